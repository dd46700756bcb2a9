// Kernels of the device-driven layer loop.  Every kernel reads the per-net
// state (current layer, active rows, buffer roles) from device memory, so one
// captured graph serves every layer and every network; grids are fixed and
// loop over the work that the state describes.
//
// Per iteration (every live network advances one layer, those of the multi-layer
// tile kernel NetState::run layers, which that kernel classifies itself):
//   layer kernel(s)  rows 0..R-1 of IN -> OUT, per-row statistics
//   k_classify       keep / prune / uncertain from the statistics and the
//                    row's error bound
//   k_replay         exact FP64 replay of the uncertain rows
//   k_compact        stable compaction of the kept rows: new lists, state
//   k_copy_rows      kept rows of OUT -> rows 0..R'-1 of the next input
// IN = y0 for layer 0, else act[in_buf]; OUT = act[in_buf ^ 1].
#pragma once

#include <type_traits>

#include "engine.cuh"
#include "replay.cuh"

namespace cospdnn {

// ---- K0: start of a run --------------------------------------------------
__global__ void k_init_run(const NetDev *__restrict__ nets, int nnets, unsigned long long *launches,
                           int *loop_guard, int *abort_flag) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (launches) *launches = 1ull;
        *loop_guard = 0;
        *abort_flag = 0;
    }
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    for (int n = 0; n < nnets; ++n) {
        const NetDev &nd = nets[n];
        if (tid == 0) {
            nd.st->layer = 0;
            nd.st->R = nd.rows;
            nd.st->done = (nd.rows == 0 || nd.L == 0);
            nd.st->nunc = 0;
            nd.st->err = 0;
            nd.st->in_buf = 0;
            nd.st->copy_R = 0;
            nd.st->l0_bits = 0;
            nd.st->gather = 0;
            nd.st->run = 1;
            nd.st->par = 0;
            nd.st->few = nd.mt && nd.rows <= (int64_t)nd.mt_few * nd.layout;
        }
        for (int64_t l = tid; l < nd.L; l += nth) {
            nd.alive_count[l] = 0;
            nd.recheck_count[l] = 0;
        }
        for (int64_t c = tid; c < (nd.rows + kCompactChunk - 1) / kCompactChunk; c += nth) nd.ccount[c] = 0;
        for (int64_t p = tid; p < nd.rows; p += nth) {
            nd.orig[0][p] = (int32_t)p;
            nd.err[0][p] = nd.err0[p];
            nd.mx[0][p] = nd.mx0[p];
            nd.stat[3 * p] = 0u;
            nd.stat[3 * p + 1] = 0u;
            nd.stat[3 * p + 2] = 0u;
        }
    }
}

// ---- K1 (CUDA cores): one warp = 4 rows x all outputs ---------------------
// Lane j of a 32-output segment accumulates output j of 4 rows over the ELL
// entries of column j (index and weight loaded once, used for 4 rows), then
// applies bias + clamp, stores the compute-type value and folds the output into
// the row statistics (max z, error bound of the stored outputs, max output).
constexpr int kPlainRows = 4;
constexpr int kPlainThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kPlainThreads)
    k_layer_plain(const NetDev *__restrict__ nets, int nnets, int prec, unsigned long long *launches) {
    count_launch(launches);
    const int lane = threadIdx.x & 31;
    const int64_t gwarp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    int64_t total = 0;
    for (int n = 0; n < nnets; ++n) {
        const NetDev &nd = nets[n];
        if (nd.kernel != COSPDNN_KERNEL_CUDA_CORE || nd.layout != 0 || nd.prec != prec || nd.st->done) continue;
        total += (nd.st->R + kPlainRows - 1) / kPlainRows;
    }
    for (int64_t unit = gwarp; unit < total; unit += nwarps) {
        int64_t u = unit;
        int n = 0;
        for (; n < nnets; ++n) {
            const NetDev &nd = nets[n];
            if (nd.kernel != COSPDNN_KERNEL_CUDA_CORE || nd.layout != 0 || nd.prec != prec || nd.st->done) continue;
            const int64_t cnt = (nd.st->R + kPlainRows - 1) / kPlainRows;
            if (u < cnt) break;
            u -= cnt;
        }
        const NetDev &nd = nets[n];
        const int N = nd.N, l = nd.st->layer, R = nd.st->R, par = nd.st->par, ib = nd.st->in_buf;
        const LayerDev lw = nd.layers[l];
        const T *in = (const T *)(l == 0 ? nd.y0 : nd.act[ib]);
        T *out = (T *)nd.act[ib ^ 1];
        const double steps = fast_steps(nd, lw);
        const T *inrow[kPlainRows];
        T *outrow[kPlainRows];
        float ez[kPlainRows], zmax[kPlainRows], emax[kPlainRows], ymax[kPlainRows];
        bool valid[kPlainRows];
#pragma unroll
        for (int r = 0; r < kPlainRows; ++r) {
            const int p = (int)(u * kPlainRows) + r;
            valid[r] = p < R;
            const int pp = valid[r] ? p : (int)(u * kPlainRows);
            inrow[r] = in + (int64_t)pp * N;
            outrow[r] = out + (int64_t)pp * N;
            ez[r] = z_error_bound(nd.err[par][pp], nd.mx[par][pp], lw.S, lw.dW, nd.bias, steps);
            zmax[r] = -INFINITY;
            emax[r] = 0.0f;
            ymax[r] = 0.0f;
        }
        for (int j0 = 0; j0 < N; j0 += 32) {
            const int j = j0 + lane;
            if (j < N) {
                float acc[kPlainRows];
#pragma unroll
                for (int r = 0; r < kPlainRows; ++r) acc[r] = 0.0f;
                const int32_t *ip = lw.ell_idx + j;
                const float *wp = lw.ell_val + j;
                for (int k = 0; k < lw.K; ++k) {
                    const int32_t i = __ldg(ip + (int64_t)k * N);
                    const float w = __ldg(wp + (int64_t)k * N);
#pragma unroll
                    for (int r = 0; r < kPlainRows; ++r)
                        acc[r] = fmaf(w, act_traits<T>::to_f(inrow[r][i]), acc[r]);
                }
#pragma unroll
                for (int r = 0; r < kPlainRows; ++r) {
                    const float z = acc[r] + nd.bias;
                    const float c = clamp32(z);
                    const T ys = act_traits<T>::from_f(c);
                    const float yf = act_traits<T>::to_f(ys);
                    if (valid[r]) outrow[r][j] = ys;
                    zmax[r] = fmaxf(zmax[r], z);
                    ymax[r] = fmaxf(ymax[r], yf);
                    if (z > -ez[r] && z <= __fadd_ru(32.0f, ez[r])) emax[r] = fmaxf(emax[r], __fadd_ru(ez[r], fabsf(yf - c)));
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kPlainRows; ++r) {
            const float zm = warp_max(zmax[r]), em = warp_max(emax[r]), ym = warp_max(ymax[r]);
            if (lane == 0 && valid[r]) {
                const int p = (int)(u * kPlainRows) + r;
                nd.stat[3 * p] = f2ord(zm);
                nd.stat[3 * p + 1] = __float_as_uint(em);
                nd.stat[3 * p + 2] = __float_as_uint(ym);
            }
        }
    }
}

// ---- K2: keep / prune / uncertain per row ---------------------------------
// A warp takes 32 consecutive rows (all in one compaction chunk) and adds its
// sure keeps to the chunk's count; k_replay adds the re-decided ones.
__global__ void k_classify(const NetDev *__restrict__ nets, int nnets, unsigned long long *launches) {
    count_launch(launches);
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int n = 0; n < nnets; ++n) {
        const NetDev &nd = nets[n];
        if (nd.st->done) continue;
        // the multi-layer tile kernel has classified its rows itself
        if (nd.mt && !nd.st->few && !(nd.st->layer == 0 && nd.st->l0_bits)) continue;
        const int l = nd.st->layer, R = nd.st->R, par = nd.st->par;
        const LayerDev &lw = nd.layers[l];
        const double steps = fast_steps(nd, lw);
        for (int64_t base = warp * 32; base < R; base += nwarps * 32) {
            const int64_t p = base + lane;
            int8_t c = CLS_PRUNE;
            if (p < R) {
                const float zm = ord2f(nd.stat[3 * p]);
                const float ez = z_error_bound(nd.err[par][p], nd.mx[par][p], lw.S, lw.dW, nd.bias, steps);
                const double lo = (double)zm - (double)ez, hi = (double)zm + (double)ez;
                if (lo > (double)nd.tau) c = CLS_KEEP;
                else if (hi <= (double)nd.tau) c = CLS_PRUNE;
                else c = CLS_UNCERTAIN;
                nd.cls[p] = c;
                if (c == CLS_UNCERTAIN) nd.ulist[atomicAdd(&nd.st->nunc, 1)] = (int32_t)p;
            }
            const unsigned keep = __ballot_sync(0xffffffffu, c == CLS_KEEP);
            if (lane == 0 && keep) atomicAdd(&nd.ccount[base / kCompactChunk], __popc(keep));
        }
    }
}

// ---- K3: exact FP64 replay of uncertain rows ------------------------------
// Recomputes the row from its exact input through the current layer in the
// oracle's order, decides keep/prune exactly, and for kept rows overwrites the
// fast output with the FP64 values rounded to the compute type.
//   Rows of up to kReplayNarrow neurons: one CTA per row, both FP64 rows in
// shared memory.  Wider rows: a cluster of kReplayCtas CTAs per row, or one CTA
// when there are many (replay_by_cluster).  Up to
// kReplaySmemDoubles every CTA holds the whole row in shared memory, computes
// a quarter of a layer's outputs and, when all have gathered, writes them into
// every CTA's row (distributed shared memory); wider rows gather from global
// scratch (L2).  The gathers bound a layer (8 bytes of
// shared memory per entry: 17 us for a row of 16384 on one SM), so a row is
// spread over four SMs: with few uncertain rows, as in most layers, the
// others would idle.  A layer of a 16384 row takes 22000 clocks: 13500 of
// gathers and sums, 4500 of exchange, 4000 of barriers (eight CTAs per row
// were slower with many rows: each receives the whole row all the same).
//   16384 neurons BF16, 6001 rows, 998 rows re-decided in 16 layers, one B200:
// 11.6 ms with one CTA per row, 2-byte index loads and a branch per zero
// input; 4.2 ms on clusters.  1024 neurons: 5 -> 2.7 us per layer of a row.
//   k_replay_any, whole runs, against one CTA of 1024 threads per row: three weight
// values, 0 to 32 entries, BF16, 1024 neurons x 20 layers, 6561 rows in doubt 3.9 ->
// 4.1 ms, 319 rows 1.58 -> 1.56; 4096 x 10, 2988 rows 4.55 -> 4.45, 104 rows 1.52 ->
// 1.09; 16384 x 8, 1417 rows 11.0 -> 10.2; 65536 x 4, 17 rows 7.2 -> 3.6; one weight
// value that is no power of two, 20 to 44 entries, 1024 x 12, 4000 rows 2.6 -> 2.1;
// 65536 x 4, one weight value, 4 to 32 entries, 6 rows 5.7 -> 2.3.
constexpr int kReplayThreads = 512;
constexpr int kReplayAnyNarrow = 512;    // and of k_replay_any, when there are many rows
constexpr int kReplayAnyThreads = 1024;  // k_replay_any, one CTA per SM
constexpr size_t kReplayTwoSmem = 200 * 1024;  // shared memory of two CTAs of k_replay_any on an SM
constexpr int kReplayCtas = 4;             // CTAs per cluster
constexpr int kReplayNarrow = 2048;        // widest row that one CTA replays
constexpr int kReplaySmemDoubles = 27648;  // 216 KB

// Doubles of shared memory that a net of width N replays in (0: global scratch):
// two rows where one CTA replays it, or, in k_replay_any, may, and they fit.
__host__ __device__ __forceinline__ bool replay_two_rows(int N, bool any) {
    return N <= kReplayNarrow || (any && 2 * replay_row_doubles(N) <= kReplaySmemDoubles);
}
__host__ __device__ __forceinline__ int replay_smem_doubles(int N, bool any) {
    const int d = replay_two_rows(N, any) ? 2 * replay_row_doubles(N)
                                          : replay_row_doubles(N) + (N + 2 * kReplayCtas - 1) / (2 * kReplayCtas) * 2;
    return d <= kReplaySmemDoubles ? d : 0;
}

// This thread's part of what outputs y[0..n-1] of a replayed row (its last
// layer) amount to: whether one is above the threshold, and in the compute
// type the bound on their rounding and the largest value.
struct ReplaySum {
    float keep, em, ym;
};
template <typename T, typename Row>
__device__ __forceinline__ ReplaySum replay_sum_as(Row y, int n, double tau) {
    ReplaySum s{0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double yj = y[j];
        const float vf = act_traits<T>::to_f(act_traits<T>::from_d(yj));
        if (yj > tau) s.keep = 1.0f;
        s.em = fmaxf(s.em, __double2float_ru(fabs((double)vf - yj)));
        s.ym = fmaxf(s.ym, vf);
    }
    return s;
}
template <typename Row>
__device__ __noinline__ ReplaySum replay_sum(const NetDev &nd, Row y, int n, float *red) {
    const double tau = (double)nd.tau;
    ReplaySum s = nd.prec == COSPDNN_PREC_FP32   ? replay_sum_as<float>(y, n, tau)
                  : nd.prec == COSPDNN_PREC_FP16 ? replay_sum_as<__half>(y, n, tau)
                                                 : replay_sum_as<__nv_bfloat16>(y, n, tau);
    s.keep = block_max(s.keep, red);
    s.em = block_max(s.em, red);
    s.ym = block_max(s.ym, red);
    return s;
}
// Outputs j0..j1-1 (y[0..j1-j0-1]) in the compute type as row p of the layer's output.
template <typename T, typename Row>
__device__ __forceinline__ void replay_store_as(const NetDev &nd, int p, Row y, int j0, int j1) {
    const int N = nd.N;
    const RowPlace at(nd.layout, N, p);
    T *__restrict__ out = (T *)nd.act[nd.st->in_buf ^ 1];
#pragma unroll 4
    for (int j = j0 + (int)threadIdx.x; j < j1; j += blockDim.x) out[at.at(N, j)] = act_traits<T>::from_d(y[j - j0]);
}
template <typename Row>
__device__ __noinline__ void replay_store(const NetDev &nd, int p, Row y, int j0, int j1) {
    if (nd.prec == COSPDNN_PREC_FP32) replay_store_as<float>(nd, p, y, j0, j1);
    else if (nd.prec == COSPDNN_PREC_FP16) replay_store_as<__half>(nd, p, y, j0, j1);
    else replay_store_as<__nv_bfloat16>(nd, p, y, j0, j1);
}
// The row's state, by one thread.
__device__ __forceinline__ void replay_decided(const NetDev &nd, int p, bool keep, float em, float ym) {
    nd.cls[p] = keep ? CLS_KEEP : CLS_PRUNE;
    if (keep) {
        atomicAdd(&nd.ccount[p / kCompactChunk], 1);
        nd.stat[3 * p + 1] = __float_as_uint(em);
        nd.stat[3 * p + 2] = __float_as_uint(ym);
    }
}

__device__ __forceinline__ void replay_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// An uncertain row: its position, the layers of this iteration from the one
// whose decision is in doubt (after several layers at once, the tile kernel
// leaves it in stat[3 p]) to the last.
struct ReplayRow {
    int p, since, l, orow;
    __device__ __forceinline__ ReplayRow(const NetDev &nd, int p_) : p(p_) {
        const int layer = nd.st->layer, run = nd.st->run;
        l = layer + run - 1;
        since = run > 1 ? layer + (int)nd.stat[3 * p] : l;
        orow = nd.orig[nd.st->par][p];
    }
};

// Counts the row as re-decided at layer `since`, by one thread.
__device__ __forceinline__ void replay_counted(const NetDev &nd, int since) {
    atomicAdd((unsigned long long *)&nd.recheck_count[since], 1ull);
}

// Counts the row as alive after the layers of the iteration from the one in
// doubt to the one before `end` (its first layer without outputs above the
// threshold, or the iteration's last layer, whose rows k_compact counts).
__device__ __forceinline__ void replay_count(const NetDev &nd, const ReplayRow &r, int end) {
    for (int ll = r.since; ll < end; ++ll) atomicAdd((unsigned long long *)&nd.alive_count[ll], 1ull);
}

// One row by this CTA; scratch: a row in global memory for the outputs of rows
// too wide for two in shared memory.
template <bool ANY, typename Ring>
__device__ __forceinline__ void replay_alone(const NetDev &nd, int p, double *smem, double *scratch, Ring &ring,
                                             float *red) {
    const ReplayRow r(nd, p);
    const bool wide = !replay_two_rows(nd.N, ANY);
    int died = 0;
    if (threadIdx.x == 0) replay_counted(nd, r.since);
    const double *y = replay_forward(nd, r.since, r.l, r.orow, smem, wide ? scratch : smem + replay_row_doubles(nd.N), wide,
                                     ring, died);
    if (!y) {
        if (threadIdx.x == 0) {
            nd.cls[p] = CLS_PRUNE;
            replay_count(nd, r, died);
        }
    } else {
        const ReplaySum s = replay_sum(nd, SharedRow(y), nd.N, red);
        if (s.keep > 0.5f) replay_store(nd, p, SharedRow(y), 0, nd.N);
        if (threadIdx.x == 0) {
            replay_decided(nd, p, s.keep > 0.5f, s.em, s.ym);
            replay_count(nd, r, r.l);
        }
    }
    __syncthreads();  // the next row reuses the buffers
}

// The address of a shared variable in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t replay_peer(const void *local, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return a;
}
__device__ __forceinline__ void replay_push2(uint32_t at, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(at), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void replay_push1(uint32_t at, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}

// What the CTAs of a cluster tell one another at the end of a row, by rank;
// two rows take turns, so that no CTA writes what another still reads.
struct ReplayVotes {
    ReplaySum by[2][kReplayCtas];
    float any[2][kReplayCtas];  // outputs above the threshold after layer ll, in slot ll % 2
};

// The row's decision and results by the cluster; y: this CTA's outputs
// j0..j1-1.  The stores come after the barrier, which would wait for them.
template <typename Row>
__device__ __forceinline__ void replay_cluster_finish(const NetDev &nd, int p, Row y, int j0, int j1, int rank,
                                                      int turn, ReplayVotes &votes, float *red) {
    const ReplaySum s = replay_sum(nd, y, j1 - j0, red);
    ReplaySum *const mine = &votes.by[turn][rank];
    if (threadIdx.x < kReplayCtas) {
        replay_push1(replay_peer(&mine->keep, threadIdx.x), s.keep);
        replay_push1(replay_peer(&mine->em, threadIdx.x), s.em);
        replay_push1(replay_peer(&mine->ym, threadIdx.x), s.ym);
    }
    replay_cluster_sync();
    ReplaySum a{0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int r = 0; r < kReplayCtas; ++r) {
        a.keep = fmaxf(a.keep, votes.by[turn][r].keep);
        a.em = fmaxf(a.em, votes.by[turn][r].em);
        a.ym = fmaxf(a.ym, votes.by[turn][r].ym);
    }
    if (a.keep > 0.5f) replay_store(nd, p, y, j0, j1);
    if (rank == 0 && threadIdx.x == 0) replay_decided(nd, p, a.keep > 0.5f, a.em, a.ym);
    __syncthreads();  // the next row reuses this CTA's buffers
}

// Outputs per CTA of a cluster, even so that they move in pairs.
__host__ __device__ __forceinline__ int replay_share(int N) { return (N + 2 * kReplayCtas - 1) / (2 * kReplayCtas) * 2; }

// One row by the whole cluster, held in every CTA's shared memory.
template <typename Ring>
__device__ __forceinline__ void replay_wide(const NetDev &nd, int p, double *row, int rank, Ring &ring,
                                            int turn, ReplayVotes &votes, float *red) {
    const ReplayRow r(nd, p);
    const int N = nd.N, l = r.l, orow = r.orow, tid = threadIdx.x;
    const int per = replay_share(N), j0 = min(N, rank * per), j1 = min(N, j0 + per);
    const double b = (double)nd.bias;
    double *const out = row + replay_row_doubles(N);  // this CTA's outputs until all have gathered
    ring.fetch(nd, 0, l);
    ring.fetch(nd, 1, l);
    replay_fill(nd, orow, row, 0, N);
    if (tid == 0) row[N] = 0.0;
    if (rank == 0 && tid == 0) replay_counted(nd, r.since);
    __syncthreads();
    typename ReplayAheadOf<typename Ring::Layer>::type ahead;
    ahead.start(ring.slot[0], N, j0 + tid, j1);
    for (int ll = 0; ll <= l; ++ll) {
        const auto &rl = ring.slot[ll & 3], &nx = ring.slot[(ll + 1) & 3];
        ring.fetch(nd, ll + 2, l);
        const bool any = replay_layer(rl, nx, ll < l, ahead, SharedRow(row), out, N, j0, j1, b, (double)nd.tau);
        if (ll == l) break;
        if (ll >= r.since) {
            const float mine = __syncthreads_or(any) ? 1.0f : 0.0f;
            if (tid < kReplayCtas) replay_push1(replay_peer(&votes.any[ll & 1][rank], tid), mine);
        }
        replay_cluster_sync();  // every CTA has gathered (and this one's outputs are in `out`)
        if (ll >= r.since) {
            float live = 0.0f;
#pragma unroll
            for (int c = 0; c < kReplayCtas; ++c) live = fmaxf(live, votes.any[ll & 1][c]);
            if (live < 0.5f) {
                if (rank == 0 && tid == 0) {
                    nd.cls[p] = CLS_PRUNE;
                    replay_count(nd, r, ll);
                }
                replay_cluster_sync();  // every CTA has read the votes
                return;
            }
        }
        // N and the shares are even: pairs
        for (int i = tid; i < (j1 - j0) / 2; i += blockDim.x) {
            const double2 v = reinterpret_cast<const double2 *>(out)[i];
#pragma unroll
            for (int c = 0; c < kReplayCtas; ++c) replay_push2(replay_peer(row + j0 + 2 * i, c), v);
        }
        replay_cluster_sync();  // every CTA's row is complete
    }
    __syncthreads();
    if (rank == 0 && tid == 0) replay_count(nd, r, l);
    replay_cluster_finish(nd, p, SharedRow(out), j0, j1, rank, turn, votes, red);
}

// The same for rows too wide for shared memory: gathers from `scratch`, two
// rows in global memory shared by the cluster.
template <bool ANY, typename Ring>
__device__ __forceinline__ void replay_global(const NetDev &nd, int p, double *scratch, int rank, Ring &ring, int turn,
                                              ReplayVotes &votes, float *red) {
    // nets this wide take one layer per iteration
    const int N = nd.N, l = nd.st->layer + nd.st->run - 1, orow = nd.orig[nd.st->par][p], tid = threadIdx.x;
    const int per = replay_share(N), j0 = min(N, rank * per), j1 = min(N, j0 + per);
    const double b = (double)nd.bias;
    double *y = scratch, *z = scratch + replay_row_doubles(N);
    ring.fetch(nd, 0, l);
    ring.fetch(nd, 1, l);
    replay_fill(nd, orow, y, j0, j1);
    if (rank == 0 && tid == 0) {
        y[N] = z[N] = 0.0;
        replay_counted(nd, l);
    }
    replay_cluster_sync();
    for (int ll = 0; ll <= l; ++ll) {
        if constexpr (ANY) {
            replay_outputs_any(ring.slot[ll & 3], GlobalRow(y), z + j0, N, j0, j1, b, 0.0);
            ring.fetch(nd, ll + 2, l);
        } else {
            const ReplayLayer rl = ReplayLayer::of(nd.layers[ll]);
#pragma unroll 2
            for (int j = j0 + tid; j < j1; j += kReplayThreads) {
                uint4 q[kReplayAhead];
                replay_load(q, rl, N, j);
                z[j] = replay_output(rl, q, GlobalRow(y), b);
            }
        }
        replay_cluster_sync();  // every CTA's outputs are in z
        double *t = y;
        y = z;
        z = t;
    }
    replay_cluster_finish(nd, p, GlobalRow(y + j0), j0, j1, rank, turn, votes, red);
    // the next row writes its input and outputs to this CTA's own shares of the
    // two rows first, and another CTA's share of y is read by that CTA only
}

// Whether a net's uncertain rows are replayed by clusters: rows too wide for
// one CTA's shared memory always; other wide ones when there are too few for
// the CTAs.  A layer of a 16384 row takes 12 us on a cluster and 31 us on one
// SM, so one CTA per row when its rounds cost no more: with 33 clusters from 67 to
// 132 rows, and from 166 on.
__device__ __forceinline__ bool replay_by_cluster(const NetDev &nd) {
    if (nd.N <= (nd.replay_any ? kReplayAnyNarrow : kReplayNarrow)) return false;
    if (!replay_smem_doubles(nd.N, nd.replay_any)) return true;
    const int ctas = gridDim.x, clusters = ctas / kReplayCtas, cnt = nd.st->nunc;
    return 8 * ((cnt + ctas - 1) / ctas) > 3 * ((cnt + clusters - 1) / clusters);
}

// Uncertain row u of the nets of one form (replay_any) replayed by clusters or of the
// others (counted over them); false past the end.
__device__ __forceinline__ bool replay_locate(const NetDev *nets, int nnets, bool any, bool clustered, int64_t u, int &n,
                                              int &i) {
    for (n = 0; n < nnets; ++n) {
        const int cnt = nets[n].st->nunc;  // 0 of a finished net
        if (!cnt || (nets[n].replay_any != 0) != any || replay_by_cluster(nets[n]) != clustered) continue;
        if (u < cnt) {
            i = (int)u;
            return true;
        }
        u -= cnt;
    }
    return false;
}

// The nets of one form each: networks of one power-of-two weight and 25 to 32
// entries in the fullest column of every layer (the Graph Challenge's), and all
// others, whose entries take more registers per thread ahead of their sums and
// rows more threads on an SM.
template <bool ANY>
__device__ __forceinline__ void replay_rows(const NetDev *__restrict__ nets, int nnets, double *__restrict__ scratch,
                                            int scratch_row) {
    using Layer = typename std::conditional<ANY, ReplayAnyLayer, ReplayLayer>::type;
    __shared__ float red[32];
    __shared__ ReplayRing<Layer> ring;
    __shared__ ReplayVotes votes;
    extern __shared__ __align__(16) double ysm[];
    // most iterations have no row in doubt
    int work = 0;
    for (int n = threadIdx.x; n < nnets; n += blockDim.x) work |= nets[n].st->nunc;
    if (!__syncthreads_or(work)) return;
    const int rank = blockIdx.x % kReplayCtas, cluster = blockIdx.x / kReplayCtas;
    // a row of scratch per CTA: its own, or four for its cluster
    double *const own = scratch + (int64_t)blockIdx.x * scratch_row;
    double *const shared = scratch + (int64_t)cluster * kReplayCtas * scratch_row;
    int n, i;
    for (int64_t u = blockIdx.x; replay_locate(nets, nnets, ANY, false, u, n, i); u += gridDim.x)
        replay_alone<ANY>(nets[n], nets[n].ulist[i], ysm, own, ring, red);
    // the clusters' rows of scratch are their CTAs' own ones: all have finished
    replay_cluster_sync();
    int turn = 0;
    for (int64_t u = cluster; replay_locate(nets, nnets, ANY, true, u, n, i); u += gridDim.x / kReplayCtas, turn ^= 1) {
        const NetDev &nd = nets[n];
        const int p = nd.ulist[i];
        if (replay_smem_doubles(nd.N, ANY)) replay_wide(nd, p, ysm, rank, ring, turn, votes, red);
        else replay_global<ANY>(nd, p, shared, rank, ring, turn, votes, red);
    }
}
__global__ void __cluster_dims__(kReplayCtas, 1, 1) __launch_bounds__(kReplayThreads, 1)
    k_replay(const NetDev *__restrict__ nets, int nnets, double *__restrict__ scratch, int scratch_row,
             unsigned long long *launches) {
    count_launch(launches);
    replay_rows<false>(nets, nnets, scratch, scratch_row);
}
__global__ void __cluster_dims__(kReplayCtas, 1, 1) __launch_bounds__(kReplayAnyThreads, 1)
    k_replay_any(const NetDev *__restrict__ nets, int nnets, double *__restrict__ scratch, int scratch_row,
                 unsigned long long *launches) {
    count_launch(launches);
    replay_rows<true>(nets, nnets, scratch, scratch_row);
}

// Nets whose layer kernel can stage its row tiles through the compaction map
// (the one-CTA row-tile kernel, k_layer_cc): kept rows need no copy.
__device__ __forceinline__ bool gathers_rows(const NetDev &nd) {
    return nd.kernel == COSPDNN_KERNEL_CUDA_CORE && nd.layout >= 2 && !nd.cc_split;
}

// ---- K4: stable compaction + state advance + loop condition ---------------
// One CTA per chunk of kCompactChunk rows (grid = chunks of all nets at full
// size; chunks past a net's current rows are idle).  A chunk's first output
// position is the sum of the keep counts of the chunks before it.  The last
// CTA to finish advances every net's state and decides whether the graph
// loop runs again.
constexpr int kCompactThreads = kCompactChunk;

// Layers that the multi-layer tile kernel takes in the next iteration, after
// one in which `run` layers left `kept` of R rows and `rest` layers remain.
// More layers per iteration save the fixed cost of an iteration (the small
// kernels, the loop and the tiles' trip through memory); fewer drop dead rows
// earlier.  With every tile on a CTA of its own there is nothing to gain from
// dropping rows; one stop at layer 16, after the layers in which rows mostly
// die, has the rows left in doubt there replayed through 16 layers and not
// through all.  Else, if a fraction q of the rows dies per layer and a layer
// takes t, m layers waste about q m^2 t / 2, which equals the fixed cost F at
// m = sqrt(2 F / (q t)).  F (about 30 us) and the rate in t (45 FMA per clock
// and SM, FP32 23) are measured on a B200.  Rows seldom die in layer 0 and mostly in the
// next few, so q says little there: the second run is one layer, and each one
// at most doubles the one before it.
__device__ __forceinline__ int next_run(const NetDev &nd, int run, int R, int kept, int rest) {
    if ((kept + nd.layout - 1) / nd.layout <= nd.mt_ctas) return nd.st->layer < 16 ? min(rest, 16 - nd.st->layer) : rest;
    const float q = (float)(R - kept) / ((float)R * (float)run);
    const float rate = nd.prec == COSPDNN_PREC_FP32 ? 6.5e6f : 1.27e7f;  // FMA per us
    const float t = (float)kept * (float)nd.N * (float)nd.layers[0].K / rate;
    const float m = q > 0.0f ? sqrtf(60.0f / (q * t)) : (float)rest;
    return max(1, min(min(nd.st->layer == 1 ? 1 : 2 * run, rest), (int)fminf(m, 1e6f)));
}

__global__ void __launch_bounds__(kCompactThreads)
    k_compact(const NetDev *__restrict__ nets, int nnets, unsigned int *finished_ctas,
              cudaGraphConditionalHandle loop, int use_cond, int max_run, int *loop_guard,
              const DevLimits *__restrict__ limits, const int *abort_flag, unsigned long long *launches) {
    count_launch(launches);
    __shared__ int red[kCompactThreads / 32];
    __shared__ int s_base;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // locate this CTA's chunk
    int64_t u = blockIdx.x;
    int n = 0;
    for (; n < nnets; ++n) {
        const NetDev &nd = nets[n];
        const int64_t cnt = nd.st->done ? 0 : (nd.st->R + kCompactChunk - 1) / kCompactChunk;
        if (u < cnt) break;
        u -= cnt;
    }
    if (n < nnets) {
        const NetDev &nd = nets[n];
        const int R = nd.st->R, par = nd.st->par, b = (int)u;
        // kept rows of the chunks before this one
        int v = 0;
        for (int t = threadIdx.x; t < b; t += kCompactThreads) v += nd.ccount[t];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[wid] = v;
        __syncthreads();
        if (wid == 0) {
            int w = red[lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
            if (lane == 0) s_base = w;
        }
        __syncthreads();
        // stable scan of this chunk's keeps
        const int p = b * kCompactChunk + threadIdx.x;
        const int keep = (p < R && nd.cls[p] == CLS_KEEP) ? 1 : 0;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) red[wid] = __popc(m);
        __syncthreads();
        if (wid == 0) {
            int w = red[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += t;
            }
            red[lane] = w;
        }
        __syncthreads();
        if (keep) {
            const int q = s_base + (wid ? red[wid - 1] : 0) + __popc(m & ((1u << lane) - 1u));
            nd.cmap[q] = p;
            nd.orig[par ^ 1][q] = nd.orig[par][p];
            nd.err[par ^ 1][q] = __uint_as_float(nd.stat[3 * p + 1]);
            nd.mx[par ^ 1][q] = __uint_as_float(nd.stat[3 * p + 2]);
        }
        if (p < R) {
            nd.stat[3 * p] = 0u;
            nd.stat[3 * p + 1] = 0u;
            nd.stat[3 * p + 2] = 0u;
        }
    }
    // the last CTA to finish advances the states and sets the loop condition
    __syncthreads();
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(finished_ctas, 1u) + 1u == gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    int deepest = 0, live = 0;  // layers done by a network of this iteration; networks that go on (thread 0)
    for (int i = 0; i < nnets; ++i) {
        const NetDev &nd = nets[i];
        if (*(volatile int *)&nd.st->done) {
            if (threadIdx.x == 0) nd.st->copy_R = 0;
            continue;
        }
        const int run = nd.st->run, l = nd.st->layer + run - 1, R = nd.st->R, nch = (R + kCompactChunk - 1) / kCompactChunk;
        int v = 0;
        for (int t = threadIdx.x; t < nch; t += kCompactThreads) {
            v += *(volatile int32_t *)&nd.ccount[t];
            nd.ccount[t] = 0;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        __syncthreads();
        if (lane == 0) red[wid] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            int kept = 0;
            for (int w = 0; w < kCompactThreads / 32; ++w) kept += red[w];
            nd.alive_count[l] = kept;
            nd.st->nunc = 0;
            nd.st->R = kept;
            nd.st->layer = l + 1;
            const bool done = kept == 0 || l + 1 >= nd.L;
            deepest = max(deepest, l + 1);
            live |= !done;
            nd.st->done = done;
            nd.st->par ^= 1;
            const bool few = nd.mt && kept <= (int64_t)nd.mt_few * nd.layout;
            nd.st->few = few;
            nd.st->run = nd.mt && !done && !few ? min(max_run, next_run(nd, run, R, kept, nd.L - l - 1)) : 1;
            if (kept == R) {
                // nothing pruned: the output buffer is the next input as it is
                nd.st->in_buf ^= 1;
                nd.st->copy_R = 0;
                nd.st->gather = 0;
            } else if (!done && gathers_rows(nd) && (nd.mt || 2 * kept >= R)) {
                // the next layer's tile kernel reads the kept rows through cmap.
                // k_layer_cc: when most rows are kept, a tile's rows come from one
                // or two source tiles (measured on one B200: S1, 1024 neurons with
                // 90% kept per layer, 23.7 -> 22.5 ms per run; with a quarter kept
                // the staging costs more than the copy).  The multi-layer kernel
                // has the source tiles fetched into L2 ahead, so always: 4096
                // neurons, 60000 rows, a quarter kept, 1.40 -> 1.34 ms per run
                nd.st->in_buf ^= 1;
                nd.st->copy_R = 0;
                nd.st->gather = 1;
            } else {
                nd.st->copy_R = kept;  // k_copy_rows moves the kept rows
                nd.st->gather = 0;
            }
        }
    }
    if (threadIdx.x == 0) {
        *finished_ctas = 0u;
        __threadfence();
        // iterations so far, or layers where a net took several in one
        const int it = max(++*loop_guard, deepest);
        if (it > limits->max_iters || *(volatile const int *)abort_flag) {
            for (int i = 0; i < nnets; ++i) nets[i].st->err = COSPDNN_ERR_DEVICE;
            live = 0;
        }
        if (use_cond) cudaGraphSetConditional(loop, live ? 1u : 0u);
    }
}

// ---- K5: move the kept rows to the front of the next input buffer ---------
// Row q of act[in_buf] <- row cmap[q] of act[in_buf ^ 1].
// Row-major nets: one warp per row, 16-byte pieces.  MMA tiles: one warp per 8
// destination rows, whose pieces of 8 features fill whole lines.  Row tiles:
// one CTA per destination tile, see copy_tile.  Bound by memory: a kept row
// costs the lines that it shares with dropped neighbours.
//   One B200: 2553 of 7500 rows x 65536 FP16 (2-row tiles) 823 -> 152 us, 2000 of
// 6001 rows x 16384 BF16 (4-row tiles) 148 -> 44 us, 36688 of 60000 rows x 4096
// FP16 (MMA tiles) 279 -> 164 us, against one 4- or 8-byte load in flight per
// thread and one warp per MMA-tile row.
constexpr int kCopyThreads = 256;
constexpr int kCopyMaxTR = 128;

// Feature columns of COLB = 4 or 8 bytes (TR values of E each): a thread
// moves 16 bytes, 16 / COLB features of all TR rows.  For RC rows at a time it
// loads the 16 bytes of those features in the row's source tile (one vector
// load, coalesced over the threads; rows of one source tile repeat it and hit
// L1), U such pieces in flight, and picks the rows' values out.
template <typename E, int COLB, int RC, int U>
__device__ __forceinline__ void copy_tile_cols(const E *__restrict__ src, E *__restrict__ dst, int N, const int *s_map) {
    constexpr int ES = (int)sizeof(E), TR = COLB / ES, F = 16 / COLB;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
    uint4 *d4 = reinterpret_cast<uint4 *>(dst);
    const int n = N / F;
#pragma unroll 1
    for (int f = threadIdx.x; f < n; f += U * kCopyThreads) {
        uint32_t o[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) o[u][0] = o[u][1] = o[u][2] = o[u][3] = 0u;
#pragma unroll
        for (int i0 = 0; i0 < TR; i0 += RC) {
            uint4 v[U][RC];
            int off[RC];  // byte offset in the column
#pragma unroll
            for (int i = 0; i < RC; ++i) {
                const int p = s_map[i0 + i];
                off[i] = (p & (TR - 1)) * ES;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    v[u][i] = p < 0 || f + u * kCopyThreads >= n
                                  ? make_uint4(0u, 0u, 0u, 0u)
                                  : __ldg(s4 + (int64_t)(p / TR) * n + f + u * kCopyThreads);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < RC; ++i) {
                    const uint32_t w[4] = {v[u][i].x, v[u][i].y, v[u][i].z, v[u][i].w};
#pragma unroll
                    for (int g = 0; g < F; ++g) {
                        // feature g's word that holds this row's value
                        uint32_t x = w[g * (COLB / 4)];
#pragma unroll
                        for (int c = 1; c < COLB / 4; ++c) x = (off[i] >> 2) == c ? w[g * (COLB / 4) + c] : x;
                        uint32_t &d = o[u][g * (COLB / 4) + (i0 + i) * ES / 4];
                        if constexpr (ES == 4) d = x;
                        else d |= ((x >> (8 * (off[i] & 3))) & 0xFFFFu) << (16 * ((i0 + i) & 1));
                    }
                }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (f + u * kCopyThreads < n) d4[f + u * kCopyThreads] = make_uint4(o[u][0], o[u][1], o[u][2], o[u][3]);
    }
}

// Columns of 16 bytes, up to eight rows of up to eight source tiles: each
// distinct column is loaded once, one at a time (loading every row's column at
// once was slower, 186 against 164 us for 13305 of 60000 rows x 4096: four
// times the loads where rows share tiles).
template <typename E>
__device__ __forceinline__ void copy_tile_cols16(const E *__restrict__ src, E *__restrict__ dst, int N, const int *s_map) {
    constexpr int ES = (int)sizeof(E), TR = 16 / ES;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
    int pm[TR];
#pragma unroll
    for (int i = 0; i < TR; ++i) pm[i] = s_map[i];
    for (int f = threadIdx.x; f < N; f += kCopyThreads) {
        uint32_t o[4] = {0u, 0u, 0u, 0u};
        int cur = -1;
        uint4 col = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < TR; ++i) {
            const int p = pm[i];
            if (p < 0) continue;
            if (p / TR != cur) {
                cur = p / TR;
                col = __ldg(s4 + (int64_t)cur * N + f);
            }
            const int off = (p & (TR - 1)) * ES;  // byte offset in the column
            const uint32_t w = off < 8 ? (off < 4 ? col.x : col.y) : (off < 12 ? col.z : col.w);
            if constexpr (ES == 4) o[i] = w;
            else o[i / 2] |= ((w >> (8 * (off & 3))) & 0xFFFFu) << (16 * (i & 1));
        }
        reinterpret_cast<uint4 *>(dst)[f] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// Row-tile copy of destination tile q of one net (a CTA's work item): rows
// q*TR .. q*TR+TR-1 of the next input <- the kept output rows cmap[...],
// rows past the kept count zero.  The tile's row map is read once into
// shared memory.  Columns wider than 16 bytes move 16-byte destination pieces
// whose values are loaded one by one (repeats hit L1).
template <typename E>
__device__ __forceinline__ void copy_tile(const NetDev &nd, int q, int *s_map) {
    constexpr int kV = 16 / (int)sizeof(E);  // values of a 16-byte piece
    const int TR = nd.layout, N = nd.N, R = nd.st->copy_R, ib = nd.st->in_buf;
    const int lg = __ffs(TR) - 1;            // TR is a power of two
    const int colb = TR * (int)sizeof(E);    // bytes of a feature column
    const E *src = (const E *)nd.act[ib ^ 1];
    E *dst = (E *)nd.act[ib] + ((int64_t)q * N << lg);
    __syncthreads();  // the previous tile is done with s_map
    for (int r = threadIdx.x; r < TR; r += blockDim.x) {
        const int row = q * TR + r;
        s_map[r] = row < R ? nd.cmap[row] : -1;
    }
    __syncthreads();
    if (colb == 16) return copy_tile_cols16<E>(src, dst, N, s_map);
    if (colb == 8) return copy_tile_cols<E, 8, 8 / (int)sizeof(E), sizeof(E) == 2 ? 1 : 2>(src, dst, N, s_map);
    if constexpr (sizeof(E) == 2)
        if (colb == 4) return copy_tile_cols<E, 4, 2, 2>(src, dst, N, s_map);
    // wider columns: 16-byte destination pieces, P per column (a power of two)
    const int lp = lg - (__ffs(kV) - 1);  // log2 of pieces per column
    const int total = N << lp;
    for (int u = threadIdx.x; u < total; u += blockDim.x) {
        const int f = u >> lp, pc = u & ((1 << lp) - 1);
        __align__(16) E v[kV];
#pragma unroll
        for (int i = 0; i < kV; ++i) {
            const int p = s_map[pc * kV + i];
            v[i] = p < 0 ? E(0) : src[(((int64_t)(p >> lg) * N + f) << lg) + (p & (TR - 1))];
        }
        *reinterpret_cast<uint4 *>(dst + ((int64_t)f << lg) + pc * kV) = *reinterpret_cast<const uint4 *>(v);
    }
}

// MMA tiles: a warp's item is 8 destination rows (8 q8 ..) and kCopyBlocks
// feature blocks of 16; lane = (block parity, 8-feature half, row) as the
// pieces lie in memory.  Rows past the kept count stay as they are.
constexpr int kCopyBlocks = 64;
__device__ __forceinline__ void copy_mma_rows(const NetDev &nd, int q8, int fb0, int lane) {
    const int N = nd.N, nbk = N / 16, ib = nd.st->in_buf, row = 8 * q8 + (lane & 7);
    if (row >= nd.st->copy_R) return;
    const int kh = (lane >> 3) & 1, p = nd.cmap[row];
    const uint4 *src = reinterpret_cast<const uint4 *>((const char *)nd.act[ib ^ 1] + 2 * act_index(1, N, p, 8 * kh));
    uint4 *dst = reinterpret_cast<uint4 *>((char *)nd.act[ib] + 2 * act_index(1, N, row, 8 * kh));
    const int fb1 = min(nbk, fb0 + kCopyBlocks);
    // a feature block is 4 KB: 256 pieces
    for (int fb = fb0 + (lane >> 4); fb < fb1; fb += 8) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (fb + 2 * u < fb1) v[u] = __ldg(src + (int64_t)(fb + 2 * u) * 256);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (fb + 2 * u < fb1) dst[(int64_t)(fb + 2 * u) * 256] = v[u];
    }
}

__global__ void __launch_bounds__(kCopyThreads, 4)
    k_copy_rows(const NetDev *__restrict__ nets, int nnets, unsigned long long *launches) {
    count_launch(launches);
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    // row-major and MMA-tile nets, items by warp
    const int lane = threadIdx.x & 31;
    const int64_t gw = tid >> 5, nw = nth >> 5;
    auto items = [](const NetDev &nd) -> int64_t {
        const int R = nd.st->copy_R;
        return nd.layout == 0 ? R : (int64_t)((R + 7) / 8) * ((nd.N / 16 + kCopyBlocks - 1) / kCopyBlocks);
    };
    int64_t total = 0;
    for (int n = 0; n < nnets; ++n)
        if (nets[n].layout < 2) total += items(nets[n]);
    for (int64_t w = gw; w < total; w += nw) {
        int64_t u = w;
        int n = 0;
        for (; n < nnets; ++n) {
            if (nets[n].layout >= 2) continue;
            const int64_t c = items(nets[n]);
            if (u < c) break;
            u -= c;
        }
        const NetDev &nd = nets[n];
        const int N = nd.N, ib = nd.st->in_buf;
        if (nd.layout == 1) {
            const int nch = (N / 16 + kCopyBlocks - 1) / kCopyBlocks;
            copy_mma_rows(nd, (int)(u / nch), (int)(u % nch) * kCopyBlocks, lane);
            continue;
        }
        const int q = (int)u, p = nd.cmap[q], es = nd.prec == COSPDNN_PREC_FP32 ? 4 : 2;
        const int64_t pieces = (int64_t)N * es / 16;
        const uint4 *src = reinterpret_cast<const uint4 *>(nd.act[ib ^ 1]) + p * pieces;
        uint4 *dst = reinterpret_cast<uint4 *>(nd.act[ib]) + q * pieces;
#pragma unroll 4
        for (int64_t f = lane; f < pieces; f += 32) dst[f] = __ldg(src + f);
    }
    // row-tile nets: one CTA per destination tile (copy_tile)
    __shared__ int s_map[kCopyMaxTR];
    int64_t tiles = 0;
    for (int n = 0; n < nnets; ++n)
        if (nets[n].layout >= 2) tiles += (nets[n].st->copy_R + nets[n].layout - 1) / nets[n].layout;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        int64_t u = t;
        int n = 0;
        for (; n < nnets; ++n) {
            const NetDev &nd = nets[n];
            if (nd.layout < 2) continue;
            const int64_t cnt = (nd.st->copy_R + nd.layout - 1) / nd.layout;
            if (u < cnt) break;
            u -= cnt;
        }
        if (nets[n].prec == COSPDNN_PREC_FP32) copy_tile<float>(nets[n], (int)u, s_map);
        else copy_tile<uint16_t>(nets[n], (int)u, s_map);
    }
}

// ---- packed result for asynchronous copies --------------------------------
// buf: int64 count, int64 alive[L], int32 categories[rows]
__global__ void k_result_pack(const NetDev *__restrict__ nd_p, long long *__restrict__ buf) {
    const NetDev &nd = *nd_p;
    const int layer = nd.st->layer, R = nd.st->R;
    const int cnt = (nd.st->done && layer >= nd.L) ? R : 0;
    int32_t *cats = (int32_t *)(buf + 1 + nd.L);
    const int32_t *src = nd.orig[nd.st->par];
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    if (tid == 0) buf[0] = cnt;
    for (int l = tid; l < nd.L; l += nth) buf[1 + l] = nd.alive_count[l];
    for (int q = tid; q < cnt; q += nth) cats[q] = src[q];
}

}  // namespace cospdnn
