// FP64 replay of one row: the parts that one CTA does.
#pragma once

#include "engine.cuh"

namespace cospdnn {

__device__ __forceinline__ float block_max(float v, float *red) {
    v = warp_max(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (int)(blockDim.x >> 5) ? red[lane] : -INFINITY;
        v = warp_max(v);
        if (lane == 0) red[0] = v;
    }
    __syncthreads();
    return red[0];
}

// Where one row's features are in an activation buffer: feature j at
// base + j * step, or (MMA tiles) at act_index(1, ...).
struct RowPlace {
    int64_t base;
    int step;  // 0: MMA tiles
    __device__ __forceinline__ RowPlace(int layout, int N, int row) {
        if (layout == 1) {
            base = row;
            step = 0;
        } else if (layout == 0) {
            base = (int64_t)row * N;
            step = 1;
        } else {
            base = (int64_t)(row / layout) * N * layout + row % layout;
            step = layout;
        }
    }
    __device__ __forceinline__ int64_t at(int N, int j) const {
        return step ? base + (int64_t)j * step : act_index(1, N, base, j);
    }
};

// y[j] = load(j) for j0 <= j < j1 by all threads of the CTA, eight loads in
// flight per thread (a store between two loads would order them).
template <typename Load>
__device__ __forceinline__ void replay_fill_with(double *y, int j0, int j1, Load load) {
    for (int j = j0 + (int)threadIdx.x; j < j1; j += 8 * blockDim.x) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (j + u * (int)blockDim.x < j1) v[u] = load(j + u * (int)blockDim.x);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (j + u * (int)blockDim.x < j1) y[j + u * (int)blockDim.x] = v[u];
    }
}

// Input features j0..j1-1 of row `orow` into y: exact FP32 values, the bit
// planes when layer 0 of this run was counted (the compute-type copy is not
// made then), else the compute-type copy (integer inputs are exact in it).
static __device__ __noinline__ void replay_fill(const NetDev &nd, int orow, double *y, int j0, int j1) {
    const int N = nd.N, prec = nd.prec;
    if (nd.y0_f32 || (prec == COSPDNN_PREC_FP32 && !nd.st->l0_bits)) {
        const RowPlace at(nd.y0_f32 ? 0 : nd.layout, N, orow);
        const float *__restrict__ src = nd.y0_f32 ? nd.y0_f32 : (const float *)nd.y0;
        replay_fill_with(y, j0, j1, [&](int j) { return (double)__ldg(src + at.at(N, j)); });
    } else if (nd.st->l0_bits) {
        const uint32_t *__restrict__ src = nd.y0bits + (int64_t)(orow >> 5) * N;
        replay_fill_with(y, j0, j1, [&](int j) { return (__ldg(src + j) >> (orow & 31)) & 1u ? 1.0 : 0.0; });
    } else {
        const RowPlace at(nd.layout, N, orow);
        const unsigned short *__restrict__ src = (const unsigned short *)nd.y0;
        replay_fill_with(y, j0, j1, [&](int j) {
            const unsigned short h = __ldg(src + at.at(N, j));
            return prec == COSPDNN_PREC_FP16 ? (double)__half2float(__ushort_as_half(h))
                                             : (double)__bfloat162float(__ushort_as_bfloat16(h));
        });
    }
}

// A replay row in shared memory, or in global memory that other CTAs write
// (read past L1).
struct SharedRow {
    uint32_t base;
    __device__ __forceinline__ explicit SharedRow(const double *p) : base((uint32_t)__cvta_generic_to_shared(p)) {}
    __device__ __forceinline__ double operator[](uint32_t i) const {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(base + i * 8u) : "memory");
        return v;
    }
};
// The same where nothing writes the row (within replay_outputs_any, which is not
// inlined): loads may be moved.
struct ConstSharedRow {
    uint32_t base;
    __device__ __forceinline__ double operator[](uint32_t i) const {
        double v;
        asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(base + i * 8u));
        return v;
    }
};
__device__ __forceinline__ ConstSharedRow replay_const_row(SharedRow y) { return ConstSharedRow{y.base}; }
struct GlobalRow {
    const double *p;
    __device__ __forceinline__ explicit GlobalRow(const double *q) : p(q) {}
    __device__ __forceinline__ double operator[](uint32_t i) const { return __ldcg(p + i); }
};

__device__ __forceinline__ GlobalRow replay_const_row(GlobalRow y) { return y; }

// What the replay needs of one layer.  The first form is for layers of one
// power-of-two weight and 25 to 32 entries in the fullest column (replay_fast):
// eight 16-bit indices per 16-byte group, kReplayAhead groups.  The second takes any
// layer: such groups of any number for one weight value, else int32 indices and
// weights.
constexpr int kReplayAhead = 4;  // index groups (of 8 entries) of an output loaded ahead of its sum
__host__ __device__ __forceinline__ bool replay_fast(const LayerDev &lw) {
    return lw.rp_idx && !lw.rp_cnt && lw.rp_pow2 && lw.rp_groups == kReplayAhead;
}
struct ReplayLayer {
    const uint4 *idx;
    float w;
    __device__ __forceinline__ static ReplayLayer of(const LayerDev &lw) { return ReplayLayer{lw.rp_idx, lw.rp_w}; }
};
struct ReplayAnyLayer {
    const uint4 *idx;       // not NULL: one weight value
    const uint16_t *cnt;    // entries per output (NULL: padding reads the zero at y[N])
    const int32_t *ell_idx;
    const float *ell_val;
    int n;                  // groups, or entries per output
    int pow2;
    float w;
    __device__ __forceinline__ static ReplayAnyLayer of(const LayerDev &lw) {
        return ReplayAnyLayer{lw.rp_idx, lw.rp_cnt, lw.ell_idx, lw.ell_val, lw.rp_idx ? lw.rp_groups : lw.K, lw.rp_pow2, lw.rp_w};
    }
};

// The records of the layers around the current one in shared memory, layer ll
// in slot ll % 4, fetched two layers ahead by one thread (a record is two
// dependent loads away).
template <typename L>
struct ReplayRing {
    using Layer = L;
    L slot[4];
    __device__ __forceinline__ void fetch(const NetDev &nd, int ll, int l) {
        if (threadIdx.x == 0 && ll <= l) slot[ll & 3] = L::of(nd.layers[ll]);
    }
};

// The index groups of output j.
__device__ __forceinline__ void replay_load(uint4 (&q)[kReplayAhead], const ReplayLayer &rl, int N, int j) {
#pragma unroll
    for (int g = 0; g < kReplayAhead; ++g) q[g] = __ldg(rl.idx + (int64_t)g * N + j);
}

// acc + the terms of one index group, in order; kScale: each input times w,
// else the inputs alone.
template <bool kScale, typename Row>
__device__ __forceinline__ double replay_group(double acc, uint4 q, double w, Row y) {
    const uint32_t e[4] = {q.x, q.y, q.z, q.w};
    double v[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) v[t] = y[t & 1 ? e[t / 2] >> 16 : e[t / 2] & 0xFFFFu];
#pragma unroll
    for (int t = 0; t < 8; ++t) acc = __dadd_rn(acc, kScale ? __dmul_rn(w, v[t]) : v[t]);
    return acc;
}

// Output j of one layer of the first form from its input row y (N doubles and a
// zero at y[N]) in the oracle's order: over the non-zeros in ascending input
// order, multiply and add rounded separately, bias last, clamp.  q: the output's
// index groups.
//   The last group is filled up with index N, whose term is an exact +-0.  A
// power-of-two weight scales every partial sum exactly, so the sum of the
// inputs alone is rounded as the oracle's and is scaled with the bias: one
// FP64 operation per entry.
template <typename Row>
__device__ __forceinline__ double replay_output(const ReplayLayer &rl, const uint4 (&q)[kReplayAhead], Row y, double b) {
    double acc = 0.0;
#pragma unroll
    for (int g = 0; g < kReplayAhead; ++g) acc = replay_group<false>(acc, q[g], 0.0, y);
    return clamp32d(__fma_rn((double)rl.w, acc, b));
}

// Outputs j0 + thread, + threads, ... < j1 of one layer of the first form into
// z[j - j0].  q0, q1: index groups of this thread's next two outputs; those of the
// outputs after them, the next layer's (nx) first ones included, are on their way
// while an output is summed.
struct ReplayAhead {
    uint4 q0[kReplayAhead], q1[kReplayAhead];
    __device__ __forceinline__ void start(const ReplayLayer &rl, int N, int j, int j1) {
        if (j < j1) replay_load(q0, rl, N, j);
        if (j + (int)blockDim.x < j1) replay_load(q1, rl, N, j + blockDim.x);
    }
};
// Returns whether one of the thread's outputs is above tau.
__device__ __forceinline__ bool replay_outputs(const ReplayLayer &rl, const ReplayLayer &nx, bool more, ReplayAhead &a,
                                               SharedRow y, double *z, int N, int j0, int j1, double b, double tau) {
    const int nt = blockDim.x;
    bool any = false;
    for (int j = j0 + (int)threadIdx.x; j < j1; j += nt) {
        uint4 c[kReplayAhead];
#pragma unroll
        for (int g = 0; g < kReplayAhead; ++g) {
            c[g] = a.q0[g];
            a.q0[g] = a.q1[g];
        }
        if (j + 2 * nt < j1) replay_load(a.q1, rl, N, j + 2 * nt);
        const double v = replay_output(rl, c, y, b);
        z[j - j0] = v;
        any |= v > tau;
    }
    if (more) a.start(nx, N, j0 + (int)threadIdx.x, j1);
    return any;
}

// acc + the terms of M entries of one output from entry k on, loaded together.
template <int M, typename Row>
__device__ __forceinline__ double replay_pairs(double acc, const int32_t *__restrict__ ip, const float *__restrict__ wp,
                                               int N, int k, Row y) {
    int i[M];
    float w[M];
#pragma unroll
    for (int t = 0; t < M; ++t) {
        i[t] = __ldg(ip + (int64_t)(k + t) * N);
        w[t] = __ldg(wp + (int64_t)(k + t) * N);
    }
    // inputs in batches; a zero input adds an exact +-0
    constexpr int B = M < 8 ? M : 8;
#pragma unroll
    for (int u = 0; u < M; u += B) {
        double v[B];
#pragma unroll
        for (int t = 0; t < B; ++t) v[t] = y[(uint32_t)i[u + t]];
#pragma unroll
        for (int t = 0; t < B; ++t) acc = __dadd_rn(acc, __dmul_rn((double)w[u + t], v[t]));
    }
    return acc;
}
template <int M, typename Row>
__device__ __forceinline__ double replay_groups(double acc, const ReplayAnyLayer &rl, int N, int j, int g, Row y) {
    uint4 q[M];
#pragma unroll
    for (int t = 0; t < M; ++t) q[t] = __ldg(rl.idx + (int64_t)(g + t) * N + j);
#pragma unroll
    for (int t = 0; t < M; ++t)
        acc = rl.pow2 ? replay_group<false>(acc, q[t], 0.0, y) : replay_group<true>(acc, q[t], (double)rl.w, y);
    return acc;
}

// Output j of one layer of the second form.
template <typename Row>
__device__ __forceinline__ double replay_output_any(const ReplayAnyLayer &rl, Row y, int N, int j, double b) {
    double acc = 0.0;
    int k = 0;
    if (rl.idx) {
        const int n = rl.cnt ? __ldg(rl.cnt + j) / 8 : rl.n;
        for (; k + 4 <= n; k += 4) acc = replay_groups<4>(acc, rl, N, j, k, y);
        for (; k < n; ++k) acc = replay_groups<1>(acc, rl, N, j, k, y);
        if (rl.cnt) {
            const int rest = __ldg(rl.cnt + j) & 7;
            const uint16_t *e = reinterpret_cast<const uint16_t *>(rl.idx + (int64_t)k * N + j);
            for (int t = 0; t < rest; ++t) {
                const double v = y[__ldg(e + t)];
                acc = __dadd_rn(acc, rl.pow2 ? v : __dmul_rn((double)rl.w, v));
            }
        }
        return clamp32d(rl.pow2 ? __fma_rn((double)rl.w, acc, b) : __dadd_rn(acc, b));
    }
    const int32_t *ip = rl.ell_idx + j;
    const float *wp = rl.ell_val + j;
    for (; k + 16 <= rl.n; k += 16) acc = replay_pairs<16>(acc, ip, wp, N, k, y);
    for (; k + 8 <= rl.n; k += 8) acc = replay_pairs<8>(acc, ip, wp, N, k, y);
    for (; k < rl.n; ++k) acc = replay_pairs<1>(acc, ip, wp, N, k, y);
    return clamp32d(__dadd_rn(acc, b));
}

// replay_outputs for the second form: up to 16 entries, or 32 of one weight value,
// loaded together.  Each group of eight loaded and summed by itself took two to
// three times as long; a ring of groups loaded ahead was no faster than that (its
// bookkeeping per group).
template <typename Row>
__device__ __noinline__ bool replay_outputs_any(const ReplayAnyLayer &rl, Row y, double *z, int N, int j0, int j1, double b,
                                                double tau) {
    const ReplayAnyLayer l = rl;
    const auto row = replay_const_row(y);
    bool any = false;
    for (int j = j0 + (int)threadIdx.x; j < j1; j += blockDim.x) {
        const double v = replay_output_any(l, row, N, j, b);
        z[j - j0] = v;
        any |= v > tau;
    }
    return any;
}

// Doubles of one replay row: N values and the zero that padding indices read,
// rounded up to keep buffers 16-byte aligned.
__host__ __device__ __forceinline__ int replay_row_doubles(int N) { return (N + 3) / 2 * 2; }

// One layer of either form.  `ahead` is the first form's.
template <typename Row>
__device__ __forceinline__ bool replay_layer(const ReplayLayer &rl, const ReplayLayer &nx, bool more, ReplayAhead &ahead,
                                             Row y, double *z, int N, int j0, int j1, double b, double tau) {
    const ReplayLayer a = rl, c = nx;
    return replay_outputs(a, c, more, ahead, y, z, N, j0, j1, b, tau);
}
struct ReplayNoAhead {
    __device__ __forceinline__ void start(const ReplayAnyLayer &, int, int, int) {}
};
template <typename Row>
__device__ __forceinline__ bool replay_layer(const ReplayAnyLayer &rl, const ReplayAnyLayer &, bool, ReplayNoAhead &, Row y,
                                             double *z, int N, int j0, int j1, double b, double tau) {
    return replay_outputs_any(rl, y, z, N, j0, j1, b, tau);
}
template <typename L>
struct ReplayAheadOf {
    using type = ReplayNoAhead;
};
template <>
struct ReplayAheadOf<ReplayLayer> {
    using type = ReplayAhead;
};

// Recomputes input row `orow` exactly through layers 0..l with all threads of
// the CTA; y and z hold a row each (replay_row_doubles), y in shared memory,
// z too or (copy_back) in this CTA's global scratch, from where each layer's
// outputs go to y for the next layer's gathers.  Returns the one in shared
// memory with the outputs of layer l, visible to every thread; or NULL, and in `died`
// the layer, when all outputs of a layer from `since` on (and before l) are
// at most tau.
template <typename Ring>
__device__ __forceinline__ const double *replay_forward(const NetDev &nd, int since, int l, int orow, double *y,
                                                        double *z, bool copy_back, Ring &ring, int &died) {
    const int N = nd.N, tid = threadIdx.x;
    ring.fetch(nd, 0, l);
    ring.fetch(nd, 1, l);
    replay_fill(nd, orow, y, 0, N);
    if (tid == 0) y[N] = z[N] = 0.0;
    __syncthreads();
    const double b = (double)nd.bias;
    typename ReplayAheadOf<typename Ring::Layer>::type ahead;
    ahead.start(ring.slot[0], N, tid, N);
    for (int ll = 0; ll <= l; ++ll) {
        const auto &rl = ring.slot[ll & 3], &nx = ring.slot[(ll + 1) & 3];
        ring.fetch(nd, ll + 2, l);
        const bool any = replay_layer(rl, nx, ll < l, ahead, SharedRow(y), z, N, 0, N, b, (double)nd.tau);
        if (!__syncthreads_or(any) && ll >= since && ll < l) {
            died = ll;
            return nullptr;
        }
        if (copy_back) {
            replay_fill_with(y, 0, N, [&](int j) { return z[j]; });
            __syncthreads();
        } else {
            double *t = y;
            y = z;
            z = t;
        }
    }
    return y;
}

}  // namespace cospdnn
