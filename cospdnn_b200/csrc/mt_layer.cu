// Multi-layer tile kernel: networks whose layers each have one weight value
// (the Graph Challenge networks), up to 7024 neurons.
//
// Rows are independent through all layers, so a CTA takes a tile of 8 rows (4
// of FP32) through as many layers as the loop state asks for (NetState::run) without
// leaving shared memory: two buffers of one tile each (feature-major, 16
// bytes of its rows per feature) take turns as input and output, the rows are
// classified after every layer by the CTA itself, and only the last layer
// writes to memory, while the CTA's next tile is copied into the buffer that
// became free.  A tile all of whose rows are dead stops early.
//
// A layer is a gather: output j of the tile is bias + w * sum of the 16-byte
// columns of its inputs.  ldmatrix.x4.trans reads 32 such columns at 32
// addresses (16 outputs x 2 steps) and delivers them as the B operand (32 x 8
// rows) of one mma.sp.m16n8k32 whose sparse A operand is constant: row m of
// the 16 x 32 matrix holds w at columns m and 16 + m, so accumulator row m
// adds w * column(m, step) for both steps.  The arithmetic is FP16/BF16
// products, exact in FP32, and FP32 sums, as on the CUDA cores.  Per 256
// multiply-adds a warp issues one ldmatrix, one MMA and about three address
// instructions, where the CUDA-core kernel (k_layer_cc) issues about 20; the
// entry order (order_entries, 8 residues) keeps every ldmatrix phase free of
// bank conflicts.  FP32 tiles sum on the CUDA cores: a lane per output, one
// 16-byte shared load and two packed FMAs per entry, in the same tiles and
// loop over layers.
//
// What bounds it: the shared-memory data pipe.  A gather is four 128-byte
// wavefronts per 256 multiply-adds (64 per clock and SM at most) and the entry
// loads pass through the same pipe (12% of it); at 4096 neurons it is 80% busy
// with 39 multiply-adds per clock and SM, 92% (52) in a loop of nothing else;
// FP32 at 1024 neurons 87%.
// One barrier per layer: the rows are decided by one warp while the others
// are in the next layer or tile.
//   Measured on one B200, FP16, XOR-mask weights, before (one CUDA-core layer,
// classification, replay and compaction launch per layer) and now:
//   4096 neurons, 60000 rows, one layer           0.731 -> 0.676 ms
//   4096 neurons x 24 layers, 8000 rows, half live   6.3 -> 2.2 ms
//   1024 neurons x 120 layers, 24000 rows live      10.5 -> 6.4 ms
//   1024 neurons x 120 layers, 64 rows               3.2 -> 0.61 ms
// FP32:
//   1024 neurons x 120 layers, 60000 rows dying     1.02 -> 0.75 ms
//   1024 neurons x 120 layers, 24000 rows live      17.6 -> 10.9 ms
//   1024 neurons x 120 layers, 64 rows               3.2 -> 0.61 ms
//   4096 neurons, 60000 rows, one layer             1.42 -> 1.23 ms
#include <algorithm>
#include <cmath>

#include "cc_layer.cuh"
#include "mt_layer.cuh"

namespace cospdnn {
namespace {

constexpr int kMtZero = kCcZeroCols;          // zero columns after a tile's N inputs
constexpr size_t kMtSmemMax = 220 * 1024;     // two tiles; the rest holds the nets' state
constexpr int kMtNets = 24;                   // networks whose state a CTA holds at a time

constexpr size_t mt_tile_bytes(int N) { return (size_t)(N + kMtZero) * 16; }

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldmatrix4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

// d += A * B: A 16 x 32 sparse (a, meta), B 32 x 8 (b).
__device__ __forceinline__ void mma_sp(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[4], uint32_t meta,
                                       __half) {
    asm(
        "mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9, %10, %11}, {%0, %1, %2, %3}, %12, 0x0;"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(meta));
}
__device__ __forceinline__ void mma_sp(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[4], uint32_t meta,
                                       __nv_bfloat16) {
    asm(
        "mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9, %10, %11}, {%0, %1, %2, %3}, %12, 0x0;"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(meta));
}

// Of row m = lane / 4 + 8 h of A, this thread holds the two kept values of the
// 4-column chunk lane % 4 (and of chunk 4 + lane % 4, where the same row has
// its second non-zero).  The non-zero of the row is column m of the first 16:
// chunk m / 4, position m % 4.  Its pair is {position, 3}, or {0, 3} with the
// value second when the position is 3; every other chunk keeps {0, 1}, zeros.
__device__ __forceinline__ uint32_t mt_meta(int lane) {
    uint32_t meta = 0u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int m = lane / 4 + 8 * h;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t pos = m % 4 < 3 ? (uint32_t)(m % 4) : 0u;
            meta |= (c == m / 4 ? pos | 0xCu : 0x4u) << (16 * h + 4 * c);
        }
    }
    return meta;
}
__device__ __forceinline__ uint32_t mt_weight(int lane, int h, uint32_t wbits) {
    const int m = lane / 4 + 8 * h;
    return m / 4 != lane % 4 ? 0u : m % 4 < 3 ? wbits & 0xFFFFu : wbits << 16;
}

__device__ __forceinline__ bool mt_net(const NetDev &nd, int prec) {
    return nd.mt && nd.prec == prec && !nd.st->done && !nd.st->few && !(nd.st->layer == 0 && nd.st->l0_bits);
}

// What the kernel needs of a network, fixed during a launch and held in shared
// memory: read from the descriptors for every tile, the dependent loads cost
// a third of a tile's time (4096 neurons, one layer).
struct MtNet {
    const MtLayer *lay;  // record of the first layer of this launch
    const uint4 *in;     // its input tiles
    uint4 *out;          // output tiles of the last layer
    const int32_t *cmap; // not NULL: rows come through the compaction map
    const float *err, *mx;
    unsigned long long *alive;  // rows kept after each layer of this launch
    int8_t *cls;
    uint32_t *stat;
    int32_t *ccount;
    const NetDev *nd;
    int N, R, tiles, run;
    int plain0;  // the first layer reads non-finite inputs (layer 0)
    float bias, tau;
};

// Rows per tile: 16-byte feature columns.
template <typename T>
constexpr int mt_rows() {
    return 16 / (int)sizeof(T);
}

// The net and tile of item u of the CTA's nets; false past the end.
__device__ __forceinline__ bool mt_locate(const MtNet *nets, int n, int64_t u, int &net, int &tile) {
    for (int i = 0; i < n; ++i) {
        if (u < nets[i].tiles) {
            net = i;
            tile = (int)u;
            return true;
        }
        u -= nets[i].tiles;
    }
    return false;
}

// Bound on |z_fast - z_FP64| (z_error_bound) in FP32 rounded up.
__device__ __forceinline__ float mt_error_bound(float e, float m, const MtLayer &ml, float bias) {
    const float ab = fabsf(bias);
    const float t = __fadd_ru(__fmul_ru(ml.S, m), ab);
    const float t64 = __fadd_ru(__fmul_ru(ml.S, __fadd_ru(m, e)), ab);
    float ez = __fadd_ru(__fmul_ru(ml.S, e), __fmul_ru(ml.dW, __fadd_ru(m, e)));
    ez = __fmaf_ru(__fmul_ru(ml.steps, 5.9604645e-08f), t, ez);  // steps * 2^-24
    return __fmaf_ru(4.4408925e-15f, t64, ez);                   // over 40 * 2^-53
}

// One chunk of a group's entries, up to 32 steps: two 16-byte blocks per lane.
__device__ __forceinline__ void mt_load(uint4 (&q)[2], const uint4 *__restrict__ p, bool second) {
    q[0] = __ldg(p);
    if (second) q[1] = __ldg(p + 32);
}

// Gathers of 32 columns (two steps of 16 outputs) and their MMAs, kBlocks x 8
// of them; the next gather is issued ahead of an MMA.  `next` loads the next
// chunk into q once the addresses are taken from it.
template <typename T, int kBlocks, typename Next>
__device__ __forceinline__ void mt_chunk(float (&c)[4], uint4 (&q)[2], uint32_t base, const uint32_t (&a)[4],
                                         uint32_t meta, Next next) {
    constexpr int n = 8 * kBlocks;
    uint32_t addr[n];
#pragma unroll
    for (int h = 0; h < kBlocks; ++h) {
        const uint32_t e[4] = {q[h].x, q[h].y, q[h].z, q[h].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            addr[8 * h + 2 * i] = base + ((e[i] & 0xFFFFu) << 4);
            addr[8 * h + 2 * i + 1] = base + ((e[i] >> 16) << 4);
        }
    }
    next();
    uint32_t y[2][4];
    ldmatrix4t(y[0], addr[0]);
#pragma unroll
    for (int i = 0; i < n; ++i) {
        if (i + 1 < n) ldmatrix4t(y[(i + 1) & 1], addr[i + 1]);
        mma_sp(c, a, y[i & 1], meta, T());
    }
}

// {lo, hi} rounded to the compute type and clamped to [0, 32] (rounding is
// monotone and 32 representable, so the order does not matter).
__device__ __forceinline__ uint32_t clamp_pack(float lo, float hi, __half) {
    uint32_t d;
    asm("{\n\t.reg .b32 t;\n\tcvt.rn.relu.f16x2.f32 t, %1, %2;\n\tmin.f16x2 %0, t, %3;\n\t}"
        : "=r"(d)
        : "f"(hi), "f"(lo), "r"(0x50005000u));
    return d;
}
__device__ __forceinline__ uint32_t clamp_pack(float lo, float hi, __nv_bfloat16) {
    uint32_t d;
    asm("{\n\t.reg .b32 t;\n\tcvt.rn.relu.bf16x2.f32 t, %1, %2;\n\tmin.bf16x2 %0, t, %3;\n\t}"
        : "=r"(d)
        : "f"(hi), "f"(lo), "r"(0x42004200u));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3_abs(float a, float b, float c) {
    float d;
    asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// {x - 16, y - 16} in one packed instruction
__device__ __forceinline__ void minus16(float x, float y, float &u, float &v) {
    asm("{\n\t.reg .b64 a, m;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 m, {%4, %4};\n\t"
        "add.rn.f32x2 a, a, m;\n\t"
        "mov.b64 {%0, %1}, a;\n\t}"
        : "=f"(u), "=f"(v)
        : "f"(x), "f"(y), "f"(-16.0f));
}

// Outputs gq and 8 + gq of a group for rows 2 q4, 2 q4 + 1: row statistics,
// clamp, store at o and o + 8 columns; the sums start again at the bias.
template <typename T>
__device__ __forceinline__ void mt_put(float (&c)[4], float bias, float (&zmax)[2], float (&zdist)[2], uint32_t *o) {
    float u[4];
    minus16(c[0], c[1], u[0], u[1]);
    minus16(c[2], c[3], u[2], u[3]);
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        zmax[v] = max3(zmax[v], c[v], c[2 + v]);
        zdist[v] = min3_abs(zdist[v], u[v], u[2 + v]);
    }
    o[0] = clamp_pack(c[0], c[1], T());
    o[32] = clamp_pack(c[2], c[3], T());
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = bias;
}

// One layer of a tile by one warp: groups warp, warp + kWarps, ... of 16
// outputs; q holds the first chunk of entries.
template <typename T, int kWarps>
__device__ __forceinline__ void mt_layer(const uint4 *__restrict__ w, int nb, uint4 (&q)[2], int ngroups, int warp,
                                         uint32_t base, const uint32_t (&a)[4], uint32_t meta, float bias,
                                         float (&zmax)[2], float (&zdist)[2], uint32_t *o) {
    const int mine = (ngroups - warp + kWarps - 1) / kWarps;  // <= 0: none
    float c[4] = {bias, bias, bias, bias};
    const uint4 *p = w + (int64_t)warp * nb * 32;
    if (nb == 2) {  // 32 entries per output: a group is one chunk
        for (int i = 1; i <= mine; ++i) {
            if (i < mine) p += kWarps * 64;
            mt_chunk<T, 2>(c, q, base, a, meta, [&] { mt_load(q, p, true); });
            mt_put<T>(c, bias, zmax, zdist, o);
            o += kWarps * 64;
        }
        return;
    }
    for (int i = 0; i < mine; ++i) {
        for (int b = 0; b < nb; b += 2) {
            // the chunk after this one
            const bool end = b + 2 >= nb;
            const int nxt = end ? 0 : b + 2;
            if (end && i + 1 < mine) p += (int64_t)kWarps * nb * 32;
            auto next = [&] { mt_load(q, p + nxt * 32, nxt + 1 < nb); };
            if (b + 1 < nb) mt_chunk<T, 2>(c, q, base, a, meta, next);
            else mt_chunk<T, 1>(c, q, base, a, meta, next);
        }
        mt_put<T>(c, bias, zmax, zdist, o);
        o += kWarps * 64;
    }
}

// acc += w * the FP32 pair (y0, y1): two IEEE FMAs in one packed instruction.
__device__ __forceinline__ void mt_ffma2(float2 &acc, float w, uint32_t y0, uint32_t y1) {
    asm("{\n\t.reg .b64 d, x, w;\n\t"
        "mov.b64 d, {%0, %1};\n\t"
        "mov.b64 x, {%2, %3};\n\t"
        "mov.b64 w, {%4, %4};\n\t"
        "fma.rn.f32x2 d, w, x, d;\n\t"
        "mov.b64 {%0, %1}, d;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "r"(y0), "r"(y1), "f"(w));
}

// One layer of an FP32 tile (4 rows) by one warp: groups of 32 outputs, one per
// lane; an entry is one 16-byte shared load (the input's 4 rows) and two packed
// FMAs.  q holds the first chunk of 16 entries; nb is even.
template <int kWarps>
__device__ __forceinline__ void mt_layer_f32(const uint4 *__restrict__ w, int nb, uint4 (&q)[2], int ngroups, int warp,
                                             uint32_t base, float weight, float bias, float (&zmax)[4],
                                             float (&zdist)[4], uint4 *o) {
    const int mine = (ngroups - warp + kWarps - 1) / kWarps;  // <= 0: none
    const uint4 *p = w + (int64_t)warp * nb * 32;
    for (int i = 0; i < mine; ++i) {
        float2 a = make_float2(0.0f, 0.0f), b = a;
        for (int c = 0; c < nb; c += 2) {
            const uint32_t e[8] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w};
            // the chunk after this one
            const bool end = c + 2 >= nb;
            if (end && i + 1 < mine) p += (int64_t)kWarps * nb * 32;
            mt_load(q, p + (end ? 0 : c + 2) * 32, true);
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                uint32_t y[4];
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(y[0]), "=r"(y[1]), "=r"(y[2]), "=r"(y[3])
                             : "r"(base + ((t & 1 ? e[t / 2] >> 16 : e[t / 2] & 0xFFFFu) << 4)));
                mt_ffma2(a, weight, y[0], y[1]);
                mt_ffma2(b, weight, y[2], y[3]);
            }
        }
        const float z[4] = {a.x + bias, a.y + bias, b.x + bias, b.y + bias};
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            zmax[v] = fmaxf(zmax[v], z[v]);
            zdist[v] = fminf(zdist[v], fabsf(z[v] - 16.0f));
        }
        *o = make_uint4(__float_as_uint(clamp32(z[0])), __float_as_uint(clamp32(z[1])), __float_as_uint(clamp32(z[2])),
                        __float_as_uint(clamp32(z[3])));
        o += kWarps * 32;
    }
}

// Layer 0 of an input with infinities or NaN: 0 * inf in the MMA would reach
// outputs that do not read it, so each output sums its own inputs.
// Returns the thread's {max z, max z, min |z - 16|, min |z - 16|} of its two rows.
template <typename T, int kWarps>
__device__ __noinline__ float4 mt_layer_plain(const NetDev &nd, const LayerDev &lw, const unsigned char *src,
                                              unsigned char *dst) {
    const int lane = threadIdx.x & 31, q4 = lane & 3;
    float zmax[2] = {-INFINITY, -INFINITY}, zdist[2] = {INFINITY, INFINITY};
    for (int j = (threadIdx.x >> 5) * 8 + (lane >> 2); j < nd.N; j += kWarps * 8) {
        float s[2] = {0.0f, 0.0f};
        for (int t = 0; t < lw.K; ++t) {
            const float w = act_traits<T>::to_f(act_traits<T>::from_f(__ldg(lw.ell_val + (int64_t)t * nd.N + j)));
            if (w == 0.0f) continue;  // padding
            const T *y = reinterpret_cast<const T *>(src) + (int64_t)__ldg(lw.ell_idx + (int64_t)t * nd.N + j) * kMtRows;
#pragma unroll
            for (int v = 0; v < 2; ++v) s[v] = fmaf(w, act_traits<T>::to_f(y[2 * q4 + v]), s[v]);
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const float z = s[v] + nd.bias;
            zmax[v] = fmaxf(zmax[v], z);
            zdist[v] = fminf(zdist[v], fabsf(z - 16.0f));
            reinterpret_cast<T *>(dst)[j * kMtRows + 2 * q4 + v] = act_traits<T>::from_f(clamp32(z));
        }
    }
    return make_float4(zmax[0], zmax[1], zdist[0], zdist[1]);
}

template <typename T, int NT, int OCC>
__global__ void __launch_bounds__(NT, OCC)
    k_layers_mt(const NetDev *__restrict__ nets, int nnets, int prec, unsigned long long *launches) {
    count_launch(launches);
    constexpr int kWarps = NT / 32, kRows = mt_rows<T>();
    constexpr bool kMma = sizeof(T) == 2;
    constexpr int kGroup = kMma ? 16 : 32;  // outputs per group of a warp
    extern __shared__ __align__(16) unsigned char mt_smem[];
    // row statistics of layer k in slot k % 3 (one is read, one filled, one cleared)
    __shared__ uint32_t s_zmax[3][kRows], s_zdist[3][kRows];
    // the rows of an item and of the next one: error bound and max of the
    // inputs, surely alive and undecided rows, the layer since when
    __shared__ float s_e[2][kRows], s_m[2][kRows];
    __shared__ int s_alive[2], s_pend[2], s_since[kRows], s_map[kRows];
    __shared__ int s_dead[2];  // no row surely alive after layer k, in slot k % 2
    // records of the layers around the current one
    __shared__ __align__(16) MtLayer s_lay[4];
    __shared__ MtNet s_nets[kMtNets];
    // the shuffle tells the compiler that the warp's number is uniform
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int q4 = lane & 3, gq = lane >> 2;
    const uint32_t meta = mt_meta(lane);
    uint32_t dyn;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    // the two buffers are a fixed distance apart whatever the net (two tiles of
    // the widest net fit), so a tile staged for the next net stays in place
    auto buf = [&](int i) { return mt_smem + (i ? dyn / 2 : 0u); };
    // networks in groups of kMtNets
    for (int n0 = 0; n0 < nnets; n0 += kMtNets) {
        __syncthreads();  // the previous group is done with s_nets
        if (threadIdx.x < kMtNets) {
            MtNet w{};
            const int n = n0 + threadIdx.x;
            if (n < nnets && mt_net(nets[n], prec)) {
                const NetDev &nd = nets[n];
                const NetState &st = *nd.st;
                w.lay = nd.mt + st.layer;
                w.in = reinterpret_cast<const uint4 *>(st.layer == 0 ? nd.y0 : nd.act[st.in_buf]);
                w.out = reinterpret_cast<uint4 *>(nd.act[st.in_buf ^ 1]);
                w.cmap = st.gather ? nd.cmap : nullptr;
                w.err = nd.err[st.par];
                w.mx = nd.mx[st.par];
                w.alive = reinterpret_cast<unsigned long long *>(nd.alive_count + st.layer);
                w.cls = nd.cls;
                w.stat = nd.stat;
                w.ccount = nd.ccount;
                w.nd = &nd;
                w.N = nd.N;
                w.R = st.R;
                w.tiles = (st.R + kRows - 1) / kRows;
                w.run = st.run;
                w.plain0 = kMma && st.layer == 0 && *nd.y0nonfin;
                w.bias = nd.bias;
                w.tau = nd.tau;
            }
            s_nets[threadIdx.x] = w;
        }
        __syncthreads();
        int64_t item = blockIdx.x;
        int net = 0, tile = 0;
        if (!mt_locate(s_nets, kMtNets, item, net, tile)) continue;
        int cur = 0;         // buffer that holds (or gets) the item's tile
        int it = 0;          // item parity: slot of the rows' state
        int lb = 0;          // slot of the item's first layer record
        int zs = 0;          // statistics slot of the current layer
        bool ready = false;  // the previous item left this one's tile and state in place
        uint4 q[2];          // the warp's first chunk of entries in the layer at hand
        // state of rows of tile t of net w into slot i, by eight threads
        auto put_rows = [&](const MtNet &w, int t, int i, float e, float m) {
            if (threadIdx.x < kRows) {
                s_e[i][threadIdx.x] = e;
                s_m[i][threadIdx.x] = m;
            }
            if (threadIdx.x == 0) {
                s_alive[i] = (1 << min(kRows, w.R - t * kRows)) - 1;
                s_pend[i] = 0;
            }
        };
        auto row_value = [&](const float *v, const MtNet &w, int t) {
            const int p = t * kRows + (int)threadIdx.x;
            return threadIdx.x < kRows && p < w.R ? v[p] : 0.0f;
        };
        auto stage_record = [&](const MtNet &w, int k, int slot) {  // by two threads
            if (k < w.run && threadIdx.x < 2)
                reinterpret_cast<uint4 *>(&s_lay[slot & 3])[threadIdx.x] =
                    __ldg(reinterpret_cast<const uint4 *>(w.lay + k) + threadIdx.x);
        };
        auto start_feed = [&](const uint4 *w, int nb, int ngroups) {
            if (warp < ngroups) mt_load(q, w + (int64_t)warp * nb * 32 + lane, nb > 1);
        };
        auto stage_tile = [&](const MtNet &w, int t, int b) {
            const uint4 *src = w.in + (int64_t)t * w.N;
            const uint32_t dst = smem_u32(buf(b));
#pragma unroll 4
            for (int f = threadIdx.x; f < w.N; f += NT)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + f * 16), "l"(src + f) : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (;;) {
            const MtNet &mn = s_nets[net];
            const int N = mn.N, R = mn.R, ngroups = N / kGroup, run = mn.run;
            const float bias = mn.bias;
            const int64_t next_item = item + gridDim.x;
            int next_net = net, next_tile = 0;
            const bool more = mt_locate(s_nets, kMtNets, next_item, next_net, next_tile);
            if (!ready) {
                // ---- the tile, its rows' state, layer records and zero columns
                const float e = row_value(mn.err, mn, tile), m = row_value(mn.mx, mn, tile);
                start_feed(mn.lay->w, mn.lay->nb, ngroups);
                __syncthreads();  // the previous item is done with the buffers and states
                if (mn.cmap) {
                    // through the compaction map: row r of the tile <- row s_map[r]
                    if (threadIdx.x < kRows) {
                        const int p = tile * kRows + threadIdx.x;
                        s_map[threadIdx.x] = p < R ? mn.cmap[p] : -1;
                    }
                    __syncthreads();
                    int pm[kRows];
#pragma unroll
                    for (int r = 0; r < kRows; ++r) pm[r] = s_map[r];
                    uint4 *dst = reinterpret_cast<uint4 *>(buf(cur));
#pragma unroll 1
                    for (int f = threadIdx.x; f < N; f += NT) {
                        uint4 col[kRows];
#pragma unroll
                        for (int r = 0; r < kRows; ++r)
                            col[r] = pm[r] < 0 ? make_uint4(0u, 0u, 0u, 0u) : __ldg(mn.in + (int64_t)(pm[r] / kRows) * N + f);
                        uint32_t v[kRows];
#pragma unroll
                        for (int r = 0; r < kRows; ++r) {
                            const int o = (pm[r] & (kRows - 1)) * (int)sizeof(T);  // byte offset in the column
                            const uint32_t w = o < 8 ? (o < 4 ? col[r].x : col[r].y) : (o < 12 ? col[r].z : col[r].w);
                            v[r] = kMma ? (w >> (8 * (o & 3))) & 0xFFFFu : w;
                        }
                        if constexpr (kMma)
                            dst[f] = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
                        else
                            dst[f] = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                } else {
                    stage_tile(mn, tile, cur);
                }
                put_rows(mn, tile, it, e, m);
                lb = 0;
                stage_record(mn, 0, 0);
                stage_record(mn, 1, 1);
                if (threadIdx.x < kMtZero) {
                    reinterpret_cast<uint4 *>(buf(0))[N + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
                    reinterpret_cast<uint4 *>(buf(1))[N + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
                }
                zs = 0;
                if (threadIdx.x < 2 * kRows) {
                    s_zmax[threadIdx.x / kRows][threadIdx.x % kRows] = 0u;
                    s_zdist[threadIdx.x / kRows][threadIdx.x % kRows] = 0x7F800000u;  // +inf
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
            }
            ready = false;
            for (int k = 0; k < run; ++k) {
                const bool last = k + 1 == run;
                const MtLayer &ml = s_lay[(lb + k) & 3];
                unsigned char *const src = buf(cur);
                // the last layer writes the output buffer in memory
                unsigned char *const dst = last ? (unsigned char *)(mn.out + (int64_t)tile * N) : buf(cur ^ 1);
                float next_e = 0.0f, next_m = 0.0f;
                const uint4 *feed = nullptr;
                int feed_nb = 0;
                bool prep = false;  // the next item is made ready during this layer
                if (!last) {
                    stage_record(mn, k + 2, lb + k + 2);
                } else if (more) {
                    // the CTA's next tile into the free buffer while this layer
                    // computes, and all that its start needs
                    const MtNet &nn = s_nets[next_net];
                    if (nn.cmap && threadIdx.x < kRows) {
                        // rows through the compaction map: their source tiles into L2
                        const int p = next_tile * kRows + threadIdx.x, src = p < nn.R ? nn.cmap[p] / kRows : -1;
                        const int before = __shfl_up_sync((1u << kRows) - 1u, src, 1);
                        if (src >= 0 && (threadIdx.x == 0 || src != before))
                            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(nn.in + (int64_t)src * nn.N),
                                         "r"(nn.N * 16)
                                         : "memory");
                    }
                    prep = !nn.cmap && nn.N == N;
                    if (prep) {
                        next_e = row_value(nn.err, nn, next_tile);
                        next_m = row_value(nn.mx, nn, next_tile);
                        feed = nn.lay->w;
                        feed_nb = nn.lay->nb;
                        stage_tile(nn, next_tile, cur ^ 1);
                        stage_record(nn, 0, lb + run);
                        stage_record(nn, 1, lb + run + 1);
                    }
                }

                // ---- the layer: groups of 16 outputs per warp
                const uint32_t base = smem_u32(src);
                // the thread's rows (2 q4 and 2 q4 + 1; FP32: all): max z, min |z - 16|
                constexpr int kMine = kMma ? 2 : 4;
                float zmax[kMine], zdist[kMine];
#pragma unroll
                for (int v = 0; v < kMine; ++v) {
                    zmax[v] = -INFINITY;
                    zdist[v] = INFINITY;
                }
                if constexpr (!kMma) {
                    mt_layer_f32<kWarps>(ml.w + lane, ml.nb, q, ngroups, warp, base, __uint_as_float(ml.wbits), bias, zmax,
                                         zdist, reinterpret_cast<uint4 *>(dst) + warp * 32 + lane);
                } else if (k == 0 && mn.plain0) {
                    const float4 z = mt_layer_plain<T, kWarps>(*mn.nd, mn.nd->layers[0], src, dst);
                    zmax[0] = z.x;
                    zmax[1] = z.y;
                    zdist[0] = z.z;
                    zdist[1] = z.w;
                } else {
                    // A repeats itself; `zero` (from memory) keeps the compiler from seeing
                    // that, so that the four registers stay one operand (else it is put
                    // together again for every MMA: 3.8 moves per MMA)
                    const uint32_t zero = ml.zero;
                    const uint32_t a[4] = {mt_weight(lane, 0, ml.wbits), mt_weight(lane, 1, ml.wbits),
                                           mt_weight(lane, 0, ml.wbits) ^ zero, mt_weight(lane, 1, ml.wbits) ^ zero};
                    mt_layer<T, kWarps>(ml.w + lane, ml.nb, q, ngroups, warp, base, a, meta, bias, zmax, zdist,
                                        reinterpret_cast<uint32_t *>(dst) + (warp * 16 + gq) * 4 + q4);
                }
                // the next layer's (or tile's) first entries, on their way during the barrier
                if (!last) start_feed(s_lay[(lb + k + 1) & 3].w, s_lay[(lb + k + 1) & 3].nb, ngroups);
                else if (prep) start_feed(feed, feed_nb, ngroups);
                // ---- row statistics
                if constexpr (!kMma) {
#pragma unroll
                    for (int v = 0; v < kMine; ++v) {
                        const uint32_t m = __reduce_max_sync(0xffffffffu, f2ord(zmax[v]));
                        const uint32_t d = __reduce_min_sync(0xffffffffu, __float_as_uint(zdist[v]));  // >= 0
                        if (lane == v) {
                            atomicMax(&s_zmax[zs][v], m);
                            atomicMin(&s_zdist[zs][v], d);
                        }
                    }
                } else {
#pragma unroll
                    for (int v = 0; v < kMine; ++v) {
#pragma unroll
                        for (int off = 4; off < 32; off <<= 1) {
                            zmax[v] = fmaxf(zmax[v], __shfl_xor_sync(0xffffffffu, zmax[v], off));
                            zdist[v] = fminf(zdist[v], __shfl_xor_sync(0xffffffffu, zdist[v], off));
                        }
                        if (gq == 0) {
                            atomicMax(&s_zmax[zs][2 * q4 + v], f2ord(zmax[v]));
                            atomicMin(&s_zdist[zs][2 * q4 + v], __float_as_uint(zdist[v]));  // >= 0
                        }
                    }
                }
                if (prep) {
                    put_rows(s_nets[next_net], next_tile, it ^ 1, next_e, next_m);
                    asm volatile("cp.async.wait_all;" ::: "memory");
                }
                __syncthreads();
                // the state that an undecided row (since layer s_since[r] of the run) or
                // a pruned one leaves behind, by thread r
                auto leave = [&](int r, bool undecided) {
                    const int p = tile * kRows + r;
                    if (p >= R) return;
                    mn.cls[p] = undecided ? CLS_UNCERTAIN : CLS_PRUNE;
                    if (undecided) {
                        mn.stat[3 * p] = (uint32_t)s_since[r];
                        mn.nd->ulist[atomicAdd(&mn.nd->st->nunc, 1)] = p;
                    }
                };
                if (!last && k > 0 && s_dead[(k - 1) & 1]) {
                    // no row was surely alive after the layer before (the outputs of
                    // undecided rows come from their replay)
                    if (threadIdx.x < kRows) leave(threadIdx.x, (s_pend[it] >> threadIdx.x) & 1);
                    break;
                }
                // ---- keep, prune or undecided (k_classify's rule), by one warp while the
                // others go on; undecided rows go on until the last layer of the run and
                // are then replayed from the layer where the doubt began
                if (threadIdx.x < kRows) {
                    const int r = threadIdx.x, clear = zs == 0 ? 2 : zs - 1;  // the slot after next
                    const float zm = ord2f(s_zmax[zs][r]), zd = __uint_as_float(s_zdist[zs][r]);
                    s_zmax[clear][r] = 0u;
                    s_zdist[clear][r] = 0x7F800000u;
                    const float ez = mt_error_bound(s_e[it][r], s_m[it][r], ml, bias);
                    float em, ym;
                    row_stats<T>(zm, zd, ez, em, ym);
                    s_e[it][r] = em;
                    s_m[it][r] = ym;
                    const int alive = s_alive[it], pend = s_pend[it];
                    const bool undec = (pend >> r) & 1, was = (alive >> r) & 1;
                    const bool keep = was && __fsub_rd(zm, ez) > mn.tau;
                    const bool unc = was && !keep && !(__fadd_ru(zm, ez) <= mn.tau);
                    if (unc) s_since[r] = k;
                    constexpr unsigned kMask = (1u << kRows) - 1u;
                    const unsigned km = __ballot_sync(kMask, keep), um = __ballot_sync(kMask, unc);
                    if (r == 0) {
                        s_alive[it] = (int)km;
                        s_pend[it] = pend | (int)um;
                        s_dead[k & 1] = km == 0;
                        // undecided rows are counted by their replay
                        if (!last && km) atomicAdd(mn.alive + k, (unsigned long long)__popc(km));
                    }
                    if (last) {
                        const int p = tile * kRows + r;
                        if (keep) {
                            mn.cls[p] = CLS_KEEP;
                            mn.stat[3 * p + 1] = __float_as_uint(em);
                            mn.stat[3 * p + 2] = __float_as_uint(ym);
                        } else {
                            leave(r, undec || unc);
                        }
                        if (r == 0 && km) atomicAdd(&mn.ccount[tile * kRows / kCompactChunk], __popc(km));
                    }
                }
                zs = zs == 2 ? 0 : zs + 1;
                ready = prep;
                if (last) break;
                cur ^= 1;
            }
            if (!more) break;
            if (ready) {
                cur ^= 1;
                it ^= 1;
                lb = (lb + run) & 3;
            }
            item = next_item;
            net = next_net;
            tile = next_tile;
        }
    }
}

}  // namespace

bool mt_supported(int N, int prec) {
    return N % (prec == COSPDNN_PREC_FP32 ? 32 : 16) == 0 && 2 * mt_tile_bytes(N) <= kMtSmemMax;
}

int mt_build_entries(const std::vector<int32_t> &colptr, const std::vector<int32_t> &rowidx,
                     const std::vector<float> &vals, int N, int prec, const LayerDev &ld, MtLayer &ml,
                     std::vector<void *> &owned) {
    std::vector<std::vector<int>> order;
    const int steps = order_entries(colptr, rowidx, N, 8, order);
    // 16-bit types: groups of 16 outputs, blocks of 16 steps; FP32: 32 and 8 (nb even)
    const bool f32 = prec == COSPDNN_PREC_FP32;
    const int padded = (steps + 15) / 16 * 16, nb = padded / (f32 ? 8 : 16);
    std::vector<uint16_t> e((size_t)padded * N);
    for (int j8 = 0; j8 < N; j8 += 8)
        for (int t = 0; t < padded; ++t) {
            uint32_t used = 0;  // residues that real entries of this step read
            for (int j = j8; j < j8 + 8; ++j)
                if (t < (int)order[j].size() && order[j][t] >= 0) used |= 1u << (rowidx[order[j][t]] % 8);
            for (int j = j8; j < j8 + 8; ++j) {
                int col;
                if (t < (int)order[j].size() && order[j][t] >= 0) {
                    col = rowidx[order[j][t]];
                } else {
                    int r = 0;
                    while (used & (1u << r)) ++r;
                    used |= 1u << r;
                    col = N + r;  // N % 8 == 0: the zero column of residue r
                }
                if (f32) {
                    e[(((size_t)(j / 32) * nb + t / 8) * 32 + j % 32) * 8 + t % 8] = (uint16_t)col;
                } else {
                    const size_t lane = (size_t)(j % 16) + 16 * (t % 2);
                    e[(((size_t)(j / 16) * nb + t / 16) * 32 + lane) * 8 + t % 16 / 2] = (uint16_t)col;
                }
            }
        }
    void *d = nullptr;
    CSP_CUDA(cudaMalloc(&d, e.size() * 2));
    owned.push_back(d);
    CSP_CUDA(cudaMemcpy(d, e.data(), e.size() * 2, cudaMemcpyHostToDevice));
    ml = MtLayer{};
    ml.w = (const uint4 *)d;
    ml.nb = nb;
    ml.wbits = compute_weight_bits(vals[0], prec);
    ml.S = ld.S;
    ml.dW = ld.dW;
    ml.steps = f32 ? (float)(ld.K + 2) : 4.0f * (float)(ld.K + 4);  // as fast_steps
    return COSPDNN_OK;
}

namespace {
// Threads per CTA and CTAs per SM by the widest net: narrow tiles leave room
// for several CTAs, whose barriers and row classifications overlap.
struct MtShape {
    int threads, per_sm;
};
MtShape mt_shape(int max_n) {
    const size_t b = 2 * mt_tile_bytes(max_n);
    if (4 * b <= kMtSmemMax - 4096) return {256, 4};
    if (2 * b <= kMtSmemMax - 4096) return {512, 2};
    return {512, 1};
}
}  // namespace

// A layer of a tile takes one CTA `tile` us here, whereas k_layer_cc spreads its
// outputs over the chip: `fixed` us per iteration (with the small kernels) and
// `share` per tile.  Measured on one B200 at 1024 to 7008 neurons, 32 to 256
// entries, 8 to 600 rows.  4096 neurons x 12 layers, FP16: 32 entries 0.35 ms
// there, 0.20 here at any number of rows; 256 entries and 8, 256 and 600 rows
// 0.41, 0.59 and 1.23 there, 1.07 here.
int mt_few_tiles(int N, int prec, double entries, int sms, int64_t rows) {
    const bool f32 = prec == COSPDNN_PREC_FP32;
    const int per_sm = mt_shape(N).per_sm, tile_rows = f32 ? kMtRows / 2 : kMtRows;
    const double each = f32 ? (per_sm == 4 ? 109e-6 : per_sm == 2 ? 85e-6 : 78e-6)
                            : (per_sm == 4 ? 176e-6 : per_sm == 2 ? 105e-6 : 90e-6);
    const double fixed = 30.0, tile = each * N * entries, share = tile_rows / (f32 ? 5.5e6 : 8.6e6) * N * entries;
    if (tile <= fixed) return 0;
    const int64_t tiles = (rows + tile_rows - 1) / tile_rows, ctas = (int64_t)sms * per_sm;
    if (fixed + share * tiles <= tile * ((tiles + ctas - 1) / ctas)) return -1;
    return (int)((tile - fixed) / share);
}

int mt_layer_ctas(int sms, int max_n) { return sms * mt_shape(max_n).per_sm; }

int mt_layer_spec(KSpec &k, NetDev *nets, int nnets, int prec, unsigned long long *launches, int sms, int max_n) {
    using F = void (*)(const NetDev *, int, int, unsigned long long *);
    static const F fns[3][3] = {
        {k_layers_mt<float, 256, 4>, k_layers_mt<float, 512, 2>, k_layers_mt<float, 512, 1>},
        {k_layers_mt<__half, 256, 4>, k_layers_mt<__half, 512, 2>, k_layers_mt<__half, 512, 1>},
        {k_layers_mt<__nv_bfloat16, 256, 4>, k_layers_mt<__nv_bfloat16, 512, 2>, k_layers_mt<__nv_bfloat16, 512, 1>}};
    const MtShape s = mt_shape(max_n);
    const F f = fns[prec][s.per_sm == 4 ? 0 : s.per_sm == 2 ? 1 : 2];
    k.fn = (void *)f;
    k.smem = 2 * mt_tile_bytes(max_n);
    CSP_CUDA(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem));
    k.grid = dim3(mt_layer_ctas(sms, max_n));
    k.block = dim3(s.threads);
    k.arg(nets).arg(nnets).arg(prec).arg(launches);
    return COSPDNN_OK;
}

}  // namespace cospdnn
