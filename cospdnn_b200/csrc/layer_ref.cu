// Drop-in operator entries in the reference's feature-major layout:
//   cospdnn_layer          <- ftxj::cospdnn_single   (src/kernels/kernel.cu:240-379)
//   cospdnn_prune_compact  <- check_active_f_col + host compaction + matrix_reshape
//                             (src/kernels/kernel.cu:129-172, src/cospdnn.cu:236-276)
// These keep the reference's [feature][batch] activations so a harness can
// call them where the reference kernels are launched.  The whole-network
// engine (engine.cu) keeps its own layouts (row-major or MMA tiles).
#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace cospdnn {

namespace {

constexpr int kLayerThreads = 128;  // one thread per batch column of the tile
constexpr int kMaxBlockVals = 32 * 32;

// Blocks that are not 16x16.  One CTA = 128 batch columns x one block column; each thread keeps the
// block column's outputs for its batch column in registers.  Block values are
// staged in shared memory and broadcast; activation loads are coalesced along
// the batch.
template <int BC, bool AF32, bool BF32>
__global__ void __launch_bounds__(kLayerThreads)
    k_layer_featmajor(const void *__restrict__ A, const void *__restrict__ B, float *__restrict__ C,
                      const int *__restrict__ fuse, const int *__restrict__ idx_ptr,
                      const int *__restrict__ index, float bias, int batch, int neuron, int br) {
    __shared__ float vs[kMaxBlockVals];
    const int bid = blockIdx.y;
    const int b = blockIdx.x * kLayerThreads + threadIdx.x;
    const bool live = b < batch;
    float acc[BC];
#pragma unroll
    for (int i = 0; i < BC; ++i) acc[i] = 0.0f;

    const int p0 = idx_ptr[bid];
    const int p1 = idx_ptr[bid + 1];
    const int bsz = BC * br;
    for (int blk = p0; blk < p1; ++blk) {
        __syncthreads();
        for (int t = threadIdx.x; t < bsz; t += kLayerThreads) {
            int64_t g = (int64_t)blk * bsz + t;
            vs[t] = BF32 ? ((const float *)B)[g] : __half2float(((const __half *)B)[g]);
        }
        __syncthreads();
        const int rs = index[blk];
        for (int k = 0; k < br; ++k) {
            const int r = rs + k;
            if (r >= neuron || r < 0) continue;
            const int f = fuse ? fuse[r] : r;
            if (f < 0 || f >= neuron || !live) continue;
            float hi, lo = 0.0f;
            if (AF32) {
                hi = ((const float *)A)[(int64_t)f * batch + b];
            } else {
                hi = __half2float(((const __half *)A)[(int64_t)f * batch + b]);
                lo = __half2float(((const __half *)A)[(int64_t)(f + neuron) * batch + b]);
            }
#pragma unroll
            for (int o = 0; o < BC; ++o) {
                // value [o*BC + k] is W[start+k][col_start+o]
                const float w = vs[o * BC + k];
                acc[o] = fmaf(w, hi, acc[o]);
                if (!AF32) acc[o] = fmaf(w, lo, acc[o]);
            }
        }
    }
    if (!live) return;
#pragma unroll
    for (int o = 0; o < BC; ++o) {
        const int out = bid * BC + o;
        if (out < neuron) C[(int64_t)out * batch + b] = clamp32(acc[o] + bias);
    }
}

// 16x16 blocks, any batch.  A CTA computes one block column (16 outputs) for
// chunks of 128 * NC batch columns, a thread NC columns.  An activation is used
// by one thread only, so it goes straight to registers (ColsShape::kAhead rows
// ahead of the rows being computed); up to two blocks' weights are staged in
// shared memory, transposed ([k][o]) for broadcast 16-byte loads, and the next
// two blocks' weights and rows are fetched while these are computed.  A thread
// sums hi + lo (exact in FP32 for the two halves of one FP32 value, as
// cospdnn_prune_compact writes them) and issues packed two-lane FMAs
// (fma.rn.f32x2: two IEEE FMAs): of two columns with one weight (NC = 4 or 2), or
// of one column with two outputs' weights (NC = 1).
//   Bound: L2 traffic for two dense blocks per column (4096 x 60032: every row
// is read by two block columns, 2.0 GB through L2 and 1.0 GB written in 0.50 ms,
// half of it from DRAM), FMA issue for many blocks.  One B200, against rows
// staged in shared memory by cp.async (batches of multiples of 8) and one column
// per thread with one load in flight (others): two blocks per column, hi/lo,
// 4096 x 60032 0.563 -> 0.501 ms, 1024 x 14098 (checked sums) 107 -> 51 us; FP32,
// 4096 x 20000 164 -> 160 us; 30 blocks, 4096 x 10000 hi/lo 1.30 -> 1.03 ms, 4096
// x 219 (checked) 188 -> 66 us, 1024 x 9999 FP32 0.655 -> 0.242 ms.  Slower than
// staged rows at some batches with two blocks: FP32 by up to 4% (1024 x 14720, 34.5
// -> 35.7 us), hi/lo by up to 7% below 12 us (4096 x 640, 10.8 -> 11.4); the host
// does not know the number of blocks.
constexpr int kColsThreads = 128;
constexpr int kColsStage = 32;  // rows staged at once (two blocks)

// acc.x += w * a.x, acc.y += w * a.y in one sm_100 packed instruction
__device__ __forceinline__ void ffma2(float2 &acc, float2 w, float2 a) {
    asm("{\n\t.reg .b64 d, x, w;\n\t"
        "mov.b64 d, {%0, %1};\n\t"
        "mov.b64 x, {%2, %3};\n\t"
        "mov.b64 w, {%4, %5};\n\t"
        "fma.rn.f32x2 d, w, x, d;\n\t"
        "mov.b64 {%0, %1}, d;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "f"(a.x), "f"(a.y), "f"(w.x), "f"(w.y));
}

// {a.x + b.x, a.y + b.y} in one packed instruction
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 d, x, y;\n\t"
        "mov.b64 x, {%2, %3};\n\t"
        "mov.b64 y, {%4, %5};\n\t"
        "add.rn.f32x2 d, x, y;\n\t"
        "mov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// {a.x - b.x, a.y - b.y} in one packed instruction
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 d, x, y;\n\t"
        "mov.b64 x, {%2, %3};\n\t"
        "mov.b64 y, {%4, %5};\n\t"
        "sub.rn.f32x2 d, x, y;\n\t"
        "mov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// Whether a thread met a pair of halves whose sum may not be exact.
struct PairSums {
    uint32_t off = 0u;
    bool larger = false;
};
// {h.x + l.x, h.y + l.y}.  `sums` notes unless both sums are surely exact: a sum is
// exact when each of the two is left when the other is taken from it (the larger
// one can be taken without rounding), so with kInOrder when the second is left
// and is not the larger, as in every split.  Sums that are not finite are noted too.
// kInOrder issues one packed operation less and needs the FMA pipe less: faster with
// four columns or two apart (4096 x 5124, two blocks 69.5 -> 63.0 us, 30 blocks 714 ->
// 685; 1024 x 25495, two blocks 104 -> 92), but not with one column, whose few
// multiply-adds per row leave that pipe free (1024 x 1565, 30 blocks 79 -> 86), nor
// with two adjacent ones at small batches (1024 x 818, two blocks by 4%).
enum Exact { kUnchecked, kAnyOrder, kInOrder };
template <Exact CHECK>
__device__ __forceinline__ float2 sum_halves(float2 h, float2 l, PairSums &sums) {
    const float2 s = add2(h, l);
    if constexpr (CHECK != kUnchecked) {
        const float2 d = sub2(s, h);
        sums.off |= (__float_as_uint(d.x) ^ __float_as_uint(l.x)) | (__float_as_uint(d.y) ^ __float_as_uint(l.y));
    }
    if constexpr (CHECK == kAnyOrder) {
        const float2 e = sub2(s, l);
        sums.off |= (__float_as_uint(e.x) ^ __float_as_uint(h.x)) | (__float_as_uint(e.y) ^ __float_as_uint(h.y));
    } else if constexpr (CHECK == kInOrder) {
        sums.larger |= fabsf(l.x) > fabsf(h.x);
        sums.larger |= fabsf(l.y) > fabsf(h.y);
    }
    return s;
}

// One row of a thread's NC columns as loaded: FP32, or the hi and lo halves.
template <bool AF32, int NC>
struct RawRow;
template <int NC>
struct RawRow<true, NC> {
    float x[NC];
    // columns i, i + 1
    template <Exact CHECK>
    __device__ __forceinline__ float2 pair(int i, PairSums &) const {
        return make_float2(x[i], x[i + 1]);
    }
};
template <int NC>
struct RawRow<false, NC> {
    __half hi[NC], lo[NC];
    template <Exact CHECK>
    __device__ __forceinline__ float2 pair(int i, PairSums &sums) const {
        return sum_halves<CHECK>(make_float2(__half2float(hi[i]), __half2float(hi[i + 1])),
                                 make_float2(__half2float(lo[i]), __half2float(lo[i + 1])), sums);
    }
};
// Column 0 of two rows.
template <Exact CHECK, int NC>
__device__ __forceinline__ float2 two_rows(const RawRow<true, NC> &a, const RawRow<true, NC> &b, PairSums &) {
    return make_float2(a.x[0], b.x[0]);
}
template <Exact CHECK, int NC>
__device__ __forceinline__ float2 two_rows(const RawRow<false, NC> &a, const RawRow<false, NC> &b, PairSums &sums) {
    return sum_halves<CHECK>(make_float2(__half2float(a.hi[0]), __half2float(b.hi[0])),
                             make_float2(__half2float(a.lo[0]), __half2float(b.lo[0])), sums);
}

// Whether weight row r reads an activation row, and which (else -1).
__device__ __forceinline__ int activation_row(const int *__restrict__ fuse, int neuron, int r) {
    if (r < 0 || r >= neuron) return -1;
    const int f = fuse ? fuse[r] : r;
    return f >= 0 && f < neuron ? f : -1;
}

// Batch column b of a block column by one thread, hi and lo with a rounding each,
// rows that do not exist left out: what a thread of k_layer_cols does again when
// a sum hi + lo was not exact or an output is NaN.
template <bool AF32, bool BF32, bool REF_ARITH>
__device__ __noinline__ void layer_column(const void *__restrict__ A, const void *__restrict__ B,
                                          float *__restrict__ C, const int *__restrict__ fuse,
                                          const int *__restrict__ index, float bias, int batch, int neuron, int bid,
                                          int p0, int p1, int b) {
    float acc[16];
#pragma unroll
    for (int o = 0; o < 16; ++o) acc[o] = 0.0f;
#pragma unroll 1
    for (int k = 0; k < (p1 - p0) * 16; ++k) {
        const int f = activation_row(fuse, neuron, index[p0 + (k >> 4)] + (k & 15));
        if (f < 0) continue;
        const int64_t at = (int64_t)f * batch + b;
        const float hi = AF32 ? ((const float *)A)[at] : __half2float(((const __half *)A)[at]);
        const float lo = AF32 ? 0.0f : __half2float(((const __half *)A)[at + (int64_t)neuron * batch]);
        const int64_t g = (int64_t)(p0 + (k >> 4)) * 256;
#pragma unroll
        for (int o = 0; o < 16; ++o) {
            const int64_t e = g + (REF_ARITH ? (k & 15) * 16 + o : o * 16 + (k & 15));
            const float w = BF32 ? ((const float *)B)[e] : __half2float(((const __half *)B)[e]);
            acc[o] = fmaf(w, hi, acc[o]);
            if constexpr (!AF32) acc[o] = fmaf(w, lo, acc[o]);
        }
    }
#pragma unroll
    for (int o = 0; o < 16; ++o)
        if (bid * 16 + o < neuron) C[(int64_t)(bid * 16 + o) * batch + b] = clamp32(acc[o] + bias);
}

// Rows of a thread in flight and CTAs per SM (which bounds the registers) for NC
// columns per thread, the fastest of 13 such pairs that were measured: 4096 x
// 10000, two blocks, hi/lo, four columns: eight rows and three CTAs 92 us, four
// and four 97; 1024 x 9999, 30 blocks, hi/lo, checked: two columns with eight rows
// and three CTAs 388 us, four columns with four rows 453.  LEAN: FP32, two adjacent
// columns in 80 registers, for batches that fill the places of the other shapes
// badly, and for two blocks per column, which wait for loads: 1024 x 2560, two
// blocks 9.6 -> 8.7 us, 30 blocks 73 -> 61; 4096 x 60032, two blocks 467 -> 443.
template <bool AF32, int NC, bool VEC, bool CHECK, bool LEAN>
struct ColsShape {
    static_assert(!LEAN || (AF32 && NC == 2 && VEC), "a shape of FP32 pairs");
    static constexpr int kAhead = LEAN ? 8 : NC == 1 ? 16 : NC == 4 ? (AF32 ? 4 : 8) : VEC && AF32 ? 16 : 8;
    static constexpr int kPerSm = LEAN ? 6 : NC == 1 ? 4 : NC == 4 ? (AF32 ? 4 : 3) : VEC ? (AF32 || CHECK ? 4 : 5) : AF32 ? 4 : 3;
};

// VEC: a thread's four columns are adjacent and aligned (vector loads and
// stores), else 128 apart.  CHECK: a thread that met a pair of halves whose sum
// is not exact computes its columns again, hi and lo apart (layer_column).
template <bool AF32, bool BF32, bool REF_ARITH, int NC, bool VEC, bool CHECK, bool LEAN = false>
__global__ void __launch_bounds__(kColsThreads, ColsShape<AF32, NC, VEC, CHECK, LEAN>::kPerSm)
    k_layer_cols(const void *__restrict__ A, const void *__restrict__ B, float *__restrict__ C,
                 const int *__restrict__ fuse, const int *__restrict__ idx_ptr, const int *__restrict__ index,
                 float bias, int batch, int neuron, int chunks) {
    static_assert(VEC ? NC > 1 : NC < 4, "vectors of two or four columns");
    static_assert(!(AF32 && CHECK), "pairs of halves");
    constexpr int kChunk = kColsThreads * NC, kAhead = ColsShape<AF32, NC, VEC, CHECK, LEAN>::kAhead;
    constexpr Exact kExact = !CHECK ? kUnchecked : NC == 4 || (NC == 2 && !VEC) ? kInOrder : kAnyOrder;
    constexpr bool kCarry = NC == 4;  // a chunk's first rows are loaded while the chunk before it is stored
    constexpr int ES = AF32 ? 4 : 2;
    __shared__ __align__(16) float wT[2][kColsStage][16];
    __shared__ int64_t s_off[2][kColsStage];  // byte offset of the row in A, -1: a zero row
    // block column fastest in the grid: CTAs running together share batch
    // columns, so activation rows read by several block columns hit L2
    const int bid = blockIdx.x, tid = threadIdx.x;
    const int p0 = idx_ptr[bid];
    const int p1 = REF_ARITH ? p0 + 2 : idx_ptr[bid + 1];
    // rows and weights of the stage of blocks q, q + 1: this thread's part in
    // registers, then in shared memory
    int row = -1;
    float w4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    auto fetch = [&](int q) {
        if (tid < kColsStage) {
            const int b = q + (tid >> 4), r = b < p1 ? index[b] + (tid & 15) : -1;
            row = activation_row(fuse, neuron, r);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            // entry e of the two blocks as they are stored
            const int e = tid + i * kColsThreads;
            const int64_t g = (int64_t)q * 256 + e;
            w4[i] = q + (e >> 8) < p1 ? (BF32 ? ((const float *)B)[g] : __half2float(((const __half *)B)[g])) : 0.0f;
        }
    };
    auto store = [&](int s) {
        if (tid < kColsStage) s_off[s][tid] = row < 0 ? -1 : (int64_t)row * batch * ES;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            // REF_ARITH: value [k*16 + o] feeds output o from input start+k (the
            // reference's ldmatrix.trans pairing); otherwise value [o*16 + k] is
            // W[start+k][col_start+o]
            const int e = tid + i * kColsThreads, hi = (e >> 4) & 15, lo = e & 15, blk = (e >> 8) * 16;
            if (REF_ARITH) wT[s][blk + hi][lo] = w4[i];
            else wT[s][blk + lo][hi] = w4[i];
        }
    };
    int s = 0;
    if (p0 < p1) fetch(p0);
    store(0);
    __syncthreads();
    const bool single = p1 - p0 <= 2;
    const int per = (chunks + (int)gridDim.y - 1) / (int)gridDim.y;
    const int c_end = min(chunks, ((int)blockIdx.y + 1) * per);
    __align__(16) RawRow<AF32, NC> raw[2][kAhead];
    bool ready = false;  // raw[0] holds the chunk's first rows
    for (int ch = blockIdx.y * per; ch < c_end; ++ch) {
        const int c0 = ch * kChunk + (VEC ? tid * NC : tid);
        auto col = [&](int i) { return VEC ? c0 + i : c0 + i * kColsThreads; };
        const char *const base = (const char *)A + (int64_t)c0 * ES;
        const int64_t lo_plane = (int64_t)neuron * batch * 2;
        const bool in = c0 < batch;
        // this thread's columns of the row at byte `off`, `step` columns on
        auto load = [&](RawRow<AF32, NC> &r, int64_t off, int step) {
            const char *const src = base + off + (int64_t)step * ES;
            const bool in = c0 + step < batch;
            if constexpr (VEC) {
                const bool ok = in && off >= 0;
                if constexpr (AF32 && NC == 2) {
                    float2 v = make_float2(0.f, 0.f);
                    if (ok) v = __ldg(reinterpret_cast<const float2 *>(src));
                    r.x[0] = v.x;
                    r.x[1] = v.y;
                } else if constexpr (NC == 2) {
                    uint32_t vh = 0u, vl = 0u;
                    if (ok) {
                        vh = __ldg(reinterpret_cast<const uint32_t *>(src));
                        vl = __ldg(reinterpret_cast<const uint32_t *>(src + lo_plane));
                    }
                    *reinterpret_cast<uint32_t *>(r.hi) = vh;
                    *reinterpret_cast<uint32_t *>(r.lo) = vl;
                } else if constexpr (AF32) {
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (ok) v = __ldg(reinterpret_cast<const float4 *>(src));
                    r.x[0] = v.x;
                    r.x[1] = v.y;
                    r.x[2] = v.z;
                    r.x[3] = v.w;
                } else {
                    uint2 vh = make_uint2(0u, 0u), vl = vh;
                    if (ok) {
                        vh = __ldg(reinterpret_cast<const uint2 *>(src));
                        vl = __ldg(reinterpret_cast<const uint2 *>(src + lo_plane));
                    }
                    *reinterpret_cast<uint2 *>(r.hi) = vh;
                    *reinterpret_cast<uint2 *>(r.lo) = vl;
                }
            } else {
#pragma unroll
                for (int i = 0; i < NC; ++i) {
                    const bool ok = off >= 0 && col(i) + step < batch;
                    const char *const at = src + (int64_t)i * (kColsThreads * ES);
                    if constexpr (AF32) {
                        r.x[i] = ok ? __ldg(reinterpret_cast<const float *>(at)) : 0.0f;
                    } else {
                        r.hi[i] = ok ? __ldg(reinterpret_cast<const __half *>(at)) : __half(0.0f);
                        r.lo[i] = ok ? __ldg(reinterpret_cast<const __half *>(at + lo_plane)) : __half(0.0f);
                    }
                }
            }
        };
        // [output][column pair]; NC = 1: [output pair]
        float2 acc[8 * NC];
#pragma unroll
        for (int i = 0; i < 8 * NC; ++i) acc[i] = make_float2(0.f, 0.f);
        PairSums sums;
        for (int q = p0; q < p1; q += 2) {
            const bool more = q + 2 < p1;
            if (more) fetch(q + 2);
            else if (!single && ch + 1 < c_end) fetch(p0);
            const int rows = min(2, p1 - q) * 16;
            if (!kCarry || !ready) {
#pragma unroll
                for (int i = 0; i < kAhead; ++i) load(raw[0][i], s_off[s][i], 0);
            }
            ready = false;
#pragma unroll 1
            for (int t0 = 0; t0 < rows; t0 += 2 * kAhead) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int t = t0 + h * kAhead;
                    if (t >= rows) break;  // one block of two in a stage of 32 rows
                    if (t + kAhead < rows) {
#pragma unroll
                        for (int i = 0; i < kAhead; ++i) load(raw[h ^ 1][i], s_off[s][t + kAhead + i], 0);
                    }
                    if constexpr (NC == 1) {
#pragma unroll
                        for (int i = 0; i < kAhead; i += 2) {
                            const float4 *w = reinterpret_cast<const float4 *>(wT[s][t + i]);
                            const float2 x = two_rows<kExact>(raw[h][i], raw[h][i + 1], sums);
#pragma unroll
                            for (int o = 0; o < 8; ++o) {
                                const float4 v = w[o];
                                const float2 a = o < 4 ? make_float2(x.x, x.x) : make_float2(x.y, x.y);
                                ffma2(acc[2 * (o & 3)], make_float2(v.x, v.y), a);
                                ffma2(acc[2 * (o & 3) + 1], make_float2(v.z, v.w), a);
                            }
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < kAhead; ++i) {
                            const RawRow<AF32, NC> &r = raw[h][i];
                            const float4 *w = reinterpret_cast<const float4 *>(wT[s][t + i]);
                            if constexpr (NC == 2) {
                                const float2 a0 = r.template pair<kExact>(0, sums);
#pragma unroll
                                for (int o = 0; o < 4; ++o) {
                                    const float4 v = w[o];
                                    const float wo[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                                    for (int k = 0; k < 4; ++k) ffma2(acc[4 * o + k], make_float2(wo[k], wo[k]), a0);
                                }
                            } else {
                                const float2 a0 = r.template pair<kExact>(0, sums), a1 = r.template pair<kExact>(2, sums);
#pragma unroll
                                for (int o = 0; o < 4; ++o) {
                                    const float4 v = w[o];
                                    const float wo[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                                    for (int k = 0; k < 4; ++k) {
                                        ffma2(acc[8 * o + 2 * k], make_float2(wo[k], wo[k]), a0);
                                        ffma2(acc[8 * o + 2 * k + 1], make_float2(wo[k], wo[k]), a1);
                                    }
                                }
                            }
                        }
                    }
                }
            }
            if (!single) {
                store(s ^ 1);
                __syncthreads();
                s ^= 1;
            }
        }
        if (kCarry && single && p0 < p1 && ch + 1 < c_end) {
#pragma unroll
            for (int i = 0; i < kAhead; ++i) load(raw[0][i], s_off[s][i], kChunk);
            ready = true;
        }
        // NaN: perhaps of a weight that is not finite on a row that does not exist
        bool again = CHECK && (sums.off != 0u || sums.larger);
#pragma unroll
        for (int i = 0; i < 8 * NC; ++i) again |= isnan(acc[i].x) || isnan(acc[i].y);
        if (again) {
#pragma unroll 1
            for (int i = 0; i < NC; ++i)
                if (col(i) < batch)
                    layer_column<AF32, BF32, REF_ARITH>(A, B, C, fuse, index, bias, batch, neuron, bid, p0, p1, col(i));
            continue;
        }
#pragma unroll
        for (int o = 0; o < 16; ++o) {
            const int out = bid * 16 + o;
            if (out >= neuron) break;
            float *dst = C + (int64_t)out * batch;
            if constexpr (NC == 2) {
                const float2 x = add2(acc[o], make_float2(bias, bias));
                if constexpr (VEC) {
                    if (in) __stcs(reinterpret_cast<float2 *>(dst + c0), make_float2(clamp32(x.x), clamp32(x.y)));
                } else {
                    if (in) dst[c0] = clamp32(x.x);
                    if (col(1) < batch) dst[col(1)] = clamp32(x.y);
                }
            } else if constexpr (NC == 4) {
                const float2 bb = make_float2(bias, bias), x = add2(acc[2 * o], bb), y = add2(acc[2 * o + 1], bb);
                if (in)
                    __stcs(reinterpret_cast<float4 *>(dst + c0),
                           make_float4(clamp32(x.x), clamp32(x.y), clamp32(y.x), clamp32(y.y)));
            } else if (c0 < batch) {
                dst[c0] = clamp32((o & 1 ? acc[o / 2].y : acc[o / 2].x) + bias);
            }
        }
    }
}

// The variant with the shortest estimated time: CTAs come in rounds of one per
// place on the chip, a round lasts as long as the CTAs of its busiest SM, and a
// last round of few CTAs at least a share `tail` of a full one (latency).  `unit`
// is a CTA's time by columns per thread: more columns read a weight from shared
// memory less often.  Fitted to 57 (FP32: 220) batches from 104 to 60032 columns at
// 1024 and 4096 neurons with 2 and 30 blocks per column on one B200: the variant
// taken is 0.5% (halves), 1.1% (halves with checked sums), 1.6% (FP32) behind the
// best on average, 8 to 19% at worst, as the host does not know the number of
// blocks.  4096 x 1280, 30 blocks, FP32: two columns 128 us, four 162 (three rounds
// of half the work against two); 4096 x 60032, two blocks, hi/lo: four 501 us, two
// 536.
struct ColsRule {
    double unit[5];  // one column, two 128 apart, two adjacent, four adjacent, two adjacent (LEAN)
    double tail;
    int rounds;  // CTAs (592 at a time) from which they take two chunks each, four from four times as many
    int per_sm[5];  // 0: no such variant
};
template <bool AF32, bool CHECK>
ColsRule cols_rule(double two_apart, double two, double four, double lean, double tail, int rounds) {
    return {{1.0, 2 * two_apart, 2 * two, 4 * four, 2 * lean},
            tail,
            rounds,
            {ColsShape<AF32, 1, false, CHECK, false>::kPerSm, ColsShape<AF32, 2, false, CHECK, false>::kPerSm,
             ColsShape<AF32, 2, true, CHECK, false>::kPerSm, ColsShape<AF32, 4, true, CHECK, false>::kPerSm,
             AF32 ? ColsShape<AF32, 2, true, CHECK, AF32>::kPerSm : 0}};
}

int launch_layer_cols(cudaStream_t s, unsigned flags, const void *A, const void *B, float *C, const int *fuse,
                      const int *idx_ptr, const int *index, float bias, int batch, int neuron, int nblockcols) {
    const bool af = flags & COSPDNN_LAYER_A_FLOAT, bf = flags & COSPDNN_LAYER_B_FLOAT;
    const bool ra = flags & COSPDNN_LAYER_REFERENCE_ARITH;
    // Batches that come in whole 16-byte pieces are summed as they are; others keep
    // a rounding each for hi and lo where their sum is not exact.
    const bool check = batch % 8 != 0 || (uintptr_t)A % 16 != 0 || (uintptr_t)C % 16 != 0;
    static const ColsRule rules[3] = {cols_rule<false, false>(1.0, 0.6, 0.5, 0.0, 0.5, 8),
                                      cols_rule<false, true>(0.7, 0.75, 0.65, 0.0, 0.5, 8),
                                      cols_rule<true, false>(0.5, 0.45, 0.42, 0.4, 0.8, 16)};
    const int type = af ? 2 : check ? 1 : 0;
    const ColsRule &rule = rules[type];
    constexpr int kSms = 148;
    static const int kCols[5] = {1, 2, 2, 4, 2};
    auto pieces = [&](int nc) { return ((int64_t)batch + nc * kColsThreads - 1) / (nc * kColsThreads); };
    auto aligned = [&](int nc) { return batch % nc == 0 && (uintptr_t)A % (4 * nc) == 0 && (uintptr_t)C % (4 * nc) == 0; };
    int variant = 0;
    double best = 0.0;
    for (int v = 0; v < 5; ++v) {
        if (!rule.per_sm[v] || (v == 3 ? !aligned(4) : v > 0 && aligned(2) != (v != 1))) continue;
        const int64_t ctas = pieces(kCols[v]) * nblockcols, places = (int64_t)kSms * rule.per_sm[v], rest = ctas % places;
        const double last = rest ? std::max((double)((rest + kSms - 1) / kSms), rule.tail * rule.per_sm[v]) : 0.0;
        const double t = rule.unit[v] * ((double)(ctas / places) * rule.per_sm[v] + last);
        if (v == 0 || t < best) {
            best = t;
            variant = v;
        }
    }
    // several chunks per CTA, whose weights and rows are then staged once, when
    // there are enough CTAs (4096 x 60032, two blocks, hi/lo: four 501 us, one 529;
    // FP32, 4096 x 15000: one and two 130 us, four 133)
    const int64_t chunks = pieces(kCols[variant]), many = (int64_t)rule.rounds * 592;
    const int64_t want = chunks * nblockcols >= 4 * many ? 4 : chunks * nblockcols >= many ? 2 : 1;
    const int64_t per = std::max(want, (chunks + 65534) / 65535);  // any batch fits the grid
    const int64_t gy = (chunks + per - 1) / per;
    const dim3 grid(nblockcols, (unsigned)gy);
    using F = void (*)(const void *, const void *, float *, const int *, const int *, const int *, float, int, int, int);
#define CSP_V(AF, BF, RA, CK)                                                                                             \
    {k_layer_cols<AF, BF, RA, 1, false, CK>, k_layer_cols<AF, BF, RA, 2, false, CK>, k_layer_cols<AF, BF, RA, 2, true, CK>, \
     k_layer_cols<AF, BF, RA, 4, true, CK>, AF ? k_layer_cols<AF, BF, RA, 2, true, CK, AF> : nullptr}
#define CSP_W(AF, CK) \
    {{CSP_V(AF, false, false, CK), CSP_V(AF, false, true, CK)}, {CSP_V(AF, true, false, CK), CSP_V(AF, true, true, CK)}}
    // halves; halves whose sums are checked; FP32
    static const F fns[3][2][2][5] = {CSP_W(false, false), CSP_W(false, true), CSP_W(true, false)};
#undef CSP_W
#undef CSP_V
    fns[type][bf][ra][variant]<<<grid, kColsThreads, 0, s>>>(A, B, C, fuse, idx_ptr, index, bias, batch, neuron, (int)chunks);
    CSP_CUDA(cudaGetLastError());
    return COSPDNN_OK;
}

template <int BC>
void launch_layer(dim3 grid, cudaStream_t s, unsigned flags, const void *A, const void *B,
                  float *C, const int *fuse, const int *idx_ptr, const int *index, float bias,
                  int batch, int neuron, int br) {
    const bool af = flags & COSPDNN_LAYER_A_FLOAT, bf = flags & COSPDNN_LAYER_B_FLOAT;
#define CSP_L(AF, BF) \
    k_layer_featmajor<BC, AF, BF><<<grid, kLayerThreads, 0, s>>>(A, B, C, fuse, idx_ptr, index, bias, batch, neuron, br)
    if (af) {
        if (bf) CSP_L(true, true);
        else CSP_L(true, false);
    } else {
        if (bf) CSP_L(false, true);
        else CSP_L(false, false);
    }
#undef CSP_L
}

// ---- pruning -----------------------------------------------------------
// Bound by memory: C is read once for the flags and once for the surviving
// columns (scattered survivors share every line), which are written once:
// 0.37 ms for 4096 x 60000 with half of the columns kept at the copy rate.
// One B200, that case, hi/lo output: flags 388 -> 155 us, scan 86 -> 5 us,
// gather 265 -> 210 us against one column per thread, one load in flight and a
// one-CTA scan; the call 742 -> 367 us.
constexpr int kPruneThreads = 128;
constexpr int kScanThreads = 1024;  // columns per chunk of the scan
constexpr int kFlagRows = 64;       // rows per CTA of the flag pass
constexpr int kGatherRows = 16;     // rows per CTA of the gather

// V adjacent floats (V = 4: one 16-byte load).
template <int V>
__device__ __forceinline__ void load_cols(const float *p, float (&x)[V]) {
    if constexpr (V == 4) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
        x[3] = v.w;
    } else {
        x[0] = __ldg(p);
    }
}

// Bit 0 of flags[k]: some C[n][k] > thr.  The other bits of a chunk's first
// word count the chunk's flagged columns.  A thread takes V adjacent columns
// (V = 4 when rows start 16-byte aligned) of a slice of rows, eight rows in
// flight, and stops when all its columns are flagged.
template <int V>
__global__ void __launch_bounds__(kPruneThreads)
    k_prune_flags(const float *__restrict__ C, int neuron, int batch, float thr, int *__restrict__ flags) {
    const int k = (blockIdx.x * kPruneThreads + threadIdx.x) * V;
    if (k >= batch) return;
    const int n0 = blockIdx.y * kFlagRows, n1 = min(neuron, n0 + kFlagRows);
    bool any[V];
#pragma unroll
    for (int v = 0; v < V; ++v) any[v] = false;
    auto all = [&] {
        bool a = true;
#pragma unroll
        for (int v = 0; v < V; ++v) a &= any[v];
        return a;
    };
    const float *p = C + (int64_t)n0 * batch + k;
    int n = n0;
    for (; n + 8 <= n1 && !all(); n += 8, p += (int64_t)8 * batch) {
        float x[8][V];
#pragma unroll
        for (int i = 0; i < 8; ++i) load_cols<V>(p + (int64_t)i * batch, x[i]);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int v = 0; v < V; ++v) any[v] |= x[i][v] > thr;
    }
    for (; n < n1 && !all(); ++n, p += batch) {
        float x[V];
        load_cols<V>(p, x);
#pragma unroll
        for (int v = 0; v < V; ++v) any[v] |= x[v] > thr;
    }
#pragma unroll
    for (int v = 0; v < V; ++v)
        if (any[v] && !(*(volatile int *)&flags[k + v] & 1) && !(atomicOr(&flags[k + v], 1) & 1))
            atomicAdd(&flags[(k + v) / kScanThreads * kScanThreads], 2);
}

// Stable compaction of the surviving columns: one CTA per chunk of 1024, whose
// first position is the sum of the counts of the chunks before it.
__global__ void __launch_bounds__(kScanThreads)
    k_prune_scan(const int *__restrict__ flags, int batch, const int *__restrict__ map_in,
                 int *__restrict__ category, int *__restrict__ map_out, int *__restrict__ count) {
    __shared__ int before[kScanThreads / 32], own[kScanThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int k = blockIdx.x * kScanThreads + threadIdx.x;
    const int f = k < batch ? flags[k] & 1 : 0;
    int v = 0;
    for (int c = threadIdx.x; c < (int)blockIdx.x; c += kScanThreads) v += (int)((unsigned)flags[(int64_t)c * kScanThreads] >> 1);
    v = __reduce_add_sync(0xffffffffu, v);
    const unsigned m = __ballot_sync(0xffffffffu, f);
    if (lane == 0) {
        before[wid] = v;
        own[wid] = __popc(m);
    }
    __syncthreads();
    const int base = __reduce_add_sync(0xffffffffu, before[lane]);
    const int w = own[lane];
    const int pre = __reduce_add_sync(0xffffffffu, lane < wid ? w : 0);
    if (f) {
        const int j = base + pre + __popc(m & ((1u << lane) - 1u));
        category[j] = k;
        map_out[j] = map_in ? map_in[k] : k;
    }
    const int total = __reduce_add_sync(0xffffffffu, w);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *count = base + total;
}

// A_out[n][j] = C[n][category[j]] for j < count, 0 up to the 128-padded stride;
// a thread takes four adjacent output columns (VEC: one vector store per row
// and plane, when A_out is 16-byte aligned), four rows in flight.
template <bool HILO, bool VEC>
__global__ void __launch_bounds__(kPruneThreads)
    k_prune_gather(const float *__restrict__ C, int neuron, int batch, const int *__restrict__ category,
                   const int *__restrict__ count, void *__restrict__ A_out) {
    const int cnt = *count;
    const int stride = (cnt + 127) / 128 * 128;
    const int j = (blockIdx.x * kPruneThreads + threadIdx.x) * 4;
    if (j >= stride) return;
    int src[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) src[v] = j + v < cnt ? category[j + v] : -1;
    const int n0 = blockIdx.y * kGatherRows, n1 = min(neuron, n0 + kGatherRows);
    auto put = [&](int n, const float (&x)[4]) {
        if constexpr (HILO) {
            // the split of floatTohalf2 (src/kernels/kernel.cu:147-148)
            __align__(8) __half hi[4], lo[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                hi[v] = __float2half(x[v]);
                lo[v] = __float2half(x[v] - __half2float(hi[v]));
            }
            __half *h = (__half *)A_out + (int64_t)n * stride + j, *l = h + (int64_t)neuron * stride;
            if constexpr (VEC) {
                *reinterpret_cast<uint2 *>(h) = *reinterpret_cast<const uint2 *>(hi);
                *reinterpret_cast<uint2 *>(l) = *reinterpret_cast<const uint2 *>(lo);
            } else {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    h[v] = hi[v];
                    l[v] = lo[v];
                }
            }
        } else {
            float *o = (float *)A_out + (int64_t)n * stride + j;
            if constexpr (VEC) {
                *reinterpret_cast<float4 *>(o) = make_float4(x[0], x[1], x[2], x[3]);
            } else {
#pragma unroll
                for (int v = 0; v < 4; ++v) o[v] = x[v];
            }
        }
    };
    int n = n0;
    for (; n + 4 <= n1; n += 4) {
        float x[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) x[i][v] = src[v] >= 0 ? __ldg(C + (int64_t)(n + i) * batch + src[v]) : 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) put(n + i, x[i]);
    }
    for (; n < n1; ++n) {
        float x[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) x[v] = src[v] >= 0 ? __ldg(C + (int64_t)n * batch + src[v]) : 0.0f;
        put(n, x);
    }
}

}  // namespace

int prune_compact_impl(const float *C, int neuron, int batch, float threshold, void *A_out,
                       int *category, const int *map_in, int *map_out, int *count_dev,
                       unsigned flags, int *flag_ws, cudaStream_t s) {
    auto ctas = [](int64_t n, int64_t per) { return (unsigned)((n + per - 1) / per); };
    CSP_CUDA(cudaMemsetAsync(flag_ws, 0, sizeof(int) * (size_t)batch, s));
    const unsigned slices = ctas(neuron, kFlagRows);
    if (batch % 4 == 0 && (uintptr_t)C % 16 == 0)
        k_prune_flags<4><<<dim3(ctas(batch, 4 * kPruneThreads), slices), kPruneThreads, 0, s>>>(C, neuron, batch, threshold,
                                                                                               flag_ws);
    else
        k_prune_flags<1><<<dim3(ctas(batch, kPruneThreads), slices), kPruneThreads, 0, s>>>(C, neuron, batch, threshold,
                                                                                           flag_ws);
    k_prune_scan<<<ctas(batch, kScanThreads), kScanThreads, 0, s>>>(flag_ws, batch, map_in, category, map_out, count_dev);
    // the padded stride can pass the batch
    const dim3 g2(ctas((batch + 127) / 128 * 128, 4 * kPruneThreads), ctas(neuron, kGatherRows));
    const bool hilo = flags & COSPDNN_PRUNE_OUT_HALF_HILO, vec = (uintptr_t)A_out % 16 == 0;
    auto *gather = hilo ? (vec ? k_prune_gather<true, true> : k_prune_gather<true, false>)
                        : (vec ? k_prune_gather<false, true> : k_prune_gather<false, false>);
    gather<<<g2, kPruneThreads, 0, s>>>(C, neuron, batch, category, count_dev, A_out);
    CSP_CUDA(cudaGetLastError());
    return COSPDNN_OK;
}

}  // namespace cospdnn

using namespace cospdnn;

extern "C" int cospdnn_layer(const void *A, const void *B, float *C, const int *fuse,
                             const int *idx_ptr, const int *index, float bias, int batch,
                             int neuron, int blocksize_c, int blocksize_r, int nblockcols,
                             unsigned flags, void *stream) {
    CSP_CHECK(A && B && C && idx_ptr && index, COSPDNN_ERR_INVALID, "cospdnn_layer: null pointer");
    CSP_CHECK(batch > 0 && neuron > 0 && nblockcols > 0, COSPDNN_ERR_INVALID, "cospdnn_layer: bad sizes");
    CSP_CHECK(nblockcols <= 65535, COSPDNN_ERR_UNSUPPORTED, "cospdnn_layer: too many block columns");
    CSP_CHECK(blocksize_r > 0 && blocksize_c * blocksize_r <= kMaxBlockVals, COSPDNN_ERR_UNSUPPORTED,
              "cospdnn_layer: block larger than 32x32");
    CSP_CHECK(!(flags & ~7u), COSPDNN_ERR_INVALID, "cospdnn_layer: unknown flag");
    if (flags & COSPDNN_LAYER_REFERENCE_ARITH)
        CSP_CHECK(blocksize_c == 16 && blocksize_r == 16, COSPDNN_ERR_UNSUPPORTED,
                  "cospdnn_layer: reference arithmetic needs 16x16 blocks");
    cudaStream_t s = (cudaStream_t)stream;
    if (blocksize_c == 16 && blocksize_r == 16)
        return launch_layer_cols(s, flags, A, B, C, fuse, idx_ptr, index, bias, batch, neuron, nblockcols);
    const dim3 grid((batch + kLayerThreads - 1) / kLayerThreads, nblockcols);
    switch (blocksize_c) {
        case 8: launch_layer<8>(grid, s, flags, A, B, C, fuse, idx_ptr, index, bias, batch, neuron, blocksize_r); break;
        case 16: launch_layer<16>(grid, s, flags, A, B, C, fuse, idx_ptr, index, bias, batch, neuron, blocksize_r); break;
        case 32: launch_layer<32>(grid, s, flags, A, B, C, fuse, idx_ptr, index, bias, batch, neuron, blocksize_r); break;
        default: return fail(COSPDNN_ERR_UNSUPPORTED, "cospdnn_layer: blocksize_c must be 8, 16 or 32");
    }
    CSP_CUDA(cudaGetLastError());
    return COSPDNN_OK;
}

extern "C" size_t cospdnn_prune_workspace_bytes(int batch) {
    if (batch <= 0) return 0;
    return ((size_t)batch * sizeof(int) + 255) / 256 * 256;
}

extern "C" int cospdnn_prune_compact(const float *C, int neuron, int batch, float threshold,
                                     void *A_out, int *category, const int *map_in, int *map_out,
                                     int *count_dev, unsigned flags, void *workspace,
                                     size_t workspace_bytes, void *stream) {
    CSP_CHECK(C && A_out && category && map_out && count_dev && workspace, COSPDNN_ERR_INVALID,
              "cospdnn_prune_compact: null pointer");
    CSP_CHECK(neuron > 0 && batch > 0, COSPDNN_ERR_INVALID, "cospdnn_prune_compact: bad sizes");
    CSP_CHECK(workspace_bytes >= cospdnn_prune_workspace_bytes(batch), COSPDNN_ERR_INVALID,
              "cospdnn_prune_compact: workspace too small");
    CSP_CHECK(!(flags & ~1u), COSPDNN_ERR_INVALID, "cospdnn_prune_compact: unknown flag");
    return prune_compact_impl(C, neuron, batch, threshold, A_out, category, map_in, map_out,
                              count_dev, flags, (int *)workspace, (cudaStream_t)stream);
}

// ---- allocation-free pruning entry ----------------------------------------
// Same computation as cospdnn_prune_compact, with the per-column flag
// scratch in a file-scope device array instead of caller-provided memory.
namespace cospdnn {
namespace {
constexpr int kNoAllocMaxBatch = 1 << 20;  // columns; 4 MiB of scratch on every GPU that loads the library
__device__ __align__(256) int g_prune_scratch[kNoAllocMaxBatch];
std::mutex g_scratch_mu;
int *g_scratch_addr[1024];  // device address of g_prune_scratch, per device ordinal

// Host code cannot use g_prune_scratch's name as a device address: ask the
// runtime for it once per device, with that device current.
int scratch_for_current_device(int **out) {
    int dev = 0;
    CSP_CUDA(cudaGetDevice(&dev));
    CSP_CHECK(dev >= 0 && dev < 1024, COSPDNN_ERR_UNSUPPORTED, "prune_compact_noalloc: device ordinal too large");
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_prune_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "prune_compact_noalloc: cudaGetSymbolAddress");
        g_scratch_addr[dev] = (int *)p;
    }
    *out = g_scratch_addr[dev];
    return COSPDNN_OK;
}
}  // namespace
}  // namespace cospdnn

extern "C" int cospdnn_prune_compact_noalloc(const float *C, int neuron, int batch, float threshold,
                                             void *A_out, int *category, const int *map_in, int *map_out,
                                             int *count_dev, unsigned flags, void *stream) {
    CSP_CHECK(C && A_out && category && map_out && count_dev, COSPDNN_ERR_INVALID,
              "cospdnn_prune_compact_noalloc: null pointer");
    CSP_CHECK(neuron > 0 && batch > 0, COSPDNN_ERR_INVALID, "cospdnn_prune_compact_noalloc: bad sizes");
    CSP_CHECK(batch <= kNoAllocMaxBatch, COSPDNN_ERR_INVALID,
              "cospdnn_prune_compact_noalloc: batch exceeds the 1048576-column scratch");
    CSP_CHECK(!(flags & ~1u), COSPDNN_ERR_INVALID, "cospdnn_prune_compact_noalloc: unknown flag");
    int *ws = nullptr;
    const int rc = scratch_for_current_device(&ws);
    if (rc) return rc;
    // prune_compact_impl clears the flags it uses (an async memset, no allocation)
    return prune_compact_impl(C, neuron, batch, threshold, A_out, category, map_in, map_out, count_dev, flags, ws,
                              (cudaStream_t)stream);
}
