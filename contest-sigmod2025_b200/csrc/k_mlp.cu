// Kernels of the learned cardinality estimator: a three-layer MLP (features
// -> 256 -> 256 -> 1, ReLU) with BF16 weights and FP32 accumulation, trained
// on the device. No reference counterpart: it stands in for the reference's
// sampling estimator (engine/query/QueryPlan.cpp:719-746) inside join
// ordering.
//
// The matrix products run on the tensor cores through mma.sync m16n8k16
// (BF16 in, FP32 accumulate): a CTA of four warps computes a 32 x 32 or 64 x
// 64 tile of C = A B from 64-deep slices of A and B, which cp.async brings
// into a ring of shared-memory stages (rows padded by 16 bytes, so
// ldmatrix reads are free of bank conflicts). A and B may each be stored with
// either dimension contiguous (the backward pass reads the forward operands
// transposed); a slice keeps its operand's own order in shared memory and
// ldmatrix transposes where the fragment needs it. A's rows may be picked by
// an index (a training batch out of the whole set). The fused epilogues are
// bias + ReLU (forward), the ReLU mask of the layer's activation (backward)
// and a plain FP32 store (weight gradients). Every output element is one
// chain of accumulations in ascending k, whatever the tile.
//
// The products are small (256 to 4096 rows, 256 columns, K up to 1792), so
// what bounds them is the length of that chain, 28 slices at K = 1792: with one
// warp a scheduler, a barrier, the copies' and ldmatrix's issue and the slice's
// MMAs (20 cycles each in a chain) follow one another. tcgen05's 128-row tiles
// would leave them on a handful of SMs, and its accumulation order is not this
// one. Measured on a B200 (one slice of 32 at a time, loaded and waited for, in
// 64 x 64 tiles, against this): 256 x 256 x 1792 about 110 -> 8 us; the two
// products of 4096 rows 147 -> 43 us.
//
// A training step of 256 rows: nine launches 215 us with the former products;
// eight launches 50 us with these; 35 us now, with six launches (products that
// do not read each other share one, row sums run beside a product), each put
// on the chip while the one before it ends (after.cuh).
#include "after.cuh"
#include "launch.h"
#include "smem.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

namespace bj {
namespace {

constexpr int kBK = 64, kPad = 8;
// Stages of the ring. The forward products' 32 x 32 tiles have 28 slices and an
// SM each: 8 stages cover the way from L2 (a step of 256 rows 34.7 us; 4: 38.4;
// 6 and 10: 38.6 and 38.2, their remainders cost what they gain). 64 x 64 tiles
// share an SM, and the backward products have 4 slices.
template <int T>
constexpr int kForwardStages = T == 32 ? 8 : 4;
constexpr int kBackwardStages = 4;
constexpr int kMaxBatch = 8192;  // rows of a batch (see bj_estimator_train)

__device__ __forceinline__ float bf2f(uint16_t v) { return __uint_as_float(uint32_t(v) << 16); }
__device__ __forceinline__ uint16_t f2bf(float f) {
    __nv_bfloat16 b = __float2bfloat16_rn(f);
    return *reinterpret_cast<uint16_t*>(&b);
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
    const uint32_t a = uint32_t(__cvta_generic_to_shared(p));
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(a));
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3,
                                                  const void* p) {
    const uint32_t a = uint32_t(__cvta_generic_to_shared(p));
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(a));
}

__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Starts copying 16 bytes to shared memory (zeros when !there).
__device__ __forceinline__ void copy16(void* dst, const void* src, bool there) {
    const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// One operand's slices in shared memory: R rows (of A, or columns of B) by
// kBK. kRowsContiguous: stored with the rows contiguous in memory, kept as
// [k][row]; else [row][k]. Element (row, k) is at p[row + k * stride] or p[row
// * stride + k]; the dimension that is not contiguous goes through idx when
// given (in shared memory when that is k), and from position `there` on it
// reads zeros (rows: from `rows` on). load() takes the slices in order.
template <int R, bool kRowsContiguous>
struct Slice {
    static constexpr int kLd = (kRowsContiguous ? R : kBK) + kPad;
    static constexpr int kWords = kLd * (kRowsContiguous ? kBK : R);
    static constexpr int kCopies = R * kBK / 8 / 128;  // 16-byte copies a thread and slice
    const uint16_t* from[kCopies];  // this thread's part of the next slice (its rows' start, under idx in k)
    int left[kCopies];              // positions before `there`, in the dimension that is not contiguous
    const uint32_t* idx;
    long stride;
    int to;                         // this thread's first element of a slice
    __device__ __forceinline__ Slice(const uint16_t* p, long stride_, const uint32_t* idx_, int there, int r0, int rows)
        : idx(idx_), stride(stride_) {
        constexpr int kLine = (kRowsContiguous ? R : kBK) / 8;  // copies a line
        const int line = threadIdx.x / kLine, at = threadIdx.x % kLine * 8;
        to = line * kLd + at;
#pragma unroll
        for (int i = 0; i < kCopies; i++) {
            const int l = line + i * (128 / kLine);
            if (kRowsContiguous) {
                left[i] = r0 + at < rows ? there - l : 0;
                from[i] = p + (left[i] > 0 ? r0 + at + (idx ? 0 : l * stride) : 0);
                idx = idx_ ? idx_ + line : nullptr;
            } else {
                const int r = r0 + l;
                left[i] = r < min(there, rows) ? 1 : 0;
                from[i] = p + (left[i] ? (idx ? long(idx[r]) : long(r)) * stride + at : 0);
            }
        }
    }
    __device__ __forceinline__ void load(uint16_t* s) {
        constexpr int kStep = 128 / ((kRowsContiguous ? R : kBK) / 8);  // lines between a thread's copies
#pragma unroll
        for (int i = 0; i < kCopies; i++) {
            const bool there = left[i] > 0;
            const uint16_t* src = from[i];
            if (kRowsContiguous) {
                if (idx) {
                    if (there) src += idx[i * kStep] * stride;
                } else if (left[i] > kBK) {
                    from[i] += kBK * stride;
                }
                left[i] -= kBK;
            } else if (there) {
                from[i] += kBK;
            }
            copy16(s + to + i * kStep * kLd, src, there);
        }
        if (kRowsContiguous && idx) idx += kBK;
    }
};

template <int T, bool kAt, bool kBt, int kStages>
constexpr size_t gemm_smem() {
    return sizeof(uint16_t) * kStages * size_t(Slice<T, kAt>::kWords + Slice<T, kBt>::kWords);
}

// A warp's operands of one slice, in registers.
template <int T>
struct Fragments {
    static constexpr int kMI = T / 32, kNJ = T / 16;  // its 16-row and 8-column MMA tiles
    uint32_t a[kBK / 16][kMI][4], b[kBK / 16][kNJ][2];
    template <bool kAt, bool kBt>
    __device__ __forceinline__ void load(const uint16_t* sA, const uint16_t* sB, int wm, int wn, int lane) {
        constexpr int kLdA = Slice<T, kAt>::kLd, kLdB = Slice<T, kBt>::kLd;
#pragma unroll
        for (int s = 0; s < kBK / 16; s++) {
            const int kk = s * 16;
#pragma unroll
            for (int i = 0; i < kMI; i++) {
                const int m = wm + i * 16;
                if (kAt)
                    ldmatrix_x4_trans(a[s][i][0], a[s][i][1], a[s][i][2], a[s][i][3],
                                      sA + (kk + (lane >> 4) * 8 + (lane & 7)) * kLdA + m + ((lane >> 3) & 1) * 8);
                else
                    ldmatrix_x4(a[s][i][0], a[s][i][1], a[s][i][2], a[s][i][3],
                                sA + (m + (lane & 15)) * kLdA + kk + (lane >> 4) * 8);
            }
#pragma unroll
            for (int j = 0; j < kNJ; j += 2) {
                const int n = wn + j * 8;
                if (kBt)
                    ldmatrix_x4_trans(b[s][j][0], b[s][j][1], b[s][j + 1][0], b[s][j + 1][1],
                                      sB + (kk + ((lane >> 3) & 1) * 8 + (lane & 7)) * kLdB + n + (lane >> 4) * 8);
                else
                    ldmatrix_x4(b[s][j][0], b[s][j][1], b[s][j + 1][0], b[s][j + 1][1],
                                sB + (n + (lane & 7) + (lane >> 4) * 8) * kLdB + kk + ((lane >> 3) & 1) * 8);
            }
        }
    }
    __device__ __forceinline__ void multiply(float (&acc)[kMI][kNJ][4]) const {
#pragma unroll
        for (int s = 0; s < kBK / 16; s++)
#pragma unroll
            for (int i = 0; i < kMI; i++)
#pragma unroll
                for (int j = 0; j < kNJ; j++) mma_bf16(acc[i][j], a[s][i], b[s][j][0], b[s][j][1]);
    }
};

// Tile (m0, n0) of g, by a block of 128 threads. kAt: A stored with m
// contiguous; kBt: B stored with n contiguous. While a slice is multiplied the
// next one's operands are on their way to registers, so what a slice takes is
// its chain of MMAs.
template <int T, bool kAt, bool kBt, int kStages>
__device__ __forceinline__ void gemm_tile(const GemmArgs& g, int m0, int n0, uint16_t* ring) {
    const uint32_t* picked = g.a_idx;
    if (kAt && picked) {  // a slice's rows would wait for their numbers
        uint32_t* const numbers = reinterpret_cast<uint32_t*>(ring + gemm_smem<T, kAt, kBt, kStages>() / sizeof(uint16_t));
        for (int k = threadIdx.x; k < g.a_there; k += 128) numbers[k] = picked[k];
        __syncthreads();
        picked = numbers;
    }
    using SA = Slice<T, kAt>;
    using SB = Slice<T, kBt>;
    using F = Fragments<T>;
    constexpr int kMI = F::kMI, kNJ = F::kNJ;
    uint16_t* ringA = ring;
    uint16_t* ringB = ring + kStages * SA::kWords;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * (T / 2), wn = (warp & 1) * (T / 2);
    const int slices = g.K / kBK;
    SA from_a(g.A, kAt ? g.a_cs : g.a_rs, picked, g.a_there, m0, g.M);
    SB from_b(g.B, kBt ? g.b_rs : g.b_cs, nullptr, kBt ? g.K : g.N, n0, g.N);
    auto fetch = [&](int t) {
        if (t < slices) {
            from_a.load(ringA + (t % kStages) * SA::kWords);
            from_b.load(ringB + (t % kStages) * SB::kWords);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int t = 0; t < kStages - 1; t++) fetch(t);
    float acc[kMI][kNJ][4] = {};
    F now, next;
    auto take = [&](F& f, int t) {
        f.template load<kAt, kBt>(ringA + (t % kStages) * SA::kWords, ringB + (t % kStages) * SB::kWords, wm, wn, lane);
    };
    auto slice = [&](const F& cur, F& other, int t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 3) : "memory");
        __syncthreads();  // slice t + 1 is there, and slice t - 1's stage is free
        fetch(t + kStages - 1);
        if (t + 1 < slices) take(other, t + 1);
        cur.multiply(acc);
    };
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    if (slices) take(now, 0);
    int t = 0;
    for (; t + 2 <= slices; t += 2) {
        slice(now, next, t);
        slice(next, now, t + 1);
    }
    if (t < slices) slice(now, next, t);
    asm volatile("cp.async.wait_all;" ::: "memory");
    // Epilogue: acc[i][j] covers rows wm + 16 i + lane / 4 (+ 8) and columns
    // wn + 8 j + 2 (lane % 4) (+ 1).
#pragma unroll
    for (int i = 0; i < kMI; i++)
#pragma unroll
        for (int j = 0; j < kNJ; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int m = m0 + wm + i * 16 + (lane >> 2) + h * 8;
                const int n = n0 + wn + j * 8 + (lane & 3) * 2;
                if (m >= g.M || n >= g.N) continue;
                float v0 = acc[i][j][2 * h], v1 = acc[i][j][2 * h + 1];
                const long o = long(m) * g.ldc + n;
                if (g.epi == kEpiBiasRelu) {
                    v0 = fmaxf(v0 + bf2f(g.bias[n]), 0.f);
                    v1 = fmaxf(v1 + bf2f(g.bias[n + 1]), 0.f);
                } else if (g.epi == kEpiReluMask) {
                    if (bf2f(g.mask[o]) <= 0.f) v0 = 0.f;
                    if (bf2f(g.mask[o + 1]) <= 0.f) v1 = 0.f;
                }
                if (g.epi == kEpiStoreF32) {
                    *reinterpret_cast<float2*>(g.Cf + o) = make_float2(v0, v1);
                } else {
                    const uint32_t packed = uint32_t(f2bf(v0)) | (uint32_t(f2bf(v1)) << 16);
                    *reinterpret_cast<uint32_t*>(g.Cb + o) = packed;
                }
            }
}

template <int T, bool kAt, bool kBt>
__global__ void __launch_bounds__(128) k_gemm_bf16(GemmArgs g) {
    extern __shared__ __align__(16) uint16_t gemm_ring[];
    begin_after_previous();
    gemm_tile<T, kAt, kBt, kForwardStages<T>>(g, blockIdx.y * T, blockIdx.x * T, gemm_ring);
}

// Two products of one step that do not read each other, in one launch: g's
// 32 x 32 tiles (A and B stored transposed: a weight gradient), then h's T x T
// ones (a row gradient). Alone, either is 64 blocks at 256 rows.
template <int T>
__global__ void __launch_bounds__(128) k_gemm_pair(GemmArgs g, GemmArgs h, int g_tiles) {
    extern __shared__ __align__(16) uint16_t gemm_ring[];
    begin_after_previous();
    const int b = blockIdx.x;
    if (b < g_tiles) {
        const int wide = (g.N + 31) / 32;
        gemm_tile<32, true, true, kBackwardStages>(g, b / wide * 32, b % wide * 32, gemm_ring);
    } else {
        const int wide = (h.N + T - 1) / T;
        gemm_tile<T, false, false, kBackwardStages>(h, (b - g_tiles) / wide * T, (b - g_tiles) % wide * T, gemm_ring);
    }
}

// Output layer and its gradient, one CTA of 256 threads per batch row:
// y = H2 . w3 + b3; with targets, loss += (y - t)^2, dy = 2 (y - t) / n_real,
// dH2 = bf16(dy * w3 * [H2 > 0]); rows at or beyond n_real get dy = 0.
__global__ void __launch_bounds__(256) k_mlp_head(MlpHeadArgs a) {
    begin_after_previous();
    const int m = blockIdx.x, n = threadIdx.x;
    const float h = bf2f(a.H2[long(m) * kMlpHidden + n]);
    const float w = bf2f(a.w3[n]);
    float p = h * w;
    for (int o = 16; o > 0; o >>= 1) p += __shfl_down_sync(0xffffffffu, p, o);
    __shared__ float part[8];
    __shared__ float dy_s;
    if ((n & 31) == 0) part[n >> 5] = p;
    __syncthreads();
    if (n == 0) {
        float y = bf2f(a.b3[0]);
        for (int i = 0; i < 8; i++) y += part[i];
        if (a.y) a.y[m] = y;
        float dy = 0.f;
        if (a.t && m < a.n_real) {
            const float d = y - a.t[a.idx ? a.idx[m] : uint32_t(m)];
            atomicAdd(a.loss, d * d);
            dy = 2.f * d / float(a.n_real);
        }
        if (a.dy) a.dy[m] = dy;
        dy_s = dy;
    }
    __syncthreads();
    if (a.dH2) a.dH2[long(m) * kMlpHidden + n] = f2bf(h > 0.f ? dy_s * w : 0.f);
}

// The gradients that are sums over the batch's rows: b2 (columns of dH2), w3
// (columns of H2 times dy) and b1 (columns of dH1), 32 columns a block of 128
// threads, and b3 (dy), a block. Rows are summed in chunks (32 rows or more, at
// most 64 chunks) and the chunks' sums in order, so the result does not depend
// on scheduling. part: 64 x 32.
constexpr int kSumColumns = 32, kRowSumBlocks = 3 * (kMlpHidden / kSumColumns) + 1;
__device__ __forceinline__ void row_sum_block(const RowSumArgs& a, int block, float (*part)[kSumColumns]) {
    constexpr int kBlocks = kMlpHidden / kSumColumns;
    const int which = block / kBlocks, t = threadIdx.x;
    if (which == 3) {
        float s[2] = {};
        for (int j = 0; j < 2; j++) {
            for (int i = t + 128 * j; i < a.rows; i += 256) s[j] += a.dy[i];
            for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_down_sync(0xffffffffu, s[j], o);
            if ((t & 31) == 0) part[(t >> 5) + 4 * j][0] = s[j];
        }
        __syncthreads();
        if (t == 0) {
            float sum = s[0];
            for (int w = 1; w < 8; w++) sum += part[w][0];
            *a.b3 = sum;
        }
        return;
    }
    const uint16_t* X = which == 0 ? a.dH2 : which == 1 ? a.H2 : a.dH1;
    float* out = which == 0 ? a.b2 : which == 1 ? a.w3 : a.b1;
    const int n = (block % kBlocks) * kSumColumns + t % kSumColumns;
    const int chunks = max(1, min(64, a.rows / 32)), per = (a.rows + chunks - 1) / chunks;
    for (int c = t / kSumColumns; c < chunks; c += 128 / kSumColumns) {
        float s = 0.f;
#pragma unroll 32
        for (int m = c * per; m < min(a.rows, c * per + per); m++)
            s += bf2f(X[long(m) * kMlpHidden + n]) * (which == 1 ? a.dy[m] : 1.f);
        part[c][t % kSumColumns] = s;
    }
    __syncthreads();
    if (t >= kSumColumns) return;
    float s = 0.f;
    for (int c = 0; c < chunks; c++) s += part[c][t];
    out[n] = s;
}

// The first layer's weight gradient (g: 32 x 32 tiles, A and B stored
// transposed) and the row sums, which its other blocks hide.
__global__ void __launch_bounds__(128) k_gemm_row_sums(GemmArgs g, RowSumArgs r) {
    extern __shared__ __align__(16) uint16_t gemm_ring[];
    begin_after_previous();
    if (blockIdx.x < kRowSumBlocks) {
        row_sum_block(r, blockIdx.x, reinterpret_cast<float(*)[kSumColumns]>(gemm_ring));
        return;
    }
    const int b = blockIdx.x - kRowSumBlocks, wide = (g.N + 31) / 32;
    gemm_tile<32, true, true, kBackwardStages>(g, b / wide * 32, b % wide * 32, gemm_ring);
}

// Adam (Kingma & Ba 2015) over every parameter, four a thread; the BF16 copy
// the products read is refreshed from the FP32 master.
__device__ __forceinline__ void adam_one(const AdamArgs& a, float g, float& am, float& av, float& aw, uint16_t& wb) {
    const float m = a.beta1 * am + (1.f - a.beta1) * g;
    const float v = a.beta2 * av + (1.f - a.beta2) * g * g;
    am = m;
    av = v;
    const float mh = m / a.bc1, vh = v / a.bc2;
    const float p = aw - a.lr * mh / (sqrtf(vh) + a.eps);
    aw = p;
    wb = f2bf(p);
}
__global__ void __launch_bounds__(128) k_adam(AdamArgs a) {
    begin_after_previous();
    const long i = 4 * (blockIdx.x * 128l + threadIdx.x);
    if (i >= a.n) return;  // n is a multiple of 4
    const float4 g = *reinterpret_cast<const float4*>(a.grad + i);
    float4 m = *reinterpret_cast<float4*>(a.m + i), v = *reinterpret_cast<float4*>(a.v + i);
    float4 w = *reinterpret_cast<float4*>(a.w + i);
    ushort4 wb;
    adam_one(a, g.x, m.x, v.x, w.x, wb.x);
    adam_one(a, g.y, m.y, v.y, w.y, wb.y);
    adam_one(a, g.z, m.z, v.z, w.z, wb.z);
    adam_one(a, g.w, m.w, v.w, w.w, wb.w);
    *reinterpret_cast<float4*>(a.m + i) = m;
    *reinterpret_cast<float4*>(a.v + i) = v;
    *reinterpret_cast<float4*>(a.w + i) = w;
    *reinterpret_cast<ushort4*>(a.wb + i) = wb;
}

__global__ void k_f32_to_bf16(const float* in, uint16_t* out, long n) {
    begin_after_previous();
    for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x)
        out[i] = f2bf(in[i]);
}

} // namespace

namespace {
template <int T, bool kAt, bool kBt>
cudaError_t launch_gemm(const GemmArgs& g, cudaStream_t st) {
    constexpr size_t smem = gemm_smem<T, kAt, kBt, kForwardStages<T>>();
    if (const cudaError_t e = allow_smem<k_gemm_bf16<T, kAt, kBt>>(smem); e != cudaSuccess) return e;
    return launch_after(k_gemm_bf16<T, kAt, kBt>, dim3((g.N + T - 1) / T, (g.M + T - 1) / T), 128, smem, st, g);
}
template <int T>
cudaError_t launch_pair(const GemmArgs& g, const GemmArgs& h, cudaStream_t st) {
    constexpr size_t smem =
        std::max(gemm_smem<32, true, true, kBackwardStages>(), gemm_smem<T, false, false, kBackwardStages>());
    if (const cudaError_t e = allow_smem<k_gemm_pair<T>>(smem); e != cudaSuccess) return e;
    const int g_tiles = (g.M + 31) / 32 * ((g.N + 31) / 32), h_tiles = (h.M + T - 1) / T * ((h.N + T - 1) / T);
    return launch_after(k_gemm_pair<T>, g_tiles + h_tiles, 128, smem, st, g, h, g_tiles);
}
// 64 x 64 tiles where they fill the chip (half the operand traffic), else
// 32 x 32 ones, four times the CTAs: the chain is as long in either.
bool wide_tiles(const GemmArgs& g) { return long((g.M + 63) / 64) * ((g.N + 63) / 64) >= 148; }
} // namespace

cudaError_t gemm_forward(const GemmArgs& g, cudaStream_t st) {
    if (g.M <= 0 || g.N <= 0) return cudaSuccess;
    return wide_tiles(g) ? launch_gemm<64, false, true>(g, st) : launch_gemm<32, false, true>(g, st);
}

cudaError_t gemm_backward(const GemmArgs& dw, const GemmArgs& dh, cudaStream_t st) {
    return wide_tiles(dh) ? launch_pair<64>(dw, dh, st) : launch_pair<32>(dw, dh, st);
}

cudaError_t gemm_row_sums(const GemmArgs& dw, const RowSumArgs& r, cudaStream_t st) {
    constexpr size_t ring = gemm_smem<32, true, true, kBackwardStages>();
    static_assert(ring >= 64 * kSumColumns * sizeof(float));
    const size_t smem = ring + (dw.a_idx ? sizeof(uint32_t) * size_t(dw.a_there) : 0);  // at most 8,192 rows a batch
    if (const cudaError_t e = allow_smem<k_gemm_row_sums>(ring + sizeof(uint32_t) * kMaxBatch); e != cudaSuccess) return e;
    return launch_after(k_gemm_row_sums, kRowSumBlocks + (dw.M + 31) / 32 * ((dw.N + 31) / 32), 128, smem, st, dw, r);
}

cudaError_t mlp_head(const MlpHeadArgs& a, int rows, cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    return launch_after(k_mlp_head, rows, kMlpHidden, 0, st, a);
}

cudaError_t adam_step(const AdamArgs& a, cudaStream_t st) {
    return launch_after(k_adam, unsigned((a.n / 4 + 127) / 128), 128, 0, st, a);
}

cudaError_t f32_to_bf16(const float* in, uint16_t* out, long n, cudaStream_t st) {
    return launch_after(k_f32_to_bf16, 592, 256, 0, st, in, out, n);
}

} // namespace bj
