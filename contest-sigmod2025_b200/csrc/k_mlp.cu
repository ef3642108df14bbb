// Kernels of the learned cardinality estimator: a three-layer MLP (features
// -> 256 -> 256 -> 1, ReLU) with BF16 weights and FP32 accumulation, trained
// on the device. No reference counterpart: it stands in for the reference's
// sampling estimator (engine/query/QueryPlan.cpp:719-746) inside join
// ordering.
//
// The matrix products run on the tensor cores through mma.sync m16n8k16
// (BF16 in, FP32 accumulate): a CTA of four warps computes a 32 x 32 or 64 x
// 64 tile of C = A B from 64-deep slices of A and B, which cp.async brings
// into a ring of four shared-memory stages (rows padded by 16 bytes, so
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
// what bounds them is the length of that chain: 112 dependent steps at
// K = 1792. tcgen05's 128-row tiles would leave them on a handful of SMs, and
// its accumulation order is not this one. Measured on a B200 (one slice of 32
// at a time, loaded and waited for, in 64 x 64 tiles, against this): 256 x 256
// x 1792 about 110 -> 12 us; the two products of 4096 rows 147 -> 43 us; a
// whole training step of 256 rows 215 -> 67 us.
#include "launch.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace bj {
namespace {

constexpr int kBK = 64, kPad = 8, kStages = 4;

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
// given, and from position `there` on it reads zeros (rows: from `rows` on).
template <int R, bool kRowsContiguous>
struct Slice {
    static constexpr int kLd = (kRowsContiguous ? R : kBK) + kPad;
    static constexpr int kWords = kLd * (kRowsContiguous ? kBK : R);
    static constexpr int kCopies = R * kBK / 8 / 128;  // 16-byte copies a thread and slice
    const uint16_t* p;
    const uint32_t* idx;
    long stride;
    int there;
    bool in_rows;                    // [k][row]: this thread's rows exist
    const uint16_t* from[kCopies];   // [row][k]: this thread's rows, at its k (null: zeros)
    __device__ __forceinline__ Slice(const uint16_t* p_, long stride_, const uint32_t* idx_, int there_, int r0, int rows)
        : p(p_), idx(idx_), stride(stride_), there(there_), in_rows(false) {
        if (kRowsContiguous) {
            const int r = r0 + (threadIdx.x % (R / 8)) * 8;
            in_rows = r < rows;
            p += in_rows ? r : 0;
        } else {
#pragma unroll
            for (int i = 0; i < kCopies; i++) {
                const int r = r0 + threadIdx.x / (kBK / 8) + i * (128 / (kBK / 8));
                const bool ok = r < min(there, rows);
                from[i] = ok ? p + (idx ? long(idx[r]) : long(r)) * stride + (threadIdx.x % (kBK / 8)) * 8 : nullptr;
            }
        }
    }
    __device__ __forceinline__ void load(uint16_t* s, int k0) const {
#pragma unroll
        for (int i = 0; i < kCopies; i++) {
            const int c = threadIdx.x + 128 * i;
            if (kRowsContiguous) {
                const int k = c / (R / 8);
                const bool ok = in_rows && k0 + k < there;
                copy16(s + k * kLd + (c % (R / 8)) * 8, p + (ok ? (idx ? long(idx[k0 + k]) : long(k0 + k)) * stride : 0),
                       ok);
            } else {
                copy16(s + (c / (kBK / 8)) * kLd + (c % (kBK / 8)) * 8, from[i] ? from[i] + k0 : p, from[i] != nullptr);
            }
        }
    }
};

template <int T, bool kAt, bool kBt>
constexpr size_t gemm_smem() {
    return sizeof(uint16_t) * kStages * size_t(Slice<T, kAt>::kWords + Slice<T, kBt>::kWords);
}

// kAt: A stored with m contiguous; kBt: B stored with n contiguous.
template <int T, bool kAt, bool kBt>
__global__ void __launch_bounds__(128) k_gemm_bf16(GemmArgs g) {
    extern __shared__ __align__(16) uint16_t gemm_ring[];
    using SA = Slice<T, kAt>;
    using SB = Slice<T, kBt>;
    constexpr int kMI = T / 32, kNJ = T / 16;  // a warp's 16-row and 8-column MMA tiles
    uint16_t* ringA = gemm_ring;
    uint16_t* ringB = gemm_ring + kStages * SA::kWords;
    const int m0 = blockIdx.y * T, n0 = blockIdx.x * T;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * (T / 2), wn = (warp & 1) * (T / 2);
    const int slices = g.K / kBK;
    const SA from_a(g.A, kAt ? g.a_cs : g.a_rs, g.a_idx, g.a_there, m0, g.M);
    const SB from_b(g.B, kBt ? g.b_rs : g.b_cs, nullptr, kBt ? g.K : g.N, n0, g.N);
    auto fetch = [&](int t) {
        if (t < slices) {
            from_a.load(ringA + (t % kStages) * SA::kWords, t * kBK);
            from_b.load(ringB + (t % kStages) * SB::kWords, t * kBK);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int t = 0; t < kStages - 1; t++) fetch(t);
    float acc[kMI][kNJ][4] = {};
    for (int t = 0; t < slices; t++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // slice t is there, and slice t - 1's stage is free
        fetch(t + kStages - 1);
        const uint16_t* sA = ringA + (t % kStages) * SA::kWords;
        const uint16_t* sB = ringB + (t % kStages) * SB::kWords;
#pragma unroll
        for (int kk = 0; kk < kBK; kk += 16) {
            uint32_t a[kMI][4], b[kNJ][2];
#pragma unroll
            for (int i = 0; i < kMI; i++) {
                const int m = wm + i * 16;
                if (kAt)
                    ldmatrix_x4_trans(a[i][0], a[i][1], a[i][2], a[i][3],
                                      sA + (kk + (lane >> 4) * 8 + (lane & 7)) * SA::kLd + m + ((lane >> 3) & 1) * 8);
                else
                    ldmatrix_x4(a[i][0], a[i][1], a[i][2], a[i][3],
                                sA + (m + (lane & 15)) * SA::kLd + kk + (lane >> 4) * 8);
            }
#pragma unroll
            for (int j = 0; j < kNJ; j += 2) {
                const int n = wn + j * 8;
                if (kBt)
                    ldmatrix_x4_trans(b[j][0], b[j][1], b[j + 1][0], b[j + 1][1],
                                      sB + (kk + ((lane >> 3) & 1) * 8 + (lane & 7)) * SB::kLd + n + (lane >> 4) * 8);
                else
                    ldmatrix_x4(b[j][0], b[j][1], b[j + 1][0], b[j + 1][1],
                                sB + (n + (lane & 7) + (lane >> 4) * 8) * SB::kLd + kk + ((lane >> 3) & 1) * 8);
            }
#pragma unroll
            for (int i = 0; i < kMI; i++)
#pragma unroll
                for (int j = 0; j < kNJ; j++) mma_bf16(acc[i][j], a[i], b[j][0], b[j][1]);
        }
    }
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

// Output layer and its gradient, one CTA of 256 threads per batch row:
// y = H2 . w3 + b3; with targets, loss += (y - t)^2, dy = 2 (y - t) / n_real,
// dH2 = bf16(dy * w3 * [H2 > 0]); rows at or beyond n_real get dy = 0.
__global__ void __launch_bounds__(256) k_mlp_head(MlpHeadArgs a) {
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

// The gradients that are sums over the batch's rows, one launch: b2 (columns
// of dH2), w3 (columns of H2 times dy) and b1 (columns of dH1), 32 columns a
// block, and b3 (dy). Rows are summed in chunks (32 rows or more, at most 64
// chunks) and the chunks' sums in order, so the result does not depend on
// scheduling.
__global__ void __launch_bounds__(256) k_row_sums(RowSumArgs a) {
    constexpr int kBlocks = kMlpHidden / 32;
    __shared__ float part[64][32];
    const int which = blockIdx.x / kBlocks, t = threadIdx.x;
    if (which == 3) {
        float s = 0.f;
        for (int i = t; i < a.rows; i += 256) s += a.dy[i];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if ((t & 31) == 0) part[0][t >> 5] = s;
        __syncthreads();
        if (t == 0) {
            for (int w = 1; w < 8; w++) s += part[0][w];
            *a.b3 = s;
        }
        return;
    }
    const uint16_t* X = which == 0 ? a.dH2 : which == 1 ? a.H2 : a.dH1;
    float* out = which == 0 ? a.b2 : which == 1 ? a.w3 : a.b1;
    const int n = (blockIdx.x % kBlocks) * 32 + (t & 31);
    const int chunks = max(1, min(64, a.rows / 32)), per = (a.rows + chunks - 1) / chunks;
    for (int c = t >> 5; c < chunks; c += 8) {
        float s = 0.f;
#pragma unroll 16
        for (int m = c * per; m < min(a.rows, c * per + per); m++)
            s += bf2f(X[long(m) * kMlpHidden + n]) * (which == 1 ? a.dy[m] : 1.f);
        part[c][t & 31] = s;
    }
    __syncthreads();
    if (t >= 32) return;
    float s = 0.f;
    for (int c = 0; c < chunks; c++) s += part[c][t];
    out[n] = s;
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
    for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x)
        out[i] = f2bf(in[i]);
}

} // namespace

namespace {
template <int T, bool kAt, bool kBt>
void launch_gemm(const GemmArgs& g, cudaStream_t st) {
    static const bool configured = [] {  // once per process
        cudaFuncSetAttribute(k_gemm_bf16<T, kAt, kBt>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(gemm_smem<T, kAt, kBt>()));
        return true;
    }();
    (void)configured;
    k_gemm_bf16<T, kAt, kBt><<<dim3((g.N + T - 1) / T, (g.M + T - 1) / T), 128, gemm_smem<T, kAt, kBt>(), st>>>(g);
}
template <int T>
void launch_gemm(const GemmArgs& g, cudaStream_t st) {
    const bool at = g.a_cs != 1, bt = g.b_rs != 1;
    if (at)
        bt ? launch_gemm<T, true, true>(g, st) : launch_gemm<T, true, false>(g, st);
    else
        bt ? launch_gemm<T, false, true>(g, st) : launch_gemm<T, false, false>(g, st);
}
} // namespace

int gemm_bf16(const GemmArgs& g, cudaStream_t st) {
    if (g.M <= 0 || g.N <= 0) return 0;
    // 64 x 64 tiles where they fill the chip (half the operand traffic), else
    // 32 x 32 ones, four times the CTAs: the chain is as long in either.
    if (long((g.M + 63) / 64) * ((g.N + 63) / 64) >= 148)
        launch_gemm<64>(g, st);
    else
        launch_gemm<32>(g, st);
    return 1;
}

int mlp_head(const MlpHeadArgs& a, int rows, cudaStream_t st) {
    if (rows <= 0) return 0;
    k_mlp_head<<<rows, kMlpHidden, 0, st>>>(a);
    return 1;
}

int row_sums(const RowSumArgs& a, cudaStream_t st) {
    k_row_sums<<<3 * (kMlpHidden / 32) + 1, 256, 0, st>>>(a);
    return 1;
}

int adam_step(const AdamArgs& a, cudaStream_t st) {
    k_adam<<<unsigned((a.n / 4 + 127) / 128), 128, 0, st>>>(a);
    return 1;
}

int f32_to_bf16(const float* in, uint16_t* out, long n, cudaStream_t st) {
    k_f32_to_bf16<<<592, 256, 0, st>>>(in, out, n);
    return 1;
}

} // namespace bj
