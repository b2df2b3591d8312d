// learn.cu — kernels of the learned early stop (include/ems_learn.h), sm_100a.
//
// A small 1-D CNN (convolutions as im2col + GEMM, then two dense layers)
// trained and run on these kernels. The GEMM runs on the tcgen05 tensor
// cores (bf16 operands from shared memory, f32 accumulator in tensor
// memory). The matrices here are small (≤ 10^5 rows, ≤ 2·10^3 columns), so
// the kernel takes A and B with arbitrary element strides (a transposed
// operand is just other strides), which keeps the backward pass free of
// transpose copies.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/ems_learn.h"

namespace {

// The GEMM C = alpha·A·B + beta·C on the fifth-generation tensor cores: one
// CTA of eight warps per 128×TN tile of C (TN the columns rounded up to 16, at
// most 128) and per share of K, the f32 accumulator in tensor memory. K runs
// in chunks of 64 through two stages of shared memory; warps 0-3 stage A,
// warps 4-7 B, each chunk's loads held in registers while the chunk before
// it multiplies. The operands lie in the no-swizzle K-major core-matrix
// layout (8 rows × 8 bf16, 16 bytes per row, per core matrix); the core
// matrices of neighbouring row groups are 144 bytes apart rather than 128, so
// that the transposing stores below meet no bank conflict. One elected thread
// issues the tcgen05.mma (M 128, N TN, K 16, bf16 in, f32 out) of a chunk and
// commits them to the stage's mbarrier (bounded waits).
//
// The matrices are small and most are bound by the latency of one CTA's chunk
// loop, so K is split over the grid's z dimension until the chip is filled
// (gemm_plan): every share writes its tile to the workspace and k_gemm_sum
// adds the shares in order. The weight gradients gain most: 32×16 over 32704
// rows took 1349 us in the single CTA of a scalar-staged kernel.
//
// An operand is read in 16-byte vectors along whichever index is contiguous
// (mode 1: k; mode 2: the row or column, transposed 8×8 in registers), or
// element by element for strides that allow neither (mode 0). An index may be
// two-level, r -> (r / per)·big + (r mod per)·stride: the rows of a valid 1-D
// convolution are overlapping spans of the channels-last input, so the
// convolutions read it in place, without columns being formed.
constexpr int TM = 128, TK = 64;
constexpr uint32_t kGroup = 144;                           // bytes between row groups of 8
constexpr uint32_t kStageOp = (TM / 8) * kGroup * (TK / 8);  // one operand's stage
constexpr uint32_t kGemmSmem = 4 * kStageOp + 64;          // three CTAs per SM, 384 of 512 tensor-memory columns
constexpr uint32_t kSumBytes = 512 * 1024;                 // shares of one tile that k_gemm_sum reads, at most
constexpr uint64_t kGemmWaitNs = 1000000000ull;

__device__ int g_learn_fail = 0;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for phase `parity`; false after kGemmWaitNs.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done = 0;
    const uint64_t t0 = now_ns();
    for (uint32_t it = 0;; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 63u) == 63u && now_ns() - t0 > kGemmWaitNs) return false;
    }
}

// Shared-memory matrix descriptor, no swizzle: start, leading and stride
// byte offsets in 16-byte units, version 1 (bits 46-47).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: f32 accumulator (bits 4-5 = 1), A
// and B bf16 (bits 7-9, 10-12 = 1), both K-major, N/8 at bit 17, M/16 at 24.
__device__ __forceinline__ uint32_t inst_desc(uint32_t tn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((tn >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
}

// One operand: rows (M or N) by k.
struct Operand {
    const uint16_t* p;
    int64_t sm, sk, big;  // element strides; big: of a two-level index's outer part
    int32_t per_m, per_k; // nonzero: that index is two-level
    int32_t mode;         // 0 scalar, 1 contiguous along k, 2 contiguous along the rows
};
__device__ __forceinline__ int64_t op_row(const Operand& o, int m) {
    return o.per_m ? (int64_t)(m / o.per_m) * o.big + (int64_t)(m % o.per_m) * o.sm : (int64_t)m * o.sm;
}
__device__ __forceinline__ int64_t op_k(const Operand& o, int k) {
    return o.per_k ? (int64_t)(k / o.per_k) * o.big + (int64_t)(k % o.per_k) * o.sk : (int64_t)k * o.sk;
}

// What happens to an element of C: C = alpha·x + beta·C or, with a bias,
// y = alpha·x + bias (kept in C if not null) and its activation in f32
// (outf) and bf16 (outb).
struct Epilogue {
    float* C;
    int64_t ldc;
    float alpha, beta;
    const float* bias;
    int act;
    float* outf;
    uint16_t* outb;
};
__device__ __forceinline__ float sigmoid(float y) { return 1.0f / (1.0f + expf(-y)); }
__device__ __forceinline__ uint16_t bf16_of(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ void finish(const Epilogue& e, int i, int j, float x) {
    const int64_t at = (int64_t)i * e.ldc + j;
    if (!e.bias) {
        e.C[at] = e.beta != 0.0f ? e.alpha * x + e.beta * e.C[at] : e.alpha * x;
        return;
    }
    const float y = e.alpha * x + e.bias[j];
    if (e.C) e.C[at] = y;
    const float a = e.act ? y * sigmoid(y) : y;
    if (e.outf) e.outf[at] = a;
    if (e.outb) e.outb[at] = bf16_of(a);
}

// A thread's part of one chunk of an operand tile of RT rows (rows r0.. of
// MN, k0.. below K), and its place in the stage. Modes 0 and 1: vector q of
// the thread holds 8 k of one row; eight lanes take eight rows of the same k
// (one 128-byte core matrix: no conflict), four groups of lanes 64 contiguous
// bytes. Mode 2: vector q holds 8 rows of k = 8·k8 + q.
struct Part {
    uint4 v[8];
};
__device__ __forceinline__ uint4 pack8(const uint16_t (&h)[8]) {
    return make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16, h[4] | (uint32_t)h[5] << 16,
                      h[6] | (uint32_t)h[7] << 16);
}
__device__ __forceinline__ void part_load(const Operand& o, int r0, int MN, int k0, int K, int RT, int t, Part& P) {
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    if (o.mode == 2) {
        const int mg = RT >> 3, m = r0 + (t % mg) * 8, k8 = t / mg;
        const bool mine = t < RT, whole = m + 8 <= MN;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = k0 + k8 * 8 + q;
            P.v[q] = zero;
            if (!mine || k >= K || m >= MN) continue;
            const uint16_t* p = o.p + op_k(o, k) + m;
            if (whole) {
                P.v[q] = __ldg(reinterpret_cast<const uint4*>(p));
            } else {
                uint16_t h[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) h[e] = m + e < MN ? p[e] : (uint16_t)0;
                P.v[q] = pack8(h);
            }
        }
        return;
    }
    const int lane = t & 31, w = t >> 5;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int tile = w + 4 * q;
        P.v[q] = zero;
        if (tile >= (RT >> 2)) continue;
        const int m = r0 + (tile >> 1) * 8 + (lane & 7), k = k0 + ((tile & 1) * 4 + (lane >> 3)) * 8;
        if (m >= MN || k >= K) continue;
        if (o.mode == 1 && k + 8 <= K) {
            P.v[q] = __ldg(reinterpret_cast<const uint4*>(o.p + op_row(o, m) + k));
        } else {
            uint16_t h[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) h[e] = k + e < K ? o.p[op_row(o, m) + op_k(o, k + e)] : (uint16_t)0;
            P.v[q] = pack8(h);
        }
    }
}
__device__ __forceinline__ uint32_t word(const uint4& v, int q) { return q == 0 ? v.x : (q == 1 ? v.y : (q == 2 ? v.z : v.w)); }
__device__ __forceinline__ void part_store(const Operand& o, unsigned char* stage, int RT, int t, const Part& P) {
    const uint32_t kstep = (uint32_t)(RT >> 3) * kGroup;
    if (o.mode == 2) {
        if (t >= RT) return;
        const int mg = RT >> 3;
        unsigned char* dst = stage + (t / mg) * kstep + (t % mg) * kGroup;
#pragma unroll
        for (int e = 0; e < 8; ++e) {  // row e: its 8 k
            const uint32_t sel = e & 1 ? 0x7632u : 0x5410u;
            uint4 r;
            r.x = __byte_perm(word(P.v[0], e >> 1), word(P.v[1], e >> 1), sel);
            r.y = __byte_perm(word(P.v[2], e >> 1), word(P.v[3], e >> 1), sel);
            r.z = __byte_perm(word(P.v[4], e >> 1), word(P.v[5], e >> 1), sel);
            r.w = __byte_perm(word(P.v[6], e >> 1), word(P.v[7], e >> 1), sel);
            *reinterpret_cast<uint4*>(dst + e * 16) = r;
        }
        return;
    }
    const int lane = t & 31, w = t >> 5;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int tile = w + 4 * q;
        if (tile >= (RT >> 2)) continue;
        *reinterpret_cast<uint4*>(stage + ((tile & 1) * 4 + (lane >> 3)) * kstep + (tile >> 1) * kGroup +
                                  (lane & 7) * 16) = P.v[q];
    }
}

// Grid: (column tiles, row tiles, shares of K). ws: null (one share), or the
// shares' tiles, [tile][share][row][TN].
__global__ void __launch_bounds__(256, 3) k_gemm_tc(const __grid_constant__ Operand A, const __grid_constant__ Operand B,
                                                    const __grid_constant__ Epilogue E, int M, int N, int K, int tn,
                                                    int per, float* ws) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 4 * kStageOp);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 4 * kStageOp + 16);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, half = tid >> 7, t = tid & 127;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * tn;
    const uint32_t cols = tn <= 32 ? 32u : (tn <= 64 ? 64u : 128u);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar + 1)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool ok = true;
    const int chunks = (K + TK - 1) / TK, c0 = blockIdx.z * per, c1 = min(chunks, c0 + per);
    const Operand& O = half ? B : A;
    const int r0 = half ? n0 : m0, MN = half ? N : M, RT = half ? tn : TM;
    const uint32_t lboA = (uint32_t)(TM >> 3) * kGroup, lboB = (uint32_t)(tn >> 3) * kGroup;
    Part P;
    part_load(O, r0, MN, c0 * TK, K, RT, t, P);
    part_store(O, smem + half * kStageOp, RT, t, P);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    for (int ch = c0; ch < c1; ++ch) {
        const int at = ch - c0, sg = at & 1;
        if (ch + 1 < c1) part_load(O, r0, MN, (ch + 1) * TK, K, RT, t, P);
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a0 = smem_addr(smem + sg * 2 * kStageOp), b0 = a0 + kStageOp;
            const uint32_t id = inst_desc((uint32_t)tn);
            const int steps = min(TK / 16, (K - ch * TK + 15) / 16);
            for (int s = 0; s < steps; ++s) {
                const uint64_t da = smem_desc(a0 + s * 2 * lboA, lboA, kGroup);
                const uint64_t db = smem_desc(b0 + s * 2 * lboB, lboB, kGroup);
                const uint32_t acc = (at > 0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(id), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_addr(bar + sg))
                         : "memory");
        }
        if (ch + 1 < c1) {
            // The other stage is free once the chunk before this one has multiplied.
            if (at > 0 && !bar_wait(bar + (sg ^ 1), (uint32_t)(((at - 1) >> 1) & 1))) ok = false;
            part_store(O, smem + ((sg ^ 1) * 2 + half) * kStageOp, RT, t, P);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
    }
    // The last chunk's commit follows every earlier one's.
    const int last = c1 - 1 - c0;
    if (!bar_wait(bar + (last & 1), (uint32_t)((last >> 1) & 1))) ok = false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // The epilogue's tensor-memory loads are warp-collective: every thread
    // takes the same branch.
    ok = __syncthreads_and(ok) != 0;
    if (!ok && tid == 0) atomicExch(&g_learn_fail, 1);
    if (ok) {
        // Warp w reads tensor-memory lanes 32(w mod 4)..: row 32(w mod 4) + lane
        // of the tile; warps 0-3 the even groups of 16 columns, 4-7 the odd ones.
        const int r = (warp & 3) * 32 + lane, i = m0 + r;
        float* share = ws ? ws + ((size_t)(blockIdx.y * gridDim.x + blockIdx.x) * gridDim.z + blockIdx.z) * TM * tn : nullptr;
        for (int cb = half * 16; cb < tn; cb += 32) {
            uint32_t v[16];
            const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cb;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                "[%16];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(taddr)
                : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (i >= M) continue;
            if (share) {
#pragma unroll
                for (int q = 0; q < 16; q += 4)
                    *reinterpret_cast<uint4*>(share + (size_t)r * tn + cb + q) = make_uint4(v[q], v[q + 1], v[q + 2], v[q + 3]);
            } else {
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    if (n0 + cb + q < N) finish(E, i, n0 + cb + q, __uint_as_float(v[q]));
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    }
}

// The shares of a split GEMM summed in order, four columns per thread, eight
// shares' loads in flight.
__global__ void __launch_bounds__(128) k_gemm_sum(const float* ws, const __grid_constant__ Epilogue E, int M, int N,
                                                  int tn, int shares, int tiles_n) {
    const int q4 = tn >> 2;
    const int q = blockIdx.x * 128 + threadIdx.x, r = q / q4, c = (q - r * q4) * 4;
    const int tile = blockIdx.y, ty = tile / tiles_n, i = ty * TM + r, j = (tile - ty * tiles_n) * tn + c;
    if (r >= TM || i >= M || j >= N) return;
    const float4* p = reinterpret_cast<const float4*>(ws + ((size_t)tile * shares * TM + r) * tn + c);
    const size_t step = (size_t)TM * q4;
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int s = 0; s < shares; s += 8) {
        float4 y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (s + e < shares) y[e] = p[(s + e) * step];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (s + e < shares) {
                x.x += y[e].x;
                x.y += y[e].y;
                x.z += y[e].z;
                x.w += y[e].w;
            }
    }
    finish(E, i, j, x.x);
    if (j + 1 < N) finish(E, i, j + 1, x.y);
    if (j + 2 < N) finish(E, i, j + 2, x.z);
    if (j + 3 < N) finish(E, i, j + 3, x.w);
}

__device__ __forceinline__ uint16_t bf16_bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

__global__ void k_to_bf16(const float* src, uint16_t* dst, size_t n) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) dst[q] = bf16_bits(src[q]);
}

__global__ void k_im2col(const float* x, uint16_t* col, int B, int T, int C, int k, int s, int To) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t F = (size_t)k * C, total = (size_t)B * To * F;
    if (q >= total) return;
    const size_t r = q / F, f = q - r * F;
    const int b = (int)(r / To), to = (int)(r - (size_t)b * To);
    const int tap = (int)(f / C), ch = (int)(f - (size_t)tap * C);
    col[q] = bf16_bits(x[((size_t)b * T + (size_t)to * s + tap) * C + ch]);
}

__global__ void k_col2im(const float* dcol, float* dx, int B, int T, int C, int k, int s, int To) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)B * T * C) return;
    const int ch = (int)(q % C);
    const size_t bt = q / C;
    const int t = (int)(bt % T), b = (int)(bt / T);
    const size_t F = (size_t)k * C;
    float acc = 0.0f;
    // t_out from high to low: taps in increasing order.
    int hi = t / s;
    if (hi > To - 1) hi = To - 1;
    for (int to = hi; to >= 0; --to) {
        const int tap = t - to * s;
        if (tap >= k) break;
        acc += dcol[((size_t)b * To + to) * F + (size_t)tap * C + ch];
    }
    dx[q] = acc;
}

__global__ void k_bias_act(float* y, const float* bias, float* a, int rows, int cols, int act) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)rows * cols) return;
    const float v = y[q] + bias[q % cols];
    y[q] = v;
    a[q] = act ? v * sigmoid(v) : v;
}

__global__ void k_act_grad(const float* y, const float* da, float* dy, int rows, int cols, int act) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)rows * cols) return;
    if (!act) {
        dy[q] = da[q];
        return;
    }
    const float s = sigmoid(y[q]);
    dy[q] = da[q] * (s + y[q] * s * (1.0f - s));
}

// One block per column: strided partial sums in a fixed order, then a tree.
__global__ void __launch_bounds__(256) k_bias_grad(const float* dy, float* db, int rows, int cols) {
    __shared__ float sh[256];
    const int j = blockIdx.x;
    float s = 0.0f;
    for (int r = threadIdx.x; r < rows; r += 256) s += dy[(size_t)r * cols + j];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) db[j] = sh[0];
}

// The adjoint of an activation, with its bf16 copy and the shares of the bias
// gradient: dy = da·act'(y) (act 0: dy = da), dyb = bf16(dy), and per block
// and column the sum of dy over the block's rows. da is read in place, or
// (k > 0) gathered from the columns' gradient as k_col2im does, da the
// gradient of a convolution's channels-last input of T positions, kernel k,
// stride s. Block: 256 threads over `rows_b` rows × 256 / cols at a time.
__global__ void __launch_bounds__(256) k_dy(const float* y, const float* da, uint16_t* dyb, float* shares, int rows,
                                            int cols, int act, int T, int k, int s, int To, int rows_b) {
    __shared__ float sh[256];
    const int wide = min(cols, 256), groups = 256 / wide;
    const int g = threadIdx.x / wide, c = blockIdx.y * 256 + threadIdx.x - g * wide;
    const int r1 = min(rows, (int)(blockIdx.x + 1) * rows_b);
    float sum = 0.0f;
    if (g < groups && c < cols)
        for (int r = blockIdx.x * rows_b + g; r < r1; r += groups) {
            const size_t at = (size_t)r * cols + c;
            float d = 0.0f;
            if (k > 0) {
                const int b = r / T, t = r - b * T;
                for (int to = min(t / s, To - 1); to >= 0; --to) {
                    const int tap = t - to * s;
                    if (tap >= k) break;
                    d += da[((size_t)b * To + to) * ((size_t)k * cols) + (size_t)tap * cols + c];
                }
            } else {
                d = da[at];
            }
            if (act) {
                const float v = y[at], q = sigmoid(v);
                d = d * (q + v * q * (1.0f - q));
            }
            dyb[at] = bf16_of(d);
            sum += d;
        }
    sh[threadIdx.x] = sum;
    __syncthreads();
    if (g == 0 && c < cols) {
        for (int q = 1; q < groups; ++q) sum += sh[q * wide + threadIdx.x];
        shares[(size_t)blockIdx.x * cols + c] = sum;
    }
}

// Column sums of the shares [blocks][cols], one warp per column.
__global__ void __launch_bounds__(256) k_share_sum(const float* shares, float* out, int blocks, int cols, float scale) {
    const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= cols) return;
    float s = 0.0f;
    for (int b = lane; b < blocks; b += 32) s += shares[(size_t)b * cols + c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) out[c] = s * scale;
}

// The MSE gradient, and the loss's shares (k_share_sum ends it).
__global__ void __launch_bounds__(256) k_mse(const float* out, const float* target, float* grad, float* shares, size_t n) {
    __shared__ float sh[8];
    float s = 0.0f;
    for (size_t q = (size_t)blockIdx.x * 256 + threadIdx.x; q < n; q += (size_t)gridDim.x * 256) {
        const float d = out[q] - target[q];
        grad[q] = 2.0f * d / (float)n;
        s += d * d;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) s += sh[w];
        shares[blockIdx.x] = s;
    }
}

__global__ void k_mse_grad(const float* out, const float* target, float* grad, size_t n) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) grad[q] = 2.0f * (out[q] - target[q]) / (float)n;
}

__global__ void __launch_bounds__(1024) k_mse_loss(const float* out, const float* target, float* loss, size_t n) {
    __shared__ float sh[1024];
    float s = 0.0f;
    for (size_t q = threadIdx.x; q < n; q += 1024) {
        const float d = out[q] - target[q];
        s += d * d;
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = 512; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss[0] = sh[0] / (float)n;
}

__global__ void k_adam(float* p, uint16_t* pb, const float* g, float* m, float* v, size_t n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const float gq = g[q];
    const float mq = b1 * m[q] + (1.0f - b1) * gq;
    const float vq = b2 * v[q] + (1.0f - b2) * gq * gq;
    m[q] = mq;
    v[q] = vq;
    const float pq = p[q] - lr * (mq / c1) / (sqrtf(vq / c2) + eps);
    p[q] = pq;
    pb[q] = bf16_bits(pq);
}

inline unsigned blocks(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }
inline int launched() { return cudaGetLastError() == cudaSuccess ? 0 : 2; }

// Whether an operand's vectors can be read along k (1), along its rows (2)
// or neither (0): a contiguous index, and every vector's start on 16 bytes.
int operand_mode(const Operand& o) {
    if (((uintptr_t)o.p & 15) || o.big % 8) return 0;
    if (o.sk == 1 && !o.per_k && o.sm % 8 == 0) return 1;
    if (o.sm == 1 && !o.per_m && o.sk % 8 == 0) return 2;
    return 0;
}

// Tile width, row and column tiles and shares of K. A share takes at least
// two chunks (the second's loads overlap the first's product); more shares
// only while the chip has SMs left (148) and a tile's shares stay below what
// k_gemm_sum reads in a few microseconds.
struct GemmPlan {
    int tn, tm, tiles_n, shares, per;
};
GemmPlan gemm_plan(int M, int N, int K, size_t ws_floats) {
    GemmPlan g;
    g.tn = N >= 128 ? 128 : (N + 15) / 16 * 16;
    g.tm = (M + TM - 1) / TM;
    g.tiles_n = (N + g.tn - 1) / g.tn;
    const int64_t tiles = (int64_t)g.tm * g.tiles_n, chunks = (K + TK - 1) / TK;
    const int64_t tile = (int64_t)TM * g.tn;
    const int64_t used = (int64_t)(M < TM ? M : TM) * (N < g.tn ? N : g.tn) * 4;
    int64_t sh = 148 / tiles;
    if (sh > (chunks + 1) / 2) sh = (chunks + 1) / 2;
    if (sh > (int64_t)kSumBytes / used) sh = (int64_t)kSumBytes / used;
    if (sh > (int64_t)(ws_floats / tile) / tiles) sh = (int64_t)(ws_floats / tile) / tiles;
    if (sh > 64) sh = 64;
    if (sh < 1) sh = 1;
    g.per = (int)((chunks + sh - 1) / sh);
    g.shares = (int)((chunks + g.per - 1) / g.per);
    return g;
}

int gemm(Operand A, Operand B, const Epilogue& E, int M, int N, int K, float* ws, size_t ws_floats, cudaStream_t s) {
    if (!A.p || !B.p || M <= 0 || N <= 0 || K <= 0) return 1;
    if (E.bias ? !(E.C || E.outf || E.outb) : !E.C) return 1;
    // Element offsets are formed in 64 bits; one grid dimension per tile axis.
    if ((M + TM - 1) / TM > 65535) return 1;
    A.mode = operand_mode(A);
    B.mode = operand_mode(B);
    static const cudaError_t attr =
        cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
    if (attr != cudaSuccess) return 2;
    const GemmPlan g = gemm_plan(M, N, K, ((uintptr_t)ws & 15) ? 0 : ws_floats);
    k_gemm_tc<<<dim3(g.tiles_n, g.tm, g.shares), 256, kGemmSmem, s>>>(A, B, E, M, N, K, g.tn, g.per,
                                                                     g.shares > 1 ? ws : nullptr);
    if (g.shares > 1) {
        const int rows = M < TM ? M : TM;
        k_gemm_sum<<<dim3(blocks((size_t)rows * (g.tn / 4), 128), g.tm * g.tiles_n), 128, 0, s>>>(ws, E, M, N, g.tn, g.shares,
                                                                                               g.tiles_n);
    }
    return launched();
}

}  // namespace

extern "C" {

int ems_learn_gemm_bf16(const uint16_t* A, int64_t sa0, int64_t sa1, const uint16_t* B, int64_t sb0, int64_t sb1,
                        float* C, int64_t ldc, int M, int N, int K, float alpha, float beta, void* stream) {
    return gemm(Operand{A, sa0, sa1, 0, 0, 0, 0}, Operand{B, sb1, sb0, 0, 0, 0, 0},
                Epilogue{C, ldc, alpha, beta, nullptr, 0, nullptr, nullptr}, M, N, K, nullptr, 0, (cudaStream_t)stream);
}

int ems_learn_run(const ems_learn_cmd* cmds, size_t n, void* stream) {
    if (!cmds && n) return 1;
    cudaStream_t s = (cudaStream_t)stream;
    for (size_t q = 0; q < n; ++q) {
        const ems_learn_cmd& c = cmds[q];
        int st = 1;
        switch (c.kind) {
        case EMS_LEARN_TO_BF16: st = ems_learn_to_bf16((const float*)c.p[0], (uint16_t*)c.p[1], (size_t)c.s[0], stream); break;
        case EMS_LEARN_GEMM:
            st = gemm(Operand{(const uint16_t*)c.p[0], c.s[0], c.s[1], c.s[5], c.i[4], 0, 0},
                      Operand{(const uint16_t*)c.p[1], c.s[3], c.s[2], c.s[6], 0, c.i[5], 0},
                      Epilogue{(float*)c.p[2], c.s[4], 1.0f, 0.0f, (const float*)c.p[3], c.i[3], (float*)c.p[5],
                               (uint16_t*)c.p[4]},
                      c.i[0], c.i[1], c.i[2], (float*)c.p[6], (size_t)c.s[7], s);
            break;
        case EMS_LEARN_DY: {
            const int rows = c.i[0], cols = c.i[1], T = c.i[3], k = c.i[4], sd = c.i[5], rows_b = c.i[6];
            if (!c.p[1] || !c.p[2] || !c.p[3] || !c.p[4] || (c.i[2] && !c.p[0]) || rows <= 0 || cols <= 0 || rows_b <= 0) break;
            if (k > 0 && (sd <= 0 || T < k || rows % T)) break;
            const unsigned nb = blocks((size_t)rows, (unsigned)rows_b);
            if ((cols + 255) / 256 > 65535) break;
            k_dy<<<dim3(nb, (cols + 255) / 256), 256, 0, s>>>((const float*)c.p[0], (const float*)c.p[1], (uint16_t*)c.p[2],
                                                             (float*)c.p[3], rows, cols, c.i[2], T, k, sd,
                                                             k > 0 ? (T - k) / sd + 1 : 0, rows_b);
            k_share_sum<<<(cols + 7) / 8, 256, 0, s>>>((const float*)c.p[3], (float*)c.p[4], (int)nb, cols, 1.0f);
            st = launched();
            break;
        }
        case EMS_LEARN_MSE: {
            const size_t m = (size_t)c.s[0];
            if (!c.p[0] || !c.p[1] || !c.p[2] || !c.p[3] || !c.p[4] || !m) break;
            const unsigned nb = (unsigned)(m < 64 * 256 ? blocks(m, 256) : 64);
            k_mse<<<nb, 256, 0, s>>>((const float*)c.p[0], (const float*)c.p[1], (float*)c.p[2], (float*)c.p[4], m);
            k_share_sum<<<1, 256, 0, s>>>((const float*)c.p[4], (float*)c.p[3], (int)nb, 1, 1.0f / (float)m);
            st = launched();
            break;
        }
        default: break;
        }
        if (st) return st;
    }
    return 0;
}

int ems_learn_check(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_learn_fail, sizeof(int)) != cudaSuccess) return 2;
    if (v) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_learn_fail, &zero, sizeof(int));
        return 4;
    }
    return 0;
}

int ems_learn_to_bf16(const float* src, uint16_t* dst, size_t n, void* stream) {
    if (!n) return 0;
    if (!src || !dst) return 1;
    k_to_bf16<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(src, dst, n);
    return launched();
}

int ems_learn_im2col(const float* x, uint16_t* col, int B, int T, int C, int k, int s, void* stream) {
    if (!x || !col || B <= 0 || C <= 0 || k <= 0 || s <= 0 || T < k) return 1;
    const int To = (T - k) / s + 1;
    const size_t n = (size_t)B * To * k * C;
    k_im2col<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(x, col, B, T, C, k, s, To);
    return launched();
}

int ems_learn_col2im(const float* dcol, float* dx, int B, int T, int C, int k, int s, void* stream) {
    if (!dcol || !dx || B <= 0 || C <= 0 || k <= 0 || s <= 0 || T < k) return 1;
    const int To = (T - k) / s + 1;
    const size_t n = (size_t)B * T * C;
    k_col2im<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(dcol, dx, B, T, C, k, s, To);
    return launched();
}

int ems_learn_bias_act(float* y, const float* bias, float* a, int rows, int cols, int act, void* stream) {
    if (!y || !bias || !a || rows <= 0 || cols <= 0) return 1;
    k_bias_act<<<blocks((size_t)rows * cols, 256), 256, 0, (cudaStream_t)stream>>>(y, bias, a, rows, cols, act);
    return launched();
}

int ems_learn_act_grad(const float* y, const float* da, float* dy, int rows, int cols, int act, void* stream) {
    if (!y || !da || !dy || rows <= 0 || cols <= 0) return 1;
    k_act_grad<<<blocks((size_t)rows * cols, 256), 256, 0, (cudaStream_t)stream>>>(y, da, dy, rows, cols, act);
    return launched();
}

int ems_learn_bias_grad(const float* dy, float* db, int rows, int cols, void* stream) {
    if (!dy || !db || rows <= 0 || cols <= 0) return 1;
    k_bias_grad<<<cols, 256, 0, (cudaStream_t)stream>>>(dy, db, rows, cols);
    return launched();
}

int ems_learn_mse(const float* out, const float* target, float* grad, float* loss, size_t n, void* stream) {
    if (!out || !target || !grad || !loss || !n) return 1;
    k_mse_grad<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(out, target, grad, n);
    k_mse_loss<<<1, 1024, 0, (cudaStream_t)stream>>>(out, target, loss, n);
    return launched();
}

int ems_learn_adam(float* p, uint16_t* p_bf16, const float* g, float* m, float* v, size_t n, float lr, float b1,
                   float b2, float eps, int t, void* stream) {
    if (!p || !p_bf16 || !g || !m || !v || !n || t < 1) return 1;
    const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
    k_adam<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(p, p_bf16, g, m, v, n, lr, b1, b2, eps, c1, c2);
    return launched();
}

}  // extern "C"
