// learn.cu — kernels of the learned early stop (include/ems_learn.h), sm_100a.
//
// A small 1-D CNN (convolutions as GEMMs over rows read in place from the
// channels-last input, then two dense layers) trained and run on these
// kernels. The GEMM runs on the tcgen05 tensor cores (bf16 operands from shared
// memory, f32 accumulator in tensor memory). The matrices here are small (≤ 10^5
// rows, ≤ 2·10^3 columns), so the kernel takes A and B with arbitrary element
// strides (a transposed operand is just other strides), which keeps the backward
// pass free of transpose copies.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>

#include "../../include/ems_learn.h"

namespace {

// The GEMM C = alpha·A·B + beta·C on the fifth-generation tensor cores: one
// CTA per 128×TN tile of C (TN the columns rounded up to 16, at most 128), the
// f32 accumulator in tensor memory, K in chunks of 64 through a ring of stages
// in shared memory. Warps 0-3 feed A and warps 4-7 B by 16-byte asynchronous
// copies, several chunks ahead of the one thread of warp 8 that issues the
// tcgen05.mma (M 128, N TN, K 16, bf16 in, f32 out) of a chunk and commits them
// to the stage's mbarrier (bounded waits).
//
// Every element of C is ONE chain of products over K in order, whatever the
// other sizes: a batch's rows come out bit for bit as each would alone, and K
// is not shared out over the chip. Shares added in f32 gave other bits, with an
// error against f64 up to 3 % larger. The chain of one CTA bounds the small
// matrices: 0.25 us per chunk for the products alone, 0.27 with copies and
// hand-over (32x16 over 32704 rows: 138 us, 64x256 over 8064: 39 us, 32x64 over
// 3840: 21 us; with two stages filled through registers 1100, 300 and 160 us).
// The weight gradients therefore share a launch (Jobs).
//
// An operand is copied in vectors along whichever index is contiguous (mode 1:
// k; mode 2: the row or column), into 8×8 core matrices without swizzle that
// are K-major or MN-major accordingly, or element by element for strides that
// allow neither (mode 0). Core matrices of neighbouring row groups lie 144
// bytes apart and those of neighbouring k groups an odd multiple of 16 modulo
// 128, so that the copies of eight lanes fall on different banks (mode 2: of 64
// rows or more). An
// index may be two-level, r -> (r / per)·big + (r mod per)·stride: the rows of
// a valid 1-D convolution are overlapping spans of the channels-last input, so
// the convolutions read it in place, without columns being formed.
constexpr int TM = 128, TK = 64, kFeeders = 256, kGemmThreads = kFeeders + 32;
constexpr uint32_t kGroup = 144;  // bytes between row groups of 8
constexpr int kMaxStages = 8;
constexpr uint32_t kStageBytes = 192 * 1024;         // most shared memory of the ring
constexpr uint32_t kBarBytes = (2 * kMaxStages + 2) * 8;
// A tile of 128 columns takes at least a quarter of an SM's shared memory: four
// of them hold all of its 512 tensor-memory columns.
constexpr uint32_t kWideBytes = 48 * 1024;
// Bytes between k groups of 8, and of a chunk, of an operand of `rows` rows.
__host__ __device__ constexpr uint32_t k_step(int rows) { return (uint32_t)(rows >> 3) * kGroup + 16u; }
__host__ __device__ constexpr uint32_t chunk_bytes(int rows) { return (TK / 8) * k_step(rows); }
constexpr uint64_t kGemmWaitNs = 1000000000ull;

__device__ int g_learn_fail = 0;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for phase `parity`; false after kGemmWaitNs. The clock is read only
// once a wait drags on.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done = 0;
    uint64_t t0 = 0;
    for (uint32_t it = 0;; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 63u) != 63u) continue;
        const uint64_t now = now_ns();
        if (!t0) t0 = now;
        if (now - t0 > kGemmWaitNs) return false;
    }
}

// Shared-memory matrix descriptor, no swizzle: start, leading and stride
// byte offsets in 16-byte units, version 1 (bits 46-47).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: f32 accumulator (bits 4-5 = 1), A
// and B bf16 (bits 7-9, 10-12 = 1), MN-major operands at bits 15 (A) and 16
// (B), N/8 at bit 17, M/16 at 24.
__device__ __forceinline__ uint32_t inst_desc(uint32_t tn, bool mn_a, bool mn_b) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn_a ? 1u << 15 : 0u) | (mn_b ? 1u << 16 : 0u) | ((tn >> 3) << 17) |
           ((uint32_t)(TM >> 4) << 24);
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
    bool wide;  // rows of every array begin on 16 bytes
};
__device__ __forceinline__ float sigmoid(float y) { return 1.0f / (1.0f + expf(-y)); }
__device__ __forceinline__ uint16_t bf16_of(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float finish_y(const Epilogue& e, float x, int j) { return e.alpha * x + e.bias[j]; }
// The elements j0 .. j0 + 15 of row i from the accumulator's values v; `wide`:
// all of them exist and every array takes 16-byte stores. A lane holds a row, so
// its stores go out in pieces of 16 bytes rather than 4.
__device__ __forceinline__ void finish(const Epilogue& e, int i, int j0, int N, bool wide, const uint32_t (&v)[16]) {
    const int64_t at = (int64_t)i * e.ldc + j0;
    if (!e.bias) {
        if (wide && e.beta == 0.0f) {
#pragma unroll
            for (int q = 0; q < 16; q += 4)
                *reinterpret_cast<float4*>(e.C + at + q) =
                    make_float4(e.alpha * __uint_as_float(v[q]), e.alpha * __uint_as_float(v[q + 1]),
                                e.alpha * __uint_as_float(v[q + 2]), e.alpha * __uint_as_float(v[q + 3]));
            return;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            if (j0 + q >= N) continue;
            const float x = __uint_as_float(v[q]);
            e.C[at + q] = e.beta != 0.0f ? e.alpha * x + e.beta * e.C[at + q] : e.alpha * x;
        }
        return;
    }
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
        float y[8], a[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int j = j0 + h + q;
            y[q] = j < N ? finish_y(e, __uint_as_float(v[h + q]), j) : 0.0f;
            a[q] = e.act ? y[q] * sigmoid(y[q]) : y[q];
        }
        if (wide) {
            float4* c = reinterpret_cast<float4*>(e.C + at + h);
            float4* f = reinterpret_cast<float4*>(e.outf + at + h);
            if (e.C) c[0] = make_float4(y[0], y[1], y[2], y[3]), c[1] = make_float4(y[4], y[5], y[6], y[7]);
            if (e.outf) f[0] = make_float4(a[0], a[1], a[2], a[3]), f[1] = make_float4(a[4], a[5], a[6], a[7]);
            if (e.outb) {
                uint32_t b[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) b[q] = bf16_of(a[2 * q]) | (uint32_t)bf16_of(a[2 * q + 1]) << 16;
                *reinterpret_cast<uint4*>(e.outb + at + h) = make_uint4(b[0], b[1], b[2], b[3]);
            }
            continue;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (j0 + h + q >= N) continue;
            if (e.C) e.C[at + h + q] = y[q];
            if (e.outf) e.outf[at + h + q] = a[q];
            if (e.outb) e.outb[at + h + q] = bf16_of(a[q]);
        }
    }
}

// 16 bytes global to shared, the first `bytes` of them read, zeros behind.
// Through L1 (.ca): the copies that pass it by (.cg) took 2.3 times as long.
__device__ __forceinline__ void copy16(uint32_t dst, const uint16_t* src, uint32_t bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// A thread's copies of an operand tile of RT rows (rows r0.. of MN): up to 8
// vectors of a chunk. Modes 0 and 1: vector q is 8 k (`k` on) of row
// t / 8 + 16·q, so eight lanes read 128 contiguous bytes. Mode 2: vector q is 8
// rows of k = `k` + q·dk, the valid row groups (rounded up to a power of two)
// side by side. Rows beyond MN are left as they are: they reach only rows or
// columns of the product that are not stored. The vectors' sources are kept and
// moved on by a chunk: computed anew for each chunk they took 500 clocks, more
// than the copies and the products.
struct Feed {
    const uint16_t* src[8];  // of the coming chunk (mode 0: of k 0)
    int inner[8];            // two-level k index: k mod per_k of the vector
    int64_t next, wrap;      // elements to the next chunk; from the end of an inner run to the next one
    uint32_t dst, step, bytes;
    int k, dk, n;  // n: vectors of this thread
};
__device__ __forceinline__ void feed_init(const Operand& o, int r0, int MN, int RT, int t, Feed& f) {
    const int valid = min(RT, MN - r0);
    f.wrap = 0;
    if (o.mode == 2) {
        const int groups = (valid + 7) >> 3, lg = 32 - __clz(groups - 1), g = t & ((1 << lg) - 1);  // clz(0) = 32
        f.k = t >> lg;
        f.dk = 128 >> lg;
        f.n = g < groups && f.k < TK ? max(1, (1 << lg) >> 1) : 0;
        f.bytes = (uint32_t)min(16, 2 * (valid - 8 * g));
        f.dst = (uint32_t)(f.k >> 3) * k_step(RT) + (uint32_t)g * kGroup + (uint32_t)(f.k & 7) * 16u;
        f.step = (uint32_t)(f.dk >> 3) * k_step(RT);
        f.next = TK * o.sk;
        if (o.per_k) f.wrap = o.big - o.per_k * o.sk;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = f.k + q * f.dk;
            f.src[q] = o.p + (q < f.n ? r0 + 8 * g + op_k(o, k) : 0);
            f.inner[q] = o.per_k ? k % o.per_k : 0;
        }
        return;
    }
    const int r = t >> 3;
    f.k = (t & 7) * 8;
    f.dk = 0;
    f.bytes = 16u;
    f.n = r < valid ? min(RT >> 4, (valid - r + 15) >> 4) : 0;
    f.dst = (uint32_t)(t & 7) * k_step(RT) + (uint32_t)(r >> 3) * kGroup + (uint32_t)(r & 7) * 16u;
    f.step = 2u * kGroup;
    f.next = o.mode ? TK : 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        f.src[q] = o.p + (q < f.n ? op_row(o, r0 + r + 16 * q) + (o.mode ? f.k : 0) : 0);
        f.inner[q] = 0;
    }
}
// The copies of the chunk at k0 into the stage at `smem`, and on to the next
// chunk; k up to the next multiple of 16 beyond K are zeros.
__device__ __forceinline__ void feed(const Operand& o, Feed& f, uint32_t smem, int k0, int K) {
    const int left = K - k0;  // k that exist from k0 on
    if (o.mode && left >= TK) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q >= f.n) break;
            copy16(smem + f.dst + q * f.step, f.src[q], f.bytes);
        }
        // After all copies are issued: a copy holds its address registers until
        // it leaves the queue.
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            f.src[q] += f.next;
            if (o.per_k) {
                f.inner[q] += TK;
                while (f.inner[q] >= o.per_k) {
                    f.inner[q] -= o.per_k;
                    f.src[q] += f.wrap;
                }
            }
        }
        return;
    }
    const int end = (min(TK, left) + 15) & ~15;  // k of the chunk multiplied
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int k = f.k + q * f.dk;
        if (q >= f.n || k >= end) break;
        const uint32_t dst = smem + f.dst + q * f.step;
        if (o.mode) {
            // Mode 1: what is left of the vector's 8 k; mode 2: its one k or none.
            const uint32_t bytes = o.mode == 2 ? f.bytes : (uint32_t)min(16, 2 * (left - k));
            copy16(dst, k < left ? f.src[q] : o.p, k < left ? bytes : 0u);
        } else {
            uint32_t h[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (k + e < left) h[e >> 1] |= (uint32_t)f.src[q][op_k(o, k0 + k + e)] << (16 * (e & 1));
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3])
                         : "memory");
        }
    }
}

// The copies of one operand by its four warps, stage by stage of `deep` chunks:
// `smem` the operand's part of the first chunk of stage 0, `size` the bytes of
// a chunk. False once a wait has run out.
__device__ __forceinline__ bool feeders(const Operand o, int r0, int MN, int RT, int t, uint32_t smem, uint32_t size,
                                        int K, int stages, int deep, uint64_t* full, uint64_t* empty) {
    Feed f;
    feed_init(o, r0, MN, RT, t, f);
    const int chunks = (K - 1) / TK + 1;
    int sg = 0;
    uint32_t round = 0;
    bool ok = true;
    for (int ch = 0; ch < chunks;) {
        if (round && !bar_wait(empty + sg, (round - 1u) & 1u)) {
            ok = false;
            break;
        }
        for (int d = 0; d < deep && ch < chunks; ++d, ++ch) feed(o, f, smem + (uint32_t)(sg * deep + d) * size, ch * TK, K);
        // Arrives once the thread's copies so far are done.
        if (o.mode) asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(full + sg)) : "memory");
        else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(full + sg)) : "memory");
        if (++sg == stages) {
            sg = 0;
            ++round;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    return ok;
}

// One product of a launch: its tiles are the blocks from `first` on, row by row.
struct Job {
    Operand A, B;
    Epilogue E;
    int M, N, K, ra, tn, stages, deep, tiles_n;
};
constexpr int kJobs = 6;
struct Jobs {
    Job job[kJobs];
    int first[kJobs];  // beyond the last job: INT_MAX
};

// Grid: the tiles of up to kJobs products that do not depend on one another
// (the weight gradients: the chain of the longest, one block, hides the
// others). Dynamic shared memory: `stages` stages of `deep` chunks of A (ra
// rows) and B (tn rows), then the barriers. The products read 128 rows of A:
// those beyond ra alias what lies behind them.
__global__ void __launch_bounds__(kGemmThreads, 2) k_gemm_tc(const __grid_constant__ Jobs P) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(16) unsigned char raw[sizeof(Job)];
    int q = 0;
    while (q + 1 < kJobs && P.first[q + 1] <= (int)blockIdx.x) ++q;
    for (unsigned w = threadIdx.x; w < sizeof(Job) / 4; w += kGemmThreads)
        reinterpret_cast<uint32_t*>(raw)[w] = reinterpret_cast<const uint32_t*>(&P.job[q])[w];
    __syncthreads();
    const Job& J = *reinterpret_cast<const Job*>(raw);
    const Epilogue& E = J.E;
    const int M = J.M, N = J.N, K = J.K, ra = J.ra, tn = J.tn, stages = J.stages, deep = J.deep;
    const int tile = (int)blockIdx.x - P.first[q], ty = tile / J.tiles_n;
    const uint32_t size_a = chunk_bytes(ra), size = size_a + chunk_bytes(tn);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + stages * deep * size);
    uint64_t* empty = full + kMaxStages;
    uint64_t* all = empty + kMaxStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(all + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, half = tid >> 7, t = tid & 127;
    const int m0 = ty * TM, n0 = (tile - ty * J.tiles_n) * tn;
    const uint32_t cols = tn <= 32 ? 32u : (tn <= 64 ? 64u : 128u);
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(full + s)), "r"(kFeeders) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(empty + s)) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(all)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool ok = true;
    const int chunks = (K - 1) / TK + 1;
    // The job comes through shared memory and its operands by value, one branch
    // each: a copy of the one or the other kernel parameter chosen per warp has
    // come out as the wrong one (nvcc 12.9), and a reference to the chosen one is
    // read again after every copy.
    if (half == 0) {
        ok = feeders(J.A, m0, M, ra, t, smem_addr(smem), size, K, stages, deep, full, empty);
    } else if (half == 1) {
        ok = feeders(J.B, n0, N, tn, t, smem_addr(smem) + size_a, size, K, stages, deep, full, empty);
    } else if (lane == 0) {
        const uint32_t id = inst_desc((uint32_t)tn, J.A.mode == 2, J.B.mode == 2);
        // The descriptors of stage 0; places further on are added in units of 16
        // bytes (all of shared memory fits the address field).
        const uint32_t a0 = smem_addr(smem), step_a = k_step(ra) >> 3, step_b = k_step(tn) >> 3;
        const uint64_t da0 = smem_desc(a0, k_step(ra), kGroup), db0 = smem_desc(a0 + size_a, k_step(tn), kGroup);
        uint32_t acc = 0;
        auto product = [&](uint32_t a, uint32_t b) {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                "l"(da0 + a), "l"(db0 + b), "r"(id), "r"(acc)
                : "memory");
            acc = 1u;
        };
        int sg = 0;
        uint32_t round = 0;
        for (int ch = 0; ch < chunks;) {
            if (!bar_wait(full + sg, round & 1u)) {
                ok = false;
                break;
            }
            // The copies are writes of the generic proxy, the products read through
            // the asynchronous one. The fence stands here: a feeder's would wait
            // for its copies of the stages behind.
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int d = 0; d < deep && ch < chunks; ++d, ++ch) {
                const uint32_t at = (uint32_t)(sg * deep + d) * (size >> 4);
                const int left = K - ch * TK;
                if (left >= TK) {
#pragma unroll
                    for (uint32_t s = 0; s < TK / 16; ++s) product(at + s * step_a, at + s * step_b);
                } else {
                    for (uint32_t s = 0; s < (uint32_t)(left + 15) / 16; ++s) product(at + s * step_a, at + s * step_b);
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_addr(empty + sg))
                         : "memory");
            if (++sg == stages) {
                sg = 0;
                ++round;
            }
        }
        // Follows every product issued, also where a wait ran out.
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(all))
                     : "memory");
    }
    __syncwarp();  // warp 8: the lanes beside the issuing one do not poll
    if ((warp < 8 || lane == 0) && !bar_wait(all, 0u)) ok = false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // The epilogue's tensor-memory loads are warp-collective: every thread
    // takes the same branch.
    ok = __syncthreads_and(ok) != 0;
    if (!ok && tid == 0) atomicExch(&g_learn_fail, 1);
    if (ok && warp < 8) {
        // Warp w reads tensor-memory lanes 32(w mod 4)..: row 32(w mod 4) + lane
        // of the tile; warps 0-3 the even groups of 16 columns, 4-7 the odd ones.
        const int r = (warp & 3) * 32 + lane, i = m0 + r;
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
            if (i < M && n0 + cb < N) finish(E, i, n0 + cb, N, E.wide && n0 + cb + 16 <= N, v);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 8) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    }
}

__global__ void k_to_bf16(const float* src, uint16_t* dst, size_t n) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) dst[q] = bf16_of(src[q]);
}

__global__ void k_im2col(const float* x, uint16_t* col, int B, int T, int C, int k, int s, int To) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t F = (size_t)k * C, total = (size_t)B * To * F;
    if (q >= total) return;
    const size_t r = q / F, f = q - r * F;
    const int b = (int)(r / To), to = (int)(r - (size_t)b * To);
    const int tap = (int)(f / C), ch = (int)(f - (size_t)tap * C);
    col[q] = bf16_of(x[((size_t)b * T + (size_t)to * s + tap) * C + ch]);
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

// The adjoint of an activation: dy = da·act'(y) (act 0: dy = da) and
// bf16(dy). da is read in place, or (k > 0) gathered from the columns' gradient
// as k_col2im does, da the gradient of a convolution's channels-last input of T
// positions, kernel k, stride s. Bound by its loads; four elements per thread
// keep them in flight.
constexpr int kDyPer = 4;
__global__ void __launch_bounds__(256) k_dy(const float* y, const float* da, uint16_t* dyb, float* dy, size_t n, int cols,
                                            int act, int T, int k, int s, int To) {
    const size_t q0 = (size_t)blockIdx.x * (256 * kDyPer) + threadIdx.x;
#pragma unroll
    for (int e = 0; e < kDyPer; ++e) {
        const size_t q = q0 + (size_t)e * 256;
        if (q >= n) break;
        float d = 0.0f;
        if (k > 0) {
            const size_t r = q / cols;
            const int c = (int)(q - r * cols), b = (int)(r / T), t = (int)(r - (size_t)b * T);
            for (int to = min(t / s, To - 1); to >= 0; --to) {
                const int tap = t - to * s;
                if (tap >= k) break;
                d += da[((size_t)b * To + to) * ((size_t)k * cols) + (size_t)tap * cols + c];
            }
        } else {
            d = da[q];
        }
        if (act) {
            const float v = y[q], g = sigmoid(v);
            d = d * (g + v * g * (1.0f - g));
        }
        dy[q] = d;
        dyb[q] = bf16_of(d);
    }
}

// Column sums of up to kJobs matrices dy[rows][cols] in the order of
// k_bias_grad: 256 partial sums over every 256th row, then a tree. A warp takes
// one partial sum of 32 columns (128 contiguous bytes a row), so that 32 blocks
// share the serial sums of 32 columns, and all layers' go in one launch: 16 + 4
// us for a training step of 64 records, in place of 51 in five launches of four
// columns per block (32 columns over 32704 rows: 24 us).
struct SumJob {
    const float* dy;
    float *parts, *db;  // parts: 256 x cols
    int rows, cols;
};
struct SumJobs {
    SumJob job[kJobs];
    int first[kJobs];  // first block of the launch; beyond the last job INT_MAX
};
__device__ __forceinline__ int sum_job(const SumJobs& P) {
    int q = 0;
    while (q + 1 < kJobs && P.first[q + 1] <= (int)blockIdx.x) ++q;
    return q;
}
// Block: eight partial sums of a group of 32 columns.
__global__ void __launch_bounds__(256) k_col_parts(const __grid_constant__ SumJobs P) {
    const int q = sum_job(P), b = (int)blockIdx.x - P.first[q], rows = P.job[q].rows, cols = P.job[q].cols;
    const int c = (b >> 5) * 32 + (threadIdx.x & 31), t = (b & 31) * 8 + (threadIdx.x >> 5);
    if (c >= cols) return;
    const float* dy = P.job[q].dy;
    float s = 0.0f;
#pragma unroll 8
    for (int r = t; r < rows; r += 256) s += dy[(size_t)r * cols + c];
    P.job[q].parts[(size_t)t * cols + c] = s;
}
// Block: the trees of eight columns, a warp each.
__global__ void __launch_bounds__(256) k_col_tree(const __grid_constant__ SumJobs P) {
    const int q = sum_job(P), cols = P.job[q].cols, lane = threadIdx.x & 31;
    const int c = ((int)blockIdx.x - P.first[q]) * 8 + (threadIdx.x >> 5);
    if (c >= cols) return;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = P.job[q].parts[(size_t)(lane + 32 * k) * cols + c];
#pragma unroll
    for (int w = 4; w > 0; w >>= 1)
#pragma unroll
        for (int k = 0; k < w; ++k) v[k] += v[k + w];
    for (int w = 16; w > 0; w >>= 1) v[0] += __shfl_down_sync(0xffffffffu, v[0], w);
    if (lane == 0) P.job[q].db[c] = v[0];
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
    pb[q] = bf16_of(pq);
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

// Makes a job of C = A·B; nonzero if it is none.
int gemm_job(Operand A, Operand B, Epilogue E, int M, int N, int K, Job& J) {
    if (!A.p || !B.p || M <= 0 || N <= 0 || K <= 0) return 1;
    if (E.bias ? !(E.C || E.outf || E.outb) : !E.C) return 1;
    if ((M - 1) / TM >= 65535) return 1;
    E.wide = E.ldc % 8 == 0 && !(((uintptr_t)E.C | (uintptr_t)E.outf | (uintptr_t)E.outb) & 15);
    A.mode = operand_mode(A);
    B.mode = operand_mode(B);
    const int ra = M >= TM ? TM : (M + 15) / 16 * 16;
    // Narrower tiles while half of the SMs have none.
    int tn = N >= 128 ? 128 : (N + 15) / 16 * 16;
    while (tn > 32 && tn % 32 == 0 && ((M - 1) / TM + 1) * (int64_t)((N - 1) / tn + 1) < 74) tn /= 2;
    const int chunks = (K - 1) / TK + 1, fit = (int)(kStageBytes / (chunk_bytes(ra) + chunk_bytes(tn)));
    // A stage holds up to four chunks, where three stages of it fit: handing one
    // over costs as much as the copies and products of a small chunk.
    const int deep = std::max(1, std::min(std::min(4, fit / 3), chunks));
    const int stages = std::min(std::min((chunks - 1) / deep + 1, kMaxStages), fit / deep);
    J = Job{A, B, E, M, N, K, ra, tn, stages, deep, (N - 1) / tn + 1};
    return 0;
}

// Launches the products of `jobs` together.
int gemm(const Job* jobs, int n, cudaStream_t s) {
    static const cudaError_t attr = cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                         (int)(kStageBytes + kBarBytes));
    if (attr != cudaSuccess) return 2;
    Jobs P{};
    uint32_t bytes = 0;
    int64_t blocks = 0;
    for (int q = 0; q < kJobs; ++q) {
        P.first[q] = q < n ? (int)blocks : INT_MAX;
        if (q >= n) continue;
        const Job& J = P.job[q] = jobs[q];
        bytes = std::max(bytes, (uint32_t)(J.stages * J.deep) * (chunk_bytes(J.ra) + chunk_bytes(J.tn)) + kBarBytes);
        if (J.tn > 64) bytes = std::max(bytes, kWideBytes);
        blocks += (int64_t)((J.M - 1) / TM + 1) * J.tiles_n;
        if (blocks >= INT_MAX) return 1;
    }
    k_gemm_tc<<<(unsigned)blocks, kGemmThreads, bytes, s>>>(P);
    return launched();
}

// The column sums of `n` jobs.
int col_sums(const SumJob* jobs, int n, cudaStream_t s) {
    SumJobs P{}, T{};
    int64_t parts = 0, trees = 0;
    for (int q = 0; q < kJobs; ++q) {
        P.first[q] = q < n ? (int)parts : INT_MAX;
        T.first[q] = q < n ? (int)trees : INT_MAX;
        if (q >= n) continue;
        P.job[q] = T.job[q] = jobs[q];
        parts += ((int64_t)jobs[q].cols + 31) / 32 * 32;
        trees += ((int64_t)jobs[q].cols + 7) / 8;
        if (parts >= INT_MAX) return 1;
    }
    k_col_parts<<<(unsigned)parts, 256, 0, s>>>(P);
    k_col_tree<<<(unsigned)trees, 256, 0, s>>>(T);
    return launched();
}

}  // namespace

extern "C" {

int ems_learn_gemm_bf16(const uint16_t* A, int64_t sa0, int64_t sa1, const uint16_t* B, int64_t sb0, int64_t sb1,
                        float* C, int64_t ldc, int M, int N, int K, float alpha, float beta, void* stream) {
    Job J;
    const int st = gemm_job(Operand{A, sa0, sa1, 0, 0, 0, 0}, Operand{B, sb1, sb0, 0, 0, 0, 0},
                            Epilogue{C, ldc, alpha, beta, nullptr, 0, nullptr, nullptr, false}, M, N, K, J);
    return st ? st : gemm(&J, 1, (cudaStream_t)stream);
}

int ems_learn_run(const ems_learn_cmd* cmds, size_t n, void* stream) {
    if (!cmds && n) return 1;
    cudaStream_t s = (cudaStream_t)stream;
    SumJob sums[kJobs];  // column sums put off to the end of the list
    int n_sums = 0;
    for (size_t q = 0; q < n; ++q) {
        const ems_learn_cmd& c = cmds[q];
        int st = 1;
        switch (c.kind) {
        case EMS_LEARN_TO_BF16: st = ems_learn_to_bf16((const float*)c.p[0], (uint16_t*)c.p[1], (size_t)c.s[0], stream); break;
        case EMS_LEARN_GEMM: {
            // The GEMMs that follow without depending on it join its launch.
            Job jobs[kJobs];
            int m = 0;
            for (; m < kJobs && q + m < n && cmds[q + m].kind == EMS_LEARN_GEMM && (!m || cmds[q + m].i[6]); ++m) {
                const ems_learn_cmd& g = cmds[q + m];
                st = gemm_job(Operand{(const uint16_t*)g.p[0], g.s[0], g.s[1], g.s[5], g.i[4], 0, 0},
                              Operand{(const uint16_t*)g.p[1], g.s[3], g.s[2], g.s[6], 0, g.i[5], 0},
                              Epilogue{(float*)g.p[2], g.s[4], 1.0f, 0.0f, (const float*)g.p[3], g.i[3], (float*)g.p[5],
                                       (uint16_t*)g.p[4], false},
                              g.i[0], g.i[1], g.i[2], jobs[m]);
                if (st) break;
            }
            if (m) {
                const int launch = gemm(jobs, m, s);
                if (launch) st = launch;
                q += (size_t)(m - 1);
            }
            break;
        }
        case EMS_LEARN_DY: {
            const int rows = c.i[0], cols = c.i[1], T = c.i[3], k = c.i[4], sd = c.i[5];
            if (!c.p[1] || !c.p[2] || !c.p[3] || !c.p[4] || !c.p[5] || (c.i[2] && !c.p[0]) || rows <= 0 || cols <= 0) break;
            if (k > 0 && (sd <= 0 || T < k || rows % T)) break;
            const size_t m = (size_t)rows * cols;
            k_dy<<<blocks(m, 256 * kDyPer), 256, 0, s>>>((const float*)c.p[0], (const float*)c.p[1], (uint16_t*)c.p[2],
                                                         (float*)c.p[3], m, cols, c.i[2], T, k, sd,
                                                         k > 0 ? (T - k) / sd + 1 : 0);
            st = launched();
            if (st) break;
            sums[n_sums++] = SumJob{(const float*)c.p[3], (float*)c.p[5], (float*)c.p[4], rows, cols};
            if (!c.i[6] || n_sums == kJobs) {
                st = col_sums(sums, n_sums, s);
                n_sums = 0;
            }
            break;
        }
        case EMS_LEARN_MSE:
            st = ems_learn_mse((const float*)c.p[0], (const float*)c.p[1], (float*)c.p[2], (float*)c.p[3], (size_t)c.s[0], stream);
            break;
        default: break;
        }
        if (st) return st;
    }
    return n_sums ? col_sums(sums, n_sums, s) : 0;
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
