// resident.cuh — many steps in one launch (sm_100a).
//
// On small grids a step of the split schedule is not bound by memory but by
// its launches: a 100^3 box takes ten of them, 62 us for about 15 us of L2
// traffic (40 us here; a 24^3 box 45 -> 21 us). Here a gang of blocks advances
// a model by n steps in one cooperative launch: the phases of a step (H update
// with its CPML, E update with its CPML, poles, serial hooks) are the split
// schedule's device functions over strided work items, with a barrier of the
// gang between them in place of a kernel boundary. A batch gives every model a
// gang of its own, sized by its cells, so the models never wait for one
// another. What bounds it is the latency of a phase at 16 warps per SM (more
// registers in flight beat more warps: 512, 768 and 1024 threads take 40, 47
// and 52 us per step of the 100^3 box) and the barrier.
//
// The serial hooks run on one block of the gang in registration order, from
// amplitude tables and sample buffers on the device. Fields change within
// the launch, so they are read through the coherent path, never __ldg.
//
// A barrier wait is bounded: after wait_ns the block sets the status flags and
// leaves the kernel, and so do the others of its gang when their waits end.
#pragma once

#include "batch.cuh"

namespace emsk {

constexpr unsigned kResThreads = 512;  // most threads per block (128 registers each)

// n / d for n < 2^31 by a multiplication (round-up method, Granlund and
// Montgomery 1994): q = (mulhi(mul, n) + n) >> sh.
struct FastDiv {
    uint32_t d, mul, sh;
};
inline FastDiv fast_div(uint32_t d) {
    FastDiv f{d, 0, 0};
    while ((1ull << f.sh) < d) ++f.sh;
    f.mul = (uint32_t)((((1ull << f.sh) - d) << 32) / d + 1);
    return f;
}
__device__ __forceinline__ uint32_t quotient(const FastDiv& f, uint32_t n) { return (__umulhi(f.mul, n) + n) >> f.sh; }

// A serial hook.
struct ResOp {
    enum Kind : int32_t { SOURCE = 0, PROBE = 1, LUMPED = 2 };
    int32_t kind, electric;      // of the field (SOURCE, PROBE)
    uint32_t n, hard, axis_l, has_src;
    uint64_t n_amp, cap, interval;
    const uint32_t* node;
    const uint8_t* axis;
    const float* weight;
    const float* amp;
    const double* amp_l;
    double *values, *rec, *pv, *pi;  // series (index: step, or step / interval); null: not recorded
    double* mail;                    // host copies of the newest samples (probe; or rec, pv, pi), or null
    ProbeDevT probe;
    LumpedDevT lumped;
};

// One model as the resident kernel reads it.
struct ResModel {
    BatchModel m;
    const ResOp* ops;
    uint32_t n_ops;
    int32_t order[2];            // slab hooks in registration order: 0 CPML, 1 poles, -1 none
    int32_t fold_e, fold_h;      // the pole correction stores the saved values
    int32_t capture_first;       // fold_e, but the saved electric values are not current at the launch
    int32_t serial_h, serial_e;  // whether a post_h hook writes i, a post_e hook exists
    FastDiv div_q, div_j;        // quads per row, rows per plane
    uint32_t quads;              // nx·ny·quads per row
    uint32_t units[2];           // blocks of the shell kernels
    // The CPML comes first among the slab hooks: its corrections are part of
    // the update of the quads in `layer` (cpml_quads), `inner` the others.
    // Otherwise layer is empty and every quad inner (null: all of them in order).
    int32_t quad_cpml;
    const uint2* layer[2];
    const uint32_t* inner[2];
    uint32_t n_layer[2];
    // Every voltage probe comes after the hooks that write u: the samples of a
    // step may be taken during the next H update.
    int32_t late_probes, writes_e;
};

struct ResArgs {
    const ResModel* models;
    const uint4* blocks;     // per block: gang, rank, size
    const uint2* gangs;      // per gang: its models, [x, y) of `list`
    const uint32_t* list;
    uint32_t* bars;          // one counter per gang, 32 words apart (zeroed)
    uint32_t* bars_next;     // the next launch's, zeroed by this one
    uint32_t n_bars, n;      // counters of a set, steps to take
    uint32_t step0;          // first step (steps null)
    uint32_t* steps;         // per model: completed steps (advanced), or null
    int* status;
    int* told;               // the same flag in host memory, or null
    uint64_t wait_ns;
};

// The barrier counter of a gang: the release covers the block's writes (ordered
// before it by the block barrier), the acquire its reads after the next one.
#ifndef EMS_HOST_EMULATION
#define EMS_GANG_SHARED __shared__
__device__ __forceinline__ void gang_arrive(uint32_t* bar) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
__device__ __forceinline__ uint32_t gang_count(const uint32_t* bar) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
    return v;
}
#else
#define EMS_GANG_SHARED static thread_local
inline void gang_arrive(uint32_t* bar) { emu::gang_arrive(bar); }
inline uint32_t gang_count(const uint32_t* bar) { return emu::gang_count(bar); }
inline uint64_t global_ns() { return 0; }
#endif

// The barrier of a gang: every write of its blocks before it is visible to
// all of them after it. False once a wait has run out.
struct Gang {
    uint32_t* bar;
    uint32_t size, epoch;
};
__device__ __forceinline__ bool gang_sync(Gang& G, const ResArgs& A, int* ok) {
    __syncthreads();
    if (G.size == 1) return true;
    ++G.epoch;
    if (threadIdx.x == 0) {
        const uint32_t want = G.epoch * G.size;
        gang_arrive(G.bar);
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
            if ((int32_t)(gang_count(G.bar) - want) >= 0) break;
            if ((it & 255u) != 255u) continue;
            const uint64_t now = global_ns();
            if (!t0) t0 = now;
            if (now - t0 > A.wait_ns) {
                atomicExch(A.status, 1);
                if (A.told) *(volatile int*)A.told = 1;
                *ok = 0;
                break;
            }
        }
    }
    __syncthreads();
    return *ok != 0;
}

// A probe's sample by one warp: the products in parallel, their sum in entry
// order (src/engine/probe.rs:381-392).
__device__ __forceinline__ void probe_warp(const Fields& f, bool electric, const ProbeDevT& p, double* out, double* mail) {
    const uint32_t lane = threadIdx.x & 31u;
    double s = 0.0;
    float s32 = 0.0f;
    for (uint32_t b = 0; b < p.n; b += 32) {
        const uint32_t e = b + lane, m = p.n - b < 32u ? p.n - b : 32u;
        double t = 0.0;
        float t32 = 0.0f;
        if (e < p.n) {
            const float x = (electric ? f.u : f.i)[p.axis[e]][p.node[e]];
            if (p.f32_sum) t32 = __fmul_rn((float)p.weight[e], x);
            else t = __dmul_rn(p.weight[e], (double)x);
        }
        for (uint32_t q = 0; q < m; ++q) {
            if (p.f32_sum) s32 = __fadd_rn(s32, __shfl_sync(0xffffffffu, t32, q));
            else s = __dadd_rn(s, __shfl_sync(0xffffffffu, t, q));
        }
    }
    if (lane != 0) return;
    *out = p.f32_sum ? (double)s32 : s;
    if (mail) *mail = *out;
}

// The serial hooks of one field side at step `step`, by one block, in
// registration order (probes: the probes; writers: the others); consecutive
// probes take a warp each. STEP: the resident kernel counts below 2^31 (and
// takes probe intervals below that), the other steps in 64 bits.
template <class STEP>
__device__ __forceinline__ void serial_hooks(const Fields& f, double dt, const ResOp* ops, uint32_t n_ops, bool electric,
                                             STEP step, bool probes, bool writers) {
    for (uint32_t q = 0; q < n_ops;) {
        const ResOp& o = ops[q];
        const bool mine = (o.electric != 0) == electric && (o.kind == ResOp::PROBE ? probes : writers);
        if (!mine) {
            ++q;
            continue;
        }
        if (o.kind == ResOp::PROBE) {
            uint32_t end = q;
            while (end < n_ops && ops[end].kind == ResOp::PROBE) ++end;
            for (uint32_t r = q + (threadIdx.x >> 5); r < end; r += blockDim.x >> 5) {
                const ResOp& p = ops[r];
                if ((p.electric != 0) != electric || step % (STEP)p.interval) continue;
                const STEP at = step / (STEP)p.interval;
                if (at < p.cap) probe_warp(f, electric, p.probe, p.values + at, p.mail);
            }
            q = end;
        } else if (o.kind == ResOp::SOURCE) {
            const float a = step < o.n_amp ? o.amp[step] : 0.0f;
            if (o.hard || a != 0.0f)
                for (uint32_t e = threadIdx.x; e < o.n; e += blockDim.x) {
                    float* F = electric ? f.u[o.axis[e]] : f.i[o.axis[e]];
                    const float v = __fmul_rn(o.weight[e], a);
                    F[o.node[e]] = o.hard ? v : __fadd_rn(F[o.node[e]], v);
                }
            ++q;
        } else {
            const double val = o.has_src && step < o.n_amp ? o.amp_l[step] : 0.0;
            const bool room = step < o.cap;
            lumped_post_e_block(f.u[o.axis_l], o.lumped, val, o.has_src && val != 0.0, dt,
                                o.rec && room ? o.rec + step : nullptr, o.pv && room ? o.pv + step : nullptr,
                                o.pi && room ? o.pi + step : nullptr, o.mail);
            ++q;
        }
        __syncthreads();
    }
}

// The lumped elements' u^n before an E update (src/engine/lumped.rs:1106-1121).
__device__ __forceinline__ void serial_pre(const Fields& f, const ResOp* ops, uint32_t n_ops) {
    for (uint32_t q = 0; q < n_ops; ++q) {
        const ResOp& o = ops[q];
        if (o.kind != ResOp::LUMPED || !(o.lumped.record || o.lumped.has_branch)) continue;
        for (uint32_t e = threadIdx.x; e < o.lumped.n; e += blockDim.x) lumped_pre_e_edge(f.u[o.axis_l], o.lumped, e);
    }
}

// The serial hooks of a step that is not resident: one block, one launch for
// every hook of both sides (sides bit 0: current probes and H sources, bit 1:
// the electric ones) instead of one each: six launches of 2.5 us on a box with
// a source and five probes.
__global__ void __launch_bounds__(256) k_hooks(const __grid_constant__ Fields f, double dt, const ResOp* ops, uint32_t n_ops,
                                               uint64_t step, int sides) {
    after_previous();
    if (sides & 1) serial_hooks(f, dt, ops, n_ops, false, step, true, true);
    if (sides & 2) serial_hooks(f, dt, ops, n_ops, true, step, true, true);
}
__global__ void __launch_bounds__(256) k_hooks_pre(const __grid_constant__ Fields f, const ResOp* ops, uint32_t n_ops) {
    after_previous();
    serial_pre(f, ops, n_ops);
}

// One side of the poles: the correction, save_prev as in k_poles_blocks.
__device__ __forceinline__ void res_poles(const ResModel& R, bool electric, uint32_t t, uint32_t stride) {
    const BatchModel& M = R.m;
    const PoleSideDev& p = electric ? M.pe : M.ph;
    for (uint32_t e = t; e < (uint32_t)p.n_edges; e += stride)
        poles_edge(M.f, M.c, p, electric ? M.P.runs : M.P.runs_h, electric ? M.P.sets : M.P.sets_h,
                   M.run_of[electric ? 0 : 1], electric ? 1 : 0, M.dt, electric ? R.fold_e : R.fold_h, e);
}
__device__ __forceinline__ void res_capture(const ResModel& R, bool electric, uint32_t t, uint32_t stride) {
    const PoleSideDev& p = electric ? R.m.pe : R.m.ph;
    for (uint32_t e = t; e < (uint32_t)p.n_edges; e += stride)
        p.prev[e] = (electric ? R.m.f.u : R.m.f.i)[p.axis[e]][p.node[e]];
}

// One update (SIDE 0: H, 1: E) of the model's quads, worker t of `stride`.
template <int SIDE, bool OE>
__device__ __forceinline__ void res_update(const ResModel& R, uint32_t t, uint32_t stride) {
    const uint32_t nl = R.n_layer[SIDE];
    uint32_t x = t;
    uint2 next = x < nl ? __ldg(R.layer[SIDE] + x) : make_uint2(0u, 0u);
    for (; x < nl; x += stride) {
        const uint2 q = next;
        if (x + stride < nl) next = __ldg(R.layer[SIDE] + x + stride);
        const uint32_t row = quotient(R.div_q, q.x), i = quotient(R.div_j, row);
        const uint32_t j = row - i * R.div_j.d, k0 = (q.x - row * R.div_q.d) * 4u;
        if (SIDE == 0) split_h_at<false, OE, false, false, true>(R.m.P, i, j, k0, q.y);
        else split_e_at<OE, false, false, true>(R.m.P, i, j, k0, q.y);
    }
    const uint32_t ni = R.quads - nl;
    x -= nl;
    const uint32_t* list = R.inner[SIDE];
    uint32_t nq = list && x < ni ? __ldg(list + x) : x;
    for (; x < ni; x += stride) {
        const uint32_t q = nq;
        nq = list && x + stride < ni ? __ldg(list + x + stride) : x + stride;
        const uint32_t row = quotient(R.div_q, q), i = quotient(R.div_j, row);
        const uint32_t j = row - i * R.div_j.d, k0 = (q - row * R.div_q.d) * 4u;
        if (SIDE == 0) split_h_at<false, OE, false, false>(R.m.P, i, j, k0);
        else split_e_at<OE, false, false>(R.m.P, i, j, k0);
    }
}

// The slab hooks of one side after its update, each followed by a barrier of
// the gang; false once a wait has run out.
template <int SIDE>
__device__ __forceinline__ bool res_slabs(const ResModel& R, const ResArgs& A, Gang& G, uint32_t rank, int* ok) {
    const uint32_t t = rank * blockDim.x + threadIdx.x, stride = G.size * blockDim.x;
    for (int q = 0; q < 2 && R.order[q] >= 0; ++q) {
        if (R.order[q] == 0) {
            if (!R.units[SIDE] || R.quad_cpml) continue;
            for (uint32_t b = t >> 8; b < R.units[SIDE]; b += stride >> 8)
                shell_item<SIDE>(R.m.P, R.m.shell[SIDE], b, threadIdx.x & 255u);
        } else {
            const PoleSideDev& p = SIDE ? R.m.pe : R.m.ph;
            if (!p.n_edges) continue;
            res_poles(R, SIDE == 1, t, stride);
        }
        if (!gang_sync(G, A, ok)) return false;
    }
    return true;
}

// Barriers of a step: after the H update, after the E update, one more per
// slab operator but the CPML (and the CPML where it does not come first), one
// for hooks that write i and one for those that write u. In a gang of
// kHookGang blocks or more the last one takes no quads: it runs the hooks, the
// probes beside the other blocks' updates.
constexpr uint32_t kHookGang = 8;

template <bool OE>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(const __grid_constant__ ResArgs A) {
    __align__(16) EMS_GANG_SHARED unsigned char raw[sizeof(ResModel)];
    EMS_GANG_SHARED int ok;
    const ResModel& R = *reinterpret_cast<const ResModel*>(raw);
    const uint4 b = A.blocks[blockIdx.x];
    Gang G{A.bars + b.x * 32u, b.z, 0u};
    const uint32_t rank = b.y;
    if (blockIdx.x == 0)
        for (uint32_t w = threadIdx.x; w < A.n_bars; w += blockDim.x) A.bars_next[w * 32u] = 0u;
    if (threadIdx.x == 0) ok = 1;
    const uint2 span = A.gangs[b.x];
    for (uint32_t l = span.x; l < span.y; ++l) {
        const uint32_t id = A.list[l];
        __syncthreads();
        for (uint32_t w = threadIdx.x; w < sizeof(ResModel) / 4; w += blockDim.x)
            reinterpret_cast<uint32_t*>(raw)[w] = reinterpret_cast<const uint32_t*>(A.models + id)[w];
        __syncthreads();
        const uint32_t step0 = A.steps ? A.steps[id] : A.step0;
        const bool apart = R.n_ops && G.size >= kHookGang;
        const bool hooks = rank == (apart ? G.size - 1u : 0u);
        const uint32_t stride = (G.size - (apart ? 1u : 0u)) * blockDim.x;
        const uint32_t t = apart && hooks ? ~0u - 2u * stride : rank * blockDim.x + threadIdx.x;
        auto hook = [&](bool electric, uint32_t step, bool probes, bool writers) {
            serial_hooks(R.m.f, R.m.dt, R.ops, R.n_ops, electric, step, probes, writers);
        };
        for (uint32_t s = 0; s < A.n; ++s) {
            const uint32_t step = step0 + s;
            if (hooks) {
                // The lumped elements' u^n and the samples of u^n.
                serial_pre(R.m.f, R.ops, R.n_ops);
                if (R.late_probes && s) hook(true, step - 1u, true, false);
            }
            // The saved values of the other field's poles go beside an update: the
            // field does not change before the barrier behind it. (After that
            // barrier there may be none up to the update that writes the field.)
            if (!(apart && hooks)) {
                if (R.m.pe.n_edges && (!R.fold_e || (R.capture_first && s == 0))) res_capture(R, true, t, stride);
                res_update<0, OE>(R, t, stride);
            }
            if (!gang_sync(G, A, &ok)) return;
            if (!res_slabs<0>(R, A, G, rank, &ok)) return;
            // Hooks that write i before the E update, in order with the current
            // probes; else the probes beside it.
            if (hooks) hook(false, step, true, true);
            if (R.serial_h && !gang_sync(G, A, &ok)) return;
            if (!(apart && hooks)) {
                if (R.m.ph.n_edges && !R.fold_h) res_capture(R, false, t, stride);
                res_update<1, OE>(R, t, stride);
            }
            if (!gang_sync(G, A, &ok)) return;
            if (!res_slabs<1>(R, A, G, rank, &ok)) return;
            if (R.writes_e || (R.serial_e && !R.late_probes)) {
                if (hooks) hook(true, step, !R.late_probes, true);
                if (!gang_sync(G, A, &ok)) return;
            }
        }
        if (R.late_probes && hooks && A.n) hook(true, step0 + A.n - 1u, true, false);
        if (A.steps && hooks && threadIdx.x == 0) A.steps[id] = step0 + A.n;
    }
}

}  // namespace emsk
