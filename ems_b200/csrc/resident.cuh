// resident.cuh — many steps in one launch (sm_100a).
//
// On grids that fit in L2 a step of the split schedule is not bound by
// memory but by its launches: a 100^3 box takes ten of them, 62 us for about
// 15 us of L2 traffic. Here a gang of blocks advances a model by n steps in
// one cooperative launch: the phases of a step (H update, CPML of the H
// side, E update, CPML of the E side, poles, serial hooks) are the split
// schedule's device functions over strided work items, with a barrier of the
// gang between them in place of a kernel boundary. A batch gives every model
// a gang of its own, sized by its cells, so the models never wait for one
// another.
//
// The serial hooks run on the gang's first block in registration order, from
// amplitude tables and sample buffers on the device. Fields change within
// the launch, so they are read through the coherent path, never __ldg.
//
// A barrier wait is bounded: after kWaitNs the block sets the status flag and
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
    uint32_t n, hard, n_amp, cap;
    uint32_t interval, axis_l, has_src, pad;
    const uint32_t* node;
    const uint8_t* axis;
    const float* weight;
    const float* amp;
    const double* amp_l;
    double *values, *rec, *pv, *pi;  // series (index: step, or step / interval); null: not recorded
    ProbeDevT probe;
    LumpedDevT lumped;
};

// One model as the resident kernel reads it.
struct ResModel {
    BatchModel m;
    UpmlSideDev upml[2];
    const ResOp* ops;
    uint32_t n_ops;
    int32_t order[3];            // slab hooks in registration order: 0 CPML, 1 poles, 2 openEMS PML; -1 end
    int32_t fold_e, fold_h;      // the pole correction stores the saved values
    int32_t capture_first;       // fold_e, but the saved electric values are not current at the launch
    int32_t serial_h, serial_e;  // whether a post_h hook writes i, a post_e hook exists
    FastDiv div_q, div_j;        // quads per row, rows per plane
    uint32_t quads;              // nx·ny·quads per row
    uint32_t units[2];           // blocks of the shell kernels
    // The CPML comes first among the slab hooks: each thread applies it to the
    // quad it has just updated (quad_cpml_all). Per side, quads below z_lo or
    // reaching past z_hi may hold the slabs normal to z, z_bits.
    int32_t quad_cpml;
    uint32_t z_lo[2], z_hi[2], z_bits[2];
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
    uint64_t wait_ns;
};

// The barrier of a gang: every write of its blocks before it is visible to
// all of them after it. False once a wait has run out.
struct Gang {
    uint32_t* bar;
    uint32_t size, epoch;
    int* status;
    uint64_t wait_ns;
};
__device__ __forceinline__ bool gang_sync(Gang& G, int* ok) {
    __syncthreads();
    if (G.size == 1) return true;
    ++G.epoch;
    if (threadIdx.x == 0) {
        const uint32_t want = G.epoch * G.size;
        uint32_t v;
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(G.bar) : "memory");
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(G.bar) : "memory");
            if ((int32_t)(v - want) >= 0) break;
            if ((it & 255u) != 255u) continue;
            const uint64_t now = global_ns();
            if (!t0) t0 = now;
            if (now - t0 > G.wait_ns) {
                atomicExch(G.status, 1);
                *ok = 0;
                break;
            }
        }
        __threadfence();
    }
    __syncthreads();
    return *ok != 0;
}

// A probe's sample by one warp: the products in parallel, their sum in entry
// order (src/engine/probe.rs:381-392).
__device__ __forceinline__ void probe_warp(const Fields& f, bool electric, const ProbeDevT& p, double* out) {
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
    if (lane == 0) *out = p.f32_sum ? (double)s32 : s;
}

// The serial hooks of one field side at step `step`, by the gang's first
// block, in registration order; consecutive probes take a warp each.
__device__ __forceinline__ void serial_hooks(const ResModel& R, bool electric, uint32_t step) {
    const Fields& f = R.m.f;
    for (uint32_t q = 0; q < R.n_ops;) {
        const ResOp& o = R.ops[q];
        const bool mine = o.kind == ResOp::LUMPED ? electric : (o.electric != 0) == electric;
        if (!mine) {
            ++q;
            continue;
        }
        if (o.kind == ResOp::PROBE) {
            uint32_t end = q;
            while (end < R.n_ops && R.ops[end].kind == ResOp::PROBE) ++end;
            for (uint32_t r = q + (threadIdx.x >> 5); r < end; r += blockDim.x >> 5) {
                const ResOp& p = R.ops[r];
                if ((p.electric != 0) != electric || step % p.interval) continue;
                const uint32_t at = step / p.interval;
                if (at < p.cap) probe_warp(f, electric, p.probe, p.values + at);
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
            lumped_post_e_block(f.u[o.axis_l], o.lumped, val, o.has_src && val != 0.0, R.m.dt,
                                o.rec && room ? o.rec + step : nullptr, o.pv && room ? o.pv + step : nullptr,
                                o.pi && room ? o.pi + step : nullptr);
            ++q;
        }
        __syncthreads();
    }
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

// The CPML of one side at the quad a thread has just updated.
template <int SIDE>
__device__ __forceinline__ void res_quad_cpml(const ResModel& R, uint32_t i, uint32_t j, uint32_t k0) {
    uint32_t bits = row_slabs(R.m.P, SIDE, i, j);
    if (k0 < R.z_lo[SIDE] || k0 + 4u > R.z_hi[SIDE]) bits |= R.z_bits[SIDE];
    if (bits) quad_cpml_all<SIDE, true, false>(R.m.P, i, j, k0, bits);
}

// The slab hooks of one side after its update, each followed by a barrier of
// the gang; false once a wait has run out.
template <int SIDE>
__device__ __forceinline__ bool res_slabs(const ResModel& R, Gang& G, uint32_t rank, int* ok, bool capture) {
    const uint32_t t = rank * blockDim.x + threadIdx.x, stride = G.size * blockDim.x;
    // The saved values of the other field's poles: it does not change here.
    if (SIDE == 0 && capture) res_capture(R, true, t, stride);
    if (SIDE == 1 && R.m.ph.n_edges && !R.fold_h) res_capture(R, false, t, stride);
    for (int q = 0; q < 3 && R.order[q] >= 0; ++q) {
        if (R.order[q] == 0) {
            if (!R.units[SIDE] || R.quad_cpml) continue;
            for (uint32_t b = t >> 8; b < R.units[SIDE]; b += stride >> 8)
                shell_item<SIDE>(R.m.P, R.m.shell[SIDE], b, threadIdx.x & 255u);
        } else if (R.order[q] == 1) {
            const PoleSideDev& p = SIDE ? R.m.pe : R.m.ph;
            if (!p.n_edges) continue;
            res_poles(R, SIDE == 1, t, stride);
        } else {
            const UpmlSideDev &a = R.upml[SIDE ? 0 : 1], &r = R.upml[SIDE ? 1 : 0];
            for (uint32_t e = t; e < r.n; e += stride) r.v[e] = (SIDE ? R.m.f.i : R.m.f.u)[r.axis[e]][r.node[e]];
            for (uint32_t e = t; e < a.n; e += stride) upml_apply((SIDE ? R.m.f.u : R.m.f.i)[a.axis[e]], a, e);
        }
        if (!gang_sync(G, ok)) return false;
    }
    return true;
}

template <bool OE>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(const __grid_constant__ ResArgs A) {
    __shared__ __align__(16) unsigned char raw[sizeof(ResModel)];
    __shared__ int ok;
    const ResModel& R = *reinterpret_cast<const ResModel*>(raw);
    const uint4 b = A.blocks[blockIdx.x];
    Gang G{A.bars + b.x * 32u, b.z, 0u, A.status, A.wait_ns};
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
        const uint32_t t = rank * blockDim.x + threadIdx.x, stride = G.size * blockDim.x;
        for (uint32_t s = 0; s < A.n; ++s) {
            const uint32_t step = step0 + s;
            // The lumped elements' u^n: the E update is two barriers away.
            if (rank == 0)
                for (uint32_t q = 0; q < R.n_ops; ++q) {
                    const ResOp& o = R.ops[q];
                    if (o.kind != ResOp::LUMPED || !(o.lumped.record || o.lumped.has_branch)) continue;
                    for (uint32_t e = threadIdx.x; e < o.lumped.n; e += blockDim.x)
                        lumped_pre_e_edge(R.m.f.u[o.axis_l], o.lumped, e);
                }
            for (uint32_t q = t; q < R.quads; q += stride) {
                const uint32_t row = quotient(R.div_q, q), i = quotient(R.div_j, row);
                const uint32_t j = row - i * R.div_j.d, k0 = (q - row * R.div_q.d) * 4u;
                split_h_at<false, OE, false, false>(R.m.P, i, j, k0);
                if (R.quad_cpml) res_quad_cpml<0>(R, i, j, k0);
            }
            if (!gang_sync(G, &ok)) return;
            if (!res_slabs<0>(R, G, rank, &ok, R.m.pe.n_edges && (!R.fold_e || (R.capture_first && s == 0)))) return;
            // Hooks that write i before the E update; current probes beside it.
            if (rank == 0) serial_hooks(R, false, step);
            if (R.serial_h && !gang_sync(G, &ok)) return;
            for (uint32_t q = t; q < R.quads; q += stride) {
                const uint32_t row = quotient(R.div_q, q), i = quotient(R.div_j, row);
                const uint32_t j = row - i * R.div_j.d, k0 = (q - row * R.div_q.d) * 4u;
                split_e_at<OE, false, false>(R.m.P, i, j, k0);
                if (R.quad_cpml) res_quad_cpml<1>(R, i, j, k0);
            }
            if (!gang_sync(G, &ok)) return;
            if (!res_slabs<1>(R, G, rank, &ok, false)) return;
            if (R.serial_e) {
                if (rank == 0) serial_hooks(R, true, step);
                if (!gang_sync(G, &ok)) return;
            }
        }
        if (A.steps && rank == 0 && threadIdx.x == 0) A.steps[id] = step0 + A.n;
    }
}

}  // namespace emsk
