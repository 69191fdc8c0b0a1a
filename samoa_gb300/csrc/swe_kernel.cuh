// The fused SWE time-step kernel (sm_103a).
//
// One launch of step_kernel = one explicit Euler time step of every instance of
// the context (one instance for the plain step, many for an ensemble) of
// t_swe_euler_timestep_traversal (src/SWE/SWE_euler_timestep.f90); on meshes
// that fit the GPU at once a launch of multi_step_kernel (at the end of this
// file) runs many. Cells are cut into segments of consecutive cells of the
// space-filling curve; a segment never spans two instances. A persistent grid
// of CTAs walks the segments; per segment:
//   1. stage h, hu, hv, b into shared memory with 1-D TMA bulk copies
//      (cp.async.bulk, completion on an mbarrier with a bounded wait), then
//      the depth h - b and sqrt(g * depth) once per cell;
//   2. evaluate each edge task once: the Riemann solver with the first-touched
//      cell as the left side writes left/right updates into per-(cell, local
//      edge) slots in shared memory, each slot written by one task, no atomics;
//      an edge between two segments is evaluated once by cross_edges_kernel
//      before, or by both CTAs, each keeping its own side, so that no CTA waits
//      for another;
//   3. update each cell from its three slots in local edge index order, clamp
//      wet/dry, write the other state buffer, set the refinement flag, fold
//      volume / sum(len * speed) into a running minimum;
// at an instance change and at the end the CTA reduces the minimum with warp
// shuffles and folds it into the instance with one atomic; the last CTA to
// finish advances every instance's time and dt and the step counter.
// The reference's traversal direction alternates every step
// (src/SFC_generic_traversal_ringbuffer.f90:420): on odd steps the
// higher-numbered cell of an edge is touched first and the two leg updates are
// summed in the other order.
#pragma once

// The kernels are compiled twice: in namespace swe with strict IEEE rounding
// (no contraction) and in namespace swe_fma with FMA contraction (SWE_KNS).
#ifndef SWE_KNS
#define SWE_KNS swe
#endif

#include <cfloat>
#include <cstdint>

#include "swe_internal.h"
#include "swe_riemann.cuh"

namespace SWE_KNS {
using namespace ::swe;

__constant__ double c_leg[kMaxDepth + 2];  // sqrt(0.5)**i at [i + 1], i = -1..60
__constant__ double c_vol[kMaxDepth + 1];  // 0.5**(i + 1)
__constant__ double c_normal[17][3][2];    // [plotter + 8][local edge][x, y]

struct StepArgs {
    double* h[2];
    double* hu[2];
    double* hv[2];
    const double* b;
    const int8_t* depth;
    int8_t* flags;
    const int4* tasks;
    const long long* seg_ptr;
    const int4* seg_info;      // {first cell, cells, instance, halo tasks at the end of its list}
    const int32_t* seg_order;  // the order segments are handed out in (a permutation), or null: curve order
    const int4* xtasks;        // cross-segment edges (Task layout, pad = instance)
    double* xflux;             // [n_xtasks][cell a, cell b][h, hu, hv, max wave speed] of the current step
    long long n_xtasks;
    uint16_t* erec;            // branch-frozen runs: this step's edge decisions, per task ...
    uint16_t* xrec;            // ... and per cross-segment edge
    const InstParams* ip;
    const DepthRow* rows;      // [instance][max_ndepth]
    InstScalars* is;
    GlobalScalars* gs;
    uint8_t* branch;           // optional per-cell output: bit 0 wetting fix, bit 1 drying clamp (adjoint)
    const double* dt_seq;      // frozen dt sequence [k * n_inst + inst] or null
    long long dt_seq_len;      // steps in the sequence
    int32_t n_seg, n_inst, seg_cells, max_ndepth, n_cells_total;
    int32_t use_tma;
    int32_t fixed_io;          // 1: read h[0], hu[0], hv[0] and write h[1].. on every step (caller's buffers)
    int32_t stage_depth;       // 1: stage a segment, then work on it; 2: stage the next one meanwhile
    int32_t halo_solve;        // 1: solve the halo tasks here (no cross-edge pass); 0: copy the pass's updates
    double2* memo;             // per cell (d, sqrt(g d)) of an earlier step, or null: see the staging loop
    uint32_t extra_tx;         // fault injection only: bytes the staging barrier expects beyond the copies (0)
    unsigned long long wait_ns;  // limit of one mbarrier wait, in ns of the global timer
};

// Launch bounds of the step kernel: at most 256 threads; with SWE_MIN_BLOCKS
// defined, also that many resident CTAs of 256 threads (registers capped at
// 65536 / (256 * SWE_MIN_BLOCKS)). Undefined: the compiler's own register choice.
#ifdef SWE_MIN_BLOCKS
#define SWE_STEP_BOUNDS __launch_bounds__(256, SWE_MIN_BLOCKS)
#else
#define SWE_STEP_BOUNDS __launch_bounds__(256)
#endif

// An mbarrier wait gives up after wait_ns of the global timer (1 s by default;
// the copies it waits for take microseconds), or after kPollLimit polls
// whatever the timer says, so that every wait ends.
constexpr unsigned long long kWaitNs = 1000000000ull;
constexpr unsigned int kPollLimit = 1u << 30;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// 1-D bulk copy global -> this CTA's shared memory; addresses 16-byte aligned,
// size a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Prefetch into L2 the 16-byte-aligned part of [p, p + bytes), for any p (the
// bulk prefetch wants a 16-byte aligned address and size): it touches no byte
// outside the range, writes nothing, and has no completion to wait for.
__device__ __forceinline__ void prefetch_l2(const void* p, size_t bytes) {
    const uintptr_t a = ((uintptr_t)p + 15u) & ~(uintptr_t)15u, e = ((uintptr_t)p + bytes) & ~(uintptr_t)15u;
    if (e > a)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)(e - a)));
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// Warp-wide maximum of u64 values: of the high words, then of the low words among the lanes that hold it.
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
    const unsigned hi = (unsigned)(v >> 32);
    const unsigned m = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, hi == m ? (unsigned)v : 0u);
    return ((unsigned long long)m << 32) | lo;
}

// grid%r_dt clamped as in pre_traversal_grid_op (src/SWE/SWE_euler_timestep.f90:89-109)
__device__ __forceinline__ double clamp_dt(double dt, double max_time, double tout) {
    if (max_time > 0.0) dt = dmn(max_time, dt);
    if (tout > 0.0) dt = dmn(tout, dt);
    return dt;
}

// grid%r_dt_new from the reductions of a step (the smallest volume / ds, or the
// bits x of the largest ds 2^(d+1))
__device__ __forceinline__ double dt_new_of(const InstParams& P, double dt_acc, unsigned long long x) {
    return x ? dmn(dt_acc, div_one(P.scaling * P.scaling, __longlong_as_double((long long)x))) : dt_acc;
}

// The scalars after a step (post_traversal_grid_op, src/SWE/SWE_euler_timestep.f90:111-131)
__device__ __forceinline__ void advance_time(InstScalars* S, const InstParams& P, double time, double dt_acc,
                                             unsigned long long x, unsigned long long n_refine) {
    const double dtn = dt_new_of(P, dt_acc, x);
    S->time = time;
    S->dt_new = dtn;
    S->dt = P.courant * dtn;
    S->n_refine = n_refine;
}

// What the CTA's threads reduce over the cells of an instance: the bits of the
// largest ds 2^(d+1) (dt_by_max) or the complement of the bits of the smallest
// volume / ds (non-negative doubles order like their bits, and the complement
// turns the minimum into a maximum), and the refinements.
struct Reduced {
    unsigned long long key;
    int nref;
};
struct RedSlots {
    unsigned long long key[8];
    int nref[8];
};
__device__ __forceinline__ void warp_reduce(const Reduced& r, RedSlots& slots) {
    const unsigned long long k = warp_max_u64(r.key);
    const int n = __reduce_add_sync(0xffffffffu, r.nref);
    if ((threadIdx.x & 31) == 0) {
        slots.key[threadIdx.x >> 5] = k;
        slots.nref[threadIdx.x >> 5] = n;
    }
}
__device__ __forceinline__ Reduced block_reduced(const RedSlots& slots) {  // after a barrier
    Reduced r{0ull, 0};
    const int nw = (blockDim.x + 31) >> 5;
    for (int w = 0; w < nw; ++w) {
        r.key = slots.key[w] > r.key ? slots.key[w] : r.key;
        r.nref += slots.nref[w];
    }
    return r;
}
// The CTA's reductions into instance `inst`; all threads call it.
__device__ __forceinline__ void flush_instance(const StepArgs& A, int inst, bool by_max, Reduced& r, RedSlots& slots) {
    warp_reduce(r, slots);
    __syncthreads();
    if (threadIdx.x == 0) {
        const Reduced b = block_reduced(slots);
        if (by_max) {
            if (b.key) atomicMax(&A.is[inst].ds_acc, b.key);
        } else if (b.key) {
            atomicMin(&A.is[inst].dt_acc, ~b.key);
        }
        if (b.nref) atomicAdd(&A.is[inst].refine_acc, (unsigned long long)b.nref);
    }
    r = Reduced{0ull, 0};
}

// The edges between two segments, one thread each, before the step kernel:
// the same flux as the step kernel's edge tasks (orientation by the step's
// parity, pre-update states), both sides' updates stored by cell (a, then b).
// depth_terms for the cross-edge pass: sqrt(g d) from the memo when the depth has
// the same bits (the pass only reads it; the step kernel's owner CTAs write it),
// and, for the f-wave, no reciprocal for a cell with both momenta +-0 (its
// quotients are zeros with the numerator's sign, which need none).
template <int SOLVER>
__device__ __forceinline__ void cross_depth_terms(const StepArgs& A, int c, const State& Q, double drytol, double& d,
                                                  double& sq, u64& y) {
    d = Q.h - Q.b;
    const bool wet = lt(drytol, d);
    sq = 0.0;
    y = 0;
    if (!wet) return;
    bool hit = false;
    if (A.memo) {
        const double2 m = A.memo[c];
        if (dbits(m.x) == dbits(d)) {
            sq = m.y;
            hit = true;
        }
    }
    SWE_IF(!hit) sq = sqrt_fix(kG * d);
    const bool still = ((dbits(Q.p1) | dbits(Q.p2)) << 1) == 0;
    y = (SOLVER == FWAVE && still) ? 0 : recip_fix(d);
}

template <int SOLVER>
static __device__ __noinline__ void cross_edge_redo(const StepArgs& A, long long j);

template <int SOLVER, int FZ, class Ops>
__device__ __forceinline__ void cross_edge(const StepArgs& A, long long j) {
    const long long step = A.gs->step;
    const int odd = (int)(step & 1);
    const int ib = A.fixed_io ? 0 : odd;
    const double* hin = A.h[ib];
    const double* huin = A.hu[ib];
    const double* hvin = A.hv[ib];
    const int4 tk = __ldg(&A.xtasks[j]);
    const uint32_t meta = (uint32_t)tk.z;
    int L, R, iL, pL;
    if (!odd) {
        L = tk.x; iL = meta & 3u; pL = (meta >> 4) & 31u;
        R = tk.y;
    } else {
        L = tk.y; iL = (meta >> 2) & 3u; pL = (meta >> 9) & 31u;
        R = tk.x;
    }
    if ((unsigned)L >= (unsigned)A.n_cells_total || (unsigned)R >= (unsigned)A.n_cells_total || iL > 2 ||
        pL > 16 || (unsigned)tk.w >= (unsigned)A.n_inst || ((meta >> 14) & 1u)) {
        atomicOr(&A.gs->error, 1u);
        return;
    }
    const double drytol = A.ip[tk.w].drytol;
    const double n1 = c_normal[pL][iL][0], n2 = c_normal[pL][iL][1];
    const State QL{hin[L], huin[L], hvin[L], A.b[L]};
    const State QR{hin[R], huin[R], hvin[R], A.b[R]};
    double dL, dR, sqL, sqR;
    u64 yL, yR;
    cross_depth_terms<SOLVER>(A, L, QL, drytol, dL, sqL, yL);
    cross_depth_terms<SOLVER>(A, R, QR, drytol, dR, sqR, yR);
    Update fL, fR;
    Ops o;
    edge_flux<SOLVER, FZ>(n1, n2, QL, QR, dL, dR, sqL, sqR, yL, yR, drytol, fL, fR, (int)((meta >> 15) & 3u),
                          FZ ? &A.xrec[j] : nullptr, o);
    if (!o.ok) {
        cross_edge_redo<SOLVER>(A, j);
        return;
    }
    const Update& ua = odd ? fR : fL;
    const Update& ub = odd ? fL : fR;
    double2* out = reinterpret_cast<double2*>(A.xflux + 8 * j);
    out[0] = make_double2(ua.h, ua.p1);
    out[1] = make_double2(ua.p2, ua.s);
    out[2] = make_double2(ub.h, ub.p1);
    out[3] = make_double2(ub.p2, ub.s);
}

template <int SOLVER>
static __device__ __noinline__ void cross_edge_redo(const StepArgs& A, long long j) {
    cross_edge<SOLVER, 0, SafeOps>(A, j);
}

template <int SOLVER, int FZ = 0>
__global__ void __launch_bounds__(256) cross_edges_kernel(const __grid_constant__ StepArgs A) {
    const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= A.n_xtasks) return;
    if (FZ) cross_edge<SOLVER, FZ, SafeOps>(A, j);
    else cross_edge<SOLVER, 0, FastOps>(A, j);
}

// Round-up float of |x| for x = +-0 or 2^-100 <= |x| < 2^101, from the bit
// pattern (integer operations): the significand truncated to 23 bits plus one
// unit in the last place (a carry into the exponent is still an upper bound).
// False for other x (tiny, huge, inf, NaN).
__device__ __forceinline__ bool float_up(double x, float& f) {
    const unsigned long long a = (unsigned long long)abs_bits(x);
    f = 0.0f;
    if (a == 0ull) return true;
    const int e = (int)(a >> 52) - 1023;
    if (e < -100 || e > 100) return false;
    f = __uint_as_float(((unsigned)(e + 127) << 23 | (unsigned)((a >> 29) & 0x7fffffull)) + 1u);
    return true;
}

// True when the CFL key RN(ds 2^k) of a cell is certainly below the key m (bits
// of a nonnegative double), so that the cell cannot raise a maximum >= m; ds =
// RN(RN(RN(leg s0) + RN(hyp s1)) + RN(leg s2)) is the cell update's speed sum,
// up = (leg, hyp) rounded up to float. U = leg s0 + hyp s1 + leg s2 evaluated in
// float with every operand and every operation rounded up bounds the exact sum
// of the magnitudes S; the three roundings of ds give |ds| <= S (1 + 2^-53)^3
// (and an absolute error below 2^-1072 where a result is subnormal), both below
// the margin U 2^-20 of a normal float U; 2^k scales exactly, and a bound that
// is not a finite double gives false. The float work runs beside the FP64 pipe.
__device__ __forceinline__ bool key_below(float2 up, double s0, double s1, double s2, int k, unsigned long long m) {
    float f0, f1, f2;
    if (!float_up(s0, f0) || !float_up(s1, f1) || !float_up(s2, f2)) return false;
    float U = __fmaf_ru(up.x, f0, __fmaf_ru(up.y, f1, __fmul_ru(up.x, f2)));
    U = __fmul_ru(U, 1.00000095367431640625f);  // 1 + 2^-20
    const unsigned int ub = __float_as_uint(U);
    const int ef = (int)(ub >> 23);  // U >= 0
    if (ef == 0 || ef == 255) return false;
    const int eb = ef - 127 + 1023 + k;
    if (eb >= 2047) return false;
    const unsigned long long bound = ((unsigned long long)eb << 52) | ((unsigned long long)(ub & 0x7fffffu) << 29);
    return bound < m;
}

// The depth-dependent values of the running instance, in shared memory.
struct DepthTab {
    double* leg;
    double* hyp;
    double* vol;
    double* pow;  // 2^(d+1)
    double* ndv;  // -dt / volume
    float2* up;   // (leg, hyp) rounded up to float
    __device__ __forceinline__ DepthTab(double* base, int n)
        : leg(base), hyp(base + n), vol(base + 2 * n), pow(base + 3 * n), ndv(base + 4 * n),
          up(reinterpret_cast<float2*>(base + 5 * n)) {}
    __device__ __forceinline__ void load(const StepArgs& A, int inst, int i) const {
        const DepthRow* row = A.rows + (size_t)inst * A.max_ndepth + i;
        leg[i] = row->leg;
        hyp[i] = row->hyp;
        vol[i] = row->vol;
        pow[i] = row->pow;
        up[i] = make_float2(row->leg_up, row->hyp_up);
    }
};

// A segment's working set in shared memory.
struct SegMem {
    int T;
    double* h;    // staged h, hu, hv, b: [4][T]
    u64* rh;      // recip_fix(depth) where the cell is wet
    double* sq;   // sqrt(g * depth) where the cell is wet
    double* upd;  // [4 quantities][3 local edges][T]
    double* d;    // depth h - b, in an array of its own or in the staged surface's place (h)
    double* tab;  // DepthTab's
    int8_t* dep;  // the cells' refinement depths
    // The arrays after the staging buffers.
    __device__ __forceinline__ void lay_out(double* after, bool own_d, int max_ndepth) {
        rh = reinterpret_cast<u64*>(after);
        sq = after + T;
        upd = after + 2 * T;
        d = own_d ? after + 14 * T : nullptr;
        tab = after + (own_d ? 15 : 14) * T;
        dep = reinterpret_cast<int8_t*>(tab + 6 * max_ndepth);
    }
    __device__ __forceinline__ double* hu() const { return h + T; }
    __device__ __forceinline__ double* hv() const { return h + 2 * T; }
    __device__ __forceinline__ double* b() const { return h + 3 * T; }
};

__host__ __device__ constexpr bool geoclaw(int solver) { return solver == FWAVE || solver == AUG_RIEMANN; }

// One edge task (skeleton_scalar_op / bnd_skeleton_scalar_op,
// src/SWE/SWE_euler_timestep.f90:196-255): the updates of both sides into the
// slots of the cells in the segment. With SHARED_STATE other CTAs write the
// neighbours' state in this launch, so it is read past the L1 cache. DEPTHS: M.d holds
// the depths. Returns 0, kBadIndex, or kRedo where FastOps does not take the edge's
// operands (nothing is written then).
constexpr unsigned int kBadIndex = 1u, kRedo = 8u;
template <int SOLVER, int FZ, bool SHARED_STATE, bool DEPTHS, class Ops>
__device__ __forceinline__ unsigned int edge_task_with(const StepArgs& A, const SegMem& M, const int4 tk, uint16_t* erec,
                                                  int c0, int cn, int odd, double drytol, int bc, const double* hin,
                                                       const double* huin, const double* hvin) {
    const int T = M.T;
    const uint32_t meta = (uint32_t)tk.z;
    const bool bnd = (meta >> 14) & 1u;
    int L, R, iL, iR, pL;
    if (bnd || !odd) {
        L = tk.x; iL = meta & 3u; pL = (meta >> 4) & 31u;
        R = tk.y; iR = (meta >> 2) & 3u;
    } else {
        L = tk.y; iL = (meta >> 2) & 3u; pL = (meta >> 9) & 31u;
        R = tk.x; iR = meta & 3u;
    }
    if ((unsigned)L >= (unsigned)A.n_cells_total || (!bnd && (unsigned)R >= (unsigned)A.n_cells_total) || iL > 2 ||
        iR > 2 || pL > 16)
        return kBadIndex;
    const double n1 = c_normal[pL][iL][0], n2 = c_normal[pL][iL][1];
    const int sl = L - c0, sr = R - c0;
    const bool lin = (unsigned)sl < (unsigned)cn;
    const bool rin = !bnd && (unsigned)sr < (unsigned)cn;
    State QL, QR;
    double dL, dR, sqL, sqR;
    u64 yL, yR;
    auto far = [&](int c, State& Q, double& d, double& sq, u64& y) {
        if (SHARED_STATE) Q = State{__ldcg(hin + c), __ldcg(huin + c), __ldcg(hvin + c), A.b[c]};
        else Q = State{hin[c], huin[c], hvin[c], A.b[c]};
        depth_terms(Q, drytol, d, sq, y);
    };
    auto near = [&](int i, State& Q, double& d, double& sq, u64& y) {
        Q = State{M.h[i], M.hu()[i], M.hv()[i], M.b()[i]};  // (h is d where d took its place)
        d = DEPTHS ? M.d[i] : Q.h - Q.b;
        sq = M.sq[i];
        y = M.rh[i];
    };
    if (lin) near(sl, QL, dL, sqL, yL);
    else far(L, QL, dL, sqL, yL);
    if (bnd) {  // the ghost has the cell's h and b
        if (bc == BC_SLIP) QR = boundary_ghost<BC_SLIP>(n1, n2, QL);
        else if (bc == BC_NOSLIP) QR = boundary_ghost<BC_NOSLIP>(n1, n2, QL);
        else QR = QL;
        dR = dL;
        sqR = sqL;
        yR = yL;
    } else if (rin) {
        near(sr, QR, dR, sqR, yR);
    } else {
        far(R, QR, dR, sqR, yR);
    }
    Update fL, fR;
    Ops o;
    constexpr bool kSurface = SHARED_STATE || !DEPTHS;  // the multi-step kernel has the depths in an array of their own
    edge_flux<SOLVER, FZ, kSurface>(n1, n2, QL, QR, dL, dR, sqL, sqR, yL, yR, drytol, fL, fR, (int)((meta >> 15) & 3u),
                                    erec, o);
    if (!o.ok) return kRedo;
    if (lin) {
        M.upd[(0 * 3 + iL) * T + sl] = fL.h;
        M.upd[(1 * 3 + iL) * T + sl] = fL.p1;
        M.upd[(2 * 3 + iL) * T + sl] = fL.p2;
        M.upd[(3 * 3 + iL) * T + sl] = fL.s;
    }
    if (rin) {
        M.upd[(0 * 3 + iR) * T + sr] = fR.h;
        M.upd[(1 * 3 + iR) * T + sr] = fR.p1;
        M.upd[(2 * 3 + iR) * T + sr] = fR.p2;
        M.upd[(3 * 3 + iR) * T + sr] = fR.s;
    }
    return 0u;
}

// The task again with SafeOps (a call, so that the callers keep their registers;
// it reads the operands again, so that they need not hold them either).
template <int SOLVER, bool SHARED_STATE, bool DEPTHS>
static __device__ __noinline__ unsigned int edge_task_redo(const StepArgs& A, const SegMem M, const int4 tk, int c0,
                                                           int cn, int odd, double drytol, int bc, int ib) {
    return edge_task_with<SOLVER, 0, SHARED_STATE, DEPTHS, SafeOps>(A, M, tk, nullptr, c0, cn, odd, drytol, bc, A.h[ib],
                                                            A.hu[ib], A.hv[ib]);
}
template <int SOLVER, int FZ, bool SHARED_STATE, bool DEPTHS>
__device__ __forceinline__ unsigned int edge_task(const StepArgs& A, const SegMem& M, const int4 tk, uint16_t* erec,
                                                  int c0, int cn, int odd, double drytol, int bc, int ib) {
    if (FZ)
        return edge_task_with<SOLVER, FZ, SHARED_STATE, DEPTHS, SafeOps>(A, M, tk, erec, c0, cn, odd, drytol, bc, A.h[ib],
                                                                 A.hu[ib], A.hv[ib]);
    unsigned int rc = edge_task_with<SOLVER, 0, SHARED_STATE, DEPTHS, FastOps>(A, M, tk, nullptr, c0, cn, odd, drytol, bc,
                                                                       A.h[ib], A.hu[ib], A.hv[ib]);
    if (rc == kRedo) rc = edge_task_redo<SOLVER, SHARED_STATE, DEPTHS>(A, M, tk, c0, cn, odd, drytol, bc, ib);
    return rc;
}

// A cell's new state, its flag and its branch bits (cell_update_op + volume_op,
// src/SWE/SWE_euler_timestep.f90:257-355); folds its CFL term and refinement
// into r. wkey: a lower bound of the largest CFL key the lanes of this warp have
// taken so far (dt_by_max); a cell whose key is certainly below it cannot raise
// the maximum. rb: the recorded fixes of a branch-frozen run (FZ = 2).
struct CellOut {
    double h, p1, p2;
    int8_t flag;
    uint8_t branch;
};
__device__ __forceinline__ int high_word(double x) { return (int)(dbits(x) >> 32); }
static __device__ __noinline__ double quotient(double a, double b) { return div_one(a, b); }
template <int FZ>
__device__ __forceinline__ CellOut update_cell(const SegMem& M, const DepthTab& tab, const InstParams& P, int i,
                                               double h, double depth, int odd, unsigned long long wkey, uint8_t rb, Reduced& r) {
    const int T = M.T, k0 = odd ? 2 : 0, k2 = odd ? 0 : 2;
    const int d = M.dep[i];
    const int di = d - P.dmin;
    const double leg = tab.leg[di], hyp = tab.hyp[di], ndv = tab.ndv[di];
    double u[4][3];
    long long nz = 0, sz = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        u[q][0] = M.upd[(q * 3 + k0) * T + i];
        u[q][1] = M.upd[(q * 3 + 1) * T + i];
        u[q][2] = M.upd[(q * 3 + k2) * T + i];
        (q < 3 ? nz : sz) |= (dbits(u[q][0]) | dbits(u[q][1]) | dbits(u[q][2])) << 1;
    }
    // quiet: every update of h, hu, hv is +-0 (dry land, water at rest). Then
    // each sum below is +0 (positive edge lengths), RN(ndv * +0) is a zero with
    // ndv's sign, and adding it leaves the state as add_zero says: the same
    // bits, without the FP64 arithmetic. Water at rest still has wave speeds,
    // so the speed sum ds has its own test.
    const bool quiet = nz == 0 && is_finite(ndv);
    // ds is +0 when every speed is +-0 (dry land) or when the cell's key stays
    // below wkey (key_below), else it is summed
    double ds = 0.0;
    bool need_ds = sz != 0;
    if (need_ds && wkey != 0ull) need_ds = !key_below(tab.up[di], u[3][0], u[3][1], u[3][2], d + 1, wkey);
    SWE_IF(need_ds) {
        ds = z0(prod_cell(leg, u[3][0])) + prod_cell(hyp, u[3][1]);
        ds = ds + prod_cell(leg, u[3][2]);
    }
    // ds >= 0, so its bits order like its value; RN(ds * 2^(d+1))
    unsigned long long key = (unsigned long long)dbits(scaled(dbits(ds), d + 1));
    SWE_IF(!P.dt_by_max || !scales(dbits(ds), d + 1)) {
        if (P.dt_by_max) {
            key = (unsigned long long)dbits(ds * tab.pow[di]);
        } else {  // r_dt_new = min(huge, volume / ds): a NaN quotient never wins
            const double q = quotient(tab.vol[di], ds);
            key = q < DBL_MAX ? ~(unsigned long long)dbits(q) : 0ull;
        }
    }
    r.key = key > r.key ? key : r.key;
    double p1 = M.hu()[i], p2 = M.hv()[i];
    const double b = M.b()[i];
    uint8_t br = 0;
    long long nrm = 0;  // bits of |sum of the lengths times the updates of h|
    // A wet cell (sq > 0: RN(h - b) > drytol, so h > b + drytol and h >= bdry) cannot
    // be below bdry now, and not after a quiet update either: it needs no bdry.
    const bool deep = FZ == 0 && dbits(M.sq[i]) != 0;
    if (quiet) {
        const double z = bitsd(dbits(ndv) & (long long)0x8000000000000000ULL);  // RN(ndv * +0)
        double h1 = add_zero(h, z), q1 = add_zero(p1, z), q2 = add_zero(p2, z);
        SWE_IF(!deep) {
            const double bdry = b + P.drytol;
            // (no flooding: the update is not positive) a branch-frozen run takes the recorded fixes
            if (FZ == 2 && (rb & 1u) != 0) {
                h1 = bdry + z;
                q1 = q2 = 0.0 + z;
                br = 1;
            }
            if (FZ == 2 ? (rb & 2u) != 0 : lt(h1, bdry)) {  // dried out: surface to min(b, 0), at rest
                h1 = lt0(b) ? b : 0.0;
                q1 = q2 = 0.0;
                br |= 2;
            }
        }
        h = h1;
        p1 = q1;
        p2 = q2;
    }
    SWE_IF(!quiet) {
        double dh = z0(prod_cell(leg, u[0][0])) + prod_cell(hyp, u[0][1]);
        dh = dh + prod_cell(leg, u[0][2]);
        double dp1 = z0(prod_cell(leg, u[1][0])) + prod_cell(hyp, u[1][1]);
        dp1 = dp1 + prod_cell(leg, u[1][2]);
        double dp2 = z0(prod_cell(leg, u[2][0])) + prod_cell(hyp, u[2][1]);
        dp2 = dp2 + prod_cell(leg, u[2][2]);
        nrm = abs_bits(dh);
        dh = prod_cell(ndv, dh);
        dp1 = prod_cell(ndv, dp1);
        dp2 = prod_cell(ndv, dp2);
        // A wet cell that certainly stays wet, from the high words, without b + drytol: with
        // depth = RN(h - b) in [2^e, 2^(e + 1)), |dh| and drytol at most depth / 8 (and 2^(e - 23)),
        // the sums h + dh and b + drytol are at least depth / 2 apart, and with |h| and |b| below
        // 2^(e + 47) their roundings move them by less than 2^(e - 5). The words of
        // infinities and NaN are above every bound.
        const int room = high_word(depth);
        const bool stays = deep & (max(high_word(iabs(dh)), high_word(P.drytol)) <= room - (3 << 20)) &
                           (max(high_word(iabs(h)), high_word(iabs(b))) - (45 << 20) <= room) & (room < (1900 << 20));
        double bdry = 0.0;
        SWE_IF(!stays) {
            bdry = b + P.drytol;
            // flooded land starts at the dry tolerance, at rest
            if (FZ == 2 ? (rb & 1u) != 0 : (!deep && lt(h, bdry) && gt0(dh))) {
                h = bdry;
                p1 = 0.0;
                p2 = 0.0;
                br = 1;
            }
        }
        h = h + dh;
        p1 = p1 + dp1;
        p2 = p2 + dp2;
        if (!stays && (FZ == 2 ? (rb & 2u) != 0 : lt(h, bdry))) {  // dried out: surface to min(b, 0), at rest
            h = lt0(b) ? b : 0.0;
            p1 = 0.0;
            p2 = 0.0;
            br |= 2;
        }
    }
    CellOut o;
    o.flag = 0;
    // |dh| > thr and |dh| < thr / 8 on the bit patterns (thresholds are positive;
    // a NaN |dh| passes neither test, as in IEEE)
    if (d < P.max_depth && not_nan(nrm) && nrm > __double_as_longlong(P.thr_refine)) {
        o.flag = 1;
        ++r.nref;
    } else if (d > P.min_depth && nrm < __double_as_longlong(P.thr_coarsen)) {
        o.flag = -1;
    }
    o.h = h;
    o.p1 = p1;
    o.p2 = p2;
    o.branch = br;
    return o;
}

// A lower bound of the largest key in the warp: its high word.
__device__ __forceinline__ unsigned long long warp_key_bound(unsigned long long key) {
    return (unsigned long long)__reduce_max_sync(0xffffffffu, (unsigned)(key >> 32)) << 32;
}

// The GeoClaw edges read a cell's depth instead of subtracting twice per edge (3 FP64
// instructions per cell): it takes the staged surface's place, and the cell update reads
// the surface from memory again (from the L2 cache). An array of its own would take the
// place of 32 of a segment's 384 cells; a segment of 352 with it measured 2495 us for 4
// steps of a 2^22-cell bowl and 2276 of a 2^23-cell basin against 2489 and 2245. Where
// the state is in host memory (HOST) the second read would cross the link again (2^20
// cells: 294 us against 275), so there the edges subtract; the Lax-Friedrichs edges need
// the surface.
template <int SOLVER, int FZ = 0, bool HOST = false>
__global__ void SWE_STEP_BOUNDS step_kernel(const __grid_constant__ StepArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr bool kDepths = geoclaw(SOLVER) && !HOST;
    const int T = A.seg_cells;
    // staging buffers [stage_depth][h, hu, hv, b][T]: with depth 2 the next
    // segment's bulk copies land in one buffer while the CTA works on the other
    const bool depth2 = A.stage_depth > 1;
    double* stage = reinterpret_cast<double*>(smem_raw);
    SegMem M;
    M.T = T;
    M.lay_out(stage + (depth2 ? 8 : 4) * T, false, A.max_ndepth);
    const DepthTab tab(M.tab, A.max_ndepth);
    __shared__ uint64_t bar[2];
    __shared__ RedSlots red;
    __shared__ InstParams P;  // the running instance's
    __shared__ unsigned int s_error;
    __shared__ int s_last;
    __shared__ int s_seg;

    const int tid = threadIdx.x;
    // The first segment of CTA k is the k-th to be handed out; the counter deals the rest.
    int seg = A.seg_order ? __ldg(&A.seg_order[blockIdx.x]) : (int)blockIdx.x;
    const long long step = A.gs->step;
    const long long kseq = step - A.gs->dt_seq_base;
    const int odd = (int)(step & 1);
    const int ib = A.fixed_io ? 0 : odd;
    const double* hin = A.h[ib];
    const double* huin = A.hu[ib];
    const double* hvin = A.hv[ib];

    if (tid == 0) {
        s_error = 0;
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();

    Reduced r{0ull, 0};
    uint32_t phase = 0;    // bit k: parity of barrier k
    uint32_t pending = 0;  // bit k: bulk copies in flight into buffer k
    int cur = -1;

    // Stage segment `sg` into buffer k: bulk copies of the 16-byte multiple (the
    // segment starts at an even cell) completing on barrier k, plain loads for an
    // odd tail cell or for host memory. All threads call it.
    auto issue = [&](int sg, int k) {
        const int4 si = __ldg(&A.seg_info[sg]);
        const int c0 = si.x, cn = si.y;
        double* bh = stage + (size_t)k * 4 * T;
        const int cbulk = A.use_tma ? (cn & ~1) : 0;
        if (cbulk > 0) {
            if (tid == 0) {
                fence_proxy_async();
                const uint32_t bytes = (uint32_t)cbulk * 8u;
                mbar_arrive_expect_tx(&bar[k], 4u * bytes + A.extra_tx);
                bulk_g2s(bh, hin + c0, bytes, &bar[k]);
                bulk_g2s(bh + T, huin + c0, bytes, &bar[k]);
                bulk_g2s(bh + 2 * T, hvin + c0, bytes, &bar[k]);
                bulk_g2s(bh + 3 * T, A.b + c0, bytes, &bar[k]);
            }
            pending |= 1u << k;
        }
        if (tid == 0) {
            // the segment's edge tasks, memo entries and depths, read later in
            // task or thread order, are on their way to L2 while its state lands
            const long long a = __ldg(&A.seg_ptr[sg]), e = __ldg(&A.seg_ptr[sg + 1]);
            prefetch_l2(A.tasks + a, (size_t)(e - a) * 16u);
            if (A.memo) prefetch_l2(A.memo + c0, (size_t)cn * 16u);
            prefetch_l2(A.depth + c0, (size_t)cn);
        }
        for (int i = cbulk + tid; i < cn; i += blockDim.x) {
            bh[i] = hin[c0 + i];
            bh[T + i] = huin[c0 + i];
            bh[2 * T + i] = hvin[c0 + i];
            bh[3 * T + i] = A.b[c0 + i];
        }
    };
    // Wait (one thread, bounded) for buffer k's bulk copies.
    auto wait = [&](int k) {
        if (pending & (1u << k)) {
            if (tid == 0) {
                unsigned int polls = 0;
                unsigned long long t0 = 0;
                while (!mbar_try_wait(&bar[k], (phase >> k) & 1u)) {
                    ++polls;
                    if ((polls & 63u) == 1u) {
                        const unsigned long long now = global_ns();
                        if (polls == 1u) t0 = now;
                        else if (now - t0 > A.wait_ns) polls = kPollLimit;
                    }
                    if (polls >= kPollLimit) {
                        s_error = 2u;
                        break;
                    }
                }
            }
            phase ^= 1u << k;
            pending &= ~(1u << k);
        }
    };

    // segments are handed out dynamically (CTAs that draw cheap segments, e.g.
    // dry land, take more), in the order seg_order gives: spread over the
    // domain, so that the CTAs an SM holds at one time mix wet and dry work
    auto drawn = [&](unsigned int ticket) {
        const long long k = (long long)gridDim.x + ticket;
        s_seg = k < A.n_seg ? (A.seg_order ? __ldg(&A.seg_order[k]) : (int)k) : A.n_seg;
    };
    int kbuf = 0;
    issue(seg, 0);
    while (seg < A.n_seg) {
        int seg_next = A.n_seg;
        if (depth2) {  // draw and stage the next segment before working on this one
            __syncthreads();
            if (tid == 0) drawn(atomicAdd(&A.gs->next_seg, 1u));
            __syncthreads();
            seg_next = s_seg;
            if (seg_next < A.n_seg) issue(seg_next, kbuf ^ 1);
        }
        const int4 si = __ldg(&A.seg_info[seg]);
        const int c0 = si.x, cn = si.y, inst = si.z;
        if (inst != cur) {  // uniform across the CTA
            if (cur >= 0) {
                flush_instance(A, cur, P.dt_by_max != 0, r, red);
                __syncthreads();  // P and the slots are read
            }
            // the parameters, the rows of the depths and dt come in one round of loads
            if (tid < (int)(sizeof(InstParams) / 4))
                reinterpret_cast<int*>(&P)[tid] = __ldg(reinterpret_cast<const int*>(A.ip + inst) + tid);
            const int nd = __ldg(&A.ip[inst].ndepth);
            const InstParams* Pg = A.ip + inst;
            for (int i = tid; i < nd; i += blockDim.x) {
                tab.load(A, inst, i);
                double dt = A.is[inst].dt;
                const double tm = Pg->max_time, to = Pg->tout;
                if (A.dt_seq && kseq >= 0 && kseq < A.dt_seq_len) dt = A.dt_seq[kseq * A.n_inst + inst];
                else dt = clamp_dt(dt, tm, to);
                tab.ndv[i] = div_one(-dt, tab.vol[i]);
            }
            cur = inst;
        }
        // ---- 1. the segment's state, staged in buffer kbuf
        wait(kbuf);
        __syncthreads();
        if (s_error) break;
        M.h = stage + (size_t)kbuf * 4 * T;
        M.d = M.h;
        const double drytol = P.drytol;
        for (int i = tid; i < cn; i += blockDim.x) {
            // depth_terms, with the square root and reciprocal skipped by warps of dry cells.
            // The f-wave path divides only the cell's own (rotated) momenta by its depth:
            // with both momenta +-0 every such quotient is a zero with the numerator's
            // sign, so those cells skip the reciprocal
            // sqrt(g d) comes from the memo when the cell's depth has the same bits as
            // the depth it was last taken for (water at rest keeps its depth from step
            // to step); the memo holds only pairs (d, sqrt(g d)), written by the CTA
            // that owns the cell, so a hit is the value the square root would give
            M.dep[i] = A.depth[c0 + i];
            const double d = M.h[i] - M.b()[i];
            const bool wet = lt(drytol, d);
            const bool need_y = wet && (SOLVER != FWAVE || ((dbits(M.hu()[i]) | dbits(M.hv()[i])) << 1) != 0);
            double sq = 0.0;
            u64 y = 0;
            bool miss = wet;
            if (wet && A.memo) {
                const double2 m = A.memo[c0 + i];
                if (dbits(m.x) == dbits(d)) {
                    sq = m.y;
                    miss = false;
                }
            }
            SWE_IF(miss) {
                sq = sqrt_fix(kG * d);
                if (A.memo) A.memo[c0 + i] = make_double2(d, sq);
            }
            if (need_y) y = recip_fix(d);
            M.rh[i] = y;
            M.sq[i] = sq;
            if (kDepths) M.h[i] = d;
        }
        if (kDepths) fence_proxy_async();  // before a later bulk copy into this buffer (barriers follow)
        // halo tasks: the cross-edge pass computed these edges' updates; copy
        // this segment's side into its slot
        const long long t0 = __ldg(&A.seg_ptr[seg]);
        const int nt = (int)(__ldg(&A.seg_ptr[seg + 1]) - t0);
        const int nm = A.halo_solve ? nt : nt - min(max(si.w, 0), nt);
        const int4* tasks = A.tasks + t0;
        for (int t = nm + tid; t < nt; t += blockDim.x) {
            const int4 tk = __ldg(&tasks[t]);
            const uint32_t meta = (uint32_t)tk.z;
            const int sa = tk.x - c0;
            const bool ain = (unsigned)sa < (unsigned)cn;
            const int cl = ain ? sa : tk.y - c0;
            const int le = ain ? (int)(meta & 3u) : (int)((meta >> 2) & 3u);
            if ((unsigned)cl >= (unsigned)cn || le > 2 || !(meta & (1u << 17)) ||
                (unsigned long long)(unsigned)tk.w >= (unsigned long long)A.n_xtasks) {
                atomicOr(&s_error, 1u);
                continue;
            }
            const double2* u = reinterpret_cast<const double2*>(A.xflux + 8 * (long long)(unsigned)tk.w + (ain ? 0 : 4));
            const double2 u0 = u[0], u1 = u[1];
            M.upd[(0 * 3 + le) * T + cl] = u0.x;
            M.upd[(1 * 3 + le) * T + cl] = u0.y;
            M.upd[(2 * 3 + le) * T + cl] = u1.x;
            M.upd[(3 * 3 + le) * T + cl] = u1.y;
        }
        __syncthreads();

        // ---- 2. edge tasks; each thread loads its next task while it works on the current one
        {
            int4 next = make_int4(0, 0, 0, 0);
            if (tid < nm) next = __ldg(&tasks[tid]);
            for (int t = tid; t < nm; t += blockDim.x) {
                const int4 tk = next;
                if (t + (int)blockDim.x < nm) next = __ldg(&tasks[t + blockDim.x]);
                if (edge_task<SOLVER, FZ, false, kDepths>(A, M, tk, FZ ? A.erec + t0 + t : nullptr, c0, cn, odd, drytol, P.bc,
                                                 ib))
                    atomicOr(&s_error, 1u);
            }
        }
        __syncthreads();

        // ---- 3. cell updates
        // With one staging buffer, thread 0 takes the next segment's ticket now and
        // reads it after its cells, so the atomic's round trip overlaps the updates.
        unsigned int ticket = 0u;
        if (!depth2 && tid == 0) ticket = atomicAdd(&A.gs->next_seg, 1u);
        const unsigned long long wkey = P.dt_by_max ? warp_key_bound(r.key) : 0ull;
        double* hout = A.h[ib ^ 1];
        double* huout = A.hu[ib ^ 1];
        double* hvout = A.hv[ib ^ 1];
        for (int i = tid; i < cn; i += blockDim.x) {
            const int c = c0 + i;
            const double h = kDepths ? hin[c] : M.h[i], depth = kDepths ? M.d[i] : 0.0;
            const CellOut o = update_cell<FZ>(M, tab, P, i, h, depth, odd, wkey, FZ == 2 ? A.branch[c] : (uint8_t)0, r);
            if (FZ != 2 && A.branch) A.branch[c] = o.branch;
            hout[c] = o.h;
            huout[c] = o.p1;
            hvout[c] = o.p2;
            A.flags[c] = o.flag;
        }
        if (!depth2 && tid == 0) drawn(ticket);
        __syncthreads();
        if (!depth2) {  // stage the next segment now
            seg_next = s_seg;
            if (seg_next < A.n_seg) issue(seg_next, 0);
        } else {
            kbuf ^= 1;
        }
        seg = seg_next;
    }
    if (pending) {  // left early on an error: let the copies in flight land first (bounded)
        wait(0);
        wait(1);
    }

    // ---- 4. reductions and the last-CTA finalisation (post_traversal_grid_op, :111-131)
    flush_instance(A, cur, P.dt_by_max != 0, r, red);
    if (tid == 0) {
        if (s_error) atomicOr(&A.gs->error, s_error);
        __threadfence();
        s_last = atomicAdd(&A.gs->done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        for (int i = tid; i < A.n_inst; i += blockDim.x) {
            // past the L1 cache: the other CTAs' atomics wrote the accumulators
            InstScalars* S = &A.is[i];
            const InstParams* Q = A.ip + i;
            const double time = S->time, dt0 = S->dt;
            const double dt_acc = __longlong_as_double((long long)__ldcg(&S->dt_acc));
            const unsigned long long x = __ldcg(&S->ds_acc), n = __ldcg(&S->refine_acc);
            const double dt = A.dt_seq && kseq >= 0 && kseq < A.dt_seq_len ? A.dt_seq[kseq * A.n_inst + i]
                                                                           : clamp_dt(dt0, Q->max_time, Q->tout);
            advance_time(S, *Q, time + dt, dt_acc, x, n);
            S->dt_acc = (unsigned long long)__double_as_longlong(DBL_MAX);
            S->ds_acc = 0;
            S->refine_acc = 0;
        }
        if (tid == 0) {
            A.gs->done = 0;
            A.gs->next_seg = 0;
            A.gs->step = step + 1;
        }
    }
}

// Wait (one thread, bounded like the staging wait) until *count reaches target;
// other CTAs' writes before their arrivals are visible afterwards.
__device__ __forceinline__ bool wait_count(const unsigned int* count, unsigned int target, unsigned long long wait_ns) {
    unsigned int polls = 0, v;
    unsigned long long t0 = 0;
    while (true) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        if ((int)(v - target) >= 0) return true;
        ++polls;
        if ((polls & 63u) == 1u) {
            const unsigned long long now = global_ns();
            if (polls == 1u) t0 = now;
            else if (now - t0 > wait_ns) return false;
        }
        if (polls >= kPollLimit) return false;
    }
}

// Many steps of a mesh whose segments all fit the GPU at once, one CTA each, in
// one cooperative launch: a segment's state stays in its CTA's shared memory from
// step to step. On such a mesh a step launched by itself is mostly fixed cost (at
// 2^12 cells 20 us, of which the launch, the staging and the end of the step take
// about half) and the serial chain of one edge and one cell.
// The CTAs of an instance meet once per step, and the meeting is split: a CTA
// writes its new state to global memory, folds its largest CFL key into the
// instance's and counts itself as arrived; then it solves the edges inside its
// segment, which need neither neighbours nor the new dt; the warps with halo
// tasks (solved here by both segments' CTAs) and the warp that prepares dt wait
// for the count. No CTA passes a count before every CTA of its instance has
// finished reading the buffer that the next cell updates overwrite, and the ring
// slot of the key cleared after step k was last read in step k (its next use is
// in step k + 2, past another meeting).
// For instances with dt_by_max and a dt from the CFL condition.
template <int SOLVER>
__global__ void __launch_bounds__(256) multi_step_kernel(const __grid_constant__ StepArgs A, const int n_steps) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int T = A.seg_cells, tid = threadIdx.x, bd = blockDim.x;
    SegMem M;
    M.T = T;
    M.h = reinterpret_cast<double*>(smem_raw);
    M.lay_out(M.h + 4 * T, true, A.max_ndepth);
    const DepthTab tab(M.tab, A.max_ndepth);
    __shared__ RedSlots red;
    __shared__ InstParams P;
    __shared__ unsigned int s_error;

    const int seg = (int)blockIdx.x;
    const int4 si = __ldg(&A.seg_info[seg]);
    const int c0 = si.x, cn = si.y, inst = si.z;
    const long long t0 = __ldg(&A.seg_ptr[seg]);
    const int nt = (int)(__ldg(&A.seg_ptr[seg + 1]) - t0);
    const int halo = min(max(si.w, 0), nt), nm = nt - halo;
    const int4* tasks = A.tasks + t0;
    const long long step0 = A.gs->step;
    InstScalars* S = &A.is[inst];
    const int nd = __ldg(&A.ip[inst].ndepth);
    if (tid < (int)(sizeof(InstParams) / 4))
        reinterpret_cast<int*>(&P)[tid] = __ldg(reinterpret_cast<const int*>(A.ip + inst) + tid);
    for (int i = tid; i < nd; i += bd) tab.load(A, inst, i);
    if (tid == 0) s_error = 0;
    {
        const int ib = (int)(step0 & 1);
        const double *hin = A.h[ib] + c0, *huin = A.hu[ib] + c0, *hvin = A.hv[ib] + c0;
        for (int i = tid; i < cn; i += bd) {
            M.h[i] = hin[i];
            M.hu()[i] = huin[i];
            M.hv()[i] = hvin[i];
            M.b()[i] = A.b[c0 + i];
            M.dep[i] = A.depth[c0 + i];
        }
    }
    // sqrt(g d) and the reciprocal of a cell, as in the step kernel's staging loop; a
    // cell whose depth kept its bits keeps them (a reciprocal left out while the
    // cell was at rest is taken when it moves)
    auto terms = [&](int i, double drytol, bool same_depth) {
        const double d = M.h[i] - M.b()[i];
        const bool wet = lt(drytol, d);
        const bool need_y = wet && (SOLVER != FWAVE || ((dbits(M.hu()[i]) | dbits(M.hv()[i])) << 1) != 0);
        if (!same_depth) {
            double sq = 0.0;
            SWE_IF(wet) sq = sqrt_fix(kG * d);
            M.sq[i] = sq;
        }
        if (!same_depth || (need_y && M.rh[i] == 0)) M.rh[i] = need_y ? recip_fix(d) : 0;
        M.d[i] = d;
    };
    __syncthreads();
    const double drytol = P.drytol;
    for (int i = tid; i < cn; i += bd) terms(i, drytol, false);
    // the last warp prepares dt; in the instance's first CTA its first lane keeps the time
    const bool dt_warp = tid >= bd - 32, keeper = tid == bd - 32 && seg == P.first_seg;
    double time = S->time, dt = S->dt;
    const unsigned int n_cta = (unsigned int)P.n_segs;
    __syncthreads();

    int k = 0;
    for (; k < n_steps; ++k) {
        const int odd = (int)((step0 + k) & 1);
        // ---- edges: tid, tid + bd, ... of those inside the segment, then the halo tasks
        // from the last warp down; dt before a warp's edges if it has none inside
        unsigned int bad = 0;
        bool met = k == 0;
        auto meet = [&]() {
            if (!met && !wait_count(&S->arrived, (unsigned int)k * n_cta, A.wait_ns)) bad = 4u;
            met = true;
        };
        auto prepare_dt = [&]() {
            meet();
            if (k > 0) {
                dt = P.courant * dt_new_of(P, DBL_MAX, __ldcg(&S->ds_ring[(k - 1) % 3]));
                if (keeper) S->ds_ring[(k + 1) % 3] = 0;
            }
            const double c = clamp_dt(dt, P.max_time, P.tout);
            time = time + c;
            for (int i = tid - (bd - 32); i < nd; i += 32) tab.ndv[i] = div_one(-c, tab.vol[i]);
        };
        if (dt_warp && bd - 32 >= nm) prepare_dt();
        auto after = [&](int t) {  // the thread's task after t (a task inside the segment)
            return t + bd < nm ? t + bd : nm + bd - 1 - tid;
        };
        int t = tid < nm ? tid : nm + bd - 1 - tid;
        int4 next = t < nt ? __ldg(&tasks[t]) : make_int4(0, 0, 0, 0);
        while (t < nt) {
            if (t >= nm) meet();
            if (bad) break;
            const int4 tk = next;
            t = t < nm ? after(t) : t + bd;
            if (t < nt) next = __ldg(&tasks[t]);
            bad = edge_task<SOLVER, 0, true, geoclaw(SOLVER)>(A, M, tk, nullptr, c0, cn, odd, drytol, P.bc, odd);
        }
        if (dt_warp && bd - 32 < nm) prepare_dt();
        if (bad) atomicOr(&s_error, bad);
        __syncthreads();
        if (s_error) break;

        // ---- cells
        Reduced r{0ull, 0};
        const bool last = k == n_steps - 1;
        double *hout = A.h[odd ^ 1], *huout = A.hu[odd ^ 1], *hvout = A.hv[odd ^ 1];
        for (int i = tid; i < cn; i += bd) {
            const CellOut o = update_cell<0>(M, tab, P, i, M.h[i], M.d[i], odd, 0ull, 0, r);
            const bool same = dbits(o.h) == dbits(M.h[i]);
            M.h[i] = o.h;
            M.hu()[i] = o.p1;
            M.hv()[i] = o.p2;
            const int c = c0 + i;
            hout[c] = o.h;
            huout[c] = o.p1;
            hvout[c] = o.p2;
            if (last) A.flags[c] = o.flag;
            else terms(i, drytol, same);
        }
        warp_reduce(r, red);
        __syncthreads();
        if (tid == bd - 32) {  // the last warp has the fewest edges inside the segment
            const Reduced b = block_reduced(red);
            if (b.key) atomicMax(&S->ds_ring[k % 3], b.key);
            if (last && b.nref) atomicAdd(&S->refine_acc, (unsigned long long)b.nref);
            __threadfence();
            atomicAdd(&S->arrived, 1u);
        }
    }
    // ---- the instance's scalars, and the counters for the next launch
    if (keeper && k == n_steps) {
        if (wait_count(&S->arrived, (unsigned int)n_steps * n_cta, A.wait_ns)) {
            advance_time(S, P, time, DBL_MAX, __ldcg(&S->ds_ring[(n_steps - 1) % 3]), __ldcg(&S->refine_acc));
        } else {
            atomicOr(&s_error, 4u);
        }
    }
    __syncthreads();
    if (tid == 0) {
        if (s_error) atomicOr(&A.gs->error, s_error);
        __threadfence();
        if (atomicAdd(&A.gs->done, 1u) == gridDim.x - 1) {
            __threadfence();
            for (int i = 0; i < A.n_inst; ++i) {
                A.is[i].arrived = 0;
                A.is[i].refine_acc = 0;  // also where a wait ran out and no one took it
                for (int q = 0; q < 3; ++q) A.is[i].ds_ring[q] = 0;
            }
            A.gs->done = 0;
            A.gs->step = step0 + n_steps;
        }
    }
}

}  // namespace SWE_KNS
