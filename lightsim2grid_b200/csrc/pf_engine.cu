// Batched AC Newton-Raphson on the GPU: one persistent kernel, one CTA per instance.
//
// Each CTA takes jobs (an instance, or a chain of time-series steps) from a global
// counter and runs the whole Newton loop of the reference's compute_pf for them:
//   mismatch   F = V .* conj(Ybus V) - Sbus (+ slack term)     BaseAlgo.cpp:30-118
//   J fill     dS/dVm, dS/dVa scattered into the LU array      BaseNRAlgo.tpp:202-260,
//                                                              BaseNRSingleSlackAlgo.tpp:449-490
//   refactor   LU with the plan's fixed pivots                 (KLUSolver.cpp:47-59 contract)
//   solve      forward / backward substitution                 (KLUSolver.cpp:61-69 contract)
//   update     Va, Vm, V and the convergence test              BaseNRSingleSlackAlgo.tpp:129-162,
//                                                              BaseNRAlgo.tpp:136-167
// The refactorisation (right-looking, by elimination level, with the forward substitution
// of the right-hand side fused in) and the substitutions run as phase programs: flat lists
// of independent operations, coloured on the host into conflict-free phases, one barrier
// per phase, no atomics -- the result is deterministic.  LU values live in shared memory
// when they fit, else in the CTA's global slab (L2 resident).  The mixed form (FP32 LU)
// refines the Newton steps taken close to the solution once against the FP64 Jacobian,
// computed on the fly from dS/dV (the correction solve is skipped when the FP64 residual is
// already below a hundredth of the tolerance).
#include "pf_engine.cuh"
#include "pf_device_math.cuh"

#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

namespace l2g {

namespace {



struct Shared {
    double red[32];  // block reductions; the dense tail's backward substitution (one panel's values)
    int ired[32];
    unsigned long long pc[kPhaseSlots];  // per-phase SM cycles (thread 0, when profiled)
    // the overrides: rows and columns, or (DC kernel) CSR positions, and values
    union {
        int orow[kMaxOverrides];
        int opos[kMaxOverrides];
    };
    int ocol[kMaxOverrides];
    double2 oval[kMaxOverrides];
    int novr;
    int job;
    int piv_err;
    int job_failed;
    double slack_absorbed;
};

static_assert(sizeof(Shared) + sizeof(Segment) + sizeof(QueueJob) + 16 <= kNrStaticSmem,
              "the Newton kernels' static shared memory, alignment included");
static_assert(sizeof(Shared) + 3 * sizeof(DevPlan) + 16 <= kFdpfStaticSmem, "the fast decoupled kernel's");

// load with acquire semantics at GPU scope: the job ring entries and segments written before the
// tail (by the host's copies, in stream order) are seen after it
__device__ __forceinline__ int ld_acquire_gpu(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Request loop: claims the next published job of the ring (compare-and-swap on the head, so a
// CTA never holds a job that is not there yet) into *job and returns its index, or -1 when the
// launch is closing and the ring is empty.  After idle_polls polls of an empty ring the CTA closes
// the launch (every CTA then leaves at its next empty poll), so the wait is bounded.  A function of
// its own: its registers do not add to the solver's.
__device__ __noinline__ int claim_queue_job(const QueueJob *jobs, int cap, int *head, const int *tail, int *closing,
                                            int idle_polls, QueueJob *job) {
    for (int polls = 0;;) {
        const int t = ld_acquire_gpu(tail);
        const int h = *reinterpret_cast<volatile int *>(head);
        if (h < t) {
            if (atomicCAS(head, h, h + 1) == h) {
                const QueueJob *e = jobs + (h % cap);
                *job = QueueJob{__ldcg(&e->slot), __ldcg(&e->first), __ldcg(&e->count), __ldcg(&e->req)};
                return h;
            }
            continue;  // another CTA took it: look again
        }
        if (*reinterpret_cast<volatile int *>(closing)) return -1;
        if (++polls > idle_polls) {
            atomicExch(closing, 1);
            return -1;
        }
        __nanosleep(500);
    }
}

// Request loop: the job's rows, iterations and errors (mapped host memory) are made visible before
// its instances are added to the slot's completion count.
__device__ __noinline__ void signal_queue_job(int *done, int slot, int count) {
    __threadfence_system();
    atomicAdd_system(done + slot, count);
}

// block-wide max of |F| and "any non-finite" flag; every thread receives the result
__device__ __forceinline__ void block_norm(Shared &S, double lmax, int lbad, double &norm, int &bad) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
        lbad |= __shfl_xor_sync(0xffffffffu, lbad, o);
    }
    __syncthreads();
    if (lane == 0) {
        S.red[warp] = lmax;
        S.ired[warp] = lbad;
    }
    __syncthreads();
    double r = 0.0;
    int b = 0;
    for (int w = 0; w < nw; ++w) {
        r = fmax(r, S.red[w]);
        b |= S.ired[w];
    }
    norm = r;
    bad = b;
}

__device__ __forceinline__ double block_min(Shared &S, double v) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) S.red[warp] = v;
    __syncthreads();
    double r = S.red[0];
    for (int w = 1; w < nw; ++w) r = fmin(r, S.red[w]);
    return r;
}

__device__ __forceinline__ double block_sum(Shared &S, double v) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) S.red[warp] = v;
    __syncthreads();
    double r = 0.0;
    for (int w = 0; w < nw; ++w) r += S.red[w];
    return r;
}

__device__ __forceinline__ double2 ybus_value(const DevPlan &P, const Shared &S, int p) {
    double2 y = P.Rx[p];
    for (int i = 0; i < S.novr; ++i)
        if (S.opos[i] == p) y = S.oval[i];
    return y;
}


// Stages override i of an instance (caller: one thread per override).  A position outside the pattern
// (pf_ybus_positions gives -1 there) changes no entry.
__device__ __forceinline__ void stage_override(const PlanArrays &P, Shared &S, int i, int pos, double2 val) {
    const bool in = (unsigned)pos < (unsigned)P.nnzY;
    S.oval[i] = val;
    S.orow[i] = in ? P.Rrow[pos] : -1;
    S.ocol[i] = in ? P.Rj[pos] : -1;
}

// The overrides that lie in row r, as a bit mask: rows without one (nearly all) then test nothing
// per entry.
__device__ __forceinline__ unsigned row_overrides(const Shared &S, int r) {
    unsigned mask = 0;
    for (int i = 0; i < S.novr; ++i) mask |= (unsigned)(S.orow[i] == r) << i;
    return mask;
}

__device__ __forceinline__ double2 override_value(const Shared &S, unsigned mask, int c, double2 y) {
    for (; mask; mask &= mask - 1) {
        const int i = __ffs(mask) - 1;
        if (S.ocol[i] == c) y = S.oval[i];
    }
    return y;
}

// (Ybus V)[r] of the row in `slot` (bus r, voltage vr, slice sl): the diagonal, then the off-diagonal
// entries in column order.  KEEP: t = conj(Y V_c) V_r of every entry goes to T / Td, from which the
// Jacobian fill and the refinement residual take their values (a mark where V_c is zero, see dsbus).
// The entries of a slice are 32 consecutive values per step (rows sorted by length, so a
// slice has almost no padding), and the loads of four steps are issued together.
template <bool KEEP>
__device__ __forceinline__ double2 ybus_row(const PlanArrays &P, const Shared &S, const double2 *__restrict__ V, int slot,
                                            int r, double2 vr, int2 sl, double2 *__restrict__ T,
                                            double2 *__restrict__ Td) {
    const unsigned mask = row_overrides(S, r);
    double2 yd = P.dg_val[slot];
    if (mask) yd = override_value(S, mask, r, yd);
    double2 s = cmul(yd, vr);
    if (KEEP) Td[slot] = entry_power(s, vr, vr);
    const int e0 = sl.x + (slot & 31);
    for (int u0 = 0; u0 < sl.y; u0 += 4) {
        int c[4];
        double2 y[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = u0 + u < sl.y;
            c[u] = in ? P.off_col[e0 + (u0 + u) * 32] : -1;
            y[u] = in ? P.off_val[e0 + (u0 + u) * 32] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = c[u] >= 0 ? V[c[u]] : make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (c[u] < 0) continue;
            if (mask) y[u] = override_value(S, mask, c[u], y[u]);
            const double2 b = cmul(y[u], v[u]);
            s.x += b.x;
            s.y += b.y;
            if (KEEP) T[e0 + (u0 + u) * 32] = entry_power(b, v[u], vr);
        }
    }
    return s;
}

// F at V: writes the permuted right-hand side x and, for the Jacobian fill and the residual, per
// row slot Sd = V conj(Ybus V) and (FB) the FP64 mismatch, per entry T / Td (ybus_row);
// returns ||F||_inf and a non-finite flag to every thread.
// Bound by the latency of its loads: every pass reads a few hundred KB of L2 data per CTA, which
// 20 to 24 warps cover only when the loads are coalesced and independent.  Rows by slots (against a
// thread per CSR row with 16-byte loads 58 bytes apart) and T kept for the fill and the
// residual (against a second and third gather of both voltages per entry) are what that takes.
template <typename XT, bool FB>
__device__ void mismatch(const PlanArrays &P, Shared &S, const double2 *__restrict__ V, double2 *__restrict__ T,
                         double2 *__restrict__ Td, double2 *__restrict__ Sd, double2 *__restrict__ Fb,
                         const double2 *__restrict__ Sbus, XT *x, double &norm, int &bad) {
    double lmax = 0.0;
    int lbad = 0;
    const double sa = S.slack_absorbed;
    const int ns = P.row_slots, bd = blockDim.x;
    int slot = threadIdx.x;
    int r = slot < ns ? P.row_bus[slot] : -1;
    int2 sl = slot < ns ? P.row_slice[slot >> 5] : make_int2(0, 0);
    while (slot < ns) {
        // the next slot's row and slice arrive while this one is worked on
        const int nslot = slot + bd;
        const int nr = nslot < ns ? P.row_bus[nslot] : -1;
        const int2 nsl = nslot < ns ? P.row_slice[nslot >> 5] : make_int2(0, 0);
        if (r >= 0) {
            const double2 sb = __ldcg(Sbus + r);
            const int2 eq = P.dg_eq[slot];
            const double2 vr = V[r];
            const double2 s = ybus_row<true>(P, S, V, slot, r, vr, sl, T, Td);
            const double2 d = cmul(cconj(s), vr);  // V * conj(I)
            Sd[slot] = d;
            double mr = d.x - sb.x;
            const double mi = d.y - sb.y;
            if (P.distributed) mr += sa * P.w[r];
            if (FB) Fb[slot] = make_double2(mr, mi);
            if (eq.x >= 0) {
                x[eq.x] = (XT)mr;
                lmax = fmax(lmax, fabs(mr));
                lbad |= !isfinite(mr);
            }
            if (eq.y >= 0) {
                x[eq.y] = (XT)mi;
                lmax = fmax(lmax, fabs(mi));
                lbad |= !isfinite(mi);
            }
        }
        slot = nslot;
        r = nr;
        sl = nsl;
    }
    block_norm(S, lmax, lbad, norm, bad);
}

// The four Jacobian values of an entry to their LU positions (-1: none).
template <typename LT>
__device__ __forceinline__ void put_entry(LT *lu, int4 t, double2 te, double2 d) {
    double dvar, dvai;
    double2 dvm;
    dsbus(te, d, dvar, dvai, dvm);
    if (t.x >= 0) lu[t.x] = (LT)dvar;
    if (t.y >= 0) lu[t.y] = (LT)dvai;
    if (t.z >= 0) lu[t.z] = (LT)dvm.x;
    if (t.w >= 0) lu[t.w] = (LT)dvm.y;
}

// dS/dVa and |V| dS/d|V| scattered into the LU array, from the mismatch's T, Td and Sd: every load is coalesced and none depends on another.
// ZERO_ALL: the LU region (shared memory) is cleared whole with 16-byte stores before the
// entries are written, in place of the gather of the fill-in positions.
template <typename LT, bool ZERO_ALL>
__device__ void jacobian_fill(const PlanArrays &P, const double2 *__restrict__ T, const double2 *__restrict__ Td,
                              const double2 *__restrict__ Sd, LT *lu) {
    if constexpr (ZERO_ALL) {
        // lu is 4-byte aligned; the head up to the first 16-byte boundary and the tail are scalar
        const int head = (int)(((16 - ((size_t)lu & 15)) & 15) / sizeof(LT));
        const int h = head < P.nnzLU ? head : P.nnzLU;
        if ((int)threadIdx.x < h) lu[threadIdx.x] = (LT)0;
        const int nvec = (P.nnzLU - h) * (int)sizeof(LT) / 16;
        float4 *v4 = reinterpret_cast<float4 *>(lu + h);
        for (int i = threadIdx.x; i < nvec; i += blockDim.x) v4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int t0 = h + nvec * 16 / (int)sizeof(LT);
        if ((int)threadIdx.x < P.nnzLU - t0) lu[t0 + threadIdx.x] = (LT)0;
        __syncthreads();
    }
    constexpr int U = 4;  // entries per thread whose loads are issued together
    const int bd = blockDim.x;
    const double2 zero = make_double2(0.0, 0.0);
    for (int e0 = threadIdx.x; e0 < P.row_len; e0 += U * bd) {
        int4 t[U];
        double2 te[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = e0 + u * bd;
            const bool ok = e < P.row_len;
            t[u] = ok ? P.off_target[e] : make_int4(-1, -1, -1, -1);
            te[u] = ok ? T[e] : zero;  // padding: no target
        }
#pragma unroll
        for (int u = 0; u < U; ++u) put_entry<LT>(lu, t[u], te[u], zero);
    }
    for (int s = threadIdx.x; s < P.row_slots; s += bd) {
        if (P.dg_pos[s] < 0) continue;
        put_entry<LT>(lu, P.dg_target[s], Td[s], Sd[s]);
    }
    if constexpr (!ZERO_ALL)
        for (int i = threadIdx.x; i < P.nfill; i += blockDim.x) lu[P.fillpos[i]] = (LT)0;
    for (int i = threadIdx.x; i < P.nconst; i += blockDim.x) lu[P.cpos[i]] = (LT)P.cval[i];
}

template <typename LT, typename XT>
__device__ __forceinline__ void run_op(const int4 o, LT *lu, XT *v) {
    const unsigned kind = (unsigned)o.w >> 28;
    const int w = o.w & 0x0fffffff;
    if (kind == 0u) {
        lu[o.x] -= lu[o.y] * lu_div(lu[o.z], lu[w]);
    } else if (kind == 2u) {
        v[o.x] -= lu_div((XT)lu[o.y] * v[o.z], (XT)lu[w]);
    }
    // kind 7: empty slot
}

// Packed operation of the shared-memory layout: s[x] -= s[y] * s[z] / s[w] over the one
// index space of the solve vector and the LU (empty slots write a scratch element).
template <typename T>
__device__ __forceinline__ void run_op_packed(const uint2 o, T *s) {
    const T y = s[o.x >> 16], z = s[o.y & 0xffffu], w = s[o.y >> 16];
    T *px = s + (o.x & 0xffffu);
    *px -= y * lu_div(z, w);
}

struct Trace {
    unsigned long long *buf;
    int cap, n;
    __device__ __forceinline__ void mark() {
        if (buf != nullptr && threadIdx.x == 0 && n < cap) buf[n++] = clock64();
    }
};

// Runs a phase program: one barrier per phase.  In phase p, thread t < sw[p] runs the
// operations sb[p] + t, sb[p] + t + sw[p], ... (bounds and widths staged in shared memory).
//
// Latency hiding: a block barrier also waits for the thread's global loads still in flight,
// so operation loads are not carried across more than the next barrier.  A thread loads the
// first two operations of phase p + 1 when phase p starts (they arrive while phase p works),
// and inside a phase it keeps four operations in flight.  The two register pairs swap roles
// from phase to phase through a loop unrolled by two (a register still waiting for its load
// is never copied).
template <typename OP>
struct OpPair {
    OP a, b;
};

template <typename OP>
__device__ __forceinline__ void load_first2(const OP *__restrict__ ops, const int *sb, const int *sw, int nph,
                                            int p, OpPair<OP> &r, OP none) {
    r.a = none;
    r.b = none;
    if (p < nph) {
        const int w = sw[p];
        if ((int)threadIdx.x < w) {
            const int k = sb[p] + threadIdx.x, e = sb[p + 1];
            if (k < e) r.a = ops[k];
            if (k + w < e) r.b = ops[k + w];
        }
    }
}

template <typename OP, typename F>
__device__ __forceinline__ void run_phase(const OP *__restrict__ ops, const int *sb, const int *sw, int nph, int p,
                                          OpPair<OP> &cur, OpPair<OP> &nxt, OP none, F &&apply, Trace &tr) {
    load_first2<OP>(ops, sb, sw, nph, p + 1, nxt, none);
    const int w = sw[p];
    if ((int)threadIdx.x < w) {
        const int e = sb[p + 1];
        int k = sb[p] + threadIdx.x;
        OP c = none, d = none;
        if (k + 2 * w < e) c = ops[k + 2 * w];
        if (k + 3 * w < e) d = ops[k + 3 * w];
        for (;;) {
            if (k >= e) break;
            apply(cur.a);
            if (k + 4 * w < e) cur.a = ops[k + 4 * w];
            k += w;
            if (k >= e) break;
            apply(cur.b);
            if (k + 4 * w < e) cur.b = ops[k + 4 * w];
            k += w;
            if (k >= e) break;
            apply(c);
            if (k + 4 * w < e) c = ops[k + 4 * w];
            k += w;
            if (k >= e) break;
            apply(d);
            if (k + 4 * w < e) d = ops[k + 4 * w];
            k += w;
        }
    }
    __syncthreads();
    tr.mark();
}

// Phases [a, b) of a program on the first `nwarps` warps: operations from the shared-memory copy
// `sops` (the program's operations from phase a on), one barrier of those warps per phase (no
// global load in flight at it), the other warps go straight to the closing block barrier.
template <typename OP, typename F>
__device__ __forceinline__ void run_narrow(const OP *sops, const int *sb, const int *sw, int a, int b, int nwarps,
                                           F &&apply, Trace &tr) {
    const int nt = nwarps * 32;
    if ((int)threadIdx.x < nt) {
        const int o0 = sb[a];
        for (int p = a; p < b; ++p) {
            const int w = sw[p], e = sb[p + 1] - o0;
            if ((int)threadIdx.x < w)
                for (int k = sb[p] - o0 + threadIdx.x; k < e; k += w) apply(sops[k]);
            asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
            tr.mark();
        }
    }
    __syncthreads();
}

template <typename OP, typename F>
__device__ void run_program(const OP *__restrict__ ops, const int *sb, const int *sw, int nph, OP none, F &&apply,
                            Trace &tr) {
    if (nph <= 0) return;
    OpPair<OP> A, B;
    load_first2<OP>(ops, sb, sw, nph, 0, A, none);
    for (int p = 0; p < nph; p += 2) {
        run_phase<OP>(ops, sb, sw, nph, p, A, B, none, apply, tr);
        if (p + 1 >= nph) break;
        run_phase<OP>(ops, sb, sw, nph, p + 1, B, A, none, apply, tr);
    }
}

// The same with phases [na, nb) on the first `nwarps` warps (run_narrow): block-wide phases
// [0, na), the narrow ones, block-wide [nb, nph).
template <typename OP, typename F>
__device__ void run_program_narrow(const OP *__restrict__ ops, const int *sb, const int *sw, int nph, OP none,
                                   F &&apply, Trace &tr, int na, int nb, const OP *sops, int nwarps) {
    if (nph <= 0) return;
    if (nb <= na) na = nb = nph;
    for (int part = 0; part < 2; ++part) {
        const int from = part == 0 ? 0 : nb, to = part == 0 ? na : nph;
        if (from < to) {
            OpPair<OP> A, B;
            load_first2<OP>(ops, sb, sw, to, from, A, none);
            for (int p = from; p < to; p += 2) {
                run_phase<OP>(ops, sb, sw, to, p, A, B, none, apply, tr);
                if (p + 1 >= to) break;
                run_phase<OP>(ops, sb, sw, to, p + 1, B, A, none, apply, tr);
            }
        }
        if (part == 0 && na < nb) run_narrow<OP>(sops, sb, sw, na, nb, nwarps, apply, tr);
    }
}

// An operation of a program over an LU in global memory, decoded: the written value x and an `id` that
// is distinct for every written value, the operands' LU positions y and w, and z.  A push writes and
// reads (x, z) the solve vector, an update the LU.
struct GlobalOp {
    unsigned x, y, z, w, id;
    bool none, push;
};
__device__ __forceinline__ GlobalOp decode(const int4 o, int, int) {
    const unsigned kind = (unsigned)o.w >> 28;
    return GlobalOp{(unsigned)o.x, (unsigned)o.y, (unsigned)o.z, (unsigned)o.w & 0x0fffffffu,
                    (unsigned)o.x | (kind << 28), kind == 7u, kind == 2u};
}
// packed: solve vector below `off`, LU from there on; m: the scratch element of an empty slot
__device__ __forceinline__ GlobalOp decode(const uint2 o, int m, int off) {
    const unsigned X = o.x & 0xffffu, Z = o.y & 0xffffu;
    const bool push = X < (unsigned)off;
    const unsigned d = push ? 0u : (unsigned)off;
    return GlobalOp{X - d, (o.x >> 16) - off, Z - d, (o.y >> 16) - off, X, X == (unsigned)m, push};
}
__device__ __forceinline__ uint2 none_op(uint2, int m) {
    return make_uint2((unsigned)m | ((unsigned)m << 16), (unsigned)m | ((unsigned)m << 16));
}
__device__ __forceinline__ int4 none_op(int4, int) { return make_int4(0, 0, 0, 7 << 28); }

// Runs a phase program over an LU in global memory, the solve vector in shared memory: in phase p,
// thread t < sw[p] runs the operations sb[p] + t, sb[p] + t + sw[p], ... in order, one barrier per phase.
// Bound by the latency of its scattered loads from L2: one operation after the other, each waited for the
// store of the one before.  So a thread takes U operations together (no operation reads a value that
// another one of its phase writes, and those that write one value follow one another on their thread:
// their sum stays in a register), the next U arriving meanwhile, in the packed form where 16-bit
// indices hold the LU (half the bytes: 2.4 MB of operations were read per factorisation).  2848 buses
// FP64, N-1, 3,050 outages: 14.7 -> 13.2 ms with run_pushes_global (U = 2, 4: 14.2, 13.8 ms; U = 6 and 8 spill:
// 16.7, 23.2 ms before run_pushes_global; operation loads past L1: +0.4 ms).  16-byte operations run U = 2
// (300-chord grid FP64 93.5 -> 91.0 ms).  FP32 keeps one operation at a time (run_program: 51.9 ms on the 300-chord
// grid against 55.4).
// A function of its own: inlined it spilled in the Newton loop.
template <int U, typename OP, typename T>
__device__ __noinline__ void run_program_global(const OP *__restrict__ ops, const int *sb, const int *sw, int nph,
                                                int m, int off, T *lu, T *x, Trace &tr) {
    if (nph <= 0) return;
    const int t = threadIdx.x;
    const auto load = [&](OP (&o)[U], int k, int w, int e) {
#pragma unroll
        for (int u = 0; u < U; ++u) o[u] = k + u * w < e ? __ldg(ops + k + u * w) : none_op(OP{}, m);
    };
    OP o[U], n[U];
    int w = sw[0], e = sb[1], k = t < w ? sb[0] + t : e;
    load(o, k, w, e);
    for (int p = 0;;) {
        T y[U], d[U], z[U], v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const GlobalOp g = decode(o[u], m, off);
            y[u] = d[u] = z[u] = v[u] = (T)1;
            if (!g.none) {
                const T *s = g.push ? x : lu;
                y[u] = lu[g.y];
                d[u] = lu[g.w];
                z[u] = s[g.z];
                if (u == 0 || g.id != decode(o[u > 0 ? u - 1 : 0], m, off).id) v[u] = s[g.x];
            }
        }
        // the next operations: of this phase, else the first of the next one
        k += U * w;
        const bool last = k >= e;
        if (last) {
            k = e = 0;
            if (p + 1 < nph) {
                w = sw[p + 1];
                e = sb[p + 2];
                k = t < w ? sb[p + 1] + t : e;
            }
        }
        load(n, k, w, e);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const GlobalOp g = decode(o[u], m, off);
            if (g.none) continue;
            if (u > 0 && g.id == decode(o[u > 0 ? u - 1 : 0], m, off).id) v[u] = v[u > 0 ? u - 1 : 0];
            const T q = lu_div(g.push ? y[u] * z[u] : z[u], d[u]);
            v[u] -= g.push ? q : y[u] * q;
            if (u == U - 1 || g.id != decode(o[u < U - 1 ? u + 1 : u], m, off).id) (g.push ? x : lu)[g.x] = v[u];
        }
        if (last) {
            __syncthreads();
            tr.mark();
            if (++p >= nph) break;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) o[u] = n[u];
    }
}

// A substitution program (pushes only) over an LU in global memory.  A phase waited for its operands from L2
// after its barrier; but the LU is final here, so a thread's LU values for its next U operations are loaded
// while the current ones run, and their operations one batch earlier still.  N-1: 2848 buses FP64 backward
// 111k -> 98k SM cycles a Newton step (with packed operations), 300-chord grid mixed 51.9 -> 50.1 ms (U = 1:
// 50.9 ms).
template <int U, typename OP, typename T>
__device__ __noinline__ void run_pushes_global(const OP *__restrict__ ops, const int *sb, const int *sw, int nph,
                                               int m, int off, const T *lu, T *x, Trace &tr) {
    if (nph <= 0) return;
    const int t = threadIdx.x;
    int p = 0, w = sw[0], e = sb[1], k = t < w ? sb[0] + t : e;  // the batch loaded next
    // loads a batch and moves on; whether it is its phase's last one
    const auto load = [&](OP (&o)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) o[u] = k + u * w < e ? __ldg(ops + k + u * w) : none_op(OP{}, m);
        k += U * w;
        const bool last = k >= e;
        if (last) {
            k = e = 0;
            if (++p < nph) {
                w = sw[p];
                e = sb[p + 1];
                k = t < w ? sb[p] + t : e;
            }
        }
        return last;
    };
    const auto values = [&](const OP (&o)[U], T (&y)[U], T (&d)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const GlobalOp g = decode(o[u], m, off);
            y[u] = g.none ? (T)0 : lu[g.y];
            d[u] = g.none ? (T)1 : lu[g.w];
        }
    };
    OP o[U], n[U], nn[U];
    T y[U], d[U], yn[U], dn[U];
    bool last = load(o), lastn = load(n);
    values(o, y, d);
    for (int left = nph;;) {
        values(n, yn, dn);
        const bool lastnn = load(nn);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const GlobalOp g = decode(o[u], m, off);
            if (!g.none) x[g.x] -= lu_div(y[u] * x[g.z], d[u]);
        }
        if (last) {
            __syncthreads();
            tr.mark();
            if (--left == 0) break;
        }
        last = lastn;
        lastn = lastnn;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            o[u] = n[u];
            n[u] = nn[u];
            y[u] = yn[u];
            d[u] = dn[u];
        }
    }
}

// The packed operations where a kernel variant can run them: an LU in global memory takes those whose
// placement keeps a value's operations together (null: the int4 ones).
template <bool LU_SMEM>
__device__ __forceinline__ const uint2 *packed_ops(const PlanArrays &P, const uint2 *cops) {
    return LU_SMEM || P.cops_runs ? cops : nullptr;
}

// One program over the LU layout of the kernel variant: packed operations over the shared
// index space, or packed or int4 operations over the global LU and the shared solve vector.
// PUSH: a substitution program.
// NARROW: `nar` is the narrow range of this program (phases [nar.x, nar.y) on nar.z warps,
// operations staged at `sops`), packed layout only.
template <typename LT, typename XT, bool LU_SMEM, bool PUSH, bool NARROW = false>
__device__ __forceinline__ void run_lu_program(const uint2 *cops, const int4 *ops, const int *sb, const int *sw,
                                               int nph, int m, int off, LT *lu, XT *x, Trace &tr,
                                               int3 nar = make_int3(0, 0, 0), const uint2 *sops = nullptr) {
    if constexpr (LU_SMEM) {
        static_assert(sizeof(LT) == sizeof(XT), "the packed layout needs one element type");
        const uint2 none = make_uint2((unsigned)m | ((unsigned)m << 16), (unsigned)m | ((unsigned)m << 16));
        if constexpr (NARROW)
            run_program_narrow<uint2>(cops, sb, sw, nph, none, [x](const uint2 o) { run_op_packed<XT>(o, x); }, tr,
                                      nar.x, nar.y, sops, nar.z);
        else
            run_program<uint2>(cops, sb, sw, nph, none, [x](const uint2 o) { run_op_packed<XT>(o, x); }, tr);
    } else {
        static_assert(sizeof(LT) == sizeof(XT), "one element type");
        if constexpr (PUSH) {
            if (cops != nullptr) run_pushes_global<2, uint2, XT>(cops, sb, sw, nph, m, off, lu, x, tr);
            else run_pushes_global<2, int4, XT>(ops, sb, sw, nph, m, 0, lu, x, tr);
        } else if constexpr (sizeof(LT) == 8) {
            if (cops != nullptr) run_program_global<3, uint2, XT>(cops, sb, sw, nph, m, off, lu, x, tr);
            else run_program_global<2, int4, XT>(ops, sb, sw, nph, m, 0, lu, x, tr);
        } else {
            run_program<int4>(ops, sb, sw, nph, none_op(int4{}, 0), [lu, x](const int4 o) { run_op<LT, XT>(o, lu, x); },
                              tr);
        }
    }
}

// z(k) / U(k, k): the backward program keeps z undivided.  CHECK: a zero pivot also sets
// S.piv_err (seen by every thread after the closing barrier).
template <typename LT, typename XT, bool CHECK = false>
__device__ __forceinline__ void scale_by_pivots(const PlanArrays &P, Shared &S, const LT *lu, XT *x) {
    int zero = 0;
    for (int k = threadIdx.x; k < P.m; k += blockDim.x) {
        const LT d = lu[P.dpos[k]];
        if (CHECK) zero |= d == (LT)0;
        x[k] = lu_div(x[k], (XT)d);
    }
    if (CHECK && zero) S.piv_err = 1;
    __syncthreads();
}

template <typename LT>
__device__ void check_pivots(const PlanArrays &P, Shared &S, const LT *lu) {
    int zero = 0;
    for (int k = threadIdx.x; k < P.m; k += blockDim.x) zero |= lu[P.dpos[k]] == (LT)0;
    if (zero) S.piv_err = 1;
    __syncthreads();
}

// FP64 residual of the Newton system, F - J dx, into rt (as a right-hand side), for the step x
// (dVa and u = dVm / |V|, FP32 values taken exactly).  Row r of J dx is the sum over its entries of
// dS/dVa dVa + |V| dS/d|V| u = t (u - j dVa), plus d (u_r + j dVa_r) of the diagonal (d = V conj(I);
// the dS/dVa, dS/dVm of BaseNRAlgo::_dSbus_dV, BaseNRAlgo.tpp:228-257), plus the slack-absorption
// column of a distributed slack: one pass over the mismatch's T, the step gathered from shared
// memory.  Returns max |F - J dx| to every thread (infinity when a value is not finite).
template <typename XT>
__device__ double newton_residual(const PlanArrays &P, Shared &S, const double2 *__restrict__ T,
                                  const double2 *__restrict__ Td, const double2 *__restrict__ Sd,
                                  const double2 *__restrict__ Fb, const XT *x, XT *__restrict__ rt) {
    const int ns = P.row_slots, bd = blockDim.x;
    double lmax = 0.0;
    int lbad = 0;
    for (int slot = threadIdx.x; slot < ns; slot += bd) {
        const int2 sl = P.row_slice[slot >> 5];
        const int2 eq = P.dg_eq[slot], ix = P.dg_x[slot];
        const double2 td = Td[slot], d = Sd[slot], F = Fb[slot];
        const int e0 = sl.x + (slot & 31);
        double2 j = make_double2(0.0, 0.0);
        for (int u0 = 0; u0 < sl.y; u0 += 4) {
            int2 i[4];
            double2 t[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = u0 + u < sl.y;
                i[u] = in ? P.off_x[e0 + (u0 + u) * 32] : make_int2(-1, -1);
                t[u] = in ? T[e0 + (u0 + u) * 32] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (i[u].x >= 0) {
                    const double a = (double)x[i[u].x];
                    j.x += t[u].y * a;
                    j.y -= t[u].x * a;
                }
                if (i[u].y >= 0) {
                    const double m = (double)x[i[u].y];
                    j.x += t[u].x * m;
                    j.y += t[u].y * m;
                }
            }
        }
        if (eq.x < 0 && eq.y < 0) continue;
        if (ix.x >= 0) {
            const double a = (double)x[ix.x];
            j.x += (td.y - d.y) * a;
            j.y -= (td.x - d.x) * a;
        }
        if (ix.y >= 0) {
            const double m = (double)x[ix.y];
            j.x += (td.x + d.x) * m;
            j.y += (td.y + d.y) * m;
        }
        if (P.distributed && eq.x >= 0) j.x += P.wJ[P.row_bus[slot]] * (double)x[P.xSlack];
        if (eq.x >= 0) {
            const double rp = F.x - j.x;
            rt[eq.x] = (XT)rp;
            lmax = fmax(lmax, fabs(rp));
            lbad |= !isfinite(rp);
        }
        if (eq.y >= 0) {
            const double rq = F.y - j.y;
            rt[eq.y] = (XT)rq;
            lmax = fmax(lmax, fabs(rq));
            lbad |= !isfinite(rq);
        }
    }
    double rmax;
    int bad;
    block_norm(S, lmax, lbad, rmax, bad);
    return bad ? INFINITY : rmax;
}

// The voltage update of a Newton step: Va -= dVa, Vm -= |V| (dVm / |V|) (the step x; when corrected,
// the first step dx plus the correction x, added in FP64),
// V = Vm e^(j Va) into the slab (and the shared copy Vs); returns the thread's smallest new
// magnitude.  Pairs of buses: their loads (magnitudes and angles, step positions, then
// the step values) are issued together before the arithmetic of the first bus.
// The reference re-derives Vm = |V| and Va = arg(V) before every update (BaseNRSingleSlackAlgo.tpp:
// 131-132), which changes them only where the last magnitude was negative or the angle left
// (-pi, pi]; elsewhere they equal the updated values up to rounding.  So a bus keeps its updated Vm
// and Va and only those buses take |V| and arg(V): two FP64 library calls (and their dependent
// chains) per bus fewer.  The distributed-slack form keeps its own block-wide re-derivation.
template <typename XT>
__device__ double voltage_update(const PlanArrays &P, double2 *__restrict__ V, double2 *__restrict__ Vs,
                                           double *__restrict__ Vm, double *__restrict__ Va,
                                           const XT *__restrict__ dx, const XT *x, bool corrected) {
    const int n = P.n;
    double lmin = 1.0;
    constexpr int R = 2;
    const int bd = blockDim.x;
    for (int b0 = threadIdx.x; b0 < n; b0 += R * bd) {
        double vm[R], va[R];
        int ia[R], im[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int b = b0 + i * bd;
            const bool ok = b < n;
            ia[i] = ok ? P.xVa[b] : -1;
            im[i] = ok ? P.xVm[b] : -1;
            vm[i] = ok ? Vm[b] : 1.0;
            va[i] = ok ? Va[b] : 0.0;
        }
        double da[R], dm[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            da[i] = ia[i] >= 0 ? (double)x[ia[i]] + (corrected ? (double)dx[ia[i]] : 0.0) : 0.0;
            dm[i] = im[i] >= 0 ? (double)x[im[i]] + (corrected ? (double)dx[im[i]] : 0.0) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int b = b0 + i * bd;
            if (b >= n) break;
            double a = va[i], mg = vm[i];
            if (ia[i] >= 0) a -= da[i];
            if (im[i] >= 0) mg -= mg * dm[i];  // the unknown is dVm / |V|, and mg = |V|
            double sn, cs;
            sincos(a, &sn, &cs);
            const double2 v = make_double2(mg * cs, mg * sn);
            V[b] = v;
            if (Vs) Vs[b] = v;
            lmin = fmin(lmin, mg);
            if (!P.distributed && !(mg >= 0.0 && fabs(a) <= kPi)) {
                // the reference's re-derivation, where it changes the values (or they are not finite)
                mg = cabs2(v);
                a = atan2(v.y, v.x);
            }
            Vm[b] = mg;
            Va[b] = a;
        }
    }
    return lmin;
}


// ---------------------------------------------------------------- dense tail
// The trailing block of steps [tail_ct, tail_ct + k) of a plan with a dense tail, as a dense
// row-major k x k matrix D in the CTA's slab (row stride tail_ld(k), a multiple of 4 values, so
// that every row starts on 16 bytes).  After the factor program has applied the pivots before
// the block (their updates of the block are the Schur complement of the sparse part),
// tail_factor gathers the block from the LU and factorises it without pivoting, right-looking
// in panels of NB = tail_panel<LT>() columns:
// (a) the panel's diagonal block is factorised (a warp per row, a lane per column) and left in
//     shared memory;
// (b) every row below (its L values) and every column right of it (its U values) is an independent
//     triangular solve against that block: a thread per row or column, its NB values in registers,
//     the block's values by 16-byte broadcast reads; the results go to D and to shared memory
//     (As by column of L, Bs by row of U);
// (c) the trailing rows minus L U: each thread a register tile of TR x 4 outputs, 2 + 1 16-byte
//     shared-memory reads per 32 multiply-adds (FP32), D read and written with 16-byte accesses.
// With the whole panel factorised in shared memory, a barrier per pivot and 5 reads per 16
// multiply-adds, the 391-step block took 1.64M SM cycles in FP32; now 0.93M: gather 145k, (a) 185k,
// (b) 200k, (c) 400k (its multiply-adds alone: 156k).  2,848-bus grid with 300 chords, N-1: mixed
// 72.0 -> 60.1 ms, FP64 131 -> 109 ms.
// A right part wider than tail_w columns (the staging area's
// share of shared memory) is solved and applied in chunks.  The block's pivots go back to the
// LU diagonal, where the pivot scaling and the zero-pivot check read them.
template <typename LT>
__host__ __device__ constexpr int tail_panel() { return sizeof(LT) == 4 ? 32 : 16; }
__host__ __device__ inline int tail_ld(int k) { return (k + 3) & ~3; }
__host__ __device__ inline int tail_lda(int k) { return (k + 7) & ~7; }
// the diagonal block (TailPanel), As and a chunk of w columns of Bs
__host__ __device__ inline size_t tail_smem_bytes(int k, int w, int lu_bytes) {
    const int nb = lu_bytes == 4 ? 32 : 16;
    return k > 0 ? (size_t)nb * (2 * nb + 1 + tail_lda(k) + w) * lu_bytes : 0;
}

// 16 bytes at a 16-byte boundary, in shared memory (an address of __cvta_generic_to_shared: the
// functions below are not inlined, and a generic load costs more) or through a generic pointer
template <typename LT>
struct Vec16;
template <>
struct Vec16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void lds(unsigned a, float *v) {
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a));
    }
    static __device__ __forceinline__ void sts(unsigned a, const float *v) {
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
    }
    static __device__ __forceinline__ void ld(const float *p, float *v) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    static __device__ __forceinline__ void st(float *p, const float *v) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <>
struct Vec16<double> {
    static constexpr int N = 2;
    static __device__ __forceinline__ void lds(unsigned a, double *v) {
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a));
    }
    static __device__ __forceinline__ void sts(unsigned a, const double *v) {
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]) : "memory");
    }
    static __device__ __forceinline__ void ld(const double *p, double *v) {
        const double2 t = *reinterpret_cast<const double2 *>(p);
        v[0] = t.x; v[1] = t.y;
    }
    static __device__ __forceinline__ void st(double *p, const double *v) {
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    }
};
__device__ __forceinline__ float lds(unsigned a, float v) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ double lds(unsigned a, double v) {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts(unsigned a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts(unsigned a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }

// Shared memory of a panel: ush, row c = U(c, c ..) of the diagonal block from column 0, zero past its
// end; lsh, row c = (0, L(c + 1, c), L(c + 2, c), ...), zero past its end; the reciprocal pivots.  So every step of (a) and (b) reads its NB values from the same place of the row, and
// the solves are loops whose register arrays move down by one value a step: unrolled over all
// steps (half the multiply-adds) the code of (a) and (b) did not stay in the instruction cache, and
// the one warp of (a) took 34k cycles a panel, waiting for instructions.
template <typename LT>
struct TailPanel {
    static constexpr int NB = tail_panel<LT>(), N = Vec16<LT>::N, E = (int)sizeof(LT);
    static constexpr int kL = NB * NB * E, kR = 2 * NB * NB * E, kBytes = kR + NB * E;
    // v[j - 1] = v[j] - f row[j] for j < W, row at shared address r
    template <int W>
    static __device__ __forceinline__ void step(LT (&v)[NB], unsigned r, LT f) {
        LT u[W];
#pragma unroll
        for (int j = 0; j < W; j += N) Vec16<LT>::lds(r + j * E, u + j);
#pragma unroll
        for (int j = 1; j < W; ++j) v[j - 1] = v[j] - f * u[j];
    }
};

// (a) the diagonal block at row and column J (jb steps; past them the identity) to `sm` and back to D, by
// the whole CTA: a warp per row (R rows each), a lane per column, the values in registers.  Per pivot:
// its row from shared memory (`blk`, two rows used in turn), published by the row's warp after the
// previous pivot, and one barrier; what (b) reads is written after the last one.  Bound by that serial
// chain (read, shuffle, reciprocal, update, write, barrier): 322 cycles a pivot alone on an SM, against 620
// with (b)'s rows written per pivot and 660 with the block in shared memory and a read-modify-write
// per element; one warp with a row per lane took 758.
template <typename LT, int R>
__device__ __forceinline__ void tail_diagonal_rows(LT *D, int ld, int J, int jb, unsigned sm, unsigned blk) {
    using T = TailPanel<LT>;
    constexpr int NB = T::NB, E = T::E;
    const int j = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    LT *base = D + (size_t)J * ld + J;
    LT v[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int i = warp + s * nwarps;
        v[s] = i < jb && j < jb ? base[(size_t)i * ld + j] : (LT)(i == j);
    }
    for (int e = threadIdx.x; e < 2 * NB * NB; e += blockDim.x) sts(sm + e * E, (LT)0);
    if (warp == 0 && j < NB) sts(blk + j * E, v[0]);
    __syncthreads();
    for (int c = 0; c + 1 < NB; ++c) {
        const unsigned row = blk + (c & 1) * NB * E, next = blk + ((c + 1) & 1) * NB * E;
        const LT u = lds(row + (j < NB ? j : 0) * E, (LT)0), piv = __shfl_sync(0xffffffffu, u, c);
        const LT r = tail_reciprocal(piv);
#pragma unroll
        for (int s = 0; s < R; ++s) {
            const int i = warp + s * nwarps;
            const LT f = tail_quotient(__shfl_sync(0xffffffffu, v[s], c), piv, r);
            if (i > c) v[s] = j > c ? v[s] - f * u : (j == c ? f : v[s]);
            if (i == c + 1 && j < NB) sts(next + j * E, v[s]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int s = 0; s < R; ++s) {
        const int i = warp + s * nwarps;
        if (i >= NB || j >= NB) continue;
        sts(sm + (j >= i ? i * NB + j - i : NB * NB + j * NB + i - j) * E, v[s]);
        if (i == j) sts(sm + T::kR + i * E, (LT)1 / v[s]);
        if (i < jb && j < jb) base[(size_t)i * ld + j] = v[s];
    }
    __syncthreads();
}
template <typename LT>
__device__ __noinline__ void tail_diagonal(LT *D, int ld, int J, int jb, unsigned sm, unsigned blk) {
    constexpr int NB = tail_panel<LT>();
    const int nwarps = blockDim.x >> 5;
    if (nwarps >= NB) tail_diagonal_rows<LT, 1>(D, ld, J, jb, sm, blk);
    else if (nwarps * 2 >= NB) tail_diagonal_rows<LT, 2>(D, ld, J, jb, sm, blk);
    else tail_diagonal_rows<LT, NB>(D, ld, J, jb, sm, blk);  // few warps: up to all rows each
}

// (b) one row below the diagonal block: L values (a full panel)
template <typename LT>
__device__ __forceinline__ void tail_row(LT *row, unsigned sm, unsigned as, int lda) {
    using T = TailPanel<LT>;
    constexpr int NB = T::NB, N = T::N, E = T::E;
    LT a[NB];
#pragma unroll
    for (int j = 0; j < NB; j += N) Vec16<LT>::ld(row + j, a + j);
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll 1
        for (int c = half * (NB / 2); c < (half + 1) * (NB / 2); c += N) {
            LT rp[N], q[N];
            Vec16<LT>::lds(sm + T::kR + c * E, rp);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const unsigned u = sm + (c + i) * NB * E;
                q[i] = tail_quotient(a[0], lds(u, (LT)0), rp[i]);
                sts(as + (unsigned)((c + i) * lda * E), q[i]);
                if (half == 0) T::template step<NB>(a, u, q[i]);
                else T::template step<NB / 2>(a, u, q[i]);
            }
            Vec16<LT>::st(row + c, q);
        }
}

// (b) one column right of the diagonal block: U values (a full panel)
template <typename LT>
__device__ __forceinline__ void tail_column(LT *col, int ld, unsigned sm, unsigned bs, int ldb) {
    using T = TailPanel<LT>;
    constexpr int NB = T::NB, N = T::N, E = T::E;
    LT v[NB];
#pragma unroll
    for (int r = 0; r < NB; ++r) v[r] = col[(size_t)r * ld];
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll 1
        for (int c = half * (NB / 2); c < (half + 1) * (NB / 2); c += N)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const LT u = v[0];
                col[(size_t)(c + i) * ld] = u;
                sts(bs + (unsigned)((c + i) * ldb * E), u);
                if (half == 0) T::template step<NB>(v, sm + T::kL + (c + i) * NB * E, u);
                else T::template step<NB / 2>(v, sm + T::kL + (c + i) * NB * E, u);
            }
}

// The stages of tail_factor are functions of their own: inlined together they spilled inside
// their loops.
template <typename LT>
__device__ __noinline__ void tail_gather(const int *__restrict__ map, const LT *lu, LT *D, int k) {
    const int ld = tail_ld(k), bd = blockDim.x, kk = k * k;
    // four entries per thread in flight
    for (int e0 = threadIdx.x; e0 < kk; e0 += 4 * bd) {
        int p[4];
        LT v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = e0 + u * bd < kk ? __ldg(map + e0 + u * bd) : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = p[u] >= 0 ? lu[p[u]] : (LT)0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * bd;
            if (e < kk) D[(size_t)(e / k) * ld + e % k] = v[u];
        }
    }
    __syncthreads();
}

// (b): `rows` rows below the diagonal block at (J, J) and the w columns from j0
template <typename LT>
__device__ __noinline__ void tail_solves(LT *D, int k, int J, int j0, int rows, int w, int W, unsigned sm) {
    constexpr int NB = tail_panel<LT>(), E = (int)sizeof(LT);
    const int ld = tail_ld(k), lda = tail_lda(k);
    const unsigned as = sm + TailPanel<LT>::kBytes, bs = as + (unsigned)(NB * lda * E);
    for (int t = threadIdx.x; t < rows + w; t += blockDim.x) {
        if (t < rows)
            tail_row<LT>(D + (size_t)(J + NB + t) * ld + J, sm, as + (unsigned)(t * E), lda);
        else
            tail_column<LT>(D + (size_t)J * ld + j0 + (t - rows), ld, sm, bs + (unsigned)((t - rows) * E), W);
    }
    __syncthreads();
}

// (c): rows and columns right of the panel (M rows from J1, w columns from j0) minus As Bs.  A warp per
// 4 x 8 register tiles of TR x 4 values (the lanes of a row read 128 consecutive bytes of Bs; columns past the
// block's last fall in the row padding, their values are never read as entries).
template <typename LT>
__device__ __noinline__ void tail_update(LT *D, int k, int J1, int j0, int w, int W, unsigned sm) {
    constexpr int NB = tail_panel<LT>(), N = Vec16<LT>::N, E = (int)sizeof(LT);
    constexpr int TR = E == 4 ? 8 : 4;
    const int ld = tail_ld(k), lda = tail_lda(k), M = k - J1;
    const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const unsigned as = sm + TailPanel<LT>::kBytes, bs = as + (unsigned)(NB * lda * E);
    const int sr = (M + 4 * TR - 1) / (4 * TR), sc = (w + 31) / 32;
    for (int t = threadIdx.x >> 5; t < sr * sc; t += nwarps) {
        const int ti = t / sc, i0 = (ti * 4 + (lane >> 3)) * TR, q0 = (t - ti * sc) * 32 + (lane & 7) * 4;
        if (i0 >= M || q0 >= w) continue;
        LT *C = D + (size_t)(J1 + i0) * ld + j0 + q0;
        LT acc[TR][4];
#pragma unroll
        for (int r = 0; r < TR; ++r)
#pragma unroll
            for (int q = 0; q < 4; q += N) {
                if (i0 + r < M) Vec16<LT>::ld(C + (size_t)r * ld + q, &acc[r][q]);
                else
#pragma unroll
                    for (int i = 0; i < N; ++i) acc[r][q + i] = (LT)0;
            }
        const unsigned pa = as + (unsigned)(i0 * E), pb = bs + (unsigned)(q0 * E);
#pragma unroll 4
        for (int c = 0; c < NB; ++c) {
            LT av[TR], bv[4];
#pragma unroll
            for (int r = 0; r < TR; r += N) Vec16<LT>::lds(pa + (unsigned)((c * lda + r) * E), av + r);
#pragma unroll
            for (int q = 0; q < 4; q += N) Vec16<LT>::lds(pb + (unsigned)((c * W + q) * E), bv + q);
#pragma unroll
            for (int r = 0; r < TR; ++r)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[r][q] -= av[r] * bv[q];
        }
#pragma unroll
        for (int r = 0; r < TR; ++r)
#pragma unroll
            for (int q = 0; q < 4; q += N)
                if (i0 + r < M) Vec16<LT>::st(C + (size_t)r * ld + q, &acc[r][q]);
    }
    __syncthreads();
}

template <typename LT>
__device__ __noinline__ void tail_factor(const PlanArrays &P, LT *lu, LT *D, LT *smem) {
    constexpr int NB = tail_panel<LT>();
    const int k = P.tail_k, ld = tail_ld(k), W = P.tail_w;
    tail_gather<LT>(P.tail_map, lu, D, k);
    const unsigned sm = (unsigned)__cvta_generic_to_shared(smem);
    for (int J = 0; J < k; J += NB) {
        const int jb = min(NB, k - J), J1 = J + jb, M = k - J1;
        tail_diagonal<LT>(D, ld, J, jb, sm, sm + TailPanel<LT>::kBytes);  // As is not in use yet
        for (int j0 = J1; j0 < k; j0 += W) {
            const int w = min(W, k - j0);
            tail_solves<LT>(D, k, J, j0, j0 == J1 ? M : 0, w, W, sm);
            tail_update<LT>(D, k, J1, j0, w, W, sm);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < k; c += blockDim.x) lu[P.dpos[P.tail_ct + c]] = D[(size_t)c * ld + c];
    __syncthreads();
}

// Forward substitution of the block (unit lower L of tail_factor) on x[tail_ct, tail_ct + k),
// after the forward pushes of the pivots before the block: per panel of 32 rows, the diagonal
// block staged in shared memory (`sm`, row stride 33), warp 0 solves it (a lane per row, values exchanged by
// shuffles), then every thread updates rows below it.  Warp 0's chain bounds it: the loop runs a fixed 32
// steps, so that the block's values are read ahead of the shuffles.
template <typename LT, typename XT>
__device__ __noinline__ void tail_forward(const PlanArrays &P, const LT *D, XT *x, LT *sm) {
    const int k = P.tail_k, ld = tail_ld(k), tid = threadIdx.x, bd = blockDim.x;
    XT *xt = x + P.tail_ct;
    for (int J = 0; J < k; J += 32) {
        const int jb = min(32, k - J), J1 = J + jb;
        for (int e = tid; e < jb * 32; e += bd) {
            const int a = e >> 5, b = e & 31;
            sm[a * 33 + b] = b < jb ? D[(size_t)(J + a) * ld + J + b] : (LT)0;
        }
        __syncthreads();
        if (tid < 32) {
            XT v = tid < jb ? xt[J + tid] : (XT)0;
            const LT *row = sm + min(tid, jb - 1) * 33;  // zero past the panel
#pragma unroll 8
            for (int c = 0; c < 32; ++c) {
                const XT a = (XT)row[c], vc = __shfl_sync(0xffffffffu, v, c);
                if (tid > c) v -= a * vc;
            }
            if (tid < jb) xt[J + tid] = v;
        }
        __syncthreads();
        for (int i = J1 + tid; i < k; i += bd) {
            XT v = xt[i];
            const LT *row = D + (size_t)i * ld + J;
            // the panel is full here (rows below it exist): 16-byte reads of the row
#pragma unroll
            for (int c = 0; c < 32; c += Vec16<LT>::N) {
                LT r[Vec16<LT>::N];
                Vec16<LT>::ld(row + c, r);
#pragma unroll
                for (int u = 0; u < Vec16<LT>::N; ++u) v -= (XT)r[u] * xt[J + c + u];
            }
            xt[i] = v;
        }
        __syncthreads();
    }
}

// Backward substitution of the block, before the backward program, in its convention: the values
// stay undivided (z(c) = U(c, c) x(c)) and a push divides by the pivot; the pivot scaling after
// the program divides them.  Per panel from the last: the diagonal block staged in shared
// memory, warp 0 solves it and leaves the panel's z(c) / U(c, c) in S.red, then every thread
// updates the rows above it.  A step of warp 0's chain is a quotient from the lane's reciprocal
// pivot, a shuffle and a multiply-add; with the division operator after the shuffle and the block read
// in the chain, here and in tail_forward, the 300-chord N-1 batch took 49.9 instead of 48.3 ms mixed and 91.1
// instead of 88.8 ms in FP64, the same bits.
template <typename LT, typename XT>
__device__ __noinline__ void tail_backward(const PlanArrays &P, Shared &S, const LT *D, XT *x, LT *sm) {
    const int k = P.tail_k, ld = tail_ld(k), tid = threadIdx.x, bd = blockDim.x;
    XT *xt = x + P.tail_ct;
    const int last = ((k - 1) / 32) * 32;
    for (int J = last; J >= 0; J -= 32) {
        const int jb = min(32, k - J);
        for (int e = tid; e < jb * 32; e += bd) {
            const int a = e >> 5, b = e & 31;
            sm[a * 33 + b] = b < jb ? D[(size_t)(J + a) * ld + J + b] : (LT)0;
        }
        __syncthreads();
        if (tid < 32) {
            XT z = tid < jb ? xt[J + tid] : (XT)0, q = (XT)0;
            const LT *row = sm + min(tid, jb - 1) * 33;
            const XT u = tid < jb ? (XT)row[tid] : (XT)1, r = (XT)1 / u;
#pragma unroll 8
            for (int c = 31; c >= 0; --c) {
                // every lane's quotient so far; column c's is final (zero past the panel)
                const XT a = (XT)row[c], w = __shfl_sync(0xffffffffu, tail_quotient(z, u, r), c);
                if (tid == c) q = w;
                if (tid < c) z -= a * w;
            }
            if (tid < jb) {
                xt[J + tid] = z;
                S.red[tid] = (double)q;
            }
        }
        __syncthreads();
        for (int i = tid; i < J; i += bd) {
            XT v = xt[i];
            const LT *row = D + (size_t)i * ld + J;
            if (jb == 32) {
#pragma unroll
                for (int c = 0; c < 32; c += Vec16<LT>::N) {
                    LT r[Vec16<LT>::N];
                    Vec16<LT>::ld(row + c, r);
#pragma unroll
                    for (int u = 0; u < Vec16<LT>::N; ++u) v -= (XT)r[u] * (XT)S.red[c + u];
                }
            } else {
                for (int c = 0; c < jb; ++c) v -= (XT)row[c] * (XT)S.red[c];
            }
            xt[i] = v;
        }
        __syncthreads();
    }
}

// Where one plan's data lives for a CTA: shared memory x | LU (LU_SMEM: one index space, LU at
// element lu_offset) | phase tables, and the CTA's slab of the scratch memory.
// The slab's part before the LU: V (16 B per bus), Vm, Va (8 B per bus), Td, Sd (16 B per row
// slot), T (16 B per off-diagonal slot); FP32 plans also the FP64 mismatch (16 B per row slot), the
// first step of a refinement and its residual (a value per unknown).
__host__ __device__ inline size_t bus_slab_bytes(const PlanArrays &P, int x_bytes) {
    size_t b = (size_t)P.n * 32 + (size_t)P.row_slots * 32 + (size_t)P.row_len * 16;
    if (x_bytes == 4) b += (size_t)P.row_slots * 16 + (size_t)P.m * 8;
    return (b + 255) & ~(size_t)255;
}
template <typename LT, typename XT>
struct Layout {
    XT *x;
    LT *lu;
    LT *D;    // dense tail block (global-memory LU plans with a tail)
    LT *tsm;  // its staging area in shared memory
    double2 *V, *Td, *Sd, *T, *Fb;
    double *Vm, *Va;
    XT *dx, *rt;
    int *sb_fac, *sb_bwd, *sb_fwd, *sw_fac, *sw_bwd, *sw_fwd;
    uint2 *nar_ops[3];  // staged operations of the narrow phases (packed layout)
};

template <typename LT, typename XT, bool LU_SMEM>
__device__ __forceinline__ Layout<LT, XT> make_layout(const PlanArrays &P, const BatchArgs &A, unsigned char *dyn) {
    Layout<LT, XT> L;
    const int n = P.n, m = P.m;
    const size_t xbytes = LU_SMEM ? (size_t)P.lu_offset * sizeof(XT) : (((size_t)m * sizeof(XT) + 15) & ~(size_t)15);
    L.x = reinterpret_cast<XT *>(dyn);
    // opaque to the optimiser: every pass of a Newton step derives its pointers again instead of
    // keeping all of them live (or spilled) across the others
    unsigned char *slab = A.scratch + (size_t)blockIdx.x * (size_t)A.slab_bytes;
    asm volatile("" : "+l"(slab));
    L.V = reinterpret_cast<double2 *>(slab);
    L.Td = L.V + n;
    L.Sd = L.Td + P.row_slots;
    L.T = L.Sd + P.row_slots;
    L.Vm = reinterpret_cast<double *>(L.T + P.row_len);
    L.Va = L.Vm + n;
    L.Fb = reinterpret_cast<double2 *>(L.Va + n);  // FP32 plans: Fb, dx, rt
    L.dx = reinterpret_cast<XT *>(L.Fb + P.row_slots);
    L.rt = L.dx + m;
    const size_t bus_bytes = bus_slab_bytes(P, sizeof(XT));
    L.lu = LU_SMEM ? reinterpret_cast<LT *>(dyn + xbytes) : reinterpret_cast<LT *>(slab + bus_bytes);
    L.D = LU_SMEM ? nullptr
                  : reinterpret_cast<LT *>(slab + bus_bytes + (((size_t)P.nnzLU * sizeof(LT) + 255) & ~(size_t)255));
    L.sb_fac = reinterpret_cast<int *>(dyn + xbytes +
                                       (LU_SMEM ? (((size_t)P.nnzLU * sizeof(LT) + 15) & ~(size_t)15) : 0));
    L.sb_bwd = L.sb_fac + P.fac_nph + 1;
    L.sb_fwd = L.sb_bwd + P.bwd_nph + 1;
    L.sw_fac = L.sb_fwd + P.fwd_nph + 1;
    L.sw_bwd = L.sw_fac + P.fac_nph;
    L.sw_fwd = L.sw_bwd + P.bwd_nph;
    {
        // the narrow phases' operations after the tables, 8-byte aligned
        const size_t off = (size_t)((reinterpret_cast<unsigned char *>(L.sw_fwd + P.fwd_nph) - dyn + 7) & ~(size_t)7);
        uint2 *base = reinterpret_cast<uint2 *>(dyn + off);
        for (int k = 0; k < 3; ++k) L.nar_ops[k] = base + P.nar_off[k];
        // the dense tail's staging area after the tables, 16-byte aligned (global-memory LU)
        L.tsm = LU_SMEM ? nullptr : reinterpret_cast<LT *>(dyn + ((off + 15) & ~(size_t)15));
    }
    return L;
}

// Phase bounds and widths of the three programs into shared memory (caller synchronises).
template <typename LT, typename XT>
__device__ __forceinline__ void stage_tables(const PlanArrays &P, const Layout<LT, XT> &L) {
    for (int i = threadIdx.x; i <= P.fac_nph; i += blockDim.x) L.sb_fac[i] = P.fac_base[i];
    for (int i = threadIdx.x; i <= P.bwd_nph; i += blockDim.x) L.sb_bwd[i] = P.bwd_base[i];
    for (int i = threadIdx.x; i <= P.fwd_nph; i += blockDim.x) L.sb_fwd[i] = P.fwd_base[i];
    for (int i = threadIdx.x; i < P.fac_nph; i += blockDim.x) L.sw_fac[i] = P.fac_width[i];
    for (int i = threadIdx.x; i < P.bwd_nph; i += blockDim.x) L.sw_bwd[i] = P.bwd_width[i];
    for (int i = threadIdx.x; i < P.fwd_nph; i += blockDim.x) L.sw_fwd[i] = P.fwd_width[i];
    if (P.compact) {
        const uint2 *cops[3] = {P.fac_cops, P.bwd_cops, P.fwd_cops};
        for (int k = 0; k < 3; ++k) {
            const int cnt = P.nar_off[k + 1] - P.nar_off[k];
            for (int i = threadIdx.x; i < cnt; i += blockDim.x) L.nar_ops[k][i] = cops[k][P.nar_first[k] + i];
        }
    }
}

// Per-phase SM cycles, measured by thread 0 between the barriers that end each phase.
struct Prof {
    bool on;
    int traced;
    unsigned long long tmark;
    unsigned long long *pc;  // Shared::pc: the counters stay out of the registers
    __device__ __forceinline__ void start(bool o, unsigned long long *counters) {
        on = o;
        traced = 0;
        pc = counters;
        tmark = o ? clock64() : 0;
        if (o)
            for (int i = 0; i < kPhaseSlots; ++i) pc[i] = 0;
    }
    __device__ __forceinline__ void mark(int slot) {
        if (on) {
            const unsigned long long t = clock64();
            pc[slot] += t - tmark;
            tmark = t;
        }
    }
};

// One job: instances [first, first + count) of a batch, chained for a time series.  The batch's
// inputs (start voltages, injections, overrides) are read through L2 only (ld.global.cg): in the
// device-resident request loop one launch serves many requests whose inputs reuse device
// addresses, and an SM's L1 could still hold an earlier request's lines.
// NARROW: the narrow phases of the packed programs run on their few warps (the 512- and
// 640-thread variants; at 768 threads the registers it takes cost more than it saves).
template <typename LT, typename XT, bool LU_SMEM, bool REFINE, bool NARROW>
__device__ __forceinline__ void solve_job(const PlanArrays &P, const BatchArgs &A, Shared &S, unsigned char *dyn, int first, int count, Prof &pr) {
    const int tid = threadIdx.x;
    const int n = P.n, m = P.m;
    const auto lay = [&]() { return make_layout<LT, XT, LU_SMEM>(P, A, dyn); };
    XT *const x = reinterpret_cast<XT *>(dyn);
    // With the LU in shared memory, the LU region is dead from the voltage update to the next
    // Jacobian fill: the voltages are also written there (Vs) and the mismatch gathers them from
    // shared memory instead of the slab.  Not when the LU must survive the mismatch (LU reuse).
    double2 *Vs = nullptr;
    if constexpr (LU_SMEM) {
        if (!(REFINE && A.reuse_below > 0.0) && (size_t)n * sizeof(double2) <= (size_t)P.nnzLU * sizeof(LT))
            Vs = reinterpret_cast<double2 *>(lay().lu);
    }
    for (int step = 0; step < count; ++step) {
        const int inst = first + step;
        const double2 *Sb = A.Sbus + (long long)inst * A.sbus_stride;
        if (step == 0 || !A.chain) {
            const Layout<LT, XT> L = lay();
            const double2 *v0 = A.v0_from_out ? out_row(A, inst, n) : A.V0 + (long long)inst * A.v0_stride;
            for (int b = tid; b < n; b += blockDim.x) {
                const double2 v = __ldcg(v0 + b);
                L.V[b] = v;
                if (Vs) Vs[b] = v;
                L.Vm[b] = cabs2(v);
                L.Va[b] = atan2(v.y, v.x);
            }
        } else {
            const Layout<LT, XT> L = lay();
            for (int b = tid; b < n; b += blockDim.x) {
                const double2 v = L.V[b];
                if (Vs) Vs[b] = v;
                L.Vm[b] = cabs2(v);
                L.Va[b] = atan2(v.y, v.x);
            }
        }
        // the mismatch reads the injections in row-slot order: bring the row into L2 in bus order first
        for (int b = 8 * tid; b < n; b += 8 * blockDim.x)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(Sb + b));
        if (tid == 0) {
            int k0 = 0, k1 = 0;
            if (A.ovr_ptr) {
                k0 = __ldcg(A.ovr_ptr + inst);
                k1 = __ldcg(A.ovr_ptr + inst + 1);
            }
            S.novr = k1 - k0 > kMaxOverrides ? -1 : k1 - k0;  // -1: too many to stage
            S.piv_err = 0;
            S.slack_absorbed = 0.0;
        }
        __syncthreads();
        if (tid < S.novr) {
            const int k0 = __ldcg(A.ovr_ptr + inst);
            stage_override(P, S, tid, __ldcg(A.ovr_pos + k0 + tid), __ldcg(A.ovr_val + k0 + tid));
        }
        if (P.distributed) {
            double ls = 0.0;
            for (int b = tid; b < n; b += blockDim.x) ls += __ldcg(Sb + b).x;
            const double tot = block_sum(S, ls);
            if (tid == 0) S.slack_absorbed = tot;
        }
        __syncthreads();
        if (S.novr < 0) {
            // more Ybus overrides than the kernel stages: not computed (start voltages out)
            double2 *vo = out_row(A, inst, n);
            const double2 *V = lay().V;
            for (int b = tid; b < n; b += blockDim.x) vo[b] = A.zero_failed ? make_double2(0.0, 0.0) : V[b];
            if (tid == 0) {
                A.iters[inst] = 0;
                A.errs[inst] = 8;  // NotInitError
            }
            __syncthreads();
            if (A.chain) {
                for (int s2 = step + 1 + tid; s2 < count; s2 += blockDim.x) {
                    A.iters[first + s2] = 0;
                    A.errs[first + s2] = 8;
                }
                break;
            }
            continue;
        }
        double norm;
        int bad;
        const auto step_mismatch = [&]() {
            const Layout<LT, XT> L = lay();
            mismatch<XT, REFINE>(P, S, Vs ? Vs : L.V, L.T, L.Td, L.Sd, L.Fb, Sb, x, norm, bad);
        };
        pr.mark(6);
        step_mismatch();
        pr.mark(0);
        bool conv = !bad && norm < A.tol;
        int it = A.it_start ? A.it_start[inst] : 0, err = 0;
        double2 *const Vlast = inst == A.j_inst ? A.Vlast : nullptr;
        Trace tr{(A.trace != nullptr && blockIdx.x == 0 && pr.traced == 0) ? A.trace : nullptr, A.trace_cap, 0};
        pr.traced = 1;
        const auto program_factor = [&]() {
            const Layout<LT, XT> L = lay();
            run_lu_program<LT, XT, LU_SMEM, false, NARROW>(packed_ops<LU_SMEM>(P, P.fac_cops), P.fac_ops, L.sb_fac, L.sw_fac,
                                                          P.fac_nph, m, P.lu_offset, L.lu, x, tr,
                                                          make_int3(P.nar_a[0], P.nar_b[0], P.nar_warps), L.nar_ops[0]);
        };
        const auto program_backward = [&]() {
            const Layout<LT, XT> L = lay();
            run_lu_program<LT, XT, LU_SMEM, true, NARROW>(packed_ops<LU_SMEM>(P, P.bwd_cops), P.bwd_ops, L.sb_bwd, L.sw_bwd,
                                                          P.bwd_nph, m, P.lu_offset, L.lu, x, tr,
                                                          make_int3(P.nar_a[1], P.nar_b[1], P.nar_warps), L.nar_ops[1]);
        };
        const auto program_forward = [&]() {
            const Layout<LT, XT> L = lay();
            run_lu_program<LT, XT, LU_SMEM, true, NARROW>(packed_ops<LU_SMEM>(P, P.fwd_cops), P.fwd_ops, L.sb_fwd, L.sw_fwd,
                                                          P.fwd_nph, m, P.lu_offset, L.lu, x, tr,
                                                          make_int3(P.nar_a[2], P.nar_b[2], P.nar_warps), L.nar_ops[2]);
        };
        bool have_lu = false;  // this instance's LU from an earlier iteration is in place
        while (!conv && it < A.max_iter) {
            ++it;
            const bool refine_now = REFINE && norm < A.refine_below;
            // close to the solution the Jacobian barely moves between iterations: the step is
            // solved with the previous iteration's LU and refined against the current FP64
            // Jacobian (refine_now holds: reuse_below <= refine_below)
            const bool reuse = REFINE && have_lu && Vlast == nullptr && norm < A.reuse_below;
            tr.mark();
            if (Vlast)  // one instance of a single power flow
                for (int b = tid; b < n; b += blockDim.x) Vlast[b] = lay().V[b];
            if (!reuse) {
                {
                    const Layout<LT, XT> L = lay();
                    jacobian_fill<LT, LU_SMEM>(P, L.T, L.Td, L.Sd, L.lu);
                }
                __syncthreads();
                pr.mark(1);
                // refactorisation with the forward substitution of the right-hand side fused in
                program_factor();
                if constexpr (!LU_SMEM) {
                    if (P.tail_k > 0) {
                        tail_factor<LT>(P, lay().lu, lay().D, lay().tsm);
                        tail_forward<LT, XT>(P, lay().D, x, lay().tsm);
                    }
                }
                pr.mark(2);
                have_lu = true;
            } else {
                program_forward();
                if constexpr (!LU_SMEM) {
                    if (P.tail_k > 0) tail_forward<LT, XT>(P, lay().D, x, lay().tsm);
                }
                pr.mark(3);
            }
            if constexpr (!LU_SMEM) {
                if (P.tail_k > 0) tail_backward<LT, XT>(P, S, lay().D, x, lay().tsm);
            }
            program_backward();
            // a zero pivot of the refactorisation is detected here: the backward program ran on
            // non-finite values, which are dropped with the step
            scale_by_pivots<LT, XT, true>(P, S, lay().lu, x);
            if (S.piv_err) {
                err = 6;  // SolverReFactor
                break;
            }
            pr.mark(4);
            // the refinement's correction solve is skipped when the residual of the FP32 step is
            // below a hundredth of the tolerance: the correction would move the next mismatch by
            // less than that (J e = r), and the final voltages by at most |J^-1| tol / 100
            bool corrected = false;
            if constexpr (REFINE) {
                if (refine_now) {
                    const Layout<LT, XT> L = lay();
                    corrected = !(newton_residual<XT>(P, S, L.T, L.Td, L.Sd, L.Fb, x, L.rt) < 0.01 * A.tol);
                }
            }
            if (corrected) {
                const Layout<LT, XT> L = lay();
                for (int k = tid; k < m; k += blockDim.x) {
                    L.dx[k] = x[k];
                    x[k] = L.rt[k];
                }
                __syncthreads();
                program_forward();
                if constexpr (!LU_SMEM) {
                    if (P.tail_k > 0) {
                        tail_forward<LT, XT>(P, lay().D, x, lay().tsm);
                        tail_backward<LT, XT>(P, S, lay().D, x, lay().tsm);
                    }
                }
                program_backward();
                scale_by_pivots<LT, XT>(P, S, lay().lu, x);
            }
            if (refine_now) pr.mark(5);
            // voltage update
            const Layout<LT, XT> L = lay();
            const double lmin = voltage_update<XT>(P, L.V, Vs, L.Vm, L.Va, L.dx, x, corrected);
            if (P.distributed) {
                const double dxs = (double)x[P.xSlack] + (corrected ? (double)L.dx[P.xSlack] : 0.0);
                const double vmin = block_min(S, lmin);  // contains barriers
                if (tid == 0) S.slack_absorbed -= dxs;
                if (vmin < 0.0) {
                    for (int b = tid; b < n; b += blockDim.x) {
                        const double2 v = L.V[b];
                        L.Vm[b] = cabs2(v);
                        L.Va[b] = atan2(v.y, v.x);
                    }
                }
            }
            __syncthreads();
            tr.mark();
            tr.buf = nullptr;
            pr.mark(6);
            step_mismatch();
            pr.mark(0);
            if (bad) {
                err = 3;  // InifiniteValue
                break;
            }
            conv = norm < A.tol;
        }
        if (!conv && err == 0) err = 2;  // TooManyIterations
        double2 *vo = out_row(A, inst, n);
        const bool zero = A.zero_failed && err != 0;
        const double2 *V = lay().V;
        for (int b = tid; b < n; b += blockDim.x) __stcs(vo + b, zero ? make_double2(0.0, 0.0) : V[b]);
        if (tid == 0) {
            A.iters[inst] = it;
            A.errs[inst] = err;
            if (pr.on) pr.pc[7] += 1;
        }
        __syncthreads();
        if (A.chain && err != 0) {
            // the reference stops a time series at its first divergence
            for (int s2 = step + 1 + tid; s2 < count; s2 += blockDim.x) {
                A.iters[first + s2] = 0;
                A.errs[first + s2] = 8;  // NotInitError: not computed
            }
            break;
        }
    }
}

// The mixed form's FP64 fallback inside the launch: a job with an instance that did not converge
// in FP32 is solved again in FP64 by the same CTA, with the solve vector in the shared memory
// the FP32 LU used (the next job refills it) and the FP64 LU in the CTA's slab.  The same code
// as a separate FP64 launch (solve_job with FP64 LU in global memory); a function of its own so
// that its registers do not add to the FP32 path's.
__device__ __noinline__ void fp64_rerun(const PlanArrays &P, const BatchArgs &A, Shared &S, unsigned char *dyn,
                                        int first, int count) {
    const Layout<double, double> L = make_layout<double, double, false>(P, A, dyn);
    stage_tables<double, double>(P, L);
    __syncthreads();
    Prof pr;
    pr.start(false, S.pc);
    solve_job<double, double, false, false, false>(P, A, S, dyn, first, count, pr);
}

// QUEUE: the device-resident request loop (jobs from M.q); a variant of its own so that the
// other launches keep their registers.
// MAXT: the launch bound, 512, 640 or 768 threads.  More warps hide more of the phases' latency
// at fewer registers per thread (128, 96, 80): the large plans run 640 (mixed form, with the
// narrow phases on a few warps) or 768 threads (FP64 form).
template <typename LT, typename XT, bool LU_SMEM, bool REFINE, bool QUEUE, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) nr_batch_kernel(const DevPlan P0, const BatchArgs A0, const MultiArgs M) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ Shared S;
    // the plan and batch of the current job, in shared memory: a launch of one plan (M.segs
    // null) copies its parameters once; a launch over several plans copies the segment of a
    // job when it differs from the CTA's previous one and restages the phase tables.  Both
    // kinds run the same code, so an instance gives the same bits in either.
    __shared__ __align__(16) Segment seg;
    const int tid = threadIdx.x;
    constexpr bool queue = QUEUE;
    const bool multi = M.segs != nullptr || queue;
    int *const counter = multi ? M.job_counter : A0.job_counter;
    const int njobs = multi ? M.njobs : (A0.njobs_dev ? min(A0.njobs, *A0.njobs_dev) : A0.njobs);
    Prof pr;
    pr.start(A0.phase_cycles != nullptr && tid == 0, S.pc);
    int cur = -1;
    __shared__ QueueJob qjob;
    for (;;) {
        if constexpr (QUEUE) {
            // request loop: claim the next published job (compare-and-swap on the head, so a CTA
            // never holds a job that is not there yet); after idle_polls empty polls, leave
            if (tid == 0)
                S.job = claim_queue_job(M.q.jobs, M.q.cap, M.q.head, M.q.tail, M.q.closing, M.q.idle_polls, &qjob);
            __syncthreads();
            const int got = S.job;
            __syncthreads();
            if (got < 0) break;
        } else {
            if (tid == 0) S.job = atomicAdd(counter, 1);
            __syncthreads();
            const int job = S.job;
            __syncthreads();
            if (job >= njobs) break;
        }
        const int job = S.job;
        // a request loop keys the segment a CTA holds by the request's sequence number (slots
        // are reused by later requests)
        const int sj = queue ? qjob.req : (multi ? M.job_seg[job] : 0);
        if (sj != cur) {
            if (multi) {
                static_assert(sizeof(Segment) % sizeof(int4) == 0, "segment records are copied as int4");
                const int4 *src = reinterpret_cast<const int4 *>(queue ? M.q.segs + qjob.slot : M.segs + sj);
                int4 *dst = reinterpret_cast<int4 *>(&seg);
                for (int i = tid; i < (int)(sizeof(Segment) / sizeof(int4)); i += blockDim.x) dst[i] = __ldcg(src + i);
            } else if (tid == 0) {
                seg.P = P0;
                seg.A = A0;
            }
            __syncthreads();
            cur = sj;
            stage_tables<LT, XT>(seg.P, make_layout<LT, XT, LU_SMEM>(seg.P, seg.A, dyn));
            __syncthreads();
        }
        const int first = queue ? qjob.first : (multi ? M.job_first[job] : A0.job_first[job]);
        const int count = queue ? qjob.count : (multi ? M.job_count[job] : A0.job_count[job]);
        solve_job<LT, XT, LU_SMEM, REFINE, (MAXT <= 640)>(seg.P, seg.A, S, dyn, first, count, pr);
        __syncthreads();
        if constexpr (REFINE) {
            if (seg.A.fp64_inline) {
                if (tid == 0) {
                    int bad = 0;
                    for (int i = first; i < first + count; ++i) bad |= seg.A.errs[i] != 0;
                    S.job_failed = bad;
                }
                __syncthreads();
                if (S.job_failed) {
                    // the word after the job counter counts the instances re-solved in FP64; the
                    // re-solve starts afresh from the instance's start voltages
                    const int *its = seg.A.it_start;
                    const int vfo = seg.A.v0_from_out;
                    if (tid == 0) {
                        if (seg.A.job_counter != nullptr) atomicAdd(seg.A.job_counter + 1, count);
                        seg.A.it_start = nullptr;
                        seg.A.v0_from_out = 0;
                    }
                    __syncthreads();
                    fp64_rerun(seg.P, seg.A, S, dyn, first, count);
                    __syncthreads();
                    if (tid == 0) {
                        seg.A.it_start = its;
                        seg.A.v0_from_out = vfo;
                    }
                    // the FP64 solve vector covered them
                    stage_tables<LT, XT>(seg.P, make_layout<LT, XT, LU_SMEM>(seg.P, seg.A, dyn));
                    __syncthreads();
                }
            }
        }
        if constexpr (QUEUE) {
            if (tid == 0) signal_queue_job(M.q.done, qjob.slot, count);
        }
    }
    if (pr.on)
        for (int i = 0; i < kPhaseSlots; ++i) A0.phase_cycles[(size_t)blockIdx.x * kPhaseSlots + i] = pr.pc[i];
}

}  // namespace

// Raises a kernel's dynamic shared-memory limit to everything the device allows, once per
// kernel and device (launches then pass their own size; setting the attribute on every
// launch would make concurrent launches on other streams wait on the driver).
cudaError_t allow_max_smem(const void *fn) {
    static std::mutex mu;
    static std::set<std::pair<const void *, int>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (done.count({fn, dev})) return cudaSuccess;
    int optin = 0;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    if (e != cudaSuccess) return e;
    done.insert({fn, dev});
    return cudaSuccess;
}

namespace {

// DC power flow of a batch (BaseDCAlgo::compute_pf, src/powerflow_algorithm/BaseDCAlgo.tpp:
// 86-175), FP64, one CTA per instance: B from the real parts of the instance's Ybus (overrides
// applied), right-hand side Re(Sbus) at the non-slack buses, refactorisation with the forward
// substitution fused, backward substitution; the angles are shifted by the slack's start angle,
// the magnitudes are the start magnitudes.  A non-finite solution or one with |theta| >= 1e6 is
// SolverSolve (:115-123): zero voltages.  One linear solve: iters = 1.
template <bool LU_SMEM>
__global__ void __launch_bounds__(512, 1) dc_batch_kernel(const DevPlan P, const BatchArgs A) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ Shared S;
    const int tid = threadIdx.x;
    const int n = P.n, m = P.m;
    const Layout<double, double> L = make_layout<double, double, LU_SMEM>(P, A, dyn);
    stage_tables<double, double>(P, L);
    __syncthreads();
    double *x = L.x, *lu = L.lu;
    Trace tr{nullptr, 0, 0};
    for (;;) {
        if (tid == 0) S.job = atomicAdd(A.job_counter, 1);
        __syncthreads();
        const int job = S.job;
        __syncthreads();
        if (job >= A.njobs) break;
        const int first = A.job_first[job], count = A.job_count[job];
        for (int inst = first; inst < first + count; ++inst) {
            if (tid == 0) {
                int k0 = 0, k1 = 0;
                if (A.ovr_ptr) {
                    k0 = A.ovr_ptr[inst];
                    k1 = A.ovr_ptr[inst + 1];
                }
                S.novr = k1 - k0 > kMaxOverrides ? -1 : k1 - k0;  // -1: too many to stage
                S.piv_err = 0;
            }
            __syncthreads();
            if (tid < S.novr) {
                const int k0 = A.ovr_ptr[inst];
                S.opos[tid] = A.ovr_pos[k0 + tid];
                S.oval[tid] = A.ovr_val[k0 + tid];
            }
            __syncthreads();
            if (S.novr < 0) {
                // more Ybus overrides than the kernel stages: not computed (start voltages out)
                const double2 *v0 = A.V0 + (long long)inst * A.v0_stride;
                double2 *vo = out_row(A, inst, n);
                for (int b = tid; b < n; b += blockDim.x) vo[b] = A.zero_failed ? make_double2(0.0, 0.0) : v0[b];
                if (tid == 0) {
                    A.iters[inst] = 0;
                    A.errs[inst] = 8;  // NotInitError
                }
                __syncthreads();
                continue;
            }
            for (int p = tid; p < P.nnzY; p += blockDim.x) {
                const int t = P.ytarget[p].x;
                if (t >= 0) lu[t] = ybus_value(P, S, p).x;
            }
            for (int i = tid; i < P.nfill; i += blockDim.x) lu[P.fillpos[i]] = 0.0;
            const double2 *Sb = A.Sbus + (long long)inst * A.sbus_stride;
            for (int b = tid; b < n; b += blockDim.x) {
                const int ip = P.xP[b];
                if (ip >= 0) x[ip] = Sb[b].x;
            }
            __syncthreads();
            run_lu_program<double, double, LU_SMEM, false>(packed_ops<LU_SMEM>(P, P.fac_cops), P.fac_ops, L.sb_fac, L.sw_fac,
                                                           P.fac_nph, m, P.lu_offset, lu, x, tr);
            check_pivots<double>(P, S, lu);
            int err = 0;
            if (S.piv_err) {
                err = 6;  // SolverReFactor
            } else {
                run_lu_program<double, double, LU_SMEM, true>(packed_ops<LU_SMEM>(P, P.bwd_cops), P.bwd_ops, L.sb_bwd,
                                                              L.sw_bwd, P.bwd_nph, m, P.lu_offset, lu, x, tr);
                scale_by_pivots<double, double>(P, S, lu, x);
                double lmax = 0.0;
                int lbad = 0;
                for (int k = tid; k < m; k += blockDim.x) {
                    lmax = fmax(lmax, fabs(x[k]));
                    lbad |= !isfinite(x[k]);
                }
                double nrm;
                int bad;
                block_norm(S, lmax, lbad, nrm, bad);
                if (bad || nrm >= 1e6) err = 7;  // SolverSolve
            }
            const double2 *v0 = A.V0 + (long long)inst * A.v0_stride;
            double2 *vo = out_row(A, inst, n);
            const double2 vs = v0[P.slack0];
            const double a0 = atan2(vs.y, vs.x);
            for (int b = tid; b < n; b += blockDim.x) {
                double2 v = make_double2(0.0, 0.0);
                if (err == 0) {
                    const int ia = P.xVa[b];
                    const double va = (ia >= 0 ? x[ia] : 0.0) + a0;
                    const double vm = cabs2(v0[b]);
                    double sn, cs;
                    sincos(va, &sn, &cs);
                    v = make_double2(vm * cs, vm * sn);
                }
                vo[b] = v;
            }
            if (tid == 0) {
                A.iters[inst] = err == 0 ? 1 : 0;
                A.errs[inst] = err;
            }
            __syncthreads();
        }
    }
}

// Fast decoupled power flow of a batch (BaseFDPFAlgo::compute_pf, src/powerflow_algorithm/
// BaseFDPFAlgo.tpp:11-173, with has_converged, BaseFDPFAlgo.hpp:118-170), FP64, one CTA per
// instance.  B' (over pvpq) and B'' (over pq) were factorised when the plan was built and do
// not change between instances (the reference's batch computers keep the base factors for
// every contingency and step); each CTA copies both factors into its shared memory once when
// they fit, else reads them from global memory (one copy, L2 resident).  An iteration:
//   P half-step  dVa = B'^-1 P, Va[pvpq] -= dVa, t = exp(j Va), V = Vm t, (Vm, Va) = (|V|, arg V)
//   Q half-step  dVm = B''^-1 Q, Vm[pq] -= dVm, V = Vm t, (Vm, Va) = (|V|, arg V)
// each followed by the mismatch  mis = (V conj(Ybus V) - Sbus + slack_absorbed w) / Vm,
// P = Re(mis)[pvpq], Q = Im(mis)[pq], converged when max(|P|, |Q|) < tol, InifiniteValue when
// any bus's mis is not finite; slack_absorbed = Re(sum Sbus), the reference's start value,
// which its FDPF never updates.
// Only one of P and Q is needed at a time (P before a B' solve, Q before a B'' solve), so the
// two systems share one solve vector; with the factors in shared memory the index space is
// x | LU(B') | LU(B''), each system's packed operations addressing its LU at its lu_offset.
struct FdpfLayout {
    double *x[2];         // the shared solve vector (both entries equal)
    // factors in shared memory: their values, and the programs' phase bounds and widths
    const double *lu[2];
    int *sbf[2], *swf[2], *sbb[2], *swb[2];
    double2 *V, *T;       // voltages, exp(j Va) of the last P half-step
    double *Vm, *Va;
};

__host__ __device__ __forceinline__ size_t fdpf_region_bytes(const DevPlan &B0, const DevPlan &B1, bool lu_in_smem) {
    const size_t e0 = lu_in_smem ? (size_t)B0.lu_offset + (size_t)B0.nnzLU : (size_t)B0.m + 1;
    const size_t e1 = lu_in_smem ? (size_t)B1.lu_offset + (size_t)B1.nnzLU : (size_t)B1.m + 1;
    const size_t e = e0 > e1 ? e0 : e1;
    return (e * sizeof(double) + 15) & ~(size_t)15;
}

// B: the two systems' plans (in shared memory)
template <bool LU_SMEM>
__device__ __forceinline__ FdpfLayout fdpf_layout(const DevPlan &P, const DevPlan *B, const BatchArgs &A,
                                                  unsigned char *dyn) {
    FdpfLayout L;
    double *x = reinterpret_cast<double *>(dyn);
    for (int k = 0; k < 2; ++k) {
        L.x[k] = x;
        L.lu[k] = LU_SMEM ? x + B[k].lu_offset : nullptr;
    }
    if constexpr (LU_SMEM) {
        int *t = reinterpret_cast<int *>(dyn + fdpf_region_bytes(B[0], B[1], true));
        for (int k = 0; k < 2; ++k) {
            L.sbf[k] = t;
            t += B[k].fwd_nph + 1;
            L.sbb[k] = t;
            t += B[k].bwd_nph + 1;
            L.swf[k] = t;
            t += B[k].fwd_nph;
            L.swb[k] = t;
            t += B[k].bwd_nph;
        }
    }
    unsigned char *slab = A.scratch + (size_t)blockIdx.x * (size_t)A.slab_bytes;
    L.V = reinterpret_cast<double2 *>(slab);
    L.T = L.V + P.n;
    L.Vm = reinterpret_cast<double *>(L.T + P.n);
    L.Va = L.Vm + P.n;
    return L;
}

// A substitution program over constant factors: every thread runs its operation of every row (rows are
// padded, so there is no bounds test), loaded kPushAhead rows ahead and across phases.  The loads are
// unconditional: one behind a test is merged with the register's old value, which waits for it.
// The factors' quotients are formed once per plan, so an operation is 12 streamed bytes and one
// multiply-add; reading both factors and dividing (16-byte operations, a scattered load of each
// factor, the quotient's chain) N-1 batches took 68.1 ms (2,848 buses, BX) against 27.8 ms now, 1,354 buses
// 13.2 -> 8.5 ms, 118 buses 1.40 -> 0.51 ms (this change alone, CUDA events around one launch).
__device__ __forceinline__ void run_pushes(const DevPushes R, double *v) {
    constexpr int A = kPushAhead;
    const unsigned *pi = R.idx + threadIdx.x;
    const double *pc = R.coef + threadIdx.x;
    const int bd = blockDim.x, rows = R.rows;
    unsigned qi[A];
    double qc[A];
#pragma unroll
    for (int i = 0; i < A; ++i) {
        qi[i] = __ldg(pi + i * bd);
        qc[i] = __ldg(pc + i * bd);
    }
    unsigned m = __ldg(R.mask), mn = __ldg(R.mask + (rows > 32 ? 1 : 0));
    for (int r = 0; r < rows; r += A) {
        pi += A * bd;
        pc += A * bd;
#pragma unroll
        for (int i = 0; i < A; ++i) {
            v[qi[i] & 0xffffu] -= qc[i] * v[qi[i] >> 16];
            qi[i] = __ldg(pi + i * bd);
            qc[i] = __ldg(pc + i * bd);
            if (m & 1u) __syncthreads();
            m >>= 1;
        }
        if (((r + A) & 31) == 0) {
            m = mn;
            mn = __ldg(R.mask + min((r + A) / 32 + 1, rows / 32));
        }
    }
}

// B x = b for one decoupled system: forward and backward programs over the constant factors,
// then the division by the pivots (the backward program keeps z undivided).
template <bool LU_SMEM>
__device__ __forceinline__ void fdpf_solve(const DevPlan &B, const FdpfLayout &L, int k, Trace &tr) {
    double *x = L.x[k];
    if constexpr (LU_SMEM) {
        double *lu = const_cast<double *>(L.lu[k]);  // read only: substitutions do not write the LU
        run_lu_program<double, double, true, true>(B.fwd_cops, B.fwd_ops, L.sbf[k], L.swf[k], B.fwd_nph, B.m, B.lu_offset,
                                                   lu, x, tr);
        run_lu_program<double, double, true, true>(B.bwd_cops, B.bwd_ops, L.sbb[k], L.swb[k], B.bwd_nph, B.m, B.lu_offset,
                                                   lu, x, tr);
    } else {
        run_pushes(B.push[0], x);
        run_pushes(B.push[1], x);
    }
    for (int i = threadIdx.x; i < B.m; i += blockDim.x) x[i] = lu_div(x[i], __ldg(B.dval + i));
    __syncthreads();
}

// mis = (V conj(Ybus V) - Sbus + slack_absorbed w) / Vm: P into x at xP (which 0, for the next
// B' solve) or Q into x at xQ (which 1, for the next B'' solve); returns max(|P|, |Q|) and "some
// bus's mis is not finite" to every thread.
__device__ void fdpf_mismatch(const DevPlan &P, Shared &S, const double2 *__restrict__ V,
                              const double *__restrict__ Vm, const double2 *__restrict__ Sbus, double *x, int which,
                              double &norm, int &bad) {
    double lmax = 0.0;
    int lbad = 0;
    const double sa = S.slack_absorbed;
    for (int slot = threadIdx.x; slot < P.row_slots; slot += blockDim.x) {
        const int r = P.row_bus[slot];
        if (r < 0) continue;
        const double2 vr = V[r], sb = Sbus[r];
        const double2 s = ybus_row<false>(P, S, V, slot, r, vr, P.row_slice[slot >> 5], nullptr, nullptr);
        double mr = vr.x * s.x + vr.y * s.y - sb.x;  // V * conj(I) - S + slack_absorbed * w
        double mi = vr.y * s.x - vr.x * s.y - sb.y;
        mr += sa * P.w[r];
        const double vm = Vm[r];
        mr = lu_div(mr, vm);
        mi = lu_div(mi, vm);
        lbad |= !isfinite(mr) || !isfinite(mi);
        const int ip = P.dg_eq[slot].x, iq = P.dg_eq[slot].y;
        if (ip >= 0) {
            if (which == 0) x[ip] = mr;
            lmax = fmax(lmax, fabs(mr));
        }
        if (iq >= 0) {
            if (which == 1) x[iq] = mi;
            lmax = fmax(lmax, fabs(mi));
        }
    }
    block_norm(S, lmax, lbad, norm, bad);
}

// MAXT / MINB: launch bounds.  With the factors in global memory (read by every CTA of an SM
// through L1) small CTAs, many per SM, hide the latency of the substitution phases.
template <bool LU_SMEM, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) fdpf_batch_kernel(const DevPlan P0, const DevPlan B0, const DevPlan B1,
                                                                const BatchArgs A) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ Shared S;
    // the three plans in shared memory: indexed by system without copies of kernel parameters
    __shared__ __align__(16) DevPlan sp[3];
    const int tid = threadIdx.x;
    if (tid == 0) {
        sp[0] = P0;
        sp[1] = B0;
        sp[2] = B1;
    }
    __syncthreads();
    const DevPlan &P = sp[0];
    const DevPlan *B = sp + 1;
    const int n = P.n;
    const FdpfLayout L = fdpf_layout<LU_SMEM>(P, B, A, dyn);
    {
        for (int k = 0; k < 2; ++k) {
            const DevPlan &b = B[k];
            if constexpr (LU_SMEM) {
                for (int i = tid; i <= b.fwd_nph; i += blockDim.x) L.sbf[k][i] = b.fwd_base[i];
                for (int i = tid; i <= b.bwd_nph; i += blockDim.x) L.sbb[k][i] = b.bwd_base[i];
                for (int i = tid; i < b.fwd_nph; i += blockDim.x) L.swf[k][i] = b.fwd_width[i];
                for (int i = tid; i < b.bwd_nph; i += blockDim.x) L.swb[k][i] = b.bwd_width[i];
                for (int i = tid; i < b.nnzLU; i += blockDim.x) L.x[k][b.lu_offset + i] = b.luval[i];
            } else if (tid == 0) {
                L.x[k][b.m] = 0.0;  // the padding operations' element (later any value of the other system)
            }
        }
    }
    __syncthreads();
    double2 *V = L.V, *T = L.T;
    double *Vm = L.Vm, *Va = L.Va;
    Trace tr{nullptr, 0, 0};
    for (;;) {
        if (tid == 0) S.job = atomicAdd(A.job_counter, 1);
        __syncthreads();
        const int job = S.job;
        __syncthreads();
        if (job >= A.njobs) break;
        const int first = A.job_first[job], count = A.job_count[job];
        for (int step = 0; step < count; ++step) {
            const int inst = first + step;
            const double2 *Sb = A.Sbus + (long long)inst * A.sbus_stride;
            if (step == 0 || !A.chain) {
                const double2 *v0 = A.V0 + (long long)inst * A.v0_stride;
                for (int b = tid; b < n; b += blockDim.x) V[b] = v0[b];
            }
            for (int b = tid; b < n; b += blockDim.x) {
                const double2 v = V[b];
                Vm[b] = cabs2(v);
                Va[b] = atan2(v.y, v.x);
            }
            if (tid == 0) {
                int k0 = 0, k1 = 0;
                if (A.ovr_ptr) {
                    k0 = A.ovr_ptr[inst];
                    k1 = A.ovr_ptr[inst + 1];
                }
                S.novr = k1 - k0 > kMaxOverrides ? -1 : k1 - k0;  // -1: too many to stage
            }
            __syncthreads();
            if (tid < S.novr) {
                const int k0 = A.ovr_ptr[inst];
                stage_override(P, S, tid, A.ovr_pos[k0 + tid], A.ovr_val[k0 + tid]);
            }
            double ls = 0.0;
            for (int b = tid; b < n; b += blockDim.x) ls += Sb[b].x;
            const double tot = block_sum(S, ls);  // contains barriers
            if (tid == 0) S.slack_absorbed = tot;
            __syncthreads();
            if (S.novr < 0) {
                // more Ybus overrides than the kernel stages: not computed (start voltages out)
                double2 *vo = out_row(A, inst, n);
                for (int b = tid; b < n; b += blockDim.x) vo[b] = A.zero_failed ? make_double2(0.0, 0.0) : V[b];
                if (tid == 0) {
                    A.iters[inst] = 0;
                    A.errs[inst] = 8;  // NotInitError
                }
                __syncthreads();
                if (A.chain) {
                    for (int s2 = step + 1 + tid; s2 < count; s2 += blockDim.x) {
                        A.iters[first + s2] = 0;
                        A.errs[first + s2] = 8;
                    }
                    break;
                }
                continue;
            }
            double norm;
            int bad;
            fdpf_mismatch(P, S, V, Vm, Sb, L.x[0], 0, norm, bad);
            bool conv = !bad && norm < A.tol;
            int it = 0, err = 0;
            while (!conv && it < A.max_iter) {
                ++it;
                // P half-step
                fdpf_solve<LU_SMEM>(B[0], L, 0, tr);
                for (int b = tid; b < n; b += blockDim.x) {
                    double va = Va[b];
                    const int ia = P.xVa[b];
                    if (ia >= 0) va -= L.x[0][ia];
                    double sn, cs;
                    sincos(va, &sn, &cs);
                    T[b] = make_double2(cs, sn);
                    const double vm = Vm[b];
                    const double2 v = make_double2(vm * cs, vm * sn);
                    V[b] = v;
                    // |V| and arg(V) only where they differ from the updated values (voltage_update)
                    if (!(vm >= 0.0 && fabs(va) <= kPi)) {
                        Vm[b] = cabs2(v);
                        va = atan2(v.y, v.x);
                    }
                    Va[b] = va;
                }
                __syncthreads();
                fdpf_mismatch(P, S, V, Vm, Sb, L.x[0], 1, norm, bad);
                if (bad) {
                    err = 3;  // InifiniteValue
                    break;
                }
                if (norm < A.tol) {
                    conv = true;
                    break;
                }
                // Q half-step
                fdpf_solve<LU_SMEM>(B[1], L, 1, tr);
                for (int b = tid; b < n; b += blockDim.x) {
                    double vm = Vm[b];
                    const int im = P.xVm[b];
                    if (im >= 0) vm -= L.x[1][im];
                    const double2 t = T[b];
                    const double2 v = make_double2(vm * t.x, vm * t.y);
                    V[b] = v;
                    if (!(vm >= 0.0)) {  // negative (or not finite): re-derived, with the angle turned
                        vm = cabs2(v);
                        Va[b] = atan2(v.y, v.x);
                    }
                    Vm[b] = vm;
                }
                __syncthreads();
                fdpf_mismatch(P, S, V, Vm, Sb, L.x[0], 0, norm, bad);
                if (bad) {
                    // the reference notices the error after the next iteration's B' solve
                    err = 3;
                    if (it < A.max_iter) ++it;
                    break;
                }
                conv = norm < A.tol;
            }
            if (!conv && err == 0) err = 2;  // TooManyIterations
            double2 *vo = out_row(A, inst, n);
            const bool zero = A.zero_failed && err != 0;
            for (int b = tid; b < n; b += blockDim.x) vo[b] = zero ? make_double2(0.0, 0.0) : V[b];
            if (tid == 0) {
                A.iters[inst] = it;
                A.errs[inst] = err;
            }
            __syncthreads();
            if (A.chain && err != 0) {
                // the reference stops a time series at its first divergence
                for (int s2 = step + 1 + tid; s2 < count; s2 += blockDim.x) {
                    A.iters[first + s2] = 0;
                    A.errs[first + s2] = 8;  // NotInitError: not computed
                }
                break;
            }
        }
        __syncthreads();
    }
}

template <typename LT, typename XT, bool SM, bool RF, bool Q, int MAXT>
cudaError_t launch_variant_t(const DevPlan &P, const BatchArgs &A, const MultiArgs &M, int threads, int grid,
                             size_t smem, cudaStream_t st) {
    cudaError_t e = allow_max_smem(reinterpret_cast<const void *>(nr_batch_kernel<LT, XT, SM, RF, Q, MAXT>));
    if (e != cudaSuccess) return e;
    nr_batch_kernel<LT, XT, SM, RF, Q, MAXT><<<grid, threads, smem, st>>>(P, A, M);
    return cudaGetLastError();
}

// the variant of the smallest launch bound (512, 640, 768) that covers `threads`
template <typename LT, typename XT, bool SM, bool RF, bool Q>
cudaError_t launch_variant_q(const DevPlan &P, const BatchArgs &A, const MultiArgs &M, int threads, int grid,
                             size_t smem, cudaStream_t st) {
    if (threads > 768) return cudaErrorInvalidValue;
    if (threads > 640) return launch_variant_t<LT, XT, SM, RF, Q, 768>(P, A, M, threads, grid, smem, st);
    if (threads > 512) return launch_variant_t<LT, XT, SM, RF, Q, 640>(P, A, M, threads, grid, smem, st);
    return launch_variant_t<LT, XT, SM, RF, Q, 512>(P, A, M, threads, grid, smem, st);
}

template <typename LT, typename XT, bool SM, bool RF>
cudaError_t launch_variant(const DevPlan &P, const BatchArgs &A, const MultiArgs &M, int threads, int grid,
                           size_t smem, cudaStream_t st) {
    if (M.q.jobs != nullptr) return launch_variant_q<LT, XT, SM, RF, true>(P, A, M, threads, grid, smem, st);
    return launch_variant_q<LT, XT, SM, RF, false>(P, A, M, threads, grid, smem, st);
}

template <typename LT, typename XT, bool SM, bool RF>
int occupancy_variant(int threads, size_t smem) {
    int nb = 0;
    if (threads > 768) return 0;
    const void *fn = threads > 640   ? reinterpret_cast<const void *>(nr_batch_kernel<LT, XT, SM, RF, false, 768>)
                     : threads > 512 ? reinterpret_cast<const void *>(nr_batch_kernel<LT, XT, SM, RF, false, 640>)
                                     : reinterpret_cast<const void *>(nr_batch_kernel<LT, XT, SM, RF, false, 512>);
    if (allow_max_smem(fn) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, smem) != cudaSuccess) return 0;
    return nb;
}

// The reference's Jacobian (dS/dVa, dS/d|V|) at V, in J order: a thread per row slot, its row product
// for the diagonal, then the entries.  A kernel of its own over the whole GPU: written by
// the one CTA of a single power flow in every iteration it took 20k cycles a time.
__global__ void jacobian_values_kernel(const DevPlan P, const double2 *__restrict__ V, double *__restrict__ Jout) {
    for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < P.row_slots; slot += gridDim.x * blockDim.x) {
        const int r = P.row_bus[slot];
        if (r < 0) continue;
        const int2 sl = P.row_slice[slot >> 5];
        const int e0 = sl.x + (slot & 31);
        const double2 vr = V[r];
        double2 s = cmul(P.dg_val[slot], vr);
        const double2 td = cmul(cconj(s), vr);
        for (int u = 0; u <= sl.y; ++u) {
            // the off-diagonal entries, then the diagonal (whose value needs the row's sum)
            const bool diag = u == sl.y;
            const int e = e0 + 32 * u, p = diag ? P.dg_pos[slot] : P.off_pos[e], c = diag ? r : P.off_col[e];
            if (p < 0) continue;
            const double2 vc = V[c];
            double2 t = td, d = make_double2(0.0, 0.0);
            if (diag) {
                d = cmul(cconj(s), vr);
            } else {
                const double2 b = cmul(P.off_val[e], vc);
                s.x += b.x;
                s.y += b.y;
                t = cmul(cconj(b), vr);
            }
            double dvar, dvai;
            double2 dvm;
            dsbus(t, d, dvar, dvai, dvm);
            const double vm = cabs2(vc);
            const int4 j = P.yjpos[p];
            if (j.x >= 0) Jout[j.x] = dvar;
            if (j.y >= 0) Jout[j.y] = dvai;
            if (j.z >= 0) Jout[j.z] = dvm.x / vm;
            if (j.w >= 0) Jout[j.w] = dvm.y / vm;
        }
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.nconst; i += gridDim.x * blockDim.x)
        Jout[P.cjpos[i]] = P.cval[i];
}

// Ybus values (storage order) into Rx and the row slots.
__global__ void set_ybus_kernel(const double2 *__restrict__ src, const int *__restrict__ of_csr, int nnz,
                                double2 *__restrict__ Rx, double2 *__restrict__ off, double2 *__restrict__ dg) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += gridDim.x * blockDim.x) {
        const double2 y = src[p];
        if (Rx != src) Rx[p] = y;
        if (of_csr != nullptr) {
            const int at = of_csr[p];
            if (at >= 0) off[at] = y;
            else dg[-1 - at] = y;
        }
    }
}

// Result rows in case order: row c = the converged voltages of compact instance map[c], or
// zeros (islanded case, map[c] < 0, or an instance that did not converge).
__global__ void scatter_case_rows(const double2 *__restrict__ src, const int *__restrict__ errs,
                                  const int *__restrict__ map, int ncases, int n, double2 *__restrict__ dst) {
    const long long total = (long long)ncases * n;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), b = (int)(t - (long long)c * n);
        const int i = map[c];
        dst[t] = (i >= 0 && errs[i] == 0) ? src[(long long)i * n + b] : make_double2(0.0, 0.0);
    }
}

}  // namespace

cudaError_t launch_scatter_case_rows(const double2 *src, const int *errs, const int *map, int ncases, int n,
                                     double2 *dst, int num_sms, cudaStream_t st) {
    if (ncases <= 0) return cudaSuccess;
    scatter_case_rows<<<num_sms * 8, 256, 0, st>>>(src, errs, map, ncases, n, dst);
    return cudaGetLastError();
}

cudaError_t launch_jacobian_values(const DevPlan &P, const double2 *V, double *Jout, int num_sms, cudaStream_t st) {
    if (P.row_slots <= 0) return cudaSuccess;
    jacobian_values_kernel<<<std::min((P.row_slots + 63) / 64, num_sms * 8), 64, 0, st>>>(P, V, Jout);
    return cudaGetLastError();
}

cudaError_t launch_set_ybus(const DevPlan &P, const double2 *src, int num_sms, cudaStream_t st) {
    if (P.nnzY <= 0) return cudaSuccess;
    set_ybus_kernel<<<std::min((P.nnzY + 255) / 256, num_sms * 8), 256, 0, st>>>(
        src, P.row_slots > 0 ? P.row_of_csr : nullptr, P.nnzY, const_cast<double2 *>(P.Rx),
        const_cast<double2 *>(P.off_val), const_cast<double2 *>(P.dg_val));
    return cudaGetLastError();
}

size_t slab_bytes(const DevPlan &P, int lu_bytes, bool lu_in_smem) {
    size_t bus = bus_slab_bytes(P, lu_bytes);
    size_t lu = lu_in_smem ? 0 : (((size_t)P.nnzLU * lu_bytes + 255) & ~(size_t)255);
    // the dense tail block after the LU (global-memory LU plans only)
    size_t tail = lu_in_smem ? 0 : (((size_t)P.tail_k * (size_t)tail_ld(P.tail_k) * lu_bytes + 255) & ~(size_t)255);
    return bus + lu + tail;
}

size_t smem_bytes(const DevPlan &P, int lu_bytes, int x_bytes, bool lu_in_smem) {
    size_t xb = lu_in_smem ? (size_t)P.lu_offset * x_bytes : (((size_t)P.m * x_bytes + 15) & ~(size_t)15);
    size_t lb = lu_in_smem ? (((size_t)P.nnzLU * lu_bytes + 15) & ~(size_t)15) : 0;
    size_t bb = (size_t)(2 * (P.fac_nph + P.bwd_nph + P.fwd_nph) + 3) * sizeof(int);
    // staged operations of the narrow phases (make_layout places them after the tables)
    const size_t nb = P.nar_off[3] > 0 ? (((xb + lb + bb + 7) & ~(size_t)7) - (xb + lb + bb)) + (size_t)P.nar_off[3] * 8 : 0;
    // the dense tail's staging area, 16-byte aligned after the tables (global-memory LU)
    if (!lu_in_smem && P.tail_k > 0)
        return ((xb + lb + bb + nb + 7) & ~(size_t)7) + 16 + tail_smem_bytes(P.tail_k, P.tail_w, lu_bytes);
    return xb + lb + bb + nb;
}

template <bool SM>
cudaError_t launch_dc_variant(const DevPlan &P, const BatchArgs &A, int threads, int grid, size_t smem,
                              cudaStream_t st) {
    cudaError_t e = allow_max_smem(reinterpret_cast<const void *>(dc_batch_kernel<SM>));
    if (e != cudaSuccess) return e;
    dc_batch_kernel<SM><<<grid, threads, smem, st>>>(P, A);
    return cudaGetLastError();
}

template <bool SM, int MAXT, int MINB>
cudaError_t launch_fdpf_variant(const DevPlan &P, const DevPlan &B0, const DevPlan &B1, const BatchArgs &A,
                                int threads, int grid, size_t smem, cudaStream_t st) {
    cudaError_t e = allow_max_smem(reinterpret_cast<const void *>(fdpf_batch_kernel<SM, MAXT, MINB>));
    if (e != cudaSuccess) return e;
    fdpf_batch_kernel<SM, MAXT, MINB><<<grid, threads, smem, st>>>(P, B0, B1, A);
    return cudaGetLastError();
}

// the kernel variant of a configuration: factors in shared memory (512 threads, 1 CTA per SM),
// or in global memory with 128-thread CTAs, 4 (registers unconstrained) or 8 (64 registers) per
// SM, or wider CTAs
const void *fdpf_kernel(bool lu_in_smem, int threads, int ctas_per_sm) {
    if (lu_in_smem) return reinterpret_cast<const void *>(fdpf_batch_kernel<true, 512, 1>);
    if (threads <= 128 && ctas_per_sm > 4) return reinterpret_cast<const void *>(fdpf_batch_kernel<false, 128, 8>);
    if (threads <= 128) return reinterpret_cast<const void *>(fdpf_batch_kernel<false, 128, 4>);
    return reinterpret_cast<const void *>(fdpf_batch_kernel<false, 512, 1>);
}

cudaError_t launch_fdpf_batch(const DevPlan &P, const DevPlan &B0, const DevPlan &B1, const BatchArgs &A,
                              int threads, int ctas_per_sm, int grid, size_t smem, cudaStream_t stream) {
    if (A.lu_in_smem) return launch_fdpf_variant<true, 512, 1>(P, B0, B1, A, threads, grid, smem, stream);
    if (threads <= 128 && ctas_per_sm > 4)
        return launch_fdpf_variant<false, 128, 8>(P, B0, B1, A, threads, grid, smem, stream);
    if (threads <= 128) return launch_fdpf_variant<false, 128, 4>(P, B0, B1, A, threads, grid, smem, stream);
    return launch_fdpf_variant<false, 512, 1>(P, B0, B1, A, threads, grid, smem, stream);
}

size_t fdpf_smem_bytes(const DevPlan &B0, const DevPlan &B1, bool lu_in_smem) {
    size_t b = fdpf_region_bytes(B0, B1, lu_in_smem);
    if (!lu_in_smem) return b;
    for (const DevPlan *B : {&B0, &B1}) b += (size_t)(2 * (B->fwd_nph + B->bwd_nph) + 2) * sizeof(int);
    return (b + 15) & ~(size_t)15;
}

size_t fdpf_slab_bytes(const DevPlan &P) { return ((size_t)P.n * 48 + 255) & ~(size_t)255; }

int fdpf_occupancy(bool lu_in_smem, int threads, int ctas_per_sm, size_t smem) {
    const void *fn = fdpf_kernel(lu_in_smem, threads, ctas_per_sm);
    int nb = 0;
    if (allow_max_smem(fn) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, smem) != cudaSuccess) return 0;
    return nb;
}

cudaError_t launch_nr_batch(const DevPlan &P, const BatchArgs &A, int precision, int threads, int grid,
                            size_t smem, cudaStream_t stream, const MultiArgs &M) {
    const bool sm = A.lu_in_smem != 0;
    if (P.dc) {
        if (M.segs != nullptr) return cudaErrorInvalidValue;  // DC plans run one plan per launch
        return sm ? launch_dc_variant<true>(P, A, threads, grid, smem, stream)
                  : launch_dc_variant<false>(P, A, threads, grid, smem, stream);
    }
    if (precision == 0) {
        return sm ? launch_variant<double, double, true, false>(P, A, M, threads, grid, smem, stream)
                  : launch_variant<double, double, false, false>(P, A, M, threads, grid, smem, stream);
    }
    if (A.refine)
        return sm ? launch_variant<float, float, true, true>(P, A, M, threads, grid, smem, stream)
                  : launch_variant<float, float, false, true>(P, A, M, threads, grid, smem, stream);
    return sm ? launch_variant<float, float, true, false>(P, A, M, threads, grid, smem, stream)
              : launch_variant<float, float, false, false>(P, A, M, threads, grid, smem, stream);
}

int nr_occupancy(int precision, bool lu_in_smem, bool refine, int threads, size_t smem) {
    if (precision == 0)
        return lu_in_smem ? occupancy_variant<double, double, true, false>(threads, smem)
                          : occupancy_variant<double, double, false, false>(threads, smem);
    if (refine)
        return lu_in_smem ? occupancy_variant<float, float, true, true>(threads, smem)
                          : occupancy_variant<float, float, false, true>(threads, smem);
    return lu_in_smem ? occupancy_variant<float, float, true, false>(threads, smem)
                      : occupancy_variant<float, float, false, false>(threads, smem);
}

}  // namespace l2g
