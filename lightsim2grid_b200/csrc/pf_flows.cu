// Branch flows of a batch of power-flow results on the GPU.
//
// Restates BaseBatchSolverSynch::compute_amps_flows / compute_active_power_flows
// (src/batch_algorithm/BaseBatchSolverSynch.hpp:87-192) for AC results and
// ContingencyAnalysis::clean_flows (src/batch_algorithm/ContingencyAnalysis.cpp:237-250):
//   I_ft = conj(y_ff E_f + y_ft E_t),  S_ft = E_f I_ft
//   amps = |S_ft| sn_mva / (sqrt(3) |E_f| vn_kv(from))   [kA]
//   p    = Re(S_ft) sn_mva                                [MW]
// A branch out of service keeps 0 (the reference skips it in zeroed matrices); a result row
// whose voltages are all zero (a failed or islanded case) gives NaN amps (0 / 0) and 0 MW, as
// the reference's arithmetic does; clean_flows then sets each case's removed branches to 0
// where the value is finite.
//
// Layout: one CTA per result row; the row's outputs are written coalesced, its voltages are
// gathered per branch end, the per-branch data comes from L2.
#include "pf_flows.cuh"

#include <algorithm>
#include <cmath>

namespace l2g {
namespace {

__device__ __forceinline__ double2 cmulf(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Source row of result row r (-1: zero voltages).
__device__ __forceinline__ int source_row(const FlowArgs &A, int r) {
    int src = A.map ? A.map[r] : r;
    if (src >= 0 && A.errs && A.errs[src] != 0) src = -1;  // failed instance: zero voltages
    return src;
}

// Flows of one branch at one row's voltages ef (from) and et (to); ka = sn_mva / (sqrt(3) vn).  The
// reference divides |E_f I_ft| by |E_f|, which leaves |I_ft| (one square root instead of two and a
// division: FP64 arithmetic was a third of the time); a zero or non-finite E_f gives the NaN of that
// quotient.
__device__ __forceinline__ void branch_flow(double2 yf, double2 yt, double ka, double sn, double2 ef, double2 et,
                                            double &a, double &p) {
    const double2 i1 = cmulf(yf, ef), i2 = cmulf(yt, et);
    const double2 ift = make_double2(i1.x + i2.x, -(i1.y + i2.y));  // conj
    const double e2 = ef.x * ef.x + ef.y * ef.y;
    a = sqrt(ift.x * ift.x + ift.y * ift.y) * ka;
    if (!(e2 > 0.0 && isfinite(e2))) a = nan("");
    p = (ef.x * ift.x - ef.y * ift.y) * sn;
}

__device__ __forceinline__ double amps_factor(double sn, double vn) { return sn / (1.7320508075688772 * vn); }

// One CTA per row (grid-stride over rows); each thread takes every NT-th branch and gathers its two
// voltages through L1.  Bound by those random 16-byte gathers: the rows in work on an SM have to stay in
// its L1.  So rows of which six do not fit it (kWideRow) run two CTAs of 1024 threads per SM, smaller ones six
// of 256 (and 40 registers).  CUDA events around one launch, buffers flushed from L2, 4,500 rows, six narrow against
// two wide CTAs: 300 buses 22.5 and 36.9 us, 1600 96 and 113, 2000 120 and 127, 2200 135 and 131, 2848 182
// and 178, 4500 338 and 268, 6515 473 and 453; the 2848-bus N-1 results (3776 rows, 726 of them islanded):
// 137 and 143 us, 178 with eight CTAs of 256 and two square roots and a division per flow.
// Few rows are spread over more threads: with at most as many rows as wide CTAs run at once (30 rows of 1200 buses:
// 16.4 -> 10.2 us), or twice as many where a narrow CTA takes long (450 rows of 2000 buses: 25.6 -> 24.6 us, 600
// rows the same).  Two or four rows per CTA (branch data read once for all) and tiles of rows staged in shared memory
// were slower.
constexpr size_t kWideRow = 34000, kLongRow = 24000;
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) branch_flows_kernel(const FlowArgs A) {
    for (int row = blockIdx.x; row < A.nrows; row += gridDim.x) {
        const int src = source_row(A, row);
        const double2 *V = src >= 0 ? A.V + (long long)src * A.v_stride : nullptr;
        const int o0 = A.out_ptr ? A.out_ptr[row] : 0, o1 = A.out_ptr ? A.out_ptr[row + 1] : 0;
        const int first = o0 < o1 ? A.out_ids[o0] : -1;
        for (int k = threadIdx.x; k < A.nbr; k += NT) {
            double a = 0.0, p = 0.0;
            if (A.status == nullptr || __ldg(A.status + k)) {
                const int f = __ldg(A.from + k), t = __ldg(A.to + k);
                const double2 yf = __ldg(A.yff + k), yt = __ldg(A.yft + k);
                const double ka = A.amps ? amps_factor(A.sn_mva, __ldg(A.vn_kv_from + k)) : 0.0;
                const double2 ef = V ? __ldg(V + f) : make_double2(0.0, 0.0);
                const double2 et = V ? __ldg(V + t) : make_double2(0.0, 0.0);
                branch_flow(yf, yt, ka, A.sn_mva, ef, et, a, p);
            }
            // clean_flows: the branches removed in this row's case are 0 where finite
            bool out = first == k;
            for (int o = o0 + 1; o < o1; ++o) out |= A.out_ids[o] == k;
            if (out) {
                if (isfinite(a)) a = 0.0;
                if (isfinite(p)) p = 0.0;
            }
            const long long at = (long long)row * A.nbr + k;
            if (A.amps) __stcs(A.amps + at, a);
            if (A.p_mw) __stcs(A.p_mw + at, p);
        }
    }
}

}  // namespace

cudaError_t launch_branch_flows(const FlowArgs &A, int num_sms, cudaStream_t st) {
    if (A.nrows <= 0 || A.nbr <= 0) return cudaSuccess;
    const size_t row = (size_t)A.n * sizeof(double2);
    const bool few = A.nbr > 512 && A.nrows <= (row >= kLongRow ? 4 : 2) * num_sms;
    if (few || row >= kWideRow)
        branch_flows_kernel<1024, 2><<<std::min(A.nrows, num_sms * 2), 1024, 0, st>>>(A);
    else
        branch_flows_kernel<256, 6><<<std::min(A.nrows, num_sms * 6), 256, 0, st>>>(A);
    return cudaGetLastError();
}

}  // namespace l2g
