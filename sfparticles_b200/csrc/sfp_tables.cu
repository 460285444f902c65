// sfp_tables.cu -- the QED rate tables generated on the GPU (no counterpart
// kernel in the reference, which builds them with scipy on the CPU).
//
// Restates the reference's generators with their own algorithm, so that the
// tables reproduce its entries:
//   * rejection sampling (qed/rejection_sampling_tables.py:80-112): on a z
//     grid, int_Ai(z) = quad(Ai, z, inf) and Ai'(z);
//   * optical depth (qed/optical_depth_tables.py:136-198): per chi row the
//     total rate quad(P, 0, 1) and the cumulative row
//       integ[0] = quad(P, 0, delta_0),
//       integ[i] = integ[i-1] + P(delta_i) (delta_i - delta_{i-1}),
//     with the differential rate
//       photon: P(delta) = factor (int_Ai(z) + (2/z + chi_g sqrt z) Ai'(z)),
//               chi_g = delta chi_e, z = (chi_g / chi_e / (chi_e - chi_g))^(2/3);
//       pair:   P(delta) = factor (int_Ai(z) + (2/z - chi_g sqrt z) Ai'(z)),
//               chi_e = delta chi_g, z = (chi_g / chi_e / (chi_g - chi_e))^(2/3);
//     P(1) = 0, and int_Ai = Ai' = 0 from z = 108 on (the product's tables'
//     convention: their float64 values there are 0; the reference's scipy
//     returns NaN at z ~ 1e8, which leaves its low-chi pair rows NaN).
// quad is QUADPACK's QAGS / QAGI as scipy runs it (sfp_quadpack.h) and Ai,
// Ai' come from sfp_airy.h.  The grids (z, chi rows, log-spaced delta) and
// the rate prefactor are computed by the caller exactly as the reference
// computes them (numpy linspace / logspace, -alpha m c^2 / hbar) and passed
// in.  A warp per z point, a thread per (chi row, delta column), a block of 21
// warps per total rate.
#include <cuda_runtime.h>

#include <string>

#include "sfp.h"
#include "sfp_internal.h"
#include "sfp_table_math.h"

namespace {

using sfp_tab::RateFn;

// One quadrature inside another is a long serial chain: a total rate takes
// up to 50 bisections of the 21-point rule, each node a rate, each rate an
// integral of Ai by bisections of the 15-point rule, each node a continued
// fraction of tens of dependent divisions (a few microseconds).  With one
// thread per row that chain is the whole time (1.16 s for 96 photon rows,
// 192 threads on the GPU).  The nodes of one rule are independent, so
//   * a warp evaluates a rate: the two halves of a bisected interval are 30
//     nodes, one per lane (WarpAi);
//   * a block of 21 warps evaluates the outer rule, a node per warp (BlockRate).
// Every lane then adds the node values in the one-thread order
// (combine15 / combine21), so the bisections taken and the results are those
// of the one-thread code.  96 photon rows: 1.16 s -> 9.5 ms (totals 8.1 ms,
// still that chain; rates 1.9 ms, accumulation 0.03 ms).
struct WarpAi {};

// node of the 15-point rule that a lane evaluates: lane 0 (of its half warp)
// the centre, 2j + 1 / 2j + 2 the nodes centre -/+ hlgth xgk15(j); lane 15 idle
__device__ __forceinline__ double node15(double a, double b, int l) {
    const double centr = 0.5 * (a + b), hlgth = 0.5 * (b - a);
    if (l == 0 || l == 15) return centr;
    const double absc = hlgth * sfp_gk::xgk15((l - 1) >> 1);
    return (l & 1) ? centr - absc : centr + absc;
}

// each half warp combines its own interval's nodes
__device__ __forceinline__ void half_combine15(double fx, double a, double b, sfp_quad::RuleValue& v) {
    double fv1[7], fv2[7];
    const double fc = __shfl_sync(0xffffffffu, fx, 0, 16);
#pragma unroll
    for (int j = 0; j < 7; ++j) {
        fv1[j] = __shfl_sync(0xffffffffu, fx, 2 * j + 1, 16);
        fv2[j] = __shfl_sync(0xffffffffu, fx, 2 * j + 2, 16);
    }
    sfp_quad::combine15(fc, fv1, fv2, 0.5 * (b - a), v);
}

__device__ __forceinline__ void from_lane(const sfp_quad::RuleValue& v, int lane, sfp_quad::RuleValue& out) {
    out.result = __shfl_sync(0xffffffffu, v.result, lane);
    out.abserr = __shfl_sync(0xffffffffu, v.abserr, lane);
    out.resabs = __shfl_sync(0xffffffffu, v.resabs, lane);
    out.resasc = __shfl_sync(0xffffffffu, v.resasc, lane);
}

__device__ void rule_two(sfp_quad::Interval<true>, const WarpAi&, double bound, double a1, double b1, double a2,
                         double b2, sfp_quad::RuleValue& v1, sfp_quad::RuleValue& v2) {
    const int lane = threadIdx.x & 31;
    const double a = lane < 16 ? a1 : a2, b = lane < 16 ? b1 : b2;
    const double t = node15(a, b, lane & 15);
    sfp_quad::RuleValue v;
    half_combine15(sfp_quad::transformed(sfp_tab::AiFn{}, bound, t), a, b, v);
    from_lane(v, 0, v1);
    from_lane(v, 16, v2);
}
__device__ void rule_one(sfp_quad::Interval<true> tag, const WarpAi& f, double bound, double a, double b,
                         sfp_quad::RuleValue& v) {
    sfp_quad::RuleValue same;
    rule_two(tag, f, bound, a, b, a, b, v, same);
}

// a rate whose warp evaluates it together (every lane gets the value)
using WarpRate = sfp_tab::RateFnBy<WarpAi>;

constexpr int kNodes = 21;

// What the warps of a block share: the control warp (warp 0) runs the
// adaptive quadrature and asks for the nodes of one or two intervals; each
// warp evaluates node `warp` of them.
struct RateBoard {
    double a[2], b[2];
    int count;  // intervals asked for; 0 ends the block's work
    double f[2][kNodes];
};

struct BlockRate {
    WarpRate rate;
    RateBoard* board;
};

// the block's barrier: the control warp and the others arrive from different
// places of the code
__device__ __forceinline__ void board_sync() {
    asm volatile("barrier.sync 1, %0;" ::"n"(32 * kNodes) : "memory");
}

// node `w` of the 21-point rule: 0 the centre, 2j + 1 / 2j + 2 centre -/+ hlgth xgk21(j)
__device__ __forceinline__ void eval_nodes(const WarpRate& rate, RateBoard* B) {
    const int w = threadIdx.x >> 5;
    const int n = B->count;
    for (int k = 0; k < n; ++k) {
        const double centr = 0.5 * (B->a[k] + B->b[k]), hlgth = 0.5 * (B->b[k] - B->a[k]);
        double d = centr;
        if (w > 0) {
            const double absc = hlgth * sfp_gk::xgk21((w - 1) >> 1);
            d = (w & 1) ? centr - absc : centr + absc;
        }
        const double v = rate(d);
        if ((threadIdx.x & 31) == 0) B->f[k][w] = v;
    }
}

// control warp: ask, evaluate its own node with the others, combine
__device__ __forceinline__ void ask(const BlockRate& f, int n) {
    if (threadIdx.x == 0) f.board->count = n;
    __syncwarp();
    board_sync();  // the request is written
    if (n) {
        eval_nodes(f.rate, f.board);
        board_sync();  // every node is in
    }
}
__device__ __forceinline__ void board_combine21(const BlockRate& f, int k, sfp_quad::RuleValue& v) {
    const RateBoard* B = f.board;
    double fv1[10], fv2[10];
    for (int j = 0; j < 10; ++j) {
        fv1[j] = B->f[k][2 * j + 1];
        fv2[j] = B->f[k][2 * j + 2];
    }
    sfp_quad::combine21(B->f[k][0], fv1, fv2, 0.5 * (B->b[k] - B->a[k]), v);
}
__device__ void rule_one(sfp_quad::Interval<false>, const BlockRate& f, double, double a, double b,
                         sfp_quad::RuleValue& v) {
    if (threadIdx.x == 0) {
        f.board->a[0] = a;
        f.board->b[0] = b;
    }
    ask(f, 1);
    board_combine21(f, 0, v);
    __syncwarp();  // read before the next request
}
__device__ void rule_two(sfp_quad::Interval<false>, const BlockRate& f, double, double a1, double b1, double a2,
                         double b2, sfp_quad::RuleValue& v1, sfp_quad::RuleValue& v2) {
    if (threadIdx.x == 0) {
        f.board->a[0] = a1;
        f.board->b[0] = b1;
        f.board->a[1] = a2;
        f.board->b[1] = b2;
    }
    ask(f, 2);
    board_combine21(f, 0, v1);
    board_combine21(f, 1, v2);
    __syncwarp();
}

// a warp per z point
__global__ void k_rs_table(const double* __restrict__ z, long long n, double* __restrict__ int_ai,
                           double* __restrict__ aip) {
    const long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long stride = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = first; i < n; i += stride) {
        double ia, d;
        sfp_tab::airy_terms_by(WarpAi{}, z[i], ia, d);
        if ((threadIdx.x & 31) == 0) {
            int_ai[i] = ia;
            aip[i] = d;
        }
    }
}

// per chi row the total rate, then per chi row the first cumulative entry (few
// bisections): the long quadratures start first
__global__ void __launch_bounds__(32 * kNodes) k_od_totals(int kind, double factor, const double* __restrict__ chi,
                                                           long long n_chi, const double* __restrict__ delta,
                                                           double* __restrict__ total, double* __restrict__ first) {
    __shared__ RateBoard board;
    for (long long job = blockIdx.x; job < 2 * n_chi; job += gridDim.x) {
        const bool whole = job < n_chi;
        const long long r = whole ? job : job - n_chi;
        const BlockRate f{WarpRate{chi[r], factor, kind}, &board};
        if (threadIdx.x < 32) {
            const double v = sfp_quad::quad(f, 0.0, whole ? 1.0 : delta[0]);
            ask(f, 0);
            if (threadIdx.x == 0) (whole ? total : first)[r] = v;
        } else {
            for (;;) {
                board_sync();  // a request
                if (board.count == 0) break;
                eval_nodes(f.rate, &board);
                board_sync();  // its nodes
            }
        }
        board_sync();  // the board is free
    }
}

// P(delta_i) on every (row, column >= 1)
__global__ void k_od_rates(int kind, double factor, const double* __restrict__ chi, long long n_chi,
                           const double* __restrict__ delta, long long n_delta, double* __restrict__ rate) {
    const long long n = n_chi * n_delta;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long r = k / n_delta, i = k % n_delta;
        rate[k] = i == 0 ? 0.0 : RateFn{chi[r], factor, kind}(delta[i]);
    }
}

// the left-Riemann accumulation of each row, in the reference's order and
// rounding (product rounded, then added).  A warp per row: the products are
// formed and the sums stored 32 at a time, only the chain of additions is
// serial (each lane runs it, fed by shuffles).
__global__ void k_od_accumulate(const double* __restrict__ first, const double* __restrict__ delta, long long n_delta,
                                long long n_chi, double* __restrict__ cum) {
    const int lane = threadIdx.x & 31;
    const long long row0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long stride = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = row0; r < n_chi; r += stride) {
        double* row = cum + r * n_delta;  // holds P(delta_i) on entry
        double acc = first[r];
        if (lane == 0) row[0] = acc;
        for (long long i0 = 1; i0 < n_delta; i0 += 32) {
            const long long i = i0 + lane;
            const double p = i < n_delta ? __dmul_rn(row[i], __dsub_rn(delta[i], delta[i - 1])) : 0.0;
            double mine = 0.0;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                acc = __dadd_rn(acc, __shfl_sync(0xffffffffu, p, k));
                if (k == lane) mine = acc;
            }
            if (i < n_delta) row[i] = mine;
        }
    }
}

unsigned grid_of(long long n, int block) {
    long long g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > 65535) g = 65535;
    return (unsigned)g;
}

}  // namespace

extern "C" {

int sfp_table_rs(const double* z, int64_t n, double* int_ai, double* aip, void* stream) {
    if (n > 0 && (!z || !int_ai || !aip)) return sfp_set_error(SFP_EINVAL, "sfp_table_rs: NULL argument");
    if (n <= 0) return SFP_OK;
    k_rs_table<<<grid_of(n, 4), 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(z, n, int_ai, aip);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return sfp_set_error(SFP_ECUDA, std::string("sfp_table_rs: ") + cudaGetErrorString(e));
    return SFP_OK;
}

int sfp_table_od(int kind, double factor, const double* chi, int64_t n_chi, const double* delta, int64_t n_delta,
                 double* total, double* cumulative, double* first, void* stream) {
    if (kind != 0 && kind != 1) return sfp_set_error(SFP_EINVAL, "sfp_table_od: kind is 0 (photon) or 1 (pair)");
    if (n_chi > 0 && (!chi || !delta || !total || !cumulative || !first || n_delta < 1))
        return sfp_set_error(SFP_EINVAL, "sfp_table_od: NULL argument or empty delta grid");
    if (n_chi <= 0) return SFP_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    k_od_totals<<<grid_of(2 * n_chi, 1), 32 * kNodes, 0, s>>>(kind, factor, chi, n_chi, delta, total, first);
    k_od_rates<<<grid_of(n_chi * n_delta, 64), 64, 0, s>>>(kind, factor, chi, n_chi, delta, n_delta, cumulative);
    k_od_accumulate<<<grid_of(n_chi, 2), 64, 0, s>>>(first, delta, n_delta, n_chi, cumulative);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return sfp_set_error(SFP_ECUDA, std::string("sfp_table_od: ") + cudaGetErrorString(e));
    return SFP_OK;
}

}  // extern "C"
