// dg_2d.cu -- the 2D quadrilateral path (Solver<2> with LagrangeQuad): the
// residual and RK stage on periodic meshes of parallelograms, FP64, and its C
// ABI (dg2d_* in dg_b200.h).
//
// Reference path replaced (the 2D instantiation of the 3D path's functions,
// citations relative to the reference root): Solver<2>::get_residual
// (src/solver/base.cpp:401-561) with evaluate_state (helpers.cpp:185-198),
// VolumeFluxesFunctor (flux_functors_impl.h:46-115), the grad-basis^T
// contraction (solver/tools.cpp:7-35), construct_face_states / the face flux
// functor / construct_flux_state (base.cpp:287-374,
// flux_functors_impl.h:168-264), the face lift (tools.cpp:38-63),
// mult_inv_mass_matrix (tools.cpp:124-139) and the RK4 / FE stage updates
// (stepper.cpp:23-142).
//
// Two launches per stage, or all steps of a call in one on small meshes (steps2d_kernel).
//   edge2d_kernel   every interior edge's numerical flux once: one thread per
//       (edge, Gauss point), the p + 1 threads of an edge in one warp.  Each holds
//       one edge node of both sides (the other basis functions vanish on the edge
//       exactly, so the traces equal the reference's dense B_f U term by term);
//       traces, and the lift onto either side's nodes (-F on the left, +F on the
//       right, times the edge weights), are sums over the warp's shuffles.
//   stage2d_kernel  a warp per E = 32 / (p+2) elements, no block barriers: the x
//       interpolation from the rows of a state to shared memory; one lane per
//       quadrature column: the y interpolation to its p+2 points, the Euler flux,
//       the contravariant transform and the y contraction in registers; the x
//       contraction of a row, its edges' lifts, and the fused RK / FE update
//       straight to global memory.  The 1D inverse mass is folded into the
//       contraction tables and the lifts (the residual output takes the plain ones).
// An edge that is no interior edge keeps a zero lift: it adds nothing, as in the
// reference, whose residual loops over the interior faces.
//
// Why: the kernel this replaces ran one task per value through shared memory, two
// loads to a multiply-add, and each edge's flux twice (512^2, p = 3: load/store and
// issue bound at 31 % of the FP64 pipe).  RK stage, HLLC, 256^2: p = 1 108 -> 23, p = 2
// 141 -> 42, p = 3 179 -> 60, p = 4 319 -> 103, p = 5 463 -> 135 us (both kernels); 64^2,
// p = 3 16.5 -> 9.8 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/dg_b200.h"
#include "../host/numerics.h"
#include "dg_small.cuh"

namespace dgi {
int fail(dg_ctx* c, int code, const std::string& msg);
unsigned* take_status_slot();
void give_status_slot(unsigned* p);
}

namespace d2 {

constexpr int kNS = 4;
constexpr int kMaxN = 6, kMaxM = 7;

constexpr int kSyncWord = 32, kStatusWords = 64;  // the status word, and a counter kSyncWord words on

enum Mode : int { kResidual = 0, kRK1 = 2, kRK2 = 3, kRK3 = 4, kRK4 = 5, kFE = 6 };
enum Status : unsigned { kRho = 1u, kPressure = 2u, kNaN = 4u, kHLLC = 8u };

// the order's tables of the edges (copied to shared memory by every CTA): trace
// of edge node m at edge point j of face f, its product with the 1D inverse mass
// (the lift of the update), and the weights
struct Tab {
    double FB[4 * kMaxN * kMaxN];  // [f][j][m]
    double MF[4 * kMaxN * kMaxN];
    double fw[kMaxN];
};

struct Geo {
    double jd[4];  // (ijac * djac)[d1][d2]
    double idj;    // 1 / djac
    double pad[3];
};

// one interior edge, by its left element: unit normal as the numerical flux wants
// it and |N|, both elements, and left face | right face << 2 | flip << 4 |
// (left orientation) << 5
struct Edge {
    double n[2];
    double nmag;
    int eL, eR;
    int code;
    int pad;
};

// an edge of a block's elements in the one-launch steps, and where in the block's shared
// memory the lift of either side goes (-1: an element of another block)
struct BlockEdge {
    int edge, oL, oR;
};

struct Args {
    const double* Us;
    double* out;
    const double* U0;
    double* acc;
    const Geo* geo;
    const Edge* edges;
    // one-launch steps: block b's edges are block_edges[i], block_first[b] <= i < block_first[b + 1]
    const BlockEdge* block_edges;
    const int* block_first;
    double* elift;  // [ne][4 faces][4][n], zero for edges that are no interior ones
    const Tab* tab;
    unsigned* status;
    int ne, nedge, mode, flux;
    double dt, gamma;
    // 1D tables: basis and weights at the volume points; contraction tables and end
    // columns of the inverse mass (plain ones and the identity's for the residual)
    double B[kMaxM * kMaxN], MB[kMaxM * kMaxN], MD[kMaxM * kMaxN], W[kMaxM];
    double ME[2][kMaxN];
};

constexpr int kEdgeThreads = 128;

__device__ __forceinline__ void load_tab(const Args& a, Tab& T)
{
    const double* src = reinterpret_cast<const double*>(a.tab);
    double* dst = reinterpret_cast<double*>(&T);
    for (int i = threadIdx.x; i < static_cast<int>(sizeof(Tab) / 8); i += blockDim.x) dst[i] = src[i];
    __syncthreads();
}

// the flux at this lane's point of edge ed, the N = P + 1 lanes from k N on holding the
// edge's points, times the point's weight
template <int P>
__device__ __forceinline__ void edge_flux(const Args& a, const double* Us, const Tab& T, const Edge& ed, double (&F)[kNS],
                                          unsigned& bad)
{
    constexpr int N = P + 1, NB = N * N;
    const int lane = threadIdx.x & 31, k = lane / N, j = lane - k * N;
    const int fL = ed.code & 3, fR = (ed.code >> 2) & 3, flip = (ed.code >> 4) & 1, mine = (ed.code >> 5) & 1;
    // edge node m of face f: basis index o + m s
    auto node = [](int f, int m) { return (f == 1 ? N - 1 : f == 2 ? (N - 1) * N : 0) + m * (f == 1 || f == 3 ? N : 1); };
    const int jr = flip ? N - 1 - j : j;           // the right side's point
    const int q = mine ? N - 1 - j : j;            // the face's quadrature point
    const double* pL = Us + static_cast<size_t>(ed.eL) * kNS * NB + node(fL, j);
    const double* pR = Us + static_cast<size_t>(ed.eR) * kNS * NB + node(fR, j);
    double uL[kNS], uR[kNS], tL[N], tR[N];
#pragma unroll
    for (int v = 0; v < kNS; ++v) {
        uL[v] = pL[v * NB];
        uR[v] = pR[v * NB];
    }
#pragma unroll
    for (int m = 0; m < N; ++m) {
        tL[m] = T.FB[(fL * N + j) * N + m];
        tR[m] = T.FB[(fR * N + jr) * N + m];
    }
    constexpr int s3[4] = {0, 1, 2, 4};
    double UL[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, UR[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int v = 0; v < kNS; ++v) {
        double sl = 0.0, sr = 0.0;
#pragma unroll
        for (int m = 0; m < N; ++m) {
            sl += tL[m] * __shfl_sync(0xffffffffu, uL[v], k * N + m);
            sr += tR[m] * __shfl_sync(0xffffffffu, uR[v], k * N + m);
        }
        UL[s3[v]] = sl;
        UR[s3[v]] = sr;
    }
    const double n3[3] = {ed.n[0], ed.n[1], 0.0};
    double F5[5];
    bad = 0;
    if (a.flux == DG_FLUX_HLLC) {
        if (!dgp::flux_hllc_n(a.gamma, UL, UR, n3, ed.nmag, F5)) bad = kHLLC;
    } else {
        dgp::flux_lax_friedrichs_sq(a.gamma, UL, UR, n3, ed.nmag, F5);
    }
    const double w = T.fw[q];
#pragma unroll
    for (int v = 0; v < kNS; ++v) F[v] = F5[s3[v]] * w;
}

// the edges of warp `warp` of nwarp, at the state Us
template <int P>
__device__ __forceinline__ void edge_phase(const Args& a, const double* Us, int mode, const Tab& T, int warp, int nwarp,
                                           unsigned& status)
{
    constexpr int N = P + 1, EPW = 32 / N;  // edges per warp
    const double* C = mode == kResidual ? T.FB : T.MF;
    const int lane = threadIdx.x & 31, k = lane / N, j = lane - k * N;
    for (int i0 = warp * EPW; i0 < a.nedge; i0 += nwarp * EPW) {
        const bool on = k < EPW && i0 + k < a.nedge;
        const Edge ed = a.edges[on ? i0 + k : a.nedge - 1];
        const int fL = ed.code & 3, fR = (ed.code >> 2) & 3, flip = (ed.code >> 4) & 1;
        double F[kNS];
        unsigned bad;
        edge_flux<P>(a, Us, T, ed, F, bad);
        if (on) status |= bad;
        double* oL = a.elift + (static_cast<size_t>(ed.eL) * 4 + fL) * kNS * N + j;
        double* oR = a.elift + (static_cast<size_t>(ed.eR) * 4 + fR) * kNS * N + j;
#pragma unroll
        for (int v = 0; v < kNS; ++v) {
            double sl = 0.0, sr = 0.0;
#pragma unroll
            for (int m = 0; m < N; ++m) {  // point m; node j of either side
                const double Fm = __shfl_sync(0xffffffffu, F[v], k * N + m);
                sl += C[(fL * N + m) * N + j] * Fm;
                sr += C[(fR * N + (flip ? N - 1 - m : m)) * N + j] * Fm;
            }
            if (on) {
                oL[v * N] = -sl;
                oR[v * N] = sr;
            }
        }
    }
}

template <int P>
__global__ void __launch_bounds__(kEdgeThreads) edge2d_kernel(const __grid_constant__ Args a)
{
    __shared__ Tab T;
    load_tab(a, T);
    unsigned status = 0;
    edge_phase<P>(a, a.Us, a.mode, T, (blockIdx.x * kEdgeThreads + threadIdx.x) >> 5, gridDim.x * kEdgeThreads / 32, status);
    if (status) atomicOr(a.status, status);
}

template <int P>
struct Cfg {
    static constexpr int N = P + 1, M = P + 2, NB = N * N;
    static constexpr int E = 32 / M;                    // elements per warp, one lane per column
    static constexpr int MS = M | 1;                    // odd row stride
    static constexpr int kA = 2 * kNS * N * MS;         // [d][v][j][qx]
    static constexpr int ES = kA + ((M - kA) % 16 + 16) % 16;  // = M modulo 16: the elements' columns follow one another over the banks
    static constexpr int kRows = E * kNS * N, R = (kRows + 31) / 32;
    static constexpr int kL = 4 * kNS * N;              // an element's lifts
    static constexpr size_t smem = sizeof(double) * ((static_cast<size_t>(E) * (ES + kL) + 2 * N + 1) / 2 * 2);
};

// the batches of warp `warp` of nwarp; sm: the warp's shared memory. With LATE other
// warps put the (only) batch's lifts there, and lifts_ready() returns true (false: give
// up) once they have.
template <int P, bool LATE, typename Ready>
__device__ __forceinline__ void stage_phase(const Args& a, const double* Us, const double* U0, double* out, int mode, double* sm,
                                            int warp, int nwarp, unsigned& status, Ready&& lifts_ready)
{
    using C = Cfg<P>;
    constexpr int N = C::N, M = C::M, NB = C::NB, E = C::E, MS = C::MS, ES = C::ES, R = C::R, kRows = C::kRows, MN = M * N;
    double* sL = sm;                      // [E][4][4][N]
    double* sA = sL + E * C::kL;          // [E][ES]: x-interpolated rows, then the y-contracted columns
    double* sM = sA + E * ES;             // [2][N]
    const int lane = threadIdx.x & 31;
    if (lane < 2 * N) sM[lane] = a.ME[lane / N][lane % N];
    const bool need_u0 = mode >= kRK1, need_acc = mode == kRK2 || mode == kRK3 || mode == kRK4;
    const bool put_acc = mode == kRK1 || mode == kRK2 || mode == kRK3, sum_acc = mode == kRK4;
    const double cu = mode == kRK1 || mode == kRK2 ? 0.5 : (sum_acc ? 1.0 / 6.0 : 1.0), ca = mode == kRK1 ? 1.0 : 2.0;
    double un[R][N];  // rows (e, v, j), fetched a batch ahead
    auto fetch = [&](int e0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = lane + 32 * r, e = i / (kNS * N), row = i - e * (kNS * N);
            if (i < kRows) dgk::load_row<N>(Us + (static_cast<size_t>(min(e0 + e, a.ne - 1)) * kNS * N + row) * N, un[r]);
        }
    };
    const int stride = nwarp * E;
    int e0 = warp * E;
    if (e0 < a.ne) fetch(e0);
    for (; e0 < a.ne; e0 += stride) {
        // the batch's lifts, for the last pass
        auto get_lifts = [&]() {
            const int nl = min(E, a.ne - e0) * C::kL;
            for (int i = 2 * lane; i < nl; i += 64) dgk::cp_async16(sL + i, a.elift + static_cast<size_t>(e0) * C::kL + i);
            dgk::cp_async_commit();
        };
        if constexpr (!LATE) get_lifts();
        // x interpolation
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = lane + 32 * r, e = i / (kNS * N), row = i - e * (kNS * N);
            if (i < kRows) {
                double* o = sA + e * ES + row * MS;
#pragma unroll
                for (int q = 0; q < M; ++q) {
                    double s = 0.0;
#pragma unroll
                    for (int b = 0; b < N; ++b) s += dgk::sym<MN>(a.B, q * N + b) * un[r][b];
                    o[q] = s;
                }
            }
        }
        __syncwarp();
        // columns: y interpolation, flux, contravariant transform, y contraction
        if (lane < E * M) {
            const int e = lane / M, qx = lane - e * M;
            double* col = sA + e * ES + qx;
            const Geo* g = a.geo + min(e0 + e, a.ne - 1);
            double S[kNS][M];
#pragma unroll
            for (int v = 0; v < kNS; ++v) {
                double x[N];
#pragma unroll
                for (int b = 0; b < N; ++b) x[b] = col[(v * N + b) * MS];
#pragma unroll
                for (int q = 0; q < M; ++q) {
                    double s = 0.0;
#pragma unroll
                    for (int b = 0; b < N; ++b) s += dgk::sym<MN>(a.B, q * N + b) * x[b];
                    S[v][q] = s;
                }
            }
            const double jd[4] = {g->jd[0], g->jd[1], g->jd[2], g->jd[3]};
            double V[2][M], p[M];
            bool sound = true;
#pragma unroll
            for (int q = 0; q < M; ++q) {
                const double r1 = 1. / S[0][q];
                const double u = S[1][q] * r1, v = S[2][q] * r1;
                p[q] = (a.gamma - 1.0) * (S[3][q] - 0.5 * (S[1][q] * u + S[2][q] * v));
                sound = sound && S[0][q] > 0.0 && p[q] > 0.0;  // a NaN is not
                if (!sound) {
                    if (!(S[0][q] > 0.0)) status |= kRho;
                    if (!(p[q] > 0.0)) status |= kPressure;
                    if (S[0][q] != S[0][q] || p[q] != p[q]) status |= kNaN;
                }
                const double w = a.W[qx] * a.W[q];
                S[3][q] += p[q];
#pragma unroll
                for (int d = 0; d < 2; ++d) V[d][q] = (u * jd[d * 2] + v * jd[d * 2 + 1]) * w;
                p[q] *= w;
            }
#pragma unroll
            for (int v = 0; v < kNS; ++v) {
                double a0[N], a1[N];
#pragma unroll
                for (int b = 0; b < N; ++b) { a0[b] = 0.0; a1[b] = 0.0; }
#pragma unroll
                for (int q = 0; q < M; ++q) {
                    double g0 = S[v][q] * V[0][q], g1 = S[v][q] * V[1][q];
                    if (v == 1 || v == 2) {
                        g0 += p[q] * jd[v - 1];
                        g1 += p[q] * jd[2 + v - 1];
                    }
#pragma unroll
                    for (int b = 0; b < N; ++b) {
                        a0[b] += dgk::sym<MN>(a.MB, q * N + b) * g0;
                        a1[b] += dgk::asym<MN>(a.MD, q * N + b) * g1;
                    }
                }
#pragma unroll
                for (int b = 0; b < N; ++b) {
                    col[(v * N + b) * MS] = a0[b];
                    col[(kNS * N + v * N + b) * MS] = a1[b];
                }
            }
        }
        __syncwarp();
        if constexpr (LATE) {
            if (!lifts_ready()) return;
        } else {
            fetch(e0 + stride);  // past the end: the last element again
            dgk::cp_async_wait_all();
            __syncwarp();
        }
        // x contraction, the row's edges (bottom 0, right 1, top 2, left 3) and the update
#pragma unroll 1
        for (int i = lane; i < kRows; i += 32) {
            const int e = i / (kNS * N), row = i - e * (kNS * N), v = row / N, jy = row - v * N;
            const int ge = min(e0 + e, a.ne - 1);
            const size_t gi = (static_cast<size_t>(ge) * kNS * N + row) * N;
            double u0[N] = {}, ac[N] = {};
            if (need_u0) dgk::load_row<N>(U0 + gi, u0);
            if (need_acc) dgk::load_row<N>(a.acc + gi, ac);
            const double* A0 = sA + e * ES + row * MS;
            double x[N];
#pragma unroll
            for (int b = 0; b < N; ++b) x[b] = 0.0;
#pragma unroll
            for (int q = 0; q < M; ++q) {
                const double c0 = A0[q], c1 = A0[kNS * N * MS + q];
#pragma unroll
                for (int b = 0; b < N; ++b)
                    x[b] = dgk::add_two(x[b], dgk::asym<MN>(a.MD, q * N + b), c0, dgk::sym<MN>(a.MB, q * N + b), c1);
            }
            const double* Lv = sL + e * C::kL + v * N;
            const double m0 = sM[jy], m1 = sM[N + jy], l3 = Lv[3 * kNS * N + jy], l1 = Lv[kNS * N + jy];
            const double scale = mode == kResidual ? 1.0 : a.dt * a.geo[ge].idj;
            if (e0 + e >= a.ne) continue;
            double k[N], o[N];
#pragma unroll
            for (int b = 0; b < N; ++b) {
                double s = x[b];
                s += m0 * Lv[b];
                s += m1 * Lv[2 * kNS * N + b];
                s += a.ME[0][b] * l3;
                s += a.ME[1][b] * l1;
                k[b] = scale * s;
            }
            if (put_acc) {
                double ao[N];
#pragma unroll
                for (int b = 0; b < N; ++b) ao[b] = ac[b] + ca * k[b];
                dgk::store_row<N>(a.acc + gi, ao);
            }
#pragma unroll
            for (int b = 0; b < N; ++b) o[b] = u0[b] + cu * (sum_acc ? ac[b] + k[b] : k[b]);
            dgk::store_row<N>(out + gi, o);
        }
        __syncwarp();  // the columns and the lifts are the next batch's
    }
}

// one warp per CTA; registers for MB resident warps per SM
template <int P, int MB>
__global__ void __launch_bounds__(32, MB) stage2d_kernel(const __grid_constant__ Args a)
{
    extern __shared__ __align__(16) double sm[];
    unsigned status = 0;
    stage_phase<P, false>(a, a.Us, a.U0, a.out, a.mode, sm, blockIdx.x, gridDim.x, status, []() { return true; });
    if (status) atomicOr(a.status, status);
}

// Steps of a small mesh in one launch.  Every stage warp keeps one batch of elements and
// goes up to the y contraction while the block's edge warps compute the lifts of its
// elements into shared memory.  An edge between two blocks is computed by both, so that
// one wait a stage is left: the edge warps' for the neighbours' states, on a counter in
// global memory that each block raises after its update.  The wait is bounded, and the
// launch cooperative (all blocks resident) unless it is of a single stage, which waits for
// nothing.  A stage's update may overwrite what other blocks' edges read the stage before:
// they were done with it when their block's update was counted, which this block's edges
// have waited for.
// Taken while every stage warp has at most one batch, where it beats the two launches
// by their latency (RK stage, HLLC, 32^2: p = 1 7.3 -> 5.1, p = 3 8.3 -> 5.9, p = 5 11.4 ->
// 7.8 us; 6.8, 7.1 and 7.9 with each edge computed once and the lifts handed over
// between blocks too; forward Euler, 20^2: p = 1 11.6 -> 5.2, p = 3 12.6 -> 5.6 a step).
// RK: RK4 steps on U0 through Ua and Ub.  Otherwise steps of the one stage `mode`, from
// U0 to Ua and back: forward Euler, or the residual of U0 into Ua.
struct StepArgs {
    Args a;
    double *U0, *Ua, *Ub;
    int nsteps, mode;
    unsigned* sync;  // arrivals of the stage warps, one per block and stage but the launch's last
    unsigned base;   // its value before the launch
    long long wait_cycles;  // limit of a wait
};
constexpr int kStageWarps = 4, kEdgeWarps = 4, kStepThreads = 32 * (kStageWarps + kEdgeWarps);

// the batches of block b: [first_batch(b), first_batch(b + 1)), neighbouring ones, so that
// many edges have both sides in the block
__host__ __device__ inline int first_batch(int b, int batches, int nblock)
{
    return static_cast<int>(static_cast<long long>(batches) * b / nblock);
}

// the block's edges [i0, i1) by warp `warp` of nwarp; lifts to the block's shared memory
template <int P>
__device__ __forceinline__ void block_edge_phase(const Args& a, const double* Us, int mode, const Tab& T, int warp, int nwarp, int i0,
                                                 int i1, double* sm, unsigned& status)
{
    constexpr int N = P + 1, EPW = 32 / N;
    const double* C = mode == kResidual ? T.FB : T.MF;
    const int lane = threadIdx.x & 31, k = lane / N, j = lane - k * N;
    for (i0 += warp * EPW; i0 < i1; i0 += nwarp * EPW) {
        const bool on = k < EPW && i0 + k < i1;
        const BlockEdge be = a.block_edges[on ? i0 + k : i1 - 1];
        const Edge ed = a.edges[be.edge];
        const int fL = ed.code & 3, fR = (ed.code >> 2) & 3, flip = (ed.code >> 4) & 1;
        double F[kNS];
        unsigned bad;
        edge_flux<P>(a, Us, T, ed, F, bad);
        if (on) status |= bad;
#pragma unroll
        for (int v = 0; v < kNS; ++v) {
            double sl = 0.0, sr = 0.0;
#pragma unroll
            for (int m = 0; m < N; ++m) {  // point m; node j of either side
                const double Fm = __shfl_sync(0xffffffffu, F[v], k * N + m);
                sl += C[(fL * N + m) * N + j] * Fm;
                sr += C[(fR * N + (flip ? N - 1 - m : m)) * N + j] * Fm;
            }
            if (on && be.oL >= 0) sm[be.oL + v * N + j] = -sl;
            if (on && be.oR >= 0) sm[be.oR + v * N + j] = sr;
        }
    }
}

template <int P, bool RK>
__global__ void __launch_bounds__(kStepThreads, 1) steps2d_kernel(const __grid_constant__ StepArgs s)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ Tab T;
    // the edge warps' wait gave up; the stage (counted through the launch) it was of
    __shared__ int dead, gave_up;
    constexpr int kSlot = Cfg<P>::smem / sizeof(double), kL = Cfg<P>::E * Cfg<P>::kL;
    if (threadIdx.x == 0) {
        dead = 0;
        gave_up = 0x7fffffff;
    }
    for (int i = threadIdx.x; i < kStageWarps * kL; i += kStepThreads) sm[i / kL * kSlot + i % kL] = 0.0;  // edges that are no interior ones
    load_tab(s.a, T);
    const int w = threadIdx.x / 32, nb = gridDim.x, batches = (s.a.ne + Cfg<P>::E - 1) / Cfg<P>::E;
    const int batch = first_batch(blockIdx.x, batches, nb) + w, end = first_batch(blockIdx.x + 1, batches, nb);
    const int i0 = s.a.block_first[blockIdx.x], i1 = s.a.block_first[blockIdx.x + 1];
    // more edges than the edge warps take at once: the stage warps, done up to the y contraction, help
    const bool share = i1 - i0 > kEdgeWarps * (32 / (P + 1));
    const int workers = share ? kEdgeWarps + kStageWarps : kEdgeWarps;
    unsigned status = 0, target = s.base;
    bool ok = true;
    for (int step = 0; step < s.nsteps && ok; ++step)
#pragma unroll 1
        for (int stage = 1; stage <= (RK ? 4 : 1) && ok; ++stage) {
            const int count = RK ? 4 * step + stage : step + 1;
            const int back = step % 2;
            const double* Us = !RK ? (back ? s.Ua : s.U0) : stage == 1 ? s.U0 : stage == 3 ? s.Ub : s.Ua;
            double* out = !RK ? (back ? s.U0 : s.Ua) : stage == 4 ? s.U0 : stage == 2 ? s.Ub : s.Ua;
            const double* U0 = RK ? s.U0 : Us;
            const int mode = RK ? kRK1 + stage - 1 : s.mode;
            if (w < kStageWarps) {
                auto ready = [&]() {
                    if (share) {
                        dgk::named_sync<kStepThreads>(4);  // the edge warps' wait is over
                        block_edge_phase<P>(s.a, Us, mode, T, kEdgeWarps + w, workers, i0, i1, sm, status);
                    }
                    dgk::named_sync<kStepThreads>(1);
                    return ok = *reinterpret_cast<volatile int*>(&gave_up) > count;
                };
                if (batch < end)
                    stage_phase<P, true>(s.a, Us, U0, out, mode, sm + w * kSlot, batch, batches, status, ready);
                else
                    ready();
                if (ok && (step + 1 < s.nsteps || (RK && stage < 4))) dgk::role_arrive<32 * kStageWarps>(s.sync, 2, threadIdx.x);
            } else {
                if (step > 0 || stage > 1) {
                    target += nb;
                    ok = dgk::role_wait<32 * kEdgeWarps>(s.sync, target, s.wait_cycles, s.a.status, &dead, 3, threadIdx.x - 32 * kStageWarps);
                }
                if (share) asm volatile("bar.arrive 4, %0;" ::"n"(kStepThreads) : "memory");
                if (ok) block_edge_phase<P>(s.a, Us, mode, T, w - kStageWarps, workers, i0, i1, sm, status);
                else gave_up = count;
                dgk::named_sync<kStepThreads>(1);  // (after a wait that gave up too: the stage warps wait here)
            }
        }
    if (status) atomicOr(s.a.status, status);
}

using KernelFn = void (*)(const Args);
struct Kernels {
    KernelFn edge, stage;
    void (*steps)(const StepArgs);
    void (*single_steps)(const StepArgs);
    size_t smem;
    int elems, edges_per_warp;
};
template <int P, int MB>
constexpr Kernels kernels()
{
    return Kernels{edge2d_kernel<P>, stage2d_kernel<P, MB>, steps2d_kernel<P, true>, steps2d_kernel<P, false>, Cfg<P>::smem, Cfg<P>::E, 32 / (P + 1)};
}
Kernels kernels_of(int p)
{
    switch (p) {
        case 0: return kernels<0, 16>();
        case 1: return kernels<1, 16>();
        case 2: return kernels<2, 16>();
        case 3: return kernels<3, 16>();
        case 4: return kernels<4, 12>();
        default: return kernels<5, 12>();
    }
}

// [ne][4][nb] <-> [ne][nb][4]
__global__ void transpose2d_kernel(const double* __restrict__ src, double* __restrict__ dst, long long n, int nb, int to_host)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long e = i / (kNS * nb);
        const int r = static_cast<int>(i - e * kNS * nb);
        if (to_host) dst[i] = src[(e * kNS + r % kNS) * nb + r / kNS];
        else dst[i] = src[(e * nb + r % nb) * kNS + r / nb];
    }
}

// ---------------- host ----------------

// corner nodes of an edge in traversal order (get_points_on_face_quadrilateral,
// shape.cpp:69-122)
constexpr int kFaceNodes[4][2] = {{0, 1}, {1, 3}, {3, 2}, {2, 0}};
constexpr double kRefX[4] = {-1., 1., -1., 1.}, kRefY[4] = {-1., -1., 1., 1.};

// the order's edge tables: rule of p+1 points, edge traces from the 2D basis at
// the edge points computed as
// get_points_on_face_quadrilateral and get_lagrange_basis_val_2D do
bool make_tab(int p, const dgh::Tables1D& t1, Tab& T)
{
    std::memset(&T, 0, sizeof(T));
    const int n = p + 1, nf = p + 1;
    std::vector<double> s, w;
    dgh::gauss_legendre(nf, s, w);
    for (int q = 0; q < nf; ++q) T.fw[q] = w[q];
    const std::vector<double> xn = dgh::equidistant_nodes(n);
    for (int f = 0; f < 4; ++f) {
        const int a = kFaceNodes[f][0], b = kFaceNodes[f][1];
        std::vector<double> val(static_cast<size_t>(nf) * n * n);
        for (int q = 0; q < nf; ++q) {
            const double b1 = (s[q] + 1.) / 2., b0 = 1.0 - b1;
            const double x = b0 * kRefX[a] + b1 * kRefX[b], y = b0 * kRefY[a] + b1 * kRefY[b];
            double vx[kMaxN], vy[kMaxN], gx[kMaxN], gy[kMaxN];
            dgh::lagrange_1d(x, xn, vx, gx);
            dgh::lagrange_1d(y, xn, vy, gy);
            for (int jj = 0; jj < n; ++jj)
                for (int ii = 0; ii < n; ++ii) val[(static_cast<size_t>(q) * n + jj) * n + ii] = vx[ii] * vy[jj];
        }
        // the edge's nodes (basis index j n + i with j = 0, i = p, j = p, i = 0
        // on faces 0..3), in ascending index; every other basis function
        // vanishes on the edge (its Lagrange factor in the normal direction is
        // zero at the edge's coordinate)
        int cnt = 0;
        for (int k = 0; k < n * n; ++k) {
            const int i = k % n, jj = k / n;
            const bool on = (f == 0 && jj == 0) || (f == 1 && i == p) || (f == 2 && jj == p) || (f == 3 && i == 0);
            if (!on) {
                for (int q = 0; q < nf; ++q)
                    if (std::fabs(val[static_cast<size_t>(q) * n * n + k]) > 1e-14) return false;
                continue;
            }
            for (int q = 0; q < nf; ++q) T.FB[(f * n + q) * n + cnt] = val[static_cast<size_t>(q) * n * n + k];
            ++cnt;
        }
        if (cnt != n) return false;
        // the lift of the update: the edge's nodes through the 1D inverse mass
        for (int q = 0; q < nf; ++q)
            for (int mm = 0; mm < n; ++mm) {
                double v = 0.0;
                for (int k = 0; k < n; ++k) v += t1.Minv[mm * n + k] * T.FB[(f * n + q) * n + k];
                T.MF[(f * n + q) * n + mm] = v;
            }
    }
    return true;
}

}  // namespace d2

struct dg_ctx2d {
    int device = 0, p = 0, nb = 1, ne = 0, nnode = 0, flux = 0;
    double gamma = 1.4, R = 1.0;
    cudaStream_t stream = nullptr;
    double *d_U0 = nullptr, *d_Ua = nullptr, *d_Ub = nullptr, *d_acc = nullptr, *d_res = nullptr;
    d2::Geo* d_geo = nullptr;
    d2::Edge* d_edges = nullptr;
    int* d_blocks = nullptr;  // d2::Args::block_first, then block_edges
    double* d_elift = nullptr;
    d2::Tab* d_tab = nullptr;
    unsigned* d_status = nullptr;
    unsigned* h_status = nullptr;  // its pinned copy on the host (or null: see dgi::take_status_slot)
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t graph_exec = nullptr;
    double graph_dt = 0.0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int nedge = 0, grid = 1, edge_grid = 1;
    int step_grid = 0;       // blocks of the small-mesh steps, 0: the mesh is too large for them
    unsigned sync_base = 0;  // their counter's value
    d2::Args args{};  // tables and geometry of every launch
    dgh::Tables1D t1;
    std::vector<double> coords;  // [nnode][2]
    std::vector<unsigned> e2n;   // [ne][4]
    std::vector<double> djac;    // [ne]
    std::vector<double> host;    // a small state between its layouts (see to_device)
    std::string err;
};

namespace {

int fail2(dg_ctx2d* c, int code, const std::string& msg)
{
    if (c) c->err = msg;
    else dgi::fail(nullptr, code, msg);
    return code;
}

#define DG2_CUDA(c, call)                                                                               \
    do {                                                                                                \
        cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess) return fail2((c), DG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

void release(dg_ctx2d* c)
{
    if (c->graph_exec) cudaGraphExecDestroy(c->graph_exec);
    if (c->graph) cudaGraphDestroy(c->graph);
    cudaFree(c->d_U0);
    cudaFree(c->d_Ua);
    cudaFree(c->d_Ub);
    cudaFree(c->d_acc);
    cudaFree(c->d_res);
    cudaFree(c->d_geo);
    cudaFree(c->d_edges);
    cudaFree(c->d_blocks);
    cudaFree(c->d_elift);
    cudaFree(c->d_tab);
    cudaFree(c->d_status);
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->ev1) cudaEventDestroy(c->ev1);
    if (c->stream) cudaStreamDestroy(c->stream);
    dgi::give_status_slot(c->h_status);
}

d2::Args args_of(const dg_ctx2d* c, int mode, double dt)
{
    d2::Args a = c->args;
    a.mode = mode;
    a.dt = dt;
    if (mode == d2::kResidual) {  // no inverse mass
        const int n = c->p + 1;
        for (int i = 0; i < n * (n + 1); ++i) {
            a.MB[i] = c->t1.B[i];
            a.MD[i] = c->t1.D[i];
        }
        for (int b = 0; b < n; ++b) {
            a.ME[0][b] = b == 0 ? 1.0 : 0.0;
            a.ME[1][b] = b == n - 1 ? 1.0 : 0.0;
        }
    }
    return a;
}

int launch(dg_ctx2d* c, const double* Us, double* out, int mode, double dt)
{
    d2::Args a = args_of(c, mode, dt);
    a.Us = Us;
    a.out = out;
    a.U0 = c->d_U0;
    const d2::Kernels k = d2::kernels_of(c->p);
    if (c->nedge > 0) k.edge<<<c->edge_grid, d2::kEdgeThreads, 0, c->stream>>>(a);
    k.stage<<<c->grid, 32, k.smem, c->stream>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DG_OK : fail2(c, DG_ERR_CUDA, std::string("stage2d launch: ") + cudaGetErrorString(e));
}

int check_status(dg_ctx2d* c)
{
    unsigned word = 0;
    if (!c->h_status) c->h_status = dgi::take_status_slot();
    unsigned* to = c->h_status ? c->h_status : &word;
    DG2_CUDA(c, cudaMemcpyAsync(to, c->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream));
    DG2_CUDA(c, cudaStreamSynchronize(c->stream));
    const unsigned s = *to;
    if (s & dgk::kStatusTimeout) {
        DG2_CUDA(c, cudaMemsetAsync(c->d_status, 0, d2::kStatusWords * sizeof(unsigned), c->stream));
        DG2_CUDA(c, cudaStreamSynchronize(c->stream));
        c->sync_base = 0;
        return fail2(c, DG_ERR_TIMEOUT, "a bounded device wait gave up (status " + std::to_string(s) + ")");
    }
    if (s) return fail2(c, DG_ERR_NONPHYSICAL, "non-physical state (status " + std::to_string(s) + ")");
    return DG_OK;
}

// a state between its host layout [ne][nb][4] and device layout [ne][4][nb] (the same at
// p = 0), through the device scratch buffer `scratch`; one of up to kHostValues values is
// transposed on the host, which takes less than the kernel's launch (set / get, p = 3: 30
// elements 15.4 / 24.6 -> 12.7 / 19.4 us, 156 elements 23.0 / 39 -> 22.2 / 32.4)
constexpr long long kHostValues = 16384;

int to_device(dg_ctx2d* c, const double* h, double* d, double* scratch)
{
    const int nb = c->nb;
    const long long n = 1LL * c->ne * d2::kNS * nb;
    double* t = c->host.data();
    const bool on_host = nb > 1 && n <= kHostValues, on_device = nb > 1 && !on_host;
    for (long long e = 0; on_host && e < n; e += d2::kNS * nb)
        for (int b = 0; b < nb; ++b)
            for (int v = 0; v < d2::kNS; ++v) t[e + v * nb + b] = h[e + b * d2::kNS + v];
    DG2_CUDA(c, cudaMemcpyAsync(on_device ? scratch : d, on_host ? t : h, n * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    if (on_device) {
        d2::transpose2d_kernel<<<1024, 256, 0, c->stream>>>(scratch, d, n, nb, 0);
        DG2_CUDA(c, cudaGetLastError());
    }
    DG2_CUDA(c, cudaStreamSynchronize(c->stream));
    return DG_OK;
}
// (checked: once the status word is good; on its error h is left as it was)
int to_host(dg_ctx2d* c, const double* d, double* h, double* scratch, bool checked = false)
{
    const int nb = c->nb;
    const long long n = 1LL * c->ne * d2::kNS * nb;
    double* t = c->host.data();
    if (n <= kHostValues) {
        DG2_CUDA(c, cudaMemcpyAsync(t, d, n * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    } else if (nb > 1) {
        d2::transpose2d_kernel<<<1024, 256, 0, c->stream>>>(d, scratch, n, nb, 1);
        DG2_CUDA(c, cudaGetLastError());
        d = scratch;
    }
    if (checked) {
        const int rc = check_status(c);
        if (rc) return rc;
    }
    if (n > kHostValues) DG2_CUDA(c, cudaMemcpyAsync(h, d, n * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if (n > kHostValues || !checked) DG2_CUDA(c, cudaStreamSynchronize(c->stream));
    for (long long e = 0; n <= kHostValues && e < n; e += d2::kNS * nb)
        for (int b = 0; b < nb; ++b)
            for (int v = 0; v < d2::kNS; ++v) h[e + b * d2::kNS + v] = t[e + v * nb + b];
    return DG_OK;
}

// the IC families of the 2D path at (x, y): the 3D families at (x, y, 0)
// without their third momentum; DG_IC_VORTEX_2D is the x-y family centred at
// the origin with no period (the reference's 2D vortex, functions.cpp:94-145)
bool ic_state(int type, const double* data, int ndata, double gamma, double R, double x, double y, double t, double* U4)
{
    double x3[3] = {x, y, 0.0}, U5[5], d[9] = {0, 0, 0, 0, 0, 0, 0, 1e300, 1e300};
    if (type == DG_IC_VORTEX_2D) {
        for (int i = 0; i < 5 && i < ndata; ++i) d[i] = data[i];
        dgp::initial_state(DG_IC_VORTEX_XY, d, gamma, R, x3, t, U5);
    } else if (type == DG_IC_UNIFORM) {
        const double u[5] = {data[0], data[1], data[2], 0.0, data[3]};
        dgp::initial_state(DG_IC_UNIFORM, u, gamma, R, x3, t, U5);
    } else if (type == DG_IC_VORTEX_XY) {
        dgp::initial_state(DG_IC_VORTEX_XY, data, gamma, R, x3, t, U5);
    } else {
        return false;
    }
    U4[0] = U5[0];
    U4[1] = U5[1];
    U4[2] = U5[2];
    U4[3] = U5[4];
    return true;
}

bool ic_args_ok(int type, int ndata)
{
    if (type == DG_IC_VORTEX_2D) return ndata >= 5;
    if (type == DG_IC_UNIFORM) return ndata >= 4;
    if (type == DG_IC_VORTEX_XY) return ndata >= 9;
    return false;
}

// (x, y) of reference point (xi, eta) of element e (the bilinear map,
// MeshTools::ref_to_phys, mesh/tools.cpp:19-26)
void ref_to_phys(const dg_ctx2d* c, int e, double xi, double eta, double& x, double& y)
{
    const double gv[4] = {0.25 * (1 - xi) * (1 - eta), 0.25 * (1 + xi) * (1 - eta), 0.25 * (1 - xi) * (1 + eta),
                          0.25 * (1 + xi) * (1 + eta)};
    x = y = 0.0;
    for (int n = 0; n < 4; ++n) {
        x += gv[n] * c->coords[2 * c->e2n[4 * e + n]];
        y += gv[n] * c->coords[2 * c->e2n[4 * e + n] + 1];
    }
}

// the blocks' edge lists of the one-launch steps: d2::Args::block_first, then block_edges
std::vector<int> block_edges(const dg_ctx2d* c, const std::vector<d2::Edge>& edges, const d2::Kernels& k)
{
    const int nb = c->step_grid, batches = (c->ne + k.elems - 1) / k.elems, n = c->p + 1;
    std::vector<int> block(c->ne), where(c->ne);  // an element's block, its lifts' place there
    for (int b = 0; b < nb; ++b) {
        const int first = d2::first_batch(b, batches, nb);
        for (int e = first * k.elems; e < std::min(c->ne, d2::first_batch(b + 1, batches, nb) * k.elems); ++e) {
            block[e] = b;
            where[e] = (e / k.elems - first) * static_cast<int>(k.smem / sizeof(double)) + e % k.elems * 4 * d2::kNS * n;
        }
    }
    std::vector<int> data(nb + 1, 0);  // the first entries, counted one block on
    for (const d2::Edge& ed : edges) {
        ++data[block[ed.eL] + 1];
        if (block[ed.eR] != block[ed.eL]) ++data[block[ed.eR] + 1];
    }
    for (int b = 0; b < nb; ++b) data[b + 1] += data[b];
    std::vector<int> next(data.begin(), data.end() - 1);
    data.resize(nb + 1 + 3 * static_cast<size_t>(data[nb]));
    for (size_t i = 0; i < edges.size(); ++i) {
        const d2::Edge& ed = edges[i];
        const int oL = where[ed.eL] + (ed.code & 3) * d2::kNS * n, oR = where[ed.eR] + ((ed.code >> 2) & 3) * d2::kNS * n;
        const int bL = block[ed.eL], bR = block[ed.eR];
        auto put = [&](int b, int l, int r) {
            int* o = &data[nb + 1 + 3 * static_cast<size_t>(next[b]++)];
            o[0] = static_cast<int>(i);
            o[1] = l;
            o[2] = r;
        };
        put(bL, oL, bR == bL ? oR : -1);
        if (bR != bL) put(bR, -1, oR);
    }
    return data;
}

// steps of a small mesh, at most 256 to a launch (queued on the stream): RK4 steps (mode
// kRK1), or steps of one stage between d_U0 and Ua (see d2::StepArgs).  A probe of the waits
// withholds an arrival: they then run to their limit.
int launch_steps(dg_ctx2d* c, int mode, double* Ua, double dt, int nsteps, long long wait_cycles = dgk::kSmallWaitCycles,
                 unsigned withheld = 0)
{
    const d2::Kernels k = d2::kernels_of(c->p);
    const auto kernel = mode == d2::kRK1 ? k.steps : k.single_steps;
    d2::StepArgs s{};
    s.a = args_of(c, mode, dt);
    s.mode = mode;
    s.wait_cycles = wait_cycles;
    s.U0 = c->d_U0;
    s.Ua = Ua;
    s.Ub = c->d_Ub;
    s.sync = c->d_status + d2::kSyncWord;
    for (int done = 0; done < nsteps; done += s.nsteps) {
        s.nsteps = std::min(256, nsteps - done);
        s.base = c->sync_base + withheld;
        void* args[] = {&s};
        const int stages = (mode == d2::kRK1 ? 4 : 1) * s.nsteps;
        const void* fn = reinterpret_cast<const void*>(kernel);
        const dim3 grid(c->step_grid), threads(d2::kStepThreads);
        const size_t smem = k.smem * d2::kStageWarps;
        if (stages > 1) DG2_CUDA(c, cudaLaunchCooperativeKernel(fn, grid, threads, args, smem, c->stream));
        else DG2_CUDA(c, cudaLaunchKernel(fn, grid, threads, args, smem, c->stream));
        c->sync_base += static_cast<unsigned>(c->step_grid) * (stages - 1u);
    }
    return DG_OK;
}

int prepare_graph(dg_ctx2d* c, double dt)
{
    if (c->graph_exec && c->graph_dt == dt) return DG_OK;
    if (c->graph_exec) { cudaGraphExecDestroy(c->graph_exec); c->graph_exec = nullptr; }
    if (c->graph) { cudaGraphDestroy(c->graph); c->graph = nullptr; }
    DG2_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    int rc = launch(c, c->d_U0, c->d_Ua, d2::kRK1, dt);
    if (!rc) rc = launch(c, c->d_Ua, c->d_Ub, d2::kRK2, dt);
    if (!rc) rc = launch(c, c->d_Ub, c->d_Ua, d2::kRK3, dt);
    if (!rc) rc = launch(c, c->d_Ua, c->d_U0, d2::kRK4, dt);
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(c->stream, &g);
    if (rc) { if (g) cudaGraphDestroy(g); return rc; }
    if (ce != cudaSuccess) return fail2(c, DG_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(ce));
    c->graph = g;
    DG2_CUDA(c, cudaGraphInstantiate(&c->graph_exec, c->graph, 0));
    c->graph_dt = dt;
    return DG_OK;
}

}  // namespace

extern "C" {

int dg2d_create(const dg_case_desc* cd, const dg_mesh2d_desc* md, dg_ctx2d** out)
{
    if (!cd || !md || !out) return fail2(nullptr, DG_ERR_ARG, "dg2d_create: null argument");
    *out = nullptr;
    if (cd->order < 0 || cd->order > 5) return fail2(nullptr, DG_ERR_UNSUPPORTED, "dg2d_create: order must be 0..5");
    if (cd->flux != DG_FLUX_LAX_FRIEDRICHS && cd->flux != DG_FLUX_HLLC) return fail2(nullptr, DG_ERR_ARG, "dg2d_create: unknown flux");
    if (cd->precision != DG_PREC_FP64) return fail2(nullptr, DG_ERR_UNSUPPORTED, "dg2d_create: the 2D path is FP64");
    if (!(cd->gamma > 1.0)) return fail2(nullptr, DG_ERR_ARG, "dg2d_create: gamma must exceed 1");
    if (md->nnode < 4 || md->nelem < 1 || md->nface < 0 || !md->node_coords || !md->elem_to_node_ids ||
        (md->nface > 0 && !md->interior_faces))
        return fail2(nullptr, DG_ERR_ARG, "dg2d_create: empty mesh");
    if (2LL * md->nface > 4LL * md->nelem) return fail2(nullptr, DG_ERR_ARG, "dg2d_create: more faces than element edges");
    dg_ctx2d* c = new dg_ctx2d();
    c->device = cd->device;
    c->p = cd->order;
    c->nb = (c->p + 1) * (c->p + 1);
    c->ne = md->nelem;
    c->nnode = md->nnode;
    c->flux = cd->flux;
    c->gamma = cd->gamma;
    c->R = cd->gas_constant;
    auto bail = [&](int code, const std::string& msg) {
        dgi::fail(nullptr, code, "dg2d_create: " + msg);
        release(c);
        delete c;
        return code;
    };
    try {
        c->coords.assign(md->node_coords, md->node_coords + 2 * static_cast<size_t>(md->nnode));
        c->e2n.assign(md->elem_to_node_ids, md->elem_to_node_ids + 4 * static_cast<size_t>(md->nelem));
        for (unsigned v : c->e2n)
            if (v >= static_cast<unsigned>(md->nnode)) return bail(DG_ERR_ARG, "node id out of range");
        // geometry: parallelograms only (constant Jacobian), as the reference
        // computes it per point (basis/tools.cpp:42-66, linear_algebra.cpp:99-107)
        std::vector<d2::Geo> geo(c->ne);
        c->djac.resize(c->ne);
        for (int e = 0; e < c->ne; ++e) {
            double X[4][2];
            for (int n = 0; n < 4; ++n)
                for (int d = 0; d < 2; ++d) X[n][d] = c->coords[2 * c->e2n[4 * e + n] + d];
            double scale = 0.0;
            for (int n = 0; n < 4; ++n) scale = std::max(scale, std::max(std::fabs(X[n][0] - X[0][0]), std::fabs(X[n][1] - X[0][1])));
            // parallelograms up to the rounding of mesh files' coordinates
            // (1e-9 of the element's size); the Jacobian of the bilinear map
            // at the element's centre, the mean of its Jacobian over the element
            for (int d = 0; d < 2; ++d)
                if (std::fabs((X[3][d] - X[2][d]) - (X[1][d] - X[0][d])) > 1e-9 * scale)
                    return bail(DG_ERR_UNSUPPORTED, "element " + std::to_string(e) + " is not a parallelogram");
            double jac[4];
            for (int i = 0; i < 2; ++i) {
                jac[i * 2 + 0] = 0.25 * ((X[1][i] - X[0][i]) + (X[3][i] - X[2][i]));
                jac[i * 2 + 1] = 0.25 * ((X[2][i] - X[0][i]) + (X[3][i] - X[1][i]));
            }
            const double det = jac[0] * jac[3] - jac[1] * jac[2];
            if (!(det > 0.0)) return bail(DG_ERR_ARG, "element " + std::to_string(e) + " has a non-positive Jacobian");
            const double ij[4] = {jac[3] / det, -jac[1] / det, -jac[2] / det, jac[0] / det};
            for (int k = 0; k < 4; ++k) geo[e].jd[k] = ij[k] * det;
            geo[e].idj = 1.0 / det;
            c->djac[e] = det;
        }
        // interior edges: both elements and faces, the orientations, and the
        // left element's normal (boundary edges of a non-periodic mesh are not
        // listed: the reference's residual loops over the interior faces only,
        // base.cpp:470-561)
        std::vector<d2::Edge> edges;
        edges.reserve(md->nface);
        std::vector<char> seen(4 * static_cast<size_t>(c->ne), 0);
        for (int f = 0; f < md->nface; ++f) {
            const unsigned* r = md->interior_faces + 8 * static_cast<size_t>(f);
            if (r[0] != static_cast<unsigned>(md->rank) || r[4] != static_cast<unsigned>(md->rank))
                return bail(DG_ERR_ARG, "face rows must carry this rank");
            const unsigned eL = r[1], fL = r[2], oL = r[3], eR = r[5], fR = r[6], oR = r[7];
            if (eL >= static_cast<unsigned>(c->ne) || eR >= static_cast<unsigned>(c->ne) || fL > 3 || fR > 3 || oL > 1 || oR > 1)
                return bail(DG_ERR_ARG, "face row " + std::to_string(f) + " out of range");
            if (seen[4 * eL + fL] || seen[4 * eR + fR] || (eL == eR && fL == fR))
                return bail(DG_ERR_ARG, "an element face appears twice");
            seen[4 * eL + fL] = seen[4 * eR + fR] = 1;
            // normal (dy/ds, -dx/ds) of the left element's edge with the
            // LagrangeSeg p = 1 gradient (-1/2, 1/2) (shape.cpp:154-210)
            const int a = d2::kFaceNodes[fL][0], b = d2::kFaceNodes[fL][1];
            const double* XA = &c->coords[2 * c->e2n[4 * eL + a]];
            const double* XB = &c->coords[2 * c->e2n[4 * eL + b]];
            const double g0 = -0.5, g1 = 0.5;
            const double dx = XA[0] * g0 + XB[0] * g1, dy = XA[1] * g0 + XB[1] * g1;
            const double N0 = 1.0 * dy, N1 = -1.0 * 1.0 * dx;
            const int flip = static_cast<int>(oL ^ oR);
            // N / |N| (base/functions.cpp:40-49), or N (1/|N|) as HLLC takes it
            // (euler/functions.cpp:309-311)
            const double nm = std::sqrt(N0 * N0 + N1 * N1), inv = 1. / nm;
            d2::Edge ed{};
            ed.n[0] = c->flux == DG_FLUX_HLLC ? N0 * inv : N0 / nm;
            ed.n[1] = c->flux == DG_FLUX_HLLC ? N1 * inv : N1 / nm;
            ed.nmag = nm;
            ed.eL = static_cast<int>(eL);
            ed.eR = static_cast<int>(eR);
            ed.code = static_cast<int>(fL | fR << 2) | flip << 4 | static_cast<int>(oL) << 5;
            edges.push_back(ed);
        }
        if (1LL * c->ne * d2::kNS * c->nb <= kHostValues) c->host.resize(static_cast<size_t>(c->ne) * d2::kNS * c->nb);
        c->t1 = dgh::make_tables(c->p);
        d2::Tab tab;
        if (!d2::make_tab(c->p, c->t1, tab)) return bail(DG_ERR_ARG, "edge trace tables");

        if (cudaSetDevice(c->device) != cudaSuccess) return bail(DG_ERR_CUDA, "cudaSetDevice failed");
        c->nedge = static_cast<int>(edges.size());
        std::vector<int> blocks;
        const d2::Kernels k = d2::kernels_of(c->p);
        int per_sm = 0, edge_per_sm = 0, sms = 0;
        if (cudaFuncSetAttribute(reinterpret_cast<const void*>(k.stage), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(k.smem)) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void*>(k.stage), 32, k.smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&edge_per_sm, reinterpret_cast<const void*>(k.edge), d2::kEdgeThreads, 0) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device) != cudaSuccess)
            return bail(DG_ERR_CUDA, "kernel attributes");
        c->grid = std::max(1, std::min((c->ne + k.elems - 1) / k.elems, std::max(1, per_sm) * std::max(1, sms)));
        // small meshes: one batch of elements per warp, at most one block per SM
        const int warps = (c->ne + k.elems - 1) / k.elems;
        if (warps <= sms * d2::kStageWarps) {
            int steps_per_sm = 0;
            const int smem = static_cast<int>(k.smem * d2::kStageWarps);
            int fits = 1;
            for (const auto kernel : {k.steps, k.single_steps}) {
                if (cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&steps_per_sm, reinterpret_cast<const void*>(kernel), d2::kStepThreads, smem) != cudaSuccess)
                    return bail(DG_ERR_CUDA, "kernel attributes");
                fits = std::min(fits, steps_per_sm);
            }
            if (fits > 0) {
                c->step_grid = std::min(sms, warps);
                blocks = block_edges(c, edges, k);
            }
        }
        const int per_cta = k.edges_per_warp * (d2::kEdgeThreads / 32);
        c->edge_grid = std::max(1, std::min((c->nedge + per_cta - 1) / per_cta, std::max(1, edge_per_sm) * std::max(1, sms)));
        const size_t nstate = static_cast<size_t>(c->ne) * d2::kNS * c->nb * sizeof(double);
        const size_t lift_bytes = static_cast<size_t>(c->ne) * 4 * d2::kNS * (c->p + 1) * sizeof(double);
        bool ok = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) == cudaSuccess &&
                  cudaEventCreate(&c->ev0) == cudaSuccess && cudaEventCreate(&c->ev1) == cudaSuccess &&
                  cudaMalloc((void**)&c->d_U0, nstate) == cudaSuccess && cudaMalloc((void**)&c->d_Ua, nstate) == cudaSuccess &&
                  cudaMalloc((void**)&c->d_Ub, nstate) == cudaSuccess && cudaMalloc((void**)&c->d_acc, nstate) == cudaSuccess &&
                  cudaMalloc((void**)&c->d_res, nstate) == cudaSuccess &&
                  cudaMalloc((void**)&c->d_geo, geo.size() * sizeof(d2::Geo)) == cudaSuccess &&
                  cudaMalloc((void**)&c->d_edges, std::max<size_t>(1, edges.size()) * sizeof(d2::Edge)) == cudaSuccess &&
                  (blocks.empty() || cudaMalloc((void**)&c->d_blocks, blocks.size() * sizeof(int)) == cudaSuccess) &&
                  cudaMalloc((void**)&c->d_elift, lift_bytes) == cudaSuccess &&
                  cudaMalloc((void**)&c->d_tab, sizeof(d2::Tab)) == cudaSuccess &&
                  cudaMalloc((void**)&c->d_status, d2::kStatusWords * sizeof(unsigned)) == cudaSuccess;
        if (!ok) {
            cudaGetLastError();
            return bail(DG_ERR_NOMEM, "device allocation failed");
        }
        ok = cudaMemcpy(c->d_geo, geo.data(), geo.size() * sizeof(d2::Geo), cudaMemcpyHostToDevice) == cudaSuccess &&
             (edges.empty() || cudaMemcpy(c->d_edges, edges.data(), edges.size() * sizeof(d2::Edge), cudaMemcpyHostToDevice) == cudaSuccess) &&
             (blocks.empty() || cudaMemcpy(c->d_blocks, blocks.data(), blocks.size() * sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess) &&
             cudaMemset(c->d_elift, 0, lift_bytes) == cudaSuccess &&
             cudaMemcpy(c->d_tab, &tab, sizeof(d2::Tab), cudaMemcpyHostToDevice) == cudaSuccess &&
             cudaMemset(c->d_status, 0, d2::kStatusWords * sizeof(unsigned)) == cudaSuccess &&
             cudaMemset(c->d_U0, 0, nstate) == cudaSuccess && cudaMemset(c->d_acc, 0, nstate) == cudaSuccess &&
             // (the context's stream does not wait for the default stream)
             cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess;
        if (!ok) return bail(DG_ERR_CUDA, "device upload failed");
        d2::Args& a = c->args;
        a.acc = c->d_acc;
        a.geo = c->d_geo;
        a.edges = c->d_edges;
        a.block_first = c->d_blocks;
        a.block_edges = reinterpret_cast<const d2::BlockEdge*>(c->d_blocks + c->step_grid + 1);
        a.elift = c->d_elift;
        a.tab = c->d_tab;
        a.status = c->d_status;
        a.ne = c->ne;
        a.nedge = c->nedge;
        a.flux = c->flux;
        a.gamma = c->gamma;
        const int n = c->p + 1, m = c->p + 2;
        for (int q = 0; q < m; ++q) {
            a.W[q] = c->t1.wq[q];
            for (int b = 0; b < n; ++b) {
                a.B[q * n + b] = c->t1.B[q * n + b];
                long double sb = 0.0L, sd = 0.0L;
                for (int k = 0; k < n; ++k) {
                    sb += static_cast<long double>(c->t1.B[q * n + k]) * c->t1.Minv[b * n + k];
                    sd += static_cast<long double>(c->t1.D[q * n + k]) * c->t1.Minv[b * n + k];
                }
                a.MB[q * n + b] = static_cast<double>(sb);
                a.MD[q * n + b] = static_cast<double>(sd);
            }
        }
        for (int b = 0; b < n; ++b) {
            a.ME[0][b] = c->t1.Minv[b * n];
            a.ME[1][b] = c->t1.Minv[b * n + n - 1];
        }
    } catch (const std::bad_alloc&) {
        return bail(DG_ERR_NOMEM, "host allocation failed");
    }
    *out = c;
    return DG_OK;
}

void dg2d_destroy(dg_ctx2d* c)
{
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    release(c);
    delete c;
}

const char* dg2d_last_error(const dg_ctx2d* c) { return c ? c->err.c_str() : dg_last_error(nullptr); }

int dg2d_num_basis(const dg_ctx2d* c) { return c ? c->nb : 0; }

int dg2d_set_state(dg_ctx2d* c, const double* Uc)
{
    if (!c || !Uc) return fail2(c, DG_ERR_ARG, "dg2d_set_state: null argument");
    DG2_CUDA(c, cudaSetDevice(c->device));
    return to_device(c, Uc, c->d_U0, c->d_res);
}

int dg2d_get_state(dg_ctx2d* c, double* Uc)
{
    if (!c || !Uc) return fail2(c, DG_ERR_ARG, "dg2d_get_state: null argument");
    DG2_CUDA(c, cudaSetDevice(c->device));
    return to_host(c, c->d_U0, Uc, c->d_res);
}

int dg2d_residual(dg_ctx2d* c, double* res)
{
    if (!c || !res) return fail2(c, DG_ERR_ARG, "dg2d_residual: null argument");
    DG2_CUDA(c, cudaSetDevice(c->device));
    int rc = c->step_grid ? launch_steps(c, d2::kResidual, c->d_res, 0.0, 1) : launch(c, c->d_U0, c->d_res, d2::kResidual, 0.0);
    if (rc) return rc;
    return to_host(c, c->d_res, res, c->d_Ub, true);
}

int dg2d_rk4_steps_timed(dg_ctx2d* c, double dt, int nsteps, double* device_ms)
{
    if (!c || nsteps < 0 || !(dt > 0.0)) return fail2(c, DG_ERR_ARG, "dg2d_rk4_steps: bad argument");
    DG2_CUDA(c, cudaSetDevice(c->device));
    int rc = c->step_grid ? DG_OK : prepare_graph(c, dt);
    if (rc) return rc;
    DG2_CUDA(c, cudaEventRecord(c->ev0, c->stream));
    if (c->step_grid) {
        if ((rc = launch_steps(c, d2::kRK1, c->d_Ua, dt, nsteps))) return rc;
    } else {
        for (int s = 0; s < nsteps; ++s) DG2_CUDA(c, cudaGraphLaunch(c->graph_exec, c->stream));
    }
    DG2_CUDA(c, cudaEventRecord(c->ev1, c->stream));
    if ((rc = check_status(c))) return rc;
    if (device_ms) {
        float ms = 0.f;
        DG2_CUDA(c, cudaEventElapsedTime(&ms, c->ev0, c->ev1));
        *device_ms = ms;
    }
    return DG_OK;
}

int dg2d_rk4_steps(dg_ctx2d* c, double dt, int nsteps) { return dg2d_rk4_steps_timed(c, dt, nsteps, nullptr); }

int dg2d_fe_steps(dg_ctx2d* c, double dt, int nsteps)
{
    if (!c || nsteps < 0 || !(dt > 0.0)) return fail2(c, DG_ERR_ARG, "dg2d_fe_steps: bad argument");
    DG2_CUDA(c, cudaSetDevice(c->device));
    if (c->step_grid) {
        const int rc = launch_steps(c, d2::kFE, c->d_Ua, dt, nsteps);
        if (rc) return rc;
        if (nsteps % 2) std::swap(c->d_U0, c->d_Ua);
        return check_status(c);
    }
    // the update reads its neighbours' stage state, so it writes another buffer
    for (int s = 0; s < nsteps; ++s) {
        int rc = launch(c, c->d_U0, c->d_Ua, d2::kFE, dt);
        if (rc) return rc;
        std::swap(c->d_U0, c->d_Ua);
    }
    if (nsteps % 2 && c->graph_exec) {
        // the RK4 graph captured the old buffer addresses
        cudaGraphExecDestroy(c->graph_exec);
        cudaGraphDestroy(c->graph);
        c->graph_exec = nullptr;
        c->graph = nullptr;
    }
    return check_status(c);
}

int dg2d_project_ic(dg_ctx2d* c, int ic_type, const double* data, int ndata, double t, double* Uc)
{
    if (!c || (ndata > 0 && !data) || !ic_args_ok(ic_type, ndata)) return fail2(c, DG_ERR_ARG, "dg2d_project_ic: bad initial condition");
    // init_state_from_fcn + L2 projection (base.cpp:113-223) on the
    // (2 max(p,1) + 2)^2 rule, the Kronecker inverse mass over det J
    const dgh::Tables1D& tb = c->t1;
    const int n = c->p + 1, me = tb.me, nb = c->nb;
    std::vector<double> U(static_cast<size_t>(c->ne) * nb * d2::kNS);
#pragma omp parallel for schedule(static)
    for (int e = 0; e < c->ne; ++e) {
        std::vector<double> f(static_cast<size_t>(me) * me * d2::kNS), rhs(static_cast<size_t>(nb) * d2::kNS), tmp(rhs.size());
        for (int qy = 0; qy < me; ++qy)
            for (int qx = 0; qx < me; ++qx) {
                double x, y, Ue[4];
                ref_to_phys(c, e, tb.xe[qx], tb.xe[qy], x, y);
                ic_state(ic_type, data, ndata, c->gamma, c->R, x, y, t, Ue);
                const double cw = (tb.we[qx] * tb.we[qy]) * c->djac[e];
                for (int v = 0; v < d2::kNS; ++v) f[(static_cast<size_t>(qy) * me + qx) * d2::kNS + v] = Ue[v] * cw;
            }
        for (int b = 0; b < nb; ++b)
            for (int v = 0; v < d2::kNS; ++v) {
                const int i = b % n, j = b / n;
                double acc = 0.0;
                for (int qy = 0; qy < me; ++qy)
                    for (int qx = 0; qx < me; ++qx)
                        acc += (tb.Be[qx * n + i] * tb.Be[qy * n + j]) * f[(static_cast<size_t>(qy) * me + qx) * d2::kNS + v];
                rhs[b * d2::kNS + v] = acc;
            }
        for (int b = 0; b < nb; ++b)
            for (int v = 0; v < d2::kNS; ++v) {
                const int i = b % n, j = b / n;
                double acc = 0.0;
                for (int k = 0; k < n; ++k) acc += tb.Minv[i * n + k] * rhs[(j * n + k) * d2::kNS + v];
                tmp[b * d2::kNS + v] = acc;
            }
        for (int b = 0; b < nb; ++b)
            for (int v = 0; v < d2::kNS; ++v) {
                const int i = b % n, j = b / n;
                double acc = 0.0;
                for (int k = 0; k < n; ++k) acc += tb.Minv[j * n + k] * tmp[(k * n + i) * d2::kNS + v];
                U[(static_cast<size_t>(e) * nb + b) * d2::kNS + v] = acc / c->djac[e];
            }
    }
    if (Uc) std::copy(U.begin(), U.end(), Uc);
    return dg2d_set_state(c, U.data());
}

int dg2d_l2_error(dg_ctx2d* c, int ic_type, const double* data, int ndata, double t, double* err)
{
    if (!c || !err || (ndata > 0 && !data) || !ic_args_ok(ic_type, ndata)) return fail2(c, DG_ERR_ARG, "dg2d_l2_error: bad argument");
    std::vector<double> U(static_cast<size_t>(c->ne) * c->nb * d2::kNS);
    int rc = dg2d_get_state(c, U.data());
    if (rc) return rc;
    // get_error (post/main.cpp:30-201) on the (2 max(p,1) + 2)^2 rule,
    // normalised by the volume of the volume rule (mesh/tools.cpp:28-36)
    const dgh::Tables1D& tb = c->t1;
    const int n = c->p + 1, me = tb.me, nb = c->nb;
    std::vector<double> per(static_cast<size_t>(c->ne) * d2::kNS, 0.0);
#pragma omp parallel for schedule(static)
    for (int e = 0; e < c->ne; ++e) {
        const double* Ue = U.data() + static_cast<size_t>(e) * nb * d2::kNS;
        double acc[4] = {0, 0, 0, 0};
        for (int qy = 0; qy < me; ++qy)
            for (int qx = 0; qx < me; ++qx) {
                double Uq[4] = {0, 0, 0, 0}, Ex[4], x, y;
                for (int b = 0; b < nb; ++b) {
                    const double bv = tb.Be[qx * n + b % n] * tb.Be[qy * n + b / n];
                    for (int v = 0; v < d2::kNS; ++v) Uq[v] += bv * Ue[b * d2::kNS + v];
                }
                ref_to_phys(c, e, tb.xe[qx], tb.xe[qy], x, y);
                ic_state(ic_type, data, ndata, c->gamma, c->R, x, y, t, Ex);
                const double w = (tb.we[qx] * tb.we[qy]) * c->djac[e];
                for (int v = 0; v < d2::kNS; ++v) acc[v] += (Uq[v] - Ex[v]) * (Uq[v] - Ex[v]) * w;
            }
        for (int v = 0; v < d2::kNS; ++v) per[static_cast<size_t>(e) * d2::kNS + v] = acc[v];
    }
    double tot[4] = {0, 0, 0, 0}, vol = 0.0, wsum = 0.0;
    for (int q = 0; q < c->p + 2; ++q)
        for (int r = 0; r < c->p + 2; ++r) wsum += tb.wq[r] * tb.wq[q];
    for (int e = 0; e < c->ne; ++e) {
        for (int v = 0; v < d2::kNS; ++v) tot[v] += per[static_cast<size_t>(e) * d2::kNS + v];
        vol += wsum * c->djac[e];
    }
    for (int v = 0; v < d2::kNS; ++v) err[v] = std::sqrt(tot[v] / vol);
    return DG_OK;
}

int dg2d_probe_step_wait(dg_ctx2d* c, long long limit_cycles)
{
    if (!c || limit_cycles < 0 || limit_cycles > 4000000000LL)
        return fail2(c, DG_ERR_ARG, "dg2d_probe_step_wait: limit must be 0 .. 4e9 SM cycles (about 2 s)");
    if (!c->step_grid) return fail2(c, DG_ERR_UNSUPPORTED, "dg2d_probe_step_wait: steps of this mesh do not wait on the device");
    DG2_CUDA(c, cudaSetDevice(c->device));
    const int rc = launch_steps(c, d2::kRK1, c->d_Ua, 0.0, 1, limit_cycles, 1);
    return rc ? rc : check_status(c);
}

int dg2d_status(dg_ctx2d* c, unsigned* flags)
{
    if (!c || !flags) return fail2(c, DG_ERR_ARG, "dg2d_status: null argument");
    DG2_CUDA(c, cudaSetDevice(c->device));
    DG2_CUDA(c, cudaMemcpyAsync(flags, c->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream));
    DG2_CUDA(c, cudaStreamSynchronize(c->stream));
    return *flags ? DG_ERR_NONPHYSICAL : DG_OK;
}

}  // extern "C"
