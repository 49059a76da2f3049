// dg_column.cuh -- the column form of the DG stage (affine elements, orders 1..5;
// bent ones in FP64, orders 1..3 the default):
// face_lift_kernel and column_kernel, one launch each per RK stage.
//
// Same scheme as dg_stage.cuh's face kernel and stage kernel, with the work cut
// so that little of it goes through shared memory:
//
//   face_lift_kernel  every interior face's numerical flux once, and its 2D
//       lift once: [face][5][(p+1)^2] lifted values in the listed side's order
//       (the other side reads them through the face-node permutation, which
//       commutes with the lift: nodes and points are symmetric on the face).
//   column_kernel     per batch of E elements: x and y interpolation through
//       shared memory, then one thread per (x, y) quadrature column does the z
//       interpolation, the Euler flux and the z contraction in registers
//       (holding the p+2 point states and contravariant velocities of its
//       column, variable by variable for the accumulators), then the y
//       contraction, and the x contraction fused with the face lifts and the
//       stage update.  A row of p+1 coefficients along x is one task's from
//       global memory to global memory, so the state, the step-start state and
//       the accumulator go straight between global memory and registers, the
//       next batch's prefetched into L2.
//
// FP64: the 1D inverse mass matrix is folded into the contraction tables
// (MB = B Minv, MD = D Minv per direction) and a face's lift is spread along its
// normal by the inverse mass's end columns, so no separate inverse-mass passes
// run.  The FP32 residual keeps its FP64 inverse mass as three passes after the
// contraction and the stage kernel's FP32 operations in their order (the same
// bits on meshes whose face orders agree).
//
// Why: the stage kernel writes and reads every intermediate through shared
// memory between up to nine block barriers per element, and waits on them
// (40^3, p = 3, FP64: 5140 warp instructions and 1640 shared wavefronts per
// element, FP64 pipe 40 %, `barrier` the first stall).  Here a warp owns its
// elements (no block barriers up to p = 3), about 2500 instructions per element,
// the column phase keeping 27 of the point array's 45 words in registers.  The
// next batch's rows and face records wait in registers during the contractions
// (reading them at the batch's top left long_scoreboard the first stall: 48^3,
// p = 3, RK stage 0.821 -> 0.722 ms FP64, 0.769 -> 0.695 ms mixed); 12 warps per
// SM at 168 registers beat 8 at 255 (0.777 ms) there, at p = 4 and 5 the other
// way round (40^3, p = 4: 0.970 against 1.037 ms).  RK stage (both kernels), stage kernel
// -> column form, GDOF/s: FP64 11.7 -> 24.4 (72^3, p = 1), 24.5 -> 39.0 (60^3,
// p = 2), 31.9 -> 49.4 (48^3, p = 3), 30.2 -> 41.0 (40^3, p = 4), 31.9 -> 42.6
// (32^3, p = 5); mixed 19.4 -> 29.6, 33.0 -> 44.6, 39.7 -> 55.2, 44.0 -> 52.3,
// 41.8 -> 53.4.  The FP32 form is bound by instruction issue (3288 per element at
// p = 3, 68 % of the issue slots): its lift sums take one y and one z face per row
// and its residual block has constant strides (48^3, p = 3: 0.695 -> 0.641 ms).
#pragma once
#include "dg_stage.cuh"

namespace dgk {

// launch option: the column form (needs the face kernel's fluxes lifted)
constexpr int kCF = 8192;
// launch option: RK4 steps of small meshes in one launch (dg_small.cuh)
constexpr int kSM = 16384;

// Shared-memory layout of a batch element.  The point array has 15 rows (v, d)
// of [bz][qy][qx] with plane stride PS and row stride AS; the x-interpolated
// block [v][bz][by][qx] (stride X1S) sits in its rows 5.. .  Strides and task
// orders (see TaskOrd for their coding) minimise the wavefronts of the passes'
// addresses (FP64 served per half-warp on 16 bank pairs, FP32 per warp on 32).
template <int P, typename T, bool GE = false>
struct ColLay {
    static constexpr bool W8 = sizeof(T) == 8;
    static constexpr int N = P + 1, M = P + 2, NB = N * N * N, NF = M * M, N2 = N * N;
    static constexpr int PS = NF + (W8 ? (P == 1 ? 6 : P == 2 ? 4 : P == 3 ? 3 : P == 4 ? 5 : 6)
                                       : (P == 1 ? 6 : P == 2 ? 5 : P == 3 ? 0 : P == 4 ? 5 : 0));
    static constexpr int AS = W8 ? (P == 1 ? 33 : P == 2 ? 63 : P == 3 ? 111 : P == 4 ? 207 : 335)
                                 : (P == 1 ? 31 : P == 2 ? 74 : P == 3 ? 119 : P == 4 ? 207 : 301);
    static constexpr int X1S = N * N * M + (W8 ? (P == 2 || P == 3 ? 1 : 0) : (P == 2 ? 1 : P == 4 ? 3 : 0));
    // (v, qx, bz) orders of the y interpolation and the y contraction
    static constexpr int oy = W8 ? (P == 1 ? 21 : P == 2 ? 7 : P == 3 ? 11 : P == 4 ? 19 : 7)
                                 : (P == 1 ? 21 : P == 2 ? 21 : P == 3 ? 7 : P == 4 ? 11 : 19);
    static constexpr int oyc = W8 ? (P == 3 || P == 4 ? 11 : 21) : (P == 1 ? 21 : P == 2 ? 15 : P == 4 ? 11 : 19);
    static_assert(PS >= NF && AS >= (N - 1) * PS + NF && 10 * AS >= 5 * X1S, "point-array rows overlap");
    static constexpr int W = 15 * AS;                     // point array, T
    // FP32 path and general geometry: the FP64 residual block, entry (bx, by, bz) at bz SZ + by SY + bx:
    // x, y and z pencils of a variable fall on distinct bank pairs but for a few
    // (N = 4: SY = 5, SZ = 20) and their words are constant offsets apart
    static constexpr int SY = N % 2 ? N : N + 1, SZ = N * SY, VS = N * SZ;
    static constexpr int RES = W8 && !GE ? 0 : 5 * VS;
    static constexpr int LF = 30 * N2;                    // the six faces' lifts, T
    static constexpr size_t f64_words(int E) { return static_cast<size_t>(E) * RES + 2 * N; }
    static constexpr size_t t_words(int E) { return static_cast<size_t>(E) * (W + LF + 6); }
    static constexpr size_t bytes(int E) { return f64_words(E) * 8 + t_words(E) * sizeof(T) + E * sizeof(int); }
};

template <int NT>
__device__ __forceinline__ void cta_sync()
{
    if constexpr (NT == 32) __syncwarp();
    else __syncthreads();
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src)
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem_src) : "memory");
}

// a row of N consecutive doubles (16-byte aligned when N is even)
template <int N>
__device__ __forceinline__ void load_row(const double* p, double (&x)[N])
{
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 2) {
            const double2 t = *reinterpret_cast<const double2*>(p + k);
            x[k] = t.x;
            x[k + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) x[k] = p[k];
    }
}
template <int N>
__device__ __forceinline__ void store_row(double* p, const double (&x)[N])
{
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 2) *reinterpret_cast<double2*>(p + k) = make_double2(x[k], x[k + 1]);
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) p[k] = x[k];
    }
}

// Dependent launch: a kernel launched with overlap may start when the CTAs of the
// kernel before it on the stream have ended, without waiting for that kernel's own
// completion, which it does in wait_prerequisites (all writes visible); only
// data that no kernel writes is read before.  Without overlap that call does nothing.
// FP64 RK stage: p = 1, 14^3 9.3 -> 8.8 us, p = 3, 9^3 12.9 -> 11.8, 16^3 34.3 -> 34.0;
// nothing from some 20^3 on; forward Euler's steps within a call the same way (p = 3, 6^3
// 12.5 -> 11.4).  An earlier start (griddepcontrol.launch_dependents at
// the kernels' beginning) places the CTAs unevenly: 9^3 15.8 us, 24^3 100 -> 110.
__device__ __forceinline__ void wait_prerequisites() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// the column kernel of FP64 p = 5 is at its register limit and loses 3 % to the wait
template <int P, typename T>
constexpr bool column_overlaps()
{
    return !(sizeof(T) == 8 && P >= 5);
}

inline cudaError_t launch_after(void (*kernel)(StageArgs), const StageArgs& a, int overlap, int grid, int threads,
                                size_t smem, cudaStream_t s)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

// x, in a way the compiler does not see through: index arithmetic on it is redone
// in every iteration of the batch loop instead of being kept in registers across
// the column phase, which needs them
// (FP64 from p = 4 on, where it is short of registers: p = 4, eight warps, 88 B of
// spills without it)
template <bool ON>
__device__ __forceinline__ int opaque(int x)
{
    if constexpr (ON) asm volatile("" : "+r"(x));
    return x;
}

// contraction tables: with the inverse mass folded in (FP64), or the plain ones
template <typename T> struct ColTab;
template <> struct ColTab<double> {
    static __device__ __forceinline__ const double* B(const StageTables& t) { return t.MB; }
    static __device__ __forceinline__ const double* D(const StageTables& t) { return t.MD; }
};
template <> struct ColTab<float> {
    static __device__ __forceinline__ const float* B(const StageTables& t) { return t.Bf; }
    static __device__ __forceinline__ const float* D(const StageTables& t) { return t.Df; }
};

// entry (q, b) of a table of M x N values that is (anti)symmetric under the
// reversal of both indices: only its first half is read
template <int MN, typename T>
__device__ __forceinline__ T sym(const T* t, int k) { return k < MN / 2 ? t[k] : t[MN - 1 - k]; }
template <int MN, typename T>
__device__ __forceinline__ T asym(const T* t, int k) { return k < MN / 2 ? t[k] : -t[MN - 1 - k]; }

// c + (d x + b y): in FP64 two fused operations, in FP32 rounded as the stage
// kernel's passes round it
__device__ __forceinline__ double add_two(double c, double d, double x, double b, double y) { return fma(d, x, fma(b, y, c)); }
__device__ __forceinline__ float add_two(float c, float d, float x, float b, float y)
{
    return __fadd_rn(c, __fmaf_rn(d, x, __fmul_rn(b, y)));
}

// what a launch of one stage reads and writes (the arguments are passed to every
// function rather than kept by reference: loads of them stay parameter loads)
struct StageIO {
    static __device__ __forceinline__ const double* Us(const StageArgs& a) { return a.Us; }
    static __device__ __forceinline__ const double* U0(const StageArgs& a) { return a.U0; }
    static __device__ __forceinline__ double* acc(const StageArgs& a) { return a.acc; }
    static __device__ __forceinline__ double* out(const StageArgs& a) { return a.out; }
    static __device__ __forceinline__ int mode(const StageArgs& a) { return a.mode; }
    static __device__ __forceinline__ double dt(const StageArgs& a) { return a.dt; }
};
template <int NT>
struct CtaSync {
    __device__ __forceinline__ void operator()() const { cta_sync<NT>(); }
};

// One batch of E elements on NT threads that synchronise through Sync (a whole
// CTA, or the threads of one group of a larger one): thread tid0 of NT, the
// group's shared memory, the stage's buffers through IO.
// GE: general (trilinear) geometry in FP64 -- per-point metric terms, plain tables,
// and the element's dense inverse mass matrix after the contraction.
template <int P, int E, int NT, typename T, typename IO, typename Sync, bool GE = false>
struct Column {
    using L = ColLay<P, T, GE>;
    static_assert(!GE || (sizeof(T) == 8 && E == 1), "general geometry: FP64, one element at a time");
    static constexpr int N = L::N, M = L::M, NB = L::NB, NF = L::NF, N2 = L::N2;
    static constexpr int PS = L::PS, AS = L::AS, X1S = L::X1S, W = L::W, VS = L::VS, SY = L::SY, SZ = L::SZ;
    static constexpr bool F64 = sizeof(T) == 8, kShift = !F64;
    static constexpr int ROWS = E * 5 * N2;            // coefficient rows along x of a batch
    static constexpr int LT = E * 6 * N2;              // its face nodes
    static constexpr int R = (ROWS + NT - 1) / NT, RL = (LT + NT - 1) / NT;
    IO io;
    Sync sync;
    const int tid0;
    double* sRes;                                      // [E][5][VS] (FP32 path, GE)
    double* sM;                                        // [2][N] end columns of the 1D inverse mass
    T* sW;                                             // [E][W]
    T* sL;                                             // [E][6][5][N2] lifts in this element's node order
    T* sSgn;                                           // [E][6] -1 on the left side, +1 on the right
    int* sCls;                                         // [E]
    // the update: out = U0 + cu (acc + k in the last stage, else k), acc' = acc + ca k,
    // with U0 and acc zero where the mode does not read them
    bool need_u0, need_acc, put_acc, sum_acc;
    double cu, ca;
    unsigned status = 0;
    // a batch's coefficient rows and face records
    double un[R][N];
    int cl[R], fl[RL], cls;

    __device__ __forceinline__ Column(const StageArgs& a, IO io_, Sync sync_, int tid, double* smem)
        : io(io_), sync(sync_), tid0(tid)
    {
        sRes = smem;
        sM = sRes + E * L::RES;
        sW = reinterpret_cast<T*>(sM + 2 * N);
        sL = sW + E * W;
        sSgn = sL + E * L::LF;
        sCls = reinterpret_cast<int*>(sSgn + E * 6);
        if (tid0 < 2 * N) sM[tid0] = a.tab.ME[tid0 / N][tid0 % N];
        set_mode(a);
    }

    // after a change of the stage
    __device__ __forceinline__ void set_mode(const StageArgs& a)
    {
        const int mode = io.mode(a);
        need_u0 = mode >= kModeRK1;
        need_acc = mode == kModeRK2 || mode == kModeRK3 || mode == kModeRK4;
        put_acc = mode == kModeRK1 || mode == kModeRK2 || mode == kModeRK3;
        sum_acc = mode == kModeRK4;
        cu = mode == kModeRK1 || mode == kModeRK2 ? 0.5 : (sum_acc ? 1.0 / 6.0 : 1.0);
        ca = mode == kModeRK1 ? 1.0 : 2.0;
    }

    // rows and face records of the batch at e0 into registers (elements past the end repeat the last one)
    __device__ __forceinline__ void fetch(const StageArgs& a, int e0)
    {
        cls = a.geo_class[min(e0 + min(tid0, E - 1), a.ne - 1)];
        const int tid = opaque<F64 && P >= 4>(tid0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = tid + r * NT;
            if (i < ROWS) {
                const int e = i / (5 * N2), row = i - e * (5 * N2), ge = min(e0 + e, a.ne - 1);
                load_row<N>(io.Us(a) + ((size_t)ge * 5 * N2 + row) * N, un[r]);
                if constexpr (kShift) cl[r] = a.geo_class[ge];
            }
        }
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            const int i = tid + r * NT;
            if (i < LT) {
                const int f = (i / N2) % 6, e = i / (6 * N2);
                fl[r] = a.lrec[(size_t)min(e0 + e, a.ne - 1) * 6 + f];
            }
        }
    }

    // the fetched batch's geometry classes
    __device__ __forceinline__ void classes()
    {
        if (tid0 < E) sCls[tid0] = cls;
    }

    // the batch's face lifts on their way into shared memory
    __device__ __forceinline__ void lifts(const StageArgs& a, int e0)
    {
        const T* gL = reinterpret_cast<const T*>(a.fflux);
        const int tid = opaque<F64 && P >= 4>(tid0);
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            const int i = tid + r * NT;
            if (i < LT) {
                const int c = i % N2, f = (i / N2) % 6, e = i / (6 * N2);
                const int ge = min(e0 + e, a.ne - 1);
                const int pc = ((fl[r] >> 30) & 1) ? c : a.cmapn[(a.frec[(size_t)ge * 6 + f].info >> 4) * N2 + c];
                const T* src = gL + (size_t)(fl[r] & 0x3fffffff) * a.fstride + pc;
                T* dst = sL + e * L::LF + f * 5 * N2 + c;
#pragma unroll
                for (int v = 0; v < 5; ++v) cp_async_t(dst + v * N2, src + v * N2);
                if (c == 0) sSgn[e * 6 + f] = fl[r] < 0 ? T(-1) : T(1);
            }
        }
        classes();
        cp_async_commit();
    }

    // x interpolation of the fetched rows
    __device__ __forceinline__ void interp_x(const StageArgs& a)
    {
        const T* __restrict__ Bt = TabSel<T>::B(a.tab);
        const int tid = opaque<F64 && P >= 4>(tid0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = tid + r * NT;
            if (i < ROWS) {
                const int e = i / (5 * N2), row = i - e * (5 * N2), v = row / N2, byz = row - v * N2;
                const double sh = kShift && v == 4 ? a.geo[cl[r]].eref : 0.0;
                T u[N];
#pragma unroll
                for (int b = 0; b < N; ++b) u[b] = kShift ? T(un[r][b] - sh) : T(un[r][b]);
                T* o = sW + e * W + 5 * AS + v * X1S + byz * M;
#pragma unroll
                for (int q = 0; q < M; ++q) {
                    T s = T(0);
#pragma unroll
                    for (int b = 0; b < N; ++b) s += sym<M * N>(Bt, q * N + b) * u[b];
                    o[q] = s;
                }
            }
        }
    }

    // y interpolation, then per quadrature column the z interpolation, flux and z contraction
    __device__ __forceinline__ void columns(const StageArgs& a, int e0)
    {
        const T* __restrict__ Bt = TabSel<T>::B(a.tab);
        const T* __restrict__ Wt = TabSel<T>::W(a.tab);
        const T* __restrict__ Ct = ColTab<T>::B(a.tab);
        const T* __restrict__ Dt = ColTab<T>::D(a.tab);
        const T gamma = T(a.gamma);
        const int tid = opaque<F64 && P >= 5>(tid0);
        sync();
        // ---- y interpolation ----
#pragma unroll 1
        for (int i = tid; i < E * 5 * N * M; i += NT) {
            const int e = i / (5 * N * M);
            int v, qx, bz;
            task3<L::oy, 5, M, N>(i - e * (5 * N * M), v, qx, bz);
            const T* x1 = sW + e * W + 5 * AS + v * X1S + bz * N * M + qx;
            T col[N];
#pragma unroll
            for (int b = 0; b < N; ++b) col[b] = x1[b * M];
            T* o = sW + e * W + v * AS + bz * PS + qx;
#pragma unroll
            for (int q = 0; q < M; ++q) {
                T s = T(0);
#pragma unroll
                for (int b = 0; b < N; ++b) s += sym<M * N>(Bt, q * N + b) * col[b];
                o[q * M] = s;
            }
        }
        sync();
        // ---- columns: z interpolation, flux, z contraction in registers ----
#pragma unroll 1
        for (int i = tid; i < E * NF; i += NT) {
            const int e = i / NF, qxy = i - e * NF;
            T* col = sW + e * W + qxy;
            T S[5][M];  // rho, momenta, energy (then enthalpy rE + P) at the column's points
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                T x[N];
#pragma unroll
                for (int b = 0; b < N; ++b) x[b] = col[v * AS + b * PS];
#pragma unroll
                for (int q = 0; q < M; ++q) {
                    T s = T(0);
#pragma unroll
                    for (int b = 0; b < N; ++b) s += sym<M * N>(Bt, q * N + b) * x[b];
                    S[v][q] = s;
                }
            }
            const GeoDev* geo = a.geo + sCls[e];
            const T hr = kShift ? T(a.gamma * geo->eref) : T(0);
            const T pref = kShift ? T((a.gamma - 1.0) * geo->eref) : T(0);
            T vel[3][M], p[M];
            bool sound = true;
#pragma unroll
            for (int q = 0; q < M; ++q) {
                // P = (gamma-1) (rE - |m|^2 / (2 rho)), as dgp::interior_flux_r1
                const T r1 = T(1.) / S[0][q];
                p[q] = (gamma - T(1.0)) * (S[4][q] - T(0.5) * ((S[1][q] * S[1][q] + S[2][q] * S[2][q] + S[3][q] * S[3][q]) * r1));
#pragma unroll
                for (int d = 0; d < 3; ++d) vel[d][q] = S[1 + d][q] * r1;
                sound = sound && S[0][q] > T(0) && p[q] + pref > T(0);  // a NaN is not
                S[4][q] = kShift ? S[4][q] + p[q] + hr : S[4][q] + p[q];
            }
            if (!sound) {
#pragma unroll
                for (int q = 0; q < M; ++q) {
                    if (!(S[0][q] > T(0))) status |= kStatusRho;
                    if (!(p[q] + pref > T(0))) status |= kStatusPressure;
                    if (S[0][q] != S[0][q] || p[q] != p[q]) status |= kStatusNaN;
                }
            }
            // GE: entry k of the metric terms at point q of the column
            auto metric = [&](int k, int q) { return a.gjd[((size_t)min(e0 + e, a.ne - 1) * 9 + k) * (M * NF) + q * NF + qxy]; };
            T JD[9];
            if constexpr (!GE) {
#pragma unroll
                for (int k = 0; k < 9; ++k) JD[k] = T(geo->JD[k]);
            }
            const T wxy = Wt[qxy % M] * Wt[qxy / M];
            // contract the components g_d(v, q) of each variable along z
            auto contract = [&](auto&& component) {
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    T a0[N], a1[N], a2[N];
#pragma unroll
                    for (int b = 0; b < N; ++b) { a0[b] = T(0); a1[b] = T(0); a2[b] = T(0); }
#pragma unroll
                    for (int q = 0; q < M; ++q) {
                        T g[3];
                        component(v, q, g);
#pragma unroll
                        for (int b = 0; b < N; ++b) {
                            a0[b] += sym<M * N>(Ct, q * N + b) * g[0];
                            a1[b] += sym<M * N>(Ct, q * N + b) * g[1];
                            a2[b] += asym<M * N>(Dt, q * N + b) * g[2];
                        }
                    }
#pragma unroll
                    for (int b = 0; b < N; ++b) {
                        col[(3 * v + 0) * AS + b * PS] = a0[b];
                        col[(3 * v + 1) * AS + b * PS] = a1[b];
                        col[(3 * v + 2) * AS + b * PS] = a2[b];
                    }
                }
            };
            if constexpr (F64) {
                // S[v] V_d (+ P JD[d][v-1] for a momentum) with the weighted
                // contravariant velocities V_d = w JD[d] . u
#pragma unroll
                for (int q = 0; q < M; ++q) {
                    const T wq = wxy * Wt[q], u = vel[0][q], v = vel[1][q], w = vel[2][q];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        if constexpr (GE) vel[d][q] = (u * metric(d * 3, q) + v * metric(d * 3 + 1, q) + w * metric(d * 3 + 2, q)) * wq;
                        else vel[d][q] = (u * JD[d * 3 + 0] + v * JD[d * 3 + 1] + w * JD[d * 3 + 2]) * wq;
                    }
                    p[q] *= wq;
                }
                contract([&](int v, int q, T (&g)[3]) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        g[d] = S[v][q] * vel[d][q];
                        if (v >= 1 && v <= 3) g[d] += p[q] * (GE ? metric(d * 3 + v - 1, q) : JD[d * 3 + v - 1]);
                    }
                });
            } else {
                // the stage kernel's operations in its order (the same bits):
                // (F_0 JD[d][0] + F_1 JD[d][1] + F_2 JD[d][2]) w
                auto flux = [&](int v, int q, T (&F)[3]) {
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        F[d] = v == 0 ? S[1 + d][q] : (v == 1 + d ? S[v][q] * vel[d][q] + p[q] : S[v][q] * vel[d][q]);
                };
                if (JD[1] == T(0) && JD[2] == T(0) && JD[3] == T(0) && JD[5] == T(0) && JD[6] == T(0) && JD[7] == T(0))
                    contract([&](int v, int q, T (&g)[3]) {  // axis-parallel element: the other products are zeros
                        T F[3];
                        flux(v, q, F);
                        const T wq = wxy * Wt[q];
#pragma unroll
                        for (int d = 0; d < 3; ++d) g[d] = (F[d] * JD[d * 4]) * wq;
                    });
                else
                    contract([&](int v, int q, T (&g)[3]) {
                        T F[3];
                        flux(v, q, F);
                        const T wq = wxy * Wt[q];
#pragma unroll
                        for (int d = 0; d < 3; ++d) g[d] = (F[0] * JD[d * 3 + 0] + F[1] * JD[d * 3 + 1] + F[2] * JD[d * 3 + 2]) * wq;
                    });
            }
        }
        sync();
    }

    __device__ __forceinline__ void contract_y(const StageArgs& a)
    {
        const T* __restrict__ Ct = ColTab<T>::B(a.tab);
        const T* __restrict__ Dt = ColTab<T>::D(a.tab);
        const int tid = opaque<F64 && P >= 4>(tid0);
        // ---- y contraction: By^T A0 over row 3v, Dy^T A1 + By^T A2 over row 3v+1 ----
#pragma unroll 1
        for (int i = tid; i < E * 5 * N * M; i += NT) {
            const int e = i / (5 * N * M);
            int v, qx, bz;
            task3<L::oyc, 5, M, N>(i - e * (5 * N * M), v, qx, bz);
            T* A0 = sW + e * W + (3 * v) * AS + bz * PS + qx;
            T c0[N], c12[N];
#pragma unroll
            for (int b = 0; b < N; ++b) { c0[b] = T(0); c12[b] = T(0); }
#pragma unroll
            for (int q = 0; q < M; ++q) {
                const T x0 = A0[q * M], x1 = A0[AS + q * M], x2 = A0[2 * AS + q * M];
#pragma unroll
                for (int b = 0; b < N; ++b) {
                    c0[b] += sym<M * N>(Ct, q * N + b) * x0;
                    c12[b] = add_two(c12[b], asym<M * N>(Dt, q * N + b), x1, sym<M * N>(Ct, q * N + b), x2);
                }
            }
#pragma unroll
            for (int b = 0; b < N; ++b) {
                A0[b * M] = c0[b];
                A0[AS + b * M] = c12[b];
            }
        }
    }

    // GE: the element's dense inverse mass matrix, streamed from global memory, and
    // the stage update; a thread's rows (two with 16-byte loads where their number
    // is even) of all five variables
    __device__ __forceinline__ void dense_inverse_mass(const StageArgs& a, int e0)
    {
        constexpr int V2 = NB % 2 == 0 ? 2 : 1, RP = NB / V2;
        const size_t ge = e0;
        const double scale = io.dt(a) * a.geo[sCls[0]].dtf;
#pragma unroll 1
        for (int rp = tid0; rp < RP; rp += NT) {
            const double* im = a.gimm + ge * NB * NB + V2 * rp;  // iMM[V2 rp + i][k] at im[k NB + i]
            double s[V2][5] = {};
            for (int kz = 0; kz < N; ++kz)
#pragma unroll
                for (int kyx = 0; kyx < N2; ++kyx) {
                    double m[V2];
                    load_row<V2>(im + (size_t)(kz * N2 + kyx) * NB, m);
                    const double* r = sRes + kz * SZ + (kyx / N) * SY + kyx % N;
#pragma unroll
                    for (int v = 0; v < 5; ++v)
#pragma unroll
                        for (int i = 0; i < V2; ++i) s[i][v] += m[i] * r[v * VS];
                }
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                const size_t g = (ge * 5 + v) * NB + V2 * rp;
                double u0[V2] = {}, ac[V2] = {}, o[V2], ao[V2];
                if (need_u0) load_row<V2>(io.U0(a) + g, u0);
                if (need_acc) load_row<V2>(io.acc(a) + g, ac);
#pragma unroll
                for (int i = 0; i < V2; ++i) {
                    const double k = scale * s[i][v];
                    ao[i] = ac[i] + ca * k;
                    o[i] = u0[i] + cu * (sum_acc ? ac[i] + k : k);
                }
                if (put_acc) store_row<V2>(io.acc(a) + g, ao);
                store_row<V2>(io.out(a) + g, o);
            }
        }
    }

    // x contraction, face lifts, inverse mass (FP32 path) and stage update
    __device__ __forceinline__ void finish(const StageArgs& a, int e0)
    {
        const T* __restrict__ Ct = ColTab<T>::B(a.tab);
        const T* __restrict__ Dt = ColTab<T>::D(a.tab);
        [[maybe_unused]] const double* __restrict__ Mi = a.tab.Minv;
        const int tid = opaque<F64 && P >= 4>(tid0);
        // ---- x contraction, face lifts; FP64: the stage update ----
#pragma unroll 1
        for (int i = tid; i < ROWS; i += NT) {
            const int e = i / (5 * N2), row = i - e * (5 * N2), v = row / N2, byz = row - v * N2;
            const int by = byz % N, bz = byz / N;
            const size_t g = ((size_t)min(e0 + e, a.ne - 1) * 5 * N2 + row) * N;
            double u0[N] = {}, ac[N] = {};
            if constexpr (F64 && !GE) {
                if (need_u0) load_row<N>(io.U0(a) + g, u0);
                if (need_acc) load_row<N>(io.acc(a) + g, ac);
            }
            const T* C0 = sW + e * W + (3 * v) * AS + bz * PS + by * M;
            T x[N];
#pragma unroll
            for (int b = 0; b < N; ++b) x[b] = T(0);
#pragma unroll
            for (int q = 0; q < M; ++q) {
                const T c0 = C0[q], c12 = C0[AS + q];
#pragma unroll
                for (int b = 0; b < N; ++b) x[b] = add_two(x[b], asym<M * N>(Dt, q * N + b), c0, sym<M * N>(Ct, q * N + b), c12);
            }
            // lifts: faces 4 / 2 at the row's ends, 1 / 3 and 0 / 5 along it
            const T* Lv = sL + e * L::LF + v * N2;
            const T* sg = sSgn + e * 6;
            if constexpr (F64 && !GE) {
                const double l4 = sg[4] * Lv[4 * 5 * N2 + byz], l2 = sg[2] * Lv[2 * 5 * N2 + byz];
                const double c1 = sg[1] * sM[by], c3 = sg[3] * sM[N + by], c0 = sg[0] * sM[bz], c5 = sg[5] * sM[N + bz];
                const double* L1 = Lv + 1 * 5 * N2 + bz * N;
                const double* L3 = Lv + 3 * 5 * N2 + bz * N;
                const double* L0 = Lv + by * N;
                const double* L5 = Lv + 5 * 5 * N2 + by * N;
                const double scale = io.mode(a) == kModeResidual ? 1.0 : io.dt(a) * a.geo[sCls[e]].dtf * a.geo[sCls[e]].inv_djac;
                double k[N];
#pragma unroll
                for (int b = 0; b < N; ++b) {
                    double s = x[b];
                    s += a.tab.ME[0][b] * l4;
                    s += a.tab.ME[1][b] * l2;
                    s += c1 * L1[b];
                    s += c3 * L3[b];
                    s += c0 * L0[b];
                    s += c5 * L5[b];
                    k[b] = scale * s;
                }
                if (e0 + e >= a.ne) continue;
                if (put_acc) {
                    double ao[N];
#pragma unroll
                    for (int b = 0; b < N; ++b) ao[b] = ac[b] + ca * k[b];
                    store_row<N>(io.acc(a) + g, ao);
                }
                double o[N];
#pragma unroll
                for (int b = 0; b < N; ++b) o[b] = u0[b] + cu * (sum_acc ? ac[b] + k[b] : k[b]);
                store_row<N>(io.out(a) + g, o);
            } else {
                // the node's faces summed in face order (0, 1, 2, 3, 4, 5); a row meets at
                // most one y face (1 or 3) and one z face (0 or 5), its ends faces 4 and 2
                const bool y0 = by == 0, y1 = by == N - 1, z0 = bz == 0, z1 = bz == N - 1;
                const T* Ly = Lv + (y1 ? 3 : 1) * 5 * N2 + bz * N;
                const T* Lz = Lv + (z1 ? 5 : 0) * 5 * N2 + by * N;
                const T sy = y0 || y1 ? sg[y1 ? 3 : 1] : T(0), sz = z0 || z1 ? sg[z1 ? 5 : 0] : T(0);
                const double l4 = double(sg[4] * Lv[4 * 5 * N2 + byz]), l2 = double(sg[2] * Lv[2 * 5 * N2 + byz]);
                double t[N];
#pragma unroll
                for (int b = 0; b < N; ++b) {
                    const double ly = sy == T(0) ? 0.0 : double(sy * Ly[b]), lz = sz == T(0) ? 0.0 : double(sz * Lz[b]);
                    double s;
                    if (b == 0) s = ((z0 ? lz : 0.0) + ly + l4) + (z0 ? 0.0 : lz);
                    else if (b == N - 1) s = ((z0 ? lz : 0.0) + (y0 ? ly : 0.0) + l2) + (y0 ? 0.0 : ly) + (z0 ? 0.0 : lz);
                    else s = lz + ly;
                    t[b] = double(x[b]) + s;
                }
                if (io.mode(a) == kModeResidual) {
                    if (e0 + e < a.ne) store_row<N>(io.out(a) + ((size_t)(e0 + e) * 5 * N2 + row) * N, t);
                    continue;
                }
                double* res = sRes + e * L::RES + v * VS;
                if constexpr (GE) {
#pragma unroll
                    for (int j = 0; j < N; ++j) res[bz * SZ + by * SY + j] = t[j];
                    continue;
                }
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    double s = 0.0;
#pragma unroll
                    for (int k = 0; k < N; ++k) s += Mi[j * N + k] * t[k];
                    res[bz * SZ + by * SY + j] = s;
                }
            }
        }
        if constexpr (GE) {
            if (io.mode(a) != kModeResidual) {
                sync();
                dense_inverse_mass(a, e0);
            }
        }
        if constexpr (!F64) {
            if (io.mode(a) != kModeResidual) {
                // ---- FP64 inverse mass along y, then z fused with the update ----
                sync();
#pragma unroll 1
                for (int i = tid; i < ROWS; i += NT) {
                    const int e = i / (5 * N2);
                    const int r = i - e * (5 * N2), v = r / N2, bx = r % N, bz = (r / N) % N;
                    double* res = sRes + e * L::RES + v * VS;
                    double t[N];
#pragma unroll
                    for (int k = 0; k < N; ++k) t[k] = res[bz * SZ + k * SY + bx];
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        double s = 0.0;
#pragma unroll
                        for (int k = 0; k < N; ++k) s += Mi[j * N + k] * t[k];
                        res[bz * SZ + j * SY + bx] = s;
                    }
                }
                sync();
#pragma unroll 1
                for (int i = tid; i < ROWS; i += NT) {
                    const int e = i / (5 * N2), row = i - e * (5 * N2), v = row / N2, bxy = row - v * N2;
                    if (e0 + e >= a.ne) continue;
                    const size_t g0 = ((size_t)(e0 + e) * 5 + v) * NB + bxy;
                    double u0[N] = {}, ac[N] = {};
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        if (need_u0) u0[k] = io.U0(a)[g0 + k * N2];
                        if (need_acc) ac[k] = io.acc(a)[g0 + k * N2];
                    }
                    const int bx = bxy % N, by = bxy / N;
                    const GeoDev& gg = a.geo[sCls[e]];
                    const double scale = io.dt(a) * gg.dtf * gg.inv_djac;
                    const double* res = sRes + e * L::RES + v * VS;
                    double t[N];
#pragma unroll
                    for (int k = 0; k < N; ++k) t[k] = res[k * SZ + by * SY + bx];
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        double s = 0.0;
#pragma unroll
                        for (int k = 0; k < N; ++k) s += Mi[j * N + k] * t[k];
                        const double kk = scale * s;
                        const size_t g = g0 + (size_t)j * N2;
                        if (put_acc) io.acc(a)[g] = ac[j] + ca * kk;
                        io.out(a)[g] = u0[j] + cu * (sum_acc ? ac[j] + kk : kk);
                    }
                }
            }
        }
    }
};

template <int P, int E, int NT, typename T, int MB, bool GE = false>
__global__ void __launch_bounds__(NT, MB) column_kernel(const __grid_constant__ StageArgs a)
{
    extern __shared__ double csm[];
    constexpr int NB = ColLay<P, T>::NB;
    Column<P, E, NT, T, StageIO, CtaSync<NT>, GE> c(a, StageIO(), CtaSync<NT>(), threadIdx.x, csm);
    const int tid = threadIdx.x;
    const int stride = gridDim.x * E;
    int e0 = a.e_begin + blockIdx.x * E;
    if constexpr (column_overlaps<P, T>()) wait_prerequisites();  // the face kernel's lifts, and through it the stage before
    if (e0 < a.ne) c.fetch(a, e0);
    for (; e0 < a.ne; e0 += stride) {
        // this batch's RK operands (read by the last pass) and the next batch's rows on
        // their way into L2
        if (tid < 3 && (tid == 0 ? e0 + stride < a.ne : tid == 1 ? c.need_u0 && a.U0 != a.Us : c.need_acc)) {
            const int ep = tid == 0 ? e0 + stride : e0;
            prefetch_l2((tid == 0 ? a.Us : tid == 1 ? a.U0 : a.acc) + (size_t)ep * 5 * NB, min(E, a.ne - ep) * 5 * NB);
        }
        c.lifts(a, e0);
        c.interp_x(a);
        c.columns(a, e0);
        // the next batch's rows and records, in flight during the contractions (past
        // the end the last element's: a condition would keep the old rows alive)
        c.fetch(a, e0 + stride);
        // the element's inverse mass matrix, towards L2 (p = 3, 18^3: 107 -> 100 us a stage)
        if constexpr (GE)
            if (tid == 0) prefetch_l2(a.gimm + (size_t)e0 * NB * NB, NB * NB);
        c.contract_y(a);
        cp_async_wait_all();  // the lifts have landed
        cta_sync<NT>();
        c.finish(a, e0);
        cta_sync<NT>();  // the point array and the lifts are the next batch's
    }
    if (c.status) atomicOr(a.status, c.status);
}

// ---------------------------------------------------------------------------
// the face kernel with the lift, per batch of FB faces:
//   gather   both sides' boundary slices by cp.async into shared memory, one lane
//            per slice entry (a warp takes whole sides, so neighbouring lanes read
//            neighbouring coefficients), while the batch before computes its
//            fluxes and lifts;
//   traces   one task per slice (2D interpolation in registers);
//   flux     one task per point of the listed side's face grid, in the
//            reference's L/R convention, weighted, over that side's trace;
//   lift     L[b1][b0] = sum_t1 C[t1][b1] sum_t0 C[t0][b0] F[t1][t0] (C = B Minv
//            in FP64, B in FP32), one task per (face, variable, output column).
// Three buffers of face descriptors: the batch's, the next one's (for its
// gather) and the one after that in flight.
//
// Bound by its FP64 chains and shared-memory wavefronts at 16-18 warps per SM (FP64 pipe
// 48 %, LSU wavefronts 71 %). One thread per slice used to read its 16 strided coefficients, 32
// cache lines to a load (79 % of the load pipe): 40^3, p = 3, FP64 0.207 -> 0.172
// ms with the cooperative gather; descriptors, three square roots and one-warp
// CTAs bring the RK stage of 48^3 from 0.845 to 0.821 ms.
template <int P, typename T, int FB>
struct FaceLay {
    // the cooperative gather pays from p = 3 on; a slice of 4 or 9 coefficients
    // is read by its trace task itself (p = 1, 72^3, FP64: stage 0.727 against
    // 0.781 ms; p = 2, 60^3, mixed: 0.774 against 0.835 ms)
    static constexpr bool COOP = P >= 3;
    static constexpr int N = P + 1, M = P + 2, NF = M * M, N2 = N * N;
    static constexpr int FS = odd(NF), NS = odd(N2);       // trace and slice strides
    static constexpr size_t tr_bytes = (sizeof(T) * FB * 10 * FS + 15) / 16 * 16;
    static constexpr size_t sl_bytes = COOP ? (sizeof(double) * FB * 10 * NS + 15) / 16 * 16 : 0;
    static constexpr size_t bytes = tr_bytes + sl_bytes + 3 * FB * sizeof(FaceDesc);
};

// the phases of a batch of nf <= FB faces on NT threads; a synchronisation of the
// threads belongs between any two of them
template <int P, typename T, int FB, int NT>
struct FacePhases {
    using L = FaceLay<P, T, FB>;
    static constexpr int N = L::N, M = L::M, NB = N * N * N, NF = L::NF, N2 = L::N2, FS = L::FS, NS = L::NS;
    static constexpr bool kShift = sizeof(T) == 4;

    // the faces' slices (cp.async)
    static __device__ __forceinline__ void gather(const double* Us, const FaceDesc* sD, int nf, double* sSl, int tid)
    {
        for (int sj = tid / 32; sj < 2 * FB; sj += NT / 32) {
            if (sj >= 2 * nf) break;
            const FaceDesc& fd = sD[sj / 2];
            const int st = fd.strides >> (16 * (sj % 2)), s0 = st & 255, s1 = (st >> 8) & 255;
            const double* src = Us + fd.base[sj % 2];
            double* dst = sSl + sj * 5 * NS;
#pragma unroll
            for (int r = 0; r < (5 * N2 + 31) / 32; ++r) {
                const int i = tid % 32 + 32 * r, v = i / N2, c = i - v * N2;
                if (i < 5 * N2) cp_async8(dst + v * NS + c, src + v * NB + (c % N) * s0 + (c / N) * s1);
            }
        }
    }

    // both sides' traces, in the listed side's energy frame
    static __device__ __forceinline__ void traces(const StageArgs& a, const double* Us, const FaceDesc* sD, int nf,
                                                  const double* sSl, T* sTr, int tid)
    {
        const T* __restrict__ Bt = TabSel<T>::B(a.tab);
        for (int t = tid; t < FB * 10; t += NT) {
            if (t >= nf * 10) break;
            const FaceDesc& fd = sD[t / 10];
            const double sh = kShift && t % 5 == 4 ? a.geo[fd.cls].eref : 0.0;
            const double* s = sSl + t * NS;
            int s0 = 1, s1 = N;
            if constexpr (!L::COOP) {
                const int side = (t / 5) % 2, st = fd.strides >> (16 * side);
                s = Us + fd.base[side] + (t % 5) * NB;
                s0 = st & 255;
                s1 = (st >> 8) & 255;
            }
            double x[N][N];
#pragma unroll
            for (int b1 = 0; b1 < N; ++b1)
#pragma unroll
                for (int b0 = 0; b0 < N; ++b0) x[b1][b0] = s[b0 * s0 + b1 * s1];
            T sl[N][N];
#pragma unroll
            for (int b1 = 0; b1 < N; ++b1)
#pragma unroll
                for (int b0 = 0; b0 < N; ++b0) sl[b1][b0] = kShift ? T(x[b1][b0] - sh) : T(x[b1][b0]);
            interp2d<N, M, T>(Bt, sl, sTr + t * FS);
        }
    }

    // the flux at the listed side's face points, over that side's trace (GEO: with the
    // normal data of each point)
    template <bool GEO = false>
    static __device__ __forceinline__ void flux(const StageArgs& a, const FaceDesc* sD, int nf, T* sTr, unsigned& status, int tid)
    {
        const T* __restrict__ Wt = TabSel<T>::W(a.tab);
        for (int i = tid; i < FB * NF; i += NT) {
            const int c = i % NF, j = i / NF;
            if (j >= nf) continue;
            const FaceDesc& fd = sD[j];
            const int cn = a.cmap[(fd.info >> 4) * NF + c];
            const int isL = (fd.info >> 3) & 1;
            T* To = sTr + (j * 2) * 5 * FS;
            const T* Tn = To + 5 * FS;
            T UL[5], UR[5], Fo[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                const T uo = To[v * FS + c], un = Tn[v * FS + cn];
                UL[v] = isL ? uo : un;
                UR[v] = isL ? un : uo;
            }
            T nd[4] = {T(fd.n[0]), T(fd.n[1]), T(fd.n[2]), T(fd.nmag)};
            if constexpr (GEO) {
#pragma unroll
                for (int k = 0; k < 4; ++k) nd[k] = T(a.gnrm[((size_t)fd.side * 4 + k) * NF + c]);
            }
            const double eref = kShift ? a.geo[fd.cls].eref : 0.0;
            bool done = false;
            if constexpr (!kShift) {
                done = a.flux == 0;
                if (done) dgp::flux_lax_friedrichs_sq(a.gamma, UL, UR, nd, nd[3], Fo);
            }
            if (!done) numerical_flux<T, kShift>(a.flux, a.gamma, UL, UR, nd, eref, Fo, status);
            const T w = Wt[c % M] * Wt[c / M];
#pragma unroll
            for (int v = 0; v < 5; ++v) To[v * FS + c] = Fo[v] * w;
        }
    }

    // the lifts of faces f0 .. f0 + nf - 1
    static __device__ __forceinline__ void lift(const StageArgs& a, int f0, int nf, const T* sTr, int tid)
    {
        const T* __restrict__ Ct = ColTab<T>::B(a.tab);
        T* out = reinterpret_cast<T*>(a.fflux);
        for (int t = tid; t < FB * 5 * N; t += NT) {
            const int b0 = t % N, jv = t / N, v = jv % 5, j = jv / 5;
            if (j >= nf) continue;
            const T* F = sTr + (j * 2) * 5 * FS + v * FS;
            T r[M];
#pragma unroll
            for (int t1 = 0; t1 < M; ++t1) {
                T s = T(0);
#pragma unroll
                for (int t0 = 0; t0 < M; ++t0) s += Ct[t0 * N + b0] * F[t1 * M + t0];
                r[t1] = s;
            }
            T* o = out + (size_t)(f0 + j) * a.fstride + v * N2 + b0;
#pragma unroll
            for (int b1 = 0; b1 < N; ++b1) {
                T s = T(0);
#pragma unroll
                for (int t1 = 0; t1 < M; ++t1) s += Ct[t1 * N + b1] * r[t1];
                o[b1 * N] = s;
            }
        }
    }
};

template <int P, typename T, int FB, int NT, int MB, bool GEO = false>
__global__ void __launch_bounds__(NT, MB) face_lift_kernel(const __grid_constant__ StageArgs a)
{
    using L = FaceLay<P, T, FB>;
    using F = FacePhases<P, T, FB, NT>;
    extern __shared__ __align__(16) unsigned char fraw[];
    T* sTr = reinterpret_cast<T*>(fraw);                              // [FB][2][5][FS]
    double* sSl = reinterpret_cast<double*>(fraw + L::tr_bytes);      // [FB][2][5][NS]
    FaceDesc* sDesc = reinterpret_cast<FaceDesc*>(fraw + L::tr_bytes + L::sl_bytes);  // [3][FB]
    const int tid = threadIdx.x;
    unsigned status = 0;
    const int fstep = gridDim.x * FB;
    // the descriptors of batch f (the last face repeated past the end)
    auto fetch = [&](int f, int slot) {
        if (f < a.nface)
            for (int i = tid; i < FB * 4; i += NT) {
                const int j = i / 4, w = i % 4;
                cp_async16(reinterpret_cast<char*>(sDesc + slot * FB + j) + 16 * w,
                           reinterpret_cast<const char*>(a.fdesc + min(f + j, a.nface - 1)) + 16 * w);
            }
    };
    auto gather = [&](int f, int slot) {
        if (L::COOP && f < a.nface) F::gather(a.Us, sDesc + slot * FB, FB, sSl, tid);
    };
    int f0 = a.face_begin + blockIdx.x * FB;
    if (f0 < a.nface) {
        fetch(f0, 0);
        fetch(f0 + fstep, 1);
        cp_async_commit();
        cp_async_wait_all();
        cta_sync<NT>();
    }
    wait_prerequisites();  // the descriptors do not change, the state does
    if (f0 < a.nface) {
        gather(f0, 0);
        cp_async_commit();
    }
    int slot = 0;
    for (; f0 < a.nface; f0 += fstep) {
        const FaceDesc* sD = sDesc + slot * FB;
        const int next = slot == 2 ? 0 : slot + 1, after = next == 2 ? 0 : next + 1;
        const int nf = min(FB, a.nface - f0);
        cp_async_wait_all();  // this batch's slices, the next one's descriptors
        cta_sync<NT>();
        fetch(f0 + 2 * fstep, after);
        F::traces(a, a.Us, sD, FB, sSl, sTr, tid);
        cta_sync<NT>();
        gather(f0 + fstep, next);
        cp_async_commit();
        F::template flux<GEO>(a, sD, nf, sTr, status, tid);
        cta_sync<NT>();
        F::lift(a, f0, nf, sTr, tid);
        slot = next;
    }
    cp_async_wait_all();
    if (status) atomicOr(a.status, status);
}

template <int P, int E, int NT, typename T, int MB, bool GE>
cudaError_t launch_column(const StageArgs& a, int grid, cudaStream_t s)
{
    return launch_after(column_kernel<P, E, NT, T, MB, GE>, a, column_overlaps<P, T>() && a.column_overlaps, grid, NT,
                        ColLay<P, T, GE>::bytes(E), s);
}
template <int P, typename T, int FB, int NT, int MB, bool GE>
cudaError_t launch_face_lift(const StageArgs& a, int grid, cudaStream_t s)
{
    return launch_after(face_lift_kernel<P, T, FB, NT, MB, GE>, a, a.face_overlaps, grid, NT, FaceLay<P, T, FB>::bytes, s);
}

// E elements and NT threads per CTA, at least MB resident CTAs per SM asked of the
// compiler; the default from min_per_sm elements per SM on.
// The face kernel's batch FB on FNT threads (FMB resident CTAs asked of the
// compiler) is the measured best of batches of 2 .. 20 faces on 32 .. 256 threads:
// small CTAs, whose barriers hold few warps, as long as one round of threads
// covers most of the slices and points. GE: general geometry.
template <int P, int E, int NT, typename T, int MB, int FB, int FNT, int FMB, bool GE = false>
StageVariant make_column_variant(int min_per_sm)
{
    using CL = ColLay<P, T, GE>;
    static_assert(CL::bytes(E) <= 227 * 1024, "column kernel shared memory exceeds 227 KB");
    static_assert(FaceLay<P, T, FB>::bytes <= 227 * 1024, "face kernel shared memory exceeds 227 KB");
    StageVariant v{E, NT, 1, sizeof(T) == 4 ? 1 : 0, kSB | kFX | kCF | (GE ? kGE : 0), CL::bytes(E),
                   (const void*)column_kernel<P, E, NT, T, MB, GE>, launch_column<P, E, NT, T, MB, GE>};
    v.min_per_sm = min_per_sm;
    v.face_func = (const void*)face_lift_kernel<P, T, FB, FNT, FMB, GE>;
    v.face_smem = FaceLay<P, T, FB>::bytes;
    v.face_threads = FNT;
    v.face_launch = launch_face_lift<P, T, FB, FNT, FMB, GE>;
    v.face_batch = FB;
    return v;
}

}  // namespace dgk
