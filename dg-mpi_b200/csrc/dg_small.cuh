// dg_small.cuh -- RK4 steps of a small affine mesh in one cooperative launch.
//
// A mesh of a few hundred elements leaves most of the chip idle, and its steps
// take the latency of eight dependent launches each (4^3, p = 3, HLLC: 18 us a
// stage, of which the arithmetic is a few).  small_steps_kernel keeps the whole
// mesh resident -- every element has its own group of threads, so there are no
// batches -- and runs all stages of all steps of a call:
//
//   column groups   x, y, z interpolation, flux and contraction of their element
//       up to the y contraction, which need its own state only; then, once the
//       stage's lifts are there, the x contraction and the update;
//   face warps      the stage's lifted fluxes, at the same time.
//
// Two counters in global memory order them: faces start when every block has
// finished the stage before (they read neighbours' states), column groups finish
// when every block has written its lifts.  The launch is cooperative (all blocks
// resident, so every wait ends); each wait is bounded all the same, and one that
// gives up reports kStatusTimeout and ends the kernel.
//
// The arithmetic is Column's and FacePhases': the bits of the two-launch form.
//
// Bound by the latency of one stage's dependent phases.  Stage time, two-launch
// form -> this kernel (FP64, Lax-Friedrichs): 4^3 elements p = 1 7.7 -> 5.2, p = 2
// 11.3 -> 5.8, p = 3 11.3 -> 6.9, p = 4 12.8 -> 8.5, p = 5 18.0 -> 10.2 us; 8^3
// p = 1 7.7 -> 5.5, p = 2 11.3 -> 6.8, p = 3 12.2 -> 9.2 us.  Two threads' worth of
// warps per element where registers allow it (p = 3: 64 threads, 6.9 against 7.6 us
// with 32), and as many face warps as column warps need not wait for; at the
// sizes where an SM would hold more elements than the variants allow, the
// two-launch form is as fast (9^3, p = 3: 12.8 against 13.9 us).
#pragma once
#include "dg_column.cuh"
#include "dg_tc.cuh"

namespace dgk {

struct SmallArgs {
    StageArgs a;          // tables, geometry, U0, acc, fflux; Us, out and mode unused
    double *Ua, *Ub;      // stage states
    int nsteps;
    int fpt;              // faces per face task
    unsigned* sync;       // [0] column arrivals, [32] face arrivals, one per block and stage
    unsigned base;        // both counters' value before the launch
    unsigned done_base;   // and that of the finished blocks' counter, sync[64]
    unsigned* host_status;  // pinned copy of the status word, written by the last block (or null)
    long long wait_cycles;  // limit of a wait
};

// stage 1 .. 4 of a step
struct StepIO {
    double *U0b, *Ua, *Ub;
    int stage;
    __device__ __forceinline__ const double* Us(const StageArgs&) const { return stage == 1 ? U0b : stage == 3 ? Ub : Ua; }
    __device__ __forceinline__ const double* U0(const StageArgs&) const { return U0b; }
    __device__ __forceinline__ double* acc(const StageArgs& a) const { return a.acc; }
    __device__ __forceinline__ double* out(const StageArgs&) const { return stage == 4 ? U0b : stage == 2 ? Ub : Ua; }
    __device__ __forceinline__ int mode(const StageArgs&) const { return kModeRK1 + stage - 1; }
    __device__ __forceinline__ double dt(const StageArgs& a) const { return a.dt; }
};

// barrier `id` of the NT threads of a group or role
template <int NT>
__device__ __forceinline__ void named_sync(int id)
{
    if constexpr (NT == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(NT) : "memory");
}
template <int NT>
struct GroupSync {
    int id;
    __device__ __forceinline__ void operator()() const { named_sync<NT>(id); }
};

constexpr long long kSmallWaitCycles = 2000000000ll;  // about a second, the limit outside of probes

// one arrival for the block by the NT threads of a role, whose writes it publishes
template <int NT>
__device__ __forceinline__ void role_arrive(unsigned* count, int id, int tid)
{
    named_sync<NT>(id);
    if (tid == 0) {
        __threadfence();
        atomicAdd(count, 1u);
    }
}
// waits until the counter has reached target; false (for all threads) when the
// wait, after `limit` SM cycles, or another block gave up
template <int NT>
__device__ __forceinline__ bool role_wait(unsigned* count, unsigned target, long long limit, unsigned* status, int* dead, int id, int tid)
{
    if (tid == 0) {
        const long long t0 = clock64();
        while (static_cast<int>(*reinterpret_cast<volatile unsigned*>(count) - target) < 0) {
            if (*reinterpret_cast<volatile unsigned*>(status) & kStatusTimeout || clock64() - t0 > limit) {
                atomicOr(status, kStatusTimeout);
                *dead = 1;
                break;
            }
        }
        __threadfence();
    }
    named_sync<NT>(id);
    return *reinterpret_cast<volatile int*>(dead) == 0;
}

// CG column groups of NT threads (E elements each) and FW face warps (tasks of up
// to FB faces) per block
template <int P, int E, int NT, int CG, int FW, int FB, typename T>
struct SmallLay {
    static constexpr int kThreads = CG * NT + FW * 32;
    static constexpr size_t col = (ColLay<P, T>::bytes(E) + 15) / 16 * 16;
    using F = FaceLay<P, T, FB>;
    static constexpr size_t face = F::tr_bytes + F::sl_bytes + FB * sizeof(FaceDesc);
    static constexpr size_t bytes = CG * col + FW * face;
    static_assert(bytes <= 227 * 1024 && kThreads <= 1024 && CG + 3 <= 16, "small-mesh kernel does not fit");
};

template <int P, int E, int NT, int CG, int FW, int FB, typename T>
__global__ void __launch_bounds__(SmallLay<P, E, NT, CG, FW, FB, T>::kThreads, 1)
small_steps_kernel(const __grid_constant__ SmallArgs s)
{
    using L = SmallLay<P, E, NT, CG, FW, FB, T>;
    extern __shared__ __align__(16) unsigned char sraw[];
    __shared__ int dead[2];
    if (threadIdx.x < 2) dead[threadIdx.x] = 0;
    __syncthreads();
    const int nb = gridDim.x;
    if (threadIdx.x < CG * NT) {
        // ---- column groups ----
        const int g = threadIdx.x / NT, tid = threadIdx.x % NT;
        const int e0 = (g * nb + blockIdx.x) * E;
        const bool active = e0 < s.a.ne;
        Column<P, E, NT, T, StepIO, GroupSync<NT>> c(s.a, StepIO{const_cast<double*>(s.a.U0), s.Ua, s.Ub, 1}, GroupSync<NT>{3 + g},
                                                     tid, reinterpret_cast<double*>(sraw + g * L::col));
        unsigned target = s.base;
        bool ok = true;
        for (int step = 0; step < s.nsteps && ok; ++step)
#pragma unroll 1
            for (int stage = 1; stage <= 4 && ok; ++stage) {
                c.io.stage = stage;
                c.set_mode(s.a);
                if (active) {
                    c.fetch(s.a, e0);
                    c.classes();
                    c.interp_x(s.a);
                    c.columns(s.a, e0);
                    c.contract_y(s.a);
                }
                target += nb;
                ok = role_wait<CG * NT>(s.sync + 32, target, s.wait_cycles, s.a.status, dead, 1, threadIdx.x);
                if (!ok) break;
                if (active) {
                    c.lifts(s.a, e0);
                    cp_async_wait_all();
                    c.sync();
                    c.finish(s.a, e0);
                }
                role_arrive<CG * NT>(s.sync, 1, threadIdx.x);
            }
        if (c.status) atomicOr(s.a.status, c.status);
    } else {
        // ---- face warps ----
        using F = FacePhases<P, T, FB, 32>;
        const int ft = threadIdx.x - CG * NT, fw = ft / 32, lane = ft % 32;
        unsigned char* base = sraw + CG * L::col + fw * L::face;
        T* sTr = reinterpret_cast<T*>(base);
        double* sSl = reinterpret_cast<double*>(base + L::F::tr_bytes);
        FaceDesc* sD = reinterpret_cast<FaceDesc*>(base + L::F::tr_bytes + L::F::sl_bytes);
        const int ntask = (s.a.nface + s.fpt - 1) / s.fpt, first = fw * nb + blockIdx.x, step_t = FW * nb;
        StepIO io{const_cast<double*>(s.a.U0), s.Ua, s.Ub, 1};
        auto describe = [&](int task) {
            const int nf = min(s.fpt, s.a.nface - task * s.fpt);
            for (int i = lane; i < nf * 4; i += 32)
                cp_async16(reinterpret_cast<char*>(sD) + 16 * i, reinterpret_cast<const char*>(s.a.fdesc + task * s.fpt) + 16 * i);
            cp_async_commit();
            cp_async_wait_all();
            __syncwarp();
        };
        if (first < ntask) describe(first);
        const bool once = first + step_t >= ntask;  // one task: its descriptors stay
        unsigned target = s.base, status = 0;
        bool ok = true;
        for (int step = 0; step < s.nsteps && ok; ++step)
#pragma unroll 1
            for (int stage = 1; stage <= 4; ++stage) {
                if (step > 0 || stage > 1) {
                    target += nb;
                    ok = role_wait<FW * 32>(s.sync, target, s.wait_cycles, s.a.status, dead + 1, 2, ft);
                    if (!ok) break;
                }
                io.stage = stage;
                const double* Us = io.Us(s.a);
                for (int task = first; task < ntask; task += step_t) {
                    const int f0 = task * s.fpt, nf = min(s.fpt, s.a.nface - f0);
                    if (!once) describe(task);
                    if constexpr (L::F::COOP) {
                        F::gather(Us, sD, nf, sSl, lane);
                        cp_async_commit();
                        cp_async_wait_all();
                        __syncwarp();
                    }
                    F::traces(s.a, Us, sD, nf, sSl, sTr, lane);
                    __syncwarp();
                    F::flux(s.a, sD, nf, sTr, status, lane);
                    __syncwarp();
                    F::lift(s.a, f0, nf, sTr, lane);
                    __syncwarp();
                }
                role_arrive<FW * 32>(s.sync + 32, 2, ft);
            }
        if (status) atomicOr(s.a.status, status);
    }
    // the last block hands the status word to the host (a copy after the kernel
    // would wait for it a second time)
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(s.sync + 64, 1u) + 1u == s.done_base + gridDim.x && s.host_status) {
            __threadfence();
            *reinterpret_cast<volatile unsigned*>(s.host_status) = atomicOr(s.a.status, 0u);
            __threadfence_system();
        }
    }
}

template <int P, int E, int NT, int CG, int FW, int FB, typename T>
cudaError_t launch_small(SmallArgs& s, int grid, cudaStream_t stream)
{
    using L = SmallLay<P, E, NT, CG, FW, FB, T>;
    void* args[] = {&s};
    return cudaLaunchCooperativeKernel((const void*)small_steps_kernel<P, E, NT, CG, FW, FB, T>, dim3(grid), dim3(L::kThreads), args,
                                       L::bytes, stream);
}

// the small-mesh form of an order: a column variant whose RK4 steps run in
// small_steps_kernel while the mesh has at most CG E elements per SM
template <int P, int E, int NT, int CG, int FW, int FB, typename T>
StageVariant make_small_variant(StageVariant v)
{
    using L = SmallLay<P, E, NT, CG, FW, FB, T>;
    v.flags |= kSM;
    v.small_func = (const void*)small_steps_kernel<P, E, NT, CG, FW, FB, T>;
    v.small_launch = launch_small<P, E, NT, CG, FW, FB, T>;
    v.small_smem = L::bytes;
    v.small_threads = L::kThreads;
    v.small_elems = CG * E;
    v.small_group_elems = E;
    v.small_face_warps = FW;
    v.small_face_batch = FB;
    return v;
}

}  // namespace dgk
