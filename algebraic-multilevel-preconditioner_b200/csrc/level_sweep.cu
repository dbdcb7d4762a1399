// Level-synchronous sparse sweeps of the local solve (the sparse part of one triangular factor of
// every subdomain), a thread-block cluster per subdomain.
//
// What bounds a sweep is the chain of dependent hand-overs: a row's sum over the lanes, its store
// and the reads that wait for it cost some 500 to 1000 cycles whatever the data path.  The layout
// (level_layout.inl) therefore has few levels, each in one or two stages, and a stage is an
// ordinary sparse product whose rows are independent: no ready flag is polled, every warp of the
// cluster works on the stage's tasks, and a barrier ends it.  x (with a zero slot for padding and the
// slots of s) lies in the shared memory of every CTA of the cluster; a row's result is stored to all
// of them through distributed shared memory.  A warp's entries are one stream whose addresses need
// no solved value: cp.async keeps its next steps on their way into a ring of its own in shared
// memory, across tasks and barriers.  (Held in registers instead, four steps ahead, every step still
// waited some 1000 cycles for its loads: a warp has six scoreboards for all of them.)
//
// Measured on one B200: local solve of all subdomains in us, CUDA events, dataflow sweeps (kernels.cu)
// and level sweeps, one column and four columns, couplings and tails the same in both:
//   bubbles3d 48^3 / 8     FP64   481 -> 271    502 -> 328      poisson2d 200^2 / 8  FP64  220 -> 117    495 -> 144
//   bubbles3d 48^3 / 8     FP32   341 -> 215    720 -> 269      convdiff3d 48^3 / 12 FP32 1014 -> 309   1770 -> 481
//   bubbles3d 100^3 / 64   FP64  1210 -> 983   1900 -> 1790     bubbles3d 100^3 / 64 FP32  787 -> 684   1025 -> 895
// (the whole local solve; on 100^3 / 64 FP32 the two sweeps take 145 and 174 us of it).
#include "s2l_internal.cuh"

#include <type_traits>

namespace s2l {

namespace {

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// The barrier of every thread of the cluster (or of the CTA, alone), in two halves: stores before a
// thread's arrival are seen after every other thread's wait.  The aligned forms want all lanes of a
// warp at the same instruction, and the code before either half branches by lane (ragged loops over
// the right-hand sides, partial copies): the warp comes together here first.
template <bool CLUSTER>
__device__ __forceinline__ void stage_arrive()
{
    if (CLUSTER) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
}
template <bool CLUSTER>
__device__ __forceinline__ void stage_wait()
{
    if (CLUSTER) {
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// the KC values of a slot to the CTA `rank` of the cluster
template <int KC>
__device__ __forceinline__ void store_rank(double* p, uint32_t rank, const double (&v)[KC])
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    if constexpr (KC == 1) {
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v[0]) : "memory");
    } else {
#pragma unroll
        for (int r = 0; r < KC; r += 2)
            asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a + 8 * r), "d"(v[r]), "d"(v[r + 1]) : "memory");
    }
}

template <int KC>
__device__ __forceinline__ void store_rank(float* p, uint32_t rank, const float (&v)[KC])
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    if constexpr (KC == 1)
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v[0]) : "memory");
    else if constexpr (KC == 2)
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v[0]), "f"(v[1]) : "memory");
    else
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                     : "memory");
}

// KC right-hand sides per cluster: cluster b takes subdomain b / ngrp and columns grp * KC .. + KC of
// the K interleaved columns (neighbouring clusters of one subdomain share the factor stream in L2)
template <typename Real, bool FWD, int KC, bool CLUSTER, int D>
__global__ void __launch_bounds__(S2L_BS_LEVEL, 1) level_sweep_kernel(const LocalSolveArgs<Real> a)
{
    constexpr int WARPS = S2L_BS_LEVEL / 32;
    constexpr int SB = level_step_bytes(sizeof(Real));  // a step: 128 values, then 128 columns
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int cs = CLUSTER ? a.cs : 1;
    const int rank = CLUSTER ? (int)cluster_rank() : 0;
    const int K = a.K, ngrp = K / KC;
    const int cid = (int)blockIdx.x / cs;
    const int g0 = (cid % ngrp) * KC;
    const int sidx = cid / ngrp;
    const int sid = a.sub_list ? a.sub_list[sidx] : sidx;
    const LevelFactor<Real> F = a.lf[FWD ? 0 : 1];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const LevelWarp W = F.warp[((int64_t)sid * cs + rank) * WARPS + wid];
    const int64_t lo = W.lo;
    const int T = W.T;
    const unsigned char* ring = smem_raw + (size_t)wid * D * SB;
    Real* xs = reinterpret_cast<Real*>(smem_raw + (size_t)WARPS * D * SB);  // slot k, column r: xs[k * KC + r]
    // Right-hand sides (scaled by 1/diag), each into the slot that keeps it: of the rows without
    // entries all (they are x), of the others the warp's own.  The indices of the first ones are loaded
    // before all else: index and gather are two trips to memory, the first to start a sweep.
    constexpr int UA = 16 / KC, UB = 8 / KC;
    auto index = [&](int i) { return FWD ? a.gather[lo + i] : a.u2l[lo + i]; };
    // N right-hand sides of the thread, number i0 + u * step of them below end, with their indices: every
    // gather is in flight before the first store (the compiler may not move a load over a store)
    auto place = [&](auto count, int i0, int step, int end, const int* at, bool own) {
        constexpr int N = decltype(count)::value;
        Real v[N][KC], f[N];
        int to[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int i = i0 + u * step;
            if (i < end) {
                const int64_t src = (FWD ? (int64_t)at[u] : lo + at[u]) * K + g0;
                f[u] = F.dinv[lo + i];
                to[u] = own ? (int)F.rslot[lo + i] : i;
#pragma unroll
                for (int r = 0; r < KC; ++r) v[u][r] = FWD ? (Real)a.in[src + r] : a.ybuf[src + r];
            }
        }
#pragma unroll
        for (int u = 0; u < N; ++u)
            if (i0 + u * step < end)
#pragma unroll
                for (int r = 0; r < KC; ++r) xs[to[u] * KC + r] = v[u][r] * f[u];
    };
    int ia[UA], ib[UB];
#pragma unroll
    for (int u = 0; u < UB; ++u) ib[u] = lane + 32 * u < W.nrhs ? index(W.rhs + lane + 32 * u) : 0;
#pragma unroll
    for (int u = 0; u < UA; ++u)
        ia[u] = (int)threadIdx.x + S2L_BS_LEVEL * u < W.n0 ? index(threadIdx.x + S2L_BS_LEVEL * u) : 0;

    // The ring: the warp's next D steps, one copy group each (empty past the end of the stream)
    const unsigned char* vp = F.ent + W.step * SB + lane * 16;
    int left = W.nstep;  // steps not yet requested
    const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(ring) + lane * 16;
    const int pf = a.sweep_pf;
    auto request = [&](int slot) {
        if (left > 0) {  // the same for the whole warp
            --left;
            const uint32_t dst = dst0 + (uint32_t)(slot * SB);
#pragma unroll
            for (int q = 0; q < SB; q += 512)
                if (q + 512 <= SB || lane < (SB - q) / 16)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + q), "l"(vp + q) : "memory");
            // the steps after the ring are hinted into L2, one lane per 128-byte line
            if (lane < SB / 128 && left > pf) asm volatile("prefetch.global.L2 [%0];" ::"l"(vp + lane * 112 + pf * SB));
            vp += SB;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int EARLY = D < 2 ? D : 2;  // the rest follows the right-hand sides, whose loads would queue behind it
#pragma unroll
    for (int i = 0; i < EARLY; ++i) request(i);

    // task descriptors 32 at a time (coalesced loads, the next 32 on their way)
    const uint4* desc = F.task + W.task;
    const int nt = W.ntask;
    const uint32_t end = (uint32_t)W.nst << 16;  // past the last task: no rows, the stage after the last
    auto window = [&](int i) { return i + lane < nt ? __ldg(desc + i + lane) : make_uint4(end, 0u, 0u, 0u); };
    uint4 w0 = window(0), w1 = window(32);

    {
        const int e1 = W.rhs + W.nrhs;
        place(std::integral_constant<int, UB>{}, W.rhs + lane, 32, e1, ib, true);
        place(std::integral_constant<int, UA>{}, threadIdx.x, S2L_BS_LEVEL, W.n0, ia, false);
        for (int i = W.rhs + lane + 32 * UB; i < e1; i += 32 * UB) {
#pragma unroll
            for (int u = 0; u < UB; ++u) ib[u] = i + 32 * u < e1 ? index(i + 32 * u) : 0;
            place(std::integral_constant<int, UB>{}, i, 32, e1, ib, true);
        }
        for (int i = threadIdx.x + S2L_BS_LEVEL * UA; i < W.n0; i += S2L_BS_LEVEL * UA) {
#pragma unroll
            for (int u = 0; u < UA; ++u) ia[u] = i + S2L_BS_LEVEL * u < W.n0 ? index(i + S2L_BS_LEVEL * u) : 0;
            place(std::integral_constant<int, UA>{}, i, S2L_BS_LEVEL, W.n0, ia, false);
        }
    }
#pragma unroll
    for (int i = EARLY; i < D; ++i) request(i);
    if (threadIdx.x < KC) xs[T * KC + threadIdx.x] = Real(0);  // the slot of the padding entries
    stage_arrive<CLUSTER>();  // every CTA runs and has its zero slot before the first store to it

    // the warp's next step: four values and four columns per lane
    Real v[4];
    uint2 c4;
    int slot = 0;
    auto next_step = [&]() {
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
        __syncwarp();
        const unsigned char* p = ring + (uint32_t)(slot * SB);
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = reinterpret_cast<const Real*>(p)[q * 32 + lane];
        c4 = reinterpret_cast<const uint2*>(p + 128 * sizeof(Real))[lane];
        __syncwarp();  // every lane has read the slot before it is filled again
        request(slot);
        slot = slot + 1 == D ? 0 : slot + 1;
    };
    auto head = [&](int t) {  // tasks in order: descriptor t is in w0
        return make_uint3(__shfl_sync(0xffffffffu, w0.x, t & 31), __shfl_sync(0xffffffffu, w0.y, t & 31),
                          __shfl_sync(0xffffffffu, w0.z, t & 31));
    };
    uint3 d = head(0);
    Real acc[KC];
#pragma unroll
    for (int r = 0; r < KC; ++r) acc[r] = Real(0);
    next_step();
    int stage = 0;
    stage_wait<CLUSTER>();
    for (const int st = (int)(d.x >> 16); stage < st; ++stage) {  // stages before the warp's first task
        stage_arrive<CLUSTER>();
        stage_wait<CLUSTER>();
    }
    auto fma_step = [&]() {
        const int c[4] = {(int)(c4.x & 0xFFFFu), (int)(c4.x >> 16), (int)(c4.y & 0xFFFFu), (int)(c4.y >> 16)};
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int r = 0; r < KC; ++r) acc[r] += v[q] * xs[c[q] * KC + r];
    };
    for (int t = 0; t < nt; ++t) {  // the same for the whole warp
        if ((t & 31) == 31) {
            w0 = w1;
            w1 = window(t + 33);
        }
        const uint3 dn = head(t + 1);
        const int n = (int)(d.y >> 16);  // steps
        const int gl2 = (int)(d.x & 7u), R = (int)((d.x >> 3) & 63u), k = lane >> gl2, G = 1 << gl2, j = lane & (G - 1);
        const bool to_s = (d.x & S2L_LTASK_TO_S) != 0, rhs = !(d.x & S2L_LTASK_NO_RHS);
        const int oslot = rhs ? (int)(d.y & 0xFFFFu) + k : (k < R ? (int)__ldg(F.bout + d.z + k) : 0);
        Real b[KC];
#pragma unroll
        for (int r = 0; r < KC; ++r) b[r] = k < R && rhs ? xs[((int)d.z + k) * KC + r] : Real(0);
        for (int i = 1; i < n; ++i) {
            fma_step();
            next_step();
        }
        if (n > 0) fma_step();
#pragma unroll
        for (int r = 0; r < KC; ++r) {  // the sum over the row's lanes, in each of them
            switch (gl2) {
            case 5: acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 16); [[fallthrough]];
            case 4: acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 8); [[fallthrough]];
            case 3: acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 4); [[fallthrough]];
            case 2: acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 2); [[fallthrough]];
            case 1: acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 1); [[fallthrough]];
            default: break;
            }
            if (rhs) acc[r] = b[r] - acc[r];
        }
        if (k < R) {
            Real* out = xs + oslot * KC;
            if (!CLUSTER) {
                if (j == 0) {
#pragma unroll
                    for (int r = 0; r < KC; ++r) out[r] = acc[r];
                }
            } else if (to_s) {  // s: to the CTA that solves the block
                if (j == 0) store_rank<KC>(out, (d.x >> 12) & 15u, acc);
            } else {  // x: to every CTA, the row's lanes sharing the stores
                for (int q = j; q < cs; q += G) store_rank<KC>(out, (uint32_t)q, acc);
            }
        }
        // the next task's stage: arrive at once, prepare the next step, then wait
        const int st = (int)(dn.x >> 16);
        if (st > stage) stage_arrive<CLUSTER>();
        if (n > 0) next_step();
#pragma unroll
        for (int r = 0; r < KC; ++r) acc[r] = Real(0);
        d = dn;
        if (st > stage) {
            stage_wait<CLUSTER>();
            for (++stage; stage < st; ++stage) {
                stage_arrive<CLUSTER>();
                stage_wait<CLUSTER>();
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // every warp has passed the barrier of the last stage: x is complete

    // every CTA holds all of x: the results are written out by all of them
    const DevSub sd = a.subs[sid];
    const int tid = rank * S2L_BS_LEVEL + threadIdx.x, all = cs * S2L_BS_LEVEL;
    if (FWD) {
#pragma unroll 8
        for (int i = tid; i < T; i += all) {
            const int p = F.pos[lo + i];
#pragma unroll
            for (int r = 0; r < KC; ++r) a.ybuf[(lo + i) * K + g0 + r] = xs[p * KC + r];
        }
        return;
    }
    // backward: x_local[j] from its slot (< T) or tail row (>= T); four rows' loads in flight together
    const int rows = a.mode == 0 ? sd.n_owned : sd.n_local;
    constexpr int U = 4;
    for (int j0 = tid; j0 < rows; j0 += U * all) {
        int p[U];
        double v[U][KC];
#pragma unroll
        for (int u = 0; u < U; ++u) p[u] = j0 + u * all < rows ? a.gout[lo + j0 + u * all] : 0;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < KC; ++r) {
                const int64_t j = j0 + u * all;
                v[u][r] = 0.0;
                if (j >= rows) continue;
                v[u][r] = p[u] < T ? (double)xs[p[u] * KC + r] : (double)a.ybuf[(lo + p[u]) * K + g0 + r];
                if (a.mode == 0 && a.base) v[u][r] += a.base[(sd.begin + j) * K + g0 + r];
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < KC; ++r) {
                const int64_t j = j0 + u * all;
                if (j >= rows) continue;
                if (a.mode == 0) a.out[(sd.begin + j) * K + g0 + r] = v[u][r];
                else if (a.mode == 1) a.ylocal[(lo + j) * K + g0 + r] = v[u][r];
                else a.out[j] = v[u][r];
            }
    }
}

template <typename Real, bool FWD, int KC, bool CLUSTER, int D>
cudaError_t configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, cudaStream_t st, int cs, int clusters, int slots)
{
    const size_t smem = level_smem_bytes(sizeof(Real), slots, KC, D);
    if (smem > S2L_SWEEP_SMEM_CAP) return cudaErrorInvalidValue;
    // the limit is a process-wide attribute of the kernel: always the same cap, so launches of setups
    // with different shared-memory sizes from several threads cannot undercut each other
    const cudaError_t e = cudaFuncSetAttribute(level_sweep_kernel<Real, FWD, KC, CLUSTER, D>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, S2L_SWEEP_SMEM_CAP);
    if (e != cudaSuccess) return e;
    cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * cs));
    cfg.blockDim = dim3(S2L_BS_LEVEL);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    if (CLUSTER) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return cudaSuccess;
}

template <typename Real, bool FWD, int KC, bool CLUSTER>
cudaError_t launch(cudaStream_t st, const LocalSolveArgs<Real>& a, int clusters, int slots)
{
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    auto go = [&](auto ring) {
        constexpr int D = decltype(ring)::value;
        const cudaError_t e = configure<Real, FWD, KC, CLUSTER, D>(cfg, at, st, a.cs, clusters, slots);
        return e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, level_sweep_kernel<Real, FWD, KC, CLUSTER, D>, a);
    };
    switch (level_ring(sizeof(Real), slots, KC)) {
    case 8: return go(std::integral_constant<int, 8>{});
    case 4: return go(std::integral_constant<int, 4>{});
    case 3: return go(std::integral_constant<int, 3>{});
    default: return go(std::integral_constant<int, 2>{});
    }
}

}  // namespace

template <typename Real>
cudaError_t launch_level_sweep(cudaStream_t st, const LocalSolveArgs<Real>& a, bool forward, int nblocks)
{
    const int clusters = nblocks * (a.K / a.KC), slots = a.slots;
#define S2L_LVL(KC_)                                                                                              \
    if (a.KC == KC_) {                                                                                           \
        if (a.cs > 1)                                                                                            \
            return forward ? launch<Real, true, KC_, true>(st, a, clusters, slots)                              \
                           : launch<Real, false, KC_, true>(st, a, clusters, slots);                            \
        return forward ? launch<Real, true, KC_, false>(st, a, clusters, slots)                                  \
                       : launch<Real, false, KC_, false>(st, a, clusters, slots);                                \
    }
    S2L_LVL(1)
    S2L_LVL(2)
    S2L_LVL(4)
#undef S2L_LVL
    return cudaErrorInvalidValue;
}

// Clusters of cs CTAs with `slots` values of x that the device runs at once (0: none)
int level_sweep_clusters(size_t real_bytes, int slots, int cs)
{
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    int n = 0;
    cudaError_t e;
    if (real_bytes == 8) {
        e = configure<double, true, 1, true, 2>(cfg, at, nullptr, cs, 1, slots);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, level_sweep_kernel<double, true, 1, true, 2>, &cfg);
    } else {
        e = configure<float, true, 1, true, 2>(cfg, at, nullptr, cs, 1, slots);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, level_sweep_kernel<float, true, 1, true, 2>, &cfg);
    }
    if (e != cudaSuccess) {
        (void)cudaGetLastError();  // the query alone failed: fewer CTAs per subdomain
        return 0;
    }
    return n;
}

template cudaError_t launch_level_sweep<double>(cudaStream_t, const LocalSolveArgs<double>&, bool, int);
template cudaError_t launch_level_sweep<float>(cudaStream_t, const LocalSolveArgs<float>&, bool, int);

}  // namespace s2l
