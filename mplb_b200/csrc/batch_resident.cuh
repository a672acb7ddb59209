// Batched cavities held in shared memory for many steps.
//
// One step over populations in HBM moves 18 values per node and is bound by
// that traffic (67 % of the copy peak in the tile launches of
// batch_kernels.cuh).  Here a thread-block cluster takes a strip of rows of
// one cavity - all of its rows when they fit - reads it once, advances it
// `steps` steps in the cluster's shared memory and writes it once, so the
// traffic per step falls by the step count and the arithmetic is the bound.
//
// Each CTA of the cluster holds rows [R rank, R (rank + 1)) of the strip, one
// copy of each population (slot (p, k) of local node k = y n + x at
// p CAP + k), updated in place by two alternating kinds of step:
//   own    : node x has f_i in its own slot opp(i), collides, and stores g_i
//            in its own slot i;
//   gather : node x takes f_i = g_i(x - c_i) from slot i of x - c_i (from
//            its own slot opp(i) where x - c_i lies beyond a wall), collides,
//            and stores g_opp(i) where it took f_i, which is where the next
//            own step of the node at x - c_i looks for it.
// A step's reads and writes of one node touch the same slots and no other
// node's, so one cluster barrier per step is the only synchronisation.  The
// first step gathers from global memory, the last stores to it.
//
// A cavity too large for one cluster is cut into strips that overlap by
// `steps - 1` rows per cut side.  A cut edge is treated as a wall, so after
// s steps the s - 1 rows next to it (the first step reads global memory) hold
// values of a different problem; only the rows beyond them are stored.
//
// The arithmetic of a node is that of the one-step kernels, so fields,
// moments and residuals are theirs.
//
// Measured (B200, node updates per second, the tile launches in brackets):
// FP32 166 G at side 64, 139 G at 128, 121 G at 256 (61-65 G); FP64 83 G, 60 G,
// 48 G (30 G).  The bound is the FMA pipe and instruction issue (53 % and 59 %
// busy at side 64, 267 warp instructions per 64 nodes of which 106 are paired
// arithmetic), then the wait at the step's barrier (13 % of the warps' time).
#pragma once

#include "batch_kernels.cuh"

namespace mplb {

__device__ __forceinline__ uint32_t ClusterRank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t ClusterSize() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void ClusterBarrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the shared-memory address `a` in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t MapToRank(uint32_t a, uint32_t rank) {
    uint32_t d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(d)
                 : "r"(a), "r"(rank));
    return d;
}

template <typename C, bool REMOTE>
__device__ __forceinline__ C SlotLoad(uint32_t a) {
    if constexpr (sizeof(C) == 4) {
        float v;
        if constexpr (REMOTE)
            asm volatile("ld.shared::cluster.f32 %0, [%1];"
                         : "=f"(v) : "r"(a) : "memory");
        else
            asm volatile("ld.shared::cta.f32 %0, [%1];"
                         : "=f"(v) : "r"(a) : "memory");
        return v;
    } else {
        double v;
        if constexpr (REMOTE)
            asm volatile("ld.shared::cluster.f64 %0, [%1];"
                         : "=d"(v) : "r"(a) : "memory");
        else
            asm volatile("ld.shared::cta.f64 %0, [%1];"
                         : "=d"(v) : "r"(a) : "memory");
        return v;
    }
}
template <typename C, bool REMOTE>
__device__ __forceinline__ void SlotStore(uint32_t a, C v) {
    if constexpr (sizeof(C) == 4) {
        if constexpr (REMOTE)
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v)
                         : "memory");
        else
            asm volatile("st.shared::cta.f32 [%0], %1;" ::"r"(a), "f"(v)
                         : "memory");
    } else {
        if constexpr (REMOTE)
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v)
                         : "memory");
        else
            asm volatile("st.shared::cta.f64 [%0], %1;" ::"r"(a), "d"(v)
                         : "memory");
    }
}

// What every node of a CTA shares.
template <typename T>
struct ResidentCta {
    using C = typename Prec<T>::C;
    uint32_t slots;          // shared address of slot (0, 0)
    uint32_t below, above;   // the same in the CTAs of the rows below / above
    int n, nn, nodes;        // nodes: of this CTA
    int rows;                // of this CTA
    int row;                 // cavity row of the CTA's first row
    int first, last;         // local rows at the strip's ends, or -1
    int lidk;                // first local node at the moving wall
    int vlo, vhi;            // local nodes stored at the end
    int rshift;              // R n: offset between facing rows of two CTAs
    float ninv;
    long long mbase;
    C lidb[3];               // of populations 3, 4, 5
    double omc;
    float omcf;
};

// Where a step takes its populations from and leaves them.
enum ResidentIn : int { kInGlobal = 0, kInOwn = 1, kInGather = 2 };
enum ResidentOut : int { kOutOwn = 0, kOutGather = 1, kOutGlobal = 2 };

// Address of slot (i, k) of this CTA.
template <typename T, int CAP>
__device__ __forceinline__ uint32_t OwnSlot(const ResidentCta<T>& c, int k,
                                            int i) {
    return c.slots + (uint32_t)(k + i * CAP) * (uint32_t)sizeof(T);
}

// Addresses of the slots that a gather step of the local node k takes its
// populations from: slot i of the upstream node, or the node's own slot
// opp(i) when that lies beyond a wall.
template <typename T, int CAP, bool REMOTE>
__device__ __forceinline__ void GatherSlots(const ResidentCta<T>& c, int k,
                                            uint32_t* a) {
    using L = Lattice<2>;
    constexpr uint32_t kSize = (uint32_t)sizeof(T);
    const int y = (int)(((float)k + 0.5f) * c.ninv), x = k - y * c.n;
    const bool left = x == 0, right = x == c.n - 1, bottom = y == c.first,
               top = y == c.last;
    const uint32_t at = c.slots + (uint32_t)k * kSize;
    // the same column of the rows the populations with c_y = 1 / -1 come from
    uint32_t up = at - (uint32_t)c.n * kSize;
    uint32_t down = at + (uint32_t)c.n * kSize;
    if constexpr (REMOTE) {
        if (y == 0) up = c.below + (uint32_t)(k - c.n + c.rshift) * kSize;
        if (y == c.rows - 1)
            down = c.above + (uint32_t)(k + c.n - c.rshift) * kSize;
    }
    a[0] = at;
#pragma unroll
    for (int i = 1; i < 9; i++) {
        const int cx = L::cx(i), cy = L::cy(i);
        bool wall = false;
        if (cx > 0) wall = wall || left;
        if (cx < 0) wall = wall || right;
        if (cy > 0) wall = wall || bottom;
        if (cy < 0) wall = wall || top;
        const uint32_t row = cy > 0 ? up : cy < 0 ? down : at;
        // Every register an offset is added to holds an address inside the
        // shared window: an access may add its constant offset after the
        // address is widened, where a wrapped one would not wrap back.
        if (i <= 4)   // own slot opp(i) = i + 4
            a[i] = (wall ? at + (uint32_t)(4 * CAP + cx) * kSize : row) +
                   (uint32_t)(i * CAP - cx) * kSize;
        else          // own slot opp(i) = i - 4
            a[i] = (wall ? at : row + (uint32_t)(4 * CAP - cx) * kSize) +
                   (uint32_t)((i - 4) * CAP) * kSize;
    }
}

// Populations of the local node k before the lid's momentum.
template <typename T, int CAP, int IN, bool REMOTE>
__device__ __forceinline__ void ResidentLoad(const ResidentCta<T>& c, int k,
                                             const uint32_t* a, const T* s,
                                             typename Prec<T>::C* f) {
    using L = Lattice<2>;
    using C = typename Prec<T>::C;
    if constexpr (IN == kInGlobal) {
        // rows of the cavity, not of the strip: a cut edge is no wall
        const int y = (int)(((float)k + 0.5f) * c.ninv), x = k - y * c.n;
        const int gy = y + c.row, gk = c.row * c.n + k;
#pragma unroll
        for (int i = 0; i < 9; i++) {
            const int sx = x - L::cx(i), sy = gy - L::cy(i);
            const bool wall = (unsigned)sx >= (unsigned)c.n ||
                              (unsigned)sy >= (unsigned)c.n;
            f[i] = __ldcs(s + (wall ? L::opp(i) * c.nn + gk
                                    : i * c.nn + sy * c.n + sx));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 9; i++)
            f[i] = IN == kInOwn
                       ? SlotLoad<C, false>(OwnSlot<T, CAP>(c, k, L::opp(i)))
                       : SlotLoad<C, REMOTE>(a[i]);
    }
}

// Stores the collided populations g (get(i)) of the local node k.
template <typename T, int CAP, int OUT, bool REMOTE, typename Get>
__device__ __forceinline__ void ResidentStore(const ResidentCta<T>& c, int k,
                                              const uint32_t* a, T* d,
                                              Get get) {
    using L = Lattice<2>;
    using C = typename Prec<T>::C;
    if (OUT == kOutGlobal && (k < c.vlo || k >= c.vhi)) return;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        if constexpr (OUT == kOutGlobal)
            __stcs(d + i * c.nn + c.row * c.n + k, get(i));
        else if constexpr (OUT == kOutOwn)
            SlotStore<C, false>(OwnSlot<T, CAP>(c, k, i), get(i));
        else
            SlotStore<C, REMOTE>(a[i], get(L::opp(i)));
    }
}

template <typename T>
__device__ __forceinline__ void ResidentMacro(const BatchDev& bd,
                                              const ResidentCta<T>& c, int k,
                                              double rho, double u, double v) {
    if (k < c.vlo || k >= c.vhi) return;
    const long long at = c.mbase + (long long)c.row * c.n + k;
    bd.macro[0][at] = rho;
    bd.macro[1][at] = u;
    bd.macro[2][at] = v;
}

// The nodes k and k + 32 (FP32, paired arithmetic) or the node k (FP64).
template <typename T, int CAP, int IN, int OUT, bool REMOTE>
__device__ __forceinline__ void ResidentNodes(const BatchDev& bd,
                                              const PhysConst& pc,
                                              const ResidentCta<T>& c, int ka,
                                              const T* s, T* d, bool macro) {
    using L = Lattice<2>;
    constexpr bool kSlots = IN == kInGather || OUT == kOutGather;
    uint32_t a[9];
    if constexpr (kSlots) GatherSlots<T, CAP, REMOTE>(c, ka, a);
    if constexpr (sizeof(T) == 4) {
        const bool two = ka + 32 < c.nodes;
        const int kb = two ? ka + 32 : ka;
        uint32_t b[9];
        if constexpr (kSlots) GatherSlots<T, CAP, REMOTE>(c, kb, b);
        float fa[9], fb[9];
        ResidentLoad<T, CAP, IN, REMOTE>(c, ka, a, s, fa);
        ResidentLoad<T, CAP, IN, REMOTE>(c, kb, b, s, fb);
        if (kb >= c.lidk) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                if (ka >= c.lidk) fa[3 + j] += c.lidb[j];
                fb[3 + j] += c.lidb[j];
            }
        }
        float2 h[9], drho, u[3];
#pragma unroll
        for (int i = 0; i < 9; i++) h[i] = make_float2(fa[i], fb[i]);
        MomentsShiftedV<L, float2>(h, pc, false, drho, u);
        if (OUT == kOutGlobal && macro) {
            ResidentMacro(bd, c, ka, 1.0 + (double)drho.x, (double)u[0].x,
                          (double)u[1].x);
            if (two)
                ResidentMacro(bd, c, kb, 1.0 + (double)drho.y, (double)u[0].y,
                              (double)u[1].y);
        }
        CollideShiftedV<L, float2>(h, pc, false, drho, u, c.omcf);
        ResidentStore<T, CAP, OUT, REMOTE>(c, ka, a, d,
                                           [&](int i) { return h[i].x; });
        if (two)
            ResidentStore<T, CAP, OUT, REMOTE>(c, kb, b, d,
                                               [&](int i) { return h[i].y; });
    } else {
        double f[9], rho, u[3];
        ResidentLoad<T, CAP, IN, REMOTE>(c, ka, a, s, f);
        if (ka >= c.lidk) {
#pragma unroll
            for (int j = 0; j < 3; j++) f[3 + j] += c.lidb[j];
        }
        MomentsCollideT<L, T>(f, pc, false, c.omc, c.omcf, rho, u);
        if (OUT == kOutGlobal && macro) ResidentMacro(bd, c, ka, rho, u[0], u[1]);
        ResidentStore<T, CAP, OUT, REMOTE>(c, ka, a, d,
                                           [&](int i) { return f[i]; });
    }
}

template <typename T>
__host__ __device__ constexpr int ResidentGroup() {
    return sizeof(T) == 4 ? kResidentGroup32 : kResidentGroup64;
}

// One step over the CTA's nodes.  Only steps that reach into another CTA's
// slots, and only in the rows next to it, take the cluster addresses.
template <typename T, int CAP, int IN, int OUT>
__device__ __forceinline__ void ResidentStep(const BatchDev& bd,
                                             const PhysConst& pc,
                                             const ResidentCta<T>& c,
                                             const T* s,
                                             T* d, bool macro) {
    constexpr int kGroup = ResidentGroup<T>();
    constexpr bool kReach = IN == kInGather || OUT == kOutGather;
    const int lane = threadIdx.x & 31;
    for (int g = (int)(threadIdx.x >> 5) * kGroup; g < c.nodes;
         g += (int)(blockDim.x >> 5) * kGroup) {
        const int k = g + lane;
        if (k >= c.nodes) continue;
        if constexpr (kReach) {
            const bool edge = (c.first < 0 && g < c.n) ||
                              (c.last < 0 && g + kGroup > c.nodes - c.n);
            if (edge) {
                ResidentNodes<T, CAP, IN, OUT, true>(bd, pc, c, k, s, d,
                                                     macro);
                continue;
            }
        }
        ResidentNodes<T, CAP, IN, OUT, false>(bd, pc, c, k, s, d, macro);
    }
}

// 24 warps of 80 registers share an SM, whose slots one, two or four CTAs fill
// (side 24, crowded: FP32 185 G, FP64 97 G; three CTAs of 18 warps, which is
// what fits when a quarter's slots leave no room for the CTAs' own 1 KB: 166 G
// and 91 G).
template <typename T, int HALVES, int CAP>
__global__ void __launch_bounds__(768 >> HALVES, 1 << HALVES)
    BatchResidentKernel(BatchDev bd, PhysConst pc,
                        const ResidentItem* __restrict__ items, int steps,
                        int macro, const T* src, T* dst) {
    using C = typename Prec<T>::C;
    extern __shared__ __align__(16) unsigned char resident_raw[];
    const uint32_t rank = ClusterRank(), ranks = ClusterSize();
    const ResidentItem it = items[blockIdx.x / ranks];
    const BatchCav& cv = bd.cavs[it.cav];
    ResidentCta<T> c;
    c.slots = (uint32_t)__cvta_generic_to_shared(resident_raw);
    c.below = rank > 0 ? MapToRank(c.slots, rank - 1) : 0u;
    c.above = rank + 1 < ranks ? MapToRank(c.slots, rank + 1) : 0u;
    c.n = it.n;
    c.nn = it.n * it.n;
    const int y0 = (int)rank * it.rows_per_cta;
    c.rows = max(0, min(it.rows_per_cta, it.rows - y0));
    c.nodes = c.rows * c.n;
    c.row = it.row0 + y0;
    c.first = rank == 0 ? 0 : -1;
    c.last = y0 + c.rows == it.rows ? c.rows - 1 : -1;
    c.lidk = c.last >= 0 && it.row0 + it.rows == it.n ? c.last * c.n
                                                      : 0x7fffffff;
    c.vlo = (it.vrow0 - y0) * c.n;
    c.vhi = (it.vrow0 + it.vrows - y0) * c.n;
    c.rshift = it.rows_per_cta * c.n;
    c.ninv = __frcp_rn((float)c.n);
    c.mbase = cv.mbase;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        if constexpr (Prec<T>::kShifted) c.lidb[j] = (C)cv.lidbf[3 + j];
        else c.lidb[j] = (C)cv.lidb[3 + j];
    }
    c.omc = cv.omc;
    c.omcf = cv.omcf;
    const long long base = (long long)it.base * (long long)(128 / sizeof(T));
    const T* s = src + base;
    T* d = (it.whole ? const_cast<T*>(src) : dst) + base;
    // one CTA alone needs no cluster barrier (its release fence held 6 % of
    // the warps' time at side 64)
    const auto barrier = [&] {
        if (ranks == 1) __syncthreads();
        else ClusterBarrier();
    };
    barrier();   // every CTA of the cluster runs: its slots may be written
    ResidentStep<T, CAP, kInGlobal, kOutGather>(bd, pc, c, s, d, false);
    int t = 1;
    for (; t + 1 < steps; t++) {
        barrier();
        if (t & 1)
            ResidentStep<T, CAP, kInOwn, kOutOwn>(bd, pc, c, s, d, false);
        else
            ResidentStep<T, CAP, kInGather, kOutGather>(bd, pc, c, s, d,
                                                        false);
    }
    barrier();
    if (t & 1)
        ResidentStep<T, CAP, kInOwn, kOutGlobal>(bd, pc, c, s, d, macro != 0);
    else
        ResidentStep<T, CAP, kInGather, kOutGlobal>(bd, pc, c, s, d,
                                                    macro != 0);
    barrier();   // no CTA leaves while another may read its slots
}

template <typename T>
using ResidentKernelFn = void (*)(BatchDev, PhysConst, const ResidentItem*, int,
                                  int, const T*, T*);
template <typename T>
ResidentKernelFn<T> ResidentKernelOf(int halves) {
    constexpr bool kF64 = sizeof(T) == 8;
    return halves == 0   ? BatchResidentKernel<T, 0, ResidentSlots(kF64, 0)>
           : halves == 1 ? BatchResidentKernel<T, 1, ResidentSlots(kF64, 1)>
                         : BatchResidentKernel<T, 2, ResidentSlots(kF64, 2)>;
}
template <typename T>
cudaError_t PrepareResident(int halves, int ranks) {
    cudaError_t e = cudaFuncSetAttribute(
        ResidentKernelOf<T>(halves),
        cudaFuncAttributeMaxDynamicSharedMemorySize,
        ResidentSmem(sizeof(T) == 8, halves));
    if (e == cudaSuccess && ranks > 8)
        e = cudaFuncSetAttribute(ResidentKernelOf<T>(halves),
                                 cudaFuncAttributeNonPortableClusterSizeAllowed,
                                 1);
    return e;
}
struct ResidentConfig {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    ResidentConfig(int smem, int ranks, int warps, int nitems,
                   cudaStream_t s) {
        cfg.gridDim = dim3((unsigned)nitems * (unsigned)ranks);
        cfg.blockDim = dim3((unsigned)warps * 32u);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)ranks;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
};

template <typename T>
cudaError_t BatchResidentLaunch<T>::Run(int halves, int ranks, int warps,
                                        int nitems, cudaStream_t s,
                                        const BatchDev& bd,
                                        const PhysConst& pc,
                                        const ResidentItem* items, int steps,
                                        bool macro, const T* src, T* dst) {
    ResidentConfig c(ResidentSmem(sizeof(T) == 8, halves), ranks, warps, nitems,
                     s);
    const cudaError_t e = PrepareResident<T>(halves, ranks);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&c.cfg, ResidentKernelOf<T>(halves), bd, pc,
                              items, steps, macro ? 1 : 0, src, dst);
}

template <typename T>
bool BatchResidentLaunch<T>::Held(int halves, int ranks) {
    ResidentConfig c(ResidentSmem(sizeof(T) == 8, halves), ranks, 24 >> halves,
                     1, nullptr);
    int clusters = 0;
    if (PrepareResident<T>(halves, ranks) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, ResidentKernelOf<T>(halves),
                                       &c.cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return clusters > 0;
}

}  // namespace mplb
