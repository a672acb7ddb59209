// Two steps of a 2D block in one launch.
//
// A step moves 2 Q values per node and, in 2D, does little more with them:
// blocks beyond the L2 cache ran at 80-83 % of the copy peak.  Here a CTA
// takes a tile of 256 bytes by kTileH rows of nodes, computes the first step
// on the tile and one node around it (10-14 % more nodes) into shared memory,
// and the second step from there, so two steps move the populations once: 302
// MB read and written for two FP32 steps of 4096 x 1024 nodes, where single
// steps move 604.  A node's 193 warp instructions per 32 nodes and step (index
// arithmetic a third of them) and their waits at 24 warps per SM are the bound
// then: 2.0 instructions a cycle and SM.
//
// One block, every boundary programme node-local, at most one axis periodic
// (the planner's rule is DoubleSteps in mplbgpu.cu).  A position outside the
// block is the node it wraps to on the periodic axis, evaluated again, and
// elsewhere a halo cell that no transfer writes: f = 0.  So no halo is read,
// and none has to be filled between two of these launches.  The arithmetic of a
// node is the step kernel's (StepNode), the same bits.
#pragma once

#include "kernels.cuh"

namespace mplb {

constexpr int kTileH = 26;   // three CTAs of 75 KB fit on an SM
constexpr int kDoubleThreads = 256;
template <typename T>
__host__ __device__ constexpr int TileW() {   // a row of a tile: 256 bytes
    return 256 / (int)sizeof(T);
}
template <typename T>
__host__ __device__ constexpr int TileNodes() {   // with the ring around it
    return (TileW<T>() + 2) * (kTileH + 2);
}
constexpr int kBlockOps2D = 9 * kMaxOps;   // the regions 9 .. 17
template <typename T>
__host__ __device__ constexpr int DoubleSmemBytes() {
    return kBlockOps2D * (int)sizeof(WallOp) +
           9 * TileNodes<T>() * (int)sizeof(T);
}

// Stale populations of node (x, y) of region r (they keep f^0).
template <typename C>
__device__ __forceinline__ void LoadStale2D(const BlockDev& b, int r, int x,
                                            int y, C* f) {
    const int rx = r % 3, ry = (r / 3) % 3;
    const int ex = rx == 1 ? b.n[0] - 2 : 1;
    const int lx = rx == 1 ? x - 1 : 0, ly = ry == 1 ? y - 1 : 0;
    const double* st = b.stale + ((long long)b.rside[r] + ly * ex + lx) * 9;
#pragma unroll
    for (int i = 0; i < 9; i++)
        if (b.rstale[r] >> i & 1u) f[i] = (C)st[i];
}

// A node on the block's boundary before its collision: pulled populations
// (pull(i), or 0 where the region pulls none), stale ones, the boundary
// programme (own(i): population i of the node itself).
template <typename T, typename Pull, typename Own>
__device__ __forceinline__ void WallNode(const BlockDev& b,
                                         const PhysConst& pc,
                                         const WallOp* ops, int r, int x,
                                         int y, Pull pull, Own own,
                                         typename Prec<T>::C* f) {
    using L = Lattice<2>;
    using C = typename Prec<T>::C;
    const bool pure = (b.rflags[r] & 3) == kPure;
    const uint32_t mask = pure ? ~0u : b.rpull[r];
#pragma unroll
    for (int i = 0; i < 9; i++) f[i] = (mask >> i & 1u) ? pull(i) : (C)0;
    if (!pure) {
        if (b.rstale[r]) LoadStale2D(b, r, x, y, f);
        ApplyWallOps<L, T>(f, ops + (r - 9) * kMaxOps, b.rnops[r], pc, x, y, 0,
                           own);
    }
    MomentsCollideT<L, T>(f, pc, (b.rflags[r] & 4) != 0);
}

// The columns (or rows) of a ringed tile that hold the first or last node of
// an axis: the tile starts at node o, has w nodes and a ring of one, on an axis
// of n nodes.  A tile's own edges and, on a periodic axis, the nodes its ring
// wraps to; `ring`: those of the ring too.
struct EdgeLines {
    int at[4];
    int n;
    __device__ __forceinline__ void Add(int v, int lo, int hi) {
        if (v >= lo && v <= hi) at[n++] = v;
    }
    __device__ __forceinline__ EdgeLines(int o, int w, int size, bool periodic,
                                         bool ring) {
        n = 0;
        const int lo = ring ? 0 : 1, hi = ring ? w + 1 : w;
        Add(1 - o, lo, hi);            // node 0
        Add(size - o, lo, hi);         // node size - 1
        if (periodic && ring) {
            if (o == 0) Add(0, lo, hi);            // wraps to size - 1
            Add(size + 1 - o, lo, hi);             // wraps to 0
        }
    }
    __device__ __forceinline__ bool Has(int v) const {
        bool h = false;
#pragma unroll
        for (int k = 0; k < 4; k++) h = h || (k < n && at[k] == v);
        return h;
    }
};

// Calls node(column, row) for every position on the lines, spread over the
// CTA: the wall nodes of a step side by side in their warps instead of one by
// one in warps of interior nodes, which ran both programmes (128^2 in FP32 took
// 22 us a launch that way).
template <typename F>
__device__ __forceinline__ void ForEdges(const EdgeLines& cols,
                                         const EdgeLines& rows, int lo, int wx,
                                         int wy, F node) {
    const int in_cols = cols.n * wy, all = in_cols + rows.n * wx;
    for (int e = threadIdx.x; e < all; e += kDoubleThreads) {
        int c, r;
        if (e < in_cols) {
            const int k = e / wy;
            c = cols.at[k];
            r = lo + e - k * wy;
        } else {
            const int k = (e - in_cols) / wx;
            r = rows.at[k];
            c = lo + (e - in_cols) - k * wx;
            if (cols.Has(c)) continue;
        }
        node(c, r);
    }
}

// Collides two interior nodes (FP32: in paired arithmetic).
template <typename T>
__device__ __forceinline__ void CollideTwo(const PhysConst& pc, bool fluid,
                                           typename Prec<T>::C* fa,
                                           typename Prec<T>::C* fb) {
    using L = Lattice<2>;
    if constexpr (Prec<T>::kShifted) {
        MomentsCollidePair<L>(fa, fb, pc, fluid, pc.omcf);
    } else {
        MomentsCollideT<L, T>(fa, pc, fluid);
        MomentsCollideT<L, T>(fb, pc, fluid);
    }
}

// periodic: bit a set when axis a wraps.
template <typename T>
__global__ void __launch_bounds__(kDoubleThreads, 3)
    DoubleStepKernel(BlockDev b, PhysConst pc, const T* __restrict__ src,
                     T* __restrict__ dst, int periodic) {
    using L = Lattice<2>;
    using P = Prec<T>;
    using C = typename P::C;
    constexpr int kW = TileW<T>(), kRow = kW + 2, kNodes = TileNodes<T>();
    extern __shared__ __align__(16) unsigned char double_raw[];
    WallOp* ops = reinterpret_cast<WallOp*>(double_raw);
    T* mid = reinterpret_cast<T*>(ops + kBlockOps2D);
    WaitForPrevious();
    const int x0 = blockIdx.x * kW, y0 = blockIdx.y * kTileH;
    const int nx = b.n[0], ny = b.n[1];
    if (x0 <= 1 || y0 <= 1 || x0 + kW >= nx - 1 || y0 + kTileH >= ny - 1) {
        constexpr int kPieces = kBlockOps2D * (int)sizeof(WallOp) / 16;
        const char* g = reinterpret_cast<const char*>(b.wops + 9 * kMaxOps);
        for (int e = threadIdx.x; e < kPieces; e += kDoubleThreads)
            CpAsync16(reinterpret_cast<char*>(ops) + 16 * e, g + 16 * e);
        CpAsyncCommit();
        CpAsyncWait<0>();
        __syncthreads();
    }

    const bool fluid = b.center_fluid != 0;
    const bool px = periodic & 1, py = (periodic & 2) != 0;

    // First step, on the tile and its ring: position k = row kRow + column is
    // the node (x0 - 1 + column, y0 - 1 + row).
    const EdgeLines cols(x0, kW, nx, px, true), rows(y0, kTileH, ny, py, true);
    if (cols.n + rows.n > 0)
        ForEdges(cols, rows, 0, kRow, kTileH + 2, [&](int c, int r) {
            int x = x0 - 1 + c, y = y0 - 1 + r;
            if (px) x = x < 0 ? x + nx : (x == nx ? 0 : x);
            if (py) y = y < 0 ? y + ny : (y == ny ? 0 : y);
            if (x < 0 || x >= nx || y < 0 || y >= ny) return;
            const T* p = src + NodeIndexT<2, true>(b, x, y, 0);
            C f[9];
            // the upstream node, wrapped, or a halo cell that nothing writes
            const auto pull = [&](int i) -> C {
                int sx = x - L::cx(i), sy = y - L::cy(i);
                if (px) sx = sx < 0 ? sx + nx : (sx == nx ? 0 : sx);
                if (py) sy = sy < 0 ? sy + ny : (sy == ny ? 0 : sy);
                if (sx < 0 || sx >= nx || sy < 0 || sy >= ny)
                    return FromF<T>(0.0, i, pc);
                return P::Load(src + NodeIndexT<2, true>(b, sx, sy, 0),
                               b.pop_off32[i], i, pc);
            };
            WallNode<T>(b, pc, ops, RegionOf(x, y, 0, b.n, 2), x, y, pull,
                        [&](int i) { return P::Load(p, b.pop_off32[i], i, pc); },
                        f);
            T* m = mid + r * kRow + c;
#pragma unroll
            for (int i = 0; i < 9; i++) m[i * kNodes] = (T)f[i];
        });
    constexpr int kHalf = kNodes / 2;
    static_assert(kNodes % 2 == 0, "nodes in pairs");
    for (int k = threadIdx.x; k < kHalf; k += kDoubleThreads) {
        C f[2][9];
        bool in[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int at = k + j * kHalf, row = at / kRow;
            const int x = x0 - 1 + at - row * kRow, y = y0 - 1 + row;
            in[j] = x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2;
            const T* p = src + NodeIndexT<2, true>(b, in[j] ? x : 1,
                                                   in[j] ? y : 1, 0);
#pragma unroll
            for (int i = 0; i < 9; i++)
                f[j][i] = P::Load(p, b.pull_off32[i], i, pc);
            // beyond the block, not on a line above: f = 0
            if ((x < 0 && !px) || (x >= nx && !px) || (y < 0 && !py) ||
                (y >= ny && !py)) {
                T* m = mid + at;
#pragma unroll
                for (int i = 0; i < 9; i++)
                    m[i * kNodes] = (T)FromF<T>(0.0, i, pc);
            }
        }
        if (!in[0] && !in[1]) continue;
        CollideTwo<T>(pc, fluid, f[0], f[1]);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            if (!in[j]) continue;
            T* m = mid + k + j * kHalf;
#pragma unroll
            for (int i = 0; i < 9; i++) m[i * kNodes] = (T)f[j][i];
        }
    }
    // A periodic ring's interior nodes of the other axis' range are nodes of
    // the block's far side: lines above, since they are its first or last.
    __syncthreads();

    // Second step, on the tile, from the first one's populations.
    const auto pulled = [&](const T* m, int i) -> C {
        return m[i * kNodes - L::cx(i) - L::cy(i) * kRow];
    };
    if (cols.n + rows.n > 0) {
        const EdgeLines tc(x0, kW, nx, px, false),
            tr(y0, kTileH, ny, py, false);
        ForEdges(tc, tr, 1, kW, kTileH, [&](int c, int r) {
            const int x = x0 - 1 + c, y = y0 - 1 + r;
            if (x >= nx || y >= ny) return;
            const T* m = mid + r * kRow + c;
            C f[9];
            WallNode<T>(b, pc, ops, RegionOf(x, y, 0, b.n, 2), x, y,
                        [&](int i) { return pulled(m, i); },
                        [&](int i) -> C { return m[i * kNodes]; }, f);
            T* d = dst + NodeIndexT<2, true>(b, x, y, 0);
#pragma unroll
            for (int i = 0; i < 9; i++) d[b.pop_off32[i]] = (T)f[i];
        });
    }
    constexpr int kTile = kW * kTileH;
    static_assert(kTileH % 2 == 0, "pairs of rows");
    for (int t = threadIdx.x; t < kTile / 2; t += kDoubleThreads) {
        // rows r and r + kTileH / 2 of the tile, the same column
        const int r = t / kW, x = x0 + t - r * kW;
        C f[2][9];
        bool in[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int y = y0 + r + j * (kTileH / 2);
            in[j] = x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2;
            const T* m = mid + (y - y0 + 1) * kRow + 1 + x - x0;
#pragma unroll
            for (int i = 0; i < 9; i++) f[j][i] = pulled(m, i);
        }
        if (!in[0] && !in[1]) continue;
        CollideTwo<T>(pc, fluid, f[0], f[1]);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            if (!in[j]) continue;
            T* d = dst +
                   NodeIndexT<2, true>(b, x, y0 + r + j * (kTileH / 2), 0);
#pragma unroll
            for (int i = 0; i < 9; i++) d[b.pop_off32[i]] = (T)f[j][i];
        }
    }
}

}  // namespace mplb
