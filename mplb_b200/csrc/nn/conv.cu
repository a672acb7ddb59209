// Tensor-core convolution kernels (see conv.cuh for the formulation).
#include "conv.cuh"
#include "launch_next.cuh"
#include "umma.cuh"

namespace mplb {
namespace nn {

using namespace umma;

namespace {

__device__ __forceinline__ uint8_t* Align1024(uint8_t* p) {
    const uint32_t s = SmemAddr(p);
    return p + ((1024u - (s & 1023u)) & 1023u);
}

__device__ __forceinline__ void Flag(volatile int* cta_err, int* err) {
    *cta_err = 1;
    atomicExch(err, 1);
}

__device__ __forceinline__ uint32_t PackBf16(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void TapOffset(int taps, int t, int& dh, int& dw) {
    dh = 0;
    dw = 0;
    if (taps == 9) {
        dh = t / 3 - 1;
        dw = t % 3 - 1;
    }
}

// Bias, ReLU, mask and store of 16 output channels (n on) of one pixel.
template <typename Args>
__device__ __forceinline__ void StoreOutputs(const Args& a, long long pix,
                                             int n, float* v,
                                             const float* bias) {
    if (a.bias != nullptr) {
        const float4* b4 = reinterpret_cast<const float4*>(bias);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4 b = b4[q];
            v[4 * q] += b.x;
            v[4 * q + 1] += b.y;
            v[4 * q + 2] += b.z;
            v[4 * q + 3] += b.w;
        }
    }
    if (a.relu) {
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = fmaxf(v[i], 0.0f);
    }
    if (a.mask != nullptr) {
        const uint4* m4 = reinterpret_cast<const uint4*>(
            a.mask + pix * a.mask_ps + a.mask_coff + n);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint4 m = m4[q];
            const uint32_t w[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                // bf16 > 0: sign bit clear and not +0
                if ((w[e] & 0x8000u) || (w[e] & 0xFFFFu) == 0)
                    v[8 * q + 2 * e] = 0.0f;
                if ((w[e] & 0x80000000u) || (w[e] >> 16) == 0)
                    v[8 * q + 2 * e + 1] = 0.0f;
            }
        }
    }
    if (a.out_f32) {
        float4* o = reinterpret_cast<float4*>(
            static_cast<float*>(a.out) + pix * a.out_ps + a.out_coff + n);
#pragma unroll
        for (int q = 0; q < 4; q++)
            o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2],
                               v[4 * q + 3]);
    } else {
        uint4* o = reinterpret_cast<uint4*>(
            static_cast<__nv_bfloat16*>(a.out) + pix * a.out_ps +
            a.out_coff + n);
        o[0] = make_uint4(PackBf16(v[0], v[1]), PackBf16(v[2], v[3]),
                          PackBf16(v[4], v[5]), PackBf16(v[6], v[7]));
        o[1] = make_uint4(PackBf16(v[8], v[9]), PackBf16(v[10], v[11]),
                          PackBf16(v[12], v[13]), PackBf16(v[14], v[15]));
    }
}

}  // namespace

template <int BK>
__global__ void __launch_bounds__(kConvThreads, 1)
    ConvKernel(const __grid_constant__ CUtensorMap ta,
               const __grid_constant__ CUtensorMap tb, ConvArgs a) {
    constexpr int SW = BK * 2;
    constexpr uint32_t A_BYTES = kTileM * BK * 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = Align1024(smem_raw);
    const uint32_t stage_bytes = A_BYTES + (uint32_t)a.bn * BK * 2;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + a.stages * stage_bytes);
    uint64_t* empty = full + a.stages;
    uint64_t* accum = empty + a.stages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    volatile int* cta_err = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x;
    const int img = mt / a.tiles_per_img;
    const int h0 = (mt - img * a.tiles_per_img) * a.bh;
    const int n0 = blockIdx.y * a.bn;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; s++) {
            BarInit(&full[s], 1);
            BarInit(&empty[s], 1);
        }
        BarInit(accum, 1);
        *cta_err = 0;
        FenceBarrierInit();
        PrefetchTmap(&ta);
        PrefetchTmap(&tb);
    }
    if (warp == 2) TmemAlloc(tmem_slot, a.tmem_cols);
    GridWait();
    FenceBeforeSync();
    __syncthreads();
    FenceAfterSync();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        // TMA producer
        const int c_per_tap = (a.cin + BK - 1) / BK;
        int kb = 0;
        for (; kb < a.nkb; kb++) {
            const int s = kb % a.stages;
            if (kb >= a.stages &&
                !BarWait(&empty[s], ((kb / a.stages) + 1) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            const int t = kb / c_per_tap;
            const int c0 = (kb - t * c_per_tap) * BK;
            int dh, dw;
            TapOffset(a.taps, t, dh, dw);
            uint8_t* sa = smem + s * stage_bytes;
            BarArriveExpectTx(&full[s], stage_bytes);
            TmaLoad4D(sa, &ta, &full[s], c0, dw, h0 + dh, img);
            TmaLoad2D(sa + A_BYTES, &tb, &full[s], t * a.cin + c0, n0);
        }
        // the copies of the last stages issued must land before exit
        for (int j = kb > a.stages ? kb - a.stages : 0; j < kb; j++)
            if (!BarWaitDrain(&full[j % a.stages], (j / a.stages) & 1))
                Flag(cta_err, a.err);
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        const uint32_t idesc = InstrDescBf16(kTileM, a.bn, false, false);
        const uint32_t base = SmemAddr(smem);
        for (int kb = 0; kb < a.nkb; kb++) {
            const int s = kb % a.stages;
            if (!BarWait(&full[s], (kb / a.stages) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            FenceAfterSync();
            const uint32_t sa = base + s * stage_bytes;
            const uint32_t sb = sa + A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / 16; k++) {
                Mma(tmem, SmemDesc(sa + k * 32, 0, 8 * SW, SW),
                    SmemDesc(sb + k * 32, 0, 8 * SW, SW), idesc,
                    (kb | k) != 0 ? 1u : 0u);
            }
            Commit(&empty[s]);
        }
        Commit(accum);
    }
    __syncwarp();

    // Epilogue: TMEM lane = pixel row of the tile, column = output channel.
    const bool acc_ok = BarWaitDrain(accum, 0);
    FenceAfterSync();
    if (!acc_ok && threadIdx.x == 0) Flag(cta_err, a.err);
    const bool store = acc_ok && *cta_err == 0;
    const int row = warp * 32 + lane;
    const long long pix = (long long)mt * kTileM + row;
    for (int c = 0; c < a.bn; c += 16) {
        float v[16];
        TmemLoad16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
        const int n = n0 + c;
        if (!store || n >= a.cout) continue;
        StoreOutputs(a, pix, n, v, a.bias + n);
    }

    FenceBeforeSync();
    __syncthreads();
    if (warp == 2) {
        FenceAfterSync();
        TmemFree(tmem, a.tmem_cols);
    }
}

// The 3x3 convolution of a band of tiles (see conv.cuh): the band's input
// stays in shared memory for all nine taps.
template <int BK>
__global__ void __launch_bounds__(kConvThreads, 1)
    ConvBandKernel(const __grid_constant__ CUtensorMap ta,
                   const __grid_constant__ CUtensorMap tb, ConvBandArgs a) {
    constexpr int SW = BK * 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = Align1024(smem_raw);
    const uint32_t b_bytes = (uint32_t)a.bn * SW;   // weights of a k-block
    const uint32_t stage_bytes = b_bytes * a.group;
    uint8_t* ring = smem + a.chunks * a.chunk_bytes;
    float* bias = reinterpret_cast<float*>(ring + a.stages * stage_bytes);
    uint64_t* full = reinterpret_cast<uint64_t*>(bias + a.bn);
    uint64_t* empty = full + a.stages;
    uint64_t* a_full = empty + a.stages;
    uint64_t* accum = a_full + a.chunks;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    volatile int* cta_err = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int img = blockIdx.x / a.bands;
    const int j0 = (int)(blockIdx.x - img * a.bands) * a.tiles;
    const int nt = min(a.tiles, a.tiles_per_img - j0);
    const int n0 = blockIdx.y * a.bn;
    const int r0 = j0 * a.tile_step / a.pitch;   // the band's first image row
    const int q0 = j0 * a.tile_step - r0 * a.pitch;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; s++) {
            BarInit(&full[s], 1);
            BarInit(&empty[s], 1);
        }
        for (int c = 0; c < a.chunks; c++) BarInit(&a_full[c], 1);
        BarInit(accum, 1);
        *cta_err = 0;
        FenceBarrierInit();
        PrefetchTmap(&ta);
        PrefetchTmap(&tb);
    }
    if (warp == 2) TmemAlloc(tmem_slot, a.tmem_cols);
    GridWait();
    for (int n = threadIdx.x; n < a.bn; n += kConvThreads)
        bias[n] = a.bias != nullptr ? a.bias[n0 + n] : 0.0f;
    FenceBeforeSync();
    __syncthreads();
    FenceAfterSync();
    const uint32_t tmem = *tmem_slot;
    const int nkb = 9 * a.chunks;
    const int nst = (nkb + a.group - 1) / a.group;   // groups of k-blocks

    if (warp == 0 && lane == 0) {
        int c = 0, k0 = 0;   // slice and weight column of the k-block
        int chunks = 0, st = 0;
        for (; st < nst; st++) {
            const int s = st % a.stages;
            if (st >= a.stages &&
                !BarWait(&empty[s], ((st / a.stages) + 1) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            const int blocks = min(a.group, nkb - st * a.group);
            BarArriveExpectTx(&full[s], blocks * b_bytes);
            for (int g = 0; g < blocks; g++) {
                if (chunks < a.chunks) {
                    BarArriveExpectTx(&a_full[chunks], a.box_bytes);
                    TmaLoad4D(smem + chunks * a.chunk_bytes, &ta,
                              &a_full[chunks], chunks * BK, -1, r0 - 1, img);
                    chunks++;
                }
                TmaLoad2D(ring + s * stage_bytes + g * b_bytes, &tb, &full[s],
                          k0 + c * BK, n0);
                if (++c == a.chunks) {
                    c = 0;
                    k0 += a.cin;
                }
            }
        }
        // every copy issued must land before exit
        for (int i = 0; i < chunks; i++)
            if (!BarWaitDrain(&a_full[i], 0)) Flag(cta_err, a.err);
        for (int j = st > a.stages ? st - a.stages : 0; j < st; j++)
            if (!BarWaitDrain(&full[j % a.stages], (j / a.stages) & 1))
                Flag(cta_err, a.err);
    } else if (warp == 1) {
        // the whole warp walks the loop, one lane issues
        const uint32_t idesc = InstrDescBf16(kTileM, a.bn, false, false);
        constexpr uint32_t kHigh = SmemDescHigh(SW);
        const uint32_t a0 = SmemDescLow(SmemAddr(smem)) + (q0 * SW >> 4);
        const uint32_t b0 = SmemDescLow(SmemAddr(ring));
        const uint32_t step = (uint32_t)(a.tile_step * SW) >> 4;
        const uint32_t slice = (uint32_t)a.chunk_bytes >> 4;
        const uint32_t row = (uint32_t)((a.pitch - 3) * SW) >> 4;
        int kb = 0;
        for (int st = 0, s = 0, phase = 0; st < nst; st++) {
            bool ok = BarWait(&full[s], phase, cta_err);
            const int blocks = min(a.group, nkb - kb);
            for (int g = kb; g < min(kb + blocks, a.chunks); g++)
                ok = ok && BarWait(&a_full[g], 0, cta_err);
            if (!__all_sync(~0u, ok)) {
                if (lane == 0) Flag(cta_err, a.err);
                break;
            }
            FenceAfterSync();
            uint32_t lb = b0 + (s * stage_bytes >> 4);
            // the stage's first k-block: its slice, tap column and input
            const int t = kb / a.chunks;
            int c = kb - t * a.chunks, dw = t % 3;
            uint32_t in = a0 + c * slice +
                          ((uint32_t)((t / 3 * a.pitch + dw) * SW) >> 4);
            if (ElectOne()) {
                for (int g = 0; g < blocks; g++) {
                    uint32_t la = in, d = tmem;
                    for (int j = 0; j < nt; j++) {
#pragma unroll
                        for (int k = 0; k < BK / 16; k++)
                            Mma2(d, la + 2 * k, lb + 2 * k, kHigh, idesc,
                                 (kb | g | k) != 0 ? 1u : 0u);
                        la += step;
                        d += a.bn;
                    }
                    lb += b_bytes >> 4;
                    in += slice;
                    if (++c == a.chunks) {
                        c = 0;
                        in -= slice * a.chunks - (SW >> 4);
                        if (++dw == 3) {
                            dw = 0;
                            in += row;
                        }
                    }
                }
                Commit(&empty[s]);
                if (st + 1 == nst) Commit(accum);
            }
            __syncwarp();
            kb += blocks;
            if (++s == a.stages) {
                s = 0;
                phase ^= 1;
            }
        }
        if (kb < nkb && ElectOne()) Commit(accum);
    }
    __syncwarp();

    const bool acc_ok = BarWaitDrain(accum, 0);
    FenceAfterSync();
    if (!acc_ok && threadIdx.x == 0) Flag(cta_err, a.err);
    const bool store = acc_ok && *cta_err == 0;
    for (int j = 0; j < nt; j++) {
        const int q = (j0 + j) * a.tile_step + warp * 32 + lane;
        const int y = q / a.pitch, x = q - y * a.pitch;
        const bool pixel = store && x < a.W && y < a.H;
        const long long pix = ((long long)img * a.H + y) * a.W + x;
        const uint32_t t =
            tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(j * a.bn);
        int c = 0;
        for (; c + 32 <= a.bn; c += 32) {
            float v[32];
            TmemLoad32(t + c, v);
            if (pixel) {
                StoreOutputs(a, pix, n0 + c, v, bias + c);
                StoreOutputs(a, pix, n0 + c + 16, v + 16, bias + c + 16);
            }
            __syncwarp();
        }
        if (c < a.bn) {
            float v[16];
            TmemLoad16(t + c, v);
            if (pixel) StoreOutputs(a, pix, n0 + c, v, bias + c);
        }
    }

    FenceBeforeSync();
    __syncthreads();
    if (warp == 2) {
        FenceAfterSync();
        TmemFree(tmem, a.tmem_cols);
    }
}

__global__ void __launch_bounds__(kConvThreads, 1)
    WgradKernel(const __grid_constant__ CUtensorMap ta,
                const __grid_constant__ CUtensorMap tb, WgradArgs a) {
    constexpr uint32_t ATOM = 16384;   // 128 pixel rows x 64 channels
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = Align1024(smem_raw);
    const uint32_t stage_bytes = (2 + a.b_atoms) * ATOM;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + a.stages * stage_bytes);
    uint64_t* empty = full + a.stages;
    uint64_t* accum = empty + a.stages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    volatile int* cta_err = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ci_tiles = (a.cin + a.bn - 1) / a.bn;
    const int co_tiles = (a.cout + 127) / 128;
    int bx = blockIdx.x;
    const int ci_t = bx % ci_tiles;
    bx /= ci_tiles;
    const int co_t = bx % co_tiles;
    const int tap = bx / co_tiles;
    const int co0 = co_t * 128, ci0 = ci_t * a.bn;
    const int a_atoms = min(2, (a.cout - co0 + 63) / 64);
    const int b_atoms = min(a.b_atoms, (a.cin - ci0 + 63) / 64);
    const uint32_t tx = (uint32_t)(a_atoms + b_atoms) * ATOM;
    const int kb0 = blockIdx.y * a.kb_per_split;
    const int nk = min(a.kb_total, kb0 + a.kb_per_split) - kb0;
    if (nk <= 0) return;   // uniform over the CTA, before any allocation
    int dh, dw;
    TapOffset(a.taps, tap, dh, dw);

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; s++) {
            BarInit(&full[s], 1);
            BarInit(&empty[s], 1);
        }
        BarInit(accum, 1);
        *cta_err = 0;
        FenceBarrierInit();
        PrefetchTmap(&ta);
        PrefetchTmap(&tb);
    }
    if (warp == 2) TmemAlloc(tmem_slot, a.tmem_cols);
    GridWait();
    FenceBeforeSync();
    __syncthreads();
    FenceAfterSync();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        int j = 0;
        for (; j < nk; j++) {
            const int s = j % a.stages;
            if (j >= a.stages &&
                !BarWait(&empty[s], ((j / a.stages) + 1) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            const int g = kb0 + j;
            const int img = g / a.tiles_per_img;
            const int h0 = (g - img * a.tiles_per_img) * a.bh;
            uint8_t* sa = smem + s * stage_bytes;
            BarArriveExpectTx(&full[s], tx);
            for (int at = 0; at < a_atoms; at++)
                TmaLoad4D(sa + at * ATOM, &ta, &full[s], co0 + 64 * at, 0, h0,
                          img);
            for (int bt = 0; bt < b_atoms; bt++)
                TmaLoad4D(sa + (2 + bt) * ATOM, &tb, &full[s], ci0 + 64 * bt,
                          dw, h0 + dh, img);
        }
        for (int q = j > a.stages ? j - a.stages : 0; q < j; q++)
            if (!BarWaitDrain(&full[q % a.stages], (q / a.stages) & 1))
                Flag(cta_err, a.err);
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = InstrDescBf16(kTileM, a.bn, true, true);
        const uint32_t base = SmemAddr(smem);
        for (int j = 0; j < nk; j++) {
            const int s = j % a.stages;
            if (!BarWait(&full[s], (j / a.stages) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            FenceAfterSync();
            const uint32_t sa = base + s * stage_bytes;
            const uint32_t sb = sa + 2 * ATOM;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                Mma(tmem, SmemDesc(sa + k * 2048, ATOM, 1024, 128),
                    SmemDesc(sb + k * 2048, ATOM, 1024, 128), idesc,
                    (j | k) != 0 ? 1u : 0u);
            }
            Commit(&empty[s]);
        }
        Commit(accum);
    }
    __syncwarp();

    const bool acc_ok = BarWaitDrain(accum, 0);
    FenceAfterSync();
    if (!acc_ok && threadIdx.x == 0) Flag(cta_err, a.err);
    const bool store = acc_ok && *cta_err == 0;
    const int co = co0 + warp * 32 + lane;
    for (int c = 0; c < a.bn; c += 16) {
        float v[16];
        TmemLoad16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
        if (!store || co >= a.cout) continue;
        float* d = a.dw + ((long long)co * a.taps + tap) * a.cin;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int ci = ci0 + c + i;
            if (ci < a.cin) atomicAdd(d + ci, v[i]);
        }
    }

    FenceBeforeSync();
    __syncthreads();
    if (warp == 2) {
        FenceAfterSync();
        TmemFree(tmem, a.tmem_cols);
    }
}

__global__ void __launch_bounds__(kConvThreads, 1)
    WgradTKernel(const __grid_constant__ CUtensorMap tx,
                 const __grid_constant__ CUtensorMap tdy, WgradTArgs a) {
    constexpr uint32_t ATOM = 8192;   // 128 pixel rows x 32 channels
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = Align1024(smem_raw);
    const int b_atoms = a.bn / 32;
    const uint32_t stage_bytes = (4 + b_atoms) * ATOM;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + a.stages * stage_bytes);
    uint64_t* empty = full + a.stages;
    uint64_t* accum = empty + a.stages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    volatile int* cta_err = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this CTA's M tile: atoms 4 blockIdx.x .. + 3 (atom = tap * ci_chunks
    // + chunk); the last tile may hold fewer
    const int atom0 = 4 * blockIdx.x;
    const int m_atoms = min(4, a.n_atoms - atom0);
    const uint32_t tx_bytes = (uint32_t)(m_atoms + b_atoms) * ATOM;
    const int kb0 = blockIdx.y * a.kb_per_split;
    const int nk = min(a.kb_total, kb0 + a.kb_per_split) - kb0;
    if (nk <= 0 || m_atoms <= 0) return;   // uniform, before any allocation

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; s++) {
            BarInit(&full[s], 1);
            BarInit(&empty[s], 1);
        }
        BarInit(accum, 1);
        *cta_err = 0;
        FenceBarrierInit();
        PrefetchTmap(&tx);
        PrefetchTmap(&tdy);
    }
    if (warp == 2) TmemAlloc(tmem_slot, a.tmem_cols);
    GridWait();
    FenceBeforeSync();
    __syncthreads();
    FenceAfterSync();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        int j = 0;
        for (; j < nk; j++) {
            const int s = j % a.stages;
            if (j >= a.stages &&
                !BarWait(&empty[s], ((j / a.stages) + 1) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            const int g = kb0 + j;
            const int img = g / a.tiles_per_img;
            const int h0 = (g - img * a.tiles_per_img) * a.bh;
            uint8_t* sa = smem + s * stage_bytes;
            BarArriveExpectTx(&full[s], tx_bytes);
            for (int m = 0; m < m_atoms; m++) {
                const int at = atom0 + m;
                const int tap = at / a.ci_chunks;
                const int chunk = at - tap * a.ci_chunks;
                int dh, dw;
                TapOffset(a.taps, tap, dh, dw);
                TmaLoad4D(sa + m * ATOM, &tx, &full[s], 32 * chunk, dw,
                          h0 + dh, img);
            }
            for (int bt = 0; bt < b_atoms; bt++)
                TmaLoad4D(sa + (4 + bt) * ATOM, &tdy, &full[s], 32 * bt, 0,
                          h0, img);
        }
        for (int q = j > a.stages ? j - a.stages : 0; q < j; q++)
            if (!BarWaitDrain(&full[q % a.stages], (q / a.stages) & 1))
                Flag(cta_err, a.err);
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = InstrDescBf16(kTileM, a.bn, true, true);
        const uint32_t base = SmemAddr(smem);
        for (int j = 0; j < nk; j++) {
            const int s = j % a.stages;
            if (!BarWait(&full[s], (j / a.stages) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            FenceAfterSync();
            const uint32_t sa = base + s * stage_bytes;
            const uint32_t sb = sa + 4 * ATOM;
            // MN-major, 64-byte swizzle: rows of 32 channels per pixel, 8-row
            // groups 512 B apart, atoms (32 M or N rows) 8 KiB apart; 16
            // pixels per MMA
#pragma unroll
            for (int k = 0; k < 8; k++) {
                Mma(tmem, SmemDesc(sa + k * 1024, ATOM, 512, 64),
                    SmemDesc(sb + k * 1024, ATOM, 512, 64), idesc,
                    (j | k) != 0 ? 1u : 0u);
            }
            Commit(&empty[s]);
        }
        Commit(accum);
    }
    __syncwarp();

    const bool acc_ok = BarWaitDrain(accum, 0);
    FenceAfterSync();
    if (!acc_ok && threadIdx.x == 0) Flag(cta_err, a.err);
    const bool store = acc_ok && *cta_err == 0;
    // TMEM lane = M row: atom (warp), channel lane of its chunk; columns are
    // output channels
    const int at = atom0 + warp;
    const int tap = at / a.ci_chunks;
    const int ci = 32 * (at - tap * a.ci_chunks) + lane;
    const bool row_ok = warp < m_atoms && ci < a.cin;
    for (int c = 0; c < a.bn; c += 16) {
        float v[16];
        TmemLoad16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
        if (!store || !row_ok) continue;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int co = c + i;
            if (co < a.cout)
                atomicAdd(a.dw + ((long long)co * a.taps + tap) * a.cin + ci,
                          v[i]);
        }
    }

    FenceBeforeSync();
    __syncthreads();
    if (warp == 2) {
        FenceAfterSync();
        TmemFree(tmem, a.tmem_cols);
    }
}

// The weight gradient of a 3x3 convolution (see conv.cuh): one 32-channel slice
// of the input, bn output channels, a range of bands of image rows.  Cold-cache
// layer times (32 images), tap by tap in brackets: 96 -> 32 at 128^2 61 us (202),
// 32 -> 32 26 (77), 192 -> 64 at 64^2 43 (116), 384 -> 128 at 32^2 54 (78), 128 ->
// 128 22 (43).  Row by row a sum has the terms of a tap's and no others: over
// surplus columns, too, 256 -> 256 at 16^2 rounds 18/16 times as often, 3.0e-7 off
// the 64-bit sums in place of 2.9e-7, and a pixel that a tap does not use enters it
// times zero.  So rows are 16 pixels or a multiple (kWgradBandWidth).
__global__ void __launch_bounds__(kConvThreads, 1)
    WgradBandKernel(const __grid_constant__ CUtensorMap tx,
                    const __grid_constant__ CUtensorMap tdy,
                    const __grid_constant__ CUtensorMap tdw,
                    WgradBandArgs a) {
    constexpr uint32_t SW = 64;   // bytes of a position: 32 channels
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = Align1024(smem_raw);
    const int slices = a.bn / 32;
    const uint32_t stage_bytes = a.x_bytes + slices * a.dy_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(
        smem + WgradBandData(a.stages, a.x_bytes, a.dy_bytes, a.bn));
    uint64_t* empty = full + a.stages;
    uint64_t* accum = empty + a.stages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    volatile int* cta_err = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = 32 * blockIdx.y, n0 = a.bn * blockIdx.z;
    const int b0 = blockIdx.x * a.bands_per_cta;
    const int nb = min(a.bands_total, b0 + a.bands_per_cta) - b0;
    if (nb <= 0) return;   // uniform over the CTA, before any allocation

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; s++) {
            BarInit(&full[s], 1);
            BarInit(&empty[s], 1);
        }
        BarInit(accum, 1);
        *cta_err = 0;
        FenceBarrierInit();
        PrefetchTmap(&tx);
        PrefetchTmap(&tdy);
    }
    if (warp == 2) TmemAlloc(tmem_slot, a.tmem_cols);
    GridWait();
    FenceBeforeSync();
    __syncthreads();
    FenceAfterSync();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        int j = 0;
        for (; j < nb; j++) {
            const int s = j % a.stages;
            if (j >= a.stages &&
                !BarWait(&empty[s], ((j / a.stages) + 1) & 1, cta_err)) {
                Flag(cta_err, a.err);
                break;
            }
            const int img = (b0 + j) / a.bands_per_img;
            const int r0 = (b0 + j - img * a.bands_per_img) * a.rows;
            uint8_t* st = smem + s * stage_bytes;
            BarArriveExpectTx(&full[s],
                              a.x_box + (uint32_t)slices * a.dy_box);
            TmaLoad4D(st, &tx, &full[s], c0, -1, r0 - 1, img);
            for (int i = 0; i < slices; i++)
                TmaLoad4D(st + a.x_bytes + i * a.dy_bytes, &tdy, &full[s],
                          n0 + 32 * i, 0, r0, img);
        }
        for (int q = j > a.stages ? j - a.stages : 0; q < j; q++)
            if (!BarWaitDrain(&full[q % a.stages], (q / a.stages) & 1))
                Flag(cta_err, a.err);
    } else if (warp == 1) {
        // the whole warp walks the loop, one lane issues
        const uint32_t idesc = InstrDescBf16(kTileM, a.bn, true, true);
        // MN-major, 64-byte swizzle.  X: M rows 32 w + c are channel c at the
        // position w further on (lbo one position); dY: slices lbo apart
        const uint32_t base = SmemAddr(smem);
        const int ksteps = a.w / 16;   // of an image row
        int j = 0;
        for (int s = 0, phase = 0; j < nb; j++) {
            const int r0 = (b0 + j) % a.bands_per_img * a.rows;
            const int runs = min(a.rows, a.h - r0);
            if (!__all_sync(~0u, BarWait(&full[s], phase, cta_err))) {
                if (lane == 0) Flag(cta_err, a.err);
                break;
            }
            FenceAfterSync();
            const uint32_t sx = base + s * stage_bytes;
            const uint64_t db =
                SmemDesc(sx + a.x_bytes, (uint32_t)a.dy_bytes, 8 * SW, SW);
            if (ElectOne()) {
                for (int dh = 0; dh < 3; dh++) {
                    const uint64_t da = SmemDesc(sx + dh * a.pitch * SW, SW,
                                                 8 * SW, SW);
                    // a position on: four units of 16 bytes
                    for (int r = 0; r < runs; r++)
                        for (int k = 0; k < ksteps; k++) {
                            const int at = 4 * (r * a.pitch + 16 * k);
                            Mma(tmem + dh * a.bn, da + at, db + at, idesc,
                                (j | r | k) != 0 ? 1u : 0u);
                        }
                }
                Commit(&empty[s]);
                if (j + 1 == nb) Commit(accum);
            }
            __syncwarp();
            if (++s == a.stages) {
                s = 0;
                phase ^= 1;
            }
        }
        if (j < nb && ElectOne()) Commit(accum);
    }
    __syncwarp();

    const bool acc_ok = BarWaitDrain(accum, 0);
    FenceAfterSync();
    if (!acc_ok && threadIdx.x == 0) Flag(cta_err, a.err);
    const bool store = __all_sync(~0u, acc_ok && *cta_err == 0);
    // TMEM lane 32 w + c: tap column w (the fourth belongs to no tap).  The
    // stages are read by now: each warp lays its tap's 32 x bn sums out there,
    // and one bulk reduction adds them to dW, clipped at its edges.  Lane by
    // lane, at about one atomic a cycle and SM, this took most of the layers of
    // few pixels and many channels: 256 -> 256 at 16^2 56 us, in bulk 34.
    const int ci = c0 + lane;
    const uint32_t row = tmem + ((uint32_t)(warp * 32) << 16);
    float* out = reinterpret_cast<float*>(smem) + warp * a.bn * 32;
    for (int dh = 0; dh < 3 && warp < 3; dh++) {
        const int tap = 3 * dh + warp;
        if (a.bulk && dh > 0) {
            if (lane == 0) BulkWaitRead();
            __syncwarp();
        }
        for (int c = 0; c < a.bn; c += 32) {
            float v[32];
            TmemLoad32(row + (uint32_t)(dh * a.bn + c), v);
            if (a.bulk && store) {
#pragma unroll
                for (int i = 0; i < 32; i++) out[(c + i) * 32 + lane] = v[i];
            } else if (store && ci < a.cin) {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    const int co = n0 + c + i;
                    if (co < a.cout)
                        atomicAdd(a.dw + ((long long)co * 9 + tap) * a.cin + ci,
                                  v[i]);
                }
            }
            __syncwarp();
        }
        if (a.bulk && store) {
            FenceProxyAsync();
            __syncwarp();
            if (lane == 0) {
                TmaAdd3D(&tdw, out, c0, tap, n0);
                BulkCommit();
            }
        }
    }
    if (lane == 0) BulkWaitRead();

    FenceBeforeSync();
    __syncthreads();
    if (warp == 2) {
        FenceAfterSync();
        TmemFree(tmem, a.tmem_cols);
    }
}

}  // namespace nn
}  // namespace mplb

// ---------------------------------------------------------------------------
// Host side: tensor maps and launches.
// ---------------------------------------------------------------------------
#include <algorithm>
#include <mutex>
#include <string>

#include "conv_host.h"
#include "conv_plan.h"

namespace mplb {
namespace nn {

namespace {

using tma::EncodeTiledFn;
using tma::Encoder;

bool CheckView(const View& v, const char* what, std::string& err) {
    char buf[256];
    const bool ok = v.ptr != nullptr && v.nimg > 0 && v.w > 0 && v.w <= 128 &&
                    128 % v.w == 0 && v.h > 0 && (v.h * v.w) % 128 == 0 &&
                    v.c > 0 && v.c % 16 == 0 && v.ps >= v.c && v.ps % 8 == 0 &&
                    reinterpret_cast<uintptr_t>(v.ptr) % 16 == 0;
    if (!ok) {
        snprintf(buf, sizeof buf,
                 "%s view unsupported (nimg %d, h %d, w %d, c %d, ps %lld)",
                 what, v.nimg, v.h, v.w, v.c, v.ps);
        err = buf;
    }
    return ok;
}

bool EncodeAct(CUtensorMap* m, const View& v, int box_c, int box_w, int box_h,
               int swizzle, std::string& err) {
    EncodeTiledFn enc = Encoder();
    if (enc == nullptr) {
        err = "cuTensorMapEncodeTiled is not available";
        return false;
    }
    const cuuint64_t dims[4] = {(cuuint64_t)v.c, (cuuint64_t)v.w,
                                (cuuint64_t)v.h, (cuuint64_t)v.nimg};
    const cuuint64_t strides[3] = {(cuuint64_t)v.ps * 2,
                                   (cuuint64_t)v.ps * 2 * v.w,
                                   (cuuint64_t)v.ps * 2 * v.w * v.h};
    const cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)box_w,
                               (cuuint32_t)box_h, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(
        m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, v.ptr, dims, strides, box,
        estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        swizzle == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        err = "tensor map of an activation view rejected (CUresult " +
              std::to_string((int)r) + ")";
        return false;
    }
    return true;
}

// fp32 dW [cout][9][cin]: boxes of 32 input channels of one tap x bn output
// channels.
bool EncodeWeightGrad(CUtensorMap* m, float* dw, int cin, int cout, int bn,
                      std::string& err) {
    EncodeTiledFn enc = Encoder();
    if (enc == nullptr) {
        err = "cuTensorMapEncodeTiled is not available";
        return false;
    }
    const cuuint64_t dims[3] = {(cuuint64_t)cin, 9, (cuuint64_t)cout};
    const cuuint64_t strides[2] = {(cuuint64_t)cin * 4, (cuuint64_t)cin * 36};
    const cuuint32_t box[3] = {32, 1, (cuuint32_t)bn};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(
        m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, dw, dims, strides, box, estr,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
        CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        err = "tensor map of a weight gradient rejected (CUresult " +
              std::to_string((int)r) + ")";
        return false;
    }
    return true;
}

// Boxes of a 128-pixel tile.
bool EncodeTile(CUtensorMap* m, const View& v, int box_c, int swizzle,
                std::string& err) {
    return EncodeAct(m, v, box_c, v.w, 128 / v.w, swizzle, err);
}

bool EncodeRows(CUtensorMap* m, const void* ptr, int rows, int kdim,
                int box_k, int box_rows, int swizzle, std::string& err) {
    EncodeTiledFn enc = Encoder();
    if (enc == nullptr) {
        err = "cuTensorMapEncodeTiled is not available";
        return false;
    }
    if (reinterpret_cast<uintptr_t>(ptr) % 16 != 0 || kdim % 8 != 0) {
        err = "weight matrix misaligned";
        return false;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)kdim, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)kdim * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_k, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(
        m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims,
        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        swizzle == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        err = "tensor map of a weight matrix rejected (CUresult " +
              std::to_string((int)r) + ")";
        return false;
    }
    return true;
}

// Dynamic shared memory for a launch: pads the request so that the CTAs an
// SM can hold never ask for more than its 512 TMEM columns together.
int ResidencySafeSmem(int smem, int tmem_cols) {
    const int max_ctas = 512 / tmem_cols;
    const int floor_bytes = kSmemPerSm / max_ctas - 1024;
    if (smem < floor_bytes) smem = floor_bytes;
    return smem > kSmemMax ? kSmemMax : smem;
}

template <int BK>
cudaError_t SetSmemAttr() {
    static cudaError_t e = cudaFuncSetAttribute(
        ConvKernel<BK>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    return e;
}

template <int BK>
cudaError_t SetBandSmemAttr() {
    static cudaError_t e =
        cudaFuncSetAttribute(ConvBandKernel<BK>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmemMax);
    return e;
}

bool LaunchConvBand(const View& x, const void* w, const BandPlan& p, int bk,
                    const float* bias, int relu, const View& y, bool y_f32,
                    const View* mask, cudaStream_t stream, int* err_dev,
                    std::string& err) {
    ConvBandArgs a{};
    a.H = x.h;
    a.W = x.w;
    a.pitch = x.w + 2;
    a.tile_step = x.w == 128 ? a.pitch : 128;
    a.tiles_per_img =
        x.w == 128 ? x.h : ((x.h - 1) * a.pitch + x.w + 127) / 128;
    a.tiles = p.tiles;
    a.bands = (a.tiles_per_img + p.tiles - 1) / p.tiles;
    a.cin = x.c;
    a.chunks = (x.c + bk - 1) / bk;
    a.chunk_bytes = BandChunkBytes(p.rows, a.pitch, bk);
    a.box_bytes = (uint32_t)(p.rows * a.pitch * bk * 2);
    a.cout = y.c;
    a.bn = p.bn;
    a.group = p.group;
    a.stages = p.stages;
    a.tmem_cols = Pow2Cols(p.tiles * p.bn);
    a.out = y.ptr;
    a.out_ps = y.ps;
    a.out_f32 = y_f32 ? 1 : 0;
    a.bias = bias;
    a.relu = relu;
    a.mask = mask ? static_cast<const __nv_bfloat16*>(mask->ptr) : nullptr;
    a.mask_ps = mask ? mask->ps : 0;
    a.err = err_dev;
    CUtensorMap ta, tb;
    if (!EncodeAct(&ta, x, bk, a.pitch, p.rows, bk * 2, err)) return false;
    if (!EncodeRows(&tb, w, y.c, 9 * x.c, bk, p.bn, bk * 2, err)) return false;
    const int smem = ResidencySafeSmem(p.smem, a.tmem_cols);
    const dim3 grid(x.nimg * a.bands, y.c / p.bn);
    cudaError_t e = bk == 64 ? SetBandSmemAttr<64>() : SetBandSmemAttr<32>();
    if (e == cudaSuccess) {
        if (bk == 64)
            LaunchNext(ConvBandKernel<64>, grid, kConvThreads, smem, stream,
                       ta, tb, a);
        else
            LaunchNext(ConvBandKernel<32>, grid, kConvThreads, smem, stream,
                       ta, tb, a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        err = std::string("convolution launch: ") + cudaGetErrorString(e);
        return false;
    }
    return true;
}

cudaError_t SetWgradTSmemAttr() {
    static cudaError_t e = cudaFuncSetAttribute(
        WgradTKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    return e;
}

cudaError_t SetWgradSmemAttr() {
    static cudaError_t e = cudaFuncSetAttribute(
        WgradKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    return e;
}

}  // namespace

bool LaunchConv(const View& x, const void* w, int taps, const float* bias,
                int relu, const View& y, bool y_f32, const View* mask,
                int sm_count, cudaStream_t stream, int* err_dev,
                std::string& err) {
    if (!CheckView(x, "input", err) || !CheckView(y, "output", err))
        return false;
    if (mask != nullptr && !CheckView(*mask, "mask", err)) return false;
    if ((taps != 9 && taps != 1) || w == nullptr ||
        x.nimg != y.nimg || x.h != y.h || x.w != y.w ||
        (mask != nullptr &&
         (mask->nimg != y.nimg || mask->h != y.h || mask->w != y.w ||
          mask->c < y.c))) {
        err = "convolution shapes do not match";
        return false;
    }
    if (y_f32 && (y.ps % 4 != 0)) {
        err = "fp32 output pixel stride must be a multiple of 4";
        return false;
    }
    const int bk = ConvBk(x.c);
    const int bn = PickBn(y.c);
    if (bn == 0) {
        err = "output channels must be a multiple of 16";
        return false;
    }
    // 1x1 convolutions have no rows to keep in shared memory
    if (taps == 9) {
        const BandPlan p = PlanBand(x.nimg, x.h, x.w, x.c, y.c, sm_count);
        if (p.tiles > 0)
            return LaunchConvBand(x, w, p, bk, bias, relu, y, y_f32, mask,
                                  stream, err_dev, err);
    }
    CUtensorMap ta, tb;
    if (!EncodeTile(&ta, x, bk, bk * 2, err)) return false;
    if (!EncodeRows(&tb, w, y.c, taps * x.c, bk, bn, bk * 2, err)) return false;
    ConvArgs a{};
    a.H = x.h;
    a.W = x.w;
    a.tiles_per_img = x.h * x.w / kTileM;
    a.bh = kTileM / x.w;
    a.cin = x.c;
    a.taps = taps;
    a.nkb = taps * ((x.c + bk - 1) / bk);
    a.cout = y.c;
    a.bn = bn;
    a.stages = ConvStages(bk, bn);
    a.tmem_cols = Pow2Cols(bn);
    a.out = y.ptr;
    a.out_ps = y.ps;
    a.out_coff = 0;
    a.out_f32 = y_f32 ? 1 : 0;
    a.bias = bias;
    a.relu = relu;
    a.mask = mask ? static_cast<const __nv_bfloat16*>(mask->ptr) : nullptr;
    a.mask_ps = mask ? mask->ps : 0;
    a.mask_coff = 0;
    a.err = err_dev;
    const int smem = ResidencySafeSmem(ConvSmemBytes(bk, bn, a.stages),
                                       a.tmem_cols);
    const dim3 grid(x.nimg * a.tiles_per_img, y.c / bn);
    cudaError_t e;
    if (bk == 64) {
        e = SetSmemAttr<64>();
        if (e == cudaSuccess)
            LaunchNext(ConvKernel<64>, grid, kConvThreads, smem, stream,
                       ta, tb, a);
    } else {
        e = SetSmemAttr<32>();
        if (e == cudaSuccess)
            LaunchNext(ConvKernel<32>, grid, kConvThreads, smem, stream,
                       ta, tb, a);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = std::string("convolution launch: ") + cudaGetErrorString(e);
        return false;
    }
    return true;
}

bool LaunchWgradBand(const View& dy, const View& x, float* dw, int sm_count,
                     cudaStream_t stream, int* err_dev, std::string& err) {
    const WgradBandPlan p =
        PlanWgradBand(x.nimg, x.h, x.w, x.c, dy.c, sm_count);
    if (p.rows == 0) {
        err = "weight gradient: a row does not fit in shared memory";
        return false;
    }
    WgradBandArgs a{};
    a.w = x.w;
    a.h = x.h;
    a.pitch = x.w + 2;
    a.cout = dy.c;
    a.cin = x.c;
    a.bn = p.bn;
    a.rows = p.rows;
    a.stages = p.stages;
    a.x_bytes = WgradBandBytes((a.rows + 2) * a.pitch + 3);
    a.dy_bytes = WgradBandBytes(a.rows * a.pitch);
    a.x_box = (uint32_t)((a.rows + 2) * a.pitch * 64);
    a.dy_box = (uint32_t)(a.rows * a.pitch * 64);
    a.bands_per_img = p.bands_per_img;
    a.bands_total = x.nimg * a.bands_per_img;
    a.bands_per_cta = p.bands_per_cta;
    a.tmem_cols = Pow2Cols(3 * a.bn);
    a.dw = dw;
    a.err = err_dev;
    CUtensorMap tx, tdy, tdw{};
    if (!EncodeAct(&tx, x, 32, a.pitch, a.rows + 2, 64, err) ||
        !EncodeAct(&tdy, dy, 32, a.pitch, a.rows, 64, err))
        return false;
    // bulk reductions take 16-byte aligned rows; elsewhere one atomic per lane
    a.bulk = reinterpret_cast<uintptr_t>(dw) % 16 == 0 && x.c % 4 == 0 ? 1 : 0;
    if (a.bulk && !EncodeWeightGrad(&tdw, dw, x.c, dy.c, a.bn, err))
        return false;
    const dim3 grid(p.ctas, p.slices, p.groups);
    const int smem = ResidencySafeSmem(
        WgradBandSmem(a.w, a.rows, a.stages, a.bn), a.tmem_cols);
    static cudaError_t attr = cudaFuncSetAttribute(
        WgradBandKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    cudaError_t e = attr;
    if (e == cudaSuccess) {
        LaunchNext(WgradBandKernel, grid, kConvThreads, smem, stream, tx, tdy,
                   tdw, a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        err = std::string("weight-gradient launch: ") + cudaGetErrorString(e);
        return false;
    }
    return true;
}

bool LaunchWgrad(const View& dy, const View& x, int taps, float* dw,
                 int sm_count, cudaStream_t stream, int* err_dev,
                 std::string& err) {
    if (!CheckView(dy, "output gradient", err) || !CheckView(x, "input", err))
        return false;
    if ((taps != 9 && taps != 1) || dw == nullptr || x.nimg != dy.nimg ||
        x.h != dy.h || x.w != dy.w) {
        err = "weight-gradient shapes do not match";
        return false;
    }
    if (taps == 9 && x.w >= kWgradBandWidth)
        return LaunchWgradBand(dy, x, dw, sm_count, stream, err_dev, err);
    if (dy.c <= 64) {
        // few output channels: taps x input channels along M (WgradTKernel)
        CUtensorMap tx, tdy;
        if (!EncodeTile(&tx, x, 32, 64, err) ||
            !EncodeTile(&tdy, dy, 32, 64, err))
            return false;
        WgradTArgs t{};
        t.H = x.h;
        t.W = x.w;
        t.tiles_per_img = x.h * x.w / kTileM;
        t.bh = kTileM / x.w;
        t.taps = taps;
        t.cout = dy.c;
        t.cin = x.c;
        t.ci_chunks = (x.c + 31) / 32;
        t.n_atoms = taps * t.ci_chunks;
        t.bn = 32 * ((dy.c + 31) / 32);
        t.stages = 4;
        t.tmem_cols = Pow2Cols(t.bn);
        t.kb_total = x.nimg * t.tiles_per_img;
        const int mtiles = (t.n_atoms + 3) / 4;
        t.kb_per_split = WgradTapBlocks(t.kb_total, taps, x.c, dy.c, sm_count);
        const int splits = (t.kb_total + t.kb_per_split - 1) / t.kb_per_split;
        t.dw = dw;
        t.err = err_dev;
        const int smem = ResidencySafeSmem(WgradTSmemBytes(t.bn, t.stages),
                                           t.tmem_cols);
        cudaError_t e = SetWgradTSmemAttr();
        if (e == cudaSuccess)
            LaunchNext(WgradTKernel, dim3(mtiles, splits), kConvThreads, smem,
                       stream, tx, tdy, t);
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e != cudaSuccess) {
            err = std::string("weight-gradient launch: ") +
                  cudaGetErrorString(e);
            return false;
        }
        return true;
    }
    CUtensorMap ta, tb;
    if (!EncodeTile(&ta, dy, 64, 128, err) || !EncodeTile(&tb, x, 64, 128, err))
        return false;
    WgradArgs a{};
    a.H = x.h;
    a.W = x.w;
    a.tiles_per_img = x.h * x.w / kTileM;
    a.bh = kTileM / x.w;
    a.taps = taps;
    a.cout = dy.c;
    a.cin = x.c;
    a.b_atoms = (x.c + 63) / 64;
    if (a.b_atoms > 4) a.b_atoms = 4;
    a.bn = 64 * a.b_atoms;
    a.stages = a.b_atoms >= 3 ? 2 : (a.b_atoms == 2 ? 3 : 4);
    a.tmem_cols = Pow2Cols(a.bn);
    a.kb_total = x.nimg * a.tiles_per_img;
    const int blocks = taps * ((dy.c + 127) / 128) * ((x.c + a.bn - 1) / a.bn);
    a.kb_per_split = WgradTapBlocks(a.kb_total, taps, x.c, dy.c, sm_count);
    const int splits = (a.kb_total + a.kb_per_split - 1) / a.kb_per_split;
    a.dw = dw;
    a.err = err_dev;
    const int smem = ResidencySafeSmem(WgradSmemBytes(a.b_atoms, a.stages),
                                       a.tmem_cols);
    cudaError_t e = SetWgradSmemAttr();
    if (e == cudaSuccess)
        LaunchNext(WgradKernel, dim3(blocks, splits), kConvThreads, smem, stream,
                   ta, tb, a);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = std::string("weight-gradient launch: ") + cudaGetErrorString(e);
        return false;
    }
    return true;
}

}  // namespace nn
}  // namespace mplb
