// Implicit-GEMM 2D convolutions on the 5th-generation tensor cores.
//
// Activations are NHWC bf16 "views": a base pointer, a pixel stride (elements
// between consecutive pixels, >= channels, a multiple of 8) and a channel
// count, so a convolution can read or write a channel slice of a wider
// (concatenated) buffer.  Weights are bf16 [cout][taps][cin] (taps = 9 for a
// 3x3 kernel with one pixel of zero padding, 1 for 1x1).
//
// ConvKernel computes, for a tile of 128 consecutive pixels (M) and `bn`
// output channels (N), D = sum over taps t and input channels c of
// X[pixel + offset(t)][c] * Wt[n][t][c] (K = taps * cin), with the pixels of
// the tile fetched by one TMA box per k-block: box (BK channels, W pixels,
// 128 / W rows) at the tap's shifted coordinates, whose out-of-image parts
// TMA fills with zeros (the padding).  A and B are K-major, swizzled by BK * 2
// bytes; the accumulator lives in TMEM (128 lanes x bn fp32 columns).  The
// same kernel is the data gradient of a convolution when it is given the
// output gradient as X and the flipped, transposed weights
// W'[c][8 - t][n] = W[n][t][c].
//
// ConvBandKernel is the 3x3 form for inputs that fit in shared memory.
// Fetching each tap's box by itself moves the input nine times from L2 into
// shared memory, which bound the layers of 32-64 channels.  Here a CTA takes a
// band of tiles and loads the band's input rows once, with the pixel of halo on
// every side (TMA's fill gives the padding): position q = y (W + 2) + x of a
// slice of BK channels is row q of the buffer, so tap (dh, dw) of the tile
// whose first output is at position q is the same buffer read from row
// q + (dh + 1) (W + 2) + (dw + 1) on.  A tile is 128 consecutive positions; the
// two columns of halo among them are computed and not stored (images of 128
// columns step by W + 2 instead and have none).  The swizzle follows the
// shared-memory address, so a tile may start at any row of the swizzle
// pattern.  Weights stream through a ring, one (tap, slice) for all tiles of
// the band.  Tap and slice follow each other as in ConvKernel, so the sums are
// the same bits.
//
// The weight gradient of a 3x3 convolution over rows of 16 pixels or more is
// WgradBandKernel's (below); the two that follow serve narrower rows and 1x1
// convolutions.  WgradKernel computes dW[n][t][c] += sum over pixels p of
// dY[p][n] * X[p + offset(t)][c]: M = 128 output channels, N = input channels, K = a
// range of 128-pixel blocks (split over CTAs, accumulated with fp32 atomics).
// Both operands arrive pixel-major with channels contiguous, i.e. MN-major,
// as 64-channel TMA boxes swizzled by 128 bytes.
//
// Warp roles (128 threads): warp 0 issues TMA loads, warp 1 issues MMAs,
// warp 2 owns the TMEM allocation, all four warps run the epilogue (warp w
// reads TMEM lanes 32w..32w+31).  Barrier waits are bounded; a CTA that
// gives up sets `err` and skips its stores.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "conv_plan.h"

namespace mplb {
namespace nn {

constexpr int kConvThreads = 128;

struct ConvArgs {
    int H, W;              // image size in pixels
    int tiles_per_img;     // H * W / 128
    int bh;                // image rows per 128-pixel tile (128 / W)
    int cin;               // channels of the input view (K per tap, padded
                           // to BK with zeros by the tensor map)
    int taps;              // 9 or 1
    int nkb;               // k-blocks: taps * ceil(cin / BK)
    int cout;              // valid output channels
    int bn;                // UMMA N of one CTA
    int stages;            // pipeline depth
    int tmem_cols;         // TMEM columns allocated (power of two >= bn)
    // epilogue
    void* out;             // bf16 or fp32 view
    long long out_ps;      // pixel stride of out (elements)
    int out_coff;          // channel offset of out
    int out_f32;           // 1: fp32 output, 0: bf16
    const float* bias;     // per output channel, or null
    int relu;              // apply max(0, .)
    const __nv_bfloat16* mask;   // multiply by (mask > 0), or null
    long long mask_ps;
    int mask_coff;
    int* err;              // set to 1 when a wait gives up
};

struct ConvBandArgs {
    int H, W;
    int pitch;             // positions per image row: W + 2
    int tile_step;         // positions between tiles
    int tiles_per_img;
    int tiles, bands;      // tiles of a band (CTA), bands of an image
    int cin;
    int chunks;            // BK-channel slices of the input
    int chunk_bytes;       // shared memory of one slice of a band's input
    uint32_t box_bytes;    // of its TMA box
    int cout, bn;
    int group;             // k-blocks (tap, slice) per stage of the weight ring
    int stages;
    int tmem_cols;
    void* out;
    long long out_ps;
    int out_coff;
    int out_f32;
    const float* bias;
    int relu;
    const __nv_bfloat16* mask;
    long long mask_ps;
    int mask_coff;
    int* err;
};

struct WgradArgs {
    int H, W, tiles_per_img, bh;
    int taps;
    int cout, cin;         // dW is [cout][taps][cin]
    int bn;                // UMMA N: 64 * b_atoms
    int b_atoms;           // 64-channel boxes of X per stage (<= 4)
    int kb_total;          // 128-pixel blocks in the batch
    int kb_per_split;
    int stages;
    int tmem_cols;
    float* dw;
    int* err;
};

// Weight gradient of layers with few output channels (cout <= 64), with the
// roles of the operands swapped: M = 128 rows of (tap, 32-channel chunk of
// the input) pairs - four "atoms", each one 32-channel TMA box of X at its
// tap's shifted coordinates - N = the output channels (32 or 64, from
// 32-channel boxes of dY), K = 128-pixel blocks split over CTAs.  Both
// operands MN-major, swizzled by 64 bytes.  Padding M to 128 for 32 output
// channels and N to 64 for 32 input channels, as WgradKernel does for
// these layers, wasted 7/8 of the tensor work.
struct WgradTArgs {
    int H, W, tiles_per_img, bh;
    int taps;
    int cout, cin;         // dW is [cout][taps][cin]
    int ci_chunks;         // 32-channel chunks of the input
    int n_atoms;           // taps * ci_chunks
    int bn;                // UMMA N: 32 * ceil(cout / 32)
    int kb_total;          // 128-pixel blocks in the batch
    int kb_per_split;
    int stages;
    int tmem_cols;
    float* dw;
    int* err;
};

// Weight gradient of a 3x3 convolution with its operands resident: a band of
// image rows of one 32-channel slice of X (with its halo) and of bn channels of
// dY in shared memory serve all nine taps (tap by tap X moved nine times through
// L2).  Both are laid out W + 2 positions to a row, and tap (dh, dw) pairs dY's
// position q with X's position q + dh (W + 2) + dw, for the W positions of each
// row.  M = 128 rows are the slice at four consecutive dw - three of them taps:
// the operand descriptor steps one position between its 32-row atoms - N = the
// output channels, one accumulator per dh.  CTAs sum ranges of bands and add
// them to dW in fp32 (bulk reductions).
struct WgradBandArgs {
    int w, h;              // image
    int pitch;             // positions per row: W + 2
    int rows;              // of a band
    int bands_per_img, bands_total, bands_per_cta;
    int cout, cin;         // dW is [cout][9][cin]
    int bn;                // UMMA N: 32 per slice of dY
    int x_bytes, dy_bytes; // shared memory of a slice of a band
    uint32_t x_box, dy_box;   // bytes of their TMA boxes
    int stages;
    int tmem_cols;         // >= 3 bn
    int bulk;              // dW takes bulk reductions
    float* dw;
    int* err;
};

__global__ void WgradBandKernel(const __grid_constant__ CUtensorMap tx,
                                const __grid_constant__ CUtensorMap tdy,
                                const __grid_constant__ CUtensorMap tdw,
                                WgradBandArgs a);

template <int BK>
__global__ void ConvBandKernel(const __grid_constant__ CUtensorMap ta,
                               const __grid_constant__ CUtensorMap tb,
                               ConvBandArgs a);

template <int BK>
__global__ void ConvKernel(const __grid_constant__ CUtensorMap ta,
                           const __grid_constant__ CUtensorMap tb,
                           ConvArgs a);

__global__ void WgradTKernel(const __grid_constant__ CUtensorMap tx,
                             const __grid_constant__ CUtensorMap tdy,
                             WgradTArgs a);

__global__ void WgradKernel(const __grid_constant__ CUtensorMap ta,
                            const __grid_constant__ CUtensorMap tb,
                            WgradArgs a);

// Shared memory of the weight gradients' launches (the convolutions' and a
// band's sizes are in conv_plan.h).
inline int WgradSmemBytes(int b_atoms, int stages) {
    return 1024 + stages * ((2 + b_atoms) * 16384) + 256;
}
// WgradTKernel: per stage four 8 KiB X atoms and bn / 32 8 KiB dY atoms.
inline int WgradTSmemBytes(int bn, int stages) {
    return 1024 + stages * ((4 + bn / 32) * 8192) + 256;
}

}  // namespace nn
}  // namespace mplb
