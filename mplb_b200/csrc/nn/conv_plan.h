// How a 3x3 convolution's work is cut for its kernels: plain host arithmetic
// (conv.cuh has the kernels).
#pragma once

namespace mplb {
namespace nn {

// Images narrower than this take the 3x3 weight gradient tap by tap.  A band
// (WgradBandKernel) sums whole 16-position steps of one image row; a narrower
// row would fill up its step with the row's two halo columns and the next row,
// where a zero of dY meets a pixel of X that the tap does not use, and an
// infinity or NaN there would enter the tap's sum.
constexpr int kWgradBandWidth = 16;

}  // namespace nn
}  // namespace mplb
