// How a 3x3 convolution's work is cut for its kernels: plain host arithmetic
// (conv.cuh has the kernels).
#pragma once

#include <algorithm>

#ifdef __CUDACC__
#define MPLB_HD __host__ __device__
#else
#define MPLB_HD
#endif

namespace mplb {
namespace nn {

constexpr int kTileM = 128;
constexpr int kSmemPerSm = 228 * 1024;
constexpr int kSmemMax = 227 * 1024;

inline int Pow2Cols(int n) {
    int c = 32;
    while (c < n) c *= 2;
    return c;
}

// Largest divisor of c that is a multiple of 16 and at most 256.
inline int PickBn(int c) {
    for (int bn = 256; bn >= 16; bn -= 16)
        if (c % bn == 0) return bn;
    return 0;
}

// Input channels of a k-block.
inline int ConvBk(int cin) { return cin % 64 == 0 ? 64 : 32; }

// Shared memory a launch needs (stage buffers + 1 KiB alignment slack +
// barriers).
inline int ConvSmemBytes(int bk, int bn, int stages) {
    return 1024 + stages * (kTileM * bk * 2 + bn * bk * 2) + 256;
}
inline int ConvStages(int bk, int bn) {
    int stages = 4;
    while (stages > 2 && ConvSmemBytes(bk, bn, stages) > 200 * 1024) stages--;
    return stages;
}
// ConvBandKernel: a slice of a band's input - the last tile reads up to two
// positions past its rows - and the whole launch.
inline int BandChunkBytes(int rows, int pitch, int bk) {
    return ((rows * pitch + 2) * bk * 2 + 1023) / 1024 * 1024;
}
inline int BandSmemBytes(int chunks, int chunk_bytes, int stages,
                         int stage_bytes, int bn, int bk) {
    return 1024 + chunks * chunk_bytes + stages * (stage_bytes + 16) +
           bn * 4 + 8 * chunks + 64;
}

// How a 3x3 convolution is cut into bands; tiles == 0: tap by tap instead.
struct BandPlan {
    int tiles = 0;    // per CTA
    int bn = 0;
    int rows = 0;     // image rows of a band's input box
    int group = 0;    // k-blocks of a weight stage
    int stages = 0;
    int smem = 0;
    int per_sm = 0;   // CTAs of an SM at a time
    long long ctas = 0;
};

// Microseconds of a 3x3 convolution's launch, tap by tap and in bands, roughly:
// fitted to the times of 1,696 shapes with cold caches and 977 with the input in
// L2: 2,048 to 524,288 pixels, rows of 1 to 128 pixels, 16 to 128 input and 16 to
// 384 output channels.
// `per` CTAs fall to the fullest SM, `rounds` one after the other.
//
// Tap by tap: a round's start, its k-blocks one behind the other (the loads'
// latency), the MMAs' time, the accumulators' way out, and the boxes of slices
// that are half filled (32-byte lines).
inline double TapMicroseconds(long long pixels, int cin, int cout,
                              int sm_count) {
    const int bk = ConvBk(cin), bn = PickBn(cout);
    const int nkb = 9 * ((cin + bk - 1) / bk);
    const int smem = ConvSmemBytes(bk, bn, ConvStages(bk, bn)) + 1024;
    const int per_sm = std::max(1, std::min(512 / Pow2Cols(bn),
                                            kSmemPerSm / smem));
    const long long ctas = pixels / kTileM * (cout / bn);
    const double per = (double)((ctas + sm_count - 1) / sm_count);
    const double rounds = (double)(((long long)per + per_sm - 1) / per_sm);
    const double mma = nkb * (bk / 16) * std::max(32.0, bn / 4.0) * 1e-3;
    return 2.1 + rounds * (1.25 + 0.333 * nkb) +
           per * (0.385 * mma + 0.0141 * bn + (cin % 32 ? 0.97 : 0.0));
}
// In bands: the waits for weight stages and the MMAs of a round, the input and
// the accumulators of every CTA.
inline double BandMicroseconds(const BandPlan& p, int pitch, int cin,
                               int sm_count) {
    const int bk = ConvBk(cin), chunks = (cin + bk - 1) / bk, nkb = 9 * chunks;
    const double per = (double)((p.ctas + sm_count - 1) / sm_count);
    const double rounds = (double)(((long long)per + p.per_sm - 1) / p.per_sm);
    const double mma =
        nkb * (bk / 16) * p.tiles * std::max(32.0, p.bn / 4.0) * 1e-3;
    const double input = (double)p.rows * pitch * bk * 2 * chunks * 1e-4;
    return 2.9 + rounds * (1.1 * ((nkb + p.group - 1) / p.group) + 0.24 * mma) +
           per * (0.3 * input + 0.016 * p.tiles * p.bn);
}

// Tiles and output channels of a CTA (cold-L2 times of the network's layers, 32
// images, against tap by tap: 32 -> 32 channels at 128^2 28 us, was 46; 64 -> 64
// at 64^2 24, was 28; 128 -> 128 at 32^2 19, was 22), with fewer output channels
// while the GPU is not full.  Above 128 input channels the
// band fills the shared memory that the weights stream through (192 -> 64 at
// 64^2 64 us, was 61; 384 -> 128 at 32^2 108, was 53).  Below, bands where they
// take no more time by the estimates above: they read the input once for at most
// 128 output channels (tap by tap 256) and compute W + 2 columns of W, so that
// 128 -> 256 at 16^2 takes 18 us in bands and 14 tap by tap (64 images 28 and
// 14), 128 -> 384 at 32^2, 8 images, 19 and 14, 64 -> 64 at 32768 x 4 250 and
// 220.  Within 4 % bands are taken: behind another launch of a pass they do
// better than alone (predictions of 16 images 356 us with the 4 %, 361 without).
// The choice is on average 0.8 % slower than the faster form with cold caches and
// 0.6 % with the input in L2 (always bands 14 and 6 %, always tap by tap 10 and
// 15 %), and by more than a tenth in 74 of the 2,673 shapes.
inline BandPlan PlanBand(int nimg, int H, int W, int cin, int cout,
                         int sm_count) {
    BandPlan p;
    if (cin > 128) return p;
    const int bk = ConvBk(cin);
    const int pitch = W + 2, step = W == 128 ? pitch : 128;
    const int per_img = W == 128 ? H : ((H - 1) * pitch + W + 127) / 128;
    const int chunks = (cin + bk - 1) / bk, nkb = 9 * chunks;
    int bn = 128;
    while (cout % bn != 0) bn -= 16;
    int tiles = 1;
    const auto ctas = [&] {
        return (long long)nimg * ((per_img + tiles - 1) / tiles) * (cout / bn);
    };
    while (bn % 32 == 0 && bn > 32 && ctas() < sm_count) bn /= 2;
    // Tiles of a CTA: its accumulators leave half of TMEM to another CTA.  An SM
    // gets `per` CTAs, `per_sm` at a time, each such round costs about as much as
    // a tile, and the fullest SM is the launch's time: 64 -> 64 at 64^2 (32
    // images, 33 tiles each) 28 us with 1 tile, 25 with 2, 27 with 3; 32 -> 64
    // 21, 19, 21 and with 4 17; 96 -> 32 at 128^2, 3 images, 19, 17, 12 and 15.
    long long best = 0;
    for (int most = std::min({4, bn <= 64 ? 4 : bn <= 96 ? 2 : 1, per_img});
         tiles <= most; tiles++) {
        const int rows = (W == 128 ? (tiles - 1) * step + 127
                                   : pitch - 1 + (tiles - 1) * step + 127) /
                             pitch + 3;
        if (rows > 256) break;
        const int chunk = BandChunkBytes(rows, pitch, bk);
        const int kb_bytes = bn * bk * 2;
        for (int per_sm = 2; per_sm >= 1; per_sm--) {
            const int room = std::min(kSmemPerSm / per_sm - 2048, kSmemMax);
            const int left = room - BandSmemBytes(chunks, chunk, 0, 0, bn, bk);
            if (left < std::min(3, nkb) * (kb_bytes + 16)) continue;
            const long long per = (ctas() + sm_count - 1) / sm_count;
            const long long cost = (per + per_sm - 1) / per_sm + per * tiles;
            if (p.tiles > 0 && cost > best) break;
            best = cost;
            // Waiting for a stage, committing it and forming its addresses
            // cost about 500 cycles, as much as 12 MMAs: a stage holds enough
            // k-blocks for 72, or all that fit (the other CTA of the SM runs
            // meanwhile): 96 -> 32 at 128^2 90 us, with 32 98; 128 -> 128 at
            // 32^2 18.5, with a third of what fits 20.2
            const int mmas = tiles * (bk / 16);
            p.group = std::min({nkb, (72 + mmas - 1) / mmas,
                                left / (kb_bytes + 16)});
            p.stages = std::min((nkb + p.group - 1) / p.group,
                                left / (p.group * kb_bytes + 16));
            p.tiles = tiles;
            p.bn = bn;
            p.rows = rows;
            p.smem = BandSmemBytes(chunks, chunk, p.stages,
                                   p.group * kb_bytes, bn, bk);
            p.per_sm = per_sm;
            p.ctas = ctas();
            break;
        }
    }
    if (p.tiles > 0 &&
        BandMicroseconds(p, pitch, cin, sm_count) >=
            1.04 * TapMicroseconds((long long)nimg * H * W, cin, cout,
                                   sm_count))
        p.tiles = 0;
    return p;
}

// Images narrower than this take the 3x3 weight gradient tap by tap.  A band
// (WgradBandKernel) sums whole 16-position steps of one image row; a narrower
// row would fill up its step with the row's two halo columns and the next row,
// where a zero of dY meets a pixel of X that the tap does not use, and an
// infinity or NaN there would enter the tap's sum.
constexpr int kWgradBandWidth = 16;

// WgradBandKernel: shared memory of a slice of so many positions; of the stages,
// in whose place the sums of three taps are laid out at the end; of a launch.
inline int WgradBandBytes(int positions) {
    return (positions * 64 + 1023) / 1024 * 1024;
}
MPLB_HD inline int WgradBandData(int stages, int x_bytes, int dy_bytes,
                                 int bn) {
    const int ring = stages * (x_bytes + bn / 32 * dy_bytes);
    const int sums = 3 * bn * 32 * 4;
    return ring > sums ? ring : sums;
}
inline int WgradBandSmem(int w, int rows, int stages, int bn) {
    const int pitch = w + 2;
    return 1024 + 256 +
           WgradBandData(stages, WgradBandBytes((rows + 2) * pitch + 3),
                         WgradBandBytes(rows * pitch), bn);
}

// 128-pixel blocks that one accumulator of the tap-by-tap weight gradients sums
// (WgradTKernel up to 64 output channels, WgradKernel above): two CTAs per SM.
inline int WgradTapBlocks(long long blocks, int taps, int cin, int cout,
                          int sm_count) {
    long long tiles;   // of M and N, split `splits` times over the blocks
    if (cout <= 64) {
        tiles = (taps * ((cin + 31) / 32) + 3) / 4;
    } else {
        const int bn = 64 * std::min(4, (cin + 63) / 64);
        tiles = (long long)taps * ((cout + 127) / 128) * ((cin + bn - 1) / bn);
    }
    const long long splits = std::max(
        1LL, std::min((2LL * sm_count + tiles - 1) / tiles, blocks));
    return (int)((blocks + splits - 1) / splits);
}

// How a 3x3 weight gradient is cut into bands of image rows.
struct WgradBandPlan {
    int bn = 0;              // output channels of a CTA
    int slices = 0;          // of 32 input channels
    int groups = 0;          // of bn output channels
    int rows = 0;            // of a band; 0: no plan
    int bands_per_img = 0;
    int bands_per_cta = 0;
    int ctas = 0;            // of a slice and group
    int stages = 0;
};

// One CTA is on an SM at a time (a training step, with an atomic per lane, 535
// us in these kernels, with two per SM 701).  Every height of bands that fits is
// tried with every number of rounds of CTAs, and the shortest launch taken: a
// round takes about 4.5 us and 1 ns for each 30 bytes of its CTAs' operands (a
// band reads two rows more than it has), fitted to 32 and 64 images of the
// network's layers.  Heights are even over an image (16 rows are two bands of 8,
// never 15 and 1), and a CTA has at least 128 pixels to pay for its sums' way
// out.
//
// A CTA sums its pixels in one fp32 accumulator, and the error against 64-bit
// sums grows with their number.  So it sums no more than the tap-by-tap kernels
// do (384 -> 128 at 32^2, 32 images: 1.38e-6 off with their 2,048 pixels, 1.97e-6
// with 2,912), and no more than twice an SM's share of one group of output
// channels (256 -> 256 at 16^2: 2.9e-7 with 512 pixels, 6.4e-7 with 1,024).
inline WgradBandPlan PlanWgradBand(int nimg, int h, int w, int cin, int cout,
                                   int sm_count) {
    WgradBandPlan p;
    p.bn = 32 * std::min(4, (cout + 31) / 32);
    p.slices = (cin + 31) / 32;
    p.groups = (cout + p.bn - 1) / p.bn;
    const long long pixels = (long long)nimg * h * w;
    const long long share = 2 * pixels * p.slices / sm_count;
    const long long most = std::min<long long>(
        128LL * WgradTapBlocks(pixels / 128, 9, cin, cout, sm_count),
        std::max(128LL, share));
    const long long planes = (long long)p.slices * p.groups;
    double best = 0;
    for (int rows = std::min(h, 250); rows >= 1; rows--) {
        const int per_img = (h + rows - 1) / rows;
        if ((h + per_img - 1) / per_img != rows ||
            WgradBandSmem(w, rows, 2, p.bn) > kSmemMax)
            continue;
        const long long bands = (long long)nimg * per_img;
        const long long band = (long long)rows * w;
        if (band > most) continue;
        const long long fewest = std::min(bands, (127 + band) / band);
        // rounds: from the first in which no CTA has more than `most` pixels
        const long long first = (bands + most / band - 1) / (most / band);
        long long rounds = (first * planes + sm_count - 1) / sm_count;
        for (int tries = 0; tries < 3; tries++, rounds++) {
            const long long ctas = rounds * sm_count / planes;
            const long long per =
                std::max(fewest, (bands + ctas - 1) / std::max(1LL, ctas));
            if (ctas < 1 || per * band > most) continue;
            const long long used = (bands + per - 1) / per;
            const double time =
                (double)((used * planes + sm_count - 1) / sm_count) *
                    ((double)(per * band) *
                         (64.0 * (rows + 2) / rows + 2.0 * p.bn) / 30 +
                     4500) +
                (double)used * 1e-3;
            if (p.rows != 0 && time >= best) continue;
            best = time;
            p.rows = rows;
            p.bands_per_img = per_img;
            p.bands_per_cta = (int)per;
            p.ctas = (int)used;
        }
    }
    p.stages = 2;
    while (p.rows != 0 && p.stages < 4 &&
           WgradBandSmem(w, p.rows, p.stages + 1, p.bn) <= kSmemMax)
        p.stages++;
    return p;
}

}  // namespace nn
}  // namespace mplb
