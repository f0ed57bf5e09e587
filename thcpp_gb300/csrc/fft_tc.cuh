// 3-D DFTs of many fields as tensor-core products (fft_tc.cu).
#pragma once

#include "common.cuh"

namespace thc {

// Axes of at most kFftTcMaxN (a product's work grows with n, an FFT's with log n: 131 is still
// six times faster) and at least kFftTcMin values in all (a chunk is seven launches).  Real
// fields, cuFFT against these products, ms: 24x25x27 x 30 (4.9e5 values) 0.057 / 0.070,
// x 97 (1.6e6) 0.137 / 0.112, 48^3 x 64 0.61 / 0.33, 48^3 x 256 2.39 / 1.21, 60x64x54 x 512
// 11.3 / 4.1, 17x97x131 x 64 5.1 / 0.87.  A chunk's digits take a quarter of Ctx::digit_bytes, at
// most kFftTcChunk (its default's quarter), and its buffers less than 2 GB; keeping its digits in
// L2 (64 MB) costs more in launches and last waves (1.41 at 48^3 x 256) than it saves.
constexpr int kFftTcMaxN = 256;
constexpr double kFftTcMin = 1e6;
constexpr size_t kFftTcChunk = (size_t)768 << 20;

// Whether `count` fields of n0 x n1 x n2 go this way.
bool fft_tc_fits(const Ctx* c, int n0, int n1, int n2, int count);
// Unnormalised forward DFTs of `count` fields stored back to back (C order, z fastest), real or
// (re, im) pairs: out[field][kz][ky][kx] as pairs, kz < n2 / 2 + 1 for real fields, < n2 else.
// *done = false (and THC_OK, out untouched) when its workspace is not to be had: the caller
// takes cuFFT, whose spectra have kz fastest.
int fft_tc(Ctx* c, int n0, int n1, int n2, int count, bool real, const double* in, double* out,
           bool* done);
void dft_release(Ctx* c);

}  // namespace thc
