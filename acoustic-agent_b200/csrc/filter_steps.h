// Steps and sample numbers of the band filter's blocks (band_filter.cuh), host and device.
//
// A signal may have up to 2^31 - 4 samples (synth.cu), and a block loads a few steps past the end of its longest signal.
// Sample numbers are therefore unsigned: as int they came out negative there, which a test against the length takes for
// a sample of the signal.
#pragma once

#if defined(__CUDACC__)
#define AC_HOST_DEVICE __host__ __device__
#else
#define AC_HOST_DEVICE
#endif

namespace ac {

// Steps of `step` samples that cover `n_len`.
AC_HOST_DEVICE constexpr int filter_steps(int n_len, int step) { return n_len / step + (n_len % step != 0 ? 1 : 0); }

// Sample `offset` of step k.
AC_HOST_DEVICE constexpr unsigned filter_sample(int k, int step, int offset) {
    return static_cast<unsigned>(k) * static_cast<unsigned>(step) + static_cast<unsigned>(offset);
}

AC_HOST_DEVICE constexpr bool in_signal(unsigned n, int n_len) { return n < static_cast<unsigned>(n_len); }

}  // namespace ac
