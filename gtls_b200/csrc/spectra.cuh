// Spectra (spectra.cu), shared by gtls_spectra and its allocation-free form.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace gtls {

struct SpecState {
  double count, mean_sr, mean_power;
  double sde_raw, sde;
};

constexpr int kSpecCtas = 4 * 148;                   // CTAs of a launch, at most
constexpr size_t kSpecParts = 6 * (size_t)kSpecCtas; // partial results of the launches

struct SpecScratch {
  double* part;       // [kSpecParts]
  SpecState* state;
  double* med;        // [n], read and written only where the median's tiles are not used
};

// Launches the spectra of n periods with a running median over k (none when n
// <= 2 k: state->sde is then not set).  Returns the number of launches.
int spectra_launch(const double* chi2, const uint8_t* mask, long long n, int k, double* sr, double* praw,
                   double* power, SpecScratch s, cudaStream_t st);

// Window of the running median for an oversampling factor: 30 times it, made
// odd (stats.py:108-112); 0 when that is no whole number of at least 1.  (Up to
// 4e18, so that twice the window is still a 64-bit number.)
inline long long spectra_window(double oversampling_factor) {
  const double kd = oversampling_factor * 30;
  if (!(kd >= 1 && kd <= 4e18) || kd != (double)(long long)kd) return 0;
  const long long k = (long long)kd;
  return k + 1 - k % 2;
}

}  // namespace gtls
