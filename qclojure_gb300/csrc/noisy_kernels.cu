// Kernels of the noisy trajectories (noisy.cpp): the draws of every shot, readout noise and
// the collected final states.
//
// The host did this work before: 20,000 shots of the 300-gate recipe at 10 qubits (0.1 % / 1 %
// depolarizing, about 8,000 distinct states) drew 6 million Kraus choices on the host cores,
// wrote 440 MB of op records into pinned memory allocated for the call and copied them over,
// about 40 of 58 ms. Here a shot's choices cost one Philox draw per site on the device, shots
// are grouped by a 128-bit sum of hashes that is checked against the choices themselves, and
// the tile interpreter looks each state's operators up by its choices (NoiseSites).
#include <algorithm>

#include "qgpu_internal.h"

namespace qg {

namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t x) {  // splitmix64's finaliser
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// One warp per shot: the choice of every site, and the sums of two hashes over the sites
// whose choice is not the first operator.
__global__ void __launch_bounds__(256) k_noise_choices(const NoiseChannel* __restrict__ chans,
                                                       const int32_t* __restrict__ site_chan, int sites,
                                                       uint64_t shot0, int shots, uint64_t seed, uint32_t stream,
                                                       uint8_t* __restrict__ choices, ulonglong2* __restrict__ hash) {
  const int lane = (int)threadIdx.x & 31;
  const int m = (int)(blockIdx.x * 8 + (threadIdx.x >> 5));
  if (m >= shots) return;
  uint64_t ha = 0, hb = 0;
  for (int s = lane; s < sites; s += 32) {
    const NoiseChannel& ch = chans[site_chan[s]];
    uint32_t c = 0;
    if (ch.count > 1) {
      const uint64_t u = draw64(seed, shot0 + (uint64_t)m, stream + (uint32_t)s) >> 11;
      while ((int)c < ch.count - 1 && u >= ch.below[c]) ++c;
    }
    choices[(size_t)m * sites + s] = (uint8_t)c;
    if (c) {
      const uint64_t k = mix64(((uint64_t)s << 2 | c) + 0x9E3779B97F4A7C15ull);
      ha += k;
      hb += mix64(k ^ 0xD1B54A32D192ED03ull);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    ha += __shfl_xor_sync(0xffffffffu, ha, o);
    hb += __shfl_xor_sync(0xffffffffu, hb, o);
  }
  if (lane == 0) hash[m] = make_ulonglong2(ha, hb);
}

// One warp per shot: *differ is set when a shot's choices are not those of its state's shot.
__global__ void __launch_bounds__(256) k_noise_verify(const uint8_t* __restrict__ choices, int sites, int shots,
                                                      const int32_t* __restrict__ state_of,
                                                      const int32_t* __restrict__ reps, int32_t* __restrict__ differ) {
  const int lane = (int)threadIdx.x & 31;
  const int m = (int)(blockIdx.x * 8 + (threadIdx.x >> 5));
  if (m >= shots) return;
  const int r = reps[state_of[m]];
  if (r == m) return;
  bool bad = false;
  for (int s = lane; s < sites; s += 32)
    bad |= choices[(size_t)m * sites + s] != choices[(size_t)r * sites + s];
  if (bad) *differ = 1;
}

// One thread per shot: readout noise qubit by qubit (noise.clj:107-160); factors[source * n +
// target], NaN where none is given (null: no correlations).
__global__ void __launch_bounds__(256) k_noise_readout(uint64_t* __restrict__ outcomes, int shots, int n, uint64_t seed,
                                                       uint64_t shot0, uint32_t stream, double p01, double p10,
                                                       const double* __restrict__ factors) {
  const int m = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (m >= shots) return;
  uint64_t bits = outcomes[m], flipped = 0;  // bit q: qubit q has flipped (in qubit order)
  for (int q = 0; q < n; ++q) {
    const int b = n - 1 - q;
    double f = 1.0;
    if (factors)
      for (uint64_t h = flipped; h; h &= h - 1) {
        const double c = factors[(__ffsll((long long)h) - 1) * n + q];
        if (!isnan(c)) f = __dmul_rn(f, c);
      }
    const double eff = fmin(1.0, fmax(0.0, __dmul_rn(((bits >> b) & 1) ? p10 : p01, f)));
    const double u = (double)(draw64(seed, shot0 + (uint64_t)m, stream + (uint32_t)q) >> 11) * 0x1p-53;
    if (u < eff) {
      bits ^= 1ULL << b;
      flipped |= 1ULL << q;
    }
  }
  outcomes[m] = bits;
}

// out[t] = state state_of[first + t] without its padding qubits, as complex128. The shot is the
// grid's x: up to 65536 shots of one batch are collected at once, and y ends at 65535.
template <typename T>
__global__ void __launch_bounds__(256) k_noise_collect(void* const* __restrict__ states,
                                                       const int32_t* __restrict__ state_of, int first, int n, int shift,
                                                       double2* __restrict__ out) {
  const T* s = reinterpret_cast<const T*>(states[state_of[first + (int)blockIdx.x]]);
  double2* o = out + ((uint64_t)blockIdx.x << n);
  for (uint64_t i = (uint64_t)blockIdx.y * blockDim.x + threadIdx.x; i < (1ULL << n); i += (uint64_t)gridDim.y * blockDim.x) {
    const T v = s[i << shift];
    o[i] = make_double2((double)v.x, (double)v.y);
  }
}

}  // namespace

cudaError_t launch_noise_choices(const NoiseChannel* d_chans, const int32_t* d_site_chan, int sites, uint64_t shot0,
                                 int shots, uint64_t seed, uint32_t stream, uint8_t* d_choices, void* d_hash,
                                 cudaStream_t st) {
  k_noise_choices<<<(unsigned)(shots + 7) / 8, 256, 0, st>>>(d_chans, d_site_chan, sites, shot0, shots, seed, stream,
                                                             d_choices, (ulonglong2*)d_hash);
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t launch_noise_verify(const uint8_t* d_choices, int sites, const int32_t* d_state_of, int shots,
                                const int32_t* d_reps, int32_t* d_differ, cudaStream_t st) {
  if (sites < 1) return cudaSuccess;
  k_noise_verify<<<(unsigned)(shots + 7) / 8, 256, 0, st>>>(d_choices, sites, shots, d_state_of, d_reps, d_differ);
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t launch_noise_readout(uint64_t* d_outcomes, int shots, int n, uint64_t seed, uint64_t shot0, uint32_t stream,
                                 double p01, double p10, const double* d_factors, cudaStream_t st) {
  k_noise_readout<<<(unsigned)(shots + 255) / 256, 256, 0, st>>>(d_outcomes, shots, n, seed, shot0, stream, p01, p10,
                                                                 d_factors);
  count_launch(1);
  return cudaGetLastError();
}

cudaError_t launch_noise_collect(int precision, void* const* d_states, const int32_t* d_state_of, int first, int count,
                                 int n, int shift, double* d_out, cudaStream_t st) {
  const dim3 grid((unsigned)count, (unsigned)std::min<uint64_t>(((1ULL << n) + 255) / 256, 1024));
  if (precision == QG_C64)
    k_noise_collect<float2><<<grid, 256, 0, st>>>(d_states, d_state_of, first, n, shift, (double2*)d_out);
  else
    k_noise_collect<double2><<<grid, 256, 0, st>>>(d_states, d_state_of, first, n, shift, (double2*)d_out);
  count_launch(1);
  return cudaGetLastError();
}

}  // namespace qg
