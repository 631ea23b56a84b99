// Device helpers shared by the PM kernels and the closure kernels: the
// particle's lattice point, its cell coordinates on a mesh, the means of a kick.
#ifndef MGP_DEVICE_CUH
#define MGP_DEVICE_CUH

#include "mgp_internal.h"

// Lattice coordinates of particle p (src/main.c:257-262 ordering).
__device__ __forceinline__ void lattice_ijk(long long p, int Ns, int &i, int &j, int &k) {
  long long ns2 = (long long)Ns * Ns;
  i = (int)(p / ns2);
  long long r = p - (long long)i * ns2;
  j = (int)(r / Ns);
  k = (int)(r - (long long)j * Ns);
}

// The same for p < 2^32 in unsigned 32-bit arithmetic (a 64-bit division is
// a long instruction sequence on the GPU; the results are identical).
__device__ __forceinline__ void lattice_ijk(unsigned p, int Ns, int &i, int &j, int &k) {
  const unsigned ns = (unsigned)Ns, ns2 = ns * ns;
  const unsigned ii = p / ns2, r = p - ii * ns2, jj = r / ns;
  i = (int)ii;
  j = (int)jj;
  k = (int)(r - jj * ns);
}

// Cell index and CIC fraction along one axis for the particle at lattice
// index `li` with displacement `s` (Mpc/h) and global offset `off_cells`.
// Position in cells = li*N/Ns + s*N/Box + off; the lattice part is split into
// integer and fractional parts exactly so the small displacement keeps full
// FP32 precision.  li*N < Ns*N stays far below 2^32 for any mesh and lattice
// that fit in device memory, so the split runs in unsigned 32-bit arithmetic.
__device__ __forceinline__ void cell_frac(int li, float s, float off_cells, int N, int Ns, float scale,
                                          int &idx, float &frac) {
  const unsigned qn = (unsigned)li * (unsigned)N;
  const unsigned qi = qn / (unsigned)Ns;
  float qf = (float)(qn - qi * (unsigned)Ns) / (float)Ns;
  float w = fmaf(s, scale, off_cells) + qf;
  float fl = floorf(w);
  float fr = w - fl;
  if (fr >= 1.0f) { fr -= 1.0f; fl += 1.0f; }
  int ic = (int)qi + (int)fl;
  if (ic < 0 || ic >= N) {  // a particle more than a cell outside its lattice cell's period
    ic %= N;
    if (ic < 0) ic += N;
  }
  idx = ic;
  frac = fr;
}

// Power-of-two lattices (Ns = 2^ls, the usual set-ups): the same lattice
// coordinates and cell fractions by shifts and masks.  The results are
// identical to lattice_ijk / cell_frac: the remainder of qn / Ns is below
// 2^24, so rem * (1/Ns) is exact in FP32 as rem / Ns is.
__device__ __forceinline__ void lattice_ijk_p2(unsigned p, int ls, int &i, int &j, int &k) {
  const unsigned m = (1u << ls) - 1u;
  i = (int)(p >> (2 * ls));
  j = (int)((p >> ls) & m);
  k = (int)(p & m);
}

__device__ __forceinline__ void cell_frac_p2(int li, float s, float off_cells, int N, int ls, float inv_ns, float scale,
                                             int &idx, float &frac) {
  const unsigned qn = (unsigned)li * (unsigned)N;
  const unsigned qi = qn >> ls;
  float qf = (float)(qn & ((1u << ls) - 1u)) * inv_ns;
  float w = fmaf(s, scale, off_cells) + qf;
  float fl = floorf(w);
  float fr = w - fl;
  if (fr >= 1.0f) { fr -= 1.0f; fl += 1.0f; }
  int ic = (int)qi + (int)fl;
  if (ic < 0 || ic >= N) {
    ic %= N;
    if (ic < 0) ic += N;
  }
  idx = ic;
  frac = fr;
}

// log2(Ns) when Ns is a power of two, else -1 (host and device).
__host__ __device__ __forceinline__ int lattice_log2(int Ns) {
  if (Ns <= 0 || (Ns & (Ns - 1))) return -1;
  int l = 0;
  while ((1 << l) < Ns) l++;
  return l;
}

// An FP32 sum that keeps what its additions rounded away (Knuth's TwoSum).
struct kd_sum {
  float s = 0.f, r = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float t = s + x, b = t - s;
    r += (s - (t - b)) + (x - b);
    s = t;
  }
};

// Means over all particles of the interpolated forces and the new velocities
// at the end of a kick, and the FP64 offsets they move (Kick and Drift subtract
// them, src/main.c:688-787).  Every block adds its threads' FP32 sums in FP64
// and leaves six numbers in `partials`; the block that arrives last at `done`
// adds the blocks' in index order and updates the state (done returns to 0 for
// the next launch).  acc: the forces' three sums, then the velocities'; red: 6 NT
// floats of shared memory that are free, or hold (kept) sums that the threads have put aside
// half-way, in the same order, so that a sum holds as few particles as with twice the
// threads; keep (or NULL): such sums elsewhere.
// FP64 runs at 1/64 of the FP32 rate here, so the adds are what counts: six
// warps sum NT / 32 values a lane and then one tree each, instead of six trees
// in every warp and a serial sum over warps (2^18 particles: 38 us the kick and
// 11 us a kernel for the blocks' sums; one kernel of 21 us now).
template <int NT>
__device__ __forceinline__ void kd_means(float (&acc)[6], float *red, double *partials, int block, int nblocks,
                                         unsigned *done, mgp_dstate *st, const mgp_kd_args &a,
                                         bool kept, const float *keep = nullptr) {
  __shared__ double tot[6];
  __shared__ int last;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  double x = 0.0;
  if (kept) {
    // both halves as one FP32 sum and what it rounded away, whose sum takes no FP64
    float y = 0.0f;
#pragma unroll
    for (int q = 0; q < 6; q++) {
      kd_sum h{red[q * NT + tid], 0.0f};
      h.add(acc[q]);
      acc[q] = h.s;
      red[q * NT + tid] = h.r;
    }
    __syncthreads();
    if (w < 6) {
#pragma unroll 4
      for (int i = 0; i < NT / 32; i++) y += red[w * NT + 32 * i + lane];
      x = (double)y;
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 6; q++) red[q * NT + tid] = acc[q];
  __syncthreads();
  if (w < 6) {
#pragma unroll 4
    for (int i = 0; i < NT / 32; i++) x += (double)red[w * NT + 32 * i + lane];
    if (keep)
#pragma unroll 4
      for (int i = 0; i < NT / 32; i++) x += (double)keep[w * NT + 32 * i + lane];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) {
      partials[(long long)block * 6 + w] = x;
      __threadfence();
    }
  }
  __syncthreads();
  if (tid == 0) last = atomicAdd(done, 1u) == (unsigned)nblocks - 1u;
  __syncthreads();
  if (!last) return;
  if (w < 6) {
    __threadfence();
    x = 0.0;
    for (int b = lane; b < nblocks; b += 32) x += __ldcg(partials + (long long)b * 6 + w);
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) tot[w] = x;
  }
  __syncthreads();
  if (tid < 3) {
    const double mD = tot[tid] * a.inv_np, mV = tot[3 + tid] * a.inv_np;
    st->mean_disp[tid] = mD;
    st->cv[tid] += a.dda_omega * mD;
    st->mean_v[tid] = mV;
    if (a.do_drift) st->cx[tid] -= mV * a.dyyy_d;
  }
  if (tid == 0) *done = 0u;
}

// Fourier-space filter of the fifth-force solvers per integer |k|^2 = rk
// (grid units): kind 1 SmoothDensityField (src/mg.h:268-309) with the
// smoothing filters of src/mg.h:318-338 (Gaussian, top-hat, sharp-k), kR =
// sqrt(rk) kR1, times norm; kind 2 the inverse Laplacian of DivideByLaplacian
// (src/mg.h:21-64), -norm / rk (0 at k = 0).  filter takes the
// MGP_FILTER_* values (1 Gaussian, 2 top-hat, 3 sharp-k).
__device__ __forceinline__ float mg_kfilter(int rk, int kind, int filter, float kR1, float norm) {
  if (kind == 2) return rk == 0 ? 0.0f : -norm / (float)rk;
  float kR = sqrtf((float)rk) * kR1, f = 1.0f;
  if (filter == 1) f = expf(-0.5f * kR * kR);
  else if (filter == 2) f = kR < 1e-5f ? 1.0f : 3.0f / (kR * kR * kR) * (sinf(kR) - kR * cosf(kR));
  else if (filter == 3) f = kR < 1.0f ? 1.0f : 0.0f;
  return f * norm;
}

// Screening factors (src/mg.h:174-176, 241-250 with the functions of
// src/user_defined_functions.h:725-773): min(1, |phi_crit / Phi|) where Phi < 0;
// 2 (sqrt(1 + f) - 1) / f with f = pref (1 + delta_R), 1 below f = 1e-5.
__device__ __forceinline__ float screen_pot(float ph, float phicrit) {
  float f = 1.0f;
  if (ph < 0.0f) {
    f = fabsf(phicrit / ph);
    if (f > 1.0f) f = 1.0f;
  }
  return f;
}
__device__ __forceinline__ float screen_den(float dsm, float pref) {
  float fac = pref * (1.0f + dsm);
  return fac < 1e-5f ? 1.0f : 2.0f * (sqrtf(1.0f + fac) - 1.0f) / fac;
}

#endif
