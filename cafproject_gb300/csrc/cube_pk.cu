// cube_pk.cu -- the matter power spectrum of the resident particles on the
// device: the CIC density of cicpower.f90:100-133 (mass 1, position
// (cell + frac)*ng/nc - 0.5), its density contrast (:171-176), and the binned
// auto/cross power of powerspectrum.f90:cross_power (:21-135) with linear bins
// ibin = nint(|k|), the CIC window 1/sinc^4 and the 4 pi k^3 weight.
//
// The mesh buffers of the fine PM are borrowed as scratch (the spectrum is an
// analysis call between steps): force plane 0 holds the particles' density
// and spectrum, plane 1 the optional second field, plane 2 the per-block
// partial sums.  Sums over modes run in FP32 inside a warp and in FP64
// across warps and blocks (the reference sums in real(4) throughout).
#include <algorithm>
#include <cmath>
#include <vector>

#include "cube_internal.cuh"

namespace {

constexpr int PK_Q = 7;        // accumulated quantities per bin (xi(1:7))
constexpr int PK_WARPS = 8;    // warps of a block, fewer where their bins need more shared memory
constexpr int PK_T = 32 * PK_WARPS;
constexpr size_t PK_SMEM = 200 * 1024;

// rho/mean - 1 over the ng^3 interior of a padded mesh (cicpower.f90:171-176);
// ng is even, so rows are pairs; blockDim.y rows at a time.  Bound by memory
// (one float at a time took 282 us for 512^3 cells, 228 in pairs; 158 at the copy rate)
__global__ void __launch_bounds__(256) k_pk_delta(float* rho, int ng, float inv_mean) {
  const int64_t rows = (int64_t)ng * ng;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.y + threadIdx.y; r < rows; r += (int64_t)gridDim.x * blockDim.y) {
    float2* row = reinterpret_cast<float2*>(rho + r * (ng + 2));
    for (int x = threadIdx.x; x < ng / 2; x += blockDim.x) {
      const float2 v = row[x];
      row[x] = make_float2(__fmaf_rn(v.x, inv_mean, -1.0f), __fmaf_rn(v.y, inv_mean, -1.0f));
    }
  }
}

// sin(pi k/ng)/(pi k/ng), 1 at k = 0
__device__ __forceinline__ float pk_sinc(int k, int ng) {
  return k == 0 ? 1.0f : sinf(CUBE_PI_F * k / ng) / (CUBE_PI_F * k / ng);
}

// Binned sums over the half spectrum.  A warp takes the rows (ky, kz) of one
// pair |ky|, |kz| together, 32 kx at a time: the two to four modes of a lane
// have the same |k|, bin and window, which are worked out once, and the lanes'
// bins grow with kx, so lanes of one bin are adjacent and a segmented sum
// leaves one addition per bin and warp.  Every warp adds into bins of its own
// (no atomics, the same sums in every run), and the block adds its warps' in
// FP64.  The spectrum is read once, consecutively (80 us for 512^3 cells at the
// copy rate): 2152 us with a thread per row (a stride of half a row between
// lanes) and shared FP32 atomics at every change of bin, 220 this way.
// Auto power (kCross false) has its second and cross power equal to the first.
template <bool kCross>
__global__ void __launch_bounds__(PK_T) k_pk_bin(const float2* __restrict__ c1, const float2* __restrict__ c2, int ng,
                                                 int nbin, double* __restrict__ part) {
  constexpr int NQ = kCross ? 7 : 5;  // modes, k, power 1 (, power 2, cross), 1/s^2, 1/s^4
  extern __shared__ float sb[];       // NQ * nbin per warp, then sinc(k) for k up to Nyquist
  const int nyq = ng / 2, nh = nyq + 1, lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* sinc = sb + nw * NQ * nbin;
  for (int i = threadIdx.x; i < nw * NQ * nbin; i += blockDim.x) sb[i] = 0.f;
  for (int i = threadIdx.x; i < nh; i += blockDim.x) sinc[i] = pk_sinc(i, ng);
  __syncthreads();
  float* mine = sb + w * NQ * nbin;
  const float inv_n3 = 1.0f / ((float)ng * (float)ng * (float)ng);  // cx=cxyz/ng^3
  const float four_pi = 4.0f * CUBE_PI_F;
  const int groups = nh * nh;
  for (int gi = blockIdx.x * nw + w; gi < groups; gi += gridDim.x * nw) {
    const int ky = gi % nh, kz = gi / nh;
    const float sy = sinc[ky], sz = sinc[kz];
    const int jn = ky == 0 || ky == nyq ? 1 : 2, kn = kz == 0 || kz == nyq ? 1 : 2;
    // rows (j, k): the mode itself, then its images; index 0 lies below Nyquist
    const int64_t row00 = ((int64_t)ky + (int64_t)ng * kz) * nh;
    const int64_t dj = (int64_t)(ng - 2 * ky) * nh, dk = (int64_t)ng * (ng - 2 * kz) * nh;
    for (int i0 = 0; i0 < nh; i0 += 32) {
      const int i = i0 + lane;
      float q[NQ];
#pragma unroll
      for (int t = 0; t < NQ; t++) q[t] = 0.f;
      int bin = -1 - lane;  // lanes past the row: bins of their own
      if (i < nh) {
        // powerspectrum.f90:60-62: the zero mode, and the conjugate duplicates
        // on the i = 0 and i = nyquist planes, are left out
        const bool edge = i == 0 || i == nyq;
        const int64_t at = row00 + i;
        float p1 = 0.f, p2 = 0.f, px = 0.f;
        int n = 0;
        auto add = [&](int64_t o) {
          const float2 a = __ldcs(c1 + o);
          p1 += a.x * a.x + a.y * a.y;
          if (kCross) {
            const float2 b = __ldcs(c2 + o);
            p2 += b.x * b.x + b.y * b.y;
            px += a.x * b.x + a.y * b.y;
          }
          n++;
        };
        if (!(i == 0 && ky == 0 && kz == 0)) add(at);
        if (jn == 2 && !edge) add(at + dj);                   // j > nyquist
        if (kn == 2 && !(edge && jn == 1)) add(at + dk);      // k > nyquist
        if (jn == 2 && kn == 2 && !edge) add(at + dj + dk);
        const int kx = i;
        const float kr = sqrtf((float)(kx * kx + ky * ky + kz * kz));
        const float s = sinc[kx] * sy * sz, s2 = s * s, s4 = s2 * s2;
        const float wt = four_pi * kr * kr * kr / s4 * inv_n3 * inv_n3, m = (float)n;
        bin = (int)roundf(kr) - 1;  // ibin = nint(kr), 1-based
        q[0] = m;                   // number of modes
        q[1] = m * kr;              // k
        q[2] = p1 * wt;             // auto power 1
        if (kCross) {
          q[3] = p2 * wt;           // auto power 2
          q[4] = px * wt;           // cross power
        }
        q[NQ - 2] = m / s2;         // kernel 1
        q[NQ - 1] = m / s4;         // kernel 2
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const bool same = __shfl_down_sync(0xffffffffu, bin, o) == bin && lane + o < 32;
#pragma unroll
        for (int t = 0; t < NQ; t++) {
          const float x = __shfl_down_sync(0xffffffffu, q[t], o);
          if (same) q[t] += x;
        }
      }
      const int left = __shfl_up_sync(0xffffffffu, bin, 1);
      if ((lane == 0 || left != bin) && bin >= 0 && bin < nbin) {
#pragma unroll
        for (int t = 0; t < NQ; t++) mine[t * nbin + bin] += q[t];
      }
      __syncwarp();
    }
  }
  __syncthreads();
  double* out = part + (int64_t)blockIdx.x * PK_Q * nbin;
  for (int i = threadIdx.x; i < PK_Q * nbin; i += blockDim.x) {
    const int t = i / nbin, b = i - t * nbin;
    // auto power: powers 2 and cross are power 1
    const int src = kCross || t <= 2 ? t : (t <= 4 ? 2 : t - 2);
    double v = 0.0;
    for (int k = 0; k < nw; k++) v += (double)sb[(k * NQ + src) * nbin + b];
    out[i] = v;
  }
}

// sum of the per-block partial bins: a warp's lanes take consecutive entries,
// the block's warps every eighth partial, then the warps' sums are added
__global__ void __launch_bounds__(PK_T) k_pk_reduce(const double* __restrict__ part, int nblocks, int n,
                                                    double* __restrict__ out) {
  __shared__ double s[PK_WARPS][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  double v = 0.0;
  if (i < n)
#pragma unroll 4
    for (int b = w; b < nblocks; b += PK_WARPS) v += part[(int64_t)b * n + i];
  s[w][lane] = v;
  __syncthreads();
  if (w != 0 || i >= n) return;
  for (int k = 1; k < PK_WARPS; k++) v += s[k][lane];
  out[i] = v;
}

}  // namespace

// nbin=nint(nyquest*sqrt(3.)) in real(4) (powerspectrum.f90:11)
extern "C" int cube_pk_nbin(int ng) { return (int)std::lround((double)((float)(ng / 2) * std::sqrt(3.0f))); }

extern "C" int cube_power_spectrum(cube_ctx* c, int ng, float box, const float* delta2, double* xi, int nbin) {
  if (!c || !xi) return CUBE_ERR_ARG;
  if (!c->have_state) return cube_fail(c, CUBE_ERR_STATE, "no state uploaded");
  if (ng != c->p.nc && ng != 2 * c->p.nc && ng != 4 * c->p.nc)
    return cube_fail(c, CUBE_ERR_ARG, "power-spectrum mesh must be nc, 2nc or 4nc per dimension");
  if (ng % 2) return cube_fail(c, CUBE_ERR_ARG, "power-spectrum mesh must be even");
  const int need = cube_pk_nbin(ng);
  if (nbin < need) return cube_fail(c, CUBE_ERR_ARG, "xi needs nint(ng/2*sqrt(3)) bins");
  CUBE_CUDA(c, cudaSetDevice(c->device));
  if (int r = cube_upload_join(c)) return r;
  cudaStream_t s = c->stream;
  if (int rf = cube_force_foreign(c, 0)) return rf;
  float* m1 = c->force_f[0];
  float* m2 = c->force_f[1];
  double* part = reinterpret_cast<double*>(c->force_f[2]);
  // 1. CIC density, mass 1 (the deposit writes every cell), and its exact total
  CUBE_CUDA(c, cudaMemsetAsync(&c->dstats->rhof_fix, 0, 8, s));
  int r = cube_pk_deposit(c, ng, m1, &c->dstats->rhof_fix);
  if (r) return r;
  r = cube_stats_fetch(c);
  if (r) return r;
  const double total = std::ldexp((double)c->hstats->rhof_fix, -dep_shift(1.0f));
  if (!(total > 0.0)) return cube_fail(c, CUBE_ERR_STATE, "no mass on the mesh");
  const double mean = total / ((double)ng * ng * ng);
  int bx = 32;
  while (bx < 256 && bx < ng / 2) bx *= 2;
  k_pk_delta<<<cube_grid((int64_t)ng * ng, 256 / bx, 8), dim3(bx, 256 / bx), 0, s>>>(m1, ng, (float)(1.0 / mean));
  CUBE_CUDA(c, cudaGetLastError());
  // 2. transforms: the fine or coarse plan when the mesh matches, else one made here
  cufftHandle plan = 0;
  bool own = false;
  if (ng == c->nf) {
    plan = c->plan_f_r2c;
  } else if (ng == c->p.nc) {
    plan = c->plan_c_r2c;
  } else {
    CUBE_FFT(c, cufftPlan3d(&plan, ng, ng, ng, CUFFT_R2C));
    CUBE_FFT(c, cufftSetStream(plan, s));
    own = true;
  }
  cufftResult fr = cufftExecR2C(plan, m1, (cufftComplex*)m1);
  if (fr == CUFFT_SUCCESS && delta2) {
    cudaError_t e = cudaMemcpy2DAsync(m2, sizeof(float) * (ng + 2), delta2, sizeof(float) * ng, sizeof(float) * ng,
                                      (size_t)ng * ng, cudaMemcpyHostToDevice, s);
    fr = e == cudaSuccess ? cufftExecR2C(plan, m2, (cufftComplex*)m2) : CUFFT_EXEC_FAILED;
  }
  if (own) cufftDestroy(plan);
  if (fr != CUFFT_SUCCESS) return cube_fail(c, CUBE_ERR_CUDA, "power-spectrum FFT failed");
  // 3. binned sums
  const size_t per_warp = sizeof(float) * (delta2 ? 7 : 5) * need;
  const int warps = (int)std::max<size_t>(1, std::min<size_t>(PK_WARPS, PK_SMEM / per_warp));
  const size_t smem = per_warp * warps + sizeof(float) * (ng / 2 + 1);
  auto bin = delta2 ? k_pk_bin<true> : k_pk_bin<false>;
  CUBE_CUDA(c, cudaFuncSetAttribute(bin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int resident = 1;
  CUBE_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, bin, 32 * warps, smem));
  const int nb = cube_grid((int64_t)(ng / 2 + 1) * (ng / 2 + 1), warps, std::max(1, resident));
  bin<<<nb, 32 * warps, smem, s>>>((const float2*)m1, (const float2*)m2, ng, need, part);
  CUBE_CUDA(c, cudaGetLastError());
  double* sums = part + (size_t)nb * PK_Q * need;
  k_pk_reduce<<<(PK_Q * need + 31) / 32, PK_T, 0, s>>>(part, nb, PK_Q * need, sums);
  CUBE_CUDA(c, cudaGetLastError());
  std::vector<double> h((size_t)PK_Q * need);
  CUBE_CUDA(c, cudaMemcpyAsync(h.data(), sums, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s));
  CUBE_CUDA(c, cudaStreamSynchronize(s));
  // 4. normalisation (powerspectrum.f90:121-133); empty bins divide by zero
  //    as in the reference
  const double two_pi = 2.0 * (double)CUBE_PI_F;
  for (int b = 0; b < nbin; b++) {
    double* o = xi + 10 * (size_t)b;
    if (b >= need) {
      for (int q = 0; q < 10; q++) o[q] = 0.0;
      continue;
    }
    double v[PK_Q];
    for (int q = 0; q < PK_Q; q++) v[q] = h[(size_t)q * need + b];
    o[0] = v[0];
    o[1] = v[1] / v[0] * two_pi / (double)box;
    for (int q = 2; q < PK_Q; q++) o[q] = v[q] / v[0];
    o[7] = o[4] / std::sqrt(o[2] * o[3]);
    o[8] = std::sqrt(o[3] / o[2]);
    o[9] = std::pow(o[7], 4) / (o[8] * o[8]) * o[3];
  }
  return CUBE_OK;
}
