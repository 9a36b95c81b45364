// cube_pm.cu -- particle_mesh (pm.f90:2-415) on one GB300.
//
// Fine level: one periodic nf^3 mesh (nf = nc*ncell) instead of the
// reference's nnt^3 tile boxes of nfe^3: the fine kernel is the 31^3 table
// (offsets -15..15 < nfb=24), so the force on each tile's physical region is
// the same linear convolution either way; the global mesh does (nf/nft)^3
// fewer cells of FFT work and needs no buffer deposit.
//   deposit (CIC, tile-local real(4) tempx as pm.f90:63) -> cuFFT R2C ->
//   multiply by i*K_d (pm.f90:119-120) -> 3 x cuFFT C2R -> f2 max -> kick
//   (pm.f90:129-189, decode sigma_vi, encode sigma_vi_new).
// Coarse level: nc^3 periodic mesh, deposit with the -0.5 shift
// (pm.f90:221), R2C, i*K_c, C2R, kick (pm.f90:322-387) with vmax.
// The 1/n^3 normalisation is folded into the stored kernels.
#include <algorithm>
#include <cmath>
#include <vector>

#include "cube_internal.cuh"

namespace {

// ----------------------------------------------------------- Green's functions
// odd-mirrored fine table in the periodic nf^3 box (kernel_f.f90:25-31)
__global__ void k_fill_fine_table(const float* __restrict__ tab, int nfc, int pp_zero, int dim, int nf,
                                  float* __restrict__ box) {
  int w = 2 * nfc - 1;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= w * w * w) return;
  int ox = t % w - (nfc - 1), oy = (t / w) % w - (nfc - 1), oz = t / (w * w) - (nfc - 1);
  int ax = abs(ox), ay = abs(oy), az = abs(oz);
  float v = tab[ax + nfc * (ay + nfc * (az + nfc * dim))];  // fk_table(i,j,k,d)
  if (ax <= pp_zero && ay <= pp_zero && az <= pp_zero) v = 0.f;
  int neg = dim == 0 ? ox < 0 : (dim == 1 ? oy < 0 : oz < 0);
  if (neg) v = -v;
  box[mesh_idx(nf, wrapi(ox, nf), wrapi(oy, nf), wrapi(oz, nf))] = v;
}

// kern[idx] = Im(fft)[idx] * scale
__global__ void k_take_imag(const float2* __restrict__ spec, int64_t n, float scale, float* __restrict__ kern) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    kern[i] = spec[i].y * scale;
}

// LRCKCORR (kernel_c.f90:102-116): for |k|<=8 and k_d != 0 replace K by
// K*0.25*pi*ksin_d/sum(ksin^2)/Im(FFT(raw)).  At nc = 16 the sphere reaches the
// Nyquist plane, where the odd raw kernel's transform is exactly zero and the
// reference would divide 0 by 0; there K keeps its value (also zero).
__global__ void k_lrck(float* __restrict__ kern, const float2* __restrict__ raw, int nc, int dim) {
  int nh = nc / 2 + 1;
  int64_t n = (int64_t)nh * nc * nc;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int ix = (int)(i % nh), iy = (int)((i / nh) % nc), iz = (int)(i / ((int64_t)nh * nc));
    float k[3];
    k[0] = (float)(((ix + nc / 2) % nc) - nc / 2);
    k[1] = (float)(((iy + nc / 2) % nc) - nc / 2);
    k[2] = (float)(((iz + nc / 2) % nc) - nc / 2);
    float kr = sqrtf(k[0] * k[0] + k[1] * k[1] + k[2] * k[2]);
    if (kr > 8.0f || k[dim] == 0.f) continue;
    float s[3];
    for (int d = 0; d < 3; d++) s[d] = 2.f * sinf(CUBE_PI_F * k[d] / (float)nc);
    float ss = (s[0] * s[0] + s[1] * s[1]) + s[2] * s[2];
    if (raw[i].y == 0.f) continue;
    float v = kern[i];
    v = v * 0.25f;
    v = v * CUBE_PI_F;
    v = v * s[dim];
    v = v / ss;
    v = v / raw[i].y;
    kern[i] = v;
  }
}

__global__ void k_scale(float* __restrict__ a, int64_t n, float s) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] *= s;
}

// ---------------------------------------------------------------- deposit
// Deterministic CIC deposit.  One CTA owns a brick of BX x BY x BZ coarse
// cells and every mesh cell inside it: it reads the particles of the brick's
// coarse cells and of the LO/HI neighbouring layers whose CIC stencils reach
// into it (fine mesh: the +1 spill of the layer below; coarse mesh with its
// -0.5 shift: one layer on each side), accumulates the weights in shared
// memory as 2^-32 fixed point with 64-bit integer atomics (integer addition is
// associative, so the sum does not depend on thread order), and writes each
// owned cell once.  No memset, no global atomics, bitwise reproducible.
// The weights are the reference's real(4) products (pm.f90:63-77, 221-233),
// computed from tempx in the tile-local frame.
struct DepArgs {
  Geo g;
  const void* xp;
  const int32_t* rhoc;
  const int64_t* cstart;
  float mass;
  float* rho;                 // padded periodic mesh, row stride n+2
  unsigned long long* total;  // sum of all owned cells in fixed point (exact)
  int ng;                     // power-spectrum mesh (kPk only)
  float rnc;                  // kPk: RN(1/nc)
  float qscale, qinv;         // fixed-point scale 2^s and 2^-s (dep_shift)
  int accumulate;             // add to the mesh (a second species) instead of writing it
};



// kPk: the power-spectrum deposit of cicpower.f90:100-133 (position
// (cell + frac)*ng/nc - 0.5 in real(4), global frame) instead of the PM ones
template <int MPC, int BX, int BY, int BZ, int LO, int HI, bool kPk = false>
__global__ void __launch_bounds__(256) k_deposit_det(DepArgs a) {
  constexpr int SX = BX + LO + HI, SY = BY + LO + HI, SZ = BZ + LO + HI;
  constexpr int NSRC = SX * SY * SZ;
  constexpr int MX = MPC * BX, MY = MPC * BY, MZ = MPC * BZ;
  extern __shared__ __align__(16) unsigned acc[];  // low words [0, MX*MY*MZ), carry words after them
  unsigned* carry = acc + MX * MY * MZ;
  __shared__ int pref[NSRC];
  __shared__ long long sstart[NSRC];
  // kAxis: the fine deposit tests the stencil per axis (a 2-bit mask each,
  // the whole stencil skipped when one is empty) and shares the x*y weight
  // products between z's two corners; the coarse deposit, whose stencils more
  // often straddle the brick's edge, measured faster with the plain per-corner
  // test (0.21 ms of 2.70 at 512^3), the fine one slower (0.37 ms of 5.54)
  constexpr bool kAxis = MPC > 1;
  // per source cell, 16 bits a dimension: the 1-based tile-local coordinate
  // (kPk: the global coarse coordinate) that the particle's frame needs
  __shared__ unsigned long long sframe[NSRC];
  __shared__ unsigned long long btot;
  const Geo& g = a.g;
  const int nc = g.nc, n = kPk ? a.ng : (MPC == 1 ? g.nc : g.nf);
  int nbx = (nc + BX - 1) / BX, nby = (nc + BY - 1) / BY;
  int b = blockIdx.x;
  int C0[3] = {(b % nbx) * BX, ((b / nbx) % nby) * BY, (b / (nbx * nby)) * BZ};
  int B[3] = {min(BX, nc - C0[0]), min(BY, nc - C0[1]), min(BZ, nc - C0[2])};
  // 2*MX*MY*MZ is a multiple of 4: 16-byte stores
  for (int i = 4 * threadIdx.x; i < 2 * MX * MY * MZ; i += 4 * blockDim.x)
    *reinterpret_cast<uint4*>(acc + i) = make_uint4(0u, 0u, 0u, 0u);
  if (threadIdx.x == 0) btot = 0ull;
  // source cells, their particle counts and frames
  for (int t = threadIdx.x; t < NSRC; t += blockDim.x) {
    const int sl[3] = {t % SX - LO, (t / SX) % SY - LO, t / (SX * SY) - LO};
    int cnt = 0;
    long long st = 0;
    unsigned long long fr = 0;
    if (sl[0] < B[0] + HI && sl[1] < B[1] + HI && sl[2] < B[2] + HI) {
      int gc[3];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        gc[d] = wrap1(C0[d] + sl[d], nc);
        int Tq, L;
        tile_local(g, gc[d], Tq, L);
        fr |= (unsigned long long)(unsigned)(kPk ? gc[d] : L) << (16 * d);
      }
      int64_t c = cell_id(g, gc[0], gc[1], gc[2]);
      cnt = a.rhoc[c];
      st = a.cstart[c];
    }
    pref[t] = cnt;
    sstart[t] = st;
    sframe[t] = fr;
  }
  __syncthreads();
  const int total = block_exclusive_scan(pref, NSRC);
  const int lim[3] = {MPC * B[0], MPC * B[1], MPC * B[2]};
  for_box_particles<SX>(pref, sstart, SX, SY * SZ, total, [&](int64_t p, int sxi, int row) {
    const int sl[3] = {sxi - LO, row % SY - LO, row / SY - LO};
    const unsigned long long fr = sframe[sxi + SX * row];
    int rel[3];
    unsigned ok[3];  // bit o: mesh index rel + o lies in the brick
    float d1[3], d2[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const int v = (int)((fr >> (16 * d)) & 0xffffu);  // L, or kPk the global coordinate
      int code = load_code(a.xp, 3 * p + d, g.izipx);
      float tx;
      if (kPk) {
        float frac = __fmul_rn(pos_off_f(code, g.izipx), g.izipx == 1 ? 1.0f / 256.0f : 1.0f / 65536.0f);
        // the particle's own global frame, as the reference rounds it
        float pos = __fadd_rn((float)v, frac);
        // the quotient by nc, correctly rounded: Markstein's correction step as
        // in div_const (nc is a whole number, its reciprocal rounded to nearest)
        const float num = __fmul_rn(pos, (float)a.ng), q = __fmul_rn(num, a.rnc);
        tx = __fsub_rn(__fmaf_rn(__fmaf_rn(-q, (float)nc, num), a.rnc, q), 0.5f);
      } else {
        tx = MPC == 1 ? coarse_tempx(v, code, g.izipx) : fine_tempx(MPC, v, code, g.izipx);
      }
      float fl = floorf(tx);
      d1[d] = __fsub_rn(__fadd_rn(fl, 1.0f), tx);
      d2[d] = __fsub_rn(1.0f, d1[d]);
      // mesh index relative to the brick
      // (kPk: unwrap the ring cell's periodic image, then relative to the brick)
      rel[d] = kPk ? (int)fl + MPC * (sl[d] - v) : MPC * sl[d] + (int)fl - MPC * (v - 1);
      ok[d] = (unsigned)(rel[d] >= 0 && rel[d] < lim[d]) | ((unsigned)(rel[d] >= -1 && rel[d] + 1 < lim[d]) << 1);
    }
    if (kAxis && !(ok[0] && ok[1] && ok[2])) return;  // the whole stencil lies outside the brick
    // the reference's product order ((d_x * d_y) * d_z) * mass
    float wxy[4];
#pragma unroll
    for (int k = 0; k < 4; k++) wxy[k] = kAxis ? __fmul_rn(k & 1 ? d2[0] : d1[0], k & 2 ? d2[1] : d1[1]) : 0.f;
    const int e0 = rel[0] + MX * (rel[1] + MY * rel[2]);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int ox = k & 1, oy = (k >> 1) & 1, oz = k >> 2;
      if (kAxis) {
        if (!((ok[0] >> ox) & (ok[1] >> oy) & (ok[2] >> oz) & 1u)) continue;
      } else {
        const int x = rel[0] + ox, y = rel[1] + oy, z = rel[2] + oz;
        if (x < 0 || y < 0 || z < 0 || x >= lim[0] || y >= lim[1] || z >= lim[2]) continue;
      }
      const float wxyk = kAxis ? wxy[k & 3] : __fmul_rn(ox ? d2[0] : d1[0], oy ? d2[1] : d1[1]);
      float w = __fmul_rn(__fmul_rn(wxyk, oz ? d2[2] : d1[2]), a.mass);
      // w * 2^s (exact scaling, truncated) < 2^31; carry out of the low word
      const unsigned q = __float2uint_rz(__fmul_rn(w, a.qscale));
      const int e = kAxis ? e0 + ox + MX * (oy + MY * oz) : (rel[0] + ox) + MX * ((rel[1] + oy) + MY * (rel[2] + oz));
      const unsigned old = atomicAdd(&acc[e], q);
      if (old + q < old) atomicAdd(&carry[e], 1u);
    }
  });
  __syncthreads();
  unsigned long long mysum = 0;
  // (hi*2^32 + lo) * 2^-s as float
  const float qhi = __fmul_rn(a.qinv, 4294967296.0f);
  if (kAxis) {
    // KX neighbouring x cells a thread, written as KX/2 pairs: KX divides
    // MPC, so MX and the brick's extent MPC*B[0] are multiples of KX, and n
    // is even, so x starts an 8-byte aligned stretch of the padded mesh
    // (row stride n+2)
    constexpr int KX = MPC >= 4 ? 4 : 2;
    for (int i = KX * threadIdx.x; i < MX * MY * MZ; i += KX * blockDim.x) {
      const int x = i % MX, y = (i / MX) % MY, z = i / (MX * MY);
      if (x >= MPC * B[0] || y >= MPC * B[1] || z >= MPC * B[2]) continue;
      unsigned lo[KX], hi[KX];
      if constexpr (KX == 4) {
        const uint4 l = *reinterpret_cast<const uint4*>(acc + i), h = *reinterpret_cast<const uint4*>(carry + i);
        lo[0] = l.x, lo[1] = l.y, lo[2] = l.z, lo[3] = l.w;
        hi[0] = h.x, hi[1] = h.y, hi[2] = h.z, hi[3] = h.w;
      } else {
        const uint2 l = *reinterpret_cast<const uint2*>(acc + i), h = *reinterpret_cast<const uint2*>(carry + i);
        lo[0] = l.x, lo[1] = l.y;
        hi[0] = h.x, hi[1] = h.y;
      }
      float2* cell = reinterpret_cast<float2*>(a.rho + mesh_idx(n, MPC * C0[0] + x, MPC * C0[1] + y, MPC * C0[2] + z));
#pragma unroll
      for (int q = 0; q < KX / 2; q++) {
        mysum += (((unsigned long long)hi[2 * q] << 32) | lo[2 * q]) +
                 (((unsigned long long)hi[2 * q + 1] << 32) | lo[2 * q + 1]);
        float2 r = make_float2(__fmaf_rn((float)lo[2 * q], a.qinv, __fmul_rn((float)hi[2 * q], qhi)),
                               __fmaf_rn((float)lo[2 * q + 1], a.qinv, __fmul_rn((float)hi[2 * q + 1], qhi)));
        if (a.accumulate) {
          const float2 o = cell[q];
          r = make_float2(__fadd_rn(o.x, r.x), __fadd_rn(o.y, r.y));
        }
        cell[q] = r;
      }
    }
  } else {
    for (int i = threadIdx.x; i < MX * MY * MZ; i += blockDim.x) {
      const int x = i % MX, y = (i / MX) % MY, z = i / (MX * MY);
      if (x >= MPC * B[0] || y >= MPC * B[1] || z >= MPC * B[2]) continue;
      const unsigned lo = acc[i], hi = carry[i];
      mysum += ((unsigned long long)hi << 32) | lo;
      float r = __fmaf_rn((float)lo, a.qinv, __fmul_rn((float)hi, qhi));
      float* cell = a.rho + mesh_idx(n, MPC * C0[0] + x, MPC * C0[1] + y, MPC * C0[2] + z);
      *cell = a.accumulate ? __fadd_rn(*cell, r) : r;
    }
  }
  for (int o = 16; o > 0; o >>= 1) mysum += __shfl_xor_sync(0xffffffffu, mysum, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&btot, mysum);
  __syncthreads();
  if (threadIdx.x == 0 && a.total) atomicAdd(a.total, btot);
}

template <int MPC, int BX, int BY, int BZ, int LO, int HI, bool kPk = false>
int launch_deposit(cube_ctx* c, const DepArgs& a) {
  int nc = c->p.nc;
  int nb = ((nc + BX - 1) / BX) * ((nc + BY - 1) / BY) * ((nc + BZ - 1) / BZ);
  size_t smem = 2 * sizeof(unsigned) * (MPC * BX) * (MPC * BY) * (MPC * BZ);
  auto kern = k_deposit_det<MPC, BX, BY, BZ, LO, HI, kPk>;
  CUBE_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<nb, 256, smem, c->stream>>>(a);
  CUBE_CUDA(c, cudaGetLastError());
  return CUBE_OK;
}

// The deposits' brick shapes (cube_set_option CUBE_OPT_DEPOSIT_FINE / _COARSE):
// larger bricks re-read fewer neighbour particles, smaller ones hold less
// shared memory per CTA (more CTAs per SM) and give small meshes more CTAs.
// Every shape writes the same exact fixed-point sums.  Unless one is set, the
// number of 8x4x4 (8x8x8) bricks decides: below one a multiprocessor the smallest
// bricks fill the chip (nc 24: 16 against 24 us fine, 22 against 53 coarse), above
// it they re-read too many neighbours (nc 64: 105 against 83, 92 against 77).  The
// fine deposit then takes the half-high brick (nc 48: 45 against 48 us, nc 256:
// 4.53 against 4.58 ms); the coarse one takes it up to three bricks a
// multiprocessor (nc 48: 52 against 72, nc 64: 76.5 against 78.6, nc 96: 189
// against 173).
int64_t default_bricks(const cube_ctx* c, int bx, int by, int bz) {
  const int64_t nc = c->p.nc;
  return ((nc + bx - 1) / bx) * ((nc + by - 1) / by) * ((nc + bz - 1) / bz);
}
int sm_count() { return cube_grid((int64_t)1 << 40, 1, 1); }
int launch_fine_deposit(cube_ctx* c, const DepArgs& a) {
  int shape = c->opt_dep_fine;
  if (shape < 0) shape = default_bricks(c, 8, 4, 4) < sm_count() ? 3 : 2;
  switch (shape) {
    case 1: return launch_deposit<4, 4, 4, 4, 1, 0>(c, a);  // 16^3 fine cells, 32 KB
    case 2: return launch_deposit<4, 8, 4, 2, 1, 0>(c, a);  // 32x16x8, 32 KB
    case 3: return launch_deposit<4, 4, 4, 2, 1, 0>(c, a);  // 16x16x8, 16 KB
    default: return launch_deposit<4, 8, 4, 4, 1, 0>(c, a);  // 32x16x16, 64 KB
  }
}
int launch_coarse_deposit(cube_ctx* c, const DepArgs& a) {
  int shape = c->opt_dep_coarse;
  if (shape < 0) {
    const int64_t nb = default_bricks(c, 8, 8, 8);
    shape = nb < sm_count() ? 3 : (nb < 3 * sm_count() ? 2 : 0);
  }
  switch (shape) {
    case 1: return launch_deposit<1, 16, 8, 8, 1, 1>(c, a);
    case 2: return launch_deposit<1, 8, 8, 4, 1, 1>(c, a);
    case 3: return launch_deposit<1, 4, 4, 4, 1, 1>(c, a);
    default: return launch_deposit<1, 8, 8, 8, 1, 1>(c, a);
  }
}

// ------------------------------------------------------- spectral multiply
// out_d = i*K_d*rho_k for the three components in one pass (pm.f90:119-120)
// (and *f2 cleared for the forces' maximum)
__global__ void k_green3(const float2* __restrict__ rk, const float* __restrict__ kern, int64_t n,
                         float2* __restrict__ o0, float2* __restrict__ o1, float2* __restrict__ o2,
                         unsigned* __restrict__ f2) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *f2 = 0u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float2 r = rk[i];
    float k0 = kern[i], k1 = kern[n + i], k2 = kern[2 * n + i];
    o0[i] = make_float2(-r.y * k0, r.x * k0);
    o1[i] = make_float2(-r.y * k1, r.x * k1);
    o2[i] = make_float2(-r.y * k2, r.x * k2);
  }
}

// maxval(sum(force**2,1)) over the mesh (pm.f90:126, 315).  Bound by memory (12
// bytes a cell): the three padded meshes are walked as flat arrays of 16 bytes,
// F2_LOADS of each in flight a thread, and the two values of padding behind each
// row (n even) are left out of the maximum.  While it also rewrote each force as
// its kick factor (24 bytes a cell) it took 4.10 ms at 1024^3; 1.77 now, 1.90 at
// the copy rate.
__device__ __forceinline__ float f2sum(float a, float b, float c) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b)), __fmul_rn(c, c));
}
constexpr int F2_LOADS = 2;
__global__ void __launch_bounds__(256) k_f2max(const float4* __restrict__ f0, const float4* __restrict__ f1,
                                               const float4* __restrict__ f2, int64_t quads, FastDiv drow,
                                               uint32_t wrap, unsigned int* __restrict__ out,
                                               unsigned int* __restrict__ out2) {
  // value pairs: drow.d of them a row, the last one padding; wrap = 2^32 mod
  // drow.d brings the pair index of a mesh beyond 2^32 pairs (n > 2046) back
  auto in_row = [&](uint64_t k) {
    uint32_t r = (uint32_t)k;
    r -= fdiv(r, drow) * drow.d;
    if (k >> 32) {
      r += (uint32_t)(k >> 32) * wrap;
      r -= fdiv(r, drow) * drow.d;
    }
    return r;
  };
  __shared__ unsigned s_max;
  if (threadIdx.x == 0) s_max = 0u;
  __syncthreads();
  float m = 0.f;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < quads; i0 += F2_LOADS * step) {
    float4 u[F2_LOADS], v[F2_LOADS], w[F2_LOADS];
#pragma unroll
    for (int j = 0; j < F2_LOADS; j++) {
      const int64_t i = i0 + j * step;
      if (i < quads) {
        u[j] = f0[i];
        v[j] = f1[i];
        w[j] = f2[i];
      }
    }
#pragma unroll
    for (int j = 0; j < F2_LOADS; j++) {
      const int64_t i = i0 + j * step;
      if (i >= quads) break;
      const uint32_t r = in_row(2 * (uint64_t)i);  // the second pair follows it, or starts the next row
      const float a = fmaxf(f2sum(u[j].x, v[j].x, w[j].x), f2sum(u[j].y, v[j].y, w[j].y));
      const float b = fmaxf(f2sum(u[j].z, v[j].z, w[j].z), f2sum(u[j].w, v[j].w, w[j].w));
      if (r != drow.d - 1) m = fmaxf(m, a);
      if (r != drow.d - 2) m = fmaxf(m, b);
    }
  }
  warp_max_pos(&s_max, m);
  __syncthreads();
  if (threadIdx.x < 2) atomicMax(threadIdx.x ? out2 : out, s_max);
}

// the maxima pass over n^3 cells of three padded meshes
void launch_f2max(cube_ctx* c, float* const f[3], int n, unsigned int* out, unsigned int* out2) {
  const int64_t quads = (int64_t)(n + 2) * n * n / 4;
  k_f2max<<<cube_grid(quads, 256 * F2_LOADS, 8), 256, 0, c->stream>>>(
      (const float4*)f[0], (const float4*)f[1], (const float4*)f[2], quads, make_fastdiv((uint32_t)(n / 2 + 1)),
      (uint32_t)((1ull << 32) % (uint64_t)(n / 2 + 1)), out, out2);
}

// ------------------------------------------------------------------- kicks
struct KickArgs {
  Geo g;
  int64_t np;
  const void* xp;
  const void* vp_in;
  void* vp_out;            // may equal vp_in (fine kick updates in place)
  const int32_t* pcell;
  const float* vfield;
  const float* f[3];
  const unsigned* f2;      // bits of the maximum of force^2 over these meshes, or NaN
  CodecView cin, cout;     // decode with sigma_in, encode with sigma_out
  float a_mid, dt;
  unsigned int* vmax_bits; // coarse kick only: exact vmax per component
  float tau[3];            // coarse kick: lanes whose |v+vfield| may reach tau are evaluated exactly
  unsigned int* vmax_lo;   // coarse kick: the largest lower bound of |v+vfield| (certain to be <= vmax)
  int vmax_only;           // rerun for the exact vmax (write nothing): lanes whose bound reaches vmax_lo
  int exact_only;          // skip the certified fast path
  const StepDev* sd;       // graph mode: a_mid, dt, tau from the device
  unsigned int* vmax_est;        // fine kick: record max |v + vfield| (FP32) here when set
  const unsigned int* tau_est;   // coarse kick: tau = 0.7 of this estimate when set
  const float* fpp;              // fine kick: when set, first the PP kick by these pair forces
  float pp_kf;                   // its factor a_mid*dt/6/pi, float and double
  double pp_kd;
  const unsigned* pp_act;        // PP prefilter: set bits are the particles PP has kicked, the others take zero kicks
};
__device__ __forceinline__ float kick_amid(const KickArgs& a) { return a.sd ? __ldg(&a.sd->h.a_mid) : a.a_mid; }
__device__ __forceinline__ float kick_dt(const KickArgs& a) { return a.sd ? __ldg(&a.sd->h.dt) : a.dt; }
__device__ __forceinline__ float kick_tau(const KickArgs& a, int d) {
  if (a.sd) return __ldg(&a.sd->h.tau[d]);
  return a.tau_est ? __fmul_rn(0.7f, __uint_as_float(__ldg(a.tau_est + d))) : a.tau[d];
}

// The kick velocity of the reference is the FP64 chain
//   v = decode; v = v + t1; ...; v = v + t8       (pm.f90:145-153)
// with t_i the real(4) CIC terms force*a_mid*dt/6/pi*w*w*w (seven roundings
// each).  The fast path forms the eight weights w*K*w*w once a particle, K =
// kick_pre(1) (three roundings, and three more), S = sum force*weight by FMAs
// (eight) and V_f = fl32(hi(decode) + S); its distance from the reference value
// is bounded by
//   gamma_21 sum|force*weight| + 2^-24 (|decode| + |V_f|) + 9*2^-53 (|decode| + sum + |V_f|)
// (gamma_21 = 21u/(1-21u), 21u = 1.2517e-6, u = 2^-24; the decode table's float
// hi is within half an ulp), and 1e-24 for products in the denormal range (a
// term's lose 2^-150 each, of which the first is multiplied by dt < 1e20).
// Forces or factors so large that the reference's own products may overflow (by
// the mesh's maximum) are left to the exact chain, as is a factor below the
// normal floats' range (kick_factor).
// certify_code keeps the code only when every double inside that bound encodes
// to it; otherwise the lane runs the exact chain, so the stored code is always
// the reference's.
//
// The exact chain (and, in the coarse kick, the exact |v + vfield| of lanes
// that may set vmax) is needed by a few components in a hundred, but a warp
// would run it whenever one of its 32 lanes needs it, on the FP64 pipe.  So each
// warp queues those (particle, component, code) entries in shared memory and
// runs the chain 32 entries at a time, each lane recomputing its entry's CIC
// corners and terms (the same arithmetic, the same bits).  An entry packs
// the particle index (bits 18 and up), the 16-bit code and the component.
//
// Bound by the L1: the force gathers are 8 corners x 3 components of 4 bytes
// (a warp's 32 particles spread over four or so cells, so about ten sectors a
// gather) plus what the velocity codec gathers, and by issue slots.  Hence the
// table-free certificate and the 4-byte decode table (one table gather a
// component instead of five), one row address per pair of x corners, and every
// component unrolled (indexing the codes in a loop had put them in local
// memory): 6.74 -> 4.38 ms fine and 6.43 -> 3.70 ms coarse at 512^3 particles,
// 63 % of the L1's wavefront rate.  The forces as the transforms leave them,
// their factor in the particle's weights, cost the kicks 0.1 ms (4.29 and 3.75)
// and spare the maxima pass 2.3 ms of writing; more than 64 registers, or spills
// to hold the factor in one (it lies in shared memory), cost more than that.
constexpr int KICK_Q = 64;  // queue entries per warp: at most 31 pending + 32 from one component
__device__ __forceinline__ unsigned long long kick_qkey(int64_t p, int d, int code) {
  return ((unsigned long long)p << 18) | ((unsigned long long)(code & 0xffff) << 2) | (unsigned long long)d;
}

// A stencil's lower x, its upper x relative to it, and the row y + n*z of its
// four corners (lower and upper y, lower and upper z).
struct KickCorners {
  int x, dx;
  uint32_t row[2][2];  // [z][y]
  float d1[3], d2[3];
  int cell;
};

template <bool kFine>
__device__ __forceinline__ void kick_corners(const KickArgs& a, int64_t p, KickCorners& k) {
  const Geo& g = a.g;
  k.cell = a.pcell[p];
  int T[3], l[3], i1[3], i2[3];
  cell_tile(g, k.cell, T, l);
  const int n = kFine ? g.nf : g.nc;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int code = load_code(a.xp, 3 * p + d, g.izipx);
    float tx, fl;
    int base;
    if (kFine) {
      tx = fine_tempx(g.ncell, l[d] + 1, code, g.izipx);  // tile-local frame (pm.f90:138)
      fl = floorf(tx);
      base = T[d] * g.nt * g.ncell + (int)fl;
    } else {
      tx = coarse_tempx(T[d] * g.nt + l[d] + 1, code, g.izipx);  // global frame (pm.f90:335)
      fl = floorf(tx);
      base = (int)fl;
    }
    k.d1[d] = __fsub_rn(__fadd_rn(fl, 1.0f), tx);
    k.d2[d] = __fsub_rn(1.0f, k.d1[d]);
    i1[d] = wrap1(base, n);
    i2[d] = wrap1(base + 1, n);
  }
  k.x = i1[0];
  k.dx = i2[0] - i1[0];
  k.row[0][0] = (uint32_t)i1[1] + (uint32_t)n * (uint32_t)i1[2];
  k.row[0][1] = (uint32_t)i2[1] + (uint32_t)n * (uint32_t)i1[2];
  k.row[1][0] = (uint32_t)i1[1] + (uint32_t)n * (uint32_t)i2[2];
  k.row[1][1] = (uint32_t)i2[1] + (uint32_t)n * (uint32_t)i2[2];
}

// K, or NaN (which no certificate passes) where the fast path does not apply: it
// takes K = 0 or a normal float with room for a weight below it, and no product
// of a force near overflow.  f2 is the maximum of force^2 over the mesh, NaN when
// that is not known
__device__ __forceinline__ float kick_factor(float a_mid, float dt, float f2) {
  const float K = kick_pre(1.0f, a_mid, dt);
  const float big = fmaxf(fabsf(a_mid), fmaxf(fabsf(dt), fabsf(__fmul_rn(a_mid, dt))));
  const bool ok = (a_mid == 0.f || dt == 0.f || fabsf(K) >= 1.0e-30f) && big < 1.0e20f && f2 < 1.0e30f;
  return ok ? K : __int_as_float(0x7fffffff);
}

// the force of the component whose mesh is F at the eight corners, [z][y][x]
template <bool kFine>
__device__ __forceinline__ void kick_gather(const KickArgs& a, const KickCorners& k, const float* F,
                                            float v[2][2][2]) {
  const uint32_t stride = (uint32_t)((kFine ? a.g.nf : a.g.nc) + 2) * 4u;  // bytes of a padded row
  const char* base = reinterpret_cast<const char*>(F + k.x);
#pragma unroll
  for (int z = 0; z < 2; z++)
#pragma unroll
    for (int y = 0; y < 2; y++) {
      const float* r = reinterpret_cast<const float*>(base + (uint64_t)k.row[z][y] * stride);
      v[z][y][0] = __ldg(r);
      v[z][y][1] = __ldg(r + k.dx);
    }
}

// one queued component on the reference's FP64 chain: its code, and in the
// coarse kick vmax=max(vmax,abs(vreal+vfield)) (pm.f90:349) as real(4)
template <bool kFine>
__device__ __noinline__ void kick_exact_entry(const KickArgs& a, unsigned long long key, float vm[3]) {
  const int64_t p = (int64_t)(key >> 18);
  const int d = (int)(key & 3ull);
  const int code = (int)(int16_t)(uint16_t)((key >> 2) & 0xffffull);
  KickCorners k;
  kick_corners<kFine>(a, p, k);
  float f[2][2][2];
  kick_gather<kFine>(a, k, d == 0 ? a.f[0] : (d == 1 ? a.f[1] : a.f[2]), f);
  double v = codec_decode(a.cin, code);
  // the real(4) CIC terms in the reference's order: corners c111, c211, c121,
  // c112, c122, c212, c221, c222
  constexpr int kX = 0xe2, kY = 0xd4, kZ = 0xb8;  // bit i: the upper corner of term i
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int x = (kX >> i) & 1, y = (kY >> i) & 1, z = (kZ >> i) & 1;
    v = __dadd_rn(v, (double)kick_term(f[z][y][x], kick_amid(a), kick_dt(a), x ? k.d2[0] : k.d1[0],
                                       y ? k.d2[1] : k.d1[1], z ? k.d2[2] : k.d1[2]));
  }
  if (!kFine) {
    const double w = fabs(__dadd_rn(v, (double)a.vfield[3 * (int64_t)k.cell + d]));
    const float wf = __double2float_rn(w);
    vm[0] = d == 0 ? fmaxf(vm[0], wf) : vm[0];
    vm[1] = d == 1 ? fmaxf(vm[1], wf) : vm[1];
    vm[2] = d == 2 ? fmaxf(vm[2], wf) : vm[2];
  }
  if (!a.vmax_only) store_code(a.vp_out, 3 * p + d, a.g.izipv, codec_encode(a.cout, v));
}

template <bool kFine>
__global__ void __launch_bounds__(256, 4) k_kick(KickArgs a) {
  if (a.vmax_only && a.sd) {  // graph mode: the exact vmax rerun runs only when some component needs it
    bool need = false;
    for (int d = 0; d < 3; d++)
      if (!(__uint_as_float(*(volatile unsigned int*)&a.vmax_bits[d]) >= kick_tau(a, d))) need = true;
    if (!need) return;
  }
  __shared__ unsigned long long s_q[8][KICK_Q];  // 256 threads: 8 warps
  const Geo& g = a.g;
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  int qn = 0;                      // queued entries of this warp (warp-uniform)
  float vm[3] = {0.f, 0.f, 0.f};  // coarse: exact vmax; fine: the FP32 estimate
  float vlo[3] = {0.f, 0.f, 0.f};  // coarse: lower bounds of |v + vfield|
  // the zero-kick codes are the codes themselves, but for -nvbin/2, when the
  // table's count says so
  __shared__ float s_K;
  __shared__ unsigned s_max[6];  // float bits: vm, vlo
  if (threadIdx.x < 6) s_max[threadIdx.x] = 0u;
  if (threadIdx.x == 0)
    s_K = a.exact_only ? __int_as_float(0x7fffffff)
                       : kick_factor(kick_amid(a), kick_dt(a), __uint_as_float(__ldg(a.f2)));
  __syncthreads();
  const bool rt_same = kFine && a.pp_act && __ldg(a.cin.rt + 2 * a.cin.half) == 0;
  // whole warps iterate together (the queue's ballots); lanes past the end
  // compute on the last particle and store nothing
  for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p0 - lane < a.np;
       p0 += (int64_t)gridDim.x * blockDim.x) {
    const bool valid = p0 < a.np;
    const int64_t p = valid ? p0 : a.np - 1;
    KickCorners k;
    kick_corners<kFine>(a, p, k);
    const float w0 = __fmul_rn(k.d1[0], s_K), w1 = __fmul_rn(k.d2[0], s_K);
    const float w[2][2] = {{__fmul_rn(k.d1[1], k.d1[2]), __fmul_rn(k.d2[1], k.d1[2])},
                           {__fmul_rn(k.d1[1], k.d2[2]), __fmul_rn(k.d2[1], k.d2[2])}};  // [z][y]
    int codes[3];
#pragma unroll
    for (int d = 0; d < 3; d++) codes[d] = load_code(a.vp_in, 3 * p + d, g.izipv);
    if (kFine && a.pp_act) {
      // ext_pp_force's kick (ext_pp_force.f90:116-121) before the fine kick:
      // the prefilter's active particles were kicked by PP already; the
      // others' force is zero, their PP code the zero-kick code of theirs
      const bool on = (__ldg(a.pp_act + (p >> 5)) >> (p & 31)) & 1u;
#pragma unroll
      for (int d = 0; d < 3; d++)
        if (!on && (!rt_same || codes[d] == -a.cin.half)) codes[d] = __ldg(a.cin.rt + codes[d] + a.cin.half);
    } else if (kFine && a.fpp) {
      // ext_pp_force's kick before the fine kick, both in this pass: the PP
      // code (decoded and encoded with sigma_vi) is the one the fine kick decodes
      const float F[3] = {a.fpp[3 * p], a.fpp[3 * p + 1], a.fpp[3 * p + 2]};
      pp_kick3(a.cin, codes, F, a.pp_kf, a.pp_kd, a.exact_only);
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      float f[2][2][2];
      kick_gather<kFine>(a, k, a.f[d], f);
      const float dh = codec_decode_f(a.cin, codes[d]);
      float S = 0.f, T = 0.f;
#pragma unroll
      for (int z = 0; z < 2; z++)
#pragma unroll
        for (int y = 0; y < 2; y++) {
          const float f0 = f[z][y][0], f1 = f[z][y][1];
          S = __fmaf_rn(__fmaf_rn(f1, w1, __fmul_rn(f0, w0)), w[z][y], S);
          T = __fmaf_rn(__fmaf_rn(fabsf(f1), fabsf(w1), fabsf(__fmul_rn(f0, w0))), w[z][y], T);
        }
      const float vf = __fadd_rn(dh, S);
      const float E = __fmaf_rn(T * 1.3e-6f + (fabsf(dh) + fabsf(vf)) * 6.0e-8f, 1.25f, 1.0e-24f);
      int n;
      bool fast = certify_code(fabsf(vf), E, a.cout, &n);
      if (!kFine) {
        const float vfd = a.vfield[3 * (int64_t)k.cell + d];
        // |v + vfield| of the reference's FP64 v lies in [lo, ub]
        const float ub = (fabsf(vf) + E + fabsf(vfd)) * 1.000001f;
        const float lo = __fmul_rn(__fsub_rn(fabsf(__fadd_rn(vf, vfd)), E), 0.99999f);
        if (valid) vlo[d] = fmaxf(vlo[d], lo);
        // the first pass: lanes that may reach tau; the rerun: lanes that may
        // reach the largest lower bound, which the maximum does
        if (ub >= (a.vmax_only ? __uint_as_float(__ldg(&a.vmax_lo[d])) : kick_tau(a, d))) fast = false;
      } else if (a.vmax_est && valid) {
        vm[d] = fmaxf(vm[d], fabsf(__fadd_rn(vf, a.vfield[3 * (int64_t)k.cell + d])));
      }
      if (fast && valid && !a.vmax_only) store_code_i(a.vp_out, 3 * p + d, g.izipv, vf < 0.f ? -n : n);
      const bool defer = valid && !fast;
      const unsigned m = __ballot_sync(0xffffffffu, defer);
      if (m) {
        if (defer) s_q[wq][qn + __popc(m & ((1u << lane) - 1u))] = kick_qkey(p, d, codes[d]);
        qn += __popc(m);
        // the chain for 32 queued entries at a time, one per lane
        if (qn >= 32) {
          __syncwarp();
          kick_exact_entry<kFine>(a, s_q[wq][qn - 32 + lane], vm);
          qn -= 32;
          __syncwarp();
        }
      }
    }
  }
  __syncwarp();
  if (lane < qn) {
    kick_exact_entry<kFine>(a, s_q[wq][lane], vm);
  }
  // the block's maxima first: an atomic per warp and maximum, all on one
  // sector, took a third of a millisecond of 256^3 particles' coarse kick
  const bool mv = !kFine || a.vmax_est, ml = !kFine && !a.vmax_only;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (mv) warp_max_pos(&s_max[d], vm[d]);
    if (ml) warp_max_pos(&s_max[3 + d], vlo[d]);
  }
  __syncthreads();
  const int t = threadIdx.x;
  if (t < 3 && mv) atomicMax(kFine ? &a.vmax_est[t] : &a.vmax_bits[t], s_max[t]);
  if (t >= 3 && t < 6 && ml) atomicMax(&a.vmax_lo[t - 3], s_max[t]);
}

// The blocks that an SM holds, once: every block ends in its warps' part-filled
// queues, which cost as much as full ones, so fewer blocks are better.  Above 2^25
// particles the queues' share is small and the balance of more blocks gives more.
// Fine / coarse kick in ms with 4 and with 16 blocks an SM, uniform states (at
// z = 3 the same within 1 %): 256^3 particles 0.541 / 0.463 and 0.559 / 0.468,
// 320^3 1.042 / 0.898 and 1.064 / 0.895, 352^3 1.384 / 1.191 and 1.402 / 1.163,
// 384^3 1.818 / 1.570 and 1.814 / 1.532, 448^3 2.856 / 2.482 and 2.847 / 2.412,
// 512^3 4.320 / 3.696 and 4.286 / 3.595.
template <bool kFine>
void launch_kick(cube_ctx* c, const KickArgs& k) {
  k_kick<kFine><<<cube_grid(k.np, 256, k.np > (int64_t)1 << 25 ? 16 : 4), 256, 0, c->stream>>>(k);
}

}  // namespace

// Fixed-point scale of the deposits: each weight w <= mass becomes the integer
// w*2^s < 2^31 with the largest such s, so a 32-bit atomic adds it (64-bit
// shared-memory atomics are several times slower); a second 32-bit counter per
// mesh point takes the carries out of the first.
int dep_shift(float mass) {
  int s = 31;
  float lim = 1.0f;
  while (lim < mass && s > 1) {
    lim *= 2.0f;
    s--;
  }
  return s;
}

// -------------------------------------------------------------- init
int cube_kernels_init(cube_ctx* c, const float* fine_table, const float* coarse_table) {
  int nf = c->nf, nc = c->p.nc, nfc = c->p.nf_cutoff;
  cudaStream_t s = c->stream;
  // ---- fine: fill the odd-mirrored table, R2C, keep Im/nf^3
  float* dtab = nullptr;
  CUBE_CUDA(c, cudaMalloc(&dtab, sizeof(float) * 3 * nfc * nfc * nfc));
  CUBE_CUDA(c, cudaMemcpyAsync(dtab, fine_table, sizeof(float) * 3 * nfc * nfc * nfc, cudaMemcpyHostToDevice, s));
  int64_t nfh = nf / 2 + 1;
  int64_t nspec = nfh * nf * (int64_t)nf;
  int64_t fpad = 2 * nspec;
  float scale_f = (float)(1.0 / ((double)nf * nf * nf));
  int w = 2 * nfc - 1;
  for (int d = 0; d < 3; d++) {
    CUBE_CUDA(c, cudaMemsetAsync(c->rho_f, 0, 4 * fpad, s));
    k_fill_fine_table<<<(w * w * w + 255) / 256, 256, 0, s>>>(dtab, nfc, c->p.pp_on ? c->p.pp_range : -1, d, nf,
                                                               c->rho_f);
    CUBE_FFT(c, cufftExecR2C(c->plan_f_r2c, c->rho_f, (cufftComplex*)c->rho_f));
    k_take_imag<<<cube_grid(nspec, 256), 256, 0, s>>>((const float2*)c->rho_f, nspec, scale_f,
                                                       c->kern_f + d * nspec);
  }
  CUBE_CUDA(c, cudaGetLastError());
  CUBE_CUDA(c, cudaStreamSynchronize(s));
  cudaFree(dtab);

  // ---- coarse: -r/r^3 with the near-field table (kernel_c.f90:16-72), on the host
  int64_t n3 = (int64_t)nc * nc * nc;
  int ncell = c->p.ncell;
  std::vector<float> ck(3 * n3), raw(3 * n3);
  auto rcoord = [&](int i) { return (float)(ncell * (((i + nc / 2) % nc) - nc / 2)); };
  for (int k = 0; k < nc; k++)
    for (int j = 0; j < nc; j++)
      for (int i = 0; i < nc; i++) {
        float rx[3] = {rcoord(i), rcoord(j), rcoord(k)};
        float r = std::sqrt(rx[0] * rx[0] + rx[1] * rx[1] + rx[2] * rx[2]);
        float r3 = (r * r) * r;
        int64_t idx = i + (int64_t)nc * (j + (int64_t)nc * k);
        for (int d = 0; d < 3; d++) raw[d * n3 + idx] = r == 0.f ? 0.f : -rx[d] / r3;
      }
  ck = raw;
  // octant copies of ck_table (kernel_c.f90:43-72); with one image all eight apply in order
  auto T = [&](int d, int i, int j, int k) { return coarse_table[d + 3 * (i + 4 * (j + 4 * k))]; };
  auto CK = [&](int d, int i, int j, int k) -> float& {  // 1-based Fortran indices into ck(d,i,j,k)
    return ck[(d - 1) * n3 + (i - 1) + (int64_t)nc * ((j - 1) + (int64_t)nc * (k - 1))];
  };
  // rev(a) maps Fortran nc-2..nc to table 4..2
  for (int k = 1; k <= 4; k++)
    for (int j = 1; j <= 4; j++)
      for (int i = 1; i <= 4; i++)
        for (int d = 1; d <= 3; d++) CK(d, i, j, k) = T(d - 1, i - 1, j - 1, k - 1);  // 1
  for (int m = 0; m < 3; m++) {  // index nc-2+m <-> table 4-m
    for (int j = 1; j <= 4; j++)
      for (int k = 1; k <= 4; k++) {
        int a = nc - 2 + m, t = 4 - m;
        // 5 x
        CK(1, a, j, k) = -T(0, t - 1, j - 1, k - 1);
        CK(2, a, j, k) = T(1, t - 1, j - 1, k - 1);
        CK(3, a, j, k) = T(2, t - 1, j - 1, k - 1);
      }
    for (int i = 1; i <= 4; i++)
      for (int k = 1; k <= 4; k++) {
        int a = nc - 2 + m, t = 4 - m;
        // 3 y
        CK(1, i, a, k) = T(0, i - 1, t - 1, k - 1);
        CK(3, i, a, k) = T(2, i - 1, t - 1, k - 1);
        CK(2, i, a, k) = -T(1, i - 1, t - 1, k - 1);
      }
    for (int i = 1; i <= 4; i++)
      for (int j = 1; j <= 4; j++) {
        int a = nc - 2 + m, t = 4 - m;
        // 2 z
        CK(1, i, j, a) = T(0, i - 1, j - 1, t - 1);
        CK(2, i, j, a) = T(1, i - 1, j - 1, t - 1);
        CK(3, i, j, a) = -T(2, i - 1, j - 1, t - 1);
      }
  }
  for (int m1 = 0; m1 < 3; m1++)
    for (int m2 = 0; m2 < 3; m2++) {
      int a1 = nc - 2 + m1, t1 = 4 - m1, a2 = nc - 2 + m2, t2 = 4 - m2;
      for (int i = 1; i <= 4; i++) {  // 4 yz: (j=a1,k=a2)
        CK(1, i, a1, a2) = T(0, i - 1, t1 - 1, t2 - 1);
        CK(2, i, a1, a2) = -T(1, i - 1, t1 - 1, t2 - 1);
        CK(3, i, a1, a2) = -T(2, i - 1, t1 - 1, t2 - 1);
      }
      for (int j = 1; j <= 4; j++) {  // 6 xz: (i=a1,k=a2)
        CK(1, a1, j, a2) = -T(0, t1 - 1, j - 1, t2 - 1);
        CK(3, a1, j, a2) = -T(2, t1 - 1, j - 1, t2 - 1);
        CK(2, a1, j, a2) = T(1, t1 - 1, j - 1, t2 - 1);
      }
      for (int k = 1; k <= 4; k++) {  // 7 xy: (i=a1,j=a2)
        CK(1, a1, a2, k) = -T(0, t1 - 1, t2 - 1, k - 1);
        CK(2, a1, a2, k) = -T(1, t1 - 1, t2 - 1, k - 1);
        CK(3, a1, a2, k) = T(2, t1 - 1, t2 - 1, k - 1);
      }
    }
  for (int m1 = 0; m1 < 3; m1++)
    for (int m2 = 0; m2 < 3; m2++)
      for (int m3 = 0; m3 < 3; m3++)  // 8 xyz
        for (int d = 1; d <= 3; d++)
          CK(d, nc - 2 + m1, nc - 2 + m2, nc - 2 + m3) = -T(d - 1, 4 - m1 - 1, 4 - m2 - 1, 4 - m3 - 1);

  // ---- FFTs and LRCKCORR; stage through force_c[0] (padded)
  int64_t nch = nc / 2 + 1;
  int64_t cspec = nch * nc * (int64_t)nc;
  float* buf = c->force_c[0];
  float* bufr = c->force_c[1];
  size_t row = (size_t)nc * 4, pitch = (size_t)(nc + 2) * 4;
  for (int d = 0; d < 3; d++) {
    CUBE_CUDA(c, cudaMemcpy2DAsync(buf, pitch, ck.data() + d * n3, row, row, (size_t)nc * nc,
                                   cudaMemcpyHostToDevice, s));
    CUBE_FFT(c, cufftExecR2C(c->plan_c_r2c, buf, (cufftComplex*)buf));
    k_take_imag<<<cube_grid(cspec, 256), 256, 0, s>>>((const float2*)buf, cspec, 1.0f, c->kern_c + d * cspec);
    CUBE_CUDA(c, cudaMemcpy2DAsync(bufr, pitch, raw.data() + d * n3, row, row, (size_t)nc * nc,
                                   cudaMemcpyHostToDevice, s));
    CUBE_FFT(c, cufftExecR2C(c->plan_c_r2c, bufr, (cufftComplex*)bufr));
    k_lrck<<<cube_grid(cspec, 256), 256, 0, s>>>(c->kern_c + d * cspec, (const float2*)bufr, nc, d);
  }
  // fold 1/nc^3 (a power of two: exact)
  k_scale<<<cube_grid(3 * cspec, 256), 256, 0, s>>>(c->kern_c, 3 * cspec, (float)(1.0 / ((double)nc * nc * nc)));
  CUBE_CUDA(c, cudaGetLastError());
  CUBE_CUDA(c, cudaStreamSynchronize(s));
  return CUBE_OK;
}

namespace {
__global__ void k_force_pre(float* __restrict__ f, int64_t n, float a_mid, float dt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    f[i] = kick_pre(f[i], a_mid, dt);
}
}  // namespace

// the meshes hold the transforms' forces, their maximum behind them
static void force_transformed(cube_ctx* c, int coarse) {
  cube_ctx* o = c->owner ? c->owner : c;
  o->force_pre[coarse].on = false;
  o->f2_known[coarse] = true;
}

int cube_force_foreign(cube_ctx* c, int coarse) {
  cube_ctx* o = c->owner ? c->owner : c;
  o->force_pre[coarse].on = o->f2_known[coarse] = false;
  CUBE_CUDA(c, cudaMemsetAsync(c->f2_kick + coarse, 0xff, 4, c->stream));
  return CUBE_OK;
}

int cube_force_settle(cube_ctx* c, int coarse) {
  const cube_ctx::ForcePre pre = (c->owner ? c->owner : c)->force_pre[coarse];
  if (!pre.on) return CUBE_OK;
  const int n = coarse ? c->p.nc : c->nf;
  const int64_t cells = (int64_t)(n + 2) * n * n;
  for (int d = 0; d < 3; d++)
    k_force_pre<<<cube_grid(cells, 256), 256, 0, c->stream>>>(coarse ? c->force_c[d] : c->force_f[d], cells, pre.a_mid,
                                                               pre.dt);
  CUBE_CUDA(c, cudaGetLastError());
  return cube_force_foreign(c, coarse);
}

// (the pass over the mesh takes a fraction of the FP64 chain for every component,
// which is the kick's way without the maximum)
int cube_force_ready(cube_ctx* c, int coarse) {
  if (int r = cube_force_settle(c, coarse)) return r;
  cube_ctx* o = c->owner ? c->owner : c;
  if (o->f2_known[coarse]) return CUBE_OK;
  CUBE_CUDA(c, cudaMemsetAsync(c->f2_kick + coarse, 0, 4, c->stream));
  launch_f2max(c, coarse ? c->force_c : c->force_f, coarse ? c->p.nc : c->nf, c->f2_kick + coarse, c->f2_kick + coarse);
  CUBE_CUDA(c, cudaGetLastError());
  o->f2_known[coarse] = true;
  return CUBE_OK;
}

// ----------------------------------------------------------------- fine
int cube_fine_density_impl(cube_ctx* c, cube_stats* st, bool accumulate, bool fresh) {
  cudaStream_t s = c->stream;
  Geo g = make_geo(c);
  if (!c->graph_mode && !fresh)  // (a captured step's head zeroes them)
    CUBE_CUDA(c, cudaMemsetAsync(c->dstats, 0, sizeof(DevStats), s));
  const int sh = dep_shift(c->p.mass_p);
  DepArgs a{g, c->xp[c->cur], c->rhoc[c->cur], c->cstart[c->cur], c->p.mass_p, c->rho_f, &c->dstats->rhof_fix, 0, 0.f,
            std::ldexp(1.0f, sh), std::ldexp(1.0f, -sh), accumulate ? 1 : 0};
  cube_phase_begin(c, PH_F_DEPOSIT);
  int r = launch_fine_deposit(c, a);
  cube_phase_end(c, PH_F_DEPOSIT);
  if (r) return r;
  if (st) {
    r = cube_stats_fetch(c);
    if (r) return r;
    st->testrhof = std::ldexp((double)c->hstats->rhof_fix, -dep_shift(c->p.mass_p));
  }
  return CUBE_OK;
}

void cube_fine_stats(const cube_ctx* c, cube_stats* st) {
  st->f2_max_fine = bits_float(c->hstats->f2_fine_bits);
  st->testrhof = std::ldexp((double)c->hstats->rhof_fix, -dep_shift(c->p.mass_p));
}

int cube_forces_fork(cube_ctx* c) {
  if (!c->graph_mode) CUBE_CUDA(c, cudaMemsetAsync(c->dstats, 0, sizeof(DevStats), c->stream));
  CUBE_CUDA(c, cudaEventRecord(c->ev_aux, c->stream));
  return CUBE_OK;
}

int cube_coarse_beside(cube_ctx* c) {
  cudaStream_t s = c->stream;
  CUBE_CUDA(c, cudaStreamWaitEvent(c->stream_aux, c->ev_aux, 0));
  for (cufftHandle h : {c->plan_c_r2c, c->plan_c_c2r}) CUBE_FFT(c, cufftSetStream(h, c->stream_aux));
  c->stream = c->stream_aux;
  const int r = cube_coarse_forces_impl(c, nullptr, true);
  c->stream = s;
  for (cufftHandle h : {c->plan_c_r2c, c->plan_c_c2r}) CUBE_FFT(c, cufftSetStream(h, s));
  if (r) return r;
  CUBE_CUDA(c, cudaEventRecord(c->ev_coarse, c->stream_aux));
  return CUBE_OK;
}

int cube_forces_join(cube_ctx* c) {
  CUBE_CUDA(c, cudaStreamWaitEvent(c->stream, c->ev_coarse, 0));
  return CUBE_OK;
}

int cube_fine_forces_impl(cube_ctx* c, cube_stats* st, bool fresh) {
  int r0 = cube_fine_density_impl(c, nullptr, false, fresh);
  if (r0) return r0;
  return cube_fine_spectral_impl(c, st);
}

// forces from the density on the fine mesh (pm.f90:112-126)
int cube_fine_spectral_impl(cube_ctx* c, cube_stats* st) {
  cudaStream_t s = c->stream;
  int64_t nfh = c->nf / 2 + 1;
  int64_t nspec = nfh * c->nf * (int64_t)c->nf;
  cube_phase_begin(c, PH_F_R2C);
  CUBE_FFT(c, cufftExecR2C(c->plan_f_r2c, c->rho_f, (cufftComplex*)c->rho_f));
  cube_phase_end(c, PH_F_R2C);
  cube_phase_begin(c, PH_F_GREEN);
  k_green3<<<cube_grid(nspec, 256), 256, 0, s>>>((const float2*)c->rho_f, c->kern_f, nspec, (float2*)c->force_f[0],
                                                  (float2*)c->force_f[1], (float2*)c->force_f[2], c->f2_kick);
  cube_phase_end(c, PH_F_GREEN);
  cube_phase_begin(c, PH_F_C2R);
  for (int d = 0; d < 3; d += c->f_c2r_batch)
    CUBE_FFT(c, cufftExecC2R(c->plan_f_c2r, (cufftComplex*)c->force_f[d], c->force_f[d]));
  cube_phase_end(c, PH_F_C2R);
  cube_phase_begin(c, PH_F_F2MAX);
  launch_f2max(c, c->force_f, c->nf, &c->dstats->f2_fine_bits, c->f2_kick);
  force_transformed(c, 0);
  cube_phase_end(c, PH_F_F2MAX);
  CUBE_CUDA(c, cudaGetLastError());
  if (st) {
    int r = cube_stats_fetch(c);
    if (r) return r;
    cube_fine_stats(c, st);
  }
  return CUBE_OK;
}

int cube_fine_kick_impl(cube_ctx* c, float a_mid, float dt, bool with_pp) {
  KickArgs k{};
  if (with_pp) {  // the PP kick of cube_pp_launch(.., defer_kick), applied here
    if (c->graph_mode || !c->fpp) return cube_fail(c, CUBE_ERR_ARG, "PP kick in the fine kick: eager mode with PP only");
    if (c->pp_act_valid)
      k.pp_act = c->pp_act;  // the active particles are kicked; the others take the zero-kick codes here
    else
      k.fpp = c->fpp;
    k.pp_kd = (((double)a_mid * (double)dt) / 6.0) / (double)CUBE_PI_F;
    k.pp_kf = (float)k.pp_kd;
  }
  if (c->graph_mode) {  // decode with sigma_vi, encode with sigma_vi_new
    CUBE_CUDA(c, cudaStreamWaitEvent(c->stream, c->ev_codec, 0));
    cube_codec_view_dev(c, c->graph_slot, &c->sd->h.cf_vi, &k.cin);
    cube_codec_view_dev(c, 1 - c->graph_slot, &c->sd->cf_new, &k.cout);
    k.sd = c->sd;
  } else {
    int r = cube_codec_pair(c, c->sigma_vi, c->sigma_vi_new, &k.cin, &k.cout);
    if (r) return r;
  }
  k.g = make_geo(c);
  k.np = c->np;
  k.xp = c->xp[c->cur];
  k.vp_in = c->vp[c->cur];
  k.vp_out = c->vp[c->cur];
  k.pcell = c->pcell[c->cur];
  k.vfield = c->vfield[c->cur];
  for (int d = 0; d < 3; d++) k.f[d] = c->force_f[d];
  k.f2 = c->f2_kick;
  k.a_mid = a_mid;
  k.dt = dt;
  k.vmax_bits = nullptr;
  k.exact_only = c->opt_exact_kicks;
  // after an upload or initial conditions the last vmax is unknown: the fine
  // kick then records the velocities' maxima for the coarse kick's threshold
  // (the fine density of this step zeroed the estimate)
  if (!c->graph_mode && c->vmax_prev[0] == 0.f && c->vmax_prev[1] == 0.f && c->vmax_prev[2] == 0.f)
    k.vmax_est = c->dstats->vmax_est_bits;
  cube_phase_begin(c, PH_F_KICK);
  launch_kick<true>(c, k);
  cube_phase_end(c, PH_F_KICK);
  CUBE_CUDA(c, cudaGetLastError());
  return CUBE_OK;
}

// CIC density of the particles on an ng^3 mesh (ng = nc, 2 nc or 4 nc) for the
// power spectrum, mass 1 per particle (cicpower.f90:79,100-133), into the
// padded mesh rho; *total receives the exact fixed-point sum.
int cube_pk_deposit(cube_ctx* c, int ng, float* rho, unsigned long long* total) {
  const int sh = dep_shift(1.0f);
  DepArgs a{make_geo(c), c->xp[c->cur], c->rhoc[c->cur], c->cstart[c->cur], 1.0f, rho, total, ng,
            1.0f / (float)c->p.nc, std::ldexp(1.0f, sh), std::ldexp(1.0f, -sh), 0};
  int nc = c->p.nc;
  if (ng == nc) return launch_deposit<1, 8, 8, 8, 1, 1, true>(c, a);
  if (ng == 2 * nc) return launch_deposit<2, 8, 8, 4, 1, 1, true>(c, a);
  if (ng == 4 * nc) return launch_deposit<4, 8, 4, 4, 1, 1, true>(c, a);
  return cube_fail(c, CUBE_ERR_ARG, "power-spectrum mesh must be nc, 2nc or 4nc per dimension");
}

// --------------------------------------------------------------- coarse
int cube_coarse_density_impl(cube_ctx* c, cube_stats* st, bool accumulate, bool fresh) {
  Geo g = make_geo(c);
  if (!fresh) {
    CUBE_CUDA(c, cudaMemsetAsync(&c->dstats->f2_coarse_bits, 0, 4, c->stream));
    CUBE_CUDA(c, cudaMemsetAsync(&c->dstats->rhoc_fix, 0, 8, c->stream));
  }
  const int sh = dep_shift(c->p.mass_p);
  DepArgs a{g, c->xp[c->cur], c->rhoc[c->cur], c->cstart[c->cur], c->p.mass_p, c->rho_c, &c->dstats->rhoc_fix, 0, 0.f,
            std::ldexp(1.0f, sh), std::ldexp(1.0f, -sh), accumulate ? 1 : 0};
  cube_phase_begin(c, PH_C_DEPOSIT);
  int r = launch_coarse_deposit(c, a);
  cube_phase_end(c, PH_C_DEPOSIT);
  if (r) return r;
  if (st) {
    r = cube_stats_fetch(c);
    if (r) return r;
    st->testrhoc = std::ldexp((double)c->hstats->rhoc_fix, -dep_shift(c->p.mass_p));
  }
  return CUBE_OK;
}

int cube_coarse_forces_impl(cube_ctx* c, cube_stats* st, bool fresh) {
  int r0 = cube_coarse_density_impl(c, nullptr, false, fresh);
  if (r0) return r0;
  return cube_coarse_spectral_impl(c, st);
}

// forces from the density on the coarse mesh (pm.f90:275-315)
int cube_coarse_spectral_impl(cube_ctx* c, cube_stats* st) {
  cudaStream_t s = c->stream;
  int nc = c->p.nc;
  int64_t nch = nc / 2 + 1;
  int64_t cspec = nch * nc * (int64_t)nc;
  cube_phase_begin(c, PH_C_FFT);
  CUBE_FFT(c, cufftExecR2C(c->plan_c_r2c, c->rho_c, (cufftComplex*)c->rho_c));
  k_green3<<<cube_grid(cspec, 256), 256, 0, s>>>((const float2*)c->rho_c, c->kern_c, cspec, (float2*)c->force_c[0],
                                                  (float2*)c->force_c[1], (float2*)c->force_c[2], c->f2_kick + 1);
  for (int d = 0; d < 3; d += c->c_c2r_batch)
    CUBE_FFT(c, cufftExecC2R(c->plan_c_c2r, (cufftComplex*)c->force_c[d], c->force_c[d]));
  launch_f2max(c, c->force_c, nc, &c->dstats->f2_coarse_bits, c->f2_kick + 1);
  force_transformed(c, 1);
  cube_phase_end(c, PH_C_FFT);
  CUBE_CUDA(c, cudaGetLastError());
  if (st) {
    int r = cube_stats_fetch(c);
    if (r) return r;
    st->f2_max_coarse = bits_float(c->hstats->f2_coarse_bits);
    st->testrhoc = std::ldexp((double)c->hstats->rhoc_fix, -dep_shift(c->p.mass_p));
  }
  return CUBE_OK;
}

int cube_coarse_kick_impl(cube_ctx* c, float a_mid, float dt, cube_stats* st, bool fresh) {
  KickArgs k{};
  int r;
  if (c->graph_mode) {  // sigma_vi is now sigma_vi_new for both
    cube_codec_view_dev(c, 1 - c->graph_slot, &c->sd->cf_new, &k.cin);
    cube_codec_view_dev(c, 1 - c->graph_slot, &c->sd->cf_new, &k.cout);
    k.sd = c->sd;
  } else {
    r = cube_codec_pair(c, c->sigma_vi, c->sigma_vi, &k.cin, &k.cout);
    if (r) return r;
  }
  int cur = c->cur, alt = 1 - cur;
  if (!fresh) {
    CUBE_CUDA(c, cudaMemsetAsync(c->dstats->vmax_bits, 0, 12, c->stream));
    CUBE_CUDA(c, cudaMemsetAsync(c->dstats->vmax_lo_bits, 0, 12, c->stream));
  }
  k.g = make_geo(c);
  k.np = c->np;
  k.xp = c->xp[cur];
  k.vp_in = c->vp[cur];
  k.vp_out = c->vp[alt];  // the input codes stay intact for an exact vmax rerun
  k.pcell = c->pcell[cur];
  k.vfield = c->vfield[cur];
  k.f2 = c->f2_kick + 1;
  for (int d = 0; d < 3; d++) {
    k.f[d] = c->force_c[d];
    // velocities change little per step: every lane that could reach 0.95 of
    // the last vmax is evaluated exactly; if the maximum ends below that, a
    // rerun evaluates the lanes that could reach this pass's largest lower
    // bound (the maximum's lane among them)
    k.tau[d] = kVmaxTau * c->vmax_prev[d];
  }
  // last vmax unknown: 0.7 of the fine kick's FP32 maxima instead (zero when
  // no fine kick recorded them: every lane exact)
  const bool est = !c->graph_mode && c->vmax_prev[0] == 0.f && c->vmax_prev[1] == 0.f && c->vmax_prev[2] == 0.f;
  if (est) k.tau_est = c->dstats->vmax_est_bits;
  k.a_mid = a_mid;
  k.dt = dt;
  k.vmax_bits = c->dstats->vmax_bits;
  k.vmax_lo = c->dstats->vmax_lo_bits;
  k.vmax_only = 0;
  k.exact_only = c->opt_exact_kicks;
  cube_phase_begin(c, PH_C_KICK);
  if (c->vp_host && !c->graph_mode) {
    // a download is waiting for vp: kick in pieces of particles, each piece's
    // codes going to the host while the next is kicked; eight, or fewer of at
    // least 2^18 (below that a piece's launch and copy cost more than they hide)
    const size_t bx = 3 * (size_t)c->p.izipx, bv = 3 * (size_t)c->p.izipv;
    const int pieces = (int)std::max<int64_t>(1, std::min<int64_t>(8, c->np >> 18));
    for (int i = 0; i < pieces; i++) {
      const int64_t p0 = c->np * i / pieces, p1 = c->np * (i + 1) / pieces;
      if (p1 <= p0) continue;
      KickArgs kp = k;
      kp.np = p1 - p0;
      kp.xp = (const char*)k.xp + bx * p0;
      kp.vp_in = (const char*)k.vp_in + bv * p0;
      kp.vp_out = (char*)k.vp_out + bv * p0;
      kp.pcell = k.pcell + p0;
      launch_kick<false>(c, kp);
      CUBE_CUDA(c, cudaEventRecord(c->ev_copy_start, c->stream));
      CUBE_CUDA(c, cudaStreamWaitEvent(c->stream_copy, c->ev_copy_start, 0));
      CUBE_CUDA(c, cudaMemcpyAsync((char*)c->vp_host + bv * p0, kp.vp_out, bv * (p1 - p0), cudaMemcpyDeviceToHost,
                                   c->stream_copy));
    }
    CUBE_CUDA(c, cudaEventRecord(c->ev_copy, c->stream_copy));
    c->copy_pending = true;
    c->vp_host = nullptr;
  } else launch_kick<false>(c, k);
  cube_phase_end(c, PH_C_KICK);
  CUBE_CUDA(c, cudaGetLastError());
  if (c->graph_mode) {
    // the exact rerun decides on the device whether it runs
    k.vmax_only = 1;
    launch_kick<false>(c, k);
    CUBE_CUDA(c, cudaGetLastError());
    void* t = c->vp[cur];
    c->vp[cur] = c->vp[alt];
    c->vp[alt] = t;
    return CUBE_OK;
  }
  r = cube_stats_fetch(c);
  if (r) return r;
  c->codec_ahead = -1;  // the kicks waited for the tables and are done
  float vm[3];
  bool rerun = false;
  for (int d = 0; d < 3; d++) {
    vm[d] = bits_float(c->hstats->vmax_bits[d]);
    const float tau = est ? 0.7f * bits_float(c->hstats->vmax_est_bits[d]) : k.tau[d];
    if (!(vm[d] >= tau)) rerun = true;
  }
  if (rerun) {
    CUBE_CUDA(c, cudaMemsetAsync(c->dstats->vmax_bits, 0, 12, c->stream));
    k.vmax_only = 1;
    launch_kick<false>(c, k);
    CUBE_CUDA(c, cudaGetLastError());
    r = cube_stats_fetch(c);
    if (r) return r;
    for (int d = 0; d < 3; d++) vm[d] = bits_float(c->hstats->vmax_bits[d]);
  }
  void* t = c->vp[cur];
  c->vp[cur] = c->vp[alt];
  c->vp[alt] = t;
  for (int d = 0; d < 3; d++) c->vmax_prev[d] = vm[d];
  if (st) {
    for (int d = 0; d < 3; d++) st->vmax[d] = vm[d];
    st->f2_max_coarse = bits_float(c->hstats->f2_coarse_bits);
    st->testrhoc = std::ldexp((double)c->hstats->rhoc_fix, -dep_shift(c->p.mass_p));
  }
  return CUBE_OK;
}
