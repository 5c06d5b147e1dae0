// Device kernels that prepare the multislice inputs: Kirkland atom windows,
// the transmission slices exp(i sigma V), the k-space probe and its
// normalisation, and the propagator table.
#include "msx_bessel.cuh"
#include "msx_internal.h"

#include <cooperative_groups.h>

#include <cmath>
#include <map>
#include <mutex>

namespace msx {

__constant__ CoshTable kCosh{};

// ------------------------------------------------------------------ atom windows
// Follows _get_potential (namsa/msa.py:180-196) and bin_2d_array
// (namsa/utils.py:101-108): oversampled inclusive grid
// x_i = -range/2 + i*range/(n-1), Kirkland sum
//   v = 4 pi^2 a0 e sum_i a_i K0(2 pi r sqrt(b_i) + 0.1) + 2 pi^2 a0 e sum_i c_i/d_i exp(-pi^2 r^2/d_i)
// with a0 = 0.529, e = 14.4, the oversample x oversample mean, minus the window
// minimum, rounded to float32.  All arithmetic is double.
//
// The grid is symmetric about its centre, so bins (i, j), (H-1-i, j), (i, W-1-j)
// and (H-1-i, W-1-j) are equal and one quadrant is evaluated.  Every Kirkland
// coefficient is positive, so v decreases with r and the window minimum is the
// corner bin, which each CTA evaluates beside its own bins.
//
// Bound by double-precision instructions (about two fused multiply-adds a
// clock and SM): an exponential per quadrature term.  The quadrant takes a
// quarter of the samples, the table the cosh of every term, the coarser step
// half of the terms of x < 3, and one thread per oversampled row of a bin
// fills the chip.  94 x 94 bins of one species at oversample 2: 938 us with
// every bin evaluated by one thread, 116 us so.
constexpr int kWinThreads = 128;

// sum over b (in order) of the samples (i os + a, j os + b)
__device__ double window_row(const double* c, int i, int j, int a, int os, double sx, double sy, double start) {
  const double pi = 3.14159265358979323846;
  const double pre = 4.0 * pi * pi * 0.529 * 14.4;
  double accr = 0;
  for (int b = 0; b < os; ++b) {
    const double gx = (double)(i * os + a) * sx + start;
    const double gy = (double)(j * os + b) * sy + start;
    const double r = sqrt(gx * gx + gy * gy);
    double v = 0;
    for (int k = 0; k < 3; ++k) {
      const double ak = c[k], bk = c[3 + k], ck = c[6 + k], dk = c[9 + k];
      const double term = pre * ak * bessel_k0(2 * pi * r * sqrt(bk) + 0.1, kCosh.v) + pre / 2. * ck / dk * exp(-pi * pi * r * r / dk);
      v = (k == 0) ? term : v + term;
    }
    accr = (b == 0) ? v : accr + v;
  }
  return accr / os;
}

// Grid: blocks of bins of the quadrant, species after species.  `rows` threads share a bin
// (the oversampled rows a, a + rows, ...); slot 0 is the corner bin, slots
// 1 .. bins are the block's own.  numpy's order: mean over the last axis, then
// over the second-to-last.
__global__ void __launch_bounds__(kWinThreads)
atom_window_kernel(const double* __restrict__ coeff, int n0, int n1, int os, int rows, int bins, double range,
                   float* __restrict__ out) {
  __shared__ double part[kWinThreads];
  __shared__ double val[kWinThreads];
  const int h0 = n0 / os, h1 = n1 / os;
  const int q1 = (h1 + 1) / 2, quad = ((h0 + 1) / 2) * q1;
  const int blocks = (quad + bins - 1) / bins;  // of a species
  const int species = blockIdx.x / blocks, block = blockIdx.x - species * blocks;
  const double* c = coeff + 12 * species;
  const double start = -range / 2, sx = range / (double)(n0 - 1), sy = range / (double)(n1 - 1);
  const int slot = threadIdx.x / rows, a0 = threadIdx.x % rows;
  const int bin = slot == 0 ? 0 : block * bins + slot - 1;  // bin 0 is the corner
  const bool live = slot <= bins && bin < quad;
  double acc = 0;
  for (int base = 0; base < os; base += rows) {
    const int a = base + a0;
    part[threadIdx.x] = live && a < os ? window_row(c, bin / q1, bin % q1, a, os, sx, sy, start) : 0.0;
    __syncthreads();
    if (live && a0 == 0)
      for (int k = 0; k < rows && base + k < os; ++k) {
        const double v = part[threadIdx.x + k];
        acc = (base + k == 0) ? v : acc + v;
      }
    __syncthreads();
  }
  if (a0 == 0) val[slot] = acc / os;
  __syncthreads();
  if (live && slot > 0 && a0 == 0) {
    const float v = (float)(val[slot] - val[0]);
    const int i = bin / q1, j = bin % q1;
    float* o = out + (size_t)species * h0 * h1;
    o[(size_t)i * h1 + j] = v;
    o[(size_t)(h0 - 1 - i) * h1 + j] = v;
    o[(size_t)i * h1 + h1 - 1 - j] = v;
    o[(size_t)(h0 - 1 - i) * h1 + h1 - 1 - j] = v;
  }
}

// ------------------------------------------------------------------ transmission slices
// One CTA per 32x32 pixel tile of one slice.  Follows BuildScatteringPotential
// (namsa/potential_kernels.cu:5-60): a site (zidx, yc, xc) covers rows
// [rintf(yc - H/2), rintf(yc + H/2)) and the matching columns, clipped to the
// grid (no wrap) and to the window extent.  Each pixel sums the windows of its
// slice's sites in site order in float32 (the order of the reference's
// per-pixel atomicAdds, which come from one thread per pixel), then
// t = (cos(sigma V), sin(sigma V)) with NaN -> 1.
//
// Sites are binned per tile in shared memory: each chunk of 256 sites is
// tested against the tile and the overlapping ones are compacted in order.
//
// Bound by instructions (at eight overlapping sites a pixel the 8-byte results
// need a sixth of the time): the thread that finds a site clips its rectangle
// once, a warp's rows are tested with warp-uniform branches, and the windows of
// four sites are read before the first is added (sixteen loads in flight per
// thread, the additions still in site order; a pixel outside a window adds +0,
// which leaves the sum as it is).  199 slices of 512^2, 128 sites of 94 x 94
// each: 391 us with the tests in the inner loop, 290 us so.
constexpr int kPotTile = 32;
constexpr int kPotThreads = 256;
constexpr int kPotBatch = 4;

__global__ void __launch_bounds__(kPotThreads)
potential_kernel(const int4* __restrict__ sites, const int* __restrict__ slice_off, const float* __restrict__ windows,
                 int H, int W, int Ny, int Nx, float sigma, float2* __restrict__ trans, float* __restrict__ pot) {
  __shared__ int4 rect[kPotThreads];        // rows [x, y), columns [z, w) of a site's window inside the grid
  __shared__ const float* base[kPotThreads];  // the window's element of pixel (0, 0)
  __shared__ int warp_count[kPotThreads / 32];
  const int s = blockIdx.z;
  const int ty0 = blockIdx.y * kPotTile, tx0 = blockIdx.x * kPotTile;
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int px = tx0 + lane;
  const int py0 = ty0 + warp;  // rows py0 + 8*k, k = 0..3
  float acc[kPotTile / 8] = {0.f, 0.f, 0.f, 0.f};
  const int begin = slice_off[s], end = slice_off[s + 1];
  const float hh = H * 0.5f, hw = W * 0.5f;
  for (int chunk = begin; chunk < end; chunk += kPotThreads) {
    const int idx = chunk + threadIdx.x;
    int4 r = make_int4(0, 0, 0, 0);
    const float* w0 = windows;
    bool hit = false;
    if (idx < end) {
      const int4 st = sites[idx];
      const int ys = (int)rintf((float)st.y - hh), ye = (int)rintf((float)st.y + hh);
      const int xs = (int)rintf((float)st.z - hw), xe = (int)rintf((float)st.z + hw);
      r = make_int4(max(ys, 0), min(min(ye, Ny), ys + H), max(xs, 0), min(min(xe, Nx), xs + W));
      hit = min(r.y, ty0 + kPotTile) > max(r.x, ty0) && min(r.w, tx0 + kPotTile) > max(r.z, tx0);
      w0 = windows + ((size_t)st.x * H * W - ((long long)ys * W + xs));
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) warp_count[warp] = __popc(ballot);
    __syncthreads();
    int offset = 0, total = 0;
    for (int w = 0; w < kPotThreads / 32; ++w) {
      if (w < warp) offset += warp_count[w];
      total += warp_count[w];
    }
    if (hit) {
      const int at = offset + __popc(ballot & ((1u << lane) - 1u));
      rect[at] = r;
      base[at] = w0;
    }
    __syncthreads();
    for (int i0 = 0; i0 < total; i0 += kPotBatch) {
      float v[kPotBatch][kPotTile / 8];
#pragma unroll
      for (int u = 0; u < kPotBatch; ++u) {
        const int i = min(i0 + u, total - 1);
        const int4 q = rect[i];
        const float* w = base[i] + px;
        const bool colok = i0 + u < total && px >= q.z && px < q.w;
#pragma unroll
        for (int k = 0; k < kPotTile / 8; ++k) {
          const int py = py0 + 8 * k;
          v[u][k] = 0.f;
          if (py >= q.x && py < q.y && colok) v[u][k] = __ldg(w + (long long)py * W);
        }
      }
#pragma unroll
      for (int u = 0; u < kPotBatch; ++u)
#pragma unroll
        for (int k = 0; k < kPotTile / 8; ++k) acc[k] += v[u][k];
    }
    __syncthreads();
  }
  if (px < Nx) {
#pragma unroll
    for (int k = 0; k < kPotTile / 8; ++k) {
      const int py = py0 + 8 * k;
      if (py < Ny) {
        const size_t o = ((size_t)s * Ny + py) * Nx + px;
        const float arg = acc[k] * sigma;
        float2 tv;
        sincosf(arg, &tv.y, &tv.x);
        if (isnan(tv.x)) tv.x = 1.f;
        if (isnan(tv.y)) tv.y = 1.f;
        trans[o] = tv;
        if (pot) pot[o] = acc[k];
      }
    }
  }
}

// ------------------------------------------------------------------ probe
// |k| on the centred grid, evaluated with the reference's operation order
// (calc_krad, probe_kernels.cu:11-16) and without FMA contraction, so that the
// float32 aperture and bandwidth decisions are reproducible on the host.
__device__ __forceinline__ double kaxis_exact(int j, int n, float kmax) {
  const double km = (double)kmax;
  return __dsub_rn(__ddiv_rn(__dmul_rn((double)j, km), (double)(n - 1)), __ddiv_rn(km, 2.0));
}
__device__ __forceinline__ double krad_of(double kx, double ky) {
  return __dsqrt_rn(__dadd_rn(__dmul_rn(kx, kx), __dmul_rn(ky, ky)));
}
__device__ __forceinline__ double krad_exact(int x, int y, int Nx, int Ny, float kmax) {
  return krad_of(kaxis_exact(x, Nx, kmax), kaxis_exact(y, Ny, kmax));
}

// k-space probe psi_k = A(k) exp(-i chi(k)) on the centred grid
// k = j*kmax/(N-1) - kmax/2 (probe_kernels.cu:11-16).  A is the smooth
// aperture 1/(1 + exp(-160 (k_semi - k))) (probe_kernels.cu:196-206, smoothing
// fixed at 80) or the hard one k < k_semi compared in float32
// (probe_kernels.cu:180-194); chi = 2 pi/lambda (-C1/2 (k lambda)^2 +
// C3/4 (k lambda)^4 + C5/6 (k lambda)^6) (probe_kernels.cu:208-222).  Evaluated
// in double, stored as complex64 like the reference's psi_k (msa.py:710-717).
//
// A thread takes kProbeRows rows of one column, so that the divisions of kx and
// ky are done once per thread.  Bound by double-precision instructions: 34 us at
// 512^2 with one pixel per thread, 30 us so.
constexpr int kProbeRows = 8;
__global__ void __launch_bounds__(128) probe_kernel(int Ny, int Nx, float kmax, double lambda, float k_semi, double C1,
                                                    double C3, double C5, int smooth, float2* __restrict__ psik,
                                                    float* __restrict__ aperture) {
  __shared__ double ky_s[kProbeRows];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y0 = blockIdx.y * kProbeRows;
  if (threadIdx.x < kProbeRows) ky_s[threadIdx.x] = kaxis_exact(y0 + threadIdx.x, Ny, kmax);
  __syncthreads();
  if (x >= Nx) return;
  const double kx = kaxis_exact(x, Nx, kmax);
  const bool finite = isfinite(C1 + C3 + C5);  // else every value is NaN
  for (int r = 0; r < kProbeRows && y0 + r < Ny; ++r) {
    const double k = krad_of(kx, ky_s[r]);
    const size_t o = (size_t)(y0 + r) * Nx + x;
    double a;
    bool zero;
    if (smooth) {
      // 1 / (1 + exp(u)): exactly 1 in double below u = -38, and 0 after rounding to
      // float32 above u = 104 (the smallest float32 is 1.4e-45), where the phase is
      // not needed: most of the grid.
      const double u = -160.0 * ((double)k_semi - k);
      zero = u > 104.0;
      a = zero ? 0.0 : u < -38.0 ? 1.0 : 1.0 / (1.0 + exp(u));
    } else {
      a = ((float)k < k_semi) ? 1.0 : 0.0;
      zero = a == 0.0;
    }
    if (zero && finite) {
      psik[o] = make_float2(0.f, 0.f);
    } else {
      const double kl = k * lambda, kl2 = kl * kl;
      const double chi = 2.0 * 3.14159265358979323846 / lambda * (-0.5 * C1 * kl2 + 0.25 * C3 * kl2 * kl2 + C5 / 6.0 * kl2 * kl2 * kl2);
      double sn, cs;
      sincos(chi, &sn, &cs);
      psik[o] = make_float2((float)(a * cs), (float)(-a * sn));
    }
    if (aperture) aperture[o] = (float)a;
  }
}

// normalisation = sum |fftshift(ifft2_u(psi_k))|^2 = N * sum |psi_k|^2 (Parseval),
// accumulated in double in a fixed order (msa.py:721-727) by one cluster of 16
// CTAs: strided partial sums per thread, a tree per CTA, and the CTAs' sums in
// rank order through distributed shared memory, which needs no scratch in
// global memory.  Bound by double-precision instructions (three a value on
// about two lanes a clock and SM): 512^2 368 us on one CTA, 28 us so.
constexpr int kNormCtas = 16, kNormThreads = 512;
__global__ void __launch_bounds__(kNormThreads) probe_norm_kernel(const float2* __restrict__ psik, long long n,
                                                                  double* __restrict__ out) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double red[kNormThreads];
  __shared__ double ranks[kNormCtas];
  const int rank = (int)cl.block_rank(), nr = (int)cl.num_blocks();
  cl.sync();  // every CTA runs before its shared memory is written
  double acc = 0;
  for (long long i = (long long)rank * kNormThreads + threadIdx.x; i < n; i += (long long)nr * kNormThreads) {
    const float2 v = psik[i];
    acc += (double)v.x * v.x + (double)v.y * v.y;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kNormThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *cl.map_shared_rank(&ranks[rank], 0) = red[0];
  cl.sync();  // rank 0's array is complete
  if (rank == 0 && threadIdx.x == 0) {
    double sum = 0;
    for (int r = 0; r < nr; ++r) sum += ranks[r];
    out[0] = sum * (double)n;
  }
}

// ------------------------------------------------------------------ propagator table
// P(k) * mask(k) / N with P = exp(-i pi lambda t k^2) (probe_kernels.cu:167-178)
// and mask = float(k) < float(bandwidth*kmax) (hard_aperture, msa.py:833-839).
// The phase is reduced in double (pi lambda t k^2 = 2 pi * f, f taken modulo 1).
__global__ void ptab_kernel(int Ny, int Nx, float kmax, double lambda, double slice_t, float k_band, float2* __restrict__ ptab) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= Nx) return;
  const double k = krad_exact(x, y, Nx, Ny, kmax);
  const double k2 = k * k;
  const float kf = (float)k;
  float2 v = make_float2(0.f, 0.f);
  if (kf < k_band) {
    double f = 0.5 * lambda * slice_t * k2;  // phase / (2 pi)
    f -= rint(f);
    float sn, cs;
    sincospif(2.0f * (float)f, &sn, &cs);
    const float inv_n = (float)(1.0 / ((double)Ny * (double)Nx));
    v = make_float2(cs * inv_n, -sn * inv_n);
  }
  ptab[(size_t)y * Nx + x] = v;
}

// Separable propagator factors for the persistent column pass:
// py[y] = exp(-i pi lambda t ky^2), px[x] = exp(-i pi lambda t kx^2) / N, and per
// column x the band [lo, hi] of rows whose float32 |k| passes the mask test
// (the same comparison as ptab_kernel).  |k| is monotone in |ky|, so the rows
// that pass form one interval.
__global__ void pfac_kernel(int Ny, int Nx, float kmax, double lambda, double slice_t, float k_band,
                            float2* __restrict__ pyx, int2* __restrict__ band) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const double km = (double)kmax;
  if (i < Ny) {
    const double ky = __dsub_rn(__ddiv_rn(__dmul_rn((double)i, km), (double)(Ny - 1)), __ddiv_rn(km, 2.0));
    double f = 0.5 * lambda * slice_t * ky * ky;
    f -= rint(f);
    float sn, cs;
    sincospif(2.0f * (float)f, &sn, &cs);
    pyx[i] = make_float2(cs, -sn);
  }
  if (i < Nx) {
    const double kx = __dsub_rn(__ddiv_rn(__dmul_rn((double)i, km), (double)(Nx - 1)), __ddiv_rn(km, 2.0));
    double f = 0.5 * lambda * slice_t * kx * kx;
    f -= rint(f);
    float sn, cs;
    sincospif(2.0f * (float)f, &sn, &cs);
    const float inv_n = (float)(1.0 / ((double)Ny * (double)Nx));
    pyx[Ny + i] = make_float2(cs * inv_n, -sn * inv_n);
  }
  // Band of column x, one warp per column.  ky rises with y and every step of the
  // float32 test is monotone in |ky|, so on each side of the centre the passing
  // rows are those nearest to it.  Half a warp per side tests sixteen rows around
  // the edge that |ky| = sqrt(k_band^2 - kx^2) gives; where that does not show the
  // edge, the half warp searches sixteen ways.  A test costs two double divisions
  // and a root: 19 us at 512^2 with a test of every row, 7 us with a 32-way search
  // from the centre, 6.7 us so.
  const int warp = i >> 5, lane = i & 31;
  if (warp < Nx) {
    const double kx = kaxis_exact(warp, Nx, kmax);
    const int side = lane >> 4, l = lane & 15;
    const int from = side ? Ny / 2 : (Ny - 1) / 2;  // the centre row of this side
    const int reach = side ? Ny - 1 - from : from;  // rows from + s, s = 0 .. reach, outwards
    auto pass = [&](int s) { return (float)krad_of(kx, kaxis_exact(side ? from + s : from - s, Ny, kmax)) < k_band; };
    auto count = [&](bool ok) {  // the passing lanes of this half come first
      return __popc((__ballot_sync(0xffffffffu, ok) >> (16 * side)) & 0xffffu);
    };
    int good = -1, bad = reach + 1;  // s = good passes (or -1), s = bad does not (or is past the end)
    const float rest = fmaxf(k_band * k_band - (float)(kx * kx), 0.f);
    const float edge = fminf(sqrtf(rest) * (float)(Ny - 1) / kmax, (float)reach);
    int base = max((int)edge - 8, 0);
    {
      const bool ok = base + l <= reach && pass(base + l);
      const int n = count(ok);
      if (n > 0) good = base + n - 1;
      if (n < 16) bad = min(bad, base + n);
      if (n == 0) bad = min(bad, base);
    }
    while (__any_sync(0xffffffffu, bad - good > 1)) {
      const int step = max((bad - good + 15) / 16, 1), s = good + 1 + l * step;
      const int n = count(s < bad && pass(s));
      bad = min(bad, good + 1 + n * step);
      if (n > 0) good = good + 1 + (n - 1) * step;
    }
    const int other = __shfl_xor_sync(0xffffffffu, good, 16);
    if (lane == 0) {
      const int lo = good >= 0 ? (Ny - 1) / 2 - good : Ny / 2, hi = other >= 0 ? Ny / 2 + other : (Ny - 1) / 2;
      band[warp] = good < 0 && other < 0 ? make_int2(1, 0) : make_int2(lo, hi);
    }
  }
}

__global__ void store_double_kernel(double* dst, double value) { *dst = value; }

cudaError_t launch_store_double(double* dst, double value, cudaStream_t st) {
  store_double_kernel<<<1, 1, 0, st>>>(dst, value);
  return cudaGetLastError();
}

cudaError_t launch_pfac(int Ny, int Nx, float kmax, double lambda, double slice_t, float k_band, float2* pyx,
                        int2* band, cudaStream_t st) {
  // 32 threads per column for the bands; that also covers the Ny + Nx factors
  const long long threads = 32LL * Nx > (long long)(Ny > Nx ? Ny : Nx) ? 32LL * Nx : (long long)(Ny > Nx ? Ny : Nx);
  pfac_kernel<<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(Ny, Nx, kmax, lambda, slice_t, k_band, pyx, band);
  return cudaGetLastError();
}

// Detector signals: out[p][d] = sum over column tiles of partial[p][tile][d],
// in tile order (deterministic).
__global__ void detect_reduce_kernel(const float* __restrict__ partial, int G, int tiles, int ndet,
                                     float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= G * ndet) return;
  const int p = i / ndet, d = i % ndet;
  float s = 0.f;
  for (int k = 0; k < tiles; ++k) s += partial[((size_t)p * tiles + k) * ndet + d];
  out[i] = s;
}

cudaError_t launch_detect_reduce(const float* partial, int G, int tiles, int ndet, float* out, cudaStream_t st) {
  const int n = G * ndet;
  detect_reduce_kernel<<<(n + 127) / 128, 128, 0, st>>>(partial, G, tiles, ndet, out);
  return cudaGetLastError();
}

cudaError_t launch_atom_windows(const double* coeff, int nspecies, int n0, int n1, int os, double range, float* out,
                                cudaStream_t st) {
  const int rows = os < kWinThreads / 2 ? os : kWinThreads / 2;  // threads per bin
  const int bins = kWinThreads / rows - 1;                       // a block's own bins; one slot is the corner
  const int quad = ((n0 / os + 1) / 2) * ((n1 / os + 1) / 2);
  const long long grid = (long long)nspecies * ((quad + bins - 1) / bins);
  if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  atom_window_kernel<<<(unsigned)grid, kWinThreads, 0, st>>>(coeff, n0, n1, os, rows, bins, range, out);
  return cudaGetLastError();
}

cudaError_t launch_potential(const int4* sites, const int* slice_off, int num_slices, const float* windows, int H, int W,
                             int Ny, int Nx, float sigma, float2* trans, float* pot, cudaStream_t st) {
  dim3 grid((Nx + kPotTile - 1) / kPotTile, (Ny + kPotTile - 1) / kPotTile, num_slices);
  potential_kernel<<<grid, kPotThreads, 0, st>>>(sites, slice_off, windows, H, W, Ny, Nx, sigma, trans, pot);
  return cudaGetLastError();
}

cudaError_t launch_probe(int Ny, int Nx, float kmax, double lambda, float k_semi, double C1, double C3, double C5,
                         int smooth, float2* psik, float* aperture, double* norm, cudaStream_t st) {
  dim3 grid((Nx + 127) / 128, (Ny + kProbeRows - 1) / kProbeRows);
  probe_kernel<<<grid, 128, 0, st>>>(Ny, Nx, kmax, lambda, k_semi, C1, C3, C5, smooth, psik, aperture);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || norm == nullptr) return e;
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kNormCtas);
  cfg.blockDim = dim3(kNormThreads);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kNormCtas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  // clusters of 16 are above the portable size: asked once per device; one CTA sums where
  // they are refused (part of a GPU)
  static std::mutex m;
  static std::map<int, FormState> form;
  bool cluster;
  {
    std::lock_guard<std::mutex> lock(m);
    cluster = form[dev].ready([&] {
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      cudaError_t r = cudaThreadExchangeStreamCaptureMode(&mode);
      if (r != cudaSuccess) return r;
      int n = 0;
      r = cudaFuncSetAttribute(probe_norm_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (r == cudaSuccess) r = cudaOccupancyMaxActiveClusters(&n, probe_norm_kernel, &cfg);
      cudaThreadExchangeStreamCaptureMode(&mode);
      return r == cudaSuccess && n < 1 ? cudaErrorInvalidConfiguration : r;
    });
  }
  if (!cluster) {
    cfg.gridDim = dim3(1);
    cfg.numAttrs = 0;
  }
  return cudaLaunchKernelEx(&cfg, probe_norm_kernel, psik, (long long)Ny * Nx, norm);
}

cudaError_t launch_ptab(int Ny, int Nx, float kmax, double lambda, double slice_t, float k_band, float2* ptab,
                        cudaStream_t st) {
  dim3 grid((Nx + 127) / 128, Ny);
  ptab_kernel<<<grid, 128, 0, st>>>(Ny, Nx, kmax, lambda, slice_t, k_band, ptab);
  return cudaGetLastError();
}

}  // namespace msx
