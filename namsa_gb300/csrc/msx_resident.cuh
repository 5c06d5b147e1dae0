// A wave held in the shared memory of a thread-block cluster through all slices.
//
// Calls with few positions on small grids are bound by latency: a slice costs two
// launches, each with its prologue, a load from L2 and a store.  Here a cluster of
// CTAs owns one wave.  In the row phase a CTA transforms its share of the rows
// (inverse FFT_x -> * t_i -> forward FFT_x) and sends every band column's values
// to the CTA that owns the column; in the column phase the owner does the same
// along y (forward FFT_y -> * P/N -> inverse FFT_y) and sends the rows back.  Only
// the transmission rows come from memory, a slice or two ahead.  The last column
// phase writes the pattern.
//
// The exchange is by blocks of (rows of one CTA) x (columns of another).  Both
// buffers are made of such blocks -- rows: one block per column owner, each [row]
// [own column]; columns: [y][own column], that is, one block per row owner -- and
// a phase leaves its results in place, so a block goes to its new owner with one
// bulk copy that counts itself off on the owner's mbarrier: no barrier over the
// cluster in the loop.  (64^2, us per slice: 8-byte remote stores and a cluster
// barrier per phase 3.4, 8-byte st.async counted one by one 2.9, blocks 2.6.)
// Nothing is overwritten early: a CTA receives block o of its rows only from CTA
// o and only after that has received the block sent from there, and it sends a
// column block only after its last read of those columns.
//
// Waits are bounded as in msx_tma.cuh.  When one runs out, bit 0 of *err is set, the CTA
// ends its phase on incomplete values, waits for the next phase's blocks (bounded, as
// ever) and stops there; the others then miss its blocks, time out and stop the
// same way.  So a CTA leaves only after a wait, complete or a second long, that
// followed every block sent to it, and after one for its own transmission rows: no
// copy is in flight when the shared memory is released.  The flag is read
// ahead of a wait, one word per kind of phase (a word is written in one phase and
// read in the next, on the other side of a barrier), which costs nothing measurable; a barrier
// with a reduction in either phase took 3 % of a slice at 256^2.
#pragma once
#include "msx_tma.cuh"

namespace msx {

template <int N_, int T_, int R1_, int R2_>
struct ResidentLine {
  static constexpr int N = N_, T = T_, R1 = R1_, R2 = R2_;
  using FFT = LineFFT<N_, T_, Radices<R1_, R2_>>;
  static constexpr int E = FFT::E;
  static constexpr int SH = swizzle_shift(R1_);
};

struct ResidentArgs {
  const float2* psi;      // (P, Ny, Nx) mixed waves of the probe formation (read once)
  const float2* trans;    // (slices, Ny, Nx), 16-byte aligned
  const float2* tw_row;
  const float2* tw_col;
  const float2* pyx;      // py[Ny] then px[Nx]
  const int2* band;
  const double* norm;
  float* cbed;            // (P, crop_y, crop_x)
  int* err;
  int slices;
  int tbufs;              // transmission buffers
  int x_lo, x_hi;         // band columns
  int x0, y0, crop_y, crop_x;
};

constexpr int kResidentThreads = 256;

// Shared-memory words (float2) of a CTA in a cluster of `cl`.
template <class LR, class LC>
struct Resident {
  static constexpr int NX = LR::N, NY = LC::N;
  static constexpr int RPR = kResidentThreads / LR::T;  // rows per round
  static constexpr int CPR = kResidentThreads / LC::T;  // columns per round
  static constexpr int TWRN = LR::FFT::tw_words(), TWCN = LC::FFT::tw_words();
  static constexpr int TWR = (TWRN + 15) / 16 * 16, TWC = (TWCN + 15) / 16 * 16;
  static __host__ __device__ int cols(int w, int cl) { return (w + cl - 1) / cl; }
  static __host__ __device__ size_t words(int w, int cl, int tbufs) {
    const int rows = NY / cl, live = rows < RPR ? rows : RPR;
    return (size_t)tbufs * rows * NX       // transmission rows (first: bulk-copied)
           + (size_t)live * NX             // exchange lines of a row round
           + 2 * (size_t)NY * cols(w, cl) + TWR + TWC + NY;  // the row blocks, the columns, tables
  }
  static __host__ size_t bytes(int w, int cl, int tbufs) { return sizeof(float2) * words(w, cl, tbufs) + 64; }  // + barriers, flags
  // two transmission buffers where they fit
  static __host__ int tbufs(int w, int cl) { return bytes(w, cl, 2) <= 232448 ? 2 : 1; }
  static __host__ size_t smem(int w, int cl) { return bytes(w, cl, tbufs(w, cl)); }
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// shared-memory address of another CTA of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// bulk copy of shared memory into a CTA of the cluster, counted on a barrier of that CTA
__device__ __forceinline__ void bulk_s2s(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
        "p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > (1LL << 31)) return false;
  }
}

template <class LR, class LC>
__global__ void __launch_bounds__(kResidentThreads, 1) resident_kernel(const ResidentArgs a) {
  using K = Resident<LR, LC>;
  constexpr int NX = K::NX, NY = K::NY;
  extern __shared__ __align__(1024) float2 smem[];
  const int rank = (int)cluster_rank(), cl = (int)cluster_size();
  const int wave = blockIdx.x / cl;
  const int rows = NY / cl, W = a.x_hi - a.x_lo, wc = K::cols(W, cl);
  const int live = rows < K::RPR ? rows : K::RPR;
  float2* const tbuf = smem;
  float2* const lines = tbuf + a.tbufs * rows * NX;
  const int block = rows * wc;              // words of a block, a multiple of 4
  float2* const rbuf = lines + live * NX;   // [column owner][row][own column]
  float2* const cbuf = rbuf + NY * wc;      // [y][own column]
  float2* const twr = cbuf + NY * wc;
  float2* const twc = twr + K::TWR;
  float2* const py = twc + K::TWC;
  uint64_t* const tfull = reinterpret_cast<uint64_t*>(py + NY);  // one per transmission buffer
  uint64_t* const rfull = tfull + 2;
  uint64_t* const cfull = tfull + 3;
  volatile int* const failed = reinterpret_cast<volatile int*>(tfull + 4);  // a wait ran out: in a row phase, in a column phase
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int mycols = min(wc, max(0, W - rank * wc));
  const uint32_t tbytes = (uint32_t)(rows * NX * sizeof(float2));
  const uint32_t bbytes = (uint32_t)(block * sizeof(float2)), phase_bytes = bbytes * cl;  // every block of a phase
  auto fetch = [&](int s) {  // thread 0: this CTA's transmission rows of slice s
    const int b = s % a.tbufs;
    mbar_expect_tx(&tfull[b], tbytes);
    bulk_g2s(tbuf + b * rows * NX, a.trans + ((size_t)s * NY + (size_t)rank * rows) * NX, tbytes, &tfull[b]);
  };
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(&tfull[i], 1);
    failed[0] = failed[1] = 0;
    fence_mbar_init();
    for (int s = 0; s < a.tbufs && s < a.slices; ++s) fetch(s);
  }
  for (int i = tid; i < K::TWRN; i += blockDim.x) twr[i] = a.tw_row[i];
  for (int i = tid; i < K::TWCN; i += blockDim.x) twc[i] = a.tw_col[i];
  for (int i = tid; i < NY; i += blockDim.x) py[i] = a.pyx[i];
  // pattern columns outside the band, rows shared among the CTAs
  float* const out = a.cbed + (size_t)wave * a.crop_y * a.crop_x;
  for (int i = rank * blockDim.x + tid; i < a.crop_y * a.crop_x; i += cl * blockDim.x) {
    const int x = a.x0 + i % a.crop_x;
    if (x < a.x_lo || x >= a.x_hi) out[i] = 0.f;
  }
  cluster_sync_all();  // every CTA runs before its shared memory is written; tables and barriers are set
  const uint32_t rbuf_s = smem_u32(rbuf), cbuf_s = smem_u32(cbuf);
  const uint32_t rfull_s = smem_u32(rfull), cfull_s = smem_u32(cfull);
  // v / wc == (v winv) >> 16: winv = 65536 / wc + e with e <= (wc - 1) / wc, so the product is off by less
  // than the 65536 / wc to the next quotient while v (wc - 1) < 65536 (clusters have at least 4 CTAs)
  static_assert((NX - 1) * (NX / 4 - 1) < 65536, "the quotient by multiplication");
  const uint32_t winv = (65536u + wc - 1) / wc;
  int stopped = -1;  // the slice in which the CTA stopped

  for (int s = 0; s < a.slices; ++s) {
    // ------------------------------------------------------------------ row phase
    const int tb = s % a.tbufs;
    const float2* const trow = tbuf + tb * rows * NX;
    const int failed_before = failed[1];
    bool ok = mbar_wait_bounded(&tfull[tb], (uint32_t)((s / a.tbufs) & 1));
    if (s > 0) {
      if (tid == 0) mbar_expect_tx(rfull, phase_bytes);  // the values may have been arriving before
      ok = wait_cluster(rfull, (uint32_t)((s - 1) & 1)) && ok;
    }
    if (!__all_sync(0xffffffffu, ok) && lane == 0) {
      failed[0] = 1;
      atomicOr(a.err, 1);
    }
    if (failed_before) {  // the same for every thread
      stopped = s;
      break;
    }
    {
      constexpr int T = LR::T, E = LR::E;
      const int lw = lane / T, tt = lane % T;
      const int slot = warp * (32 / T) + lw;
      for (int r0 = 0; r0 < rows; r0 += K::RPR) {
        // rows is a multiple of a warp's 32 / T rows (4 or more): whole warps take part or not
        const int r = r0 + slot;
        if (r < rows) {
          const SwizzledLine<LR::SH> line{lines + slot * NX, T == 8 ? (lw & 1) * 8 : 0};
          float2 v[E], o[E];
          if (s == 0) {
            const float2* src = a.psi + ((size_t)wave * NY + rank * rows + r) * NX;
#pragma unroll
            for (int m = 0; m < E; ++m) v[m] = __ldg(src + tt + T * m);
          } else {
#pragma unroll
            for (int m = 0; m < E; ++m) {
              const int x = tt + T * m - a.x_lo;
              const int owner = (int)(((uint32_t)x * winv) >> 16);
              v[m] = x >= 0 && x < W ? rbuf[owner * block + r * wc + x - owner * wc] : make_float2(0.f, 0.f);
            }
          }
          LR::FFT::template butterflies<LR::R1, 1, 0, true>(v, o, twr, tt);
          __syncwarp();
          LR::FFT::template scatter<LR::R1, 1>(o, line, tt);
          __syncwarp();
          LR::FFT::gather(v, line, tt);
          LR::FFT::template butterflies<LR::R2, LR::R1, 0, true>(v, o, twr, tt);
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = cmul(o[m], trow[r * NX + tt + T * m]);
          LR::FFT::template butterflies<LR::R1, 1, 0, false>(v, o, twr, tt);
          __syncwarp();
          LR::FFT::template scatter<LR::R1, 1>(o, line, tt);
          __syncwarp();
          LR::FFT::gather(v, line, tt);
          LR::FFT::template butterflies<LR::R2, LR::R1, 0, false>(v, o, twr, tt);
#pragma unroll
          for (int m = 0; m < E; ++m) {  // in place: the words that this thread has read
            const int x = tt + T * m - a.x_lo;
            const int owner = (int)(((uint32_t)x * winv) >> 16);
            if (x >= 0 && x < W) rbuf[owner * block + r * wc + x - owner * wc] = o[m];
          }
        }
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (tid < cl)
      bulk_s2s(map_rank(cbuf_s + rank * bbytes, (uint32_t)tid), rbuf_s + tid * bbytes, bbytes, map_rank(cfull_s, (uint32_t)tid));
    // --------------------------------------------------------------- column phase
    const int failed_rows = failed[0];
    if (tid == 0) mbar_expect_tx(cfull, phase_bytes);
    if (!__all_sync(0xffffffffu, wait_cluster(cfull, (uint32_t)(s & 1)) ? 1 : 0) && lane == 0) {
      failed[1] = 1;
      atomicOr(a.err, 1);
    }
    if (failed_rows) {
      stopped = s;
      break;
    }
    {
      constexpr int T = LC::T, E = LC::E, C = K::CPR;
      const bool last = s + 1 == a.slices;
      const int c = tid % C, tt = tid / C;
      for (int c0 = 0; c0 < wc; c0 += C) {
        const bool active = c0 + c < mycols;
        const int cc = active ? c0 + c : 0;  // idle threads keep to the barriers
        const int x = a.x_lo + rank * wc + cc;
        float2 v[E], o[E];
        int2 bd = make_int2(1, 0);
        float2* const col = cbuf + cc;
        if (active) {
          bd = __ldg(a.band + x);
#pragma unroll
          for (int m = 0; m < E; ++m) v[m] = col[(tt + T * m) * wc];
          LC::FFT::template butterflies<LC::R1, 1, 0, false>(v, o, twc, tt);
        }
        struct Line {
          float2* base;
          int wc;
          __device__ __forceinline__ float2& operator[](int i) const { return base[i * wc]; }
        };
        const Line line{col, wc};
        __syncthreads();
        if (tid == 0 && c0 == 0 && s + a.tbufs < a.slices) {  // every row has read its transmission values
          fence_proxy_async();
          fetch(s + a.tbufs);
        }
        if (active) LC::FFT::template scatter<LC::R1, 1>(o, line, tt);
        __syncthreads();
        if (active) {
          LC::FFT::gather(v, line, tt);
          LC::FFT::template butterflies<LC::R2, LC::R1, 0, false>(v, o, twc, tt);
        }
        if (last) {
          if (active && x >= a.x0 && x < a.x0 + a.crop_x) {
            const float inv_n = (float)(1.0 / ((double)NY * (double)NX));
            const float scale = (float)((double)NY * (double)NX / *a.norm);
#pragma unroll
            for (int m = 0; m < E; ++m) {
              const int ky = tt + T * m;
              const float2 f = cscale(o[m], ky >= bd.x && ky <= bd.y ? inv_n : 0.f);
              const int yo = ky - a.y0;
              if (yo >= 0 && yo < a.crop_y) out[(size_t)yo * a.crop_x + x - a.x0] = fmaf(f.x, f.x, f.y * f.y) * scale;
            }
          }
          continue;
        }
        if (active) {
          const float2 px = __ldg(a.pyx + NY + x);
#pragma unroll
          for (int m = 0; m < E; ++m) {
            const int ky = tt + T * m;
            v[m] = cmul(o[m], ky >= bd.x && ky <= bd.y ? cmul(px, py[ky]) : make_float2(0.f, 0.f));
          }
          LC::FFT::template butterflies<LC::R1, 1, 0, true>(v, o, twc, tt);
        }
        __syncthreads();
        if (active) LC::FFT::template scatter<LC::R1, 1>(o, line, tt);
        __syncthreads();
        if (active) {
          LC::FFT::gather(v, line, tt);
          LC::FFT::template butterflies<LC::R2, LC::R1, 0, true>(v, o, twc, tt);
#pragma unroll
          for (int m = 0; m < E; ++m) line[tt + T * m] = o[m];  // the words that this thread has read
        }
      }
      if (!last) {
        fence_proxy_async();
        __syncthreads();
        if (tid < cl)
          bulk_s2s(map_rank(rbuf_s + rank * bbytes, (uint32_t)tid), cbuf_s + tid * bbytes, bbytes,
                   map_rank(rfull_s, (uint32_t)tid));
      }
    }
  }
  if (stopped >= 0 && tid == 0)  // rows asked for: those of the slices before stopped + tbufs
    for (int s = stopped; s < stopped + a.tbufs && s < a.slices; ++s)
      mbar_wait_bounded(&tfull[s % a.tbufs], (uint32_t)((s / a.tbufs) & 1));
  cluster_sync_all();  // no CTA leaves while another may still write to it
}

struct ResidentOps {
  int twr_words, twc_words;
  void (*tw_row)(float2*);
  void (*tw_col)(float2*);
  cudaError_t (*configure)();
  // no more clusters of `cl` CTAs than this run at the same time, by shared memory and threads alone
  int (*most)(int w, int cl, int sms);
  // clusters of `cl` CTAs that run at the same time with `w` band columns (0: does not fit)
  cudaError_t (*clusters)(int w, int cl, int* n);
  cudaError_t (*launch)(ResidentArgs a, int waves, int cl, cudaStream_t st);
};
const ResidentOps* resident_ops(int ny, int nx);

}  // namespace msx
