// All slices of a group of waves in one persistent kernel.
//
// The separate row and column passes (msx_tma.cuh) cost two launches per
// slice, each with a last wave of tiles that leaves SMs idle, and between them
// every wave crosses HBM.  Here one kernel runs the row and column tiles of
// every slice of a group small enough to stay in L2: a tile starts as soon as
// the tiles that it reads from are done, so tiles of one chunk of waves fill
// the SMs while another chunk's last tiles finish.
//
// Tasks.  A chunk is `wpt` consecutive waves.  Per slice, in this order:
//   row tiles     (chunk, y block): wpt waves x ypt rows, wpt * ypt = L lines:
//                 inverse FFT_x -> * t_i -> forward FFT_x;
//   column tiles  (wave, column tile): C columns x Ny rows:
//                 forward FFT_y -> * P/N -> inverse FFT_y.
// CTA b takes tasks b, b + grid, b + 2 grid, ...  A row tile of slice i > 0
// waits for all column tiles of its chunk of slice i - 1, a column tile for all
// row tiles of its chunk of slice i; both precede it in the task order.  The
// launch is cooperative (every CTA resident) and each CTA finishes its tasks in
// order, so the first unfinished task of the order can always run: no deadlock.
//
// Roles.  CT compute threads, a loader warp and a publisher warp.  The loader
// (one lane) waits for a stage and for the tile's dependency (a counter per
// chunk, acquire at gpu scope, then a proxy fence: the data were written by
// other CTAs and are read by bulk copies) and issues the copies, up to NS - 1
// tiles ahead of the compute warps.  The publisher (one lane) waits until the
// compute warps are done with a tile, writes a column tile back by a tiled bulk
// store and waits for it, and then adds 1 to the chunk's counter (release at
// gpu scope).  Blocking is safe in both: neither holds up a tile in front of
// the one it waits for.
//
// Band limit as in msx_tma.cuh: from slice `first` on only columns
// [x_lo, x_hi) of a row are copied and written; the rest of a row counts as
// zero.  Slice 0 of a group reads whole rows (an aperture may reach beyond the
// band).  Columns outside the band are never written again.
//
// Waits are bounded as in msx_tma.cuh (about one second each): on a timeout a
// role sets bit 0 of *err and stops, the others then time out in turn, and the
// loader waits (bounded) for its copies in flight before the CTA exits.
#pragma once
#include <type_traits>

#include "msx_tma.cuh"

namespace msx {

// Tasks of one launch, the same arithmetic on host and device.
struct StreamShape {
  int G, wpt, ypt;       // waves, waves and rows per row tile
  int Ny, tiles_x;       // rows, column tiles of a wave
  int slices;            // slices of this launch
  int last_col;          // 1: the last slice has its column pass too
  __host__ __device__ int chunks() const { return (G + wpt - 1) / wpt; }
  __host__ __device__ int row_tiles() const { return Ny / ypt; }  // per chunk
  __host__ __device__ int per_slice() const { return chunks() * row_tiles() + G * tiles_x; }
  __host__ __device__ long long tasks() const {
    return (long long)slices * per_slice() - (last_col ? 0 : (long long)G * tiles_x);
  }
  __host__ __device__ int chunk_waves(int c) const { return G - c * wpt < wpt ? G - c * wpt : wpt; }
};
struct StreamTask {
  int slice, chunk;
  bool row;
  int a, b;              // row: first row, -; column: wave, column tile
  int need;              // value of the awaited counter (0: none)
};
__host__ __device__ __forceinline__ StreamTask stream_task(const StreamShape& sh, long long u) {
  StreamTask t;
  const int per = sh.per_slice(), rt = sh.row_tiles(), rows = sh.chunks() * rt;
  t.slice = (int)(u / per);
  const int r = (int)(u - (long long)t.slice * per);
  t.row = r < rows;
  if (t.row) {
    t.chunk = r / rt;
    t.a = (r - t.chunk * rt) * sh.ypt;
    t.b = 0;
    t.need = t.slice * sh.chunk_waves(t.chunk) * sh.tiles_x;  // column tiles of the chunk, slices before
  } else {
    const int q = r - rows;
    t.a = q / sh.tiles_x;
    t.b = q - t.a * sh.tiles_x;
    t.chunk = t.a / sh.wpt;
    t.need = (t.slice + 1) * rt;  // row tiles of the chunk, this slice included
  }
  return t;
}

__host__ __device__ __forceinline__ int4 task_desc(const StreamShape& sh, long long u) {
  const StreamTask t = stream_task(sh, u);
  return make_int4((t.row ? 1 : 0) | (t.slice << 1), t.chunk, t.a, t.b);
}

struct StreamArgs {
  float2* psi;            // (G, Ny, Nx) workspace
  const float2* trans;    // (slices, Ny, Nx)
  const float2* tw_row;
  const float2* tw_col;
  const float2* pyx;      // py[Ny] then px[Nx]
  const int2* band;
  int* counters;          // row tiles done [chunks], column tiles done [chunks], zero at launch
  int* err;
  int first;              // 1: slice 0 of the launch reads whole rows
  int x_lo, x_hi;         // multiples of the column tile
  StreamShape sh;
};

// whether the barrier's phase of this parity is complete, without waiting
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// orders earlier generic-proxy accesses (also those acquired from other threads) before later bulk copies
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Exchange positions of a column in a tile of C interleaved columns.
template <int C>
struct StreamColumn {
  float2* base;
  __device__ __forceinline__ float2& operator[](int i) const { return base[i * C]; }
};

// One two-stage line schedule of the persistent kernel.
template <int N_, int T_, int R1_, int R2_>
struct StreamLineSched {
  static constexpr int N = N_, T = T_, R1 = R1_, R2 = R2_;
  using FFT = LineFFT<N_, T_, Radices<R1_, R2_>>;
  static constexpr int E = FFT::E;
  static constexpr int SH = swizzle_shift(R1_);  // of the exchange through staged rows
};

// CT compute threads and a warpgroup of helpers, which hand their registers to the
// compute warps (setmaxnreg): one CTA per SM (256 + 128) x 168 = 256 x 232 + 128 x 40,
// two CTAs per SM (256 + 128) x 80 = 256 x 104 + 128 x 32 (at most).
template <class LR, class LC, int MINB_>
struct Stream {
  static_assert(MINB_ == 1 || MINB_ == 2, "the register split is made for one or two CTAs per SM");
  static constexpr int CT = 256, WARPS = CT / 32, THREADS = CT + 128, MINB = MINB_;
  static constexpr size_t LIMIT = MINB == 2 ? 115712 : 232448;  // shared memory of a CTA
  static constexpr int NX = LR::N, NY = LC::N;
  static constexpr int L = CT / LR::T;              // lines per row tile
  static constexpr int C = CT / LC::T;              // columns per column tile
  static constexpr int BOXR = NY < 128 ? NY : 128, NBOX = NY / BOXR;
  static constexpr int COL_WORDS = C * NY;
  static constexpr int TWR = LR::FFT::tw_words(), TWC = LC::FFT::tw_words();
  static constexpr bool SHARE = std::is_same_v<LR, LC>;
  static constexpr int TW = (TWR + (SHARE ? 0 : TWC) + 15) / 16 * 16;
  // L rows and the transmission rows of a tile of wpt waves, or a column tile
  static constexpr int stage_words(int wpt) {
    return (((L + L / wpt) * NX > COL_WORDS ? (L + L / wpt) * NX : COL_WORDS) + 15) / 16 * 16;
  }
  static constexpr size_t bytes(int ns, int wpt) {
    return sizeof(float2) * ((size_t)ns * stage_words(wpt) + TW) + ns * (sizeof(int4) + 3 * sizeof(uint64_t));
  }
  // As few waves per row tile as two stages hold the transmission rows for: small
  // chunks keep more of them apart when there are few waves, and full lines in
  // the tiles of the last chunk.
  static constexpr int WPT = bytes(2, 2) <= LIMIT ? 2 : bytes(2, 4) <= LIMIT ? 4 : 8;
  static constexpr int YPT = L / WPT;               // rows per row tile
  static constexpr int STAGE = stage_words(WPT);
  static constexpr int NS = bytes(3, WPT) <= LIMIT ? 3 : 2;
  static_assert(L % WPT == 0 && bytes(NS, WPT) <= LIMIT, "stages do not fit");
  static constexpr size_t smem() { return bytes(NS, WPT); }
};

template <class K>
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(K::CT) : "memory"); }
// the same barrier; true on all compute threads iff `ok` on all of them
template <class K>
__device__ __forceinline__ bool compute_all(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)ok), "n"(K::CT)
      : "memory");
  return r != 0;
}

template <class LR, class LC, int MINB>
__global__ void __launch_bounds__(384, MINB) stream_kernel(const __grid_constant__ CUtensorMap map, const StreamArgs a) {
  using K = Stream<LR, LC, MINB>;
  constexpr int NX = K::NX, NY = K::NY, NS = K::NS, STAGE = K::STAGE, L = K::L, C = K::C;
  extern __shared__ __align__(1024) float2 smem[];
  float2* const stage = smem;
  float2* const twr = smem + NS * STAGE;
  float2* const twc = K::SHARE ? twr : twr + K::TWR;
  int4* const desc = reinterpret_cast<int4*>(twr + K::TW);  // the stage's task: row tile | 2 slice, chunk, a, b
  uint64_t* const full = reinterpret_cast<uint64_t*>(desc + NS);
  uint64_t* const done = full + NS;    // compute warps are finished with the tile
  uint64_t* const empty = done + NS;   // ... and the publisher has stored and released it
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < K::TWR; i += blockDim.x) twr[i] = a.tw_row[i];
  if constexpr (!K::SHARE)
    for (int i = tid; i < K::TWC; i += blockDim.x) twc[i] = a.tw_col[i];
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&done[s], K::WARPS);
      mbar_init(&empty[s], 1);
    }
    fence_mbar_init();
  }
  __syncthreads();
  const StreamShape sh = a.sh;
  const long long tasks = sh.tasks();
  const int grid = gridDim.x;
  const long long mine = blockIdx.x < tasks ? (tasks - 1 - blockIdx.x) / grid + 1 : 0;
  const int chunks = sh.chunks();
  int* const row_done = a.counters;
  int* const col_done = a.counters + chunks;

  if (warp >= K::WARPS) {
    if constexpr (MINB == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == K::WARPS) {  // --------------------------------------------------- loader
      long long issued = 0;
      for (; issued < mine; ++issued) {
        const int s = (int)(issued % NS);
        const StreamTask t = stream_task(sh, blockIdx.x + issued * grid);
        int ok = 1;
        if (lane == 0) {
          if (issued >= NS) ok = mbar_wait_bounded(&empty[s], (uint32_t)(((issued / NS) - 1) & 1)) ? 1 : 0;
          if (ok && t.need > 0) {
            const int* ctr = (t.row ? col_done : row_done) + t.chunk;
            const long long t0 = clock64();
            while (ld_acquire(ctr) < t.need && ok) ok = clock64() - t0 < (1LL << 31) ? 1 : 0;
          }
          if (!ok) atomicOr(a.err, 1);
        }
        if (!__shfl_sync(0xffffffffu, ok, 0)) break;
        __syncwarp();             // lane 0's acquire before what follows in the other lanes (a shuffle orders nothing)
        fence_proxy_async_all();  // in every lane that issues copies: the awaited data before its own copies
        float2* const dst = stage + s * STAGE;
        if (t.row) {
          const bool whole = a.first && t.slice == 0;
          const int x0 = whole ? 0 : a.x_lo, nx = (whole ? NX : a.x_hi) - x0;
          const int lines = sh.chunk_waves(t.chunk) * K::YPT;
          if (lane == 0) {
            desc[s] = make_int4(1 | (t.slice << 1), t.chunk, t.a, t.b);  // published by the arrival on full[s]
            mbar_expect_tx(&full[s], (uint32_t)((lines * nx + K::YPT * NX) * sizeof(float2)));
            bulk_g2s(dst + L * NX, a.trans + ((size_t)t.slice * NY + t.a) * NX, (uint32_t)(K::YPT * NX * sizeof(float2)),
                     &full[s]);
          }
          __syncwarp();
          for (int j = lane; j < lines; j += 32)
            bulk_g2s(dst + j * NX + x0, a.psi + ((size_t)(t.chunk * K::WPT + j / K::YPT) * NY + t.a + j % K::YPT) * NX + x0,
                     (uint32_t)(nx * sizeof(float2)), &full[s]);
        } else if (lane == 0) {
          desc[s] = make_int4(t.slice << 1, t.chunk, t.a, t.b);
          mbar_expect_tx(&full[s], (uint32_t)(K::COL_WORDS * sizeof(float2)));
#pragma unroll
          for (int b = 0; b < K::NBOX; ++b)
            tma2d_g2s(dst + b * K::BOXR * C, &map, a.x_lo + t.b * C, t.a * NY + b * K::BOXR, &full[s]);
        }
      }
      // copies in flight land before the CTA's shared memory is released
      for (long long j = issued > NS ? issued - NS : 0; j < issued; ++j)
        mbar_wait_bounded(&full[j % NS], (uint32_t)((j / NS) & 1));
    } else if (warp == K::WARPS + 1 && lane == 0) {  // ------------------------------ publisher
      // A column tile's store is left in flight while the next tile is awaited, but
      // only if that one is ready: nothing here waits with a finished tile unpublished.
      int pending = -1;  // chunk of the column tile whose store is in flight
      auto publish = [&](int* ctr) {
        fence_proxy_async_all();
        add_release(ctr, 1);
      };
      for (long long k = 0; k < mine; ++k) {
        const int s = (int)(k % NS);
        const uint32_t par = (uint32_t)((k / NS) & 1);
        if (pending >= 0 && !mbar_test(&done[s], par)) {
          bulk_wait_all();
          publish(col_done + pending);
          pending = -1;
        }
        if (!mbar_wait_bounded(&done[s], par)) {
          atomicOr(a.err, 1);
          break;
        }
        const int4 t = desc[s];
        if (t.x & 1) {
          mbar_arrive(&empty[s]);
          publish(row_done + t.y);
        } else {
          const float2* src = stage + s * STAGE;
#pragma unroll
          for (int b = 0; b < K::NBOX; ++b)
            tma2d_s2g(&map, a.x_lo + t.w * C, t.z * NY + b * K::BOXR, src + b * K::BOXR * C);
          bulk_commit();
        }
        if (pending >= 0) {
          if (t.x & 1) bulk_wait_all();
          else asm volatile("cp.async.bulk.wait_group 1;" ::: "memory");  // all but the store just issued
          publish(col_done + pending);
          pending = -1;
        }
        if (!(t.x & 1)) {
          bulk_wait_read_all();
          mbar_arrive(&empty[s]);
          pending = t.y;
        }
      }
      bulk_wait_all();
      if (pending >= 0) publish(col_done + pending);
    }
  } else {  // ---------------------------------------------------------------- compute
    if constexpr (MINB == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    // A warp whose wait ran out (`dead`) does no more work but still takes part in
    // the first barrier of a column tile, where all compute warps leave together.
    bool dead = false;
    for (long long k = 0; k < mine; ++k) {
      const int s = (int)(k % NS);
      float2* const st = stage + s * STAGE;
      if (!dead && !__all_sync(0xffffffffu, mbar_wait_bounded(&full[s], (uint32_t)((k / NS) & 1)) ? 1 : 0)) {
        dead = true;
        if (lane == 0) atomicOr(a.err, 1);
      }
      const int4 t = dead ? task_desc(sh, blockIdx.x + k * grid) : desc[s];
      if (t.x & 1) {
        if (dead) continue;
        constexpr int T = LR::T, E = LR::E;
        const int lw = lane / T, tt = lane % T;
        const int slot = warp * (32 / T) + lw;
        const bool whole = a.first && t.x == 1;
        const int xr0 = whole ? 0 : a.x_lo, xr1 = whole ? NX : a.x_hi;
        const SwizzledLine<LR::SH> line{st + slot * NX, T == 8 ? (lw & 1) * 8 : 0};
        const float2* trow = st + (L + slot % K::YPT) * NX;
        float2 v[E], out[E];
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int x = tt + T * m;
          v[m] = x >= xr0 && x < xr1 ? line.base[x] : make_float2(0.f, 0.f);
        }
        LR::FFT::template butterflies<LR::R1, 1, 0, true>(v, out, twr, tt);
        __syncwarp();
        LR::FFT::template scatter<LR::R1, 1>(out, line, tt);
        __syncwarp();
        LR::FFT::gather(v, line, tt);
        LR::FFT::template butterflies<LR::R2, LR::R1, 0, true>(v, out, twr, tt);
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = cmul(out[m], trow[tt + T * m]);
        LR::FFT::template butterflies<LR::R1, 1, 0, false>(v, out, twr, tt);
        __syncwarp();
        LR::FFT::template scatter<LR::R1, 1>(out, line, tt);
        __syncwarp();
        LR::FFT::gather(v, line, tt);
        LR::FFT::template butterflies<LR::R2, LR::R1, 0, false>(v, out, twr, tt);
        const int wave = t.y * K::WPT + slot / K::YPT;
        if (wave < sh.G) {
          float2* o = a.psi + ((size_t)wave * NY + t.z + slot % K::YPT) * NX;
#pragma unroll
          for (int m = 0; m < E; ++m) {
            const int x = tt + T * m;
            if (x >= a.x_lo && x < a.x_hi) o[x] = out[m];
          }
        }
      } else {
        constexpr int T = LC::T, E = LC::E;
        const int c = tid % C, tt = tid / C;
        const int x = a.x_lo + t.w * C + c;
        const float2 px = __ldg(a.pyx + NY + x);
        const int2 bd = __ldg(a.band + x);
        static_assert(C >= 16, "a half warp stays within a row: no two of its accesses share a bank");
        const StreamColumn<C> in{st + c};
        float2 v[E], out[E];
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = st[(tt + T * m) * C + c];
        LC::FFT::template butterflies<LC::R1, 1, 0, false>(v, out, twc, tt);
        if (!compute_all<K>(!dead)) break;
        LC::FFT::template scatter<LC::R1, 1>(out, in, tt);
        compute_sync<K>();
        LC::FFT::gather(v, in, tt);
        LC::FFT::template butterflies<LC::R2, LC::R1, 0, false>(v, out, twc, tt);
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const int ky = tt + T * m;
          const float2 f = ky >= bd.x && ky <= bd.y ? cmul(px, __ldg(a.pyx + ky)) : make_float2(0.f, 0.f);
          v[m] = cmul(out[m], f);
        }
        LC::FFT::template butterflies<LC::R1, 1, 0, true>(v, out, twc, tt);
        compute_sync<K>();
        LC::FFT::template scatter<LC::R1, 1>(out, in, tt);
        compute_sync<K>();
        LC::FFT::gather(v, in, tt);
        LC::FFT::template butterflies<LC::R2, LC::R1, 0, true>(v, out, twc, tt);
        // at the words of this warp's last gather: nobody else reads them any more
#pragma unroll
        for (int m = 0; m < E; ++m) st[(tt + T * m) * C + c] = out[m];
      }
      fence_proxy_async();  // shared-memory accesses before the next bulk copy into (or out of) the stage
      __syncwarp();
      if (lane == 0) mbar_arrive(&done[s]);
    }
  }
}

// Lines of 256 hold 16 values per thread, so that two CTAs fit an SM and hide each
// other's waits: 0.31 us per wave and slice at 64 waves of 256^2 against 0.36 with
// one CTA.  With few waves the CTAs run out of tiles and one is faster (0.40
// against 0.45 at 32 waves, 0.63 against 0.75 at 16), so 256^2 has both.
constexpr int kStreamWaves2 = 48;  // from this many waves on

// Launchers of one (ny, nx) instance.
struct StreamOps {
  int col_c, col_boxr;     // columns per tile, rows per tensor-map box
  int wpt, ypt;            // waves and rows per row tile
  int twr_words, twc_words;
  void (*tw_row)(float2*);
  void (*tw_col)(float2*);
  cudaError_t (*configure)();
  cudaError_t (*launch)(const CUtensorMap& map, const StreamArgs& a, int sms, cudaStream_t st);
};

template <class LR, class LC, int MINB>
struct StreamImpl {
  using K = Stream<LR, LC, MINB>;
  static cudaError_t configure() {
    if constexpr (LR::N == 256 && LC::N == 256 && MINB == 1) {
      // the same tiles, so that a launch may take either
      using K2 = Stream<LR, LC, 2>;
      static_assert(K2::WPT == K::WPT && K2::YPT == K::YPT && K2::C == K::C);
      const cudaError_t e = StreamImpl<LR, LC, 2>::configure();
      if (e != cudaSuccess) return e;
    }
    // the registers the roles take must be there at launch, or setmaxnreg waits for good
    cudaFuncAttributes fa{};
    cudaError_t e = cudaFuncGetAttributes(&fa, stream_kernel<LR, LC, MINB>);
    if (e != cudaSuccess) return e;
    if (fa.numRegs * K::THREADS < (MINB == 2 ? 256 * 104 + 128 * 32 : 256 * 232 + 128 * 40)) return cudaErrorInvalidConfiguration;
    e = cudaFuncSetAttribute(stream_kernel<LR, LC, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem());
    if (e != cudaSuccess) return e;
    // every CTA of a launch resident, MINB to an SM
    int dev = 0, cooperative = 0, ctas = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, stream_kernel<LR, LC, MINB>, K::THREADS, K::smem());
    return e == cudaSuccess && (!cooperative || ctas < MINB) ? cudaErrorInvalidConfiguration : e;
  }
  static cudaError_t launch(const CUtensorMap& map, const StreamArgs& a, int sms, cudaStream_t st) {
    const long long tasks = a.sh.tasks();
    if (tasks <= 0) return cudaSuccess;
    cudaLaunchConfig_t cfg{};
    if constexpr (LR::N == 256 && LC::N == 256 && MINB == 1)
      if (a.sh.G >= kStreamWaves2) return StreamImpl<LR, LC, 2>::launch(map, a, sms, st);
    const long long most = (long long)sms * K::MINB;
    cfg.gridDim = dim3((unsigned)(tasks < most ? tasks : most));
    cfg.blockDim = dim3(K::THREADS);
    cfg.dynamicSmemBytes = K::smem();
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;  // CTAs wait for one another: all of them resident, or an error
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, stream_kernel<LR, LC, MINB>, map, a);
  }
  static StreamOps ops() {
    return StreamOps{K::C, K::BOXR, K::WPT, K::YPT, K::TWR, K::TWC, &LR::FFT::host_twiddles, &LC::FFT::host_twiddles,
                     &configure, &launch};
  }
};

using StreamLine256 = StreamLineSched<256, 16, 16, 16>;
using StreamLine384 = StreamLineSched<384, 8, 48, 8>;
using StreamLine512 = StreamLineSched<512, 16, 32, 16>;
using StreamLine768 = StreamLineSched<768, 16, 48, 16>;

template <class LR>
const StreamOps* stream_ops_of(int ny) {
  static const StreamOps table[] = {StreamImpl<LR, StreamLine256, 1>::ops(), StreamImpl<LR, StreamLine384, 1>::ops(),
                                    StreamImpl<LR, StreamLine512, 1>::ops(), StreamImpl<LR, StreamLine768, 1>::ops()};
  switch (ny) {
    case 256: return &table[0];
    case 384: return &table[1];
    case 512: return &table[2];
    case 768: return &table[3];
    default: return nullptr;
  }
}
// One translation unit per row length.
const StreamOps* stream_ops_256(int ny);
const StreamOps* stream_ops_384(int ny);
const StreamOps* stream_ops_512(int ny);
const StreamOps* stream_ops_768(int ny);

}  // namespace msx
