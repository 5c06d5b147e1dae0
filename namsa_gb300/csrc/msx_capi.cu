// C ABI of libmsx.so (declared in include/msx.h): argument checks, plans,
// schedule tables and the multislice launch sequence.
#include "msx.h"
#include "msx_internal.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <map>
#include <mutex>
#include <string>
#include <vector>

using namespace msx;

namespace {

thread_local std::string g_err;

int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  return fail(MSX_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
}

#define MSX_CUDA(call, what)                   \
  do {                                         \
    cudaError_t e_ = (call);                   \
    if (e_ != cudaSuccess) return cuda_fail(e_, what); \
  } while (0)

int schedule_table(int n, const SchedOps** ops) {
  switch (n) {
    case 64: return schedules_64(ops);
    case 128: return schedules_128(ops);
    case 256: return schedules_256(ops);
    case 384: return schedules_384(ops);
    case 512: return schedules_512(ops);
    case 768: return schedules_768(ops);
    case 1024: return schedules_1024(ops);
    default: *ops = nullptr; return 0;
  }
}

// The all-slices kernel of a grid, or null.
const StreamOps* stream_ops(int ny, int nx) {
  switch (nx) {
    case 256: return stream_ops_256(ny);
    case 384: return stream_ops_384(ny);
    case 512: return stream_ops_512(ny);
    case 768: return stream_ops_768(ny);
    default: return nullptr;
  }
}

// cudaFuncSetAttribute must run once per device for every kernel of a schedule.
constexpr int kMaxDevices = 64;
constexpr int kMaxSchedPerSize = 8;
bool g_configured[kMaxDevices][8][kMaxSchedPerSize];

int size_slot(int n) {
  switch (n) {
    case 64: return 0; case 128: return 1; case 256: return 2; case 384: return 3;
    case 512: return 4; case 768: return 5; case 1024: return 6; default: return 7;
  }
}

int ensure_configured(int device, int n, int idx, const SchedOps& op) {
  if (device < 0 || device >= kMaxDevices || idx >= kMaxSchedPerSize) return fail(MSX_ERR_INVALID, "device/schedule index out of range");
  bool& done = g_configured[device][size_slot(n)][idx];
  if (!done) {
    MSX_CUDA(op.configure(), "configuring pass kernels");
    done = true;
  }
  return MSX_OK;
}

bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }
// Every pointer on an 8-byte boundary (null is): complex values and position pairs are loaded whole.
bool aligned8(std::initializer_list<const void*> ps) {
  for (const void* p : ps)
    if (!aligned(p, 8)) return false;
  return true;
}
constexpr const char* kAlign8 = "complex inputs, positions and the normalisation must be 8-byte aligned";

}  // namespace

void msx::set_last_error(const char* msg) { g_err = msg; }

struct msx_plan {
  int ny = 0, nx = 0, device = 0;
  int group = 0;
  int row_sched = 0, col_sched = 0;
  const SchedOps* row_ops = nullptr;
  const SchedOps* col_ops = nullptr;
  float2* psi = nullptr;
  size_t psi_waves = 0;
  float2* ptab = nullptr;
  float2* tw_row = nullptr;
  float2* tw_col = nullptr;
  cudaStream_t work = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  cudaEvent_t ev_last = nullptr;  // after the last call that used the plan's waves, tables and counters
  bool use_graph = true;
  cudaGraphExec_t gexec = nullptr;
  std::vector<unsigned char> gkey;
  cudaGraphExec_t gexec_host = nullptr;  // msx_multislice_host, page-locked buffers
  std::vector<unsigned char> gkey_host;
  // persistent TMA-pipelined passes
  bool use_tma = true;
  void* tables = nullptr;        // one allocation behind the small tables:
  int* err = nullptr;            // device error word of the bounded waits
  float2* pyx = nullptr;         // py[ny] then px[nx]
  int2* band = nullptr;          // mask band per column
  CUtensorMap map{};             // workspace as (psi_waves*ny) x nx 8-byte elements, box col_c x col_boxr
  bool map_ok = false;
  int row_ctas = 0, col_ctas = 0, sms = 0;
  // the passes of calls of a few lines (few_lines); off while schedules are set by hand
  struct FewPass {
    const SchedOps* ops = nullptr;
    float2* tw = nullptr;        // in `tables`
    int ctas = 0;
    FormState form;
  } few_row, few_col;
  CUtensorMap fmap{};            // the workspace with few_col's tile as box
  bool use_few = false;
  // all slices of a group in one kernel (msx_stream.cuh); off while schedules are set by hand
  const StreamOps* stream = nullptr;
  FormState stream_form, resident_form;  // asked by the first call that would take the form
  bool use_stream = false;       // may take `stream`
  bool use_resident = false;     // may take `resident`
  // a wave in the shared memory of a cluster (msx_resident.cuh), small grids
  const ResidentOps* resident = nullptr;
  float2* rtw_row = nullptr;     // in `tables`
  float2* rtw_col = nullptr;
  int rclusters[3] = {-1, -1, -1}, rclusters_w = -1;  // clusters of kResidentSizes at the same time, for that many band columns
  CUtensorMap smap{};            // the workspace with the kernel's column tile as box
  float2* stw_row = nullptr;     // in `tables`, like the counters (2 * kMaxChunks)
  float2* stw_col = nullptr;
  int* counters = nullptr;
  float* partial = nullptr;      // detector partial sums
  size_t partial_words = 0;
  float2* inv_n = nullptr;       // constant (1/N, 0) table for CBEDs of real-space waves
  // host-buffer calls (msx_multislice_host): a copy stream and device copies of
  // the inputs and of the CBED stack, grown as needed
  cudaStream_t copy = nullptr;
  cudaEvent_t ev_copy = nullptr;
  float2* io_trans = nullptr;
  size_t io_trans_words = 0;
  float2* io_psik = nullptr;
  size_t io_psik_words = 0;
  float* io_pos = nullptr;
  size_t io_pos_words = 0;
  double* io_norm = nullptr;
  float* io_cbed = nullptr;
  size_t io_cbed_words = 0;
};

namespace {

constexpr int kMaxChunks = 1024;  // chunks of a group of the all-slices kernel

// A schedule's twiddle table, computed once per process (they are constants; there
// are as many as compiled schedules).
const std::vector<float2>& host_twiddles(int words, void (*fill)(float2*)) {
  static std::mutex m;
  static std::map<void (*)(float2*), std::vector<float2>> tables;
  std::lock_guard<std::mutex> lock(m);
  std::vector<float2>& h = tables[fill];
  if (h.empty()) {
    h.resize(words > 0 ? words : 1);
    fill(h.data());
  }
  return h;  // a map's elements stay where they are
}

int upload_twiddles(const SchedOps& op, float2** dst) {
  const std::vector<float2>& h = host_twiddles(op.tw_words, op.host_twiddles);
  if (*dst) cudaFree(*dst);
  *dst = nullptr;
  cudaError_t e = cudaMalloc(dst, sizeof(float2) * h.size());
  if (e != cudaSuccess) return fail(MSX_ERR_ALLOC, "twiddle table allocation failed: %s", cudaGetErrorString(e));
  MSX_CUDA(cudaMemcpy(*dst, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice), "twiddle upload");
  return MSX_OK;
}

// The propagator table of the plain passes, allocated for the first call that runs
// them (which may be under a stream capture).
int ensure_ptab(msx_plan* p) {
  if (p->ptab) return MSX_OK;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  MSX_CUDA(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
  const cudaError_t e = cudaMalloc(&p->ptab, sizeof(float2) * (size_t)p->ny * p->nx);
  MSX_CUDA(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
  if (e != cudaSuccess) {
    cudaGetLastError();
    p->ptab = nullptr;
    return fail(MSX_ERR_ALLOC, "propagator table allocation failed");
  }
  return MSX_OK;
}

// The constant (1/N, 0) table, filled before the first call that reads it goes on: later
// calls may come from any stream, and the first one may be under a capture.
int ensure_inv_n(msx_plan* p) {
  if (p->inv_n) return MSX_OK;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  MSX_CUDA(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
  float2* t = nullptr;
  cudaError_t e = cudaMalloc(&t, sizeof(float2) * (size_t)p->ny * p->nx);
  const bool allocated = e == cudaSuccess;
  // P = 1 everywhere, k_band beyond every |k|: zero thickness gives (1/N, 0)
  if (e == cudaSuccess) e = launch_ptab(p->ny, p->nx, 1.0f, 1.0, 0.0, 3.0e38f, t, p->work);
  if (e == cudaSuccess) e = cudaStreamSynchronize(p->work);
  MSX_CUDA(cudaThreadExchangeStreamCaptureMode(&mode), "cudaThreadExchangeStreamCaptureMode");
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (t) cudaFree(t);
    return allocated ? cuda_fail(e, "constant table") : fail(MSX_ERR_ALLOC, "constant table allocation failed");
  }
  p->inv_n = t;
  return MSX_OK;
}

// Asks the device, also under a stream capture.
template <class F>
cudaError_t ask_device(F ask) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return e;
  const cudaError_t asked = ask();
  e = cudaThreadExchangeStreamCaptureMode(&mode);
  return asked != cudaSuccess ? asked : e;
}

// Whether the device takes the plan's optional forms; where it refuses one (no room for
// its CTAs, its clusters or its registers) the two passes with the plan's schedules run.
// Asked by the first call whose rules choose the form: the answer loads the form's
// module, and many plans never come to it (first plan of a process: 256^2 2.8 ms
// configuring every form at once, 2.3 so; 512^2 2.6, 2.2; 384 x 768 2.9, 2.3).
bool stream_ready(msx_plan* p) {
  return p->stream && p->stream_form.ready([&] { return ask_device([&] { return p->stream->configure(); }); });
}
bool resident_ready(msx_plan* p) {
  return p->resident && p->resident_form.ready([&] { return ask_device([&] { return p->resident->configure(); }); });
}
bool few_ready(msx_plan* p, msx_plan::FewPass& f) {
  auto configure = [&] {
    cudaError_t e = f.ops->configure();
    int sms = 0, rows = 0, cols = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device);
    if (e == cudaSuccess) e = f.ops->occupancy(&rows, &cols);
    f.ctas = sms * (&f == &p->few_row ? rows : cols);
    return e == cudaSuccess && f.ctas < 1 ? cudaErrorInvalidConfiguration : e;
  };
  return f.ops && f.form.ready([&] { return ask_device(configure); });
}

// The plan's small tables in one allocation: propagator factors, mask bands, the
// error word, and the all-slices kernel's counters and twiddles.
int create_tables(msx_plan* p) {
  auto round = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t pyx = 0, band = pyx + round(sizeof(float2) * (size_t)(p->ny + p->nx));
  const size_t err = band + round(sizeof(int2) * (size_t)p->nx), counters = err + 256;
  size_t at = counters + (p->stream ? round(sizeof(int) * 2 * kMaxChunks) : 0);
  const size_t twiddles = at;
  std::vector<char> h;
  auto table = [&](int words, void (*fill)(float2*)) {  // its offset
    const std::vector<float2>& t = host_twiddles(words, fill);
    const size_t off = at;
    at += round(sizeof(float2) * words);
    h.resize(at - twiddles, 0);
    std::memcpy(h.data() + (off - twiddles), t.data(), sizeof(float2) * words);
    return off;
  };
  size_t srow = 0, scol = 0, rrow = 0, rcol = 0, frow = 0, fcol = 0;
  if (p->few_row.ops) frow = table(p->few_row.ops->tw_words, p->few_row.ops->host_twiddles);
  if (p->few_col.ops) fcol = table(p->few_col.ops->tw_words, p->few_col.ops->host_twiddles);
  if (p->stream) {
    srow = table(p->stream->twr_words, p->stream->tw_row);
    scol = table(p->stream->twc_words, p->stream->tw_col);
  }
  if (p->resident) {
    rrow = table(p->resident->twr_words, p->resident->tw_row);
    rcol = table(p->resident->twc_words, p->resident->tw_col);
  }
  const size_t total = at;
  if (cudaMalloc(&p->tables, total) != cudaSuccess) return fail(MSX_ERR_ALLOC, "plan table allocation failed");
  char* base = static_cast<char*>(p->tables);
  p->pyx = reinterpret_cast<float2*>(base + pyx);
  p->band = reinterpret_cast<int2*>(base + band);
  p->err = reinterpret_cast<int*>(base + err);
  MSX_CUDA(cudaMemset(p->err, 0, sizeof(int)), "clearing the plan error word");
  if (!h.empty()) MSX_CUDA(cudaMemcpy(base + twiddles, h.data(), h.size(), cudaMemcpyHostToDevice), "twiddle upload");
  if (p->stream) {
    p->counters = reinterpret_cast<int*>(base + counters);
    p->stw_row = reinterpret_cast<float2*>(base + srow);
    p->stw_col = reinterpret_cast<float2*>(base + scol);
  }
  if (p->resident) {
    p->rtw_row = reinterpret_cast<float2*>(base + rrow);
    p->rtw_col = reinterpret_cast<float2*>(base + rcol);
  }
  p->few_row.tw = reinterpret_cast<float2*>(base + frow);
  p->few_col.tw = reinterpret_cast<float2*>(base + fcol);
  p->use_few = true;
  p->use_stream = true;
  p->use_resident = true;
  return MSX_OK;
}

// Grows the wave workspace to `waves`.  The new buffer is allocated before the
// old one is released, so on failure the plan keeps its previous workspace.
int ensure_workspace(msx_plan* p, size_t waves) {
  if (waves <= p->psi_waves) return MSX_OK;
  float2* fresh = nullptr;
  cudaError_t e = cudaMalloc(&fresh, sizeof(float2) * waves * (size_t)p->ny * p->nx);
  if (e != cudaSuccess) {
    cudaGetLastError();  // clear the sticky-free allocation error
    return fail(MSX_ERR_ALLOC, "workspace of %zu waves (%d x %d) failed: %s", waves, p->ny, p->nx,
                cudaGetErrorString(e));
  }
  if (p->psi) cudaFree(p->psi);
  p->psi = fresh;
  p->psi_waves = waves;
  p->map_ok = false;  // the tensor map describes the old buffer until prepare_tma runs
  return MSX_OK;
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  static EncodeTiled fn = nullptr;
  if (!fn) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(f);
  }
  return fn;
}

// Tensor map of the wave workspace for the column pass's tile loads, and the
// persistent grid sizes of the current schedules.
int prepare_tma(msx_plan* p) {
  p->map_ok = false;
  EncodeTiled enc = encode_tiled();
  if (!enc) return fail(MSX_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t dims[2] = {(cuuint64_t)p->nx, (cuuint64_t)p->psi_waves * p->ny};
  const cuuint64_t strides[1] = {(cuuint64_t)p->nx * sizeof(float2)};
  const cuuint32_t estr[2] = {1, 1};
  auto encode = [&](CUtensorMap* map, int c, int boxr) {
    const cuuint32_t box[2] = {(cuuint32_t)c, (cuuint32_t)boxr};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, p->psi, dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode(&p->map, p->col_ops->col_c, p->col_ops->col_boxr);
  if (r == CUDA_SUCCESS && p->stream) r = encode(&p->smap, p->stream->col_c, p->stream->col_boxr);
  if (r == CUDA_SUCCESS && p->few_col.ops) r = encode(&p->fmap, p->few_col.ops->col_c, p->few_col.ops->col_boxr);
  if (r != CUDA_SUCCESS) return fail(MSX_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  int sms = 0, rr = 0, cr = 0, dummy = 0;
  MSX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device), "SM count");
  MSX_CUDA(p->row_ops->occupancy(&rr, &dummy), "occupancy");
  MSX_CUDA(p->col_ops->occupancy(&dummy, &cr), "occupancy");
  if (rr < 1 || cr < 1) return fail(MSX_ERR_CUDA, "persistent passes do not fit on an SM");
  p->sms = sms;
  p->row_ctas = sms * rr;
  p->col_ctas = sms * cr;
  p->map_ok = true;
  return MSX_OK;
}

void drop_graph(msx_plan* p) {
  if (p->gexec) cudaGraphExecDestroy(p->gexec);
  p->gexec = nullptr;
  p->gkey.clear();
  if (p->gexec_host) cudaGraphExecDestroy(p->gexec_host);
  p->gexec_host = nullptr;
  p->gkey_host.clear();
}

int auto_group(int ny, int nx) {
  // A resident group of about 1 GiB of waves (complex64), 4 to 512 waves: the
  // persistent passes run faster per wave on large groups than on groups small
  // enough to stay in L2 (tiles flow without launch tails); the plan autotuner
  // picks the same on GB300 for every supported grid.
  const size_t wave = sizeof(float2) * (size_t)ny * nx;
  size_t g = ((size_t)1 << 30) / wave;
  if (g < 4) g = 4;
  if (g > 512) g = 512;
  return (int)g;
}

// Schedules a plan starts with, by event timings on GB300 of groups of about
// 1 GiB at bandwidth 1/3 (us per pass):
//   rows of 256     in CTAs of four warps 149, of eight 159 (912 waves)
//   rows of 384     48 x 8 199, 8 x 8 x 6 231 (400 waves)
//   rows of 512     32 x 16 in CTAs of four warps 355, of eight 365, paired
//                   transform 364 (512 waves)
//   rows of 768     48 x 16 422, 8 x 8 x 12 496 (228 waves)
//   columns of 384  48 x 8 117, 8 x 8 x 6 149
//   columns of 768  48 x 16 265, 8 x 8 x 12 342 in 16-column tiles, 391 in 8-column ones
// and the first schedule elsewhere.
int schedule_index(int n, const char* name) {
  const SchedOps* ops = nullptr;
  const int k = schedule_table(n, &ops);
  for (int i = 0; i < k; ++i)
    if (std::strcmp(ops[i].name, name) == 0) return i;
  return 0;
}
int default_row_schedule(int nx) {
  switch (nx) {
    case 256: return schedule_index(256, "t16_r16x16_c8");
    case 384: return schedule_index(384, "t8_r48x8");
    case 512: return schedule_index(512, "t16_r32x16_c8");
    case 768: return schedule_index(768, "t16_r48x16");
    default: return 0;
  }
}
int default_col_schedule(int ny) {
  return ny == 768 ? schedule_index(768, "t16_r48x16") : ny == 384 ? schedule_index(384, "t8_r48x8") : 0;
}

// Schedules of calls whose passes do not fill the GPU, where the shortest line counts
// and not the most lines: the radices above win by fewer operations and exchanges
// per line but are a longer chain.  -1: the default serves them too.
int few_row_schedule(int nx) {
  switch (nx) {
    case 384: return schedule_index(384, "t16_r8x8x6");
    case 512: return schedule_index(512, "t32_r16x2x16_pair");
    case 768: return schedule_index(768, "t32_r8x8x12");
    default: return -1;
  }
}
int few_col_schedule(int ny) { return ny == 384 || ny == 768 ? few_row_schedule(ny) : -1; }

struct MsArgs {
  const float* trans; int num_slices; const float* psik; const double* norm; const float* pos; int num_probes;
  float kmax; double lambda, slice_t; float k_band; float* cbed; int crop_y, crop_x;
  int group, row_sched, col_sched;
  const float* det; int ndet; float* signals;  // detector mode (det != nullptr): signals (P, ndet) instead of cbed
};

// One slice's row pass and (mid) column pass over a group of gn waves.
// Band-limited column range.  A column whose |kx| reaches the mask radius has
// |k| >= k_band for every ky, so the column pass zeroes it whole; from the second
// slice on those columns are zero on entry, stay zero through the row pass (which
// then need not write them) and need no column pass.  [x_lo, x_hi) is the range
// of column tiles (width C) holding every column with |kx| < k_band, with a
// 1e-6 relative margin on k_band so that it contains every column the device's
// float32 mask test keeps.  The whole grid when no column is in the band.
void band_columns(int nx, float kmax, float k_band, int C, int* x_lo, int* x_hi) {
  const double km = (double)kmax, lim = (double)k_band * (1.0 + 1e-6);
  int lo = nx, hi = -1;
  for (int j = 0; j < nx; ++j) {
    const double kx = (double)j * km / (double)(nx - 1) - km / 2.0;
    if (std::fabs(kx) < lim) {
      lo = j < lo ? j : lo;
      hi = j;
    }
  }
  if (hi < 0 || C <= 0) {
    *x_lo = 0;
    *x_hi = nx;
    return;
  }
  *x_lo = (lo / C) * C;
  *x_hi = (hi / C + 1) * C < nx ? (hi / C + 1) * C : nx;
}

// Whether the row (column) pass over gn waves runs with the schedule for few lines:
// while its tiles are at most one to an SM; at 768 also for one tile a row, since the
// default's CTAs are alone on their SM.  Event timings on GB300, us per slice of both
// passes, default / few:
//   rows     64 x 384   P 1 9.9/9.0   32 12.2/11.5  64 14.4/16.0     256 x 384  P 4 12.6/14.3
//           128 x 384   P 4 11.7/10.9 16 12.6/11.9  24 14.7/16.5
//            64 x 768   P 1 11.2/9.6  16 13.2/11.0  24 13.9/15.0
//           384 x 768   P 1 25.3/21.0  8 27.3/23.5  12 31.8/36.5
//            64 x 512   P 1 8.8/8.2   16 9.9/9.2    24 10.6/10.7
//   columns 384 x 128   P 1 14.4/13.0 24 15.9/14.7  32 17.4/17.8
//           384 x 384   P 1 19.5/18.2  8 20.2/18.9  12 21.6/21.8
//           768 x 64    P 1 16.1/14.1 24 18.5/16.6  32 19.5/20.9
//           768 x 256   P 1 16.5/14.3  4 16.7/14.5   8 17.4/19.0
bool few_rows(msx_plan* p, int gn) {
  if (!p->use_few || !p->few_row.ops) return false;
  const int tiles = (gn + p->few_row.ops->row_lines - 1) / p->few_row.ops->row_lines;
  return (tiles * p->ny <= p->sms || (p->nx == 768 && tiles == 1)) && few_ready(p, p->few_row);
}
bool few_cols(msx_plan* p, int gn, float kmax, float k_band, int* x_lo, int* x_hi) {
  if (p->use_few && p->few_col.ops) {
    band_columns(p->nx, kmax, k_band, p->few_col.ops->col_c, x_lo, x_hi);
    if ((*x_hi - *x_lo) / p->few_col.ops->col_c * gn <= p->sms && few_ready(p, p->few_col)) return true;
  }
  band_columns(p->nx, kmax, k_band, p->col_ops->col_c, x_lo, x_hi);
  return false;
}

// Whether the passes run as persistent kernels: their bulk copies of transmission rows
// start on 16-byte boundaries.
bool tma_passes(const msx_plan* p, const void* trans) { return p->use_tma && p->map_ok && aligned(trans, 16); }

// x_lo, x_hi: the column range of the TMA passes (0, 0 = all columns); the
// plain passes always cover every column.  fr, fc: the row, column pass with the
// schedule for few lines.
int slice_passes(msx_plan* p, const float2* trans_s, int gn, const ColArgs& c, bool with_col, cudaStream_t st,
                 int x_lo, int x_hi, bool tma, bool fr = false, bool fc = false) {
  if (tma) {
    TmaPassArgs ta{};
    ta.psi = p->psi; ta.trans = trans_s; ta.tw = fr ? p->few_row.tw : p->tw_row; ta.pyx = p->pyx; ta.band = p->band;
    ta.err = p->err; ta.G = gn; ta.Ny = p->ny; ta.Nx = p->nx; ta.x_lo = x_lo; ta.x_hi = x_hi;
    MSX_CUDA((fr ? p->few_row.ops : p->row_ops)->row_tma(ta, fr ? p->few_row.ctas : p->row_ctas, st), "row pass");
    if (with_col) {
      ta.tw = fc ? p->few_col.tw : p->tw_col;
      MSX_CUDA(fc ? p->few_col.ops->col_tma(p->fmap, ta, p->few_col.ctas, st)
                  : p->col_ops->col_tma(p->map, ta, p->col_ctas, st), "column pass");
    }
  } else {
    MSX_CUDA(p->row_ops->row(p->psi, trans_s, p->tw_row, gn, p->ny, st), "row pass");
    if (with_col) MSX_CUDA(p->col_ops->col(COL_MID, c, st), "column pass");
  }
  return MSX_OK;
}

// Copy pipeline of msx_multislice_host: the first group waits for each chunk of
// uploaded slices only when it reaches it, and each group's CBED block goes
// back to the host on the copy stream while the next group computes.
struct HostPipe {
  cudaStream_t copy;
  int chunk;                              // slices per upload chunk
  const std::vector<cudaEvent_t>* chunk_ev;  // recorded on the copy stream after each chunk
  std::vector<cudaEvent_t>* group_ev;        // recorded on the work stream after each group
  float* cbed_host;
  size_t pattern_words;                   // crop_y * crop_x
};

// A plan can only run groups its workspace holds (an allocation that failed
// leaves the previous workspace, or none).
bool workspace_holds(const msx_plan* p, int waves) { return p->psi && waves >= 0 && (size_t)waves <= p->psi_waves; }

// Grows a plan-owned device buffer of `words` elements of T.
template <class T>
int grow(T** buf, size_t* have, size_t words, const char* what) {
  if (words <= *have && *buf) return MSX_OK;
  T* fresh = nullptr;
  const cudaError_t e = cudaMalloc(&fresh, sizeof(T) * (words ? words : 1));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(MSX_ERR_ALLOC, "%s: allocation of %zu bytes failed", what, sizeof(T) * words);
  }
  if (*buf) cudaFree(*buf);
  *buf = fresh;
  *have = words;
  return MSX_OK;
}

// Whether a call runs through the all-slices kernel, and the waves of its groups.
// A group is as many waves as stay in L2 (kStreamBytes of their band columns: the
// row and column tiles read and write nothing else), in equal parts.
//
// The line between it and the separate passes is that of event timings on GB300
// of every pair of its line lengths from 1 to 512 positions (24 slices, bandwidth
// 1/3): from `few` positions on, and up to `most` MB of band columns of all
// waves, it was the faster one.  The passes gain with long launches (no
// part-filled last waves of tiles); the kernel's waits between the passes of one
// wave cost most on short lines.  Passes (with the schedules of few lines where a
// call has few) / all slices, us, at 1, 8, 16, 64, 256 positions:
//   256 x 256   212/235   235/253   304/276   647/529    2130/2012
//   384 x 384   438/457   462/504   551/543   1438/1241  5195/4844
//   512 x 512   385/351   491/412   700/569   2256/2117  8349/8333
//   768 x 768   724/727   966/947   1555/1261 5121/4904  (128: 9653/10068)
//   768 x 256   349/367   418/413   637/548   1801/1826  6114/7251
//   256 x 768   343/331   413/421   593/516   1784/1702  6530/6747
constexpr size_t kStreamBytes = (size_t)80 << 20;
struct StreamRange {
  int few, most;
};
constexpr StreamRange kStreamRange[4][4] = {  // [ny][nx], lines of 256, 384, 512, 768
    {{12, 180}, {24, 130}, {12, 60}, {1, 130}},
    {{24, 36}, {16, 400}, {12, 130}, {12, 300}},
    {{8, 60}, {1, 500}, {1, 360}, {1, 500}},
    {{8, 36}, {1, 300}, {1, 380}, {1, 310}}};
int stream_group(msx_plan* p, const MsArgs& a) {
  if (!p->use_stream || !p->stream || !p->use_tma || !p->map_ok || a.num_slices < 2 || a.num_probes < 1 ||
      !aligned(a.trans, 16))
    return 0;
  auto line = [](int n) { return n == 256 ? 0 : n == 384 ? 1 : n == 512 ? 2 : 3; };
  const StreamRange range = kStreamRange[line(p->ny)][line(p->nx)];
  int lo = 0, hi = 0;
  band_columns(p->nx, a.kmax, a.k_band, p->stream->col_c, &lo, &hi);
  const size_t bytes = sizeof(float2) * (size_t)p->ny * (hi - lo);
  if (a.num_probes < range.few || bytes * a.num_probes > ((size_t)range.most << 20)) return 0;
  constexpr int unit = 8;  // whole chunks of every instance
  size_t most = kStreamBytes / bytes / unit * unit;
  if (most < unit) most = unit;
  if (most > (size_t)p->stream->wpt * kMaxChunks) most = (size_t)p->stream->wpt * kMaxChunks;
  const int groups = (int)((a.num_probes + most - 1) / most);
  int g = ((a.num_probes + groups - 1) / groups + unit - 1) / unit * unit;
  if (g > a.num_probes) g = a.num_probes;
  return workspace_holds(p, g) && stream_ready(p) ? g : 0;
}

// Whether a call keeps each wave in a cluster, and the CTAs of a cluster: as many as
// let all positions run at the same time (more CTAs shorten a slice).  Event
// timings on GB300, us per slice in the passes / clusters of 16 / 8 / 4:
//   256^2      P 1 8.7 / 6.0 / 10.0 / -     8 9.3 / 11.4 / 10.0 / -
//   128 x 256  P 1 7.8 / 5.1 / 5.7 / 10.0   8 8.4 / 9.4 / 5.7 / 9.9   32 11.5 / 22 / 16 / 10.0
//   128^2      P 4 8.9 / 5.1 / 5.0 / 6.1   16 9.3 / 14 / 8.9 / 6.1   64 13.2 / 43 / 21 / 11.5
//   64^2       P 1 6.4 / 3.6 / 3.1 / 3.2   64 7.6 / 31 / 14 / 5.7   128 9.1 / 58 / 24 / 10.9
// so 16 only above 128^2, fewer only below 256^2, and the smallest grids take up
// to two rounds of clusters of four.
constexpr int kResidentSizes[3] = {16, 8, 4};
int resident_cluster(msx_plan* p, const MsArgs& a) {
  if (!p->use_resident || !p->resident || !p->use_tma || !p->map_ok || a.det || a.num_slices < 2 || a.num_probes < 1 ||
      !workspace_holds(p, a.num_probes) || !aligned(a.trans, 16))
    return 0;
  int lo = 0, hi = 0;
  band_columns(p->nx, a.kmax, a.k_band, 1, &lo, &hi);
  const int w = hi - lo;
  // whether all positions run in `rounds` rounds of clusters of kResidentSizes[i]; the
  // device is asked where the shared memory alone does not rule it out
  auto fits = [&](int i, int rounds) -> bool {
    const int cl = kResidentSizes[i];
    if (a.num_probes > rounds * p->resident->most(w, cl, p->sms) || !resident_ready(p)) return false;
    if (p->rclusters_w != w) {
      for (int& n : p->rclusters) n = -1;
      p->rclusters_w = w;
    }
    int& n = p->rclusters[i];
    if (n < 0 && ask_device([&] { return p->resident->clusters(w, cl, &n); }) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    return a.num_probes <= rounds * n;
  };
  const int area = p->ny * p->nx;
  if (area > 128 * 128 && fits(0, 1)) return kResidentSizes[0];
  if (area >= 256 * 256) return 0;
  if (fits(1, 1)) return kResidentSizes[1];
  if (p->nx > p->ny && area > 128 * 128 && a.num_probes < 24) return 0;  // 128 x 256: P 16 9.0 / 9.7, 24 9.8 / 9.7
  const int rounds = area <= 128 * 128 && p->nx <= 128 ? 2 : 1;  // 64 x 256: P 64 10.9 / 11.1 in two
  if (fits(2, rounds)) return kResidentSizes[2];
  return 0;
}

// Slices [s0, s1) of a group of gn waves; `more`: slices follow, so the last one has its column pass.
int stream_slices(msx_plan* p, const MsArgs& a, int s0, int s1, bool more, int gn, cudaStream_t st) {
  StreamArgs sa{};
  sa.psi = p->psi;
  sa.trans = reinterpret_cast<const float2*>(a.trans) + (size_t)s0 * p->ny * p->nx;
  sa.tw_row = p->stw_row;
  sa.tw_col = p->stw_col;
  sa.pyx = p->pyx;
  sa.band = p->band;
  sa.counters = p->counters;
  sa.err = p->err;
  sa.first = s0 == 0 ? 1 : 0;
  band_columns(p->nx, a.kmax, a.k_band, p->stream->col_c, &sa.x_lo, &sa.x_hi);
  sa.sh = StreamShape{gn, p->stream->wpt, p->stream->ypt, p->ny, (sa.x_hi - sa.x_lo) / p->stream->col_c, s1 - s0, more ? 1 : 0};
  MSX_CUDA(cudaMemsetAsync(p->counters, 0, sizeof(int) * 2 * sa.sh.chunks(), st), "clearing the tile counters");
  MSX_CUDA(p->stream->launch(p->smap, sa, p->sms, st), "all-slices kernel");
  return MSX_OK;
}

// A call of so few launches that issuing them costs less than recording a graph
// for every new set of buffers (an output allocated by the caller is one).
bool few_launches(msx_plan* p, const MsArgs& a) {
  if (resident_cluster(p, a)) return true;
  const int g = stream_group(p, a);
  return g > 0 && a.num_probes <= 2 * g;
}

// Calls of one plan share its waves, tables, partial sums and counters, so each follows
// the last one (ev_last), whichever streams they come from.  Under a capture a call
// joins the caller's stream, and the caller keeps the captured work apart from the
// plan's other calls.
int after_last_call(msx_plan* p, cudaStream_t st) {
  MSX_CUDA(cudaStreamWaitEvent(st, p->ev_last, 0), "cudaStreamWaitEvent");
  return MSX_OK;
}

// Runs enqueue(stream) in that order: on the caller's stream, or for recorded graphs and
// calls of a few launches on the plan's, which follows the caller's and is followed by it.
// A failed call is ordered too: what was enqueued before the failure uses the caller's buffers.
template <class F>
int in_call_order(msx_plan* p, cudaStream_t caller, bool own_stream, F enqueue) {
  cudaStream_t st = caller;
  if (own_stream) {
    MSX_CUDA(cudaEventRecord(p->ev_in, caller), "cudaEventRecord");
    MSX_CUDA(cudaStreamWaitEvent(p->work, p->ev_in, 0), "cudaStreamWaitEvent");
    st = p->work;
  }
  const int ordered = after_last_call(p, st);
  if (ordered != MSX_OK) return ordered;
  const int rc = enqueue(st);
  const std::string msg = g_err;
  MSX_CUDA(cudaEventRecord(p->ev_last, st), "cudaEventRecord");
  if (own_stream) MSX_CUDA(cudaStreamWaitEvent(caller, p->ev_last, 0), "cudaStreamWaitEvent");
  if (rc != MSX_OK) g_err = msg;
  return rc;
}

bool capturing(cudaStream_t st, int* rc) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const cudaError_t e = cudaStreamIsCapturing(st, &cap);
  *rc = e == cudaSuccess ? MSX_OK : cuda_fail(e, "cudaStreamIsCapturing");
  return cap != cudaStreamCaptureStatusNone;
}

int enqueue_multislice(msx_plan* p, const MsArgs& a, cudaStream_t st, const HostPipe* hp = nullptr) {
  const int ny = p->ny, nx = p->nx;
  const int cluster = resident_cluster(p, a);
  const int streamed = cluster ? 0 : stream_group(p, a);
  const int group = cluster ? a.num_probes : streamed ? streamed : a.group;
  const int gmax = a.num_probes < group ? a.num_probes : group;
  if (!workspace_holds(p, gmax))
    return fail(MSX_ERR_ALLOC, "the plan's workspace does not hold %d waves (an earlier allocation failed)", gmax);
  // the persistent passes form the propagator from its factors and the mask band;
  // the table of N values (26 us of double precision at 512^2, 89 us at 1024^2)
  // serves the plain passes
  const bool tma = tma_passes(p, a.trans);
  const bool factors = tma;
  if (!factors) {
    const int rc = ensure_ptab(p);
    if (rc != MSX_OK) return rc;
  }
  if (factors)
    MSX_CUDA(launch_pfac(ny, nx, a.kmax, a.lambda, a.slice_t, a.k_band, p->pyx, p->band, st), "propagator factors");
  else
    MSX_CUDA(launch_ptab(ny, nx, a.kmax, a.lambda, a.slice_t, a.k_band, p->ptab, st), "propagator table");
  const size_t wave = (size_t)ny * nx;
  const int y0 = ny / 2 - a.crop_y / 2, x0 = nx / 2 - a.crop_x / 2;
  const float2* trans = reinterpret_cast<const float2*>(a.trans);
  // group done: hand its CBED block to the copy stream (host-buffer calls)
  auto hand_off = [&](int gi, int g0, int gn) -> int {
    if (!hp) return MSX_OK;
    cudaEvent_t ev = (*hp->group_ev)[gi];
    MSX_CUDA(cudaEventRecord(ev, st), "cudaEventRecord");
    MSX_CUDA(cudaStreamWaitEvent(hp->copy, ev, 0), "cudaStreamWaitEvent");
    MSX_CUDA(cudaMemcpyAsync(hp->cbed_host + (size_t)g0 * hp->pattern_words, a.cbed + (size_t)g0 * hp->pattern_words,
                             sizeof(float) * (size_t)gn * hp->pattern_words, cudaMemcpyDeviceToHost, hp->copy),
             "CBED download");
    return MSX_OK;
  };
  for (int g0 = 0, gi = 0; g0 < a.num_probes; g0 += group, ++gi) {
    const int gn = (a.num_probes - g0 < group) ? a.num_probes - g0 : group;
    ColArgs c{};
    c.psi = p->psi;
    c.ptab = p->ptab;  // null where the persistent passes run
    c.psik = reinterpret_cast<const float2*>(a.psik);
    c.pos_yx = a.pos + 2 * (size_t)g0;
    c.tw = p->tw_col;
    c.norm = a.norm;
    c.cbed = a.cbed + (size_t)g0 * a.crop_y * a.crop_x;
    c.G = gn;
    c.Nx = nx;
    c.kmax = a.kmax;
    c.y0 = y0;
    c.crop_y = a.crop_y;
    if (factors) {
      c.band = p->band;
      c.inv_n = (float)(1.0 / ((double)ny * (double)nx));
    }
    if (a.num_slices == 0) {
      c.x_begin = x0;
      c.ncols = a.crop_x;
      MSX_CUDA(p->col_ops->col(COL_INIT_FINAL, c, st), "probe-only pass");
      const int rc = hand_off(gi, g0, gn);
      if (rc != MSX_OK) return rc;
      continue;
    }
    c.x_begin = 0;
    c.ncols = nx;
    MSX_CUDA(p->col_ops->col(COL_INIT, c, st), "probe formation pass");
    if (cluster) {  // one group of every position
      if (hp)
        for (int i = 0; i * hp->chunk < a.num_slices; ++i)
          MSX_CUDA(cudaStreamWaitEvent(st, (*hp->chunk_ev)[i], 0), "cudaStreamWaitEvent");
      ResidentArgs ra{};
      ra.psi = p->psi; ra.trans = trans; ra.tw_row = p->rtw_row; ra.tw_col = p->rtw_col; ra.pyx = p->pyx;
      ra.band = p->band; ra.norm = a.norm; ra.cbed = c.cbed; ra.err = p->err; ra.slices = a.num_slices;
      band_columns(nx, a.kmax, a.k_band, 1, &ra.x_lo, &ra.x_hi);
      ra.x0 = x0; ra.y0 = y0; ra.crop_y = a.crop_y; ra.crop_x = a.crop_x;
      MSX_CUDA(p->resident->launch(ra, gn, cluster, st), "cluster-resident kernel");
      const int rc = hand_off(gi, g0, gn);
      if (rc != MSX_OK) return rc;
      continue;
    }
    int bx_lo = 0, bx_hi = 0;
    const bool fr = few_rows(p, gn), fc = few_cols(p, gn, a.kmax, a.k_band, &bx_lo, &bx_hi);
    for (int s = 0; s < a.num_slices; ++s) {
      if (hp && gi == 0 && s % hp->chunk == 0)
        MSX_CUDA(cudaStreamWaitEvent(st, (*hp->chunk_ev)[s / hp->chunk], 0), "cudaStreamWaitEvent");
      int rc;
      if (streamed) {  // all slices, or those of one upload
        const int s0 = s, step = hp && gi == 0 ? hp->chunk : a.num_slices;
        s = (s0 + step < a.num_slices ? s0 + step : a.num_slices) - 1;
        rc = stream_slices(p, a, s0, s + 1, s + 1 < a.num_slices, gn, st);
      } else {
        // the first slice covers every column (the probe may reach beyond the band)
        rc = slice_passes(p, trans + (size_t)s * wave, gn, c, s + 1 < a.num_slices, st, s > 0 ? bx_lo : 0,
                          s > 0 ? bx_hi : 0, tma, fr, fc);
      }
      if (rc != MSX_OK) return rc;
      if (s + 1 == a.num_slices) {
        ColArgs f = c;
        if (a.det) {
          f.det = a.det;
          f.ndet = a.ndet;
          f.partial = p->partial;
          MSX_CUDA(p->col_ops->col(COL_DETECT, f, st), "detector pass");
          MSX_CUDA(launch_detect_reduce(p->partial, gn, nx / p->col_ops->col_c, a.ndet,
                                        a.signals + (size_t)g0 * a.ndet, st), "detector reduction");
        } else {
          f.x_begin = x0;
          f.ncols = a.crop_x;
          MSX_CUDA(p->col_ops->col(COL_FINAL, f, st), "final column pass");
          const int rc2 = hand_off(gi, g0, gn);
          if (rc2 != MSX_OK) return rc2;
        }
      }
    }
  }
  return MSX_OK;
}

}  // namespace

extern "C" {

int msx_version(void) { return 1 * 10000 + 0 * 100 + 0; }

int msx_last_error(char* buf, size_t len) {
  if (buf && len) {
    std::strncpy(buf, g_err.c_str(), len - 1);
    buf[len - 1] = '\0';
  }
  return (int)g_err.size();
}

int msx_supported_size(int n) {
  const SchedOps* ops;
  return schedule_table(n, &ops) > 0 ? 1 : 0;
}

int msx_num_schedules(int n) {
  const SchedOps* ops;
  return schedule_table(n, &ops);
}

int msx_schedule_name(int n, int index, char* buf, size_t len) {
  const SchedOps* ops;
  const int cnt = schedule_table(n, &ops);
  if (index < 0 || index >= cnt) return fail(MSX_ERR_INVALID, "no schedule %d for length %d", index, n);
  if (buf && len) {
    std::strncpy(buf, ops[index].name, len - 1);
    buf[len - 1] = '\0';
  }
  return MSX_OK;
}

int msx_schedule_col_tile(int n, int index, int* tile) {
  const SchedOps* ops;
  const int cnt = schedule_table(n, &ops);
  if (index < 0 || index >= cnt || !tile) return fail(MSX_ERR_INVALID, "no schedule %d for length %d", index, n);
  *tile = ops[index].col_c;
  return MSX_OK;
}

int msx_band_columns(int nx, float kmax, float k_band, int tile, int* x_lo, int* x_hi) {
  if (nx <= 1 || tile <= 0 || !x_lo || !x_hi || !(kmax > 0)) return fail(MSX_ERR_INVALID, "band_columns arguments");
  band_columns(nx, kmax, k_band, tile, x_lo, x_hi);
  return MSX_OK;
}

int msx_atom_windows(const double* coeff_dev, int nspecies, int n0, int n1, int oversample, double potential_range,
                     float* windows_out_dev, void* stream) {
  if (!coeff_dev || !windows_out_dev) return fail(MSX_ERR_INVALID, "null pointer");
  if (nspecies <= 0 || oversample <= 0 || n0 < 2 || n1 < 2 || n0 % oversample || n1 % oversample)
    return fail(MSX_ERR_INVALID, "bad window grid %d x %d (oversample %d, %d species)", n0, n1, oversample, nspecies);
  if (!(potential_range > 0)) return fail(MSX_ERR_INVALID, "potential range must be positive");
  if ((size_t)(n0 / oversample) * (n1 / oversample) > (size_t)65535 * 128)
    return fail(MSX_ERR_INVALID, "window %d x %d too large", n0 / oversample, n1 / oversample);
  MSX_CUDA(launch_atom_windows(coeff_dev, nspecies, n0, n1, oversample, potential_range, windows_out_dev,
                               (cudaStream_t)stream), "atom windows");
  return MSX_OK;
}

int msx_build_transmission(const int* sites_dev, const int* slice_offsets_dev, int num_slices, const float* windows_dev,
                           int window_h, int window_w, int ny, int nx, float sigma, float* trans_out_dev,
                           float* potential_out_dev, void* stream) {
  if (num_slices < 0 || ny <= 0 || nx <= 0 || window_h <= 0 || window_w <= 0)
    return fail(MSX_ERR_INVALID, "bad sizes (slices %d, grid %d x %d, window %d x %d)", num_slices, ny, nx, window_h,
                window_w);
  if (num_slices == 0) return MSX_OK;
  if (!sites_dev || !slice_offsets_dev || !windows_dev || !trans_out_dev) return fail(MSX_ERR_INVALID, "null pointer");
  if (!aligned(sites_dev, 16)) return fail(MSX_ERR_INVALID, "sites must be 16-byte aligned (int32 rows of 4)");
  if (!aligned(trans_out_dev, 8)) return fail(MSX_ERR_INVALID, "transmission output must be 8-byte aligned");
  if (num_slices > 65535) return fail(MSX_ERR_INVALID, "at most 65535 slices");
  MSX_CUDA(launch_potential(reinterpret_cast<const int4*>(sites_dev), slice_offsets_dev, num_slices, windows_dev, window_h,
                            window_w, ny, nx, sigma, reinterpret_cast<float2*>(trans_out_dev), potential_out_dev,
                            (cudaStream_t)stream), "transmission slices");
  return MSX_OK;
}

int msx_build_probe(int ny, int nx, float kmax, double lambda, float k_semi, double c1, double c3, double c5,
                    int smooth_aperture, float* psi_k_out_dev, float* aperture_out_dev, double* normalization_dev,
                    void* stream) {
  if (ny < 2 || nx < 2 || ny > 65535) return fail(MSX_ERR_INVALID, "bad grid %d x %d", ny, nx);
  if (!psi_k_out_dev) return fail(MSX_ERR_INVALID, "null psi_k output");
  if (!aligned(psi_k_out_dev, 8)) return fail(MSX_ERR_INVALID, "psi_k must be 8-byte aligned");
  if (!(lambda > 0) || !(kmax > 0)) return fail(MSX_ERR_INVALID, "lambda and kmax must be positive");
  MSX_CUDA(launch_probe(ny, nx, kmax, lambda, k_semi, c1, c3, c5, smooth_aperture,
                        reinterpret_cast<float2*>(psi_k_out_dev), aperture_out_dev, normalization_dev,
                        (cudaStream_t)stream), "probe");
  return MSX_OK;
}

int msx_plan_create(int ny, int nx, int group, msx_plan** out) {
  if (!out) return fail(MSX_ERR_INVALID, "null plan pointer");
  *out = nullptr;
  if (!msx_supported_size(ny) || !msx_supported_size(nx))
    return fail(MSX_ERR_UNSUPPORTED, "grid %d x %d: supported line lengths are 64, 128, 256, 384, 512, 768, 1024", ny, nx);
  if (group < 0) return fail(MSX_ERR_INVALID, "group must be >= 0");
  int device = 0;
  MSX_CUDA(cudaGetDevice(&device), "cudaGetDevice");
  msx_plan* p = new msx_plan();
  p->ny = ny;
  p->nx = nx;
  p->device = device;
  p->stream = stream_ops(ny, nx);
  p->resident = resident_ops(ny, nx);
  int rc = MSX_OK;
  const SchedOps *rops, *cops;
  schedule_table(nx, &rops);
  schedule_table(ny, &cops);
  const int fr = few_row_schedule(nx), fc = few_col_schedule(ny);
  if (fr >= 0) p->few_row.ops = &rops[fr];
  if (fc >= 0) p->few_col.ops = &cops[fc];
  rc = msx_plan_set_schedule(p, default_row_schedule(nx), default_col_schedule(ny),
                             group > 0 ? group : auto_group(ny, nx));
  if (rc == MSX_OK) rc = create_tables(p);
  if (rc == MSX_OK) {
    cudaError_t e = cudaStreamCreateWithFlags(&p->work, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p->ev_in, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p->ev_out, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p->ev_last, cudaEventDisableTiming);
    if (e != cudaSuccess) rc = cuda_fail(e, "plan stream/events");
  }
  if (rc != MSX_OK) {
    msx_plan_destroy(p);
    return rc;
  }
  *out = p;
  return MSX_OK;
}

int msx_plan_destroy(msx_plan* p) {
  if (!p) return MSX_OK;
  drop_graph(p);
  if (p->psi) cudaFree(p->psi);
  if (p->ptab) cudaFree(p->ptab);
  if (p->tables) cudaFree(p->tables);
  if (p->partial) cudaFree(p->partial);
  if (p->inv_n) cudaFree(p->inv_n);
  if (p->tw_row) cudaFree(p->tw_row);
  if (p->tw_col) cudaFree(p->tw_col);
  for (void* q : {(void*)p->io_trans, (void*)p->io_psik, (void*)p->io_pos, (void*)p->io_norm, (void*)p->io_cbed})
    if (q) cudaFree(q);
  if (p->ev_copy) cudaEventDestroy(p->ev_copy);
  if (p->copy) cudaStreamDestroy(p->copy);
  if (p->ev_in) cudaEventDestroy(p->ev_in);
  if (p->ev_out) cudaEventDestroy(p->ev_out);
  if (p->ev_last) cudaEventDestroy(p->ev_last);
  if (p->work) cudaStreamDestroy(p->work);
  delete p;
  return MSX_OK;
}

int msx_plan_set_schedule(msx_plan* p, int row_schedule, int col_schedule, int group) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  const SchedOps *rops, *cops;
  const int nr = schedule_table(p->nx, &rops), nc = schedule_table(p->ny, &cops);
  if (row_schedule < 0 || row_schedule >= nr || col_schedule < 0 || col_schedule >= nc)
    return fail(MSX_ERR_INVALID, "schedule (%d, %d) out of range (%d, %d)", row_schedule, col_schedule, nr, nc);
  if (group < 0 || group > 65535) return fail(MSX_ERR_INVALID, "group %d out of range", group);
  int rc = ensure_configured(p->device, p->nx, row_schedule, rops[row_schedule]);
  if (rc == MSX_OK) rc = ensure_configured(p->device, p->ny, col_schedule, cops[col_schedule]);
  if (rc != MSX_OK) return rc;
  if (!p->row_ops || p->row_sched != row_schedule) {
    rc = upload_twiddles(rops[row_schedule], &p->tw_row);
    if (rc != MSX_OK) return rc;
  }
  if (!p->col_ops || p->col_sched != col_schedule) {
    rc = upload_twiddles(cops[col_schedule], &p->tw_col);
    if (rc != MSX_OK) return rc;
  }
  p->use_stream = p->use_resident = p->use_few = false;  // schedules set by hand are the passes that run
  p->row_sched = row_schedule;
  p->col_sched = col_schedule;
  p->row_ops = &rops[row_schedule];
  p->col_ops = &cops[col_schedule];
  const int old_group = p->group;
  if (group > 0) p->group = group;
  drop_graph(p);
  rc = ensure_workspace(p, (size_t)p->group);
  if (rc != MSX_OK) {
    // keep the previous group (and its workspace); the new schedule still applies
    const std::string msg = g_err;
    p->group = old_group;
    const int rc2 = (p->psi && (size_t)p->group <= p->psi_waves) ? prepare_tma(p) : MSX_OK;
    if (rc2 != MSX_OK) return rc2;
    g_err = msg;
    return MSX_ERR_ALLOC;
  }
  return prepare_tma(p);
}

int msx_plan_get_schedule(const msx_plan* p, int* row_schedule, int* col_schedule, int* group) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  if (row_schedule) *row_schedule = p->row_sched;
  if (col_schedule) *col_schedule = p->col_sched;
  if (group) *group = p->group;
  return MSX_OK;
}

int msx_plan_route(msx_plan* p, int num_slices, int num_probes, float kmax, float k_band, int detector, int* form,
                   int* size, int* few) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  if (num_slices < 0 || num_probes < 1 || !(kmax > 0) || !(k_band >= 0))
    return fail(MSX_ERR_INVALID, "route: needs probes, kmax > 0, non-negative slices and k_band");
  MsArgs a;
  std::memset(&a, 0, sizeof(a));
  a.num_slices = num_slices; a.num_probes = num_probes; a.kmax = kmax; a.k_band = k_band; a.group = p->group;
  const float any = 0.f;
  a.det = detector ? &any : nullptr;
  const int cluster = resident_cluster(p, a), streamed = cluster ? 0 : stream_group(p, a);
  const int waves = num_probes < p->group ? num_probes : p->group;
  int lo = 0, hi = 0;
  if (form) *form = cluster ? MSX_FORM_CLUSTER : streamed ? MSX_FORM_ALL_SLICES : MSX_FORM_PASSES;
  if (size) *size = cluster ? cluster : streamed ? streamed : waves;
  if (few) {
    *few = 0;
    if (!cluster && !streamed && num_slices > 0 && p->use_tma && p->map_ok)
      *few = (few_rows(p, waves) ? 1 : 0) + (few_cols(p, waves, kmax, k_band, &lo, &hi) ? 2 : 0);
  }
  return MSX_OK;
}

int msx_plan_set_tma(msx_plan* p, int enable) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  p->use_tma = enable != 0;
  drop_graph(p);
  return MSX_OK;
}

int msx_plan_check(msx_plan* p) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  int h = 0;
  MSX_CUDA(cudaDeviceSynchronize(), "synchronising the device");  // a copy alone does not wait for non-blocking streams
  MSX_CUDA(cudaMemcpy(&h, p->err, sizeof(int), cudaMemcpyDeviceToHost), "reading the plan error word");
  if (h) {
    MSX_CUDA(cudaMemset(p->err, 0, sizeof(int)), "clearing the plan error word");
    if (h & 2)  // bit 1: the paired row pass found its shared memory misaligned and did nothing
      return fail(MSX_ERR_CUDA, "the paired row pass found its shared memory misaligned (error word 0x%x)", h);
    return fail(MSX_ERR_TIMEOUT, "a pipelined pass gave up waiting for its tile copy (error word 0x%x)", h);
  }
  return MSX_OK;
}

int msx_plan_set_graph(msx_plan* p, int enable) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  p->use_graph = enable != 0;
  if (!p->use_graph) drop_graph(p);
  return MSX_OK;
}

int msx_multislice(msx_plan* p, const float* trans_dev, int num_slices, const float* psi_k_dev,
                   const double* normalization_dev, const float* positions_dev, int num_probes, float kmax,
                   double lambda, double slice_t, float k_band, float* cbed_out_dev, int crop_y, int crop_x,
                   void* stream) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  if (num_probes < 0 || num_slices < 0) return fail(MSX_ERR_INVALID, "negative probe or slice count");
  if (num_probes == 0) return MSX_OK;
  if (crop_y <= 0 || crop_x <= 0 || crop_y > p->ny || crop_x > p->nx)
    return fail(MSX_ERR_INVALID, "crop %d x %d outside the %d x %d grid", crop_y, crop_x, p->ny, p->nx);
  if (!psi_k_dev || !normalization_dev || !positions_dev || !cbed_out_dev || (num_slices > 0 && !trans_dev))
    return fail(MSX_ERR_INVALID, "null pointer");
  if (!aligned8({trans_dev, psi_k_dev, positions_dev, normalization_dev})) return fail(MSX_ERR_INVALID, kAlign8);
  if (!(kmax > 0) || !(lambda > 0) || !(slice_t >= 0) || !(k_band >= 0))
    return fail(MSX_ERR_INVALID, "kmax, lambda must be positive; slice thickness and k_band non-negative");
  int dev = 0;
  MSX_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev != p->device) return fail(MSX_ERR_INVALID, "plan belongs to device %d, current device is %d", p->device, dev);

  MsArgs a;
  std::memset(&a, 0, sizeof(a));  // the struct doubles as the graph cache key: no stray padding bytes
  a.trans = trans_dev; a.num_slices = num_slices; a.psik = psi_k_dev; a.norm = normalization_dev;
  a.pos = positions_dev; a.num_probes = num_probes; a.kmax = kmax; a.lambda = lambda; a.slice_t = slice_t;
  a.k_band = k_band; a.cbed = cbed_out_dev; a.crop_y = crop_y; a.crop_x = crop_x;
  a.group = p->group; a.row_sched = p->row_sched; a.col_sched = p->col_sched;
  cudaStream_t caller = (cudaStream_t)stream;
  int rc = MSX_OK;
  const bool captured = capturing(caller, &rc);
  if (rc != MSX_OK) return rc;
  if (captured) return enqueue_multislice(p, a, caller);
  return in_call_order(p, caller, p->use_graph, [&](cudaStream_t st) -> int {
    if (!p->use_graph || few_launches(p, a)) return enqueue_multislice(p, a, st);
    std::vector<unsigned char> key(sizeof(MsArgs));
    std::memcpy(key.data(), &a, sizeof(MsArgs));
    if (!p->gexec || key != p->gkey) {
      drop_graph(p);
      cudaGraph_t graph = nullptr;
      MSX_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
      const int rc = enqueue_multislice(p, a, st);
      cudaError_t e = cudaStreamEndCapture(st, &graph);
      if (rc != MSX_OK) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
      }
      if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
      e = cudaGraphInstantiate(&p->gexec, graph, 0);
      cudaGraphDestroy(graph);
      if (e != cudaSuccess) {
        p->gexec = nullptr;
        return cuda_fail(e, "cudaGraphInstantiate");
      }
      p->gkey = key;
    }
    MSX_CUDA(cudaGraphLaunch(p->gexec, st), "cudaGraphLaunch");
    return MSX_OK;
  });
}

int msx_multislice_detect(msx_plan* p, const float* trans_dev, int num_slices, const float* psi_k_dev,
                          const double* normalization_dev, const float* positions_dev, int num_probes, float kmax,
                          double lambda, double slice_t, float k_band, const float* detectors_dev, int num_detectors,
                          float* signals_out_dev, void* stream) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  if (num_probes < 0 || num_slices < 1) return fail(MSX_ERR_INVALID, "detector mode needs num_slices >= 1");
  if (num_probes == 0) return MSX_OK;
  if (num_detectors < 1 || num_detectors > kMaxDetectors)
    return fail(MSX_ERR_INVALID, "1..%d detectors supported, got %d", kMaxDetectors, num_detectors);
  if (!trans_dev || !psi_k_dev || !normalization_dev || !positions_dev || !detectors_dev || !signals_out_dev)
    return fail(MSX_ERR_INVALID, "null pointer");
  if (!aligned8({trans_dev, psi_k_dev, positions_dev, normalization_dev})) return fail(MSX_ERR_INVALID, kAlign8);
  if (!(kmax > 0) || !(lambda > 0) || !(slice_t >= 0) || !(k_band >= 0))
    return fail(MSX_ERR_INVALID, "kmax, lambda must be positive; slice thickness and k_band non-negative");
  MsArgs a;
  std::memset(&a, 0, sizeof(a));
  a.trans = trans_dev; a.num_slices = num_slices; a.psik = psi_k_dev; a.norm = normalization_dev;
  a.pos = positions_dev; a.num_probes = num_probes; a.kmax = kmax; a.lambda = lambda; a.slice_t = slice_t;
  a.k_band = k_band; a.crop_y = p->ny; a.crop_x = p->nx; a.group = p->group; a.row_sched = p->row_sched;
  a.col_sched = p->col_sched; a.det = detectors_dev; a.ndet = num_detectors; a.signals = signals_out_dev;
  const int waves = std::max(p->group, stream_group(p, a));  // of a group, whichever form runs
  const size_t need = (size_t)waves * (p->nx / p->col_ops->col_c) * num_detectors;
  if (need > p->partial_words) {
    if (p->partial) cudaFree(p->partial);
    p->partial = nullptr;
    p->partial_words = 0;
    if (cudaMalloc(&p->partial, need * sizeof(float)) != cudaSuccess)
      return fail(MSX_ERR_ALLOC, "detector partial sums allocation failed");
    p->partial_words = need;
  }
  drop_graph(p);  // the detector sequence is launched directly
  cudaStream_t caller = (cudaStream_t)stream;
  int rc = MSX_OK;
  const bool captured = capturing(caller, &rc);
  if (rc != MSX_OK) return rc;
  if (captured) return enqueue_multislice(p, a, caller);
  return in_call_order(p, caller, false, [&](cudaStream_t st) -> int { return enqueue_multislice(p, a, st); });
}

int msx_propagator_table(int ny, int nx, float kmax, double lambda, double slice_t, float k_band, float* ptab_out_dev,
                         void* stream) {
  if (ny < 2 || nx < 2 || ny > 65535 || !ptab_out_dev || !(kmax > 0) || !(lambda > 0) || !(slice_t >= 0))
    return fail(MSX_ERR_INVALID, "propagator table: bad arguments");
  MSX_CUDA(launch_ptab(ny, nx, kmax, lambda, slice_t, k_band, reinterpret_cast<float2*>(ptab_out_dev),
                       (cudaStream_t)stream), "propagator table");
  return MSX_OK;
}

int msx_plan_probe_waves(msx_plan* p, const float* psi_k_dev, const float* positions_dev, int num_probes, float kmax,
                         float* waves_out_dev, void* stream) {
  if (!p || num_probes < 0 || !psi_k_dev || !positions_dev || !waves_out_dev || !(kmax > 0))
    return fail(MSX_ERR_INVALID, "probe waves: bad arguments");
  if (!aligned8({psi_k_dev, positions_dev, waves_out_dev})) return fail(MSX_ERR_INVALID, kAlign8);
  if (num_probes == 0) return MSX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  ColArgs c{};
  c.psi = reinterpret_cast<float2*>(waves_out_dev); c.psik = reinterpret_cast<const float2*>(psi_k_dev);
  c.pos_yx = positions_dev; c.tw = p->tw_col; c.G = num_probes; c.Nx = p->nx; c.kmax = kmax; c.x_begin = 0;
  c.ncols = p->nx;
  MSX_CUDA(p->col_ops->col(COL_INIT, c, st), "probe formation pass");
  MSX_CUDA(p->row_ops->row_mode(ROW_I, c.psi, nullptr, p->tw_row, num_probes, p->ny, st), "inverse row transform");
  return MSX_OK;
}

int msx_plan_probe_stack(msx_plan* p, const float* psi_k_dev, const double* normalization_dev,
                         const float* positions_dev, int num_probes, float kmax, float* probes_out_dev, void* stream) {
  if (!p || num_probes < 0 || !psi_k_dev || !normalization_dev || !positions_dev || !probes_out_dev || !(kmax > 0))
    return fail(MSX_ERR_INVALID, "probe stack: bad arguments");
  if (!aligned8({psi_k_dev, normalization_dev, positions_dev, probes_out_dev}))
    return fail(MSX_ERR_INVALID, "probe stack: arrays must be 8-byte aligned");
  if (num_probes == 0) return MSX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  ColArgs c{};
  c.psi = reinterpret_cast<float2*>(probes_out_dev); c.psik = reinterpret_cast<const float2*>(psi_k_dev);
  c.pos_yx = positions_dev; c.tw = p->tw_col; c.G = num_probes; c.Nx = p->nx; c.kmax = kmax; c.x_begin = 0;
  c.ncols = p->nx; c.init_norm = normalization_dev;
  MSX_CUDA(p->col_ops->col(COL_INIT, c, st), "probe formation pass");
  MSX_CUDA(p->row_ops->row_mode(ROW_I, c.psi, nullptr, p->tw_row, num_probes, p->ny, st), "inverse row transform");
  return MSX_OK;
}

int msx_plan_step_waves(msx_plan* p, float* waves_dev, int num_waves, const float* trans_dev, const float* ptab_dev,
                        void* stream) {
  if (!p || num_waves < 0 || !waves_dev || !trans_dev || !ptab_dev) return fail(MSX_ERR_INVALID, "step waves: bad arguments");
  if (!aligned8({waves_dev, trans_dev, ptab_dev})) return fail(MSX_ERR_INVALID, kAlign8);
  if (num_waves == 0) return MSX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  float2* w = reinterpret_cast<float2*>(waves_dev);
  ColArgs c{};
  c.psi = w; c.ptab = reinterpret_cast<const float2*>(ptab_dev); c.tw = p->tw_col; c.G = num_waves; c.Nx = p->nx;
  c.x_begin = 0; c.ncols = p->nx;
  MSX_CUDA(p->row_ops->row_mode(ROW_TF, w, reinterpret_cast<const float2*>(trans_dev), p->tw_row, num_waves, p->ny, st),
           "transmit + forward row transform");
  MSX_CUDA(p->col_ops->col(COL_MID, c, st), "column pass");
  MSX_CUDA(p->row_ops->row_mode(ROW_I, w, nullptr, p->tw_row, num_waves, p->ny, st), "inverse row transform");
  return MSX_OK;
}

int msx_plan_cbed_waves(msx_plan* p, float* waves_dev, int num_waves, const double* normalization_dev,
                        float* cbed_out_dev, int crop_y, int crop_x, void* stream) {
  if (!p || num_waves < 0 || !waves_dev || !normalization_dev || !cbed_out_dev || crop_y <= 0 || crop_x <= 0 ||
      crop_y > p->ny || crop_x > p->nx)
    return fail(MSX_ERR_INVALID, "cbed of waves: bad arguments");
  if (!aligned8({waves_dev, normalization_dev})) return fail(MSX_ERR_INVALID, kAlign8);
  if (num_waves == 0) return MSX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int rc = ensure_inv_n(p);
  if (rc != MSX_OK) return rc;
  float2* w = reinterpret_cast<float2*>(waves_dev);
  MSX_CUDA(p->row_ops->row_mode(ROW_F, w, nullptr, p->tw_row, num_waves, p->ny, st), "forward row transform");
  ColArgs c{};
  c.psi = w; c.ptab = p->inv_n; c.tw = p->tw_col; c.norm = normalization_dev; c.cbed = cbed_out_dev; c.G = num_waves;
  c.Nx = p->nx; c.x_begin = p->nx / 2 - crop_x / 2; c.ncols = crop_x; c.y0 = p->ny / 2 - crop_y / 2; c.crop_y = crop_y;
  MSX_CUDA(p->col_ops->col(COL_FINAL, c, st), "final column pass");
  return MSX_OK;
}

int msx_multislice_host(msx_plan* p, const float* trans_host, int num_slices, const float* psi_k_host,
                        double normalization, const float* positions_host, int num_probes, float kmax, double lambda,
                        double slice_t, float k_band, float* cbed_host, int crop_y, int crop_x, void* stream) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  if (num_probes < 0 || num_slices < 0) return fail(MSX_ERR_INVALID, "negative probe or slice count");
  if (num_probes == 0) return MSX_OK;
  if (crop_y <= 0 || crop_x <= 0 || crop_y > p->ny || crop_x > p->nx)
    return fail(MSX_ERR_INVALID, "crop %d x %d outside the %d x %d grid", crop_y, crop_x, p->ny, p->nx);
  if (!psi_k_host || !positions_host || !cbed_host || (num_slices > 0 && !trans_host))
    return fail(MSX_ERR_INVALID, "null pointer");
  if (!(normalization > 0) || !(kmax > 0) || !(lambda > 0) || !(slice_t >= 0) || !(k_band >= 0))
    return fail(MSX_ERR_INVALID, "normalisation, kmax, lambda must be positive; slice thickness and k_band non-negative");
  int dev = 0;
  MSX_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev != p->device) return fail(MSX_ERR_INVALID, "plan belongs to device %d, current device is %d", p->device, dev);
  if (!p->copy) {
    MSX_CUDA(cudaStreamCreateWithFlags(&p->copy, cudaStreamNonBlocking), "copy stream");
    MSX_CUDA(cudaEventCreateWithFlags(&p->ev_copy, cudaEventDisableTiming), "cudaEventCreate");
  }
  const size_t wave = (size_t)p->ny * p->nx, pattern = (size_t)crop_y * crop_x;
  int rc = grow(&p->io_trans, &p->io_trans_words, wave * num_slices, "transmission slices");
  if (rc == MSX_OK) rc = grow(&p->io_psik, &p->io_psik_words, wave, "k-space probe");
  if (rc == MSX_OK) rc = grow(&p->io_pos, &p->io_pos_words, 2 * (size_t)num_probes, "positions");
  size_t one = p->io_norm ? 1 : 0;
  if (rc == MSX_OK) rc = grow(&p->io_norm, &one, 1, "normalisation");
  if (rc == MSX_OK) rc = grow(&p->io_cbed, &p->io_cbed_words, pattern * num_probes, "CBED stack");
  if (rc != MSX_OK) return rc;

  cudaStream_t caller = (cudaStream_t)stream, w = p->work, cp = p->copy;
  // The whole call is captured into a CUDA graph and replayed while its
  // arguments (host and device buffers included) repeat, when every host buffer
  // is page-locked: copies from pageable memory stay outside graphs.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  MSX_CUDA(cudaStreamIsCapturing(caller, &cap), "cudaStreamIsCapturing");
  auto locked = [](const void* q) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, q) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return at.type == cudaMemoryTypeHost;
  };
  const bool graph = p->use_graph && cap == cudaStreamCaptureStatusNone && locked(psi_k_host) &&
                     locked(positions_host) && locked(cbed_host) && (num_slices == 0 || locked(trans_host));
  struct HostKey {
    const void *trans, *psik, *pos, *cbed, *d_trans, *d_psik, *d_pos, *d_norm, *d_cbed;
    double normalization, lambda, slice_t;
    float kmax, k_band;
    int num_slices, num_probes, crop_y, crop_x, group, row_sched, col_sched, tma;
  } hk;
  std::memset(&hk, 0, sizeof(hk));  // the struct is the cache key: no stray padding bytes
  hk.trans = trans_host; hk.psik = psi_k_host; hk.pos = positions_host; hk.cbed = cbed_host;
  hk.d_trans = p->io_trans; hk.d_psik = p->io_psik; hk.d_pos = p->io_pos; hk.d_norm = p->io_norm;
  hk.d_cbed = p->io_cbed; hk.normalization = normalization; hk.lambda = lambda; hk.slice_t = slice_t;
  hk.kmax = kmax; hk.k_band = k_band; hk.num_slices = num_slices; hk.num_probes = num_probes; hk.crop_y = crop_y;
  hk.crop_x = crop_x; hk.group = p->group; hk.row_sched = p->row_sched; hk.col_sched = p->col_sched;
  hk.tma = (p->use_tma ? 1 : 0) + (p->use_stream ? 2 : 0) + (p->use_resident ? 4 : 0) + (p->use_few ? 8 : 0);
  std::vector<unsigned char> key(sizeof(hk));
  std::memcpy(key.data(), &hk, sizeof(hk));
  // everything here follows the caller's earlier work and this plan's earlier calls
  MSX_CUDA(cudaEventRecord(p->ev_in, caller), "cudaEventRecord");
  MSX_CUDA(cudaStreamWaitEvent(w, p->ev_in, 0), "cudaStreamWaitEvent");
  if (cap == cudaStreamCaptureStatusNone) {
    rc = after_last_call(p, w);
    if (rc != MSX_OK) return rc;
  }
  if (graph && p->gexec_host && key == p->gkey_host) {
    MSX_CUDA(cudaGraphLaunch(p->gexec_host, w), "cudaGraphLaunch");
    MSX_CUDA(cudaEventRecord(p->ev_last, w), "cudaEventRecord");
    MSX_CUDA(cudaStreamWaitEvent(caller, p->ev_last, 0), "cudaStreamWaitEvent");
    return MSX_OK;
  }
  if (graph) {
    if (p->gexec_host) cudaGraphExecDestroy(p->gexec_host);
    p->gexec_host = nullptr;
    p->gkey_host.clear();
    MSX_CUDA(cudaStreamBeginCapture(w, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
  }
  MsArgs a;
  std::memset(&a, 0, sizeof(a));
  a.trans = reinterpret_cast<const float*>(p->io_trans); a.num_slices = num_slices;
  a.psik = reinterpret_cast<const float*>(p->io_psik); a.norm = p->io_norm; a.pos = p->io_pos;
  a.num_probes = num_probes; a.kmax = kmax; a.lambda = lambda; a.slice_t = slice_t; a.k_band = k_band;
  a.cbed = p->io_cbed; a.crop_y = crop_y; a.crop_x = crop_x;
  a.group = p->group; a.row_sched = p->row_sched; a.col_sched = p->col_sched;
  const bool cluster = resident_cluster(p, a) > 0;
  const int streamed = cluster ? 0 : stream_group(p, a), step = cluster ? num_probes : streamed ? streamed : p->group;
  const int ngroups = (num_probes + step - 1) / step;
  const int chunk = 8;
  const int nchunks = (num_slices + chunk - 1) / chunk;
  std::vector<cudaEvent_t> chunk_ev(nchunks + 1, nullptr), group_ev;
  auto release = [&]() {  // events still pending are released when they complete
    for (cudaEvent_t e : chunk_ev) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : group_ev) if (e) cudaEventDestroy(e);
  };
  // everything between the start and the end of a capture: any failure returns
  // through here, so that the capture is always ended
  auto run = [&]() -> int {
    group_ev.resize(ngroups, nullptr);
    for (auto& e : chunk_ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return fail(MSX_ERR_CUDA, "cudaEventCreate");
    for (auto& e : group_ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return fail(MSX_ERR_CUDA, "cudaEventCreate");
    // the copy stream forks from the work stream (joining the capture, if any)
    MSX_CUDA(cudaEventRecord(p->ev_out, w), "cudaEventRecord");
    MSX_CUDA(cudaStreamWaitEvent(cp, p->ev_out, 0), "cudaStreamWaitEvent");
    MSX_CUDA(cudaMemcpyAsync(p->io_psik, psi_k_host, sizeof(float2) * wave, cudaMemcpyHostToDevice, cp), "probe upload");
    MSX_CUDA(cudaMemcpyAsync(p->io_pos, positions_host, sizeof(float) * 2 * num_probes, cudaMemcpyHostToDevice, cp),
             "position upload");
    // by value through a launch argument: no host memory to keep alive, no staging
    MSX_CUDA(launch_store_double(p->io_norm, normalization, cp), "normalisation");
    MSX_CUDA(cudaEventRecord(chunk_ev[nchunks], cp), "cudaEventRecord");
    for (int i = 0; i < nchunks; ++i) {
      const int s0 = i * chunk, s1 = (s0 + chunk < num_slices) ? s0 + chunk : num_slices;
      MSX_CUDA(cudaMemcpyAsync(p->io_trans + (size_t)s0 * wave, trans_host + 2 * (size_t)s0 * wave,
                               sizeof(float2) * (size_t)(s1 - s0) * wave, cudaMemcpyHostToDevice, cp),
               "slice upload");
      MSX_CUDA(cudaEventRecord(chunk_ev[i], cp), "cudaEventRecord");
    }
    MSX_CUDA(cudaStreamWaitEvent(w, chunk_ev[nchunks], 0), "cudaStreamWaitEvent");
    HostPipe hp{cp, chunk, &chunk_ev, &group_ev, cbed_host, pattern};
    int r = enqueue_multislice(p, a, w, &hp);
    if (r != MSX_OK) return r;
    // the copy stream joins back: the work stream (and through it the caller) waits for the downloads
    MSX_CUDA(cudaEventRecord(p->ev_copy, cp), "cudaEventRecord");
    MSX_CUDA(cudaStreamWaitEvent(w, p->ev_copy, 0), "cudaStreamWaitEvent");
    return MSX_OK;
  };
  rc = run();
  if (graph) {
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(w, &g);
    release();
    if (rc != MSX_OK) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
    const cudaError_t e2 = cudaGraphInstantiate(&p->gexec_host, g, 0);
    cudaGraphDestroy(g);
    if (e2 != cudaSuccess) {
      p->gexec_host = nullptr;
      return cuda_fail(e2, "cudaGraphInstantiate");
    }
    p->gkey_host = key;
    MSX_CUDA(cudaGraphLaunch(p->gexec_host, w), "cudaGraphLaunch");
  } else {
    release();
  }
  if (rc != MSX_OK) return rc;
  cudaEvent_t done = cap == cudaStreamCaptureStatusNone ? p->ev_last : p->ev_out;
  MSX_CUDA(cudaEventRecord(done, w), "cudaEventRecord");
  MSX_CUDA(cudaStreamWaitEvent(caller, done, 0), "cudaStreamWaitEvent");
  return MSX_OK;
}

int msx_plan_profile(msx_plan* p, const float* trans_dev, int num_slices, const float* psi_k_dev,
                     const double* normalization_dev, const float* positions_dev, int num_probes, float kmax,
                     double lambda, double slice_t, float k_band, int iters, float* ms_out, void* stream) {
  if (!p || !ms_out) return fail(MSX_ERR_INVALID, "null plan or output");
  if (iters <= 0 || num_slices <= 0 || num_probes <= 0 || !trans_dev || !psi_k_dev || !normalization_dev || !positions_dev)
    return fail(MSX_ERR_INVALID, "profile needs slices, probes, inputs and iters > 0");
  if (!aligned8({trans_dev, psi_k_dev, positions_dev, normalization_dev})) return fail(MSX_ERR_INVALID, kAlign8);
  const int ny = p->ny, nx = p->nx;
  const int gn = num_probes < p->group ? num_probes : p->group;
  if (!workspace_holds(p, gn))
    return fail(MSX_ERR_ALLOC, "the plan's workspace does not hold %d waves (an earlier allocation failed)", gn);
  const size_t wave = (size_t)ny * nx;
  cudaStream_t st = (cudaStream_t)stream;
  int rcp = ensure_ptab(p);
  if (rcp == MSX_OK) rcp = after_last_call(p, st);
  if (rcp != MSX_OK) return rcp;
  cudaEvent_t ev[4];
  for (auto& e : ev) MSX_CUDA(cudaEventCreate(&e), "cudaEventCreate");
  MSX_CUDA(launch_ptab(ny, nx, kmax, lambda, slice_t, k_band, p->ptab, st), "propagator table");
  MSX_CUDA(launch_pfac(ny, nx, kmax, lambda, slice_t, k_band, p->pyx, p->band, st), "propagator factors");
  ColArgs c{};
  c.psi = p->psi; c.ptab = p->ptab; c.psik = reinterpret_cast<const float2*>(psi_k_dev); c.pos_yx = positions_dev;
  c.tw = p->tw_col; c.norm = normalization_dev; c.cbed = nullptr; c.G = gn; c.Nx = nx; c.kmax = kmax;
  c.x_begin = 0; c.ncols = nx; c.y0 = 0; c.crop_y = 0;
  MSX_CUDA(p->col_ops->col(COL_INIT, c, st), "probe formation pass");
  float row_ms = 0, col_ms = 0;
  const float2* trans = reinterpret_cast<const float2*>(trans_dev);
  // the steady-state passes of multislice: the band-limited column range
  int bx_lo = 0, bx_hi = 0;
  band_columns(nx, kmax, k_band, p->col_ops->col_c, &bx_lo, &bx_hi);
  const bool tma = tma_passes(p, trans_dev);
  for (int i = 0; i < iters; ++i) {
    const int s = i % num_slices;
    MSX_CUDA(cudaEventRecord(ev[0], st), "cudaEventRecord");
    int rc = slice_passes(p, trans + (size_t)s * wave, gn, c, false, st, bx_lo, bx_hi, tma);
    if (rc != MSX_OK) return rc;
    MSX_CUDA(cudaEventRecord(ev[1], st), "cudaEventRecord");
    if (tma) {
      TmaPassArgs ta{};
      ta.psi = p->psi; ta.tw = p->tw_col; ta.pyx = p->pyx; ta.band = p->band; ta.err = p->err;
      ta.G = gn; ta.Ny = ny; ta.Nx = nx; ta.x_lo = bx_lo; ta.x_hi = bx_hi;
      MSX_CUDA(p->col_ops->col_tma(p->map, ta, p->col_ctas, st), "column pass");
    } else {
      MSX_CUDA(p->col_ops->col(COL_MID, c, st), "column pass");
    }
    MSX_CUDA(cudaEventRecord(ev[2], st), "cudaEventRecord");
    MSX_CUDA(cudaEventSynchronize(ev[2]), "cudaEventSynchronize");
    float a = 0, b = 0;
    MSX_CUDA(cudaEventElapsedTime(&a, ev[0], ev[1]), "cudaEventElapsedTime");
    MSX_CUDA(cudaEventElapsedTime(&b, ev[1], ev[2]), "cudaEventElapsedTime");
    row_ms += a;
    col_ms += b;
  }
  for (auto& e : ev) cudaEventDestroy(e);
  ms_out[0] = row_ms / iters;
  ms_out[1] = col_ms / iters;
  ms_out[2] = (float)gn;
  return MSX_OK;
}

int msx_plan_autotune(msx_plan* p, const float* trans_dev, int num_slices, const float* psi_k_dev,
                      const double* normalization_dev, const float* positions_dev, int num_probes, float kmax,
                      double lambda, double slice_t, float k_band, int iters, size_t max_workspace_bytes,
                      float* best_ns_per_wave_slice, void* stream) {
  if (!p) return fail(MSX_ERR_INVALID, "null plan");
  if (iters <= 0 || num_slices <= 0 || num_probes <= 0 || !trans_dev || !psi_k_dev || !normalization_dev || !positions_dev)
    return fail(MSX_ERR_INVALID, "autotune needs slices, probes, inputs and iters > 0");
  if (!aligned8({trans_dev, psi_k_dev, positions_dev, normalization_dev})) return fail(MSX_ERR_INVALID, kAlign8);
  int rcp = ensure_ptab(p);
  if (rcp == MSX_OK) rcp = after_last_call(p, (cudaStream_t)stream);
  if (rcp != MSX_OK) return rcp;
  const SchedOps *rops, *cops;
  const int nr = schedule_table(p->nx, &rops), nc = schedule_table(p->ny, &cops);
  const size_t wave_bytes = sizeof(float2) * (size_t)p->ny * p->nx;
  if (max_workspace_bytes == 0) max_workspace_bytes = (size_t)1 << 30;
  // candidate groups: resident sets of 8 MiB .. 1 GiB, and every probe at once
  std::vector<int> groups;
  for (size_t mb : {8, 16, 32, 48, 64, 128, 256, 512, 1024}) {
    size_t g = (mb << 20) / wave_bytes;
    if (g < 1) g = 1;
    if (g > (size_t)num_probes) g = (size_t)num_probes;
    if (g * wave_bytes > max_workspace_bytes) continue;
    if (groups.empty() || groups.back() != (int)g) groups.push_back((int)g);
  }
  if (groups.empty()) groups.push_back(1);
  cudaStream_t st = (cudaStream_t)stream;
  cudaEvent_t e0, e1;
  MSX_CUDA(cudaEventCreate(&e0), "cudaEventCreate");
  MSX_CUDA(cudaEventCreate(&e1), "cudaEventCreate");
  const float2* trans = reinterpret_cast<const float2*>(trans_dev);
  const size_t wave = (size_t)p->ny * p->nx;
  // The row and column passes only share the group size, so for every group the
  // best row schedule and the best column schedule are found separately.
  float best = 1e30f;
  int br = p->row_sched, bc = p->col_sched, bg = p->group;
  int rc = MSX_OK;
  auto time_loop = [&](bool row_pass, int g, float* ms) -> int {
    ColArgs c{};
    c.psi = p->psi; c.ptab = p->ptab; c.psik = reinterpret_cast<const float2*>(psi_k_dev); c.pos_yx = positions_dev;
    c.tw = p->tw_col; c.norm = normalization_dev; c.G = g; c.Nx = p->nx; c.kmax = kmax; c.x_begin = 0; c.ncols = p->nx;
    MSX_CUDA(p->col_ops->col(COL_INIT, c, st), "probe formation pass");
    int bx_lo = 0, bx_hi = 0;  // time the steady-state (band-limited) passes
    band_columns(p->nx, kmax, k_band, p->col_ops->col_c, &bx_lo, &bx_hi);
    for (int pass = 0; pass < 2; ++pass) {  // pass 0 warms caches and clocks
      MSX_CUDA(cudaEventRecord(e0, st), "cudaEventRecord");
      for (int i = 0; i < iters; ++i) {
        if (row_pass) {
          const int r2 = slice_passes(p, trans + (size_t)(i % num_slices) * wave, g, c, false, st, bx_lo, bx_hi,
                                       tma_passes(p, trans));
          if (r2 != MSX_OK) return r2;
        } else if (tma_passes(p, trans)) {
          TmaPassArgs ta{};
          ta.psi = p->psi; ta.tw = p->tw_col; ta.pyx = p->pyx; ta.band = p->band; ta.err = p->err;
          ta.G = g; ta.Ny = p->ny; ta.Nx = p->nx; ta.x_lo = bx_lo; ta.x_hi = bx_hi;
          MSX_CUDA(p->col_ops->col_tma(p->map, ta, p->col_ctas, st), "column pass");
        } else {
          MSX_CUDA(p->col_ops->col(COL_MID, c, st), "column pass");
        }
      }
      MSX_CUDA(cudaEventRecord(e1, st), "cudaEventRecord");
    }
    MSX_CUDA(cudaEventSynchronize(e1), "cudaEventSynchronize");
    MSX_CUDA(cudaEventElapsedTime(ms, e0, e1), "cudaEventElapsedTime");
    return MSX_OK;
  };
  for (int g : groups) {
    float best_row = 1e30f, best_col = 1e30f;
    int gr = 0, gc = 0;
    for (int r = 0; r < nr && rc == MSX_OK; ++r) {
      rc = msx_plan_set_schedule(p, r, 0, g);
      if (rc != MSX_OK) break;
      MSX_CUDA(launch_ptab(p->ny, p->nx, kmax, lambda, slice_t, k_band, p->ptab, st), "propagator table");
      MSX_CUDA(launch_pfac(p->ny, p->nx, kmax, lambda, slice_t, k_band, p->pyx, p->band, st), "propagator factors");
      float ms = 0;
      rc = time_loop(true, g, &ms);
      if (rc == MSX_OK && ms < best_row) { best_row = ms; gr = r; }
    }
    for (int cidx = 0; cidx < nc && rc == MSX_OK; ++cidx) {
      rc = msx_plan_set_schedule(p, gr, cidx, g);
      if (rc != MSX_OK) break;
      MSX_CUDA(launch_ptab(p->ny, p->nx, kmax, lambda, slice_t, k_band, p->ptab, st), "propagator table");
      MSX_CUDA(launch_pfac(p->ny, p->nx, kmax, lambda, slice_t, k_band, p->pyx, p->band, st), "propagator factors");
      float ms = 0;
      rc = time_loop(false, g, &ms);
      if (rc == MSX_OK && ms < best_col) { best_col = ms; gc = cidx; }
    }
    if (rc != MSX_OK) break;
    const float ns = (best_row + best_col) * 1e6f / ((float)iters * (float)g);
    if (ns < best) { best = ns; br = gr; bc = gc; bg = g; }
  }
  if (rc == MSX_OK) rc = msx_plan_set_schedule(p, br, bc, bg);
  if (rc == MSX_OK) {  // the all-slices kernel on the same inputs, where the call would take it
    MsArgs a;
    std::memset(&a, 0, sizeof(a));
    a.trans = trans_dev; a.num_slices = num_slices; a.num_probes = num_probes; a.kmax = kmax; a.lambda = lambda;
    a.slice_t = slice_t; a.k_band = k_band; a.group = p->group;
    p->use_stream = p->use_resident = true;  // per call, unless the timing below is against the former
    const int g = stream_group(p, a), s = num_slices < iters ? num_slices : iters;
    if (g > 0 && workspace_holds(p, g)) {
      ColArgs c{};
      c.psi = p->psi; c.psik = reinterpret_cast<const float2*>(psi_k_dev); c.pos_yx = positions_dev; c.tw = p->tw_col;
      c.G = g; c.Nx = p->nx; c.kmax = kmax; c.ncols = p->nx;
      rc = [&]() -> int {
        MSX_CUDA(p->col_ops->col(COL_INIT, c, st), "probe formation pass");
        for (int pass = 0; pass < 2; ++pass) {
          MSX_CUDA(cudaEventRecord(e0, st), "cudaEventRecord");
          const int r2 = stream_slices(p, a, 0, s, true, g, st);
          if (r2 != MSX_OK) return r2;
          MSX_CUDA(cudaEventRecord(e1, st), "cudaEventRecord");
        }
        MSX_CUDA(cudaEventSynchronize(e1), "cudaEventSynchronize");
        float ms = 0;
        MSX_CUDA(cudaEventElapsedTime(&ms, e0, e1), "cudaEventElapsedTime");
        const float ns = ms * 1e6f / ((float)s * (float)g);
        if (ns < best) best = ns;
        else p->use_stream = false;
        return MSX_OK;
      }();
    }
    // the winners stand for groups of bg waves: calls of few lines keep their schedules
    // unless the timing was of few lines itself
    int lo = 0, hi = 0;
    p->use_few = true;
    if (few_rows(p, bg) || few_cols(p, bg, kmax, k_band, &lo, &hi)) p->use_few = false;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc != MSX_OK) return rc;
  if (best_ns_per_wave_slice) *best_ns_per_wave_slice = best;
  return rc;
}

}  // extern "C"

// ============================================================================ uneven batches
// A batch runs many independent jobs (crystals of different grid size,
// thickness, voltage and probe count) as one CUDA graph: the jobs are spread
// over `branches` parallel streams inside the capture (longest first onto the
// least loaded branch), each branch owning one plan per grid size, so the GPU
// overlaps jobs of different shapes.  The graph is replayed while the job list
// repeats.
struct msx_batch {
  int branches = 4;
  int device = 0;
  std::vector<std::vector<std::pair<long long, msx_plan*>>> plans;  // per branch: (ny<<32|nx, plan)
  std::vector<cudaStream_t> streams;
  std::vector<cudaEvent_t> events;  // fork/join events, 2 per branch
  cudaStream_t origin = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  cudaGraphExec_t gexec = nullptr;
  std::vector<unsigned char> gkey;
  std::vector<std::pair<long long, std::array<int, 4>>> sched;  // (ny<<32|nx) -> row, col, group, forms
};

namespace {

// Forms besides the two passes with the given schedules that a plan may take: 1 the
// all-slices kernel, 2 clusters, 4 the schedules of few lines.
void allow_forms(msx_plan* p, int forms) {
  p->use_stream = (forms & 1) != 0;
  p->use_resident = (forms & 2) != 0;
  p->use_few = (forms & 4) != 0;
}
int allowed_forms(const msx_plan* p) {
  return (p->use_stream ? 1 : 0) + (p->use_resident ? 2 : 0) + (p->use_few ? 4 : 0);
}

// Persistent passes amortise their start-up over large groups: up to 1 GiB of
// waves per branch (the jobs of a branch run one after another).
int batch_waves(int ny, int nx) {
  const int g = (int)(((size_t)1 << 30) / (sizeof(float2) * (size_t)ny * nx));
  return g < 2 ? 2 : g;
}

msx_plan* batch_plan(msx_batch* b, int branch, int ny, int nx, int* rc) {
  const long long key = ((long long)ny << 32) | (unsigned)nx;
  for (auto& kv : b->plans[branch])
    if (kv.first == key) return kv.second;
  int group = batch_waves(ny, nx), waves = group;
  int r = 0, c = 0;
  bool tuned = false;  // schedules set for this grid (else the plan's defaults)
  int forms = 0;
  for (auto& kv : b->sched)
    if (kv.first == key) {
      r = kv.second[0]; c = kv.second[1]; tuned = true; forms = kv.second[3];
      if (kv.second[2] > 0) group = kv.second[2];
      // forms that choose their own groups need the room that the tuned plan had
      if (!(forms & 3) || waves < group) waves = group;
    }
  msx_plan* p = nullptr;
  *rc = msx_plan_create(ny, nx, waves, &p);
  if (*rc == MSX_ERR_ALLOC && group < waves) *rc = msx_plan_create(ny, nx, group, &p);  // the passes need no more
  if (*rc != MSX_OK) return nullptr;
  if (tuned) {
    *rc = msx_plan_set_schedule(p, r, c, group);
    if (*rc != MSX_OK) { msx_plan_destroy(p); return nullptr; }
    allow_forms(p, forms);
  }
  b->plans[branch].push_back({key, p});
  return p;
}

int batch_set_schedule(msx_batch* b, int ny, int nx, int row_schedule, int col_schedule, int group, int forms) {
  if (!b) return fail(MSX_ERR_INVALID, "null batch");
  if (!msx_supported_size(ny) || !msx_supported_size(nx)) return fail(MSX_ERR_UNSUPPORTED, "grid %d x %d", ny, nx);
  if (row_schedule < 0 || row_schedule >= msx_num_schedules(nx) || col_schedule < 0 ||
      col_schedule >= msx_num_schedules(ny) || group < 0)
    return fail(MSX_ERR_INVALID, "schedule (%d, %d, group %d) out of range", row_schedule, col_schedule, group);
  const long long key = ((long long)ny << 32) | (unsigned)nx;
  bool found = false;
  for (auto& kv : b->sched)
    if (kv.first == key) { kv.second = {row_schedule, col_schedule, group, forms}; found = true; }
  if (!found) b->sched.push_back({key, {row_schedule, col_schedule, group, forms}});
  for (auto& br : b->plans)
    for (auto& kv : br)
      if (kv.first == key) {
        int rc = msx_plan_set_schedule(kv.second, row_schedule, col_schedule, group);
        if (rc != MSX_OK) return rc;
        allow_forms(kv.second, forms);
        if (forms & 3) {
          rc = ensure_workspace(kv.second, (size_t)batch_waves(ny, nx));  // or the forms go without
          if (rc == MSX_OK || rc == MSX_ERR_ALLOC) rc = prepare_tma(kv.second);
          if (rc != MSX_OK) return rc;
        }
      }
  if (b->gexec) cudaGraphExecDestroy(b->gexec);
  b->gexec = nullptr;
  b->gkey.clear();
  return MSX_OK;
}

}  // namespace

extern "C" {

int msx_batch_create(int branches, msx_batch** out) {
  if (!out) return fail(MSX_ERR_INVALID, "null batch pointer");
  *out = nullptr;
  if (branches < 0 || branches > 16) return fail(MSX_ERR_INVALID, "branches must be 0..16");
  msx_batch* b = new msx_batch();
  b->branches = branches ? branches : 4;
  cudaError_t e = cudaGetDevice(&b->device);
  b->plans.resize(b->branches);
  b->streams.resize(b->branches, nullptr);
  b->events.resize(2 * b->branches, nullptr);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->origin, cudaStreamNonBlocking);
  for (int i = 0; i < b->branches && e == cudaSuccess; ++i) e = cudaStreamCreateWithFlags(&b->streams[i], cudaStreamNonBlocking);
  for (auto& ev : b->events)
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_in, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_out, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    msx_batch_destroy(b);
    return cuda_fail(e, "batch streams/events");
  }
  *out = b;
  return MSX_OK;
}

int msx_batch_destroy(msx_batch* b) {
  if (!b) return MSX_OK;
  if (b->gexec) cudaGraphExecDestroy(b->gexec);
  for (auto& br : b->plans)
    for (auto& kv : br) msx_plan_destroy(kv.second);
  for (auto s : b->streams)
    if (s) cudaStreamDestroy(s);
  for (auto ev : b->events)
    if (ev) cudaEventDestroy(ev);
  if (b->ev_in) cudaEventDestroy(b->ev_in);
  if (b->ev_out) cudaEventDestroy(b->ev_out);
  if (b->origin) cudaStreamDestroy(b->origin);
  delete b;
  return MSX_OK;
}

int msx_batch_set_schedule(msx_batch* b, int ny, int nx, int row_schedule, int col_schedule, int group) {
  return batch_set_schedule(b, ny, nx, row_schedule, col_schedule, group, 0);
}

int msx_batch_autotune(msx_batch* b, const msx_job* jobs, int njobs, int iters, void* stream) {
  if (!b || (!jobs && njobs > 0) || njobs < 0 || iters <= 0) return fail(MSX_ERR_INVALID, "bad batch autotune arguments");
  // one representative per grid: the job with the most positions (ties: the first)
  std::vector<int> rep;
  for (int i = 0; i < njobs; ++i) {
    const msx_job& j = jobs[i];
    if (j.num_slices <= 0 || j.num_probes <= 0) continue;
    bool seen = false;
    for (int& r : rep)
      if (jobs[r].ny == j.ny && jobs[r].nx == j.nx) {
        seen = true;
        if (j.num_probes > jobs[r].num_probes) r = i;
      }
    if (!seen) rep.push_back(i);
  }
  for (int r : rep) {
    const msx_job& j = jobs[r];
    msx_plan* p = nullptr;
    int rc = msx_plan_create(j.ny, j.nx, 0, &p);
    if (rc != MSX_OK) return rc;
    // the batch keeps at most 1 GiB of waves per plan and branch
    rc = msx_plan_autotune(p, j.trans_dev, j.num_slices, j.psi_k_dev, j.normalization_dev, j.positions_dev,
                           j.num_probes, j.kmax, j.lambda, j.slice_t, j.k_band, iters, (size_t)1 << 30, nullptr,
                           stream);
    int row = 0, col = 0, group = 0;
    if (rc == MSX_OK) rc = msx_plan_get_schedule(p, &row, &col, &group);
    const int forms = rc == MSX_OK ? allowed_forms(p) : 0;
    msx_plan_destroy(p);
    if (rc == MSX_OK) rc = batch_set_schedule(b, j.ny, j.nx, row, col, group, forms);
    if (rc != MSX_OK) return rc;
  }
  return MSX_OK;
}

int msx_batch_run(msx_batch* b, const msx_job* jobs, int njobs, void* stream) {
  if (!b) return fail(MSX_ERR_INVALID, "null batch");
  if (njobs < 0 || (njobs > 0 && !jobs)) return fail(MSX_ERR_INVALID, "bad job list");
  if (njobs == 0) return MSX_OK;
  int dev = 0;
  MSX_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev != b->device) return fail(MSX_ERR_INVALID, "batch belongs to device %d, current device is %d", b->device, dev);
  for (int i = 0; i < njobs; ++i) {
    const msx_job& j = jobs[i];
    if (!msx_supported_size(j.ny) || !msx_supported_size(j.nx))
      return fail(MSX_ERR_UNSUPPORTED, "job %d: grid %d x %d", i, j.ny, j.nx);
    if (j.num_probes < 0 || j.num_slices < 0 || j.crop_y <= 0 || j.crop_x <= 0 || j.crop_y > j.ny || j.crop_x > j.nx)
      return fail(MSX_ERR_INVALID, "job %d: bad probe/slice count or crop", i);
    if (j.num_probes > 0 && (!j.psi_k_dev || !j.normalization_dev || !j.positions_dev || !j.cbed_out_dev ||
                             (j.num_slices > 0 && !j.trans_dev)))
      return fail(MSX_ERR_INVALID, "job %d: null pointer", i);
    if (j.num_probes > 0 && !aligned8({j.trans_dev, j.psi_k_dev, j.positions_dev, j.normalization_dev}))
      return fail(MSX_ERR_INVALID, "job %d: %s", i, kAlign8);
    if (!(j.kmax > 0) || !(j.lambda > 0) || !(j.slice_t >= 0) || !(j.k_band >= 0))
      return fail(MSX_ERR_INVALID, "job %d: kmax, lambda must be positive", i);
  }
  cudaStream_t caller = (cudaStream_t)stream;
  std::vector<unsigned char> key(sizeof(msx_job) * (size_t)njobs);
  std::memcpy(key.data(), jobs, key.size());
  if (!b->gexec || key != b->gkey) {
    if (b->gexec) cudaGraphExecDestroy(b->gexec);
    b->gexec = nullptr;
    b->gkey.clear();
    // longest job first onto the least loaded branch
    std::vector<int> order(njobs);
    for (int i = 0; i < njobs; ++i) order[i] = i;
    auto cost = [&](int i) {
      const msx_job& j = jobs[i];
      const double n = (double)j.ny * j.nx;
      return (double)j.num_probes * (j.num_slices + 1) * n * std::log2(n);
    };
    std::sort(order.begin(), order.end(), [&](int x, int y) { return cost(x) > cost(y); });
    std::vector<double> load(b->branches, 0.0);
    std::vector<std::vector<int>> assign(b->branches);
    for (int i : order) {
      int best = 0;
      for (int k = 1; k < b->branches; ++k)
        if (load[k] < load[best]) best = k;
      load[best] += cost(i);
      assign[best].push_back(i);
    }
    // plans are created (allocating) before the capture
    for (int k = 0; k < b->branches; ++k)
      for (int i : assign[k]) {
        int rc = MSX_OK;
        if (!batch_plan(b, k, jobs[i].ny, jobs[i].nx, &rc)) return rc;
      }
    cudaGraph_t graph = nullptr;
    MSX_CUDA(cudaStreamBeginCapture(b->origin, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
    int rc = MSX_OK;
    for (int k = 0; k < b->branches && rc == MSX_OK; ++k) {
      cudaError_t e = cudaEventRecord(b->events[2 * k], b->origin);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(b->streams[k], b->events[2 * k], 0);
      if (e != cudaSuccess) rc = cuda_fail(e, "batch fork");
      for (int i : assign[k]) {
        if (rc != MSX_OK) break;
        const msx_job& j = jobs[i];
        if (j.num_probes == 0) continue;
        msx_plan* p = batch_plan(b, k, j.ny, j.nx, &rc);
        MsArgs a;
        std::memset(&a, 0, sizeof(a));
        a.trans = j.trans_dev; a.num_slices = j.num_slices; a.psik = j.psi_k_dev; a.norm = j.normalization_dev;
        a.pos = j.positions_dev; a.num_probes = j.num_probes; a.kmax = j.kmax; a.lambda = j.lambda;
        a.slice_t = j.slice_t; a.k_band = j.k_band; a.cbed = j.cbed_out_dev; a.crop_y = j.crop_y; a.crop_x = j.crop_x;
        a.group = p->group; a.row_sched = p->row_sched; a.col_sched = p->col_sched;
        rc = enqueue_multislice(p, a, b->streams[k]);
      }
      if (rc == MSX_OK) {
        e = cudaEventRecord(b->events[2 * k + 1], b->streams[k]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(b->origin, b->events[2 * k + 1], 0);
        if (e != cudaSuccess) rc = cuda_fail(e, "batch join");
      }
    }
    cudaError_t e = cudaStreamEndCapture(b->origin, &graph);
    if (rc != MSX_OK) {
      if (graph) cudaGraphDestroy(graph);
      return rc;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
    e = cudaGraphInstantiate(&b->gexec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      b->gexec = nullptr;
      return cuda_fail(e, "cudaGraphInstantiate");
    }
    b->gkey = key;
  }
  MSX_CUDA(cudaEventRecord(b->ev_in, caller), "cudaEventRecord");
  MSX_CUDA(cudaStreamWaitEvent(b->origin, b->ev_in, 0), "cudaStreamWaitEvent");
  MSX_CUDA(cudaGraphLaunch(b->gexec, b->origin), "cudaGraphLaunch");
  MSX_CUDA(cudaEventRecord(b->ev_out, b->origin), "cudaEventRecord");
  MSX_CUDA(cudaStreamWaitEvent(caller, b->ev_out, 0), "cudaStreamWaitEvent");
  return MSX_OK;
}

int msx_batch_check(msx_batch* b) {
  if (!b) return fail(MSX_ERR_INVALID, "null batch");
  for (auto& br : b->plans)
    for (auto& kv : br) {
      const int rc = msx_plan_check(kv.second);
      if (rc != MSX_OK) return rc;
    }
  return MSX_OK;
}

}  // extern "C"
