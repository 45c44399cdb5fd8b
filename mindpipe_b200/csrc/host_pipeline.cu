// W4A16 linears on page-locked host activations: a recorded set of independent linears as one chain of launches, in which
// rows and results cross PCIe beside the products.
//
// What bounds it: PCIe (about 50 GB/s each way), the products, the first rows' way in and the last result's way out.  While
// results leave, reads of host memory wait behind them (131 KB: 6 us alone, 59 beside a long copy out), so all rows come in
// before the first result goes: a copy kernel brings the first linear's, and its product, on the weight stream, the others'
// in a warp of its own.  So a linear that runs there goes first (outputs 1024, 1024 and 4096 of 4096 columns, given in that
// order, at 16 rows 38.1 -> 33.5 us); where none does, a copy kernel on the side stream brings the others' rows beside the
// first product (four linears of 256x11008 at 16 rows 66.3 us, by a launch behind that product 72.5).  Results leave by the copy
// engine, on a stream of their own, while the next product runs (the events between products do not end the overlap of one's
// beginning with the end of the one before), so the linear with the smallest result goes last: a copy kernel takes it.  Up to
// kDirectBytes each way one such kernel brings everything and one takes everything back.
// A 7B layer's four linears at 16 rows, 0.75 MB in and 1.36 MB out, 42 us of products: 68 us; 81 with the others' rows
// on a stream of their own, where they kept the first one's from arriving (21 us); 76 with each product bringing the next
// one's rows, against the results; 76 with the products taking the results along too, since a kernel that has stored to host
// memory ends 5 us after its last store; 154 in stream order, a copy per tensor.
#include <map>
#include <mutex>
#include <new>
#include <utility>

#include "common.cuh"

namespace mp {

// Whether mp_w4a16_linear takes copies along for such a call (with scratch and 16-byte aligned weights).  w4a16_decode.cu
bool w4a16_linear_takes_copies(int M, int N, int K, int group);
// mp_w4a16_linear with the kernels' weights requested before the kernel before has finished (early > 0), or as the
// process-wide switch says (early < 0); `copies` go along where *carried says so afterwards.  w4a16_decode.cu
int w4a16_linear(const void* x, const void* packed, const void* sz, const void* bias, void* y, int M, int N, int K, int group,
                 void* workspace, size_t workspace_bytes, int* error_word, int early, mp_stream_t stream,
                 const HostCopies* copies, bool* carried);

namespace {
constexpr int kMaxLinears = kMaxHostCopies;
// At 50 GB/s 256 KB are 5 us, about what the results' own stream and events cost.
constexpr size_t kDirectBytes = 256 * 1024;

__global__ void __launch_bounds__(256) host_copy_kernel(const __grid_constant__ HostCopies list, bool from_host) {
  chain_wait();
  chain_release();
  copy_pieces(list, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256, from_host);
}

int launch_copy(const HostCopies& list, bool from_host, cudaStream_t st) {
  const int blocks = (list.end[list.count - 1] + 255) / 256;
  return launch_chained(host_copy_kernel, dim3(blocks < 2 * kSmCount ? blocks : 2 * kSmCount), dim3(256), 0, st, list, from_host);
}

void add_copy(HostCopies& list, const void* src, void* dst, size_t bytes) {
  list.src[list.count] = static_cast<const uint4*>(src);
  list.dst[list.count] = static_cast<uint4*>(dst);
  list.end[list.count] = (list.count ? list.end[list.count - 1] : 0) + static_cast<int>(bytes / 16);
  ++list.count;
}

size_t row_bytes(const mp_host_linear& c) { return (size_t)c.M * c.K * 2; }
size_t result_bytes(const mp_host_linear& c) { return (size_t)c.M * c.N * 2; }
bool takes_copies(const mp_host_linear& c) {
  return w4a16_linear_takes_copies(c.M, c.N, c.K, c.group) && c.workspace &&
         c.workspace_bytes >= mp_w4a16_linear_workspace_bytes(c.M, c.N, c.K, c.group) && aligned(c.packed_i32, 16) &&
         aligned(c.sz_f16x2, 16);
}
}  // namespace

// The stream for results (and rows) beside a caller's stream, shared by all pipelines that run there and given back with the
// last of them (making one takes some 150 us; with two or four of them in turn a 7B layer took 73 to 87 us instead of 68 to 71).
struct SideStream {
  cudaStream_t out = nullptr;
  int users = 0;
};
static std::mutex g_sides_mutex;
static std::map<std::pair<int, cudaStream_t>, SideStream>& sides() {
  static auto* all = new std::map<std::pair<int, cudaStream_t>, SideStream>;
  return *all;
}

struct HostPipeline {
  int device = 0, count = 0;
  cudaStream_t stream = nullptr;                   // the caller's
  bool has_side = false;
  mp_host_linear linear[kMaxLinears];              // in the order they run
  HostCopies first{}, others{}, back{};            // rows of the first linear (or of all), of the others; the last result (or all)
  bool direct_out = false;
  bool beside = false;                             // the others' rows come on the side stream, not with the first product
  cudaStream_t out = nullptr;
  cudaEvent_t begun = nullptr, arrived = nullptr, sent = nullptr, done[kMaxLinears] = {};
  std::mutex enqueue;                              // a call's events are recorded and waited for before the next call's
  ~HostPipeline() {
    for (cudaEvent_t e : {begun, arrived, sent})
      if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : done)
      if (e) cudaEventDestroy(e);
    if (has_side) {
      std::lock_guard<std::mutex> lock(g_sides_mutex);
      auto at = sides().find({device, stream});
      if (at != sides().end() && --at->second.users == 0) {
        cudaStreamDestroy(at->second.out);
        sides().erase(at);
      }
    }
  }
};

static int make_pipeline(HostPipeline& p, const mp_host_linear* linears, int count) {
  MP_CUDA_TRY(cudaGetDevice(&p.device));
  size_t x_bytes = 0, y_bytes = 0;
  for (int i = 0; i < count; ++i) {
    const mp_host_linear& c = linears[i];
    if (!c.x_host_f16 || !c.x_stage_f16 || !c.y_stage_f16 || !c.y_host_f16 || c.M <= 0 || c.K <= 0 || c.N <= 0)
      return MP_ERR_INVALID_ARG;
    const size_t xb = row_bytes(c), yb = result_bytes(c);
    if (c.M > 16 || xb % 16 || yb % 16 || xb + yb > ((size_t)1 << 28)) return MP_ERR_UNSUPPORTED;
    void* alias = nullptr;
    int rc = mp_host_buffer_device_alias(c.x_host_f16, xb, &alias);
    if (rc != MP_OK) return rc;
    if (alias != c.x_host_f16) return MP_ERR_UNSUPPORTED;
    rc = mp_host_buffer_device_alias(c.y_host_f16, yb, &alias);
    if (rc != MP_OK) return rc;
    if (alias != c.y_host_f16) return MP_ERR_UNSUPPORTED;
    if (!aligned(c.x_stage_f16, 16) || !aligned(c.y_stage_f16, 16)) return MP_ERR_ALIGNMENT;
    x_bytes += xb;
    y_bytes += yb;
  }
  auto smallest_but = [&](int not_this) {
    int best = -1;
    for (int i = 0; i < count; ++i)
      if (i != not_this && (best < 0 || result_bytes(linears[i]) < result_bytes(linears[best]))) best = i;
    return best;
  };
  const bool rows_apart = count > 1 && x_bytes > kDirectBytes;
  int first = -1, last = smallest_but(-1);
  if (rows_apart) {
    for (int i = 0; i < count && first < 0; ++i)
      if (i != last && takes_copies(linears[i])) first = i;
    if (first < 0 && takes_copies(linears[last])) {
      first = last;
      last = smallest_but(first);
    }
    p.beside = first < 0;
  }
  p.count = count;
  int at = 0;
  if (first >= 0) p.linear[at++] = linears[first];
  for (int i = 0; i < count; ++i)
    if (i != first && i != last) p.linear[at++] = linears[i];
  p.linear[at] = linears[last];
  for (int i = 0; i < count; ++i) {
    const mp_host_linear& c = p.linear[i];
    add_copy(i == 0 || x_bytes <= kDirectBytes ? p.first : p.others, c.x_host_f16, c.x_stage_f16, row_bytes(c));
    if (i == count - 1 || y_bytes <= kDirectBytes) add_copy(p.back, c.y_stage_f16, c.y_host_f16, result_bytes(c));
  }
  p.direct_out = count == 1 || y_bytes <= kDirectBytes;
  if (!p.direct_out || p.beside) {
    std::lock_guard<std::mutex> lock(g_sides_mutex);
    SideStream side;
    auto at = sides().find({p.device, p.stream});
    if (at != sides().end()) {
      side = at->second;
    } else {
      MP_CUDA_TRY(cudaStreamCreateWithFlags(&side.out, cudaStreamNonBlocking));
    }
    ++side.users;
    sides()[{p.device, p.stream}] = side;
    p.has_side = true;
    p.out = side.out;
  }
  if (p.beside) {
    for (cudaEvent_t* e : {&p.begun, &p.arrived}) MP_CUDA_TRY(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  }
  if (p.has_side) MP_CUDA_TRY(cudaEventCreateWithFlags(&p.sent, cudaEventDisableTiming));
  if (!p.direct_out) {
    for (int i = 0; i < count; ++i) MP_CUDA_TRY(cudaEventCreateWithFlags(&p.done[i], cudaEventDisableTiming));
  }
  return MP_OK;
}

// `apart`: work of this run is on the side stream and the caller's does not wait for it yet.
static int enqueue_run(HostPipeline& p, bool& apart) {
  const cudaStream_t st = p.stream;
  int rc;
  if (p.beside) {
    MP_CUDA_TRY(cudaEventRecord(p.begun, st));               // the call before still reads its rows until here
    MP_CUDA_TRY(cudaStreamWaitEvent(p.out, p.begun, 0));
  }
  if ((rc = launch_copy(p.first, true, st)) != MP_OK) return rc;
  for (int i = 0; i < p.count; ++i) {
    const mp_host_linear& c = p.linear[i];
    const HostCopies* others = i == 0 && p.others.count && !p.beside ? &p.others : nullptr;
    bool carried = false;
    // the kernel before in the stream is this pipeline's own and writes no weights
    rc = w4a16_linear(c.x_stage_f16, c.packed_i32, c.sz_f16x2, c.bias_f16, c.y_stage_f16, c.M, c.N, c.K, c.group, c.workspace,
                      c.workspace ? c.workspace_bytes : 0, nullptr, 1, st, others, &carried);
    if (rc != MP_OK) return rc;
    if (others && !carried && (rc = launch_copy(p.others, true, st)) != MP_OK) return rc;    // (the kernel was switched since)
    if (i == 0 && p.beside) {
      apart = true;
      if ((rc = launch_copy(p.others, true, p.out)) != MP_OK) return rc;
      MP_CUDA_TRY(cudaEventRecord(p.arrived, p.out));
      MP_CUDA_TRY(cudaStreamWaitEvent(st, p.arrived, 0));
      apart = false;
    }
    if (!p.direct_out && i < p.count - 1) {
      MP_CUDA_TRY(cudaEventRecord(p.done[i], st));
      MP_CUDA_TRY(cudaStreamWaitEvent(p.out, p.done[i], 0));
      apart = true;
      MP_CUDA_TRY(cudaMemcpyAsync(c.y_host_f16, c.y_stage_f16, result_bytes(c), cudaMemcpyDeviceToHost, p.out));
    }
  }
  return launch_copy(p.back, false, st);
}

static int run_pipeline(HostPipeline& p) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  MP_CUDA_TRY(cudaStreamIsCapturing(p.stream, &capturing));
  if (capturing != cudaStreamCaptureStatusNone) return mp_w4a16_linear_decode_host_many(p.linear, p.count, p.stream);
  std::lock_guard<std::mutex> lock(p.enqueue);
  bool apart = false;
  const int rc = enqueue_run(p, apart);
  if (!apart) return rc;
  // also after an error: a caller who then waits for the stream may write its buffers again
  const cudaError_t recorded = cudaEventRecord(p.sent, p.out);
  const cudaError_t joined = recorded == cudaSuccess ? cudaStreamWaitEvent(p.stream, p.sent, 0) : recorded;
  if (rc != MP_OK) return rc;
  MP_CUDA_TRY(joined);
  return MP_OK;
}

}  // namespace mp

using namespace mp;

extern "C" int mp_host_pipeline_create(const mp_host_linear* linears, int count, mp_stream_t stream, void** pipeline) {
  if (!linears || !pipeline || count <= 0) return MP_ERR_INVALID_ARG;
  *pipeline = nullptr;
  if (count > kMaxLinears) return MP_ERR_UNSUPPORTED;
  HostPipeline* p = new (std::nothrow) HostPipeline;
  if (!p) return MP_ERR_CUDA;
  p->stream = static_cast<cudaStream_t>(stream);
  const int rc = make_pipeline(*p, linears, count);
  if (rc != MP_OK) {
    delete p;
    return rc;
  }
  *pipeline = p;
  return MP_OK;
}

extern "C" int mp_host_pipeline_run(void* pipeline) {
  if (!pipeline) return MP_ERR_INVALID_ARG;
  return run_pipeline(*static_cast<HostPipeline*>(pipeline));
}

extern "C" void mp_host_pipeline_destroy(void* pipeline) { delete static_cast<HostPipeline*>(pipeline); }
