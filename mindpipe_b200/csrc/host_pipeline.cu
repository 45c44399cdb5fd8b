// W4A16 linears on page-locked host activations: a recorded set of independent linears as a pipeline of copies and products.
//
// What bounds it: PCIe (about 50 GB/s each way), the launches and, behind the last product, its results' way home.  One copy
// per tensor and direction in stream order took 2 to 4 us each before its first byte and ran beside nothing: a 7B layer's
// four linears at 16 rows, 0.75 MB in and 1.36 MB out, took 154 us, 48 of them products.  Here
//   * the rows come in by a kernel that reads host memory itself, all tensors of a launch at once;
//   * up to kDirectBytes each way one such launch brings everything and one takes everything back (2 us + 4 us);
//   * beyond that the first linear's rows come alone and the others' beside its product, and every result leaves by the copy
//     engine, on a stream of its own, while the next product runs.  The linear with the smallest result goes last.
#include <map>
#include <mutex>
#include <new>
#include <utility>

#include "common.cuh"

namespace mp {

// mp_w4a16_linear with the kernels' weights requested before the kernel before has finished (early > 0), or as the
// process-wide switch says (early < 0).  w4a16_decode.cu
int w4a16_linear(const void* x, const void* packed, const void* sz, const void* bias, void* y, int M, int N, int K, int group,
                 void* workspace, size_t workspace_bytes, int* error_word, int early, mp_stream_t stream);

namespace {
constexpr int kMaxLinears = 16;
// At 50 GB/s 256 KB are 5 us, about what the copies' own streams and events cost.
constexpr size_t kDirectBytes = 256 * 1024;

struct CopyList {
  const uint4* src[kMaxLinears];
  uint4* dst[kMaxLinears];
  int end[kMaxLinears];        // running count of 16-byte pieces
  int count;
};

// Host memory is written again between calls, so its loads bypass the caches; four are in flight per thread.
__global__ void __launch_bounds__(256) host_copy_kernel(const __grid_constant__ CopyList list, bool from_host) {
  chain_wait();
  chain_release();
  const int total = list.end[list.count - 1], step = gridDim.x * 256;
  for (int i0 = blockIdx.x * 256 + threadIdx.x; i0 < total; i0 += 4 * step) {
    uint4 v[4];
    uint4* to[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + j * step;
      to[j] = nullptr;
      if (i >= total) continue;
      int e = 0;
      while (i >= list.end[e]) ++e;
      const int at = i - (e ? list.end[e - 1] : 0);
      v[j] = from_host ? __ldcv(list.src[e] + at) : __ldcg(list.src[e] + at);
      to[j] = list.dst[e] + at;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (to[j]) *to[j] = v[j];
  }
}

int launch_copy(const CopyList& list, bool from_host, cudaStream_t st) {
  const int blocks = (list.end[list.count - 1] + 255) / 256;
  return launch_chained(host_copy_kernel, dim3(blocks < 2 * kSmCount ? blocks : 2 * kSmCount), dim3(256), 0, st, list, from_host);
}

void add_copy(CopyList& list, const void* src, void* dst, size_t bytes) {
  list.src[list.count] = static_cast<const uint4*>(src);
  list.dst[list.count] = static_cast<uint4*>(dst);
  list.end[list.count] = (list.count ? list.end[list.count - 1] : 0) + static_cast<int>(bytes / 16);
  ++list.count;
}
}  // namespace

// The two streams beside a caller's stream, shared by all pipelines that run there and given back with the last of them
// (making one takes some 300 us).
struct SideStreams {
  cudaStream_t in = nullptr, out = nullptr;
  int users = 0;
};
static std::mutex g_sides_mutex;
static std::map<std::pair<int, cudaStream_t>, SideStreams>& sides() {
  static auto* all = new std::map<std::pair<int, cudaStream_t>, SideStreams>;
  return *all;
}

struct HostPipeline {
  int device = 0, count = 0;
  cudaStream_t stream = nullptr;                   // the caller's
  bool has_sides = false;
  mp_host_linear linear[kMaxLinears];              // in the order they run
  CopyList first{}, others{}, back{};              // rows of the first linear (or of all), of the others; all results
  bool direct_in = false, direct_out = false;
  cudaStream_t in = nullptr, out = nullptr;
  cudaEvent_t begun = nullptr, arrived = nullptr, sent = nullptr, done[kMaxLinears] = {};
  std::mutex enqueue;                              // a call's events are recorded and waited for before the next call's
  ~HostPipeline() {
    for (cudaEvent_t e : {begun, arrived, sent})
      if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : done)
      if (e) cudaEventDestroy(e);
    if (has_sides) {
      std::lock_guard<std::mutex> lock(g_sides_mutex);
      auto at = sides().find({device, stream});
      if (at != sides().end() && --at->second.users == 0) {
        cudaStreamDestroy(at->second.in);
        cudaStreamDestroy(at->second.out);
        sides().erase(at);
      }
    }
  }
};

static int make_pipeline(HostPipeline& p, const mp_host_linear* linears, int count) {
  MP_CUDA_TRY(cudaGetDevice(&p.device));
  size_t x_bytes = 0, y_bytes = 0;
  int smallest = 0;
  for (int i = 0; i < count; ++i) {
    const mp_host_linear& c = linears[i];
    if (!c.x_host_f16 || !c.x_stage_f16 || !c.y_stage_f16 || !c.y_host_f16 || c.M <= 0 || c.K <= 0 || c.N <= 0)
      return MP_ERR_INVALID_ARG;
    const size_t xb = (size_t)c.M * c.K * 2, yb = (size_t)c.M * c.N * 2;
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
    if ((size_t)c.M * c.N < (size_t)linears[smallest].M * linears[smallest].N) smallest = i;
  }
  p.count = count;
  p.direct_in = count == 1 || x_bytes <= kDirectBytes;
  p.direct_out = y_bytes <= kDirectBytes;
  for (int i = 0, at = 0; i < count; ++i)
    if (i != smallest) p.linear[at++] = linears[i];
  p.linear[count - 1] = linears[smallest];
  for (int i = 0; i < count; ++i) {
    const mp_host_linear& c = p.linear[i];
    add_copy(i == 0 || p.direct_in ? p.first : p.others, c.x_host_f16, c.x_stage_f16, (size_t)c.M * c.K * 2);
    add_copy(p.back, c.y_stage_f16, c.y_host_f16, (size_t)c.M * c.N * 2);
  }
  if (!p.direct_in || !p.direct_out) {
    std::lock_guard<std::mutex> lock(g_sides_mutex);
    SideStreams side;
    auto at = sides().find({p.device, p.stream});
    if (at != sides().end()) {
      side = at->second;
    } else {
      MP_CUDA_TRY(cudaStreamCreateWithFlags(&side.in, cudaStreamNonBlocking));
      const cudaError_t e = cudaStreamCreateWithFlags(&side.out, cudaStreamNonBlocking);
      if (e != cudaSuccess) {
        cudaStreamDestroy(side.in);
        return cuda_fail(e);
      }
    }
    ++side.users;
    sides()[{p.device, p.stream}] = side;
    p.has_sides = true;
    p.in = side.in;
    p.out = side.out;
  }
  if (!p.direct_in) {
    for (cudaEvent_t* e : {&p.begun, &p.arrived}) MP_CUDA_TRY(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  }
  if (!p.direct_out) {
    MP_CUDA_TRY(cudaEventCreateWithFlags(&p.sent, cudaEventDisableTiming));
    for (int i = 0; i < count; ++i) MP_CUDA_TRY(cudaEventCreateWithFlags(&p.done[i], cudaEventDisableTiming));
  }
  return MP_OK;
}

static int run_pipeline(HostPipeline& p) {
  const cudaStream_t st = p.stream;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  MP_CUDA_TRY(cudaStreamIsCapturing(st, &capturing));
  if (capturing != cudaStreamCaptureStatusNone) return mp_w4a16_linear_decode_host_many(p.linear, p.count, st);
  std::lock_guard<std::mutex> lock(p.enqueue);
  int rc;
  if (!p.direct_in) {
    MP_CUDA_TRY(cudaEventRecord(p.begun, st));               // the call before still reads its rows until here
    MP_CUDA_TRY(cudaStreamWaitEvent(p.in, p.begun, 0));
  }
  if ((rc = launch_copy(p.first, true, st)) != MP_OK) return rc;
  for (int i = 0; i < p.count; ++i) {
    const mp_host_linear& c = p.linear[i];
    // the kernel before in the stream is this pipeline's own and writes no weights
    rc = w4a16_linear(c.x_stage_f16, c.packed_i32, c.sz_f16x2, c.bias_f16, c.y_stage_f16, c.M, c.N, c.K, c.group, c.workspace,
                      c.workspace ? c.workspace_bytes : 0, nullptr, 1, st);
    if (rc != MP_OK) return rc;
    if (i == 0 && !p.direct_in) {
      if ((rc = launch_copy(p.others, true, p.in)) != MP_OK) return rc;
      MP_CUDA_TRY(cudaEventRecord(p.arrived, p.in));
      MP_CUDA_TRY(cudaStreamWaitEvent(st, p.arrived, 0));
    }
    if (!p.direct_out) {
      MP_CUDA_TRY(cudaEventRecord(p.done[i], st));
      MP_CUDA_TRY(cudaStreamWaitEvent(p.out, p.done[i], 0));
      MP_CUDA_TRY(cudaMemcpyAsync(c.y_host_f16, c.y_stage_f16, (size_t)c.M * c.N * 2, cudaMemcpyDeviceToHost, p.out));
    }
  }
  if (p.direct_out) return launch_copy(p.back, false, st);
  MP_CUDA_TRY(cudaEventRecord(p.sent, p.out));
  MP_CUDA_TRY(cudaStreamWaitEvent(st, p.sent, 0));
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
