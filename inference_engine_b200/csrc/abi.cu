// Version and error-string entry points of the b200kv C ABI.
#include "b200kv.h"

#include <cuda_runtime.h>

#include <atomic>
#include <new>

namespace b200kv {
static std::atomic<int> g_chained{0};
static bool chained() { return g_chained.load(std::memory_order_relaxed) != 0; }

// A recording stream's place in its graph is the set of nodes that the next one will wait for: up to `room` of them to `to`;
// -1: not recording, or more than that.
constexpr int kBranchNodes = 16;
static int place(cudaStream_t stream, cudaGraphNode_t* to, int room) {
  cudaStreamCaptureStatus status;
  const cudaGraphNode_t* nodes = nullptr;
  size_t num = 0;
  if (cudaStreamGetCaptureInfo_v2(stream, &status, nullptr, nullptr, &nodes, &num) != cudaSuccess) {
    (void)cudaGetLastError();
    return -1;
  }
  if (status != cudaStreamCaptureStatusActive || num > (size_t)room) return -1;
  for (size_t i = 0; i < num; ++i) to[i] = nodes[i];
  return (int)num;
}

// The places where a fork or a join of branches left a stream: a launch by this thread that finds its stream still there is not chained.
// One that finds it elsewhere stands behind another library's node, as any other does.  One mark per stream, taken off by the next
// launch there; the sixteen latest are kept, as a mark may never be asked for.
struct Mark {
  cudaStream_t stream;
  int num;
  cudaGraphNode_t nodes[kBranchNodes];
};
constexpr int kMarks = 16;
static thread_local Mark t_marks[kMarks];
static thread_local int t_num_marks = 0;
static int marked(cudaStream_t stream) {
  for (int i = 0; i < t_num_marks; ++i)
    if (t_marks[i].stream == stream) return i;
  return -1;
}
static void take_off(int i) {
  for (--t_num_marks; i < t_num_marks; ++i) t_marks[i] = t_marks[i + 1];
}
static void mark_place(cudaStream_t stream) {
  Mark m;
  m.stream = stream;
  m.num = place(stream, m.nodes, kBranchNodes);
  const int old = marked(stream);
  if (old >= 0) take_off(old);
  if (m.num < 0) return;
  if (t_num_marks == kMarks) take_off(0);
  t_marks[t_num_marks++] = m;
}
bool take_plain_launch(cudaStream_t stream) {
  const int at = marked(stream);
  if (at < 0) return false;
  const Mark m = t_marks[at];
  take_off(at);
  cudaGraphNode_t now[kBranchNodes];
  if (place(stream, now, kBranchNodes) != m.num) return false;
  for (int i = 0; i < m.num; ++i) {  // in any order
    bool found = false;
    for (int j = 0; j < m.num; ++j) found = found || now[i] == m.nodes[j];
    if (!found) return false;
  }
  return true;
}
bool take_chained_launch(cudaStream_t stream) { return !take_plain_launch(stream) && chained(); }

struct Branches {
  cudaStream_t stream;
  int num_from = 0, num_ends = 0;
  cudaGraphNode_t from[kBranchNodes], ends[kBranchNodes];

  bool move_to(cudaGraphNode_t* nodes, int num) {
    const bool ok = cudaStreamUpdateCaptureDependencies(stream, nodes, num, cudaStreamSetCaptureDependencies) == cudaSuccess;
    mark_place(stream);
    return ok;
  }
  // The end of the branch at hand joins `ends`.
  bool keep_end() {
    const int n = place(stream, ends + num_ends, kBranchNodes - num_ends);
    if (n < 0) return false;
    num_ends += n;
    return true;
  }
};
}  // namespace b200kv

// One kernel after the other leaves the multiprocessors half empty where one is short of blocks and the next of bandwidth.
// Branches need no second stream, whose tensors' lifetimes would have to be told to the allocator, and no events.
extern "C" void* b200kv_branches_begin(void* stream) {
  b200kv::Branches* b = new (std::nothrow) b200kv::Branches;
  if (!b) return nullptr;
  b->stream = (cudaStream_t)stream;
  b->num_from = b200kv::place(b->stream, b->from, b200kv::kBranchNodes);
  if (b->num_from < 0) {
    delete b;
    return nullptr;
  }
  b200kv::mark_place(b->stream);
  return b;
}
extern "C" int b200kv_branches_next(void* branches) {
  b200kv::Branches* b = (b200kv::Branches*)branches;
  if (!b) return B200KV_OK;
  return b->keep_end() && b->move_to(b->from, b->num_from) ? B200KV_OK : B200KV_E_LAUNCH;
}
extern "C" int b200kv_branches_end(void* branches) {
  b200kv::Branches* b = (b200kv::Branches*)branches;
  if (!b) return B200KV_OK;
  const bool ok = b->keep_end() && b->move_to(b->ends, b->num_ends);
  delete b;
  return ok ? B200KV_OK : B200KV_E_LAUNCH;
}

extern "C" void b200kv_set_chained_launch(int enabled) { b200kv::g_chained.store(enabled ? 1 : 0, std::memory_order_relaxed); }
extern "C" int b200kv_get_chained_launch(void) { return b200kv::chained() ? 1 : 0; }

extern "C" void b200kv_plain_next(void* stream) { b200kv::mark_place((cudaStream_t)stream); }

extern "C" int b200kv_version(void) { return B200KV_VERSION; }

extern "C" const char* b200kv_error_string(int code) {
  switch (code) {
    case B200KV_OK: return "ok";
    case B200KV_E_NULL: return "a required pointer is NULL";
    case B200KV_E_SHAPE: return "unsupported geometry (head_dim must be 128, Hq a multiple of Hkv with ratio <= 8, page_size a multiple of 16 when paged)";
    case B200KV_E_ALIGN: return "pointer or stride not aligned (bf16 rows need 8-byte, q/out of decode attention 16-byte alignment)";
    case B200KV_E_WORKSPACE: return "workspace too small (see b200kv_decode_attn_workspace_bytes)";
    case B200KV_E_LAUNCH: return "CUDA launch failed";
    case B200KV_E_RANGE: return "size argument out of range";
    case B200KV_E_STATIC_LIMIT: return "this batch needs more scratch than the 8 MiB built into the library: use b200kv_decode_attn with a caller workspace";
    default: return "unknown b200kv error";
  }
}
