// tpcf_ctx.h -- the context object behind the opaque tpcf_ctx handle and the
// host helpers shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <cstdint>
#include <string>
#include <vector>

#include "tpcf_b200.h"

namespace tpcf {

// Internal failure carried to the C boundary, where it becomes a status code.
struct Failure {
  tpcf_status status;
  std::string msg;
  Failure(tpcf_status s, std::string m) : status(s), msg(std::move(m)) {}
};
// The exception being handled, as a Failure (for the handlers of the C entry points,
// which let none through).
Failure caught();

// NVTX range over one phase of a call (grid build, pair kernel, reduction,
// k-means, resampling), visible in Nsight timelines; free when no tool is
// attached.
struct Phase {
  explicit Phase(const char* name) { nvtxRangePushA(name); }
  ~Phase() { nvtxRangePop(); }
  Phase(const Phase&) = delete;
  Phase& operator=(const Phase&) = delete;
};

// Grow-only device buffer.  A call takes slots in a fixed order, so repeated
// calls of the same shape allocate nothing after the first.
struct Slot {
  void* ptr;
  size_t bytes;
};

}  // namespace tpcf

struct tpcf_ctx {
  int device = 0;
  int num_sms = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  cudaStream_t aux_stream = nullptr;  // second stream of a call (aux_stream()), made on first use
  tpcf_opts opts{};
  std::string err;
  std::vector<tpcf::Slot> slots;
  size_t next_slot = 0;
  void* stage = nullptr;  // kStageBytes of staging for large outputs (copy_out_large), until the context goes
  void* stage_map = nullptr;
  size_t stage_map_bytes = 0;
  bool stage_failed = false;
  int64_t launches = 0;
  int64_t h2d_bytes = 0;
  // statistics of the last call
  bool time_pairs = false;
  cudaEvent_t pending_ev0 = nullptr, pending_ev1 = nullptr;
  double last_pair_ms = 0.0;
  double last_call_ms = 0.0;
  int64_t last_pairs = 0;
  // fault injection for tests (tpcf_debug_inject): the fail_alloc-th workspace
  // allocation from now fails with TPCF_ERR_OOM (-1: none); pair-kernel tile
  // whose copy is never issued (-1: none) and the poll limit of the waits
  int64_t fail_alloc = -1;
  int32_t skip_tile = -1;
  uint32_t wait_limit = 0;
};

namespace tpcf {
void* ws_alloc(tpcf_ctx* c, size_t bytes);
bool is_device_ptr(const void* p);
void check(cudaError_t e, const char* what);
void counted(tpcf_ctx* c, cudaError_t e, const char* what);
template <class T>
const T* stage(tpcf_ctx* c, const T* p, int64_t n);
// Puts `bytes` of host memory at dst (host or device; a device copy is complete
// for the caller once the stream is).
void put_out(tpcf_ctx* c, void* dst, const void* src, size_t bytes);
void copy_out(tpcf_ctx* c, void* dst, const void* src, size_t bytes);
// Large outputs to pageable host memory.  A plain copy is one driver thread that also
// takes the page faults of fresh memory one by one: 32 MB 16.3 ms, against 1.6 ms into
// pages that are there.  expect_outputs(), called while the GPU still works on them,
// has their pages made (contents stay as they are), or from kStagedBytes on the
// context's staging memory, through which copy_out_large() brings them in pieces that
// host threads copy on, faults included, while the next pieces land.
struct HostOut {
  const void* dst;
  size_t bytes;
};
struct HostCopy {
  void* dst;
  const void* src;
  size_t bytes;
};
constexpr size_t kStagePiece = (size_t)2 << 20, kStageBytes = (size_t)16 << 20, kStagedBytes = (size_t)12 << 20;
void expect_outputs(tpcf_ctx* c, const std::vector<HostOut>& outs);
// Complete when it returns for host destinations.
void copy_out_large(tpcf_ctx* c, const std::vector<HostCopy>& v);
void stage_free(tpcf_ctx* c);
void begin_call(tpcf_ctx* c);
cudaStream_t aux_stream(tpcf_ctx* c);
// The bounding boxes, counts and patch ranges of ncat catalogues on the device
// (launch_bbox accumulates into them) and their copy on the host.
struct Boxes {
  int ncat = 0;
  unsigned long long* d_cnt = nullptr;  // [ncat], then box_ord [8 ncat], pr [2 ncat]
  int* d_box = nullptr;
  int* d_pr = nullptr;
  std::vector<float> box;               // [8 ncat]: minx miny maxx maxy minz maxz max|m| 0
  std::vector<unsigned long long> cnt;
  std::vector<int> pr;
  void begin(tpcf_ctx* c, int n);       // allocates and clears
  void read(tpcf_ctx* c);               // one copy, one wait
};
// Sort-key bits of n lenses in n_patch patches: 2 half Hilbert bits (cells of
// less than a sixteenth of an object on average; a radix sort pays per 8 bits)
// under the patch bits; wide: more than 32 in all (64-bit keys).
struct LensKeyBits {
  int half, total;
  bool wide;
};
LensKeyBits lens_key_bits(int64_t n, int n_patch);
// Hilbert bits within a cell of the source sort key.
int cell_hilbert_bits(int64_t n, unsigned ncells, int cell_bits);
struct TaskDesc;
struct LensDesc;
struct GridDesc;
// The work items of the ranges {task, first item} (n in all) on the device,
// costliest first; with shard_count > 1 every shard_count-th of them.
int2* order_items(tpcf_ctx* c, const std::vector<int2>& ranges, int n, const TaskDesc* tasks, const LensDesc* lenses,
                  const GridDesc* grids, float R, bool sph, int shard_index, int shard_count, int* n_run);

// An event of one call (no timing); destroyed with the object, which CUDA
// defers until the event has completed.
struct Event {
  cudaEvent_t e = nullptr;
  Event() { check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event"); }
  ~Event() { cudaEventDestroy(e); }
  Event(const Event&) = delete;
  Event& operator=(const Event&) = delete;
};
tpcf_status canonical_edges(const tpcf_bins* b, double* e, double* e2);
// How the kernels find a bin: for log spacing t = lg2(theta^2) A + B in FP32, with a
// guard band eps around whole numbers that covers its error; on = false: a search of
// the squared edges with a relative guard eps.  sph: angle edges e, squared chords e2.
struct BinRule {
  bool on;
  float A, B, eps;
};
BinRule bin_rule(const tpcf_bins* b, const double* e, const double* e2, bool sph);
}  // namespace tpcf
