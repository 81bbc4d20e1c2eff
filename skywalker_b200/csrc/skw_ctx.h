// Host-side state behind the opaque skw_ctx handle, and the helpers every translation unit of
// the library uses to report errors and count launches.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/skywalker_b200.h"
#include "skw_device.cuh"

namespace skw {

// Spare slots allocated past the table's E entries (room for the padded last chunk of an in-place
// all-gather over up to 1024 ranks).
constexpr uint32_t kSlotSlack = 1024;

}  // namespace skw

struct skw_ctx {
  int device = 0;
  int sm_count = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  cudaStream_t side_stream = nullptr;  // result copies that overlap kernels of `stream`
  cudaStream_t copy_stream = nullptr;  // skw_walk_packed: the packed rows of each slice
  // skw_walk_packed, per slice: rows packed (and their count on the host); start and end of the walk
  static constexpr int kPackSlices = 8;
  cudaEvent_t pk_ready[kPackSlices] = {}, pk_t0[kPackSlices] = {}, pk_t1[kPackSlices] = {},
              pk_in[kPackSlices] = {};
  uint64_t* h_tot = nullptr;  // cells each slice's packed result needs: mapped, written by the packing kernel
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // the builders of one build run side by side: those of lists of more than 512 weights on streams of their own,
  // forked from and joined back into `stream` by events
  static constexpr int kBuilderStreams = 5;
  cudaStream_t bstream[kBuilderStreams] = {};
  cudaEvent_t bfork = nullptr, bjoin[kBuilderStreams] = {};
  bool queued = false;          // walks on the current stream that no call has waited for
  bool queued_before = false;   // ... and on the stream before it
  // behind the last queued call that builds tables, whatever stream it went to: the builders' work lists and scratch and
  // the tables of an online call are the context's
  cudaEvent_t tables_used = nullptr;
  bool tables_queued = false;
  std::string err;
  uint64_t launches = 0;

  // resident CSR
  uint32_t V = 0;
  uint64_t E = 0;
  uint32_t max_degree = 0;
  uint32_t empty_lists = 0;  // vertices without out-edges
  static constexpr uint32_t kLongLeast = 16385, kLongMost = 65536;
  uint32_t long_lists = 0;   // vertices of degree kLongLeast to kLongMost
  static constexpr uint32_t kEdgeSample = 4096;
  uint32_t dead_ends = 0;    // of kEdgeSample edges spread over the list of all, those into vertices without out-edges
  uint32_t* xadj = nullptr;
  uint32_t* adjncy = nullptr;
  float* adjwgt = nullptr;
  bool owns_graph = false;
  bool owns_weights = false;

  // alias table
  skw::Slot* slots = nullptr;
  uint8_t* valid = nullptr;
  bool slots_marked = false;  // slots that no build has reached hold prob = -1
  bool table_ready = false;
  // tables of one online call (the table above stays as it is); their memory is kept for the next
  skw::Slot* online_slots = nullptr;
  uint8_t* online_valid = nullptr;
  bool online_in_use = false;  // by the call that is being made: not to be given up
  // optional fused walk records (32 B per edge slot) and per-vertex {offset, usable degree}
  void* records = nullptr;
  void* vinfo = nullptr;
  void* vbits = nullptr;  // one bit per vertex: usable degree != 0
  bool records_ready = false;  // set once records, vinfo and vbits were all written
  bool records_building = false;  // between their allocation and that: not to be given up
  bool records_all_usable = false;  // ... and no vertex with out-edges lacks a usable table

  // status words on the device and in mapped host memory: the error records of synchronous and of queued calls (4 words
  // each) and four 64-bit sums (edges of a synchronous call, of queued calls, of packed calls; vertices without a usable table)
  uint32_t* d_err = nullptr;
  uint32_t* launch_err = nullptr;  // the record that the kernels of the current call write
  uint32_t* h_err = nullptr;
  uint64_t* d_sum = nullptr;
  uint64_t* h_sum = nullptr;
  bool status_clean = true;  // the record of synchronous calls and sums 0 and 3 are zero

  // builder scratch, grown on demand
  uint32_t* worklist = nullptr;      // vertices by degree class, one list per class
  size_t worklist_cap = 0;
  // Counts and cursors of the degree classes, a set of words a build.  A build takes the next set, which is zero; the kernel
  // that reports a call's status clears them all again, so that a build needs no memset of its own (1 M edges: 50 -> 47 us).
  static constexpr unsigned kClassSets = 8, kClassWords = 32;
  uint32_t* cls_counts = nullptr;
  unsigned cls_used = 0;  // sets that are not zero; the last one belongs to graphs
  void* cta_scratch = nullptr;       // slabs of the global-memory CTA builder
  size_t cta_scratch_bytes = 0;
  bool scratch_short = false;        // no memory for those of this graph's smaller teams: the largest do without

  // online mode: per-frontier work lists (one per degree class) and the claim stamps that make
  // every distinct frontier vertex be built once per round
  uint32_t* frontier_lists = nullptr;
  size_t frontier_lists_bytes = 0;
  uint32_t* stamp = nullptr;         // V entries, last round that claimed the vertex
  uint32_t stamp_round = 0;
  // online direct walks: per-vertex memo of {call stamp, largest weight, total quantised weight}
  void* prep_memo = nullptr;
  uint32_t prep_stamp = 0;
  void* prep_ckpt = nullptr;  // prefix-sum checkpoints of long lists, valid together with the memo entry

  // skw_walk with host rows, large batches: pinned staging for the packed result and the host threads
  // that scatter it into the caller's matrix
  uint32_t* h_pack = nullptr;
  size_t h_pack_cells = 0;
  void* host_pool = nullptr;  // skw::HostPool
  bool counted = false;       // among the contexts for which freed device memory is kept

  // staging buffers of the host-pointer entry points, grown on demand
  static constexpr int kStages = 14;
  void* stage[kStages] = {};
  size_t stage_bytes[kStages] = {};
  static constexpr int kHeadStage = kStages - 1;  // for speed only: given up when another allocation fails
  bool heads_in_use = false;
};

namespace skw {

int fail(skw_ctx* ctx, int code, const char* fmt, ...);
// after the CSR pointers are set: compute max_degree, empty_lists, long_lists and dead_ends
int finish_graph(skw_ctx* ctx);
// allocate slots[E] / valid[V] if absent; a call that writes only a part of the table has the rest marked unusable
enum class TableUse {
  kAll,      // writes every slot
  kSome,     // a range of vertices, the others may be drawn from later
  kFrontier  // draws only from the slots that it writes
};
int alloc_table(skw_ctx* ctx, TableUse use);
// the calls that write a table or its records in place wait for walks that were queued on other streams
int settle_queued(skw_ctx* ctx);
// the calls that queue builders wait on the GPU for the last queued call that did, if it was on another stream
int builders_begin(skw_ctx* ctx);
int builders_queued(skw_ctx* ctx);
// memory that the builders of the tables of so many vertices need besides the tables
int reserve_builders(skw_ctx* ctx, uint32_t vertices);
// queue the construction of the tables of vertices [v_begin, v_end)
int enqueue_tables(skw_ctx* ctx, uint32_t v_begin, uint32_t v_end, Slot* slots, uint8_t* valid);
// free the memory of an online call's tables
void drop_online_tables(skw_ctx* ctx);
// forget the fused walk records (they are derived from the table and die with it) and free their memory
void drop_records(skw_ctx* ctx);
// Device memory, from blocks freed earlier where one fits; gives up the memory of records that are no longer valid, then
// that of an online call's tables, then that for heads of rows, before it fails.  dev_free waits for the GPU.
cudaError_t dev_malloc_bytes(skw_ctx* ctx, void** p, size_t bytes);
template <class T>
cudaError_t dev_malloc(skw_ctx* ctx, T** p, size_t bytes) {
  void* q = nullptr;
  const cudaError_t e = dev_malloc_bytes(ctx, &q, bytes);
  if (e == cudaSuccess) *p = static_cast<T*>(q);
  return e;
}
void dev_free(void* p);
void dev_give_back(int device);  // what dev_free kept
int fail_cuda(skw_ctx* ctx, cudaError_t e, const char* what, const char* file, int line);
void set_global_error(const char* msg);

// Whether the context's stream is being captured into a graph: no allocation then, and no memory that may change later.
bool capturing(const skw_ctx* ctx);
// Grow-only device buffer.
int ensure_bytes(skw_ctx* ctx, void** p, size_t* cap, size_t want);
// Bracket of a synchronous call: its error record and sums 0 and 3 are zero after err_reset; err_check brings all
// status words to the host, waits for the stream, clears them but for those of queued calls and reports an error.
// queued: what queued calls reported, cleared as well.
int err_reset(skw_ctx* ctx);
int err_check(skw_ctx* ctx, const char* where, bool queued = false);
// Kernels launched while this lives write the record of queued calls.
struct QueuedErrors {
  skw_ctx* ctx;
  explicit QueuedErrors(skw_ctx* c) : ctx(c) { ctx->launch_err = ctx->d_err + 4; }
  ~QueuedErrors() { ctx->launch_err = ctx->d_err; }
};

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
    else prev = -1;
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

}  // namespace skw

#define SKW_CUDA(ctx, call)                                                          \
  do {                                                                               \
    cudaError_t e__ = (call);                                                        \
    if (e__ != cudaSuccess) return skw::fail_cuda((ctx), e__, #call, __FILE__, __LINE__); \
  } while (0)

// Count a kernel launch and surface a launch-configuration error at once.
#define SKW_LAUNCHED(ctx)                                                            \
  do {                                                                               \
    (ctx)->launches++;                                                               \
    cudaError_t e__ = cudaGetLastError();                                            \
    if (e__ != cudaSuccess) return skw::fail_cuda((ctx), e__, "kernel launch", __FILE__, __LINE__); \
  } while (0)
