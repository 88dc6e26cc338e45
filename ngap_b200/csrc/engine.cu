// Device side of the C ABI: table upload, work planning, kernel launches,
// report compaction and results.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <memory>
#include <tuple>
#include <vector>

#include "common.h"
#include "context.h"
#include "handles.h"
#include "match_kernel.cuh"
#include "plan_rules.h"
#include "scan_kernel.cuh"
#include "sort_kernels.cuh"
#include "tables.h"

using namespace ngap;

namespace {

#define CUDA_TRY(expr)                                                                     \
  do {                                                                                     \
    cudaError_t _e = (expr);                                                               \
    if (_e != cudaSuccess) {                                                               \
      set_error("CUDA error %s at %s:%d: %s", cudaGetErrorName(_e), __FILE__, __LINE__,    \
                cudaGetErrorString(_e));                                                   \
      return NGAP_E_CUDA;                                                                  \
    }                                                                                      \
  } while (0)

// Device counters of an engine (kNumCounters words, zeroed by the last kernel
// of a match, HostOut): [0] raw reports, [1] unique reports, [2..3] work, [4]
// error bits, [5..6] the standalone sort's counts, [kRadixCount] keys left to
// the radix pipeline after the small-set sort, [kCursors ...] the unit cursors
// of the three launches, [kSliceCtl ...] the control words of the slices.
constexpr int kDefaultQueue = 1 << 16;  // overflow-stack entries per warp
constexpr int kQueueSpare = 128;  // more of them: a worklist holds the caller's capacity and 512 entries
static_assert(kStackCap + kQueueSpare == 512, "512 entries, in shared memory or beyond it");
constexpr int kRadixCount = 8;
constexpr int kCursors = 10;
constexpr int kSliceCtl = 16;
static_assert(kRunWarps % kWarpsPerCta == 0, "the runs' warps share what match_kernel's have");

// Overflow-stack entries of a run's warp, where a warp of match_kernel has ovf_cap.
// There are twice as many, so that equal shares would need twice the memory
// (1.24 GB on 148 SMs at the default capacity, 0.62 GB with halves); they inject no
// more than a quarter of their worklist at a time (mark_inject) and work depth
// first past half of it, which bounds what they need. Small capacities are kept whole.
int run_queue(int ovf_cap) { return std::max(ovf_cap / 2, std::min(ovf_cap, 8192 + kQueueSpare)); }
constexpr int kSliceSlots = 8;  // slices that run without zeroing control words in between
static_assert(kSliceCtl * 8 + kSliceSlots * kCtlWords * 4 <= kNumCounters * 8, "counters");

int bits_for(uint64_t x) {  // bits needed to hold values < x (x >= 1)
  int b = 0;
  while (b < 64 && (x - 1) >> b) b++;
  return b;
}

// Bits [lo, lo + n) of a key.
uint64_t bit_range(int lo, int n) { return n <= 0 ? 0ull : ((n >= 64 ? ~0ull : (1ull << n) - 1) << lo); }

// The 8-bit digits that cover the bits of a key that can vary, least
// significant first.
std::vector<int> digits_of(uint64_t bits) {
  std::vector<int> shifts;
  while (bits) {
    const int b = __builtin_ctzll(bits);
    shifts.push_back(b);
    bits &= ~bit_range(b, kDigitBits);
  }
  return shifts;
}

}  // namespace

// One sort of report keys: d_in[0 .. *d_n) (clamped to cap) into unique
// reports at d_out (and stream indices at d_out_stream for MODE 1).
//   MODE 0: keys offset << 32 | id, written as id << 32 | offset;
//   MODE 1: keys stream << sshift | offset << oshift | id (batched matching).
// shifts: the digits the radix pipeline sorts, least significant first.
struct SortJob {
  int mode;
  uint64_t* d_in;
  const unsigned long long* d_n;
  uint64_t cap;
  std::vector<int> shifts;
  int oshift, sshift;
  uint64_t* d_out;
  uint32_t* d_out_stream;
  unsigned long long* d_unique_n;
};

// A report sort captured as a CUDA graph (see sort_reports).
struct SortGraph {
  std::vector<uint64_t> key;
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  int chain = 0;  // kernels in the conditional radix pipeline
  void release() {
    if (ge) cudaGraphExecDestroy(ge);
    if (g) cudaGraphDestroy(g);
    ge = nullptr;
    g = nullptr;
  }
};

// Plan caches key on these serial numbers, not on addresses: a new object
// may be allocated where a destroyed one was.
std::atomic<uint64_t> g_next_serial{1};

struct ngap_tables {
  uint64_t serial = g_next_serial.fetch_add(1);
  int device = 0;
  int num_groups = 0;
  int sid_bits = 0;  // bits of the largest group-local state id
  uint64_t report_states = 0;
  double report_paths = 0;  // most reports a position can give, duplicates included
  bool paths_meet = false;  // in some tile that the blocking algorithm follows paths in (many_paths)
  std::vector<TileHost> tiles;
  std::vector<TileDev> dev_desc;
  TileDev* d_tiles = nullptr;
  std::vector<void*> allocs;
  int64_t bytes = 0;
  int32_t max_states = 0;
  std::vector<char> tile_lean;      // per tile: plain, no sticky states (the lean kernel runs it)
  std::vector<int32_t> run_len;     // per tile: candidates per run
  std::vector<int32_t> pair_nact;  // activation slots of each (activation, layered) tile pair
  int32_t max_nact = 0;            // largest pair

  ~ngap_tables() {
    for (void* p : allocs) cudaFree(p);
  }
  template <class T>
  int upload(const std::vector<T>& v, const T** out) {
    *out = nullptr;
    if (v.empty()) return NGAP_OK;
    void* p = nullptr;
    size_t b = v.size() * sizeof(T);
    CUDA_TRY(cudaMalloc(&p, b));
    allocs.push_back(p);
    bytes += (int64_t)b;
    CUDA_TRY(cudaMemcpy(p, v.data(), b, cudaMemcpyHostToDevice));
    *out = static_cast<const T*>(p);
    return NGAP_OK;
  }
};

struct UnitPlanKey {
  int64_t num_seg, seg_len;
  int is_dup, window, chunk;
  int64_t first_seg;
  int depth;      // prefix depth of the algorithm
  bool blocking;
  bool filtered;  // tiles with a filter may be scanned (off for the wait test hook)
  bool operator<(const UnitPlanKey& o) const {
    return std::tie(num_seg, seg_len, is_dup, window, chunk, first_seg, depth, blocking, filtered) <
           std::tie(o.num_seg, o.seg_len, o.is_dup, o.window, o.chunk, o.first_seg, o.depth,
                    o.blocking, o.filtered);
  }
};

// What the launches of a plan run: units of the three launches of
// match_kernel (make_units) and slices of pieces (make_slices).
struct PlanRanges {
  int32_t begin[3] = {0, 0, 0}, count[3] = {0, 0, 0};
  int32_t one_tile[3] = {-1, -1, -1};  // the one tile of a launch's units, or -1
  std::vector<Slice> slices;
};

struct ngap_engine {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  // input
  uint8_t* d_input = nullptr;
  size_t input_cap = 0;
  // units (cached plan for one tables object)
  uint64_t plan_tables = 0;  // serial of the tables the plain plan was made for
  UnitPlanKey plan_key{-1, -1, -1, -1, -1, -1, -1, false, true};
  UnitDev* d_units = nullptr;
  size_t units_cap = 0;
  int32_t nunits = 0;
  int64_t longest_unit = 0;  // positions of the plan's longest unit
  PlanRanges ranges;
  PieceDev* d_pieces = nullptr;  // pieces of filtered tiles (trace records follow the units')
  size_t pieces_cap = 0;
  uint16_t* d_cand = nullptr;    // candidates and runs of one slice
  int64_t cand_cap = 0;
  RunDev* d_runs = nullptr;
  int64_t runs_cap = 0;
  // worklist traces
  bool trace = false;
  unsigned long long* d_unit_work = nullptr;
  size_t unit_work_cap = 0;
  std::vector<UnitDev> h_units;  // the current plan's units (host copy)
  int64_t trace_seg_len = 0;     // plain matching: unit positions are made segment-relative
  int64_t act_entries = 0;   // activation slots the plan uses
  uint32_t* d_act = nullptr;
  uint32_t* d_act_list = nullptr;  // per row: slots with a first match (compacted)
  int64_t act_cap = 0;
  int32_t act_rows = 0;            // rows of the plan
  int64_t* d_row_off = nullptr;    // per row: first slot
  int32_t* d_row_n = nullptr;      // per row: slots
  uint32_t* d_act_cnt = nullptr;   // per row: matched slots
  int32_t rows_cap = 0;
  uint32_t* d_stk = nullptr; // per-slot sticky lists of layered units (beyond shared memory)
  int stk_cap = 0;
  // reports
  uint64_t rep_cap = 0;
  uint64_t* d_reports = nullptr;
  uint64_t* d_tmp = nullptr;
  uint64_t* d_unique = nullptr;
  uint32_t* d_hist = nullptr;
  size_t hist_cap = 0;
  unsigned long long* d_counters = nullptr;
  bool counters_dirty = false;  // a match was left half enqueued: zero them first
  HostOut ho;                   // what the last kernel of a match leaves in pinned memory
  // per-warp scratch
  uint32_t* d_carry = nullptr;
  uint32_t* d_marks = nullptr;
  uint32_t* d_ovf = nullptr;
  size_t slots = 0;
  size_t ovf_words = 0;
  int carry_cap = 0, mark_words = 0, ovf_cap = 0;
  int max_smem_set = -1;
  int bps_smem = -1, bps_val = 0;  // resident CTAs per SM at the last shared-memory size
  // pinned staging of plan uploads (grow-only) and the event of the last one
  uint8_t* h_plan = nullptr;
  size_t h_plan_cap = 0;
  cudaEvent_t plan_ev = nullptr;
  bool plan_ev_pending = false;
  // timing
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  float match_ms = 0.f, sort_ms = 0.f;
  int launches = 0;
  int pending_status = NGAP_OK;
  bool ran = false;
  int grid = 0;
  // batched matching
  uint64_t batch_ts = 0;     // serial of the tableset the batched plan was made for
  std::vector<ngap_batch_stream> batch_streams;
  int batch_window = -1, batch_chunk = -1, batch_depth = -1;
  bool batch_blocking = false;
  uint32_t* d_stream_ids = nullptr;
  uint64_t stream_ids_cap = 0;
  cudaGraphExec_t graph = nullptr;
  std::vector<uint64_t> graph_key;
  uint64_t buffers = 0;  // counts allocations of device buffers: a captured batch holds their addresses
  bool graph_mode = false;
  int graph_launches = 0;
  cudaStream_t cap_stream = nullptr;  // capture/replay stream of the batched graph
  cudaEvent_t cap_ev[2] = {nullptr, nullptr};
  // report sorts as graphs with a conditional radix pipeline, per configuration
  std::vector<SortGraph> sort_graphs;
  cudaStream_t sort_cs = nullptr;     // capture stream of those graphs
  bool sort_graph_off = false;
  int sort_chain_pending = 0;         // pipeline kernels of the last graph sort, if it ran
  bool sort_open = false;             // the last sort may have left keys to the pipeline (finish_sort)
  SortJob sort_job;                   // that sort
  // test hook for the bounded device wait (ngap_engine_test_wait_timeout): armed for the
  // next ngap_match only
  int32_t test_skip_unit = -1;
  int32_t test_wait_rounds = 0;

  ~ngap_engine() {
    cudaFree(d_input);
    cudaFree(d_units);
    cudaFree(d_pieces);
    cudaFree(d_cand);
    cudaFree(d_runs);
    cudaFree(d_reports);
    cudaFree(d_tmp);
    cudaFree(d_unique);
    cudaFree(d_hist);
    cudaFree(d_counters);
    cudaFree(d_carry);
    cudaFree(d_marks);
    cudaFree(d_ovf);
    cudaFree(d_unit_work);
    cudaFree(d_act);
    cudaFree(d_act_list);
    cudaFree(d_row_off);
    cudaFree(d_row_n);
    cudaFree(d_act_cnt);
    cudaFree(d_stk);
    cudaFree(d_stream_ids);
    if (graph) cudaGraphExecDestroy(graph);
    for (auto& g : sort_graphs) g.release();
    if (sort_cs) cudaStreamDestroy(sort_cs);
    for (auto& c : cap_ev)
      if (c) cudaEventDestroy(c);
    if (cap_stream) cudaStreamDestroy(cap_stream);
    if (ho.counters) cudaFreeHost(ho.counters);
    if (ho.reports) cudaFreeHost(ho.reports);
    if (ho.streams) cudaFreeHost(ho.streams);
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
    if (plan_ev) cudaEventSynchronize(plan_ev);
    if (plan_ev) cudaEventDestroy(plan_ev);
    if (h_plan) cudaFreeHost(h_plan);
  }
};

namespace {

// Candidates per run: one injection of a warp, and no more lists than a few
// refills of its worklist when they are long (tables of one level: hundreds
// of states per position), so that such runs spread over the warps.
int run_len(const TileHost& th) { return std::max(4, std::min(64, 2 * th.inj_batch)); }

}  // namespace

extern "C" {

int ngap_tables_build(const ngap_groups* g, const ngap_table_opts* opts, ngap_tables** out) {
  if (!g || !out) {
    set_error("ngap_tables_build: null argument");
    return NGAP_E_INVALID;
  }
  *out = nullptr;
  TableOpts to;
  int device = 0;
  int rc = table_opts_from(opts, "ngap_tables_build", to, &device);
  if (rc != NGAP_OK) return rc;
  std::unique_ptr<ngap_tables> t(new ngap_tables());
  t->device = device;
  CUDA_TRY(cudaSetDevice(device));
  rc = build_tiles(g->gs, to, t->tiles);
  if (rc != NGAP_OK) return rc;
  build_filters(t->tiles);
  t->num_groups = (int)g->gs.groups.size();
  for (const GroupGraph& gg : g->gs.groups) {
    t->sid_bits = std::max(t->sid_bits, bits_for(std::max<uint64_t>(gg.attrs.size(), 1)));
    for (uint8_t a : gg.attrs) t->report_states += a & 2 ? 1 : 0;
  }
  for (auto& th : t->tiles) {
    count_paths(th);
    t->report_paths += th.report_paths;
    t->paths_meet = t->paths_meet || (th.max_paths > 1 && !many_paths(th.max_paths));
    if (th.nstates >= kMaxTileStates - 1) {
      set_error("a connected component has %d states; at most %d are supported per tile",
                th.nstates, kMaxTileStates - 2);
      return NGAP_E_UNSUPPORTED;
    }
    t->max_states = std::max(t->max_states, th.nstates);
    t->tile_lean.push_back(th.nsticky == 0 && th.phase == 0 ? 1 : 0);
    t->run_len.push_back(run_len(th));
    TileDev d;
    d.group = th.group;
    d.nstates = th.nstates;
    d.naas = (int32_t)th.aas.size();
    d.nstart = (int32_t)th.start.size();
    d.depth = th.depth;
    d.max_path = th.max_path;
    d.ncls = th.ncls;
    d.cw = th.cw;
    d.nlive = th.nlive;
    d.image_bytes = (int32_t)th.image.size();
    d.off_cmask = th.off_cmask;
    d.off_rep = th.off_rep;
    d.off_cls = th.off_cls;
    d.inj_batch = th.inj_batch;
    d.inj_batch0 = th.inj_batch0;
    d.nsticky = th.nsticky;
    d.off_sticky = th.off_sticky;
    d.phase = th.phase;
    d.nact = th.nact;
    if (th.pair >= 0) {
      if ((int)t->pair_nact.size() <= th.pair) t->pair_nact.resize(th.pair + 1, 0);
      t->pair_nact[th.pair] = th.nact;
      t->max_nact = std::max(t->max_nact, th.nact);
    }
    if ((rc = t->upload(th.act_local, &d.act_local)) != NGAP_OK) return rc;
    if ((rc = t->upload(th.stk_union, &d.stk_union)) != NGAP_OK) return rc;
    if ((rc = t->upload(th.image, &d.image)) != NGAP_OK) return rc;
    if ((rc = t->upload(th.sid, &d.sid)) != NGAP_OK) return rc;
    if ((rc = t->upload(th.aas, &d.aas)) != NGAP_OK) return rc;
    if ((rc = t->upload(th.start, &d.start)) != NGAP_OK) return rc;
    d.run_len = run_len(th);
    d.one_by_one = many_paths(th.max_paths) ? 1 : 0;
    d.filt.len = th.filt.len;
    d.filt.min_rep = th.filt.min_rep;
    d.filt.shift = th.filt.shift;
    d.filt.drop = th.filt.drop;
    if ((rc = t->upload(th.filt.blocks, &d.filt.blocks)) != NGAP_OK) return rc;
    for (int k = 0; k < kMaxDepth; k++) {
      const PrefixTableHost& ph = th.pt[k];
      PrefixTableDev& pd = d.pt[k];
      pd.dense = ph.dense ? 1 : 0;
      pd.inline1 = ph.inline1 ? 1 : 0;
      pd.hmask = ph.hmask;
      pd.cutoff = ph.cutoff;
      pd.has_reports = ph.rlist.empty() ? 0 : 1;
      d.rep_levels |= (uint32_t)pd.has_reports << k;
      if ((rc = t->upload(ph.voff, &pd.voff)) != NGAP_OK) return rc;
      if ((rc = t->upload(ph.roff, &pd.roff)) != NGAP_OK) return rc;
      const uint32_t* slots = nullptr;
      if ((rc = t->upload(ph.slots, &slots)) != NGAP_OK) return rc;
      pd.slots = reinterpret_cast<const uint4*>(slots);
      if ((rc = t->upload(ph.vlist, &pd.vlist)) != NGAP_OK) return rc;
      if ((rc = t->upload(ph.rlist, &pd.rlist)) != NGAP_OK) return rc;
    }
    t->dev_desc.push_back(d);
  }
  const TileDev* dt = nullptr;
  if ((rc = t->upload(t->dev_desc, &dt)) != NGAP_OK) return rc;
  t->d_tiles = const_cast<TileDev*>(dt);
  *out = t.release();
  return NGAP_OK;
}

void ngap_tables_destroy(ngap_tables* t) { delete t; }

int64_t ngap_tables_device_bytes(const ngap_tables* t) { return t ? t->bytes : 0; }

int ngap_engine_create(int device, ngap_engine** out) {
  if (!out) {
    set_error("ngap_engine_create: null argument");
    return NGAP_E_INVALID;
  }
  *out = nullptr;
  int ndev = 0;
  CUDA_TRY(cudaGetDeviceCount(&ndev));
  if (device < 0 || device >= ndev) {
    set_error("no CUDA device %d (%d present)", device, ndev);
    return NGAP_E_CUDA;
  }
  CUDA_TRY(cudaSetDevice(device));
  std::unique_ptr<ngap_engine> e(new ngap_engine());
  e->device = device;
  CUDA_TRY(cudaDeviceGetAttribute(&e->num_sms, cudaDevAttrMultiProcessorCount, device));
  CUDA_TRY(cudaMalloc(&e->d_counters, kNumCounters * sizeof(unsigned long long)));
  CUDA_TRY(cudaMemset(e->d_counters, 0, kNumCounters * sizeof(unsigned long long)));
  CUDA_TRY(cudaFuncSetAttribute(sort_unique_cta<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSmallSortSmem));
  CUDA_TRY(cudaFuncSetAttribute(sort_unique_cta<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSmallSortSmem));
  CUDA_TRY(cudaFuncSetAttribute(scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kScanWarps * kScanWarpBytes));
  for (auto kernel : {run_kernel<false, false>, run_kernel<false, true>, run_kernel<true, false>,
                      run_kernel<true, true>})
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, run_smem_bytes()));
  CUDA_TRY(cudaMallocHost(&e->ho.counters, kNumCounters * sizeof(unsigned long long)));
  CUDA_TRY(cudaMallocHost(&e->ho.reports, kHostReports * sizeof(uint64_t)));
  CUDA_TRY(cudaMallocHost(&e->ho.streams, kHostReports * sizeof(uint32_t)));
  std::memset(e->ho.counters, 0, kNumCounters * sizeof(unsigned long long));
  e->ho.d_counters = e->d_counters;
  for (auto& ev : e->ev) CUDA_TRY(cudaEventCreate(&ev));
  *out = e.release();
  return NGAP_OK;
}

void ngap_engine_destroy(ngap_engine* e) {
  if (e) {
    cudaSetDevice(e->device);
    delete e;
  }
}

}  // extern "C"

namespace {

// New capacity of a grow-only buffer that must hold `need` elements: at
// least twice the old one, so that a run of growing plans reallocates (a
// cudaMalloc, which waits for the device) only a few times.
template <class T>
T grown(T cap, T need) {
  return std::max(need, cap * 2);
}

// One host array to copy to a device buffer.
struct Upload {
  void* dst;
  const void* src;
  size_t bytes;
};

// Copies plan arrays to the device on stream st through the engine's pinned
// staging buffer, so that the host does not wait: a synchronous copy from
// pageable memory queues behind other streams' transfers on the copy
// engine (in a serving loop, the other slot's input copy). The staging
// buffer is written again only once the last upload has ended (an event).
// Inside a stream capture the copies stay synchronous, so that no captured
// node reads the reusable staging buffer.
int upload_plan(ngap_engine* e, cudaStream_t st, const std::vector<Upload>& parts) {
  size_t total = 0;
  for (const Upload& u : parts) total += (u.bytes + 15) & ~(size_t)15;
  if (total == 0) return NGAP_OK;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CUDA_TRY(cudaStreamIsCapturing(st, &cs));
  if (cs != cudaStreamCaptureStatusNone) {
    for (const Upload& u : parts)
      if (u.bytes) CUDA_TRY(cudaMemcpy(u.dst, u.src, u.bytes, cudaMemcpyHostToDevice));
    return NGAP_OK;
  }
  if (e->plan_ev_pending) {
    CUDA_TRY(cudaEventSynchronize(e->plan_ev));
    e->plan_ev_pending = false;
  }
  if (total > e->h_plan_cap) {
    const size_t cap = grown(e->h_plan_cap, total);
    if (e->h_plan) cudaFreeHost(e->h_plan);
    e->h_plan = nullptr;
    e->h_plan_cap = 0;
    CUDA_TRY(cudaMallocHost(&e->h_plan, cap));
    e->h_plan_cap = cap;
  }
  if (!e->plan_ev) CUDA_TRY(cudaEventCreateWithFlags(&e->plan_ev, cudaEventDisableTiming));
  size_t off = 0;
  for (const Upload& u : parts) {
    if (u.bytes == 0) continue;
    std::memcpy(e->h_plan + off, u.src, u.bytes);
    CUDA_TRY(cudaMemcpyAsync(u.dst, e->h_plan + off, u.bytes, cudaMemcpyHostToDevice, st));
    off += (u.bytes + 15) & ~(size_t)15;
  }
  CUDA_TRY(cudaEventRecord(e->plan_ev, st));
  e->plan_ev_pending = true;
  return NGAP_OK;
}

// Whether a match reads its input where the caller has it: device memory of
// this GPU whose start and length are multiples of 16. Otherwise it is copied into
// the engine's padded buffer (16 MiB: 10 us of a 190 us call on a B200).
bool input_in_place(const ngap_engine* e, const uint8_t* input, int on_device, uint64_t bytes) {
  return reads_in_place(input, on_device != 0, bytes, e->device, [](const void* p) {
    InputMemory m;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) {
      m.device = a.type == cudaMemoryTypeDevice;
      m.owner = a.device;
    } else {
      cudaGetLastError();  // an address the runtime does not know is copied
    }
    return m;
  });
}

// Last input byte that the scan may read. (A count would not fit: the 16-byte
// units of an input just below 4 GiB end at 2^32.)
uint32_t last_readable(uint64_t bytes) { return (uint32_t)((bytes - 1) | 15u); }

// The engine's input buffer, padded for those reads.
int ensure_input(ngap_engine* e, uint64_t bytes) {
  const size_t need = ((bytes + 15) & ~(uint64_t)15) + 64;
  if (need <= e->input_cap) return NGAP_OK;
  e->buffers++;
  cudaFree(e->d_input);
  e->d_input = nullptr;
  e->input_cap = 0;
  CUDA_TRY(cudaMalloc(&e->d_input, need));
  e->input_cap = need;
  return NGAP_OK;
}

int ensure_reports(ngap_engine* e, uint64_t cap) {
  if (cap <= e->rep_cap) return NGAP_OK;
  e->buffers++;
  cudaFree(e->d_reports);
  cudaFree(e->d_tmp);
  cudaFree(e->d_unique);
  cudaFree(e->d_hist);
  e->d_reports = e->d_tmp = e->d_unique = nullptr;
  e->d_hist = nullptr;
  e->rep_cap = 0;
  CUDA_TRY(cudaMalloc(&e->d_reports, cap * sizeof(uint64_t)));
  CUDA_TRY(cudaMalloc(&e->d_tmp, cap * sizeof(uint64_t)));
  CUDA_TRY(cudaMalloc(&e->d_unique, cap * sizeof(uint64_t)));
  size_t ntiles = (cap + kSortTile - 1) / kSortTile;
  e->hist_cap = kDigits * ntiles + kDigits;
  CUDA_TRY(cudaMalloc(&e->d_hist, e->hist_cap * sizeof(uint32_t)));
  e->rep_cap = cap;
  return NGAP_OK;
}

// Scratch of the resident warps of `ctas` CTAs: carry lists, bitmaps and sticky
// lists for the warps of match_kernel, worklists for those and for the runs' warps,
// which use the same memory in turn (run_queue).
int ensure_slots(ngap_engine* e, size_t ctas, int max_states, int max_nact, int queue) {
  int ovf_cap = queue + kQueueSpare;
  int carry_cap = std::max(max_states, 32);
  int mark_words = (max_states + 31) / 32 + 1;
  size_t slots = ctas * kWarpsPerCta;
  // the overflow stacks only grow: a request for fewer entries than held
  // keeps them (more room changes no result, while reallocating would
  // cudaFree, which waits for every stream of the device)
  if (e->d_ovf && ovf_cap < e->ovf_cap) ovf_cap = e->ovf_cap;
  if (ovf_cap != e->ovf_cap && e->d_ovf) {  // queue capacity grew: reallocate everything
    e->slots = std::max(e->slots, slots);
    slots = e->slots;
    e->carry_cap = 0;
  }
  const int stk_cap = max_nact > kStickyCap ? max_nact : 0;
  if (slots <= e->slots && stk_cap > e->stk_cap) {  // only the sticky lists grow
    e->buffers++;
    cudaFree(e->d_stk);
    e->d_stk = nullptr;
    e->stk_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_stk, e->slots * 2 * (size_t)stk_cap * sizeof(uint32_t)));
    e->stk_cap = stk_cap;
  }
  if (slots <= e->slots && carry_cap <= e->carry_cap && mark_words <= e->mark_words) return NGAP_OK;
  e->buffers++;
  cudaFree(e->d_carry);
  cudaFree(e->d_marks);
  cudaFree(e->d_ovf);
  cudaFree(e->d_stk);
  e->d_carry = e->d_marks = e->d_ovf = e->d_stk = nullptr;
  e->stk_cap = 0;
  e->ovf_words = 0;
  slots = std::max(slots, e->slots);
  e->slots = 0;
  if (stk_cap > 0) {
    CUDA_TRY(cudaMalloc(&e->d_stk, slots * 2 * (size_t)stk_cap * sizeof(uint32_t)));
    e->stk_cap = stk_cap;
  }
  CUDA_TRY(cudaMalloc(&e->d_carry, slots * (size_t)carry_cap * sizeof(uint32_t)));
  CUDA_TRY(cudaMalloc(&e->d_marks, slots * (size_t)mark_words * sizeof(uint32_t)));
  CUDA_TRY(cudaMemset(e->d_marks, 0, slots * (size_t)mark_words * sizeof(uint32_t)));
  const size_t words = slots * std::max<size_t>(ovf_cap, (size_t)run_queue(ovf_cap) * kRunWarps / kWarpsPerCta);
  CUDA_TRY(cudaMalloc(&e->d_ovf, words * sizeof(uint32_t)));
  e->ovf_words = words;
  e->slots = slots;
  e->carry_cap = carry_cap;
  e->mark_words = mark_words;
  e->ovf_cap = ovf_cap;
  return NGAP_OK;
}

// Splits the work into units: unbounded tiles get one unit per segment;
// bounded tiles are cut into chunks of emitted positions (AutoChunk when the
// caller gives no length), each with max_path - 1 positions of warm-up (clamped
// at the segment start).
// One independent input range (a segment, or a whole stream in batched mode).
struct SegSpec {
  int64_t lo, hi;
  bool starts;      // start-of-data states active at lo
  uint64_t key_hi;  // stream index in the report key
  int64_t base;     // offsets in reports are relative to this
  int32_t index;    // segment or stream index
};

// The launch that runs a tile (make_units): 0 activation tiles, 1 plain tiles
// without sticky states, 2 the rest.
int launch_of(const TileHost& th) {
  return th.phase == 1 ? 0 : (th.phase == 0 && th.nsticky == 0 ? 1 : 2);
}

// Chunk length of bounded tiles when the caller gives none. Long inputs: the
// window's length less the warm-up (a unit is then one window), which is best
// while it gives every warp several units. Shorter ones (positions: those of
// the launch's bounded tiles) are cut to one unit per warp, because a warp
// walks its unit serially and idle warps gain nothing; below 128 positions the
// warm-up and a unit's start cost more than the shorter walk gains. Match times
// on a B200 by chunk length (128, 384, 1024, 2048): 64 literals on 1 MiB 61, 43,
// 47, 61 us; 200 25-mers on 3 MB 1769, 1617, 1516, 2646 us; a server's burst
// of four batches 748, 809, 1090, 1484 us; 1000 25-mers on 16 MiB (more units
// than warps at any of them) 895, 405, 258, 260 us.
struct AutoChunk {
  static constexpr int64_t kShortest = 1024;  // unless that gives fewer units than warps
  int64_t positions[3] = {0, 0, 0};  // of bounded tiles, per launch
  int64_t warps = 1;
  void add(const TileHost& th, int64_t len) {
    if (th.max_path >= 0) positions[launch_of(th)] += len;
  }
  int64_t chunk(const TileHost& th, int window) const {
    const int64_t warm = th.max_path > 0 ? th.max_path - 1 : 0;
    const int64_t base = std::max<int64_t>(window, 2048);
    const int64_t longest = std::max<int64_t>(base - warm, base / 2);
    const int64_t share = (positions[launch_of(th)] + warps - 1) / warps;
    return std::min(longest, std::max<int64_t>({(share + 63) & ~(int64_t)63, 128, warm}));
  }
};

// Tiles that are scanned: acyclic ones with a filter, in plans with at least
// kScanMin of work (scan_work). Below, a scan and its runs are two kernels whose
// start costs more than looking every position up: an 81-byte line matches
// in 22 us in match_kernel and 30 us scanned, 64 literals on 1 MiB in 43 and 33.
bool is_scanned(const TileHost& th, bool blocking) {
  return th.filt.len > 0 && th.max_path >= 0 && !(blocking && many_paths(th.max_paths));
}

// Positions and the states that a look-up of each would inject at prefix depth
// `depth` (keys equally likely), with the levels that follow; layered tiles test
// their sticky states instead.
double scan_work(const TileHost& th, int depth, bool blocking, int64_t positions) {
  if (!is_scanned(th, blocking)) return 0.0;
  if (th.phase == 2) return (double)positions * (1 + th.nact);
  const int d = std::max(1, std::min(depth, th.depth));
  return (double)positions * (1 + 4 * (double)th.pt[d - 1].entries / std::pow((double)std::max(1, th.nlive), d));
}

void add_pieces(const TileHost& th, int tile, const SegSpec& s, int64_t len,
                std::pair<int64_t, int32_t> act, std::vector<PieceDev> pieces[2]) {
  PieceDev p{};
  p.tile = tile;
  p.end = (uint32_t)s.hi;
  p.base = (uint32_t)s.base;
  p.key_hi = s.key_hi;
  p.act_row = act.first;
  p.act_rowid = act.second;
  p.pad = s.index;
  const bool starts = s.starts && !th.start.empty();
  int64_t hi = s.lo;
  for (int64_t lo = s.lo; lo < s.hi; lo = hi) {
    hi = std::min((lo + len) & ~(int64_t)7, s.hi);  // later pieces start where the scan reads, at multiples of 8
    p.lo = (uint32_t)lo;
    p.hi = (uint32_t)hi;
    p.flags = starts && lo == s.lo ? 1u : 0u;
    pieces[th.phase == 2 ? 1 : 0].push_back(p);
  }
}

void add_units(const TileHost& th, int tile, const SegSpec& s, int64_t chunk,
               std::pair<int64_t, int32_t> act, std::vector<UnitDev>& pass1,
               std::vector<UnitDev>& unbounded, std::vector<UnitDev>& bounded) {
  UnitDev u{};
  u.tile = tile;
  u.key_hi = s.key_hi;
  u.base = s.base;
  u.act_row = act.first;
  u.act_rowid = act.second;
  u.stream = s.index;
  std::vector<UnitDev>& chunks = th.phase == 1 ? pass1 : bounded;
  const bool starts = s.starts && !th.start.empty();
  if (th.max_path < 0) {
    u.flags = starts ? 1u : 0u;
    u.lo = s.lo;
    u.hi = s.hi;
    u.emit_lo = s.lo;
    unbounded.push_back(u);
    return;
  }
  const int64_t warm = th.max_path > 0 ? th.max_path - 1 : 0;
  for (int64_t em = s.lo; em < s.hi; em += chunk) {
    u.lo = std::max(s.lo, em - warm);
    u.hi = std::min(em + chunk, s.hi);
    u.emit_lo = em;
    u.flags = (starts && u.lo == s.lo) ? 1u : 0u;
    chunks.push_back(u);
  }
}

// Activation rows: one per (tables index, pair, segment), nact slots each;
// the slots of pair q of tables n start at base[n][q], its rows at rbase[n][q].
struct ActRows {
  std::vector<std::vector<int64_t>> base;
  std::vector<std::vector<int32_t>> rbase;
  std::vector<int64_t> row_off;  // per row: first slot
  std::vector<int32_t> row_n;    // per row: slots
  int64_t total = 0;
  ActRows(const std::vector<const ngap_tables*>& ts, int64_t nseg) {
    for (const ngap_tables* t : ts) {
      base.emplace_back();
      rbase.emplace_back();
      for (int32_t nact : t->pair_nact) {
        base.back().push_back(total);
        rbase.back().push_back((int32_t)row_off.size());
        for (int64_t g = 0; g < nseg; g++) {
          row_off.push_back(total + g * nact);
          row_n.push_back(nact);
        }
        total += (int64_t)nact * nseg;
      }
    }
  }
  // (first slot, row id) of a unit of tile th over segment seg; (-1, -1) for plain tiles
  std::pair<int64_t, int32_t> row(int n, const TileHost& th, int64_t seg) const {
    if (th.pair < 0) return {-1, -1};
    return {base[n][th.pair] + seg * th.nact, rbase[n][th.pair] + (int32_t)seg};
  }
};

// Units (already grouped by tile) in launch order: the activation tiles; the
// plain tiles without sticky states (is_lean: the lean kernel instance, with
// fewer registers spilled and a smaller code path); the rest. Within a launch the long
// units of cyclic tiles come first. A launch whose units all belong to one
// tile has its CTAs stage that tile's descriptors in shared memory.
PlanRanges make_units(std::vector<UnitDev>& units, const std::vector<UnitDev>& pass1,
                      const std::vector<UnitDev>& unbounded, const std::vector<UnitDev>& bounded,
                      const std::vector<char>& lean) {
  PlanRanges r;
  units.clear();
  auto append = [&](const std::vector<UnitDev>& v, int which) {
    for (const UnitDev& u : v)
      if (which == 0 || (lean[u.tile] != 0) == (which == 1)) units.push_back(u);
  };
  for (int which = 0; which < 3; which++) {
    r.begin[which] = (int32_t)units.size();
    if (which == 0) {
      append(pass1, 0);
    } else {
      append(unbounded, which);
      append(bounded, which);
    }
    r.count[which] = (int32_t)units.size() - r.begin[which];
    for (int32_t i = r.begin[which]; i < (int32_t)units.size(); i++) {
      if (i == r.begin[which]) r.one_tile[which] = units[i].tile;
      else if (units[i].tile != r.one_tile[which]) r.one_tile[which] = -1;
    }
  }
  return r;
}

ActRows plan_units(const ngap_tables* t, const UnitPlanKey& k, int grid,
                   std::vector<UnitDev>& units, std::vector<PieceDev> pieces[2], PlanRanges& ranges) {
  std::vector<UnitDev> pass1, unbounded, bounded;
  ActRows rows({t}, k.num_seg);
  AutoChunk ac;
  ac.warps = (int64_t)grid * kWarpsPerCta;
  int64_t scanned = 0;
  double work = 0;
  for (const TileHost& th : t->tiles) work += scan_work(th, k.depth, k.blocking, k.num_seg * k.seg_len);
  const bool scan = k.filtered && work >= kScanMin;
  auto scans = [&](const TileHost& th) { return scan && is_scanned(th, k.blocking); };
  for (const TileHost& th : t->tiles) {
    if (scans(th)) scanned += k.num_seg * k.seg_len;
    else ac.add(th, k.num_seg * k.seg_len);
  }
  const int64_t piece = piece_len(scanned, (int64_t)grid * kScanWarps, k.chunk);
  for (int ti = 0; ti < (int)t->tiles.size(); ti++) {
    const TileHost& th = t->tiles[ti];
    const int64_t chunk = k.chunk > 0 ? k.chunk : ac.chunk(th, k.window);
    for (int64_t s = 0; s < k.num_seg; s++) {
      SegSpec sp{s * k.seg_len, (s + 1) * k.seg_len, k.first_seg + s == 0 || k.is_dup != 0, 0ull,
                 0, (int32_t)s};
      if (scans(th))
        add_pieces(th, ti, sp, piece, rows.row(0, th, s), pieces);
      else
        add_units(th, ti, sp, chunk, rows.row(0, th, s), pass1, unbounded, bounded);
    }
  }
  ranges = make_units(units, pass1, unbounded, bounded, t->tile_lean);
  return rows;
}

int64_t longest_unit(const std::vector<UnitDev>& units) {
  int64_t n = 0;
  for (const UnitDev& u : units) n = std::max(n, u.hi - u.lo);
  return n;
}

// An automatic window no longer than the plan's longest unit: the shared
// memory that longer windows would take is left to L1, which holds small
// filters and tables (64 literals on 1 MiB, chunks of 384: 43 us with windows of
// 2048 positions, 37 us with 1024).
int fit_window(int window, int64_t longest) {
  return (int)std::min<int64_t>(window, std::max<int64_t>(64, (longest + 63) & ~(int64_t)63));
}

// Per-unit work counters when tracing (zeroed on st); null otherwise.
// d_unit_work holds two arrays of unit_work_cap words: work, then cycles
int trace_buffer(ngap_engine* e, cudaStream_t st, unsigned long long** work,
                 unsigned long long** cycles) {
  *work = *cycles = nullptr;
  if (!e->trace || e->h_units.empty()) return NGAP_OK;
  if (e->h_units.size() > e->unit_work_cap) {
    e->buffers++;
    const size_t cap = grown(e->unit_work_cap, e->h_units.size());
    cudaFree(e->d_unit_work);
    e->d_unit_work = nullptr;
    e->unit_work_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_unit_work, 2 * cap * sizeof(unsigned long long)));
    e->unit_work_cap = cap;
  }
  CUDA_TRY(cudaMemsetAsync(e->d_unit_work, 0, 2 * e->unit_work_cap * sizeof(unsigned long long), st));
  *work = e->d_unit_work;
  *cycles = e->d_unit_work + e->unit_work_cap;
  return NGAP_OK;
}

// Drops the cached plan before another one is made: a plan that cannot be
// finished (an allocation fails) leaves neither the old one, whose buffers may be
// gone, nor half of its own. The next match plans again.
void forget_plan(ngap_engine* e) {
  e->plan_tables = 0;
  e->plan_key = UnitPlanKey{-1, -1, -1, -1, -1, -1, -1, false, true};
  e->batch_ts = 0;
}

// Device copies of a plan's units and pieces, and buffers for its largest slice;
// as large as `room` asks for where that is more.
int set_plan(ngap_engine* e, const std::vector<UnitDev>& units, const std::vector<PieceDev> pieces[2],
             const std::vector<int32_t>& run_len, const PlanRoom& room, std::vector<PieceDev>& all,
             std::vector<Upload>& ups) {
  all = pieces[0];
  all.insert(all.end(), pieces[1].begin(), pieces[1].end());
  int64_t cands = 0, runs = 0;
  e->ranges.slices = make_slices(pieces, run_len, &cands, &runs);
  cands = std::max(cands, room.cands);
  runs = std::max(runs, room.runs);
  const size_t nunits = std::max(units.size(), (size_t)room.units);
  const size_t npieces = std::max(all.size(), (size_t)room.pieces);
  if (nunits > e->units_cap) {
    e->buffers++;
    const size_t cap = grown(e->units_cap, nunits);
    cudaFree(e->d_units);
    e->d_units = nullptr;
    e->units_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_units, cap * sizeof(UnitDev)));
    e->units_cap = cap;
  }
  if (npieces > e->pieces_cap) {
    e->buffers++;
    const size_t cap = grown(e->pieces_cap, npieces);
    cudaFree(e->d_pieces);
    e->d_pieces = nullptr;
    e->pieces_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_pieces, cap * sizeof(PieceDev)));
    e->pieces_cap = cap;
  }
  if (cands > e->cand_cap) {
    e->buffers++;
    const int64_t cap = std::max(cands, std::min<int64_t>(grown(e->cand_cap, cands), kSlicePositions));
    cudaFree(e->d_cand);
    e->d_cand = nullptr;
    e->cand_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_cand, (size_t)cap * sizeof(uint16_t)));
    e->cand_cap = cap;
  }
  if (runs > e->runs_cap) {
    e->buffers++;
    const int64_t cap = std::max(runs, std::min<int64_t>(grown(e->runs_cap, runs), kSliceRuns));
    cudaFree(e->d_runs);
    e->d_runs = nullptr;
    e->runs_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_runs, (size_t)cap * sizeof(RunDev)));
    e->runs_cap = cap;
  }
  if (!units.empty()) ups.push_back({e->d_units, units.data(), units.size() * sizeof(UnitDev)});
  if (!all.empty()) ups.push_back({e->d_pieces, all.data(), all.size() * sizeof(PieceDev)});
  e->nunits = (int32_t)units.size();
  e->longest_unit = longest_unit(units);
  // host records of the traces: the units, then the pieces
  e->h_units = units;
  for (const PieceDev& p : all) {
    UnitDev u{};
    u.tile = p.tile;
    u.lo = u.emit_lo = p.lo;
    u.hi = p.hi;
    u.base = p.base;
    u.stream = p.pad;
    e->h_units.push_back(u);
  }
  return NGAP_OK;
}

// Activation buffers of a plan (slots, compacted lists, row table).
int set_act_rows(ngap_engine* e, const ActRows& rows, std::vector<Upload>& ups) {
  e->act_entries = rows.total;
  e->act_rows = (int32_t)rows.row_off.size();
  if (e->act_entries > e->act_cap) {
    e->buffers++;
    const int64_t cap = grown(e->act_cap, e->act_entries);
    cudaFree(e->d_act);
    cudaFree(e->d_act_list);
    e->d_act = e->d_act_list = nullptr;
    e->act_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_act, (size_t)cap * sizeof(uint32_t)));
    CUDA_TRY(cudaMalloc(&e->d_act_list, (size_t)cap * sizeof(uint32_t)));
    e->act_cap = cap;
  }
  if (e->act_rows > e->rows_cap) {
    e->buffers++;
    const int32_t cap = grown(e->rows_cap, e->act_rows);
    cudaFree(e->d_row_off);
    cudaFree(e->d_row_n);
    cudaFree(e->d_act_cnt);
    e->d_row_off = nullptr;
    e->d_row_n = nullptr;
    e->d_act_cnt = nullptr;
    e->rows_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_row_off, (size_t)cap * sizeof(int64_t)));
    CUDA_TRY(cudaMalloc(&e->d_row_n, (size_t)cap * sizeof(int32_t)));
    CUDA_TRY(cudaMalloc(&e->d_act_cnt, (size_t)cap * sizeof(uint32_t)));
    e->rows_cap = cap;
  }
  if (e->act_rows > 0) {
    ups.push_back({e->d_row_off, rows.row_off.data(), rows.row_off.size() * sizeof(int64_t)});
    ups.push_back({e->d_row_n, rows.row_n.data(), rows.row_n.size() * sizeof(int32_t)});
  }
  return NGAP_OK;
}

// One warp per activation row: the slots with a first match, in slot order.
__global__ void act_compact(const int64_t* __restrict__ row_off, const int32_t* __restrict__ row_n,
                            int32_t nrows, const uint32_t* __restrict__ act,
                            uint32_t* __restrict__ list, uint32_t* __restrict__ cnt) {
  const int32_t row = (int32_t)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= nrows) return;  // whole warps
  const int64_t off = row_off[row];
  const int32_t n = row_n[row];
  uint32_t c = 0;
  for (int32_t i0 = 0; i0 < n; i0 += 256) {  // eight reads in flight per lane: the reads are the time
    uint32_t a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int32_t i = i0 + 32 * k + lane;
      a[k] = i < n ? act[off + i] : 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const bool ok = a[k] != 0xffffffffu;
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (ok) list[off + c + __popc(m & ((1u << lane) - 1u))] = (uint32_t)(i0 + 32 * k + lane);
      c += __popc(m);
    }
  }
  if (lane == 0) cnt[row] = c;
}

// CTAs of a launch: one per unit up to the whole grid, so that few units spread
// over as many SMs.
int launch_grid(int64_t nunits, int grid) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(grid, nunits));
}

// The matching launches of a plan: the activation tiles' work; the plain
// tiles without sticky states in the lean kernel instance; then the rest
// (the layered tiles read what the first launch recorded).
int launch_plan(ngap_engine* e, MatchParams mp, const std::vector<TileDev>& tiles, int smem,
                uint32_t last, cudaStream_t st) {
  auto set_marks = [](MatchParams& m, int longest) {
    const WorklistMarks k = worklist_marks(kStackCap + m.ovf_cap, longest);
    m.mark_inject = k.inject;
    m.mark_walk = k.walk;
    m.mark_single = k.single;
  };
  set_marks(mp, mp.window);
  MatchParams rp = mp;  // the runs': no windows, paths to their end
  rp.ovf_cap = run_queue(mp.ovf_cap);
  set_marks(rp, kMaxRunPath);
  if (e->act_entries > 0)
    CUDA_TRY(cudaMemsetAsync(e->d_act, 0xff, (size_t)e->act_entries * sizeof(uint32_t), st));
  auto run = [&](bool lean, int which) -> int {
    if (e->ranges.count[which] == 0) return NGAP_OK;
    mp.unit_begin = e->ranges.begin[which];
    mp.nunits = e->ranges.count[which];
    mp.one_tile = e->ranges.one_tile[which];
    mp.unit_cursor = reinterpret_cast<unsigned int*>(e->d_counters + kCursors + which);
    const int grid = launch_grid(mp.nunits, e->grid);
    if (lean)
      match_kernel<true><<<grid, kCtaThreads, smem, st>>>(mp);
    else
      match_kernel<false><<<grid, kCtaThreads, smem, st>>>(mp);
    CUDA_TRY(cudaGetLastError());
    e->launches++;
    return NGAP_OK;
  };
  ScanParams sp;
  sp.tiles = mp.tiles;
  sp.pieces = e->d_pieces;
  sp.input = mp.input;
  sp.last = last;
  sp.cand = e->d_cand;
  sp.runs = e->d_runs;
  sp.act_cnt = e->d_act_cnt;
  sp.cycles = mp.unit_cycles ? mp.unit_cycles + e->nunits : nullptr;
  rp.piece_unit0 = e->nunits;
  unsigned int* const ctl0 = reinterpret_cast<unsigned int*>(e->d_counters + kSliceCtl);
  auto run_slices = [&](bool layered) -> int {
    for (size_t i = 0; i < e->ranges.slices.size(); i++) {
      const Slice& s = e->ranges.slices[i];
      if (s.layered != layered) continue;
      unsigned int* ctl = ctl0 + (i % kSliceSlots) * kCtlWords;
      if (i >= kSliceSlots) CUDA_TRY(cudaMemsetAsync(ctl, 0, kCtlWords * sizeof(unsigned int), st));
      sp.piece_begin = (uint32_t)s.begin;
      sp.npieces = (uint32_t)s.count;
      sp.ctl = ctl;
      sp.one_tile = s.one_tile;
      if (s.one_tile >= 0) {  // described in the parameters: no reads before the scan
        const TileDev& td = tiles[s.one_tile];
        sp.filt = td.filt;
        sp.cls = td.image + td.off_cls;
        sp.nlive = (uint32_t)td.nlive;
        sp.run_len = td.run_len;
        sp.phase = td.phase;
      }
      // strips of 16 where a piece fills the warp with them
      sp.strip_bits = s.longest >= 32 * kStripMax ? 4 : 3;
      scan_kernel<<<launch_grid(s.count, e->grid), kScanWarps * 32, kScanWarps * kScanWarpBytes, st>>>(sp);
      const int grid = launch_grid(s.runs, e->grid);
      const auto kernel = layered ? (mp.unique ? run_kernel<true, true> : run_kernel<true, false>)
                                  : (mp.unique ? run_kernel<false, true> : run_kernel<false, false>);
      kernel<<<grid, kRunWarps * 32, run_smem_bytes(), st>>>(rp, e->d_cand, e->d_runs, ctl);
      CUDA_TRY(cudaGetLastError());
      e->launches += 2;
    }
    return NGAP_OK;
  };
  int rc = run(false, 0);
  if (rc == NGAP_OK) rc = run(true, 1);
  if (rc == NGAP_OK) rc = run_slices(false);
  if (rc != NGAP_OK) return rc;
  if (e->act_rows > 0) {
    act_compact<<<(e->act_rows + 7) / 8, 256, 0, st>>>(e->d_row_off, e->d_row_n, e->act_rows,
                                                       e->d_act, e->d_act_list, e->d_act_cnt);
    CUDA_TRY(cudaGetLastError());
    e->launches++;
  }
  if ((rc = run(false, 2)) != NGAP_OK) return rc;
  return run_slices(true);
}

__global__ void swap_halves(uint64_t* a, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t x = a[i];
    a[i] = (x << 32) | (x >> 32);
  }
}

// The dynamic shared-memory limit is an attribute of the kernel function
// (per device, shared by every engine of the process), so it only ever grows.
std::mutex g_smem_mu;
int g_smem_set[64];

int set_smem(ngap_engine* e, int smem) {
  if (e->max_smem_set >= smem) return NGAP_OK;
  std::lock_guard<std::mutex> lock(g_smem_mu);
  const int dev = e->device & 63;
  if (g_smem_set[dev] >= smem) {
    e->max_smem_set = g_smem_set[dev];
    return NGAP_OK;
  }
  const void* kernels[2] = {(const void*)match_kernel<false>, (const void*)match_kernel<true>};
  cudaError_t ce = cudaSuccess;
  for (int k = 0; k < 2 && ce == cudaSuccess; k++)
    ce = cudaFuncSetAttribute(kernels[k], cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (ce != cudaSuccess) {
    set_error("shared memory request of %d bytes rejected: %s", smem, cudaGetErrorString(ce));
    return NGAP_E_CUDA;
  }
  g_smem_set[dev] = smem;
  e->max_smem_set = smem;
  return NGAP_OK;
}

// Resident CTAs per SM, cached for the engine's last shared-memory size (the
// occupancy query costs a driver call on every match otherwise).
int blocks_per_sm(ngap_engine* e, int smem, int* out) {
  if (e->bps_smem != smem) {
    int n = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, match_kernel<false>, kCtaThreads, smem));
    if (n < 1) {
      set_error("the matching kernel does not fit on an SM with %d bytes of shared memory", smem);
      return NGAP_E_CUDA;
    }
    e->bps_smem = smem;
    e->bps_val = n;
  }
  *out = e->bps_val;
  return NGAP_OK;
}

// The radix pipeline over *radix_n keys; adds its launches to *kernels.
int radix_chain(ngap_engine* e, const SortJob& j, const unsigned long long* radix_n,
                cudaStream_t st, int* kernels) {
  const uint32_t max_tiles = (uint32_t)((j.cap + kSortTile - 1) / kSortTile);
  const int grid = (int)std::max<uint32_t>(1, std::min<uint32_t>(max_tiles, e->num_sms * 8));
  // ping-pong between d_in (an engine-owned buffer) and d_tmp
  uint64_t* src = j.d_in;
  uint64_t* dst = e->d_tmp;
  uint32_t* totals = e->d_hist + e->hist_cap - kDigits;
  for (int sh : j.shifts) {
    radix_hist<<<grid, kSortThreads, 0, st>>>(src, radix_n, j.cap, sh, e->d_hist);
    radix_scan<<<kDigits, kSortThreads, 0, st>>>(e->d_hist, radix_n, j.cap, totals);
    radix_scatter<<<grid, kSortThreads, 0, st>>>(src, dst, radix_n, j.cap, sh, e->d_hist, totals);
    *kernels += 3;
    std::swap(src, dst);
  }
  unique_count<<<grid, kSortThreads, 0, st>>>(src, radix_n, j.cap, e->d_hist);
  scan_exclusive_1block<<<1, kScanThreads, 0, st>>>(e->d_hist, radix_n, j.cap, j.d_unique_n);
  if (j.mode == 0)
    unique_write<0><<<grid, kSortThreads, 0, st>>>(src, radix_n, j.cap, e->d_hist, j.oshift, j.sshift,
                                                   j.d_out, nullptr);
  else
    unique_write<1><<<grid, kSortThreads, 0, st>>>(src, radix_n, j.cap, e->d_hist, j.oshift, j.sshift,
                                                   j.d_out, j.d_out_stream);
  *kernels += 3;
  CUDA_TRY(cudaGetLastError());
  return NGAP_OK;
}

// Last kernel of a match whose reports went through the radix pipeline.
int publish(ngap_engine* e, const SortJob& j, cudaStream_t st, int* kernels) {
  publish_results<<<1, kHostReports, 0, st>>>(e->ho, j.d_unique_n, j.d_out, j.d_out_stream);
  *kernels += 1;
  CUDA_TRY(cudaGetLastError());
  return NGAP_OK;
}

// The one-CTA sort of at most `most` keys.
int cta_sort(ngap_engine* e, const SortJob& j, uint64_t most, const HostOut& ho, cudaStream_t st) {
  unsigned long long* radix_n = e->d_counters + kRadixCount;
  const cudaGraphConditionalHandle none = 0;
  if (j.mode == 0)
    sort_unique_cta<0><<<1, kSmallThreads, kSmallSortSmem, st>>>(
        j.d_in, e->d_tmp, j.d_n, j.cap, radix_n, j.d_unique_n, j.oshift, j.sshift, j.d_out,
        j.d_out_stream, none, 0, most, ho);
  else
    sort_unique_cta<1><<<1, kSmallThreads, kSmallSortSmem, st>>>(
        j.d_in, e->d_tmp, j.d_n, j.cap, radix_n, j.d_unique_n, j.oshift, j.sshift, j.d_out,
        j.d_out_stream, none, 0, most, ho);
  CUDA_TRY(cudaGetLastError());
  e->launches++;
  return NGAP_OK;
}

// Builds the graph: the one-CTA sort, then the radix pipeline in the body of a
// conditional (IF) node whose condition the first kernel sets when it leaves
// keys to the pipeline.
int build_sort_graph(ngap_engine* e, const SortJob& j, SortGraph& sg) {
  if (!e->sort_cs) CUDA_TRY(cudaStreamCreateWithFlags(&e->sort_cs, cudaStreamNonBlocking));
  CUDA_TRY(cudaGraphCreate(&sg.g, 0));
  cudaGraphConditionalHandle h = 0;
  CUDA_TRY(cudaGraphConditionalHandleCreate(&h, sg.g, 0, cudaGraphCondAssignDefault));
  unsigned long long* radix_n = e->d_counters + kRadixCount;
  SortJob a = j;  // kernel arguments
  uint64_t* d_tmp = e->d_tmp;
  int set_cond = 1;
  uint64_t most = kSmallSort;
  HostOut ho = e->ho;
  void* args[] = {&a.d_in, &d_tmp, &a.d_n, &a.cap, &radix_n, &a.d_unique_n, &a.oshift, &a.sshift,
                  &a.d_out, &a.d_out_stream, &h, &set_cond, &most, &ho};
  cudaKernelNodeParams kp = {};
  kp.func = j.mode == 0 ? reinterpret_cast<void*>(sort_unique_cta<0>)
                        : reinterpret_cast<void*>(sort_unique_cta<1>);
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(kSmallThreads);
  kp.sharedMemBytes = kSmallSortSmem;
  kp.kernelParams = args;
  cudaGraphNode_t kn = nullptr, cn = nullptr;
  CUDA_TRY(cudaGraphAddKernelNode(&kn, sg.g, nullptr, 0, &kp));
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeIf;
  cp.conditional.size = 1;
  CUDA_TRY(cudaGraphAddNode(&cn, sg.g, &kn, 1, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  CUDA_TRY(cudaStreamBeginCaptureToGraph(e->sort_cs, body, nullptr, nullptr, 0,
                                         cudaStreamCaptureModeThreadLocal));
  int kernels = 0;
  int rc = radix_chain(e, j, radix_n, e->sort_cs, &kernels);
  if (rc == NGAP_OK) rc = publish(e, j, e->sort_cs, &kernels);
  cudaGraph_t captured = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(e->sort_cs, &captured);
  if (rc != NGAP_OK) return rc;
  CUDA_TRY(ce);
  CUDA_TRY(cudaGraphInstantiate(&sg.ge, sg.g, 0));
  sg.chain = kernels;
  return NGAP_OK;
}

// A match whose positions times its rules' report states are at most this sorts
// its reports with the one-CTA kernel, launched directly: a launch with a conditional
// graph costs 7 us more on a B200 (29 against 22 us for an empty pipeline), while
// one CTA keeps up with the pipeline only to some 30,000 reports. More keys than
// this can come all the same where several paths lead to a report, each of which
// emits it; the kernel then leaves them, and ngap_engine_sync launches the pipeline.
constexpr uint64_t kAloneReports = 1ull << 16;

// How many reports a match can give: without duplicates, and with them (positions
// times the paths that end in report states, TileHost::report_paths).
struct MostReports {
  double unique = 0, all = 0;
  void add(const ngap_tables* t, uint64_t positions) {
    if (positions == 0) return;
    unique += (double)positions * (double)t->report_states;
    all += (double)positions * t->report_paths;
  }
};

// Launches the pipeline for keys that the one-CTA kernel left, the match having ended
// on e->stream, and waits for it.
int finish_sort(ngap_engine* e) {
  if (!e->sort_open) return NGAP_OK;
  e->sort_open = false;
  if (e->ho.counters[kRadixCount] > 0) {
    int kernels = 0;
    int rc = radix_chain(e, e->sort_job, e->d_counters + kRadixCount, e->stream, &kernels);
    if (rc == NGAP_OK) rc = publish(e, e->sort_job, e->stream, &kernels);
    if (rc != NGAP_OK) return rc;
    e->launches += kernels;
    CUDA_TRY(cudaEventRecord(e->ev[3], e->stream));
    CUDA_TRY(cudaStreamSynchronize(e->stream));
  }
  e->counters_dirty = false;  // by whichever kernel came last
  return NGAP_OK;
}

// Enqueues the sort of a match's reports on st, the match's last kernels: they
// leave its counters and first reports for the host. Past
// kAloneReports, outside stream capture, it replays a cached graph (one launch; the
// radix pipeline runs only for more than kSmallSort keys); inside a
// capture, or where graphs are unavailable, it launches the one-CTA kernel and
// the pipeline, whose kernels find no keys after a small set.
int sort_reports(ngap_engine* e, const SortJob& j, const MostReports& most, cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CUDA_TRY(cudaStreamIsCapturing(st, &cs));
  if (cs == cudaStreamCaptureStatusNone && std::min(most.unique, most.all) <= kAloneReports) {
    e->sort_open = true;
    e->sort_job = j;
    return cta_sort(e, j, kAloneReports, e->ho, st);
  }
  if (cs != cudaStreamCaptureStatusNone && most.all <= kAloneReports)  // nobody would finish it
    return cta_sort(e, j, ~0ull, e->ho, st);
  if (cs == cudaStreamCaptureStatusNone && !e->sort_graph_off) {
    std::vector<uint64_t> key = {(uint64_t)j.mode,   (uint64_t)(uintptr_t)j.d_in,
                                 (uint64_t)(uintptr_t)j.d_n, j.cap,
                                 (uint64_t)j.oshift, (uint64_t)j.sshift,
                                 (uint64_t)(uintptr_t)j.d_out,
                                 (uint64_t)(uintptr_t)j.d_out_stream,
                                 (uint64_t)(uintptr_t)j.d_unique_n,
                                 (uint64_t)(uintptr_t)e->d_tmp, (uint64_t)(uintptr_t)e->d_hist};
    for (int sh : j.shifts) key.push_back((uint64_t)sh);
    SortGraph* sg = nullptr;
    for (auto& g : e->sort_graphs)
      if (g.key == key) sg = &g;
    if (!sg) {
      if (e->sort_graphs.size() >= 16) {  // keep a few configurations
        e->sort_graphs.front().release();
        e->sort_graphs.erase(e->sort_graphs.begin());
      }
      SortGraph ng;
      ng.key = key;
      if (build_sort_graph(e, j, ng) == NGAP_OK) {
        e->sort_graphs.push_back(ng);
        sg = &e->sort_graphs.back();
      } else {  // graphs unavailable here: launch the kernels directly from now on
        ng.release();
        cudaGetLastError();
        e->sort_graph_off = true;
      }
    }
    if (sg) {
      CUDA_TRY(cudaGraphLaunch(sg->ge, st));
      e->launches++;
      e->sort_chain_pending = sg->chain;
      return NGAP_OK;
    }
  }
  int rc = cta_sort(e, j, kSmallSort, HostOut(), st);
  int kernels = 0;
  if (rc == NGAP_OK) rc = radix_chain(e, j, e->d_counters + kRadixCount, st, &kernels);
  if (rc == NGAP_OK) rc = publish(e, j, st, &kernels);
  e->launches += kernels;
  return rc;
}

// Zeroes the counters when an earlier match was left half enqueued (otherwise
// its last kernel did), and marks them until this match is enqueued whole.
int begin_counters(ngap_engine* e, cudaStream_t st) {
  if (e->counters_dirty)
    CUDA_TRY(cudaMemsetAsync(e->d_counters, 0, kNumCounters * sizeof(unsigned long long), st));
  e->counters_dirty = true;
  e->sort_open = false;
  return NGAP_OK;
}

// Copies the first n reports (and stream indices) of the last match to the host.
cudaError_t copy_results(const ngap_engine* e, uint64_t n, uint64_t* reports, uint32_t* streams) {
  if (n <= (uint64_t)kHostReports) {  // left in pinned memory by the match
    std::memcpy(reports, e->ho.reports, n * sizeof(uint64_t));
    if (streams) std::memcpy(streams, e->ho.streams, n * sizeof(uint32_t));
    return cudaSuccess;
  }
  cudaError_t ce = cudaSetDevice(e->device);
  if (ce == cudaSuccess)
    ce = cudaMemcpy(reports, e->d_unique, n * sizeof(uint64_t), cudaMemcpyDeviceToHost);
  if (ce == cudaSuccess && streams)
    ce = cudaMemcpy(streams, e->d_stream_ids, n * sizeof(uint32_t), cudaMemcpyDeviceToHost);
  return ce;
}

// --algorithm -> prefix depth. The blocking algorithm scans the always-active
// list like NAP, over whole windows: windows of one position cost a TMA copy
// and a wait per position and tile (64 literals in ten groups on 1 MiB: 9466 us
// on a B200, 85 us with windows of 2048). Within a window it follows paths, not
// states: tiles in which many paths can meet (cyclic ones, above all, where they
// would double at every symbol) keep windows of one position, and where a few can
// duplicate entries of a step are dropped as with --unique (50 edit-distance rules:
// 1864 raw reports position by position, 6205 along all paths, 2119 like this, and
// 0.28 instead of 0.30 ms). R1, R2 and all ask for
// privatization, which the kernel does for every algorithm (walk_paths).
int algo_config(int algo, int table_depth, int* depth) {
  switch (algo) {
    case NGAP_ALGO_BLOCKING:
    case NGAP_ALGO_NAP: *depth = 0; break;
    case NGAP_ALGO_NONBLOCKING:
    case NGAP_ALGO_NONBLOCKING_R1:
    case NGAP_ALGO_NONBLOCKING_R2: *depth = 1; break;
    case NGAP_ALGO_NONBLOCKING_PC:
    case NGAP_ALGO_NONBLOCKING_ALL: *depth = std::max(1, table_depth); break;
    default:
      set_error("not supported algoritm %d", algo);
      return NGAP_E_INVALID;
  }
  return NGAP_OK;
}

}  // namespace

extern "C" {

int ngap_match(ngap_engine* e, const ngap_tables* t, const uint8_t* input, int input_on_device,
               const ngap_match_params* p, void* stream) {
  if (!e || !t || !p) {
    set_error("ngap_match: null argument");
    return NGAP_E_INVALID;
  }
  if (p->num_seg <= 0 || p->seg_len <= 0) {
    set_error("ngap_match: num_seg and seg_len must be positive");
    return NGAP_E_INVALID;
  }
  if (!input) {
    set_error("ngap_match: null argument (input)");
    return NGAP_E_INVALID;
  }
  // each factor below 2^32 first, so that the product cannot wrap
  const uint64_t total = p->num_seg < (1ll << 32) && p->seg_len < (1ll << 32)
                             ? (uint64_t)p->num_seg * (uint64_t)p->seg_len
                             : ~0ull;
  if (total >= (1ull << 32)) {
    set_error("ngap_match: input of %llu bytes exceeds the 32-bit offsets of the report format",
              (unsigned long long)total);
    return NGAP_E_UNSUPPORTED;
  }
  if (t->num_groups > 1024) {
    set_error("ngap_match: at most 1024 groups fit the 32-bit report id");
    return NGAP_E_UNSUPPORTED;
  }
  CUDA_TRY(cudaSetDevice(e->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  e->stream = st;
  e->launches = 0;
  e->sort_chain_pending = 0;
  e->ran = false;
  // automatic window: 2048 positions (against 1024: Hamming set 0.654 ->
  // 0.624 ms, high_frontier and the literal set 1-2 % faster; fit_window
  // shortens it below)
  int depth = 1, window = p->window > 0 ? p->window : 2048;
  int table_depth = 0;
  for (auto& th : t->tiles) table_depth = std::max(table_depth, th.depth);
  int rc = algo_config(p->algorithm, table_depth, &depth);
  if (rc != NGAP_OK) return rc;
  const bool blocking = p->algorithm == NGAP_ALGO_BLOCKING;
  window = std::min(window, kMaxWindow);
  const bool in_place = input_in_place(e, input, input_on_device, total);
  if (!in_place && (rc = ensure_input(e, total)) != NGAP_OK) return rc;
  uint64_t cap = p->result_capacity > 0 ? p->result_capacity : 54619400ull;
  if ((rc = ensure_reports(e, cap)) != NGAP_OK) return rc;
  // shared memory: the warps' (a window too large for it is shortened)
  while (window > 64 && cta_smem_bytes(window) > 227 * 1024 - 1024) window /= 2;
  int smem = cta_smem_bytes(window);
  if ((rc = set_smem(e, smem)) != NGAP_OK) return rc;
  int bps = 0;
  rc = blocks_per_sm(e, smem, &bps);
  if (rc != NGAP_OK) return rc;
  const int full_grid = e->num_sms * bps;
  // units
  UnitPlanKey key{p->num_seg, p->seg_len, p->is_dup ? 1 : 0, window, p->chunk, p->first_segment,
                  depth, blocking, e->test_skip_unit < 0};
  if (e->plan_tables != t->serial || key < e->plan_key || e->plan_key < key) {
    forget_plan(e);
    std::vector<UnitDev> units;
    std::vector<PieceDev> pieces[2], all;
    const ActRows rows = plan_units(t, key, full_grid, units, pieces, e->ranges);
    std::vector<Upload> ups;
    if ((rc = set_act_rows(e, rows, ups)) != NGAP_OK) return rc;
    if ((rc = set_plan(e, units, pieces, t->run_len, PlanRoom(), all, ups)) != NGAP_OK) return rc;
    if ((rc = upload_plan(e, st, ups)) != NGAP_OK) return rc;
    e->plan_tables = t->serial;
    e->plan_key = key;
  }
  if (p->window <= 0) {
    window = fit_window(window, e->longest_unit);
    smem = cta_smem_bytes(window);
  }
  e->grid = full_grid;
  // per-warp scratch for the full grid, whatever this plan uses: a later
  // larger plan then never reallocates (cudaMalloc waits for the device)
  rc = ensure_slots(e, (size_t)full_grid, t->max_states, t->max_nact, kDefaultQueue);
  if (rc != NGAP_OK) return rc;

  if (!in_place)
    CUDA_TRY(cudaMemcpyAsync(e->d_input, input, total,
                             input_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, st));
  if ((rc = begin_counters(e, st)) != NGAP_OK) return rc;

  MatchParams mp;
  mp.tiles = t->d_tiles;
  mp.units = e->d_units;
  mp.input = in_place ? input : e->d_input;
  mp.window = window;
  mp.depth = depth;
  mp.blocking = blocking;
  mp.unique = p->unique || (blocking && t->paths_meet);
  mp.report_off = p->report_off;
  mp.off_shift = 32;
  mp.rep_count = e->d_counters + 0;
  mp.reports = e->d_reports;
  mp.rep_cap = cap;
  mp.err = reinterpret_cast<int*>(e->d_counters + 4);
  mp.carry = e->d_carry;
  mp.marks = e->d_marks;
  mp.ovf = e->d_ovf;
  mp.carry_cap = e->carry_cap;
  mp.mark_words = e->mark_words;
  mp.ovf_cap = e->ovf_cap;
  mp.work = e->d_counters + 2;
  mp.act = e->d_act;
  mp.act_list = e->d_act_list;
  mp.act_cnt = e->d_act_cnt;
  mp.stk_g = e->d_stk;
  mp.stk_g_cap = e->stk_cap;
  mp.wait_rounds = e->test_wait_rounds > 0 ? e->test_wait_rounds : kWaitRounds;
  mp.skip_copy_unit = e->test_skip_unit;
  e->test_wait_rounds = 0;  // the hook covers one match
  e->test_skip_unit = -1;
  if ((rc = trace_buffer(e, st, &mp.unit_work, &mp.unit_cycles)) != NGAP_OK) return rc;
  e->trace_seg_len = p->seg_len;
  CUDA_TRY(cudaEventRecord(e->ev[1], st));
  if (!e->h_units.empty()) {
    rc = launch_plan(e, mp, t->dev_desc, smem, last_readable(total), st);
    if (rc != NGAP_OK) return rc;
  }
  CUDA_TRY(cudaEventRecord(e->ev[2], st));
  if (!p->report_off) {
    const uint64_t bits = bit_range(0, t->sid_bits) |
                          bit_range(22, bits_for((uint64_t)std::max(t->num_groups, 1))) |
                          bit_range(32, bits_for(total));
    const SortJob job{0,  e->d_reports, e->d_counters + 0, cap,     digits_of(bits),
                      32, 64,           e->d_unique,       nullptr, e->d_counters + 1};
    MostReports most;
    most.add(t, total);
    if ((rc = sort_reports(e, job, most, st)) != NGAP_OK) return rc;
  } else {
    publish_kernel<<<1, 32, 0, st>>>(e->ho);
    CUDA_TRY(cudaGetLastError());
    e->launches++;
  }
  CUDA_TRY(cudaEventRecord(e->ev[3], st));
  e->counters_dirty = e->sort_open;
  e->ran = true;
  return NGAP_OK;
}

int ngap_engine_sync(ngap_engine* e) {
  if (!e || !e->ran) {
    set_error("ngap_engine_sync: no match in flight");
    return NGAP_E_INVALID;
  }
  CUDA_TRY(cudaSetDevice(e->device));
  CUDA_TRY(cudaStreamSynchronize(e->stream));
  const int rc = finish_sort(e);
  if (rc != NGAP_OK) return rc;
  CUDA_TRY(cudaEventElapsedTime(&e->match_ms, e->ev[1], e->ev[2]));
  CUDA_TRY(cudaEventElapsedTime(&e->sort_ms, e->ev[2], e->ev[3]));
  if (e->sort_chain_pending > 0 && e->ho.counters[kRadixCount] > 0)  // the radix pipeline ran
    e->launches += e->sort_chain_pending;
  e->sort_chain_pending = 0;
  int err = (int)(e->ho.counters[4] & 0xffffffffull);
  if (err & kErrTimeout) {
    set_error("a bounded device wait gave up; results are incomplete");
    return NGAP_E_TIMEOUT;
  }
  if (err & (kErrQueue | kErrCarry)) {
    set_error("a worklist overflowed its capacity; results are incomplete");
    return NGAP_E_OVERFLOW_QUEUE;
  }
  if (err & kErrResults) {
    set_error("%llu reports exceed the result capacity of %llu; results are truncated",
              (unsigned long long)e->ho.counters[0], (unsigned long long)e->rep_cap);
    return NGAP_E_OVERFLOW_RESULTS;
  }
  return NGAP_OK;
}

int ngap_results_count(const ngap_engine* e, uint64_t* raw, uint64_t* unique) {
  if (!e) return NGAP_E_INVALID;
  if (raw) *raw = e->ho.counters[0];
  if (unique) *unique = e->ho.counters[1];
  return NGAP_OK;
}

const uint64_t* ngap_results_device(const ngap_engine* e) { return e ? e->d_unique : nullptr; }

int64_t ngap_results_copy(ngap_engine* e, uint64_t* host, uint64_t cap) {
  if (!e || !host) return -1;
  uint64_t n = std::min<uint64_t>(e->ho.counters[1], cap);
  if (n == 0) return 0;
  cudaError_t ce = copy_results(e, n, host, nullptr);
  if (ce != cudaSuccess) {
    set_error("cudaMemcpy: %s", cudaGetErrorString(ce));
    return -1;
  }
  return (int64_t)n;
}

int ngap_last_times_ms(const ngap_engine* e, float* match_ms, float* sort_ms) {
  if (!e) return NGAP_E_INVALID;
  if (match_ms) *match_ms = e->match_ms;
  if (sort_ms) *sort_ms = e->sort_ms;
  return NGAP_OK;
}

int ngap_last_launches(const ngap_engine* e) { return e ? e->launches : 0; }

int ngap_engine_work(const ngap_engine* e, uint64_t* expanded, uint64_t* injected) {
  if (!e) return NGAP_E_INVALID;
  if (expanded) *expanded = e->ho.counters[2];
  if (injected) *injected = e->ho.counters[3];
  return NGAP_OK;
}

int ngap_engine_memory(const ngap_engine* e, ngap_engine_mem* out) {
  if (!e || !out) {
    set_error("ngap_engine_memory: null argument");
    return NGAP_E_INVALID;
  }
  out->input = (int64_t)e->input_cap;
  out->reports = 3 * 8 * (int64_t)e->rep_cap + 4 * (int64_t)e->hist_cap + 4 * (int64_t)e->stream_ids_cap;
  out->scratch =
      (int64_t)e->slots * 4 * ((int64_t)e->carry_cap + e->mark_words + 2 * e->stk_cap) + 4 * (int64_t)e->ovf_words +
      (int64_t)sizeof(uint16_t) * e->cand_cap + (int64_t)sizeof(RunDev) * e->runs_cap;
  out->plan = 8 * (int64_t)e->act_cap + 16 * (int64_t)e->rows_cap + 16 * (int64_t)e->unit_work_cap +
              (int64_t)sizeof(UnitDev) * (int64_t)e->units_cap +
              (int64_t)sizeof(PieceDev) * (int64_t)e->pieces_cap;
  return NGAP_OK;
}

int64_t ngap_engine_device_bytes(const ngap_engine* e) {
  ngap_engine_mem m;
  if (ngap_engine_memory(e, &m) != NGAP_OK) return 0;
  return m.input + m.reports + m.scratch + m.plan;
}

int ngap_engine_test_wait_timeout(ngap_engine* e, int32_t unit, int32_t wait_rounds) {
  if (!e || unit < 0 || wait_rounds < 1) {
    set_error("ngap_engine_test_wait_timeout: needs an engine, a unit >= 0 and wait_rounds >= 1");
    return NGAP_E_INVALID;
  }
  e->test_skip_unit = unit;
  e->test_wait_rounds = wait_rounds;
  return NGAP_OK;
}

int ngap_engine_set_trace(ngap_engine* e, int enable) {
  if (!e) {
    set_error("ngap_engine_set_trace: null engine");
    return NGAP_E_INVALID;
  }
  e->trace = enable != 0;
  return NGAP_OK;
}

int ngap_trace_copy(ngap_engine* e, ngap_unit_trace* out, int64_t cap, int64_t* n) {
  if (!e || !n) {
    set_error("ngap_trace_copy: bad argument");
    return NGAP_E_INVALID;
  }
  *n = 0;
  if (!e->trace || !e->ran || e->h_units.empty() || !e->d_unit_work) return NGAP_OK;
  if (!out) {  // count query
    *n = (int64_t)e->h_units.size();
    return NGAP_OK;
  }
  std::vector<unsigned long long> work(e->h_units.size()), cycles(e->h_units.size());
  CUDA_TRY(cudaSetDevice(e->device));
  CUDA_TRY(cudaStreamSynchronize(e->stream));
  CUDA_TRY(cudaMemcpy(work.data(), e->d_unit_work, work.size() * sizeof(unsigned long long),
                      cudaMemcpyDeviceToHost));
  CUDA_TRY(cudaMemcpy(cycles.data(), e->d_unit_work + e->unit_work_cap,
                      cycles.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
  const int64_t m = std::min<int64_t>(cap, (int64_t)e->h_units.size());
  for (int64_t i = 0; i < m; i++) {
    const UnitDev& u = e->h_units[i];
    const int64_t base = e->trace_seg_len > 0 ? (int64_t)u.stream * e->trace_seg_len : u.base;
    out[i].stream = u.stream;
    out[i].tile = u.tile;
    out[i].lo = u.emit_lo - base;
    out[i].hi = u.hi - base;
    out[i].work = work[i];
    out[i].cycles = cycles[i];
  }
  *n = m;
  return NGAP_OK;
}

int ngap_tables_stats_get(const ngap_tables* t, ngap_tables_stats* out) {
  if (!t || !out) {
    set_error("ngap_tables_stats_get: null argument");
    return NGAP_E_INVALID;
  }
  ngap_tables_stats st{};
  st.tiles = (int32_t)t->tiles.size();
  for (const TileHost& th : t->tiles) {
    if (th.phase == 1) continue;  // activation tiles repeat states of their layered pair
    st.states += th.nstates;
    for (uint32_t u : th.succ) st.edges += u != kNoSucc ? 1 : 0;
    st.aas += (int32_t)th.aas.size();
    st.depth = std::max(st.depth, th.depth);
    st.max_nlive = std::max(st.max_nlive, th.nlive);
    const PrefixTableHost& pt = th.pt[th.depth - 1];
    st.list_entries += pt.entries;
    st.cutoff += pt.cutoff;
    double space = 1.0;
    for (int d = 0; d < th.depth; d++) space *= (double)std::max(1, th.nlive);
    st.exp_list += (double)pt.entries / space;
    st.max_list = std::max<int32_t>(st.max_list, pt.max_len);
  }
  *out = st;
  return NGAP_OK;
}

int ngap_reports_sort_unique(ngap_engine* e, const uint64_t* d_in, uint64_t n, uint64_t* d_out,
                             uint64_t* n_out, void* stream) {
  if (!e || (!d_in && n) || !d_out || !n_out) {
    set_error("ngap_reports_sort_unique: null argument");
    return NGAP_E_INVALID;
  }
  CUDA_TRY(cudaSetDevice(e->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  *n_out = 0;
  if (n == 0) return NGAP_OK;
  int rc = NGAP_OK;
  if (e->ran && e->sort_open) {  // the last match's reports are in the buffers used below
    CUDA_TRY(cudaStreamSynchronize(e->stream));
    if ((rc = finish_sort(e)) != NGAP_OK) return rc;
  }
  if ((rc = ensure_reports(e, n)) != NGAP_OK) return rc;
  // input arrives in the reference encoding (id << 32 | offset): swap halves
  // into sort keys in the engine's report buffer
  CUDA_TRY(cudaMemcpyAsync(e->d_reports, d_in, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
  unsigned long long hn = n;
  CUDA_TRY(cudaMemcpyAsync(e->d_counters + 5, &hn, sizeof(hn), cudaMemcpyHostToDevice, st));
  swap_halves<<<std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, 4096)), 256, 0, st>>>(e->d_reports, n);
  CUDA_TRY(cudaGetLastError());
  const SortJob job{0,  e->d_reports, e->d_counters + 5, n,       digits_of(~0ull),
                    32, 64,           d_out,             nullptr, e->d_counters + 6};
  int kernels = 0;
  rc = n <= (uint64_t)kSmallSort ? cta_sort(e, job, kSmallSort, HostOut(), st)
                                 : radix_chain(e, job, job.d_n, st, &kernels);
  if (rc != NGAP_OK) return rc;
  unsigned long long un = 0;
  CUDA_TRY(cudaMemcpyAsync(&un, e->d_counters + 6, sizeof(un), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(cudaStreamSynchronize(st));
  *n_out = un;
  return NGAP_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Batched matching: many streams, several NFAs, one persistent launch.
// ---------------------------------------------------------------------------

struct ngap_tableset {
  uint64_t serial = g_next_serial.fetch_add(1);
  std::vector<const ngap_tables*> tables;
  std::vector<int> tile_base;  // first tile of each NFA in the combined descriptor array
  TileDev* d_tiles = nullptr;
  int sid_bits = 0;
  int ntiles = 0, max_states = 0, max_groups = 1, max_depth = 1, device = 0;
  int max_nact = 0;
  bool paths_meet = false;          // in any of them
  BatchShape shape;                 // of its NFAs
  std::vector<TileDev> tiles;       // the combined array
  std::vector<char> tile_lean;      // per tile of it (ngap_tables::tile_lean)
  std::vector<int32_t> run_len;     // the same
  ~ngap_tableset() { cudaFree(d_tiles); }
};

extern "C" {

int ngap_tableset_create(const ngap_tables* const* tables, int n, ngap_tableset** out) {
  if (!tables || n <= 0 || !out) {
    set_error("ngap_tableset_create: bad argument");
    return NGAP_E_INVALID;
  }
  *out = nullptr;
  std::unique_ptr<ngap_tableset> ts(new ngap_tableset());
  std::vector<TileDev>& all = ts->tiles;
  for (int i = 0; i < n; i++) {
    const ngap_tables* t = tables[i];
    if (!t || (i > 0 && t->device != tables[0]->device)) {
      set_error("ngap_tableset_create: tables must exist and share one device");
      return NGAP_E_INVALID;
    }
    ts->tables.push_back(t);
    ts->tile_base.push_back((int)all.size());
    all.insert(all.end(), t->dev_desc.begin(), t->dev_desc.end());
    ts->tile_lean.insert(ts->tile_lean.end(), t->tile_lean.begin(), t->tile_lean.end());
    ts->run_len.insert(ts->run_len.end(), t->run_len.begin(), t->run_len.end());
    ts->max_states = std::max(ts->max_states, t->max_states);
    ts->max_groups = std::max(ts->max_groups, t->num_groups);
    ts->sid_bits = std::max(ts->sid_bits, t->sid_bits);
    ts->max_nact = std::max(ts->max_nact, t->max_nact);
    ts->paths_meet = ts->paths_meet || t->paths_meet;
    int64_t scanned = 0;
    for (auto& th : t->tiles) {
      ts->max_depth = std::max(ts->max_depth, th.depth);
      scanned += is_scanned(th, false);
    }
    BatchShape& sh = ts->shape;
    sh.tiles = std::max(sh.tiles, (int64_t)t->tiles.size());
    sh.scanned = std::max(sh.scanned, scanned);
    sh.plain = std::max(sh.plain, (int64_t)t->tiles.size() - scanned);
    for (int32_t n : t->run_len) sh.run_len = std::min<int64_t>(sh.run_len, n);
  }
  ts->device = tables[0]->device;
  ts->ntiles = (int)all.size();
  CUDA_TRY(cudaSetDevice(ts->device));
  if (!all.empty()) {
    CUDA_TRY(cudaMalloc(&ts->d_tiles, all.size() * sizeof(TileDev)));
    CUDA_TRY(cudaMemcpy(ts->d_tiles, all.data(), all.size() * sizeof(TileDev),
                        cudaMemcpyHostToDevice));
  }
  *out = ts.release();
  return NGAP_OK;
}

void ngap_tableset_destroy(ngap_tableset* ts) { delete ts; }

int ngap_batch_match(ngap_engine* e, const ngap_tableset* ts, const uint8_t* input,
                     uint64_t input_bytes, int input_on_device, const ngap_batch_stream* streams,
                     int nstreams, const ngap_batch_params* p, void* stream) {
  if (!e || !ts || !p || !streams || nstreams <= 0 || (!input && input_bytes > 0)) {
    set_error("ngap_batch_match: bad argument");
    return NGAP_E_INVALID;
  }
  uint64_t max_len = 1;
  for (int i = 0; i < nstreams; i++) {
    const ngap_batch_stream& s = streams[i];
    if (s.nfa < 0 || s.nfa >= (int)ts->tables.size() || s.offset > input_bytes ||
        s.length > input_bytes - s.offset) {  // no wrap-around of offset + length
      set_error("ngap_batch_match: stream %d is out of range", i);
      return NGAP_E_INVALID;
    }
    max_len = std::max<uint64_t>(max_len, s.length + 1);
  }
  if (input_bytes >= (1ull << 32)) {
    set_error("ngap_batch_match: batches are limited to 4 GiB of input");
    return NGAP_E_UNSUPPORTED;
  }
  // report key: stream | offset in stream | id
  const int ibits = 22 + bits_for((uint64_t)std::max(ts->max_groups, 1));
  int obits = bits_for(max_len);
  int sbits = bits_for((uint64_t)nstreams);
  // field widths rounded up to multiples of 4 bits when the key still fits: at
  // most one more 8-bit digit and far fewer distinct layouts, so that the sort's
  // CUDA graph (keyed by the layout) is reused across batches
  // of other lengths and stream counts instead of being captured again
  if (ibits + ((obits + 3) & ~3) + ((sbits + 3) & ~3) <= 64) {
    obits = (obits + 3) & ~3;
    sbits = (sbits + 3) & ~3;
  }
  const int oshift = ibits, sshift = ibits + obits;
  if (sshift + sbits > 64) {
    set_error("ngap_batch_match: stream count, stream length and group count exceed a 64-bit key");
    return NGAP_E_UNSUPPORTED;
  }
  CUDA_TRY(cudaSetDevice(e->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  e->stream = st;
  e->ran = false;
  // automatic window: 2048 positions (against 1024: Hamming set 0.654 ->
  // 0.624 ms, high_frontier and the literal set 1-2 % faster; fit_window
  // shortens it below)
  int depth = 1, window = p->window > 0 ? p->window : 2048;
  int rc = algo_config(p->algorithm, ts->max_depth, &depth);
  if (rc != NGAP_OK) return rc;
  const bool blocking = p->algorithm == NGAP_ALGO_BLOCKING;
  window = std::min(window, kMaxWindow);
  while (window > 64 && cta_smem_bytes(window) > 227 * 1024 - 1024) window /= 2;
  int smem = cta_smem_bytes(window);
  if ((rc = set_smem(e, smem)) != NGAP_OK) return rc;
  int bps = 0;
  rc = blocks_per_sm(e, smem, &bps);
  if (rc != NGAP_OK) return rc;
  const int full_grid = e->num_sms * bps;
  // buffers (before any capture)
  const bool in_place = input_in_place(e, input, input_on_device, input_bytes);
  if (!in_place && (rc = ensure_input(e, input_bytes)) != NGAP_OK) return rc;
  const uint64_t cap = p->result_capacity > 0 ? p->result_capacity : 54619400ull;
  if ((rc = ensure_reports(e, cap)) != NGAP_OK) return rc;
  if (cap > e->stream_ids_cap) {
    e->buffers++;
    cudaFree(e->d_stream_ids);
    e->d_stream_ids = nullptr;
    e->stream_ids_cap = 0;
    CUDA_TRY(cudaMalloc(&e->d_stream_ids, cap * sizeof(uint32_t)));
    e->stream_ids_cap = cap;
  }
  // plan: tiles outer, streams of the tile's NFA inner
  const std::vector<ngap_batch_stream> sv(streams, streams + nstreams);
  auto same_streams = [&]() {
    if (e->batch_streams.size() != sv.size()) return false;
    for (size_t i = 0; i < sv.size(); i++)
      if (sv[i].offset != e->batch_streams[i].offset || sv[i].length != e->batch_streams[i].length ||
          sv[i].nfa != e->batch_streams[i].nfa || sv[i].chunk != e->batch_streams[i].chunk)
        return false;
    return true;
  };
  bool replanned = false;
  if (e->batch_ts != ts->serial || e->batch_depth != depth ||
      e->batch_blocking != blocking || e->batch_window != window || e->batch_chunk != p->chunk ||
      !same_streams() || e->plan_tables != 0) {
    forget_plan(e);
    std::vector<std::vector<int>> by_nfa(ts->tables.size());
    for (int i = 0; i < nstreams; i++) by_nfa[sv[i].nfa].push_back(i);
    std::vector<UnitDev> pass1, unbounded, bounded, units;
    const ActRows rows(ts->tables, nstreams);
    AutoChunk ac;
    ac.warps = (int64_t)full_grid * kWarpsPerCta;
    int64_t scanned = 0;
    double work = 0;
    for (const ngap_batch_stream& s : sv)
      for (const TileHost& th : ts->tables[s.nfa]->tiles) work += scan_work(th, depth, blocking, (int64_t)s.length);
    auto scans = [&](const TileHost& th) { return work >= kScanMin && is_scanned(th, blocking); };
    for (const ngap_batch_stream& s : sv)
      for (const TileHost& th : ts->tables[s.nfa]->tiles) {
        if (scans(th)) scanned += (int64_t)s.length;
        else ac.add(th, (int64_t)s.length);
      }
    std::vector<PieceDev> pieces[2], all;
    for (size_t n = 0; n < ts->tables.size(); n++) {
      const ngap_tables* t = ts->tables[n];
      for (int ti = 0; ti < (int)t->tiles.size(); ti++) {
        const TileHost& th = t->tiles[ti];
        const int64_t auto_chunk = ac.chunk(th, window);
        for (int si : by_nfa[n]) {
          const ngap_batch_stream& s = sv[si];
          if (s.length == 0) continue;
          SegSpec sp{(int64_t)s.offset, (int64_t)(s.offset + s.length), true,
                     (uint64_t)si << sshift, (int64_t)s.offset, si};
          const int64_t chunk = s.chunk > 0 ? s.chunk : p->chunk;
          if (scans(th))
            add_pieces(th, ts->tile_base[n] + ti, sp,
                       piece_len(scanned, (int64_t)full_grid * kScanWarps, chunk),
                       rows.row((int)n, th, si), pieces);
          else
            add_units(th, ts->tile_base[n] + ti, sp, chunk > 0 ? chunk : auto_chunk,
                      rows.row((int)n, th, si), pass1, unbounded, bounded);
        }
      }
    }
    e->ranges = make_units(units, pass1, unbounded, bounded, ts->tile_lean);
    std::vector<Upload> ups;
    if ((rc = set_act_rows(e, rows, ups)) != NGAP_OK) return rc;
    BatchShape shape = ts->shape;
    shape.streams = nstreams;
    shape.chunk = AutoChunk::kShortest;
    for (const ngap_batch_stream& s : sv) {
      const int64_t chunk = s.chunk > 0 ? s.chunk : p->chunk;
      shape.positions += (int64_t)s.length;
      shape.chunk = std::min<int64_t>(shape.chunk, chunk > 0 ? chunk : AutoChunk::kShortest);
    }
    shape.warps = (int64_t)full_grid * kScanWarps;
    if (blocking) shape.plain = shape.tiles;  // tiles with a filter may be units too
    if ((rc = set_plan(e, units, pieces, ts->run_len, plan_room(shape), all, ups)) != NGAP_OK) return rc;
    if ((rc = upload_plan(e, st, ups)) != NGAP_OK) return rc;
    e->batch_ts = ts->serial;
    e->batch_streams = sv;
    e->batch_window = window;
    e->batch_depth = depth;
    e->batch_blocking = blocking;
    e->batch_chunk = p->chunk;
    replanned = true;
  }
  if (p->window <= 0) {
    window = fit_window(window, e->longest_unit);
    smem = cta_smem_bytes(window);
  }
  e->grid = full_grid;
  if ((rc = ensure_slots(e, (size_t)full_grid, ts->max_states, ts->max_nact,
                         p->queue_capacity > 0 ? std::max(p->queue_capacity, 1024) : kDefaultQueue)) != NGAP_OK)
    return rc;

  MatchParams mp;
  mp.tiles = ts->d_tiles;
  mp.units = e->d_units;
  mp.input = in_place ? input : e->d_input;
  mp.window = window;
  mp.depth = depth;
  mp.blocking = blocking;
  mp.unique = p->unique || (blocking && ts->paths_meet);
  mp.report_off = p->report_off;
  mp.off_shift = oshift;
  mp.rep_count = e->d_counters + 0;
  mp.reports = e->d_reports;
  mp.rep_cap = cap;
  mp.err = reinterpret_cast<int*>(e->d_counters + 4);
  mp.carry = e->d_carry;
  mp.marks = e->d_marks;
  mp.ovf = e->d_ovf;
  mp.carry_cap = e->carry_cap;
  mp.mark_words = e->mark_words;
  mp.ovf_cap = e->ovf_cap;
  mp.work = e->d_counters + 2;
  mp.act = e->d_act;
  mp.act_list = e->d_act_list;
  mp.act_cnt = e->d_act_cnt;
  mp.stk_g = e->d_stk;
  mp.stk_g_cap = e->stk_cap;
  mp.unit_work = mp.unit_cycles = nullptr;
  mp.wait_rounds = kWaitRounds;
  mp.skip_copy_unit = -1;
  e->trace_seg_len = 0;

  MostReports most;  // streams may share bytes of the input
  for (const ngap_batch_stream& s : sv) most.add(ts->tables[s.nfa], s.length);

  auto enqueue = [&](cudaStream_t qs) -> int {
    if (e->trace) {
      const int r = trace_buffer(e, qs, &mp.unit_work, &mp.unit_cycles);
      if (r != NGAP_OK) return r;
    }
    if (!in_place)
      CUDA_TRY(cudaMemcpyAsync(e->d_input, input, input_bytes,
                               input_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, qs));
    int r = NGAP_OK;
    if (!e->h_units.empty()) {
      r = launch_plan(e, mp, ts->tiles, smem, last_readable(input_bytes), qs);
      if (r != NGAP_OK) return r;
    }
    if (!p->report_off) {
      const uint64_t bits = bit_range(0, ts->sid_bits) | bit_range(22, ibits - 22) |
                            bit_range(oshift, obits) | bit_range(sshift, sbits);
      const SortJob job{1,      e->d_reports, e->d_counters + 0, cap,             digits_of(bits),
                        oshift, sshift,       e->d_unique,       e->d_stream_ids, e->d_counters + 1};
      if ((r = sort_reports(e, job, most, qs)) != NGAP_OK) return r;
    } else {
      publish_kernel<<<1, 32, 0, qs>>>(e->ho);
      CUDA_TRY(cudaGetLastError());
      e->launches++;
    }
    return NGAP_OK;
  };

  e->launches = 0;
  e->sort_chain_pending = 0;
  if (!p->use_graph) {
    e->graph_mode = false;
    CUDA_TRY(cudaEventRecord(e->ev[1], st));
    if ((rc = begin_counters(e, st)) != NGAP_OK) return rc;
    if ((rc = enqueue(st)) != NGAP_OK) return rc;
    e->counters_dirty = e->sort_open;
    CUDA_TRY(cudaEventRecord(e->ev[2], st));
    CUDA_TRY(cudaEventRecord(e->ev[3], st));
    e->ran = true;
    return NGAP_OK;
  }
  // CUDA graph: the same tableset, streams, parameters and input pointer replay
  // one captured pipeline (copy, match, sort, unique, counters). Capture and
  // replay use the engine's own stream (the legacy default stream cannot be
  // captured), ordered after and before the caller's stream by events.
  if (!e->cap_stream) {
    CUDA_TRY(cudaStreamCreateWithFlags(&e->cap_stream, cudaStreamNonBlocking));
    CUDA_TRY(cudaEventCreateWithFlags(&e->cap_ev[0], cudaEventDisableTiming));
    CUDA_TRY(cudaEventCreateWithFlags(&e->cap_ev[1], cudaEventDisableTiming));
  }
  cudaStream_t cs = e->cap_stream;
  std::vector<uint64_t> key = {ts->serial, (uint64_t)(uintptr_t)input, input_bytes,
                               (uint64_t)input_on_device, (uint64_t)in_place,
                               (uint64_t)p->algorithm,
                               (uint64_t)p->unique,
                               (uint64_t)p->report_off, cap, (uint64_t)window, (uint64_t)p->chunk,
                               (uint64_t)e->trace, (uint64_t)e->ovf_cap, e->buffers};
  if (replanned || !e->graph || key != e->graph_key) {
    if (e->graph) {
      cudaGraphExecDestroy(e->graph);
      e->graph = nullptr;
    }
    cudaGraph_t g = nullptr;
    CUDA_TRY(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    rc = enqueue(cs);
    cudaError_t ce = cudaStreamEndCapture(cs, &g);
    if (rc != NGAP_OK) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (ce != cudaSuccess) {
      set_error("CUDA graph capture failed: %s", cudaGetErrorString(ce));
      return NGAP_E_CUDA;
    }
    ce = cudaGraphInstantiate(&e->graph, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) {
      e->graph = nullptr;
      set_error("CUDA graph instantiation failed: %s", cudaGetErrorString(ce));
      return NGAP_E_CUDA;
    }
    e->graph_key = key;
    e->graph_launches = e->launches;
  }
  e->graph_mode = true;
  e->launches = e->graph_launches;
  CUDA_TRY(cudaEventRecord(e->cap_ev[0], st));  // after the caller's prior work
  CUDA_TRY(cudaStreamWaitEvent(cs, e->cap_ev[0], 0));
  CUDA_TRY(cudaEventRecord(e->ev[1], cs));
  if ((rc = begin_counters(e, cs)) != NGAP_OK) return rc;
  CUDA_TRY(cudaGraphLaunch(e->graph, cs));
  e->counters_dirty = false;
  CUDA_TRY(cudaEventRecord(e->ev[2], cs));
  CUDA_TRY(cudaEventRecord(e->ev[3], cs));
  CUDA_TRY(cudaEventRecord(e->cap_ev[1], cs));  // the caller's later work waits for the graph
  CUDA_TRY(cudaStreamWaitEvent(st, e->cap_ev[1], 0));
  e->stream = cs;
  e->ran = true;
  return NGAP_OK;
}

int ngap_batch_results(ngap_engine* e, uint64_t* reports, uint32_t* stream_ids, uint64_t cap,
                       uint64_t* n) {
  if (!e || !reports || !n) {
    set_error("ngap_batch_results: null argument");
    return NGAP_E_INVALID;
  }
  const uint64_t k = std::min<uint64_t>(e->ho.counters[1], cap);
  *n = 0;
  if (k == 0) return NGAP_OK;
  CUDA_TRY(copy_results(e, k, reports, stream_ids));
  *n = k;
  return NGAP_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Report sort + unique without any device allocation.
//
// Some callers cannot call cudaMalloc: a serving process whose device memory
// is owned by another allocator (a framework's caching allocator that has
// reserved the GPU), or a latency-critical loop where cudaMalloc's implicit
// device synchronisation is not acceptable. For them the scratch of the
// report sort lives in the file-scope array below, reserved on every GPU that
// loads this library until the process exits. It holds one ping-pong key
// buffer of kNoAllocMaxReports entries plus the digit histograms and
// counters (about 2 MiB). All calls share it and it keeps the last call's
// contents: calls whose work overlaps on the GPU (other streams, other host
// threads) race on it and must be serialised by the caller.
// ---------------------------------------------------------------------------
#include <mutex>

namespace {

constexpr uint64_t kNoAllocMaxReports = 1ull << 18;  // 262,144 reports
constexpr uint64_t kNoAllocTiles = (kNoAllocMaxReports + kSortTile - 1) / kSortTile;
constexpr size_t kNoAllocKeyBytes = kNoAllocMaxReports * sizeof(uint64_t);
constexpr size_t kNoAllocHistBytes = (kDigits * kNoAllocTiles + kDigits) * sizeof(uint32_t);
constexpr size_t kNoAllocBytes = kNoAllocKeyBytes + kNoAllocHistBytes + 4 * sizeof(unsigned long long);

static __device__ __align__(256) uint8_t g_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
constexpr int kNoAllocMaxDevices = 64;
uint8_t* g_noalloc_addr[kNoAllocMaxDevices] = {};
uint64_t g_noalloc_ctx[kNoAllocMaxDevices] = {};  // context the address belongs to

// Device address of the scratch array on the current device. In host code
// g_noalloc_scratch names a host-side stand-in, not device memory, so the
// address is looked up with that device current: once per device, and again
// whenever the device's current context is another one than at the lookup
// (after cudaDeviceReset, or a context the caller made current), whose
// address the old one is not.
int noalloc_scratch(int dev, uint8_t** out) {
  if (dev < 0 || dev >= kNoAllocMaxDevices) {
    set_error("device %d is beyond the %d devices the allocation-free path supports", dev,
              kNoAllocMaxDevices);
    return NGAP_E_INVALID;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  const uint64_t ctx = current_context_id();
  if (!g_noalloc_addr[dev] || !ctx || ctx != g_noalloc_ctx[dev]) {
    void* p = nullptr;
    cudaError_t ce = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (ce != cudaSuccess) {
      g_noalloc_addr[dev] = nullptr;
      set_error("cudaGetSymbolAddress of the sort scratch failed: %s", cudaGetErrorString(ce));
      return NGAP_E_CUDA;
    }
    g_noalloc_addr[dev] = static_cast<uint8_t*>(p);
    // the runtime may have made the primary context current just now
    g_noalloc_ctx[dev] = ctx ? ctx : current_context_id();
  }
  *out = g_noalloc_addr[dev];
  return NGAP_OK;
}

// Copies reference-encoded reports into sort keys (offset << 32 | id) and
// resets the counters: [0] = n, [1] = unique count.
__global__ void noalloc_prepare(const uint64_t* __restrict__ in, uint64_t n,
                                uint64_t* __restrict__ keys, unsigned long long* counters) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[0] = n;
    counters[1] = 0;
    counters[2] = 0;
    counters[3] = 0;
  }
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t x = in[i];
    keys[i] = (x << 32) | (x >> 32);
  }
}

}  // namespace

extern "C" int ngap_reports_sort_unique_noalloc(const uint64_t* d_in, uint64_t n, uint64_t* d_out,
                                                uint64_t* n_out, void* stream) {
  if ((!d_in && n) || !d_out || !n_out) {
    set_error("ngap_reports_sort_unique_noalloc: null argument");
    return NGAP_E_INVALID;
  }
  if (n > kNoAllocMaxReports) {
    set_error("ngap_reports_sort_unique_noalloc: %llu reports exceed the allocation-free "
              "maximum of %llu", (unsigned long long)n, (unsigned long long)kNoAllocMaxReports);
    return NGAP_E_INVALID;
  }
  *n_out = 0;
  if (n == 0) return NGAP_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  CUDA_TRY(cudaStreamIsCapturing(st, &cap));
  if (cap != cudaStreamCaptureStatusNone) {  // the call waits for the stream below
    set_error("ngap_reports_sort_unique_noalloc waits for its stream to return the unique "
              "count, so it cannot run while that stream is being captured");
    return NGAP_E_INVALID;
  }
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  uint8_t* base = nullptr;
  int rc = noalloc_scratch(dev, &base);
  if (rc != NGAP_OK) return rc;
  uint64_t* keys = reinterpret_cast<uint64_t*>(base);
  uint32_t* hist = reinterpret_cast<uint32_t*>(base + kNoAllocKeyBytes);
  unsigned long long* counters =
      reinterpret_cast<unsigned long long*>(base + kNoAllocKeyBytes + kNoAllocHistBytes);
  int sms = 0;
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint32_t tiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
  const int grid = (int)std::max<uint32_t>(1, std::min<uint32_t>(tiles, (uint32_t)sms * 8));
  // 4 digit passes over the id half and 4 over the offset half; an even count
  // leaves the sorted keys back in the scratch buffer, d_out being the other
  // half of the ping-pong
  const std::vector<int> shifts = digits_of(~0ull);
  uint32_t* totals = hist + kDigits * kNoAllocTiles;
  uint64_t* src = (shifts.size() % 2 == 0) ? keys : d_out;
  uint64_t* dst = (shifts.size() % 2 == 0) ? d_out : keys;
  noalloc_prepare<<<grid, 256, 0, st>>>(d_in, n, src, counters);
  for (int sh : shifts) {
    radix_hist<<<grid, kSortThreads, 0, st>>>(src, counters, n, sh, hist);
    radix_scan<<<kDigits, kSortThreads, 0, st>>>(hist, counters, n, totals);
    radix_scatter<<<grid, kSortThreads, 0, st>>>(src, dst, counters, n, sh, hist, totals);
    std::swap(src, dst);
  }
  unique_count<<<grid, kSortThreads, 0, st>>>(src, counters, n, hist);
  scan_exclusive_1block<<<1, kScanThreads, 0, st>>>(hist, counters, n, counters + 1);
  unique_write<0><<<grid, kSortThreads, 0, st>>>(src, counters, n, hist, 32, 64, d_out, nullptr);
  CUDA_TRY(cudaGetLastError());
  unsigned long long un = 0;
  CUDA_TRY(cudaMemcpyAsync(&un, counters + 1, sizeof(un), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(cudaStreamSynchronize(st));
  *n_out = un;
  return NGAP_OK;
}
