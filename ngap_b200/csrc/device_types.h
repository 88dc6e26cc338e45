// Structures shared by host table building and device kernels.
#pragma once

#include <vector_types.h>

#include <cstdint>

namespace ngap {

constexpr uint32_t kNoSucc = 0xffffffffu;
// act_local of layered tiles: local id of the slot's sticky state in the low
// 28 bits; bit 28 + j set when the state enables its successor j from its
// first match on (a shortcut) rather than from the next position
constexpr uint32_t kActIdMask = 0x0fffffffu;
constexpr int kMaxDepth = 12;        // prefix-memoization depth limit (the reference stops at 3)
constexpr int kEntryPosBits = 13;    // worklist entry = local_state << 13 | window offset
constexpr int kMaxWindow = (1 << kEntryPosBits) - 2;
constexpr int kMaxTileStates = 1 << (32 - kEntryPosBits);
constexpr uint64_t kDenseKeys = 1ull << 18;     // prefix tables with <= 2^18 keys are dense
constexpr uint64_t kMaxDenseKeys = 1ull << 26;  // larger ones are dense when that is smaller

constexpr uint32_t kHashEmpty = 0xffffffffu;

// One prefix-memoization table of depth d for a tile (precompute_table.h:8-101).
// The key is the live class ids c_0 .. c_{d-1} of the next d input bytes as a
// base-L number (L = TileDev::nlive): ((c_0 * L + c_1) * L + ...) + c_{d-1}.
// A byte of the dead class (accepted by no state of the tile) ends every path,
// so keys never contain it. dense: offsets indexed by the key (key space
// <= kDenseKeys); otherwise an open-addressing hash table (linear probing,
// capacity a power of two, at least twice the keys) whose slots hold
// {key, state-list begin, report-list begin, state-list length << 16 |
// report-list length}; the reference binary-searches a sorted key array
// (precompute_table.h:59-100).
// inline1 (dense tables without report lists): voff holds one word per key
// [space]: kHashEmpty for an empty list, the state itself (bit 31 clear) for
// a list of one, else bit 31 | begin << 6 | length (2..63) into vlist; most
// keys of a deep table have at most one state, so a lookup is one read.
struct PrefixTableDev {
  int32_t dense = 0;
  uint32_t hmask = 0;               // hash capacity - 1
  int32_t cutoff = 0;
  int32_t has_reports = 0;          // any report list non-empty
  int32_t inline1 = 0;
  int32_t pad = 0;
  const uint32_t* voff = nullptr;   // dense: state-list offsets [space + 1], or inline1 words
  const uint32_t* roff = nullptr;   // dense: report-list offsets [space + 1] (if reports)
  const uint4* slots = nullptr;     // hashed: [hmask + 1]
  const uint32_t* vlist = nullptr;  // local states reached after d symbols
  const uint32_t* rlist = nullptr;  // local report states reached after d symbols
};

__host__ __device__ inline uint32_t prefix_hash(uint32_t key) {
  return (key * 0x9E3779B1u) ^ (key >> 15);
}

// Look-ahead filter of a tile: a blocked Bloom filter (Putze, Sanders and
// Singler, 2007) over the next `len` class ids. A position is in it when some
// state the tile injects there leads to a path that is alive after `len` symbols
// or reports within them, so a position that is not in it needs no injection at
// all. hash = sum of c_i * kFilterMul^(len - 1 - i) over the class ids c_i, modulo
// 2^32. The top bits of hash * kFilterBlock choose a 64-bit block (one read), the
// top 15 bits of hash * kFilterBits three bits of it (filter_has). A position
// with fewer than len symbols left in its segment needs injection when at least
// min_rep are left (the shortest path to a report). len = 0: no filter.
// Measured on a B200 against a bitmap with one bit per key and twice the bits
// (match times): 200 25-mers with three table levels 387 -> 204 us, 50
// edit-distance 20-mers 175 -> 134, 1000 25-mers 156 -> 131 (4 % -> 1 % of the
// positions pass), the 32 MiB mix 616 -> 548, 512 streams 3.02 -> 2.66 ms.
constexpr int kMaxFilter = 16;       // most symbols a filter looks ahead
// odd multipliers: the first prime of xxHash32 and the two of MurmurHash3's 32-bit finalizer
constexpr uint32_t kFilterMul = 0x9E3779B1u;
constexpr uint32_t kFilterBlock = 0x85EBCA6Bu;
constexpr uint32_t kFilterBits = 0xC2B2AE35u;

struct FilterDev {
  int32_t len = 0;
  int32_t min_rep = 1;
  int32_t shift = 0;                // block = (hash * kFilterBlock) >> shift
  uint32_t drop = 0;                // kFilterMul^len: weight of the symbol that leaves a rolling hash
  const uint64_t* blocks = nullptr;
};

// The three bits of a block: two of its low word, one of its high word.
__host__ __device__ inline uint64_t filter_mask(uint32_t hash) {
  const uint32_t x = (hash * kFilterBits) >> 17;
  return 1ull << (x & 31) | 1ull << ((x >> 5) & 31) | 1ull << (32 + (x >> 10));
}

// A tile: a set of whole CCs (of one group, or of several for a global tile),
// matched by one warp per unit. Its hot tables form one contiguous image, read
// in place through L1 and L2:
//   [succ][cmask: nstates x cw x u32][rep: ceil(nstates/32) x u32][cls: 256 B]
// succ: a 32-byte record per state, so that an expansion is one read: up to 4
// tile-local successors (u32, bit 31 = report successor, kNoSucc = none), then
// for each what it accepts: its class mask in tiles of at most 32 classes (0 for
// none), otherwise the one class it accepts, kNoClass for none or
// kManyClasses (its mask is in cmask). cmask: bit c of word c/32 = the state
// accepts byte class c. cls: byte -> class id, live classes first, the dead
// class (bytes no state accepts) last.
constexpr uint32_t kNoClass = 0xfffffffeu;
constexpr uint32_t kManyClasses = 0xffffffffu;

struct TileDev {
  int32_t group = 0;        // group of the first CC (report ids are in sid)
  int32_t nstates = 0;
  int32_t naas = 0;
  int32_t nstart = 0;
  int32_t depth = 0;        // prefix depth built for this tile (>= 1)
  int32_t max_path = -1;    // longest path in states if acyclic, else -1
  int32_t ncls = 0;         // byte classes
  int32_t cw = 8;           // class-mask words per state: ceil(classes / 32), 1..8
  int32_t nlive = 0;        // live classes: key base; class id nlive = dead
  int32_t image_bytes = 0;  // multiple of 16
  int32_t off_cmask = 0, off_rep = 0, off_cls = 0;
  int32_t inj_batch = 32;   // positions injected per worklist refill (prefix tables)
  int32_t inj_batch0 = 32;  // the same when the always-active list is scanned
  int32_t nsticky = 0;      // sticky states (bitmap at off_sticky in the image)
  int32_t off_sticky = 0;
  int32_t phase = 0;        // 0 plain; 1 activation pass; 2 layered (sticky states pre-registered)
  int32_t nact = 0;         // activation slots per segment (phase 1 and 2)
  const uint32_t* act_local = nullptr;  // phase 2: [nact] each slot's sticky state (kActIdMask)
  const uint32_t* stk_union = nullptr;  // phase 2: [nact][cw] classes any successor accepts
  const uint8_t* image = nullptr;   // global copy of the image (16-byte aligned)
  const uint32_t* sid = nullptr;    // [nstates] local -> report id (sid | group << 22)
  const uint32_t* aas = nullptr;    // [naas] local ids
  const uint32_t* start = nullptr;  // [nstart] local ids
  int32_t run_len = 32;     // filter candidates per run
  int32_t one_by_one = 0;   // blocking algorithm: windows of one position (many_paths)
  uint32_t rep_levels = 0;  // bit d: the depth-(d+1) table has report lists
  FilterDev filt;
  PrefixTableDev pt[kMaxDepth];
};

// Whether so many paths can end in one state at one position that following them one
// by one is out of bounds: `most` of them, infinite in a cyclic tile. The blocking
// algorithm, which looks at a state once a position, then works in windows of
// one position, whose states are carried to the next without duplicates;
// elsewhere it takes whole windows (algo_config). The line: edit-distance rules
// (two edits in 20 symbols: at most 466 paths) are far better off in whole windows,
// where few of those paths are ever alive (50 rules on 1 MiB: 318 ms in windows of
// one position, 0.33 ms scanned on a B200); a bound far above theirs says that
// paths multiply.
constexpr double kManyPaths = 1024;
inline bool many_paths(double most) { return !(most <= kManyPaths); }

// A unit of work: one tile over input positions [lo, hi); reports are kept for
// positions >= emit_lo (the positions before are warm-up of a chunk). A report
// at position q is stored as key_hi | (q - base) << off_shift | id, where
// key_hi carries the stream index in batched matching (0 otherwise). Units of
// activation tiles record the first match of sticky state slot i of their
// segment as atomicMin(act[act_row + i], q - base); units of the paired
// layered tile read those slots.
struct UnitDev {
  int32_t tile;
  uint32_t flags;  // bit0: inject start-of-data states at lo
  int64_t lo, hi, emit_lo;
  int64_t base;      // first byte of the unit's stream
  uint64_t key_hi;   // stream index, already shifted into the report key
  int64_t act_row;   // phase 1 and 2 tiles: first activation slot of the unit's segment
  int32_t act_rowid; // its row (pair, segment) in the compacted activation lists
  int32_t stream;    // segment (plain matching) or stream (batched matching) index
};

// A piece of a filtered tile's work: the candidates among positions [lo, hi) of
// a segment that ends at `end`. Reports are stored as in UnitDev.
struct PieceDev {
  int32_t tile;
  uint32_t flags;     // bit0: inject start-of-data states at lo
  uint32_t lo, hi, end;
  uint32_t base;      // first byte of the piece's stream
  uint64_t key_hi;
  int64_t act_row;    // as in UnitDev
  int32_t act_rowid;
  int32_t pad;
};

// A run: n candidates of one piece, from cand[first], with what the piece says
// (one read instead of two that depend on each other).
struct alignas(16) RunDev {
  uint32_t piece, first, n;
  uint32_t starts;    // 1: inject the piece's start-of-data states too
  int32_t tile;
  uint32_t lo, end, base;
  uint64_t key_hi;
  int64_t act_row;
  int32_t act_rowid;
  int32_t pad[3];
};

}  // namespace ngap
