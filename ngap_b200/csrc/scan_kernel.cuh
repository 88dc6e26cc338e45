// Filtered tiles: a scan of the input with a tile's look-ahead filter
// (FilterDev), and a pass over the positions it leaves (candidates).
//
// A path that starts at a position of an acyclic tile depends on nothing but
// the input after it, so candidates are matched one by one, in any order and
// without windows, warm-up or states carried from one chunk to the next:
//  * scan_kernel: one warp per piece (a tile and up to kPieceMax positions of a
//    segment) writes the piece's candidates to a list and cuts them into runs;
//  * run_kernel: one warp per run injects the candidates through the prefix
//    tables (or the active sticky states of a layered tile) and follows their
//    paths in registers to their end, reading the input in place.
// The two have opposite needs, which is why they are two kernels: the scan is
// one filter block read per position (a gather, which takes the L1 tag stage once per
// lane: 32 warps with eight reads per lane in flight keep L1 84 % busy on the
// 25-mers, 78 us for 16.8 M positions, 215 G positions/s) with few instructions;
// runs are chains of dependent reads that want many warps and full lanes. In
// one kernel (16 warps, a window of 2048 positions at a time) each window left 80
// candidates and 20 surviving paths to one warp, which waited for all of them.
// Match times on a B200, one kernel and two: 1000 25-mers on 16 MiB 182 and 156
// us, 200 25-mers with three table levels 764 and 387, the 32 MiB mix 824 and
// 616, motifs 154 and 123, 300 dot-star regexes 133 and 111; 64 literals on
// 1 MiB 25 and 33 (two starts).
#pragma once

#include "match_kernel.cuh"
#include "slices.h"

namespace ngap {

constexpr int kMaxRunPath = 2048;  // states of the longest path of an acyclic tile (TableOpts::max_warmup)
// run entries pack offsets below kPieceMax (slices.h) + the longest path
static_assert(kPieceMax + kMaxRunPath + kMaxDepth < kMaxWindow, "offsets fit worklist entries");
constexpr int kScanWarps = 32;
// Per warp: class ids of 33 strips (4 bytes apart, so that lanes reading their
// strips word by word hit 32 banks), byte classes, one bit per position.
constexpr int kScanSymBytes = (33 * (kStripMax + 4) + 15) / 16 * 16;
constexpr int kScanPassBytes = (kPieceMax + 32 * kStripMax) / 8;
constexpr int kScanWarpBytes = kScanSymBytes + 256 + kScanPassBytes;
static_assert(kScanWarpBytes % 16 == 0, "per-warp regions stay 16-byte aligned");
// Control words of one scan and its runs (zeroed before the scan).
enum { kCtlPieces = 0, kCtlCands = 1, kCtlRuns = 2, kCtlTaken = 3, kCtlWords = 4 };

struct ScanParams {
  const TileDev* tiles;
  const PieceDev* pieces;
  uint32_t piece_begin, npieces;
  const uint8_t* input;     // 16-byte aligned
  uint32_t last;            // last byte of input that may be read (15 modulo 16)
  uint16_t* cand;           // candidates: offsets in their piece
  RunDev* runs;
  unsigned int* ctl;
  const uint32_t* act_cnt;  // activations of each row (layered tiles), or null
  int32_t one_tile;         // the one tile of the pieces (described below), or -1
  FilterDev filt;
  const uint8_t* cls;
  uint32_t nlive;
  int32_t run_len, phase;
  int32_t strip_bits;       // log2 of the positions per lane (3 or 4)
  unsigned long long* cycles;  // per piece (tracing), or null
};

// The next index of a warp past the `warps` that were handed out by number;
// n or more: none is left.
__device__ __forceinline__ unsigned next_index(unsigned int* counter, unsigned warps, unsigned n, int lane) {
  if (n <= warps) return n;
  unsigned k = 0;
  if (lane == 0) k = warps + atomicAdd(counter, 1u);
  return __shfl_sync(kFull, k, 0);
}

// The scan. A lane owns a strip of 8 or 16 consecutive positions, whose hash it
// rolls: two words of class ids per four positions and two multiply-adds per
// position. Longer strips have fewer instructions, but their symbols take L1 from
// the filters: match times on a B200 with strips of 8, 16, 32 and 64: 512
// streams 2.68, 2.60, 2.72, 3.00 ms; the 32 MiB mix 552, 519, 505, 505 us; 300
// dot-star regexes 116, 107, 110, 118 us. (Filters of up to 64 KB copied to
// shared memory gained the mix 1 % and nothing else: not kept.)
__global__ void __launch_bounds__(kScanWarps * 32, 1) scan_kernel(ScanParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* sym = smem_raw + warp * kScanWarpBytes;
  uint8_t* cls = sym + kScanSymBytes;
  uint8_t* pass = cls + 256;
  int staged = -1;  // the tile whose classes are in cls
  // eight input bytes as class ids
  auto load = [&](uint32_t at) {
    return at <= p.last ? __ldg(reinterpret_cast<const uint2*>(p.input + at)) : make_uint2(0u, 0u);
  };
  auto classes = [&](uint32_t b) {
    return cls[b & 0xff] | cls[(b >> 8) & 0xff] << 8 | cls[(b >> 16) & 0xff] << 16 |
           (uint32_t)cls[b >> 24] << 24;
  };
  const int sb = p.strip_bits, strip = 1 << sb;
  const uint32_t block_len = 32u << sb;  // positions per pass over the strips
  // class id i of the lane's strip and the ones after it, or the word that holds ids i .. i + 3
  const uint8_t* mine = sym + lane * (strip + 4);
  auto at = [&](int i) { return mine + i + ((i >> sb) << 2); };
  auto word_at = [&](int i) { return *reinterpret_cast<const uint32_t*>(at(i)); };
  // the first piece of a warp is its own number (spread over the CTAs), the
  // later ones come from a counter: short inputs start without an atomic
  unsigned k = warp * gridDim.x + blockIdx.x;
  const unsigned warps = gridDim.x * kScanWarps;
  for (; k < p.npieces; k = next_index(p.ctl + kCtlPieces, warps, p.npieces, lane)) {
    const long long t0 = clock64();
    const uint32_t index = p.piece_begin + k;
    const PieceDev pc = p.pieces[index];
    const TileDev* t = p.tiles + pc.tile;
    const bool starts = (pc.flags & 1u) != 0u;
    const bool one = p.one_tile >= 0;
    if ((one ? p.phase : t->phase) == 2 && !starts && p.act_cnt[pc.act_rowid] == 0u) {  // nothing is active
      if (p.cycles && lane == 0) p.cycles[index] = (unsigned long long)(clock64() - t0);
      continue;
    }
    const FilterDev f = one ? p.filt : t->filt;
    const uint32_t nlive = one ? p.nlive : (uint32_t)t->nlive;
    if (pc.tile != staged) {
      staged = pc.tile;
      __syncwarp();
      reinterpret_cast<uint2*>(cls)[lane] =
          __ldg(reinterpret_cast<const uint2*>(one ? p.cls : t->image + t->off_cls) + lane);
      __syncwarp();
    }
    const uint32_t a0 = pc.lo & ~7u;
    const int nblocks = (int)((pc.hi - a0 + block_len - 1) >> (5 + sb));
    for (int b = 0; b < nblocks; b++) {
      const uint32_t o = a0 + (uint32_t)b * block_len;
      __syncwarp();
      for (uint32_t c = lane; c < (block_len + 16) / 8; c += 32) {
        const uint2 in = load(o + 8 * c);
        uint32_t* dst = reinterpret_cast<uint32_t*>(sym + 8 * c + (((8 * c) >> sb) << 2));
        dst[0] = classes(in.x);
        dst[1] = classes(in.y);
      }
      __syncwarp();
      const uint32_t own = o + ((uint32_t)lane << sb);  // the lane's first position
      // whole passes inside the piece with all of the filter's symbols left need no bounds per position
      // (the sum in 64 bits: inputs reach to 4 GiB)
      const bool inside = o >= pc.lo && (uint64_t)o + block_len <= pc.hi &&
                          pc.end - (o + block_len - 1) >= (uint32_t)f.len;
      uint32_t h = 0u, left = 0u;  // left: the id that leaves before the next position
      for (int i = 0; i < f.len - 1; i++) h = h * kFilterMul + *at(i);
      const int w0 = (f.len - 1) & ~3, sh = ((f.len - 1) & 3) * 8;
      uint32_t next = word_at(w0);
      for (int i = 0; i < strip; i += kScanLane) {
        uint32_t hash[kScanLane];
        unsigned test = 0xffu, found = 0u;
#pragma unroll
        for (int g = 0; g < kScanLane / 4; g++) {
          const uint32_t out = word_at(i + 4 * g);
          const uint32_t w = next;
          next = word_at(w0 + i + 4 * g + 4);
          const uint32_t in = __funnelshift_r(w, next, sh);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            h = h * kFilterMul + (__byte_perm(in, 0, 0x4440 | j) - left * f.drop);
            left = __byte_perm(out, 0, 0x4440 | j);
            hash[4 * g + j] = h;
          }
          // positions whose own byte no state accepts need no read
          const uint32_t dead = nlive > 255u ? 0u : __vcmpgeu4(out, nlive * 0x01010101u) & 0x01010101u;
          test &= ~(((dead * 0x01020408u) >> 24 & 0xfu) << (4 * g));
        }
        if (!inside) {
#pragma unroll
          for (int j = 0; j < kScanLane; j++) {
            const uint32_t q = own + (uint32_t)(i + j);
            const bool in_piece = q >= pc.lo && q < pc.hi;
            const bool whole = in_piece && pc.end - q >= (uint32_t)f.len;
            if (in_piece && !whole && ((test >> j) & 1u) && pc.end - q >= (uint32_t)f.min_rep) found |= 1u << j;
            if (!whole) test &= ~(1u << j);
          }
        }
        uint2 block[kScanLane];
#pragma unroll
        for (int j = 0; j < kScanLane; j++) {
          const uint2* at = reinterpret_cast<const uint2*>(f.blocks) + ((hash[j] * kFilterBlock) >> f.shift);
          block[j] = (test >> j) & 1u ? __ldg(at) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int j = 0; j < kScanLane; j++) {  // filter_mask's three bits, rotated to bit 0
          const uint32_t x = (hash[j] * kFilterBits) >> 17;
          found |= (__funnelshift_r(block[j].x, block[j].x, x) & __funnelshift_r(block[j].x, block[j].x, x >> 5) &
                    __funnelshift_r(block[j].y, block[j].y, x >> 10) & 1u)
                   << j;
        }
        pass[(((uint32_t)b * block_len + ((uint32_t)lane << sb)) + (uint32_t)i) >> 3] = (uint8_t)found;
      }
    }
    __syncwarp();
    // the piece's candidates, in order, to the list; their runs
    const int nwords = nblocks << sb;
    const uint32_t* words = reinterpret_cast<const uint32_t*>(pass);
    uint32_t mine = 0;
    for (int i = lane; i < nwords; i += 32) mine += __popc(words[i]);
    const uint32_t total = __reduce_add_sync(kFull, mine);
    const uint32_t run_len = (uint32_t)(one ? p.run_len : t->run_len);
    const uint32_t nruns = max((total + run_len - 1) / run_len, starts ? 1u : 0u);
    if (nruns > 0) {
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(p.ctl + kCtlCands, total);
      if (lane == 1) at = atomicAdd(p.ctl + kCtlRuns, nruns);
      const uint32_t cbase = __shfl_sync(kFull, at, 0), rbase = __shfl_sync(kFull, at, 1);
      for (uint32_t i = lane; i < nruns; i += 32) {
        RunDev r;
        r.piece = index;
        r.first = cbase + i * run_len;
        r.n = min(run_len, total - i * run_len);
        r.starts = starts && i == 0 ? 1u : 0u;
        r.tile = pc.tile;
        r.lo = pc.lo;
        r.end = pc.end;
        r.base = pc.base;
        r.key_hi = pc.key_hi;
        r.act_row = pc.act_row;
        r.act_rowid = pc.act_rowid;
        p.runs[rbase + i] = r;
      }
      uint32_t done = cbase;
      const int shift = (int)(pc.lo - a0);
      for (int i0 = 0; i0 < nwords; i0 += 32) {
        uint32_t m = i0 + lane < nwords ? words[i0 + lane] : 0u;
        uint32_t incl = __popc(m);
        const uint32_t own = incl;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
          const uint32_t y = __shfl_up_sync(kFull, incl, s);
          if (lane >= s) incl += y;
        }
        uint32_t pos = done + incl - own;
        for (; m; m &= m - 1u) p.cand[pos++] = (uint16_t)((i0 + lane) * 32 + __ffs(m) - 1 - shift);
        done += __shfl_sync(kFull, incl, 31);
      }
    }
    if (p.cycles && lane == 0) atomicAdd(p.cycles + index, (unsigned long long)(clock64() - t0));
    __syncwarp();
  }
}

// What a run's steps share.
struct RunCtx {
  const uint8_t* in;   // input at the piece's first position
  const uint8_t* cls;  // byte -> class
  uint32_t lo;         // the piece's first position
  int lim;             // symbols from there to the segment's end
};

__device__ __forceinline__ uint32_t symbol(const RunCtx& c, int r) { return __ldg(c.cls + __ldg(c.in + r)); }

// What a run puts on its worklist before it follows the paths. Positions that
// pass a filter are the ones with long lists, and 32 of them are injected at once,
// so that a batch's lists can be many times what the worklist holds (32 URLs
// against 4000 rules on "http://www.": 128,000 entries). An injection therefore
// stops near mark_inject entries, a quarter of the worklist; the paths are
// followed, and it goes on from `resume` (0: all is done). Lists of up to that many
// entries, nearly all, are injected in one go as before.
static_assert((512 + 1024) / 4 >= kInjectLow + 4 * 32, "short lists always fit");

// Entries from the overflow stack to the empty shared one.
__device__ __forceinline__ void refill_stack(WarpSmem& ws, WarpRun& w, int lane) {
  const int m = min(w.ovf_n, kStackCap);
  for (int i = lane; i < m; i += 32) ws.stack[i] = w.ovf[w.ovf_n - m + i];
  w.ovf_n -= m;
  w.top = m;
  __syncwarp();
}

// Injects the states a tile has always active at the piece's offset r of each
// lane (valid lanes): as inject_aas, without a window to clamp to. resume: index
// into the always-active list (depth 0) or into the lanes' lists one after another.
__device__ __forceinline__ void inject_run(const MatchParams& p, WarpSmem& ws, WarpRun& w,
                                           const TileView& tv, const RunCtx& c, int lane, bool valid,
                                           int r, int depth, uint32_t& resume,
                                           unsigned long long& n_injected) {
  const TileDev& t = *tv.t;
  const uint32_t q = c.lo + (uint32_t)r;
  const uint32_t from = resume;
  resume = 0;
  if (depth == 0) {  // scan the always-active list
    const uint32_t s = valid ? symbol(c, r) : 0u;
    for (int i0 = (int)from; i0 < t.naas; i0 += kAasStep) {
      if (held(w) > p.mark_inject - 32 * kAasStep) {
        resume = (uint32_t)i0;
        return;
      }
      uint32_t a[kAasStep];
      const uint32_t ok = aas_step(tv, i0, s, valid, a);
      if (!__any_sync(kFull, ok != 0u)) continue;
#pragma unroll
      for (int j = 0; j < kAasStep; j++) {
        const bool hit = (ok >> j) & 1u;
        const bool rep = hit && is_report(tv, a[j]);
        emit_report(p, ws, w, lane, rep, rep ? __ldg(t.sid + a[j]) : 0u, q);
        push_entry(p, ws, w, lane, hit && r + 1 < c.lim, (a[j] << kEntryPosBits) | (uint32_t)r);
      }
      n_injected += __popc(ok);
    }
    return;
  }
  const int kmax = valid ? min(depth, c.lim - r) : 0;
  // the next symbols: two 16-byte reads of the granules they lie in (a byte read
  // per symbol would take the L1 tag stage kMaxDepth times per lane); the
  // second only where the first ends too soon and input is left
  const uint32_t at = q & 15u;
  const uint4* granule = reinterpret_cast<const uint4*>(c.in + r - at);
  uint4 b0 = make_uint4(0u, 0u, 0u, 0u), b1 = b0;
  if (kmax > 0) b0 = __ldg(granule);
  if (kmax > 16 - (int)at) b1 = __ldg(granule + 1);
  uint32_t byte[kMaxDepth];
  {
    const uint64_t w0 = b0.x | (uint64_t)b0.y << 32, w1 = b0.z | (uint64_t)b0.w << 32;
    const uint64_t w2 = b1.x | (uint64_t)b1.y << 32, w3 = b1.z | (uint64_t)b1.w << 32;
    const bool high = at >= 8;
    const uint64_t lo = high ? w1 : w0, mid = high ? w2 : w1, hi = high ? w3 : w2;
    const uint32_t sh = (at & 7u) * 8u;
    const uint64_t s0 = sh ? lo >> sh | mid << (64 - sh) : lo;
    const uint64_t s1 = sh ? mid >> sh | hi << (64 - sh) : mid;
#pragma unroll
    for (int d = 0; d < kMaxDepth; d++)
      byte[d] = (uint32_t)((d < 8 ? s0 >> (8 * d) : s1 >> (8 * (d - 8))) & 0xffu);
  }
  int k = kmax;
  uint32_t key = 0;  // live classes of the next k symbols, base nlive
#pragma unroll
  for (int d = 0; d < kMaxDepth; d++) {
    byte[d] = __ldg(c.cls + byte[d]);
    if (d < k) {
      if (byte[d] >= tv.nlive) k = d;
      else key = key * tv.nlive + byte[d];
    }
  }
  const bool use = k == kmax && k > 0;  // a dead class ends every path
  uint32_t vb = 0, ve = 0, one = kNoEntry;
  const PrefixTableDev& deep = tv.pt[(k > 0 ? k : 1) - 1];
  if (use) {
    uint32_t rb, re;
    pt_find(deep, key, true, false, vb, ve, rb, re, one);
  }
  if (tv.rep_levels && from == 0) {  // reports of the first k symbols, level by level
    uint32_t kk = 0;
#pragma unroll
    for (int d = 0; d < kMaxDepth; d++) {
      if (d >= depth) break;
      const bool act = d < k;
      if (act) kk = kk * tv.nlive + byte[d];
      if (!((tv.rep_levels >> d) & 1u)) continue;
      const PrefixTableDev& pt = tv.pt[d];
      uint32_t b0, e0, rb, re, o1;
      pt_find(pt, kk, false, act, b0, e0, rb, re, o1);
      const int len = (int)(re - rb);
      const int mx = __reduce_max_sync(kFull, len);
      for (int i = 0; i < mx; i++) {
        const bool ok = i < len;
        const uint32_t v = ok ? __ldg(pt.rlist + rb + i) : 0u;
        emit_report(p, ws, w, lane, ok, ok ? __ldg(t.sid + v) : 0u, q + d);
      }
    }
  }
  // entries at the segment's last position have nothing to expand
  const uint32_t len = use && r + k < c.lim ? (ve - vb) + (one != kNoEntry ? 1u : 0u) : 0u;
  if (from == 0) n_injected += len;
  uint32_t incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  uint32_t total = __shfl_sync(kFull, incl, 31);
  if (total == 0) return;
  const uint32_t off = (uint32_t)(r + k - 1);
  if (__reduce_max_sync(kFull, len) <= 4u) {  // short lists: every lane copies its own
    uint32_t v[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; j++)
      v[j] = j < len ? (one != kNoEntry ? one : __ldg(deep.vlist + vb + j)) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < 4; j++)
      if (j < len) store_entry(p, ws, w, w.top + (int)(incl - len + j), (v[j] << kEntryPosBits) | off);
  } else {  // all lanes' lists copied cooperatively
    ws.inj[lane] = incl;
    ws.inj[32 + lane] = one != kNoEntry ? one : vb;  // a lone state itself, or where the list starts
    ws.inj[64 + lane] = off | (uint32_t)(k > 0 ? k : 1) << 16 | (one != kNoEntry ? 0x1000000u : 0u);
    __syncwarp();
    const uint32_t all = total;
    total = min(all, from + (uint32_t)(p.mark_inject - held(w)));  // what there is room for
    if (total < all) resume = total;
    for (uint32_t i = from + lane; i < total; i += 32) {
      int l0 = 0, l1 = 31;
      while (l0 < l1) {  // first lane whose inclusive prefix exceeds i
        const int m = (l0 + l1) >> 1;
        if (ws.inj[m] > i) l1 = m;
        else l0 = m + 1;
      }
      const uint32_t before = l0 > 0 ? ws.inj[l0 - 1] : 0u;
      const uint32_t x = ws.inj[64 + l0];
      const uint32_t v = x >> 24 ? ws.inj[32 + l0]
                                 : __ldg(tv.pt[((x >> 16) & 0xffu) - 1].vlist + ws.inj[32 + l0] + (i - before));
      store_entry(p, ws, w, w.top + (int)(i - from), (v << kEntryPosBits) | (x & 0xffffu));
    }
    total -= from;
  }
  grow_stack(p, w, (int)total);
  __syncwarp();
}

// Start-of-data states at the piece's first position (ngap_buffer.cu:613-631),
// except sticky ones of layered tiles (registered from the activation pass).
// resume: index into the start-of-data list.
__device__ __forceinline__ void inject_starts(const MatchParams& p, WarpSmem& ws, WarpRun& w,
                                              const TileView& tv, const RunCtx& c, int lane,
                                              uint32_t& resume) {
  const TileDev& t = *tv.t;
  const uint32_t s0 = symbol(c, 0);
  int i0 = (int)resume;
  resume = 0;
  for (; i0 < t.nstart; i0 += 32) {
    if (held(w) > p.mark_inject - 32) {
      resume = (uint32_t)i0;
      return;
    }
    const int i = i0 + lane;
    const uint32_t v = i < t.nstart ? __ldg(t.start + i) : 0u;
    const bool ok = i < t.nstart && accepts(tv, v, s0);
    const bool rep = ok && is_report(tv, v);
    emit_report(p, ws, w, lane, rep, rep ? __ldg(t.sid + v) : 0u, c.lo);
    push_entry(p, ws, w, lane, ok && c.lim > 1 && !(tv.sticky && is_sticky(tv, v)), v << kEntryPosBits);
  }
}

// Layered tiles: the work of the segment's active sticky states (n matched
// slots listed at act_list + row) at the offsets rc of lanes 0 .. m - 1. The
// filter leaves few positions, so lanes hold sticky states (32 at a time, their
// slot, first match and union mask in registers) and the candidates are
// visited one by one: a pass over n states costs n / 32 steps per candidate. Same
// rule as layered_sticky_positions; reporting sticky states get no filter. resume:
// the first of 32 sticky states + the candidate.
// Measured on a B200, whole calls, layered tiles without and with a filter: the
// 32 MiB mix 2.41 -> 1.16 ms (20.8 M expansions -> 1.3 M), 512 streams against
// eight rule sets 32.5 -> 10.8 ms, 300 dot-star regexes on 4 MB 0.80 -> 0.38.
__device__ __forceinline__ void layered_run(const MatchParams& p, WarpSmem& ws, WarpRun& w,
                                            const TileView& tv, const RunCtx& c, int lane, int rc,
                                            int m, int64_t row, uint32_t n, uint32_t& resume) {
  const TileDev& t = *tv.t;
  const uint32_t cls = lane < m ? symbol(c, rc) : 0u;
  uint32_t i0 = resume & ~31u;
  int k = (int)(resume & 31u);
  resume = 0;
  uint32_t next = i0 + (uint32_t)lane < n ? __ldg(p.act_list + row + i0 + lane) : 0u;
  for (; i0 < n; i0 += 32, k = 0) {
    const uint32_t i = i0 + (uint32_t)lane;
    const uint32_t sl = next;
    if (i + 32 < n) next = __ldg(p.act_list + row + i + 32);
    const uint32_t f = i < n ? __ldg(p.act + row + sl) : kNoAct;
    const uint32_t al = i < n ? __ldg(t.act_local + sl) : 0u;
    const uint32_t* um = t.stk_union + (size_t)sl * tv.cw;
    const uint32_t u0 = i < n ? __ldg(um) : 0u;
    const uint32_t u1 = i < n && tv.cw > 1 ? __ldg(um + 1) : 0u;
    const uint32_t u2 = i < n && tv.cw > 2 ? __ldg(um + 2) : 0u;
    for (; k < m; k++) {
      const int r = __shfl_sync(kFull, rc, k);
      const uint32_t sym = __shfl_sync(kFull, cls, k);
      const uint32_t rel = c.lo + (uint32_t)r - w.base;  // position in the segment
      const uint32_t word = sym >> 5;
      const uint32_t mask = word == 0 ? u0 : word == 1 ? u1 : word == 2 ? u2 : i < n ? __ldg(um + word) : 0u;
      const bool hit = i < n && rel >= f && ((mask >> (sym & 31)) & 1u);
      if (!__any_sync(kFull, hit)) continue;
      const uint32_t on = !hit ? 0u : rel > f ? 0xfu : al >> 28;
      uint4 su = make_uint4(kNoSucc, kNoSucc, kNoSucc, kNoSucc);
      if (hit) su = load_succ(tv, al & kActIdMask);
      const uint32_t us[4] = {su.x, su.y, su.z, su.w};
      bool ok[4];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        ok[j] = ((on >> j) & 1u) && us[j] != kNoSucc && accepts(tv, us[j] & kIdMask, sym);
        cnt += ok[j];
      }
      report4(p, ws, w, tv, lane, ok, us, (int64_t)c.lo + r, true);
      if (r + 1 >= c.lim) continue;  // the segment's last position: nothing to expand
      int total;
      int pos = w.top + warp_excl<3>(cnt, lane, total);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (ok[j]) store_entry(p, ws, w, pos++, ((us[j] & kIdMask) << kEntryPosBits) | (uint32_t)r);
      grow_stack(p, w, total);
      __syncwarp();
      if (held(w) > p.mark_inject - 4 * 32) {
        resume = k + 1 < m ? i0 + (uint32_t)k + 1u : i0 + 32 < n ? i0 + 32 : 0u;
        if (resume) return;
      }
    }
  }
}

// One step of a run's worklist past mark_walk, or with --unique: expand_step without windows.
template <bool UNIQUE>
__device__ __forceinline__ void step_run(const MatchParams& p, WarpSmem& ws, WarpRun& w,
                                         const TileView& tv, const RunCtx& c, int lane,
                                         unsigned long long& n_expanded) {
  if (w.top == 0) refill_stack(ws, w, lane);
  const int n = min(w.top, held(w) > p.mark_single ? 1 : 32);
  const uint32_t e = lane < n ? ws.stack[w.top - 1 - lane] : kNoEntry;
  w.top -= n;
  __syncwarp();
  bool go = lane < n;
  if (UNIQUE) {  // identical entries once (every lane votes; those without an entry hold kNoEntry)
    const unsigned same = __match_any_sync(kFull, e);
    go = go && __ffs(same) - 1 == lane;
  }
  const uint32_t v = e >> kEntryPosBits;
  const int r = (int)(e & ((1u << kEntryPosBits) - 1));
  go = go && r + 1 < c.lim;
  uint4 sc = make_uint4(kNoSucc, kNoSucc, kNoSucc, kNoSucc);
  uint4 sm = make_uint4(0u, 0u, 0u, 0u);
  uint32_t s = 0u;
  if (go) {
    load_record(tv, v, sc, sm);
    s = symbol(c, r + 1);
  }
  n_expanded += go;
  const uint32_t u[4] = {sc.x, sc.y, sc.z, sc.w};
  const uint32_t um[4] = {sm.x, sm.y, sm.z, sm.w};
  bool ok[4];
  int cnt = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    ok[j] = go && succ_accepts(tv, u[j], um[j], s);
    cnt += ok[j];
  }
  report4(p, ws, w, tv, lane, ok, u, (int64_t)c.lo + r + 1, true);
  const int more = go && r + 2 < c.lim ? cnt : 0;  // the successors have a next symbol
  int total;
  int pos = w.top + warp_excl<3>(more, lane, total);
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (more && ok[j]) store_entry(p, ws, w, pos++, ((u[j] & kIdMask) << kEntryPosBits) | (uint32_t)(r + 1));
  grow_stack(p, w, total);
  __syncwarp();
}

// Follows every path on the stack to its end: walk_paths without windows (no
// state is carried over).
__device__ __forceinline__ void walk_run(const MatchParams& p, WarpSmem& ws, WarpRun& w,
                                         const TileView& tv, const RunCtx& c, int lane,
                                         unsigned long long& n_expanded) {
  uint32_t v = 0;
  int r = 0;
  bool act = false;
  unsigned live = 0u;
  while (true) {
    if (w.top == 0 && w.ovf_n > 0 && __popc(live) <= 16) refill_stack(ws, w, lane);
    if (w.top > 0 && __popc(live) <= 16) {  // idle lanes take the entries on top of the stack
      const int n = min(w.top, 32 - __popc(live));
      const int k = __popc(~live & lanemask_lt(lane));
      if (!act && k < n) {
        const uint32_t e = ws.stack[w.top - 1 - k];
        v = e >> kEntryPosBits;
        r = (int)(e & ((1u << kEntryPosBits) - 1));
        act = r + 1 < c.lim;
      }
      w.top -= n;
      __syncwarp();
    }
    uint4 sc = make_uint4(kNoSucc, kNoSucc, kNoSucc, kNoSucc);
    uint4 sm = make_uint4(0u, 0u, 0u, 0u);
    uint32_t s = 0u;
    if (act) {
      load_record(tv, v, sc, sm);
      s = symbol(c, r + 1);
    }
    n_expanded += act;
    const uint32_t u[4] = {sc.x, sc.y, sc.z, sc.w};
    const uint32_t um[4] = {sm.x, sm.y, sm.z, sm.w};
    bool ok[4], rep = false;
    int cnt = 0;
    uint32_t follow = 0u;
#pragma unroll
    for (int j = 3; j >= 0; j--) {
      ok[j] = act && succ_accepts(tv, u[j], um[j], s);
      rep |= ok[j] && (u[j] >> 31);
      cnt += ok[j];
      if (ok[j]) follow = u[j] & kIdMask;
    }
    const bool need = act && r + 2 < c.lim && cnt > 0;  // the successors have a next symbol
    const unsigned events = __reduce_or_sync(kFull, (rep ? 1u : 0u) | (need && cnt > 1 ? 2u : 0u));
    if (events & 1u) report4(p, ws, w, tv, lane, ok, u, (int64_t)c.lo + r + 1, true);
    if (events & 2u) {  // successors beyond the first
      const int more = need ? cnt - 1 : 0;
      int total;
      int pos = w.top + warp_excl<2>(more, lane, total);
      bool first = true;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (more && ok[j] && !first)
          store_entry(p, ws, w, pos++, ((u[j] & kIdMask) << kEntryPosBits) | (uint32_t)(r + 1));
        first = first && !ok[j];
      }
      grow_stack(p, w, total);
      __syncwarp();
    }
    act = need;
    v = follow;
    r++;
    live = __ballot_sync(kFull, act);
    // the worklist has grown past mark_walk (injections end far below it): all
    // paths back to it, and steps until it is half as full
    if ((events & 2u) && held(w) > p.mark_walk) {
      push_entry(p, ws, w, lane, act, (v << kEntryPosBits) | (uint32_t)r);
      act = false;
      live = 0u;
      while (held(w) > p.mark_inject) step_run<false>(p, ws, w, tv, c, lane, n_expanded);
    }
    if (live == 0u && w.top == 0 && w.ovf_n == 0) return;
  }
}

// Warps of a CTA: 32 of 64 registers (the plain instance spills 120 bytes) rather than 16 of 122,
// because runs wait for reads most of the time. Match times on a B200 with 16,
// 20, 24 and 32: 1000 25-mers 194, 181, 174, 160 us; 200 25-mers with three table
// levels 625, 546, 468, 394; the 32 MiB mix 639, 619, 607, 599.
constexpr int kRunWarps = 32;
// Per warp: worklist, report buffer, injection scratch. (Copies of the tile's
// descriptor and classes in shared memory cost more, in L1, than they gain.)
constexpr int kRunWarpBytes = kStackCap * 4 + kReportBuf * 8 + 3 * 32 * 4;
static_assert(kRunWarpBytes % 16 == 0, "per-warp regions stay 16-byte aligned");
__host__ __device__ inline int run_smem_bytes() { return kRunWarps * kRunWarpBytes; }

// One warp per run. LAYERED: the runs' tiles are layered tiles. UNIQUE: step by
// step, dropping duplicate entries of a step (--unique): paths that meet in a state
// at the same symbol are then followed once, as match_kernel does.
template <bool LAYERED, bool UNIQUE>
__global__ void __launch_bounds__(kRunWarps * 32, 1) run_kernel(MatchParams p, const uint16_t* cand,
                                                               const RunDev* runs, unsigned int* ctl) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* mem = smem_raw + warp * kRunWarpBytes;
  WarpSmem ws = {};
  ws.stack = reinterpret_cast<uint32_t*>(mem);
  ws.rbuf = reinterpret_cast<unsigned long long*>(mem + kStackCap * 4);
  ws.inj = reinterpret_cast<uint32_t*>(mem + kStackCap * 4 + kReportBuf * 8);
  const int slot = blockIdx.x * kRunWarps + warp;
  WarpRun w = {};
  w.ovf = p.ovf + (size_t)slot * p.ovf_cap;
  unsigned long long n_expanded = 0, n_injected = 0;
  const unsigned nruns = ctl[kCtlRuns];
  const unsigned warps = gridDim.x * kRunWarps;
  // lane 0: the next run, taken while the current one is matched
  unsigned taken = warp * gridDim.x + blockIdx.x;
  while (true) {
    const unsigned i = __shfl_sync(kFull, taken, 0);
    if (i >= nruns) break;
    const long long t0 = clock64();
    const unsigned long long work0 = n_expanded + n_injected;
    const RunDev run = runs[i];
    if (lane == 0) taken = nruns > warps ? warps + atomicAdd(ctl + kCtlTaken, 1u) : nruns;
    const TileDev* t = p.tiles + run.tile;
    const uint8_t* cls = t->image + t->off_cls;
    RunCtx c;
    c.in = p.input + run.lo;
    c.cls = cls;
    c.lo = run.lo;
    c.lim = (int)min(run.end - run.lo, 1u << 30);
    w.key_hi = run.key_hi;
    w.base = run.base;
    w.act = !LAYERED && t->phase == 1 ? p.act + run.act_row : nullptr;
    TileRun tr;
    tile_run<!LAYERED>(p, t, t->pt, cls, tr);
    const int batch = LAYERED ? 32 : min(tr.batch, 32);
    const uint32_t active = LAYERED ? p.act_cnt[run.act_rowid] : 0u;
    auto follow = [&]() {  // every path on the worklist to its end
      if (UNIQUE)
        while (held(w) > 0) step_run<true>(p, ws, w, tr.tv, c, lane, n_expanded);
      else
        walk_run(p, ws, w, tr.tv, c, lane, n_expanded);
    };
    bool starts = run.starts != 0u;
    uint32_t c0 = 0, resume = 0;
    while (starts || c0 < run.n) {
      if (starts) {
        inject_starts(p, ws, w, tr.tv, c, lane, resume);
        starts = resume != 0u;
      } else {
        const int m = (int)min((uint32_t)batch, run.n - c0);
        const int r = lane < m ? (int)__ldg(cand + run.first + c0 + lane) : 0;
        if (LAYERED)
          layered_run(p, ws, w, tr.tv, c, lane, r, m, run.act_row, active, resume);
        else
          inject_run(p, ws, w, tr.tv, c, lane, lane < m, r, tr.depth, resume, n_injected);
        if (resume == 0u) c0 += batch;
      }
      if (held(w) >= kInjectLow) follow();
    }
    if (held(w) > 0) follow();
    if (p.unit_work) {  // work of the run's piece (all lanes)
      unsigned long long d = n_expanded + n_injected - work0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(kFull, d, o);
      if (lane == 0) {
        atomicAdd(p.unit_work + p.piece_unit0 + run.piece, d);
        atomicAdd(p.unit_cycles + p.piece_unit0 + run.piece, (unsigned long long)(clock64() - t0));
      }
    }
  }
  flush_reports(p, ws, w, lane);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    n_expanded += __shfl_xor_sync(kFull, n_expanded, o);
    n_injected += __shfl_xor_sync(kFull, n_injected, o);
  }
  __shared__ unsigned long long s_work[2];
  if (threadIdx.x < 2) s_work[threadIdx.x] = 0ull;
  __syncthreads();
  if (lane == 0) {
    atomicAdd(&s_work[0], n_expanded);
    atomicAdd(&s_work[1], n_injected);
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_work[threadIdx.x]) atomicAdd(&p.work[threadIdx.x], s_work[threadIdx.x]);
}

}  // namespace ngap
