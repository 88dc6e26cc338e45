// Pieces of scanned tiles, the slices that launches take, and the room of a plan.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "device_types.h"

namespace ngap {

// Positions of a piece: a step of a scan warp at least, and what run entries can pack.
constexpr int kPieceMax = 4096;
constexpr int kScanLane = 8;     // positions per lane and step: reads in flight
constexpr int kScanMinPiece = 32 * kScanLane;
constexpr int kStripMax = 16;    // consecutive positions per lane (a strip)

// Length of a filtered tile's pieces: one per scan warp for short inputs, and
// not below one step of a warp (256 positions); a caller's chunk length bounds it.
inline int64_t piece_len(int64_t positions, int64_t warps, int64_t chunk_opt) {
  int64_t n = (positions + warps - 1) / warps;
  const int64_t step = n > kScanMinPiece ? 32 * kStripMax : kScanMinPiece;
  n = (n + step - 1) / step * step;
  if (chunk_opt > 0) n = std::min(n, chunk_opt);
  return std::max<int64_t>(kScanMinPiece, std::min<int64_t>(n, kPieceMax));
}

// Pieces scanned by one launch and matched by the next (make_slices).
struct Slice {
  int32_t begin, count;
  int64_t runs;     // most runs they can give
  bool layered;
  int32_t one_tile; // the one tile of the pieces, or -1
  int64_t longest = 0;  // positions of the longest piece
};

// Slices of consecutive pieces whose worst case (every position a candidate)
// fits the candidate and run buffers: pieces[0] (plain and activation tiles)
// first, then pieces[1] (layered tiles, after the activations are known). The
// candidate buffer takes 64 MB at most and the run buffer 256 MB: 4 to 64 candidates
// a run, so that the latter bounds only slices of tables with long lists. (With a
// quarter of it, 24 MiB against 200 25-mers with three table levels takes 1.43 ms
// instead of 1.00 on a B200, and against 50 edit-distance rules with one level
// 1.15 instead of 0.57: a slice's last runs leave most of the chip idle.)
constexpr int64_t kSlicePositions = 32 << 20;
constexpr int64_t kSliceRuns = 4 << 20;
static_assert(kSlicePositions * sizeof(uint16_t) == (64 << 20) && kSliceRuns * sizeof(RunDev) == (256 << 20),
              "as stated above");
inline std::vector<Slice> make_slices(const std::vector<PieceDev> pieces[2],
                                      const std::vector<int32_t>& run_len, int64_t* cands, int64_t* runs) {
  std::vector<Slice> out;
  *cands = *runs = 0;
  int32_t index = 0;
  for (int l = 0; l < 2; l++) {
    int64_t pos = 0;
    for (size_t i = 0; i < pieces[l].size(); i++, index++) {
      const PieceDev& p = pieces[l][i];
      const int64_t n = p.hi - p.lo, r = (n + run_len[p.tile] - 1) / run_len[p.tile] + 1;
      if (i == 0 || pos + n > kSlicePositions || out.back().runs + r > kSliceRuns) {
        out.push_back({index, 0, 0, l == 1, p.tile});
        pos = 0;
      }
      if (p.tile != out.back().one_tile) out.back().one_tile = -1;
      out.back().count++;
      out.back().runs += r;
      pos += n;
      out.back().longest = std::max(out.back().longest, n);
      *cands = std::max(*cands, pos);
      *runs = std::max(*runs, out.back().runs);
    }
  }
  return out;
}

// Plans with less work than this are not scanned (engine.cu, scan_work: at least
// one per position and tile).
constexpr int64_t kScanMin = 1 << 17;

// What bounds a batch's plan: its streams, and the NFAs they may be matched against.
struct BatchShape {
  int64_t tiles = 0, scanned = 0, plain = 0;  // of the NFA with most: all, with a filter, without
  int64_t run_len = 64;                       // shortest runs of any tile
  int64_t positions = 0, streams = 0;
  int64_t chunk = 0;                          // shortest chunk of any stream
  int64_t warps = 0;                          // resident warps
};

// Records that a plan of such a batch has at most, whatever NFAs its streams
// name. A batch reserves as much, so that a server that has matched one batch of
// its largest size never allocates (which waits for the whole device) for
// another mix of NFAs or for one that is too small to be scanned.
struct PlanRoom {
  int64_t units = 0, pieces = 0, cands = 0, runs = 0;
};
inline PlanRoom plan_room(const BatchShape& b) {
  PlanRoom r;
  const int64_t chunk = std::max<int64_t>(1, b.chunk);
  // chunks of the tiles without a filter; of the others where the plan is not
  // scanned; automatic chunks may be one per warp in each of three launches
  r.units = b.plain * (b.positions / chunk + b.streams) + b.scanned * b.streams +
            kScanMin / std::min<int64_t>(chunk, 128) + 3 * b.warps;
  if (b.scanned == 0) return r;
  // pieces end at multiples of 8; automatic ones are one per warp or kPieceMax
  const int64_t piece = std::max<int64_t>(kScanMinPiece, std::min<int64_t>(chunk, kPieceMax)) - 7;
  r.pieces = b.scanned * (b.positions / piece + b.streams) + b.warps;
  r.cands = std::min(kSlicePositions, b.scanned * b.positions);
  r.runs = std::min(kSliceRuns, b.scanned * b.positions / b.run_len + 2 * r.pieces);
  return r;
}

}  // namespace ngap
