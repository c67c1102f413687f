// Register-resident form of the fused primal-dual iteration: all iterations of one warp of a
// pyramid level in one launch, the level's state held in registers and shared memory of the
// whole GPU or, where it is small, of one thread-block cluster (one pair per launch).
//
// A level is cut into tiles of 30 x R pixels, one warp each; only tiles that hold a pixel that
// is on (or that such a pixel reads) exist.  Lane k of a warp is image column x0 - 1 + k: lanes
// 1..30 own their column, lanes 0 and 31 hold the west and east halo.  A warp keeps u, u-bar,
// v-bar, p and q of its rows in registers and shared memory, with the level's coefficients beside
// them.  One iteration streams down the rows: the dual step of row r needs u-bar and v-bar of row
// r + 1 (still the old values) and of the east lane; the threshold and primal steps of row r need T p
// and q of the west lane and of row r - 1.  The dual step of the west column and of the row above the
// tile is recomputed by the warp, so an
// iteration needs one exchange: u-bar and v-bar of the pixels around the tile.
//
// Exchange.  Every tile publishes the u-bar and v-bar of its border pixels as 16-byte words
// that carry a tag (launch epoch and iteration) beside the values, and reads the words of its
// eight neighbours until their tags are the ones it waits for.  A word is written and read by
// single 128-bit memory operations, so a reader that sees the tag has the values: no fence, no
// barrier, no grid-wide synchronisation; one store and one load through L2 are the whole
// latency.  Words live in a ring of two iterations: a tile that has the words of iteration k of
// all its neighbours knows that each of them has finished k - 1, and so has read this tile's
// words of k - 1, before it overwrites them with those of k + 1.
//
// The grid is launched cooperatively (or is one cluster), so that all its blocks are resident and
// every wait ends; a wait is bounded all the same.  A warp that gives up records it in its handle's word
// (StereoTgvImpl::checkWaits), stops waiting and runs on.
//
// The arithmetic is that of k_fused_iter (tgv_pixel.cuh, tgv_pixel_fast.cuh) with the same
// storage rounding, so the results are bit-identical to one launch per iteration, the values
// that the other ping-pong buffers hold included (the state before the last iteration is
// written there).
//
// What bounds it, on B200 (FP16 storage, 848 x 800, 2037 tiles of 8 rows, 3.7 us per iteration):
// about half of an iteration is instruction issue (1040 instructions per tile, 3.4 warps per
// scheduler, close to one per cycle), the rest the exchange: 1100 to 1500 cycles from a
// store to the load that sees it, and the wait for the slowest neighbour.  One launch per iteration
// (k_fused_iter) takes 8.0 us there alone, bound by its loads; float storage 6.3 against 10.3 us.
// Small levels are all latency, so theirs runs in one cluster whose blocks write into each other's
// shared memory (k_resident_cluster): 53 x 50 takes 0.90 us, through L2 1.39, one launch per
// iteration 3.2.
#pragma once
#include <atomic>
#include <vector>

#include "common.cuh"
#include "fused.cuh"

namespace vfs {

constexpr int kResCols = 30;       // owned columns per tile
constexpr int kResRing = 2;        // iterations of exchange words kept
constexpr int kResMaxIters = 128;  // iterations per launch (a tag's low seven bits)
// tile heights the kernel is built for (float storage: those up to 8)
constexpr int kResRows[] = {2, 4, 6, 8, 12, 16};
constexpr int kResNumRows = 6;
constexpr int kResMostWarps = 16;                   // of a block (one per SM), a tile each
constexpr int kResMostTiles = 148 * kResMostWarps;  // a bound on the tiles of a plan
// The cluster form (kernels_resident.cu, k_resident_cluster): 16 blocks, tiles of two rows, for levels of
// up to so many tiles.  Beyond, the 16 SMs have more to issue than the shorter exchange saves (us per
// iteration, cluster / whole GPU: half storage 50 tiles 0.90 / 1.39, 128 1.02 / 1.38, 200 1.19 / 1.44,
// 230 1.39 / 1.42; float 50 1.18 / 1.70, 128 1.46 / 1.7, 200 1.76 / 1.75, 230 2.06 / 1.75; tiles of four
// rows, 160 of them, 1.62 / 1.42 and 2.57 / 1.75).
constexpr int kResClusterRows = 2;
constexpr int kResClusterCtas = 16;
inline int res_cluster_tiles(bool half) { return half ? 208 : 128; }
// The drop-in path makes its plans at a mask's first solve where that runs at least so many iterations a
// level (all warps), else at its second: a plan takes the host longer than a short solve saves.  B200, ms from a new
// mask to the disparity on the host, 1 warp: 848 x 800 with plans 1.70 + 0.008 an iteration, a kernel per operation
// 1.27 + 0.09; 424 x 400 0.77 + 0.003, 0.70 + 0.065; 64 x 48 0.23, 0.29 + 0.03.
constexpr int kResPlanIters = 6;
inline int res_slots(int rows) { return 64 + 2 * rows; }  // words per tile: top, bottom, left, right

// What a tile's pixels ask of its iterations: none of the edge rules; the edge rules; or
// also the values that masked-out pixels keep (an on pixel reads one of them: it has neither its
// right nor its left, or neither its lower nor its upper, neighbour).
// kResPlain (found by the kernel): as kResKeep, with the plain division and square root.
enum ResKind { kResInner = 0, kResEdge = 1, kResKeep = 2, kResPlain = 3 };
constexpr unsigned kResBeyond = 0x80u;  // in a word's tag (epoch << 8 | iteration): from a kResPlain tile

struct ResTile {
  int x0, y0;   // first owned column and row
  int nb[8];    // tile index of the N, S, W, E, NW, NE, SW, SE neighbour (own index: none)
  int kind;     // ResKind
  int pad;
};

struct ResCtl {   // per level plan, in device memory
  unsigned epoch; // launches completed
  unsigned done;  // of the running launch: blocks that have ended, and kResGaveUp for each warp that gave up a wait
};
constexpr unsigned kResGaveUp = 1u << 16;

// One iteration's step sizes (evaluated on the host), each twice for the packed instructions.
struct ResStep {
  float2 sp, sq, tau, mu;
};

struct ResArgs {
  IterPair P;            // pointers of the first iteration (u, u-bar current; v-bar, p, q are zero)
  uint4* exch;           // [kResRing][ntiles][res_slots]
  ResCtl* ctl;
  const ResTile* tiles;
  int ntiles;
  const int2* fill;      // plain form: (x0, y0) of the tiles without a pixel to solve
  int nfill;
  int n;                 // iterations (1 .. kResMaxIters)
  int p_planes;          // p and q have two planes (result in plane n & 1); else one
  int rows, blocks;      // tile height, blocks of the grid
  bool cluster;          // the grid is one thread-block cluster
  int mute;              // tests: a tile that leaves out its first words (-1: none)
  unsigned* gave_up;     // host memory: 1 once a wait ran out
  float2 minus_zero;     // -0, where the compiler does not see it
  ResStep step[kResMaxIters];
};

// A level's tiles (host side).
struct ResTiles {
  int rows = 0, blocks = 0;
  bool cluster = false;  // the blocks are one thread-block cluster
  // Renumbers the tiles for a grid of `blocks` (tile t: warp t / blocks of block t % blocks) so that
  // those with edge rules sit on the schedulers (warp % 4) that have the fewest tiles.
  void place(int blocks);
  std::vector<ResTile> tiles;
  std::vector<int2> fill;
};
// What the tiles of any height need of a w x h level with edge codes `code` (rows of `pitch`; masked form:
// k_edge_codes of the mask, plain form: kOn inside the circle), found in one pass over it.
struct ResLevel {
  int w = 0, h = 0, tx = 0;
  bool masked = false;
  std::vector<uint8_t> need;          // per tile column and two rows: holds a pixel to solve
  std::vector<uint8_t> inner, keep;   // per row and tile column (ResKind)
  // False where the form does not apply: a masked-in pixel of column 0 (row 0) without its right
  // (lower) neighbour reads outside the image, a one-pixel-wide or -high plain level has no
  // neighbour to take, or no pixel is on.
  bool scan(const uint8_t* code, int pitch, int w, int h, bool masked);
  int count(int rows) const;  // tiles of `rows` rows
  void tiles(int rows, ResTiles& out) const;
};
// The plain form's codes (tight rows) on the host: kOn inside the circle.  A row's pixels inside are
// one run about the middle (the radius grows with the distance from it, and so does its rounded value).
std::vector<uint8_t> res_circle_codes(int w, int h);
// Picks the tile height for the level among the instances whose grid can be resident;
// false: no instance fits (or the form does not apply).
bool res_choose(const uint8_t* code, int pitch, int w, int h, bool masked, bool half, ResTiles& out);

// Device bytes a level's plan takes at most.
size_t res_bytes_bound(int w, int h);

// A level's plan on the device.
struct ResPlan {
  bool cluster = false;
  int rows = 0, blocks = 0, ntiles = 0, nfill = 0;  // ntiles = 0: the level has no plan
  const ResTile* tiles = nullptr;
  const int2* fill = nullptr;
  uint4* exch = nullptr;
  ResCtl* ctl = nullptr;
};

// most tiles an instance holds with its whole grid (cluster > 0: one cluster of that many blocks)
// resident; 0: not available
int res_capacity(bool masked, bool half, int rows, int cluster = 0);
// readies an instance for launches (once a plan has chosen it)
void res_use(bool masked, bool half, int rows, bool cluster);
// host bytes (a multiple of four) to the device, stream-ordered; they are taken before the call returns
void launch_res_upload(void* to, const void* from, size_t bytes, cudaStream_t st);
void launch_resident(const ResArgs& A, bool masked, bool half, cudaStream_t st);
// test hook: launches leave out the first words of their first tile
std::atomic<bool>& res_muted();
// reads and clears the device status (1: a bounded wait ran out)
int resident_status_take();

}  // namespace vfs
