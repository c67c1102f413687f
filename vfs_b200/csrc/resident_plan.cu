// Host side of the register-resident iteration: the tiles of a level (resident.cuh).
#include <algorithm>
#include <cstring>

#include "resident.cuh"
#include "tgv_pixel.cuh"

namespace vfs {

std::vector<uint8_t> res_circle_codes(int w, int h) {
  std::vector<uint8_t> code((size_t)w * h, 0);
  const int mid = w / 2;  // no column is nearer to the centre
  for (int y = 0; y < h; y++) {
    if (mid >= w || outside_circle(mid, y, w, h)) continue;
    int out = -1, in = mid;  // the run's first column: out is outside (or left of the image), in inside
    while (in - out > 1) {
      const int x = out + (in - out) / 2;
      if (outside_circle(x, y, w, h)) out = x;
      else in = x;
    }
    const int first = in;
    in = mid, out = w;
    while (out - in > 1) {
      const int x = in + (out - in) / 2;
      if (outside_circle(x, y, w, h)) out = x;
      else in = x;
    }
    std::memset(&code[(size_t)y * w + first], kOn, (size_t)(in - first + 1));
  }
  return code;
}

// A level is mostly tiles' rows that are on or off throughout; those take three or four 8-byte looks
// (a 1280 x 1024 disc: 2.25 ms a pixel at a time, 0.40 this way; a new mask pays it).
bool ResLevel::scan(const uint8_t* code, int pitch, int w_, int h_, bool masked_) {
  w = w_;
  h = h_;
  masked = masked_;
  tx = (w + kResCols - 1) / kResCols;
  const int ty = (h + kResRows[0] - 1) / kResRows[0];
  need.assign((size_t)tx * ty, 0);
  inner.assign((size_t)tx * h, 0);
  keep.assign((size_t)tx * h, 0);
  if (w < 2 || h < 2) return false;
  const uint8_t kAll = kOn | kR | kL | kD | kU;
  constexpr uint64_t kEach = 0x0101010101010101ull;
  // the 30 codes from p on, by bits: those that all have (AND) and those that some have (OR)
  auto bits = [](const uint8_t* p, uint64_t& all, uint64_t& some) {
    uint64_t v[4];
    for (int k = 0; k < 4; k++) std::memcpy(&v[k], p + (k < 3 ? 8 * k : kResCols - 8), 8);
    all = v[0] & v[1] & v[2] & v[3];
    some = v[0] | v[1] | v[2] | v[3];
  };
  bool any = false;
  for (int y = 0; y < h; y++) {
    const uint8_t* c = code + (size_t)y * pitch;
    auto mark = [&](int x, int yy) { need[(size_t)(yy / kResRows[0]) * tx + x / kResCols] = 1; };
    // per pixel: 1 on, 2 interior, 4 takes part in a read of a masked-out pixel
    auto flags = [&](int x) -> uint8_t {
      const uint8_t k = c[x];
      if (!(k & kOn)) return 0;
      if (!masked) return x >= 1 && y >= 1 && x + 1 < w && y + 1 < h ? 3 : 1;
      if (k == kAll) return 3;
      return !(k & (kR | kL)) || !(k & (kD | kU)) ? 5 : 1;
    };
    for (int i = 0; i < tx; i++) {
      const int x0 = i * kResCols, x1 = std::min(w, x0 + kResCols);
      uint8_t all = 7, some = 0;
      bool read = true;  // whether a pixel may read one that is off
      if (x0 + kResCols <= w) {
        uint64_t a, o;
        bits(c + x0, a, o);
        if (!(o & (kEach * kOn))) {
          all = 0;
          read = false;
        } else if (masked && a == kEach * kAll && o == a) {
          all = some = 3;
          read = false;
        } else if (!masked && (a & (kEach * kOn)) == kEach * kOn && x0 >= 1 && x1 < w && y >= 1 && y + 1 < h && (c[x1] & kOn)) {
          bits(c + pitch + x0, a, o);
          if ((a & (kEach * kOn)) == kEach * kOn) {
            all = some = 3;
            read = false;
          }
        }
      }
      if (read) {
        for (int x = x0; x < x1; x++) {
          const uint8_t k = c[x], f = flags(x);
          all &= f;
          some |= f;
          if (!(f & 1) || (masked && f == 3)) continue;
          if (masked) {
            // the neighbours an edge rule falls back to, which may be masked out
            if (!(k & kR)) {
              if (x == 0) return false;
              mark(x - 1, y);
            }
            if (!(k & kD)) {
              if (y == 0) return false;
              mark(x, y - 1);
            }
          } else {
            // a pixel outside the circle that the first iteration reads
            if (x + 1 < w && !(c[x + 1] & kOn)) mark(x + 1, y);
            if (y + 1 < h && !(c[x + pitch] & kOn)) mark(x, y + 1);
          }
        }
      }
      if (some & 1) {
        any = true;
        need[(size_t)(y / kResRows[0]) * tx + i] = 1;
      }
      inner[(size_t)y * tx + i] = x0 >= 1 && x0 + kResCols <= w && (all & 2) && (flags(x0 - 1) & 2);
      if (masked) {
        if (x0 >= 1) some |= flags(x0 - 1);
        if (x1 < w) some |= flags(x1);
      }
      keep[(size_t)y * tx + i] = some & 4;
    }
  }
  return any;
}

int ResLevel::count(int rows) const {
  const int per = rows / kResRows[0], ty2 = (int)(need.size() / tx);
  int n = 0;
  for (int j = 0; j < ty2; j += per)
    for (int i = 0; i < tx; i++) {
      uint8_t v = 0;
      for (int k = j; k < std::min(ty2, j + per); k++) v |= need[(size_t)k * tx + i];
      n += v;
    }
  return n;
}

void ResLevel::tiles(int rows, ResTiles& out) const {
  out.rows = rows;
  out.tiles.clear();
  out.fill.clear();
  const int per = rows / kResRows[0], ty2 = (int)(need.size() / tx), ty = (h + rows - 1) / rows;
  std::vector<int> id((size_t)tx * ty, -1);
  for (int j = 0; j < ty; j++)
    for (int i = 0; i < tx; i++) {
      uint8_t v = 0;
      for (int k = j * per; k < std::min(ty2, (j + 1) * per); k++) v |= need[(size_t)k * tx + i];
      if (!v) {
        if (!masked) out.fill.push_back(make_int2(i * kResCols, j * rows));
        continue;
      }
      id[(size_t)j * tx + i] = (int)out.tiles.size();
      ResTile t{};
      t.x0 = i * kResCols;
      t.y0 = j * rows;
      out.tiles.push_back(t);
    }
  for (int j = 0; j < ty; j++)
    for (int i = 0; i < tx; i++) {
      const int k = id[(size_t)j * tx + i];
      if (k < 0) continue;
      ResTile& t = out.tiles[k];
      auto at = [&](int a, int b) {
        if (a < 0 || b < 0 || a >= tx || b >= ty) return k;
        const int n = id[(size_t)b * tx + a];
        return n < 0 ? k : n;
      };
      const int nb[8] = {at(i, j - 1),     at(i, j + 1),     at(i - 1, j),     at(i + 1, j),
                         at(i - 1, j - 1), at(i + 1, j - 1), at(i - 1, j + 1), at(i + 1, j + 1)};
      std::copy(nb, nb + 8, t.nb);
      // interior: the owned pixels, the column west of them and the row above, whose steps the
      // tile evaluates, are on with all four neighbours in the image (and, masked, on)
      bool in = t.y0 >= 1 && t.y0 + rows <= h, kept = false;
      for (int y = t.y0 - 1; in && y < t.y0 + rows; y++) in = inner[(size_t)y * tx + i];
      for (int y = std::max(0, t.y0 - 1); !in && y <= std::min(h - 1, t.y0 + rows); y++) kept |= keep[(size_t)y * tx + i] != 0;
      t.kind = in ? kResInner : kept ? kResKeep : kResEdge;
    }
}

void ResTiles::place(int grid) {
  blocks = grid;
  const int n = (int)tiles.size();
  // tiles per scheduler of a block that has all its warps, or one less
  auto load = [&](int t) {
    const int b = t % grid, warps = std::max(1, (n - b + grid - 1) / grid), w = t / grid;
    return (warps - w % 4 + 3) / 4;
  };
  std::vector<int> slot(n), tile(n), to(n);
  for (int t = 0; t < n; t++) slot[t] = tile[t] = t;
  std::stable_sort(slot.begin(), slot.end(), [&](int a, int b) { return load(a) < load(b); });
  std::stable_sort(tile.begin(), tile.end(), [&](int a, int b) { return tiles[a].kind > tiles[b].kind; });
  for (int k = 0; k < n; k++) to[tile[k]] = slot[k];
  std::vector<ResTile> placed(n);
  for (int t = 0; t < n; t++) {
    ResTile r = tiles[t];
    for (int& k : r.nb) k = to[k];
    placed[to[t]] = r;
  }
  tiles.swap(placed);
}

// The smallest tile height whose tiles fit, since more warps with less to do each hide more of one
// another's latency and shorten an iteration (B200, us per iteration, FP16 / float storage: 848 x 800
// disc 8 rows 3.7 / 6.3; 640 x 480 4 rows 2.45 / 3.6, 6 rows 2.75 / 3.9, 8 rows 3.1 / 5.3; 212 x 200
// 2 rows 1.40 / 1.73, 4 rows 1.60 / 2.15).  Two rows are left to levels that fill at most three
// quarters of the warps: fuller, the row above each tile, which two rows pay for as much as four,
// costs more than it gives (424 x 400, 91 %: 2 rows 2.0, 4 rows 1.87).  12 and 16 rows (half storage) cost
// more a pixel (kernels_resident.cu) and take the levels that 8 rows do not.
bool res_choose(const uint8_t* code, int pitch, int w, int h, bool masked, bool half, ResTiles& out) {
  int dev = 0, sms = 0;
  VFS_CUDA(cudaGetDevice(&dev));
  VFS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ResLevel L;
  if (!L.scan(code, pitch, w, h, masked)) return false;
  out.cluster = false;
  // (a capacity is asked for only where the count may fit: the first question loads the kernel)
  if (const int n = L.count(kResClusterRows);
      n <= res_cluster_tiles(half) && n <= res_capacity(masked, half, kResClusterRows, kResClusterCtas)) {
    L.tiles(kResClusterRows, out);
    out.cluster = true;
    out.place(kResClusterCtas);
    return true;
  }
  for (int k = 0; k < kResNumRows; k++) {
    const int rows = kResRows[k];
    const int n = L.count(rows);
    if (n > sms * kResMostWarps) continue;
    const int cap = res_capacity(masked, half, rows);
    if (n > cap || (rows == kResRows[0] && 4 * (long long)n > 3 * (long long)cap)) continue;
    L.tiles(rows, out);
    out.place(std::min(sms, n));
    return true;
  }
  return false;
}

size_t res_bytes_bound(int w, int h) {
  size_t most = 0;
  for (int k = 0; k < kResNumRows; k++) {
    const int rows = kResRows[k];
    const size_t tiles = std::min<size_t>((size_t)((w + kResCols - 1) / kResCols) * ((h + rows - 1) / rows), kResMostTiles);
    most = std::max(most, tiles * (kResRing * res_slots(rows) * sizeof(uint4) + sizeof(ResTile) + sizeof(int2)));
  }
  return most + 4 * 256 + sizeof(ResCtl);
}

}  // namespace vfs
