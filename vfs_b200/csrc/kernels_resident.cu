// Kernels of the register-resident iteration (resident.cuh).
#include "resident.cuh"

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "tgv_exact_pairs.cuh"
#include "tgv_pixel.cuh"
#include "tgv_pixel_fast.cuh"

namespace vfs {

namespace x2 = fast::x2;

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kResLooks = 1 << 20;  // after which a wait gives up: some 0.5 to 1 s

__device__ int g_res_status;  // 1 = a wait for a neighbour's words ran out

__device__ __forceinline__ void give_up(const ResArgs& A) {
  g_res_status = 1;
  *(volatile unsigned*)A.gave_up = 1u;
}

// one exchange word as a single 128-bit memory operation at L2
__device__ __forceinline__ void st_word(uint4* p, uint4 v) {
  const unsigned long long lo = v.x | ((unsigned long long)v.y << 32), hi = v.z | ((unsigned long long)v.w << 32);
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo),
               "l"(hi)
               : "memory");
}
__device__ __forceinline__ uint4 ld_word(const uint4* p) {
  unsigned long long lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}

__device__ __forceinline__ unsigned bits(__half2 h) { return *reinterpret_cast<unsigned*>(&h); }
__device__ __forceinline__ __half2 as_half2(unsigned b) { return *reinterpret_cast<__half2*>(&b); }

// Per-warp shared memory: the coefficients (rows -1 .. R-1) and edge codes, and a place to hand
// the halo columns to lanes 0 and 31.  At a masked-out pixel a and b hold its stale T p instead
// (its tensor is not used).
// Beside them each lane's exchange offsets and pixel masks, read back at every iteration.
// half storage (up to 8 rows): rows in pairs, each coefficient's two rows side by side for the packed
// instructions: (a, b), (c, 1 / eta_u), (Iu, Iz), (1 / eta_v1, 1 / eta_v2), 1 / Iu
// float storage: (a, b), (c, Iu), Iz, and p, (q.x, q.y), (q.z, q.w) in the same pairs
// What a lane's edge rules need, bit r + 1 for row r: x (y): the pixel is on and takes its right
// (lower) neighbour; on: the pixel is on.
struct ResEdge {
  unsigned x, y, on;
};
// What a warp reads back at every iteration.
struct ResLinks {
  uint4 at[32];    // per lane: exchange words of ring slot 0 read from above, below and beside; e.x
  uint2 edge[32];  // e.y, e.on
  int kind;        // ResKind of the tile
  int t;           // tile
  int pad[2];
};
template <class ST, int R>
struct ResShared;
template <int R, bool TALL = (R > 8), bool STREAM = (R > 12)>
struct ResSharedHalf;
template <int R>
struct ResSharedHalf<R, false, false> {
  float4 top[32];
  float4 cf[R / 2][4][32];
  float2 riu[R / 2][32];
  uint2 p[R / 2][32];
  uint4 q[R / 2][32];
  uint4 pqtop[32];
  uint2 col[2][R];
  ResLinks k;
};
// tall tiles: (a, b), c, p, (q.x, q.y and q.z, q.w) and, up to 12 rows, (Iu, Iz); the row above's p and q
template <int R>
struct ResSharedHalf<R, true, true> {
  float4 top[32];
  float4 ab[R / 2][32];
  float2 c[R / 2][32];
  uint2 p[R / 2][32];
  uint4 q[R / 2][32];
  uint4 pqtop[32];
  uint2 col[2][R];
  ResLinks k;
};
template <int R>
struct ResSharedHalf<R, true, false> : ResSharedHalf<R, true, true> {
  float4 uz[R / 2][32];
};
template <int R>
struct ResShared<__half, R> : ResSharedHalf<R> {};
template <int R>
struct ResShared<float, R> {
  float4 top[32];
  float4 ab[R / 2][32], ci[R / 2][32];
  float4 p[R / 2][32], qxy[R / 2][32], qzw[R / 2][32];
  float4 qtop[32];
  float2 iz[R / 2][32];
  float2 ptop[32];
  uint4 col[2][R];
  ResLinks k;
};

__device__ __forceinline__ float lo(x2::f2 v) { return x2::upk(v).x; }
__device__ __forceinline__ x2::f2 both(float v) { return x2::pk(v, v); }
__device__ __forceinline__ float hi(x2::f2 v) { return x2::upk(v).y; }
__device__ __forceinline__ float2 unpack(unsigned h) { return __half22float2(as_half2(h)); }
__device__ __forceinline__ unsigned pack(float x, float y) { return bits(__float22half2_rn(make_float2(x, y))); }

// A tile's state and its iteration.
template <bool MASKED, class ST, int R>
struct ResState;

// Half storage.  Rows are taken two at a time, a row's value in each half of the packed FP32
// instructions, so that nearly every operation of the dual, threshold and primal steps serves
// two pixels; only the differences along a column, whose operands straddle the pairs, the
// comparisons and the conversions are per pixel.
//
// From 6 rows on p and q are in shared memory; in registers they left too few for the rest (848 x 800, 8
// rows: 276 bytes spilled, 3.93 us per iteration; 4 bytes, 3.73).
//
// Tall tiles (12 and 16 rows) hold levels that 8 rows in 16 warps do not, up to 0.85 and 1.1 million
// pixels.  The room comes from the reciprocals (formed again at every iteration, 24 instructions a
// pair of rows) and, with 16 rows, from Iu and Iz (read again from L2, 8 bytes a pixel of the
// one-iteration kernel's 96).  Their rows are taken four at a time by one piece of code, between whose
// passes the registers move up: 16 rows unrolled by eight leave the instruction cache (1280 x 1024
// disc, 2174 tiles of 16 rows: 11.6 us per iteration; by four 9.3; one launch per iteration 15.0.
// 1000 x 900, 1883 tiles of 12: 6.1; 9.85).  Instruction issue bounds both.
template <bool MASKED, int R>
struct ResState<MASKED, __half, R> {
  typedef ResShared<__half, R> Sh;
  typedef x2::f2 f2;
  static constexpr bool kTall = R > 8, kStream = R > 12;
  static constexpr int kPasses = kTall ? R / 4 : 1, kPairs = R / 2 / kPasses;
  static constexpr bool kSharedPQ = R > 4;
  static constexpr int kHeld = kSharedPQ ? 0 : R;
  f2 u[R / 2], ub[R / 2];
  unsigned v[R];                                             // v-bar
  unsigned p[kHeld + 1], q0[kHeld + 1], q1[kHeld + 1];       // rows -1 .. R-1: p, (q.x, q.y), (q.z, q.w)

  __device__ __forceinline__ void clear(Sh& sh, int lane) {
    if constexpr (kSharedPQ) {
#pragma unroll
      for (int i = 0; i < R / 2; i++) {
        sh.p[i][lane] = make_uint2(0u, 0u);
        sh.q[i][lane] = make_uint4(0u, 0u, 0u, 0u);
      }
      sh.pqtop[lane] = make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
      for (int i = 0; i <= R; i++) p[i] = q0[i] = q1[i] = 0u;
    }
  }
  // what a pixel has in memory (kept: masked out, with the other ping-pong buffer's values)
  struct Pixel {
    float4 ca;
    float2 rv, tp;
    float iu, iz, u, ub;
    unsigned v;
  };
  static __device__ __forceinline__ Pixel fetch(const IterPair& P, int r, bool in, bool kept, int pos) {
    Pixel x{make_float4(0.f, 0.f, 0.f, 1.f), make_float2(1.f, 1.f), make_float2(0.f, 0.f), 0.f, 0.f, 0.f, 0.f, 0u};
    if (in) x.ca = P.abce[pos];
    if (kept) x.tp = P.Tp[pos];
    if (r < 0) return x;
    if (!kTall && in) x.rv = P.rv[pos];
    if (in) {
      x.iu = P.Iu[pos];
      x.iz = P.Iz[pos];
      x.u = kept ? P.u_s[pos] : P.u[pos];
      x.ub = P.u_[pos];
    }
    if (kept) x.v = bits(((const __half2*)P.v_s)[pos]);
    return x;
  }
  // east / south: edge codes of the pixel's right and lower neighbour
  __device__ __forceinline__ bool set_row(Sh& sh, int lane, const IterPair&, int r, bool, bool kept, Pixel x, unsigned,
                                          unsigned east, unsigned south) {
    if (kept) {
      // read by the right / lower neighbour only where that one's other side is off too
      x.ca.x = (east & kOn) && !(east & kR) ? x.tp.x : 0.f;
      x.ca.y = (south & kOn) && !(south & kD) ? x.tp.y : 0.f;
    }
    if (r < 0) {
      sh.top[lane] = x.ca;
      return false;
    }
    const int i = r >> 1, k = r & 1;
    if constexpr (kTall) {
      reinterpret_cast<float*>(&sh.ab[i][lane])[k] = x.ca.x;
      reinterpret_cast<float*>(&sh.ab[i][lane])[2 + k] = x.ca.y;
      reinterpret_cast<float*>(&sh.c[i][lane])[k] = x.ca.z;
      if constexpr (!kStream) {
        reinterpret_cast<float*>(&sh.uz[i][lane])[k] = x.iu;
        reinterpret_cast<float*>(&sh.uz[i][lane])[2 + k] = x.iz;
      }
    } else {
      // eta_v2 = 0 (updatePrimalVariables.cu:103-105): .x takes tau itself, .y keeps its value
      if (fast::etav2_zero(x.rv.y)) x.rv = make_float2(1.f, 0.f);
      const float c[8] = {x.ca.x, x.ca.y, x.ca.z, x.ca.w, x.iu, x.iz, x.rv.x, x.rv.y};
#pragma unroll
      for (int j = 0; j < 8; j++) reinterpret_cast<float*>(&sh.cf[i][j >> 1][lane])[2 * (j & 1) + k] = c[j];
      // the Newton step -rho / Iu of the threshold; 0 where Iu = 0 (no step there)
      reinterpret_cast<float*>(&sh.riu[i][lane])[k] = x.iu == 0.0f ? 0.0f : fast::rcp(x.iu);
    }
    v[r] = 0u;
    if (kept) {
      if constexpr (kSharedPQ) (k ? sh.p[i][lane].y : sh.p[i][lane].x) = x.v;
      else p[r + 1] = x.v;
    }
    u[i] = k ? x2::pk(lo(u[i]), x.u) : x2::pk(x.u, 0.f);
    ub[i] = k ? x2::pk(lo(ub[i]), x.ub) : x2::pk(x.ub, 0.f);
    return false;
  }
  __device__ __forceinline__ float u_of(int r) const { return r & 1 ? hi(u[r >> 1]) : lo(u[r >> 1]); }
  __device__ __forceinline__ float ub_of(int r) const { return r & 1 ? hi(ub[r >> 1]) : lo(ub[r >> 1]); }
  __device__ __forceinline__ __half2 v_of(int r) const { return as_half2(v[r]); }
  __device__ __forceinline__ uint4 word(int r, unsigned tag) const {
    return make_uint4(__float_as_uint(ub_of(r)), v[r], 0u, tag);
  }
  static __device__ __forceinline__ void put_col(Sh& sh, int side, int r, uint4 w) { sh.col[side][r] = make_uint2(w.x, w.y); }
  __device__ __forceinline__ void take_col(const uint2* col) {
#pragma unroll
    for (int i = 0; i < R / 2; i++) {
      const uint4 w = *reinterpret_cast<const uint4*>(col + 2 * i);
      ub[i] = x2::pk(__uint_as_float(w.x), __uint_as_float(w.z));
      v[2 * i] = w.y;
      v[2 * i + 1] = w.w;
    }
  }
  __device__ __forceinline__ void store_pq(const Sh& sh, int lane, int r, void* po, void* qo, int pos) const {
    uint2 q;
    unsigned pv;
    if constexpr (kSharedPQ) {
      const uint2 pp = sh.p[r >> 1][lane];
      const uint4 qq = sh.q[r >> 1][lane];
      pv = r & 1 ? pp.y : pp.x;
      q = r & 1 ? make_uint2(qq.y, qq.w) : make_uint2(qq.x, qq.z);
    } else {
      pv = p[r + 1];
      q = make_uint2(q0[r + 1], q1[r + 1]);
    }
    reinterpret_cast<unsigned*>(po)[pos] = pv;
    reinterpret_cast<uint2*>(qo)[pos] = q;
  }
  // entry i of a pass to the place of the last pass's, the others' one pass up (n entries a pair)
  template <class T>
  static __device__ __forceinline__ void roll(T* a, int i, int n) {
    const T t = a[i];
#pragma unroll
    for (int k = 0; k + 1 < kPasses; k++) a[k * kPairs * n + i] = a[(k + 1) * kPairs * n + i];
    a[(kPasses - 1) * kPairs * n + i] = t;
  }
  // the reciprocals of a pair of rows: 1 / eta_u, 1 / eta_v1 and 1 / eta_v2, 1 / Iu, as in the level's
  // records (fast::etau_rcp, etav_rcp) and in set_row
  static __device__ __forceinline__ void reciprocals(f2 a, f2 b, f2 c, f2 iu, const IterPair& P, f2& re, f2& rx, f2& ry,
                                                     f2& riu) {
    using namespace x2;
    const f2 a1s = both(P.alpha1 * P.alpha1), a0s4 = both(4 * P.alpha0 * P.alpha0);
    const f2 bb = mul(b, b), ac = add(a, c), bc = add(b, c), cc = mul(c, c);
    const f2 eu = mul(fma(bc, bc, fma(ac, ac, fma(add(c, c), c, fma(a, a, bb)))), a1s);
    const f2 e1 = fma(a1s, fma(b, b, cc), a0s4), e2 = fma(a1s, fma(a, a, cc), a0s4);
    auto one = [](float e, float i, float x, float y, float& ro, float& xo, float& yo, float& io) {
      ro = e == 0.0f ? 1.0f : fast::rcp(e);
      xo = x != 0.0f && y != 0.0f ? fast::rcp(x) : 1.0f;
      yo = y != 0.0f ? fast::rcp(y) : 0.0f;
      io = i == 0.0f ? 0.0f : fast::rcp(i);
    };
    float r0, r1, x0, x1, y0, y1, i0, i1;
    one(lo(eu), lo(iu), lo(e1), lo(e2), r0, x0, y0, i0);
    one(hi(eu), hi(iu), hi(e1), hi(e2), r1, x1, y1, i1);
    re = pk(r0, r1);
    rx = pk(x0, x1);
    ry = pk(y0, y1);
    riu = pk(i0, i1);
  }

  // One iteration.  wn / ws: the words of the row above / below the tile.  KIND: ResKind of the
  // tile.  E: what the edge rules need (bit r + 1 of each mask: row r).
  //
  // Edge rules.  The x difference of an on pixel takes its right neighbour where that is on, else
  // its left one; either is the difference to the east of a lane, its own or its west lane's.
  // The threshold and primal steps take T p.x, q.x and q.w of the pixel and of its left
  // neighbour; the pixel's own count where its right neighbour is on, the left one's where that is
  // on, which is the same condition seen from the left pixel (it is on, and so is its right
  // neighbour).  So those values are replaced by zero once, at the pixel, where it is off or
  // its right neighbour is; likewise along y.  (-0 in T p, so that 0 - x is -x.)
  template <int KIND>
  __device__ __forceinline__ void iterate(Sh& sh, const ResArgs& A, int lane, const ResStep& S, ResEdge E,
                                          uint4 wn, uint4 ws, float2* tp_out, int s, unsigned tp_rows) {
    using namespace x2;
    constexpr bool EDGE = KIND != kResInner;
    constexpr bool KEEP = MASKED && KIND == kResKeep;
    const f2 sp = pk(S.sp.x, S.sp.y), sq = pk(S.sq.x, S.sq.y), tau = pk(S.tau.x, S.tau.y), mu = pk(S.mu.x, S.mu.y);
    const f2 lam = both(A.P.lambda), al0 = both(A.P.alpha0), al1 = both(A.P.alpha1);
    auto bit = [](unsigned m, int r) { return (m >> (r + 1)) & 1u; };
    // streamed: positions of the pair's two rows and of the next pair's first, rows of the image below that
    int a0 = 0, a1 = 0, at = 0, left = 0;
    auto next = [&](f2& iu, f2& iz) {
      a0 = at;
      a1 = left > 0 ? at + s : at;
      at = left > 1 ? a1 + s : a1;
      left -= 2;
      iu = pk(__ldg(A.P.Iu + a0), __ldg(A.P.Iu + a1));
      iz = pk(__ldg(A.P.Iz + a0), __ldg(A.P.Iz + a1));
    };
    if constexpr (kStream) {  // (beyond the image: some pixel of it, for lanes and rows that nothing reads)
      const ResTile& T = A.tiles[sh.k.t];
      at = min(max(T.x0 - 1 + lane, 0), A.P.w - 1) + T.y0 * s;
      left = A.P.h - 1 - T.y0;
    }
    // row -1: its dual step, for T p and q of the row above row 0
    float tpy_n, qz_n, qy_n;       // T p.y, q.z and q.y of the row above
    float du_n;                    // u-bar and v-bar less those of the row above
    float2 dv_n;
    float2 vc = unpack(v[0]);      // v-bar of the pair's first row
    {
      const float4 ca = sh.top[lane];
      const float ubc = __uint_as_float(wn.x);
      const float2 vp = unpack(wn.y), ve = unpack(__shfl_down_sync(kFull, wn.y, 1));
      float dux = __shfl_down_sync(kFull, ubc, 1) - ubc;
      float2 dvx = make_float2(ve.x - vp.x, ve.y - vp.y);
      du_n = lo(ub[0]) - ubc;
      dv_n = make_float2(vc.x - vp.x, vc.y - vp.y);
      if (EDGE) {
        const float wu = __shfl_up_sync(kFull, dux, 1);
        const float2 wv = make_float2(__shfl_up_sync(kFull, dvx.x, 1), __shfl_up_sync(kFull, dvx.y, 1));
        const bool r0 = bit(E.x, -1);
        dux = r0 ? dux : wu;
        dvx = make_float2(r0 ? dvx.x : wv.x, r0 ? dvx.y : wv.y);
      }
      const float gx = dux - vp.x, gy = du_n - vp.y;
      if constexpr (kSharedPQ) {
        const uint4 t = sh.pqtop[lane];
        p[0] = t.x;
        q0[0] = t.y;
        q1[0] = t.z;
      }
      const float2 h0 = unpack(p[0]), h1 = unpack(q0[0]), h2 = unpack(q1[0]);
      float px = __fmaf_rn(S.sp.x, __fmaf_rn(ca.x, gx, ca.z * gy), h0.x);
      float py = __fmaf_rn(S.sp.x, __fmaf_rn(ca.z, gx, ca.y * gy), h0.y);
      const float rp = fast::unit_scale(__fmaf_rn(px, px, py * py));
      px *= rp;
      py *= rp;
      float qx = __fmaf_rn(S.sq.x, dvx.x, h1.x), qy = __fmaf_rn(S.sq.x, dv_n.y, h1.y);
      float qz = __fmaf_rn(S.sq.x, dv_n.x, h2.x), qw = __fmaf_rn(S.sq.x, dvx.y, h2.y);
      const float rq = fast::unit_scale(__fmaf_rn(qx, qx, __fmaf_rn(qy, qy, __fmaf_rn(qz, qz, qw * qw))));
      qx *= rq;
      qy *= rq;
      qz *= rq;
      qw *= rq;
      p[0] = pack(px, py);
      q0[0] = pack(qx, qy);
      q1[0] = pack(qz, qw);
      if constexpr (kSharedPQ) sh.pqtop[lane] = make_uint4(p[0], q0[0], q1[0], 0u);
      tpy_n = __fmaf_rn(ca.z, px, ca.y * py);
      qz_n = qz;
      qy_n = qy;
      if (EDGE) {
        const bool d0 = bit(E.y, -1);
        const bool o0 = MASKED ? d0 : bit(E.on, -1);
        tpy_n = o0 ? tpy_n : KEEP && !bit(E.on, -1) ? ca.y : -0.0f;
        qz_n = d0 ? qz : 0.f;
        qy_n = d0 ? qy : 0.f;
      }
    }
#pragma unroll 1
    for (int pass = 0; pass < kPasses; pass++) {
#pragma unroll
      for (int i = 0; i < kPairs; i++) {
        const int r = 2 * i, is = pass * kPairs + i;
        constexpr int kNext = kTall ? kPairs : 0;  // the first pair of the next pass
        const f2 UB = ub[i];
        const float ub0 = lo(UB), ub1 = hi(UB);
        const float2 v1 = unpack(v[r + 1]);
        const bool more = kTall && pass + 1 < kPasses;
        const int in_ = i + 1 < kPairs ? i + 1 : kNext;
        const float ubd = i + 1 < kPairs || more ? lo(ub[in_]) : __uint_as_float(ws.x);
        const float2 vd = unpack(i + 1 < kPairs || more ? v[2 * in_] : ws.y);
        const f2 VX = pk(vc.x, v1.x), VY = pk(vc.y, v1.y);
        ulonglong2 ab, ce, uz, rr;
        f2 riu;
        unsigned pa, pb, qa0h, qa1h, qb0h, qb1h;  // p, (q.x, q.y), (q.z, q.w) of the two rows
        if constexpr (kTall) {
          ab = *reinterpret_cast<const ulonglong2*>(&sh.ab[is][lane]);
          ce.x = *reinterpret_cast<const f2*>(&sh.c[is][lane]);
          if constexpr (kStream) {
            next(uz.x, uz.y);
          } else {
            uz = *reinterpret_cast<const ulonglong2*>(&sh.uz[is][lane]);
          }
          reciprocals(ab.x, ab.y, ce.x, uz.x, A.P, ce.y, rr.x, rr.y, riu);
        } else {
          ab = *reinterpret_cast<const ulonglong2*>(&sh.cf[i][0][lane]);
          ce = *reinterpret_cast<const ulonglong2*>(&sh.cf[i][1][lane]);
          uz = *reinterpret_cast<const ulonglong2*>(&sh.cf[i][2][lane]);
          rr = *reinterpret_cast<const ulonglong2*>(&sh.cf[i][3][lane]);
          riu = *reinterpret_cast<const f2*>(&sh.riu[i][lane]);
        }
        if constexpr (kSharedPQ) {
          const uint2 pp = sh.p[is][lane];
          const uint4 qq = sh.q[is][lane];
          pa = pp.x, pb = pp.y, qa0h = qq.x, qa1h = qq.y, qb0h = qq.z, qb1h = qq.w;
        } else {
          pa = p[r + 1], pb = p[r + 2], qa0h = q0[r + 1], qa1h = q0[r + 2], qb0h = q1[r + 1], qb1h = q1[r + 2];
        }
        // ---- differences of u-bar and v-bar to the east and to the south -----------------
        const float2 e0 = unpack(__shfl_down_sync(kFull, v[r], 1)), e1 = unpack(__shfl_down_sync(kFull, v[r + 1], 1));
        f2 dux = sub(pk(__shfl_down_sync(kFull, ub0, 1), __shfl_down_sync(kFull, ub1, 1)), UB);
        f2 dxx = sub(pk(e0.x, e1.x), VX), dxy = sub(pk(e0.y, e1.y), VY);
        const float du0 = ub1 - ub0, du1 = ubd - ub1;
        const float2 dv0 = make_float2(v1.x - vc.x, v1.y - vc.y), dv1 = make_float2(vd.x - v1.x, vd.y - v1.y);
        f2 duy = pk(du0, du1), dyx = pk(dv0.x, dv1.x), dyy = pk(dv0.y, dv1.y);
        bool r0 = true, r1 = true, d0 = true, d1 = true;
        if (EDGE) {
          r0 = bit(E.x, r);
          r1 = bit(E.x, r + 1);
          d0 = bit(E.y, r);
          d1 = bit(E.y, r + 1);
          const float wu0 = __shfl_up_sync(kFull, lo(dux), 1), wu1 = __shfl_up_sync(kFull, hi(dux), 1);
          const float wx0 = __shfl_up_sync(kFull, lo(dxx), 1), wx1 = __shfl_up_sync(kFull, hi(dxx), 1);
          const float wy0 = __shfl_up_sync(kFull, lo(dxy), 1), wy1 = __shfl_up_sync(kFull, hi(dxy), 1);
          dux = pk(r0 ? lo(dux) : wu0, r1 ? hi(dux) : wu1);
          dxx = pk(r0 ? lo(dxx) : wx0, r1 ? hi(dxx) : wx1);
          dxy = pk(r0 ? lo(dxy) : wy0, r1 ? hi(dxy) : wy1);
          duy = pk(d0 ? du0 : du_n, d1 ? du1 : du0);
          dyx = pk(d0 ? dv0.x : dv_n.x, d1 ? dv1.x : dv0.x);
          dyy = pk(d0 ? dv0.y : dv_n.y, d1 ? dv1.y : dv0.y);
          du_n = du1;
          dv_n = dv1;
        }
        // ---- dual step ------------------------------------------------------------------
        const f2 a = ab.x, b = ab.y, c = ce.x;
        const f2 ux = sub(dux, VX), uy = sub(duy, VY);
        const float2 p0 = unpack(pa), p1 = unpack(pb);
        const float2 qa0 = unpack(qa0h), qa1 = unpack(qa1h), qb0 = unpack(qb0h), qb1 = unpack(qb1h);
        f2 px = fma(sp, fma(a, ux, mul(c, uy)), pk(p0.x, p1.x));
        f2 py = fma(sp, fma(c, ux, mul(b, uy)), pk(p0.y, p1.y));
        const f2 n2 = fma(px, px, mul(py, py));
        const f2 rp = pk(fast::unit_scale(lo(n2)), fast::unit_scale(hi(n2)));
        px = mul(px, rp);
        py = mul(py, rp);
        f2 qx = fma(sq, dxx, pk(qa0.x, qa1.x));
        f2 qy = fma(sq, dyy, pk(qa0.y, qa1.y));
        f2 qz = fma(sq, dyx, pk(qb0.x, qb1.x));
        f2 qw = fma(sq, dxy, pk(qb0.y, qb1.y));
        const f2 m2 = fma(qx, qx, fma(qy, qy, fma(qz, qz, mul(qw, qw))));
        const f2 rq = pk(fast::unit_scale(lo(m2)), fast::unit_scale(hi(m2)));
        qx = mul(qx, rq);
        qy = mul(qy, rq);
        qz = mul(qz, rq);
        qw = mul(qw, rq);
        f2 tpx = fma(a, px, mul(c, py)), tpy = fma(c, px, mul(b, py));
        unsigned pn0 = pack(lo(px), lo(py)), pn1 = pack(hi(px), hi(py));
        if constexpr (kSharedPQ) {
          sh.q[is][lane] =
              make_uint4(pack(lo(qx), lo(qy)), pack(hi(qx), hi(qy)), pack(lo(qz), lo(qw)), pack(hi(qz), hi(qw)));
        } else {
          q0[r + 1] = pack(lo(qx), lo(qy));
          q1[r + 1] = pack(lo(qz), lo(qw));
          q0[r + 2] = pack(hi(qx), hi(qy));
          q1[r + 2] = pack(hi(qz), hi(qw));
        }
        auto put = [&](int row, int pos, float2 t) {
          if constexpr (kStream) A.P.Tp[pos] = t;
          else tp_out[row * s] = t;
        };
        if (!MASKED && EDGE) {  // outside the circle p = 0: T p = T 0
          const float2 z = make_float2(0.f, 0.f);
          if ((tp_rows >> r) & 1u)
            put(r, a0, bit(E.on, r) ? make_float2(lo(tpx), lo(tpy)) : tp_math(lo(a), lo(b), lo(c), z));
          if ((tp_rows >> (r + 1)) & 1u)
            put(r + 1, a1, bit(E.on, r + 1) ? make_float2(hi(tpx), hi(tpy)) : tp_math(hi(a), hi(b), hi(c), z));
        } else {
          if ((tp_rows >> r) & 1u) put(r, a0, make_float2(lo(tpx), lo(tpy)));
          if ((tp_rows >> (r + 1)) & 1u) put(r + 1, a1, make_float2(hi(tpx), hi(tpy)));
        }
        // ---- threshold step -----------------------------------------------------------
        f2 txo = tpx, tyo = tpy;  // as counted for this pixel and its right / lower neighbour
        bool o0 = true, o1 = true;
        if (EDGE) {
          if (KEEP || !MASKED) {
            o0 = bit(E.on, r);
            o1 = bit(E.on, r + 1);
          }
          const float zx0 = KEEP && !o0 ? lo(a) : -0.0f, zx1 = KEEP && !o1 ? hi(a) : -0.0f;
          const float zy0 = KEEP && !o0 ? lo(b) : -0.0f, zy1 = KEEP && !o1 ? hi(b) : -0.0f;
          // the plain form takes the difference at the last row and column too
          txo = pk((MASKED ? r0 : o0) ? lo(tpx) : zx0, (MASKED ? r1 : o1) ? hi(tpx) : zx1);
          tyo = pk((MASKED ? d0 : o0) ? lo(tpy) : zy0, (MASKED ? d1 : o1) ? hi(tpy) : zy1);
          qx = pk(r0 ? lo(qx) : 0.f, r1 ? hi(qx) : 0.f);
          qw = pk(r0 ? lo(qw) : 0.f, r1 ? hi(qw) : 0.f);
          qz = pk(d0 ? lo(qz) : 0.f, d1 ? hi(qz) : 0.f);
          qy = pk(d0 ? lo(qy) : 0.f, d1 ? hi(qy) : 0.f);
        }
        const f2 tpw = pk(__shfl_up_sync(kFull, lo(txo), 1), __shfl_up_sync(kFull, hi(txo), 1));
        const f2 qxw = pk(__shfl_up_sync(kFull, lo(qx), 1), __shfl_up_sync(kFull, hi(qx), 1));
        const f2 qww = pk(__shfl_up_sync(kFull, lo(qw), 1), __shfl_up_sync(kFull, hi(qw), 1));
        const f2 dy = pk(lo(tyo) - tpy_n, hi(tyo) - lo(tyo));
        const f2 dqz = pk(lo(qz) - qz_n, hi(qz) - lo(qz)), dqy = pk(lo(qy) - qy_n, hi(qy) - lo(qy));
        const f2 U = u[i], iu = uz.x;
        const f2 teu = mul(tau, ce.y);
        const f2 dun = sub(fma(teu, add(sub(txo, tpw), dy), UB), U);
        const f2 rho = fma(iu, dun, uz.y);
        const f2 lt = mul(lam, teu);
        const f2 up = mul(lt, mul(iu, iu));
        f2 un;
        {
          // |rho| <= upper: the Newton step; beyond it a step of lambda tau / eta_u against the sign of
          // rho (lambda >= 0); a NaN residual leaves u
          float x[2], y[2];
          bool num[2];
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const float rh = k ? hi(rho) : lo(rho), upk_ = k ? hi(up) : lo(up), ltk = k ? hi(lt) : lo(lt);
            const bool in = fabsf(rh) <= upk_;
            num[k] = in || fabsf(rh) > upk_;
            const float away = __uint_as_float(__float_as_uint(ltk) ^ (~__float_as_uint(rh) & 0x80000000u));
            x[k] = in ? -rh : away;
            y[k] = in ? (k ? hi(riu) : lo(riu)) : (k ? hi(iu) : lo(iu));
          }
          const f2 d = fma(pk(x[0], x[1]), pk(y[0], y[1]), dun);
          un = add(U, pk(num[0] ? lo(d) : 0.0f, num[1] ? hi(d) : 0.0f));
        }
        // ---- primal step --------------------------------------------------------------
        const f2 gx = fma(al1, tpx, mul(al0, add(sub(qx, qxw), dqz)));
        const f2 gy = fma(al1, tpy, mul(al0, add(sub(qw, qww), dqy)));
        const f2 vx = fma(mul(tau, rr.x), gx, VX);
        const f2 vy = fma(mul(tau, rr.y), gy, VY);
        f2 us = fma(mu, sub(un, UB), un);
        const f2 vsx = fma(mu, sub(vx, VX), vx), vsy = fma(mu, sub(vy, VY), vy);
        unsigned vn0 = pack(lo(vsx), lo(vsy)), vn1 = pack(hi(vsx), hi(vsy));
        if (KEEP) {  // unwritten pixels alternate between the two ping-pong buffers' values
          un = pk(o0 ? lo(un) : ub0, o1 ? hi(un) : ub1);
          us = pk(o0 ? lo(us) : lo(U), o1 ? hi(us) : hi(U));
          vn0 = o0 ? vn0 : pa;
          vn1 = o1 ? vn1 : pb;
          pn0 = o0 ? pn0 : v[r];
          pn1 = o1 ? pn1 : v[r + 1];
        } else if (EDGE && !MASKED) {  // outside the circle
          un = pk(o0 ? lo(un) : 0.f, o1 ? hi(un) : 0.f);
          us = pk(o0 ? lo(us) : 0.f, o1 ? hi(us) : 0.f);
          vn0 = o0 ? vn0 : 0u;
          vn1 = o1 ? vn1 : 0u;
        }
        u[i] = un;
        ub[i] = us;
        v[r] = vn0;
        v[r + 1] = vn1;
        if constexpr (kSharedPQ) {
          sh.p[is][lane] = make_uint2(pn0, pn1);
        } else {
          p[r + 1] = pn0;
          p[r + 2] = pn1;
        }
        tpy_n = hi(tyo);
        qz_n = hi(qz);
        qy_n = hi(qy);
        vc = vd;
      }
      if constexpr (kTall) {
#pragma unroll
        for (int i = 0; i < kPairs; i++) {
          roll(u, i, 1);
          roll(ub, i, 1);
          roll(v, 2 * i, 2);
          roll(v, 2 * i + 1, 2);
        }
        E.x >>= 2 * kPairs;
        E.y >>= 2 * kPairs;
        E.on >>= 2 * kPairs;
        tp_rows >>= 2 * kPairs;
        if (!kStream) tp_out += 2 * kPairs * s;
      }
    }
  }
};

// Float storage: the operations of the drop-in kernels in their order, rows in pairs as above.
// PLAIN: quotients and roots by the plain operators.
template <bool MASKED, int R>
struct ResState<MASKED, float, R> {
  typedef ResShared<float, R> Sh;
  typedef x2::f2 f2;
  f2 u[R / 2], ub[R / 2], vx[R / 2], vy[R / 2];

  static __device__ __forceinline__ float& el(float4& v, int j) { return reinterpret_cast<float*>(&v)[j]; }
  static __device__ __forceinline__ float el(const float4& v, int j) { return reinterpret_cast<const float*>(&v)[j]; }

  __device__ __forceinline__ void clear(Sh& sh, int lane) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < R / 2; i++) sh.p[i][lane] = sh.qxy[i][lane] = sh.qzw[i][lane] = z;
    sh.qtop[lane] = z;
    sh.ptop[lane] = make_float2(0.f, 0.f);
  }
  // What keeps the squared norms finite, which the exact roots ask for: a level's values are at most
  // kMost before the first iteration, an iteration moves them by kRate at most (tau <= 1: the host
  // sees to it), so that after kResMaxIters they are below 2^30, and a dual step adds below 2^60
  // (sigma <= 2^14).  A pixel beyond any of it asks for the plain operators.
  static constexpr float kMost = 0x1p24f, kMostTp = 16.0f, kRate = 0x1p20f;
  static __device__ __forceinline__ bool beyond(float v) { return !(fabsf(v) <= kMost); }
  // in the range of the exact quotients (Iu, whose dividends are of any size: 2^-64 to 2^32; a residual that
  // takes the Newton step is then below 2^52, since lambda |Iu| <= kRate eta_u)
  static __device__ __forceinline__ bool ranged(float b) { return fabsf(b) >= 0x1p-100f && fabsf(b) <= 0x1p100f; }
  struct Pixel {
    float a, b, c, iu, iz, u, ub;
    float2 tp, v;
  };
  static __device__ __forceinline__ Pixel fetch(const IterPair& P, int r, bool in, bool kept, int pos) {
    Pixel x{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (in) {
      x.a = P.a[pos];
      x.b = P.b[pos];
      x.c = P.c[pos];
    }
    if (kept) x.tp = P.Tp[pos];
    if (r < 0) return x;
    if (in) {
      x.iu = P.Iu[pos];
      x.iz = P.Iz[pos];
      x.u = kept ? P.u_s[pos] : P.u[pos];
      x.ub = P.u_[pos];
    }
    if (kept) x.v = ((const float2*)P.v_s)[pos];
    return x;
  }
  // returns whether the pixel asks for the plain operators
  __device__ __forceinline__ bool set_row(Sh& sh, int lane, const IterPair& P, int r, bool in, bool kept, Pixel x,
                                          unsigned code, unsigned east, unsigned south) {
    bool plain = false;
    if (in && r >= 0 && (code & kOn)) {
      const float eu = etau_math(x.a, x.b, x.c, P.alpha1);
      const float e1 = etav1_math(x.b, x.c, P.alpha0, P.alpha1), e2 = etav2_math(x.a, x.c, P.alpha0, P.alpha1);
      plain = !((eu == 0.0f || ranged(eu)) && ranged(e1) && ranged(e2) &&
                (x.iu == 0.0f || (fabsf(x.iu) >= 0x1p-64f && fabsf(x.iu) <= 0x1p32f)));
      const float m = fmaxf(fmaxf(fabsf(x.a), fabsf(x.b)), fabsf(x.c)), eu1 = eu == 0.0f ? 1.0f : eu;
      const float gv = fabsf(P.alpha1) * m + 4.0f * fabsf(P.alpha0);
      plain = plain || !(m <= 0x1p8f && gv <= 0x1p14f && P.lambda * fabsf(x.iu) <= kRate * eu1 &&
                         4.0f * fmaxf(m, kMostTp) <= kRate * eu1 && gv <= kRate * e1 && gv <= kRate * e2);
    }
    if (kept) {
      // read by the right / lower neighbour only where that one's other side is off too
      x.a = (east & kOn) && !(east & kR) ? x.tp.x : 0.f;
      x.b = (south & kOn) && !(south & kD) ? x.tp.y : 0.f;
      plain = plain || !(fabsf(x.a) <= kMostTp) || !(fabsf(x.b) <= kMostTp);
    }
    if (r < 0) {
      sh.top[lane] = make_float4(x.a, x.b, x.c, 0.f);
      return plain;
    }
    const int i = r >> 1, k = r & 1;
    el(sh.ab[i][lane], k) = x.a;
    el(sh.ab[i][lane], 2 + k) = x.b;
    el(sh.ci[i][lane], k) = x.c;
    el(sh.ci[i][lane], 2 + k) = x.iu;
    reinterpret_cast<float*>(&sh.iz[i][lane])[k] = x.iz;
    plain = plain || beyond(x.u) || beyond(x.ub);
    if (kept) {
      plain = plain || beyond(x.v.x) || beyond(x.v.y);
      el(sh.p[i][lane], k) = x.v.x;
      el(sh.p[i][lane], 2 + k) = x.v.y;
    }
    u[i] = k ? x2::pk(lo(u[i]), x.u) : x2::pk(x.u, 0.f);
    ub[i] = k ? x2::pk(lo(ub[i]), x.ub) : x2::pk(x.ub, 0.f);
    vx[i] = vy[i] = x2::pk(0.f, 0.f);
    return plain;
  }
  static __device__ __forceinline__ float of(f2 v, int r) { return r & 1 ? hi(v) : lo(v); }
  __device__ __forceinline__ float u_of(int r) const { return of(u[r >> 1], r); }
  __device__ __forceinline__ float ub_of(int r) const { return of(ub[r >> 1], r); }
  __device__ __forceinline__ float2 v_of(int r) const { return make_float2(of(vx[r >> 1], r), of(vy[r >> 1], r)); }
  __device__ __forceinline__ uint4 word(int r, unsigned tag) const {
    const float2 v = v_of(r);
    return make_uint4(__float_as_uint(ub_of(r)), __float_as_uint(v.x), __float_as_uint(v.y), tag);
  }
  static __device__ __forceinline__ void put_col(Sh& sh, int side, int r, uint4 w) { sh.col[side][r] = w; }
  __device__ __forceinline__ void take_col(const uint4* col) {
#pragma unroll
    for (int i = 0; i < R / 2; i++) {
      const uint4 w0 = col[2 * i], w1 = col[2 * i + 1];
      ub[i] = x2::pk(__uint_as_float(w0.x), __uint_as_float(w1.x));
      vx[i] = x2::pk(__uint_as_float(w0.y), __uint_as_float(w1.y));
      vy[i] = x2::pk(__uint_as_float(w0.z), __uint_as_float(w1.z));
    }
  }
  __device__ __forceinline__ void store_pq(const Sh& sh, int lane, int r, void* po, void* qo, int pos) const {
    const int i = r >> 1, k = r & 1;
    ((float2*)po)[pos] = make_float2(el(sh.p[i][lane], k), el(sh.p[i][lane], 2 + k));
    ((float4*)qo)[pos] = make_float4(el(sh.qxy[i][lane], k), el(sh.qxy[i][lane], 2 + k), el(sh.qzw[i][lane], k),
                                     el(sh.qzw[i][lane], 2 + k));
  }

  // p and q projected: |.| is divided out where it is above 1
  template <bool PLAIN>
  static __device__ __forceinline__ void project(f2 n2, f2& a, f2& b) {
    using namespace x2;
    if (PLAIN) {
      const float r0 = sqrtf(lo(n2)), r1 = sqrtf(hi(n2));
      const bool k0 = r0 <= 1.0f, k1 = r1 <= 1.0f;
      a = pk(k0 ? lo(a) : lo(a) / r0, k1 ? hi(a) : hi(a) / r1);
      b = pk(k0 ? lo(b) : lo(b) / r0, k1 ? hi(b) : hi(b) / r1);
    } else {
      f2 s, y;
      exact::root(pk(max1(lo(n2)), max1(hi(n2))), s, y);
      const exact::Divisor d(s, y);
      a = exact::quot(a, d);
      b = exact::quot(b, d);
    }
  }
  // max(v, 1); a NaN stays
  static __device__ __forceinline__ float max1(float v) {
    float r;
    asm("max.NaN.f32 %0, %1, 0f3F800000;" : "=f"(r) : "f"(v));
    return r;
  }
  template <bool PLAIN>
  static __device__ __forceinline__ void project4(f2 m2, f2& x, f2& y_, f2& z, f2& w) {
    using namespace x2;
    if (PLAIN) {
      f2 a = x, b = y_;
      project<true>(m2, a, b);
      x = a;
      y_ = b;
      a = z;
      b = w;
      project<true>(m2, a, b);
      z = a;
      w = b;
    } else {
      f2 s, y;
      exact::root(pk(max1(lo(m2)), max1(hi(m2))), s, y);
      const exact::Divisor d(s, y);
      x = exact::quot(x, d);
      y_ = exact::quot(y_, d);
      z = exact::quot(z, d);
      w = exact::quot(w, d);
    }
  }
  // tau / eta; eta = 0 takes tau itself
  template <bool PLAIN>
  static __device__ __forceinline__ f2 step_of(f2 tau, f2 eta) {
    if (PLAIN)
      return x2::pk(lo(eta) == 0.0f ? lo(tau) : lo(tau) / lo(eta), hi(eta) == 0.0f ? hi(tau) : hi(tau) / hi(eta));
    return exact::quot(tau, eta, exact::recip(eta));
  }

  template <int KIND>
  __device__ __forceinline__ void iterate(Sh& sh, const ResArgs& A, int lane, const ResStep& S, const ResEdge& E,
                                          uint4 wn, uint4 ws, float2* tp_out, int s, unsigned tp_rows) {
    using namespace x2;
    constexpr bool PLAIN = KIND == kResPlain;
    constexpr bool EDGE = KIND != kResInner;
    constexpr bool KEEP = MASKED && (KIND == kResKeep || PLAIN);
    const f2 sp = pk(S.sp.x, S.sp.y), sq = pk(S.sq.x, S.sq.y), tau = pk(S.tau.x, S.tau.y), mu = pk(S.mu.x, S.mu.y);
    const f2 lam = both(A.P.lambda), al0 = both(A.P.alpha0), al1 = both(A.P.alpha1);
    const f2 a1s = both(A.P.alpha1 * A.P.alpha1), a0s4 = both(4 * A.P.alpha0 * A.P.alpha0);
    // A product that is added to something else.  ptxas contracts mul.rn.f32x2 and add.rn.f32x2 into
    // one fma (CUDA 12.9, -fmad=false notwithstanding); a fused multiply-add of -0, which it
    // cannot see, rounds the product alone.
    const f2 nz = pk(A.minus_zero.x, A.minus_zero.y);
    auto prod = [nz](f2 x, f2 y) { return fma(x, y, nz); };
    auto bit = [](unsigned m, int r) { return (m >> (r + 1)) & 1u; };
    auto pair = [](const float4& v) { return *reinterpret_cast<const ulonglong2*>(&v); };
    float tpy_n, qz_n, qy_n, du_n;
    float2 dv_n;
    {
      const float4 ca = sh.top[lane];
      const float ubc = __uint_as_float(wn.x);
      const float2 vp = make_float2(__uint_as_float(wn.y), __uint_as_float(wn.z));
      float dux = __shfl_down_sync(kFull, ubc, 1) - ubc;
      float2 dvx = make_float2(__shfl_down_sync(kFull, vp.x, 1) - vp.x, __shfl_down_sync(kFull, vp.y, 1) - vp.y);
      du_n = lo(ub[0]) - ubc;
      dv_n = make_float2(lo(vx[0]) - vp.x, lo(vy[0]) - vp.y);
      if (EDGE) {
        const float wu = __shfl_up_sync(kFull, dux, 1);
        const float2 wv = make_float2(__shfl_up_sync(kFull, dvx.x, 1), __shfl_up_sync(kFull, dvx.y, 1));
        const bool r0 = bit(E.x, -1);
        dux = r0 ? dux : wu;
        dvx = make_float2(r0 ? dvx.x : wv.x, r0 ? dvx.y : wv.y);
      }
      const float gx = dux - vp.x, gy = du_n - vp.y;
      float2 p = sh.ptop[lane];
      float4 q = sh.qtop[lane];
      const float dtx = ca.x * gx + ca.z * gy, dty = ca.z * gx + ca.y * gy;
      // both p lanes and the norms of p and q side by side
      f2 pp = pk(p.x + S.sp.x * dtx, p.y + S.sp.x * dty);
      f2 qa = pk(q.x + S.sq.x * dvx.x, q.y + S.sq.x * dv_n.y), qb = pk(q.z + S.sq.x * dv_n.x, q.w + S.sq.x * dvx.y);
      const f2 p2 = prod(pp, pp), qa2 = prod(qa, qa), qb2 = prod(qb, qb);
      const float n2 = lo(p2) + hi(p2), m2 = lo(qa2) + hi(qa2) + lo(qb2) + hi(qb2);
      if (PLAIN) {
        const float rp = sqrtf(n2), rq = sqrtf(m2);
        if (!(rp <= 1.0f)) pp = pk(lo(pp) / rp, hi(pp) / rp);
        if (!(rq <= 1.0f)) {
          qa = pk(lo(qa) / rq, hi(qa) / rq);
          qb = pk(lo(qb) / rq, hi(qb) / rq);
        }
      } else {
        f2 sr, y;
        exact::root(pk(max1(n2), max1(m2)), sr, y);
        const exact::Divisor d(sr, y);
        const exact::Divisor dp = d.low(), dq = d.high();
        pp = exact::quot(pp, dp);
        qa = exact::quot(qa, dq);
        qb = exact::quot(qb, dq);
      }
      p = upk(pp);
      sh.ptop[lane] = p;
      sh.qtop[lane] = make_float4(lo(qa), hi(qa), lo(qb), hi(qb));
      tpy_n = ca.z * p.x + ca.y * p.y;
      qz_n = lo(qb);
      qy_n = hi(qa);
      if (EDGE) {
        const bool d0 = bit(E.y, -1);
        const bool o0 = MASKED ? d0 : bit(E.on, -1);
        tpy_n = o0 ? tpy_n : KEEP && !bit(E.on, -1) ? ca.y : -0.0f;
        qz_n = d0 ? qz_n : 0.f;
        qy_n = d0 ? qy_n : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < R / 2; i++) {
      const int r = 2 * i;
      const int in_ = i + 1 < R / 2 ? i + 1 : 0;
      const f2 UB = ub[i], VX = vx[i], VY = vy[i];
      const float ub0 = lo(UB), ub1 = hi(UB);
      const float ubd = i + 1 < R / 2 ? lo(ub[in_]) : __uint_as_float(ws.x);
      const float vxd = i + 1 < R / 2 ? lo(vx[in_]) : __uint_as_float(ws.y);
      const float vyd = i + 1 < R / 2 ? lo(vy[in_]) : __uint_as_float(ws.z);
      const ulonglong2 ab = pair(sh.ab[i][lane]), ci = pair(sh.ci[i][lane]);
      // ---- differences of u-bar and v-bar to the east and to the south -----------------
      f2 dux = sub(pk(__shfl_down_sync(kFull, ub0, 1), __shfl_down_sync(kFull, ub1, 1)), UB);
      f2 dxx = sub(pk(__shfl_down_sync(kFull, lo(VX), 1), __shfl_down_sync(kFull, hi(VX), 1)), VX);
      f2 dxy = sub(pk(__shfl_down_sync(kFull, lo(VY), 1), __shfl_down_sync(kFull, hi(VY), 1)), VY);
      const float du0 = ub1 - ub0, du1 = ubd - ub1;
      const float2 dv0 = make_float2(hi(VX) - lo(VX), hi(VY) - lo(VY)), dv1 = make_float2(vxd - hi(VX), vyd - hi(VY));
      f2 duy = pk(du0, du1), dyx = pk(dv0.x, dv1.x), dyy = pk(dv0.y, dv1.y);
      bool r0 = true, r1 = true, d0 = true, d1 = true;
      if (EDGE) {
        r0 = bit(E.x, r);
        r1 = bit(E.x, r + 1);
        d0 = bit(E.y, r);
        d1 = bit(E.y, r + 1);
        const float wu0 = __shfl_up_sync(kFull, lo(dux), 1), wu1 = __shfl_up_sync(kFull, hi(dux), 1);
        const float wx0 = __shfl_up_sync(kFull, lo(dxx), 1), wx1 = __shfl_up_sync(kFull, hi(dxx), 1);
        const float wy0 = __shfl_up_sync(kFull, lo(dxy), 1), wy1 = __shfl_up_sync(kFull, hi(dxy), 1);
        dux = pk(r0 ? lo(dux) : wu0, r1 ? hi(dux) : wu1);
        dxx = pk(r0 ? lo(dxx) : wx0, r1 ? hi(dxx) : wx1);
        dxy = pk(r0 ? lo(dxy) : wy0, r1 ? hi(dxy) : wy1);
        duy = pk(d0 ? du0 : du_n, d1 ? du1 : du0);
        dyx = pk(d0 ? dv0.x : dv_n.x, d1 ? dv1.x : dv0.x);
        dyy = pk(d0 ? dv0.y : dv_n.y, d1 ? dv1.y : dv0.y);
        du_n = du1;
        dv_n = dv1;
      }
      // ---- dual step ------------------------------------------------------------------
      const f2 a = ab.x, b = ab.y, c = ci.x, iu = ci.y;
      const f2 ux = sub(dux, VX), uy = sub(duy, VY);
      const ulonglong2 p0 = pair(sh.p[i][lane]), qa = pair(sh.qxy[i][lane]), qb = pair(sh.qzw[i][lane]);
      f2 px = add(p0.x, prod(sp, add(prod(a, ux), prod(c, uy))));
      f2 py = add(p0.y, prod(sp, add(prod(c, ux), prod(b, uy))));
      project<PLAIN>(add(prod(px, px), prod(py, py)), px, py);
      f2 qx = add(qa.x, prod(sq, dxx));
      f2 qy = add(qa.y, prod(sq, dyy));
      f2 qz = add(qb.x, prod(sq, dyx));
      f2 qw = add(qb.y, prod(sq, dxy));
      project4<PLAIN>(add(add(add(prod(qx, qx), prod(qy, qy)), prod(qz, qz)), prod(qw, qw)), qx, qy, qz, qw);
      const f2 tpx = add(prod(a, px), prod(c, py)), tpy = add(prod(c, px), prod(b, py));
      f2 pnx = px, pny = py;
      *reinterpret_cast<ulonglong2*>(&sh.qxy[i][lane]) = make_ulonglong2(qx, qy);
      *reinterpret_cast<ulonglong2*>(&sh.qzw[i][lane]) = make_ulonglong2(qz, qw);
      if (!MASKED && EDGE) {  // outside the circle p = 0: T p = T 0
        const float2 z = make_float2(0.f, 0.f);
        if ((tp_rows >> r) & 1u) tp_out[r * s] = bit(E.on, r) ? make_float2(lo(tpx), lo(tpy)) : tp_math(lo(a), lo(b), lo(c), z);
        if ((tp_rows >> (r + 1)) & 1u)
          tp_out[(r + 1) * s] = bit(E.on, r + 1) ? make_float2(hi(tpx), hi(tpy)) : tp_math(hi(a), hi(b), hi(c), z);
      } else {
        if ((tp_rows >> r) & 1u) tp_out[r * s] = make_float2(lo(tpx), lo(tpy));
        if ((tp_rows >> (r + 1)) & 1u) tp_out[(r + 1) * s] = make_float2(hi(tpx), hi(tpy));
      }
      // ---- threshold step -----------------------------------------------------------
      f2 txo = tpx, tyo = tpy;  // as counted for this pixel and its right / lower neighbour
      bool o0 = true, o1 = true;
      if (EDGE) {
        if (KEEP || !MASKED) {
          o0 = bit(E.on, r);
          o1 = bit(E.on, r + 1);
        }
        const float zx0 = KEEP && !o0 ? lo(a) : -0.0f, zx1 = KEEP && !o1 ? hi(a) : -0.0f;
        const float zy0 = KEEP && !o0 ? lo(b) : -0.0f, zy1 = KEEP && !o1 ? hi(b) : -0.0f;
        // the plain form takes the difference at the last row and column too
        txo = pk((MASKED ? r0 : o0) ? lo(tpx) : zx0, (MASKED ? r1 : o1) ? hi(tpx) : zx1);
        tyo = pk((MASKED ? d0 : o0) ? lo(tpy) : zy0, (MASKED ? d1 : o1) ? hi(tpy) : zy1);
        qx = pk(r0 ? lo(qx) : 0.f, r1 ? hi(qx) : 0.f);
        qw = pk(r0 ? lo(qw) : 0.f, r1 ? hi(qw) : 0.f);
        qz = pk(d0 ? lo(qz) : 0.f, d1 ? hi(qz) : 0.f);
        qy = pk(d0 ? lo(qy) : 0.f, d1 ? hi(qy) : 0.f);
      }
      const f2 tpw = pk(__shfl_up_sync(kFull, lo(txo), 1), __shfl_up_sync(kFull, hi(txo), 1));
      const f2 qxw = pk(__shfl_up_sync(kFull, lo(qx), 1), __shfl_up_sync(kFull, hi(qx), 1));
      const f2 qww = pk(__shfl_up_sync(kFull, lo(qw), 1), __shfl_up_sync(kFull, hi(qw), 1));
      const f2 dy = pk(lo(tyo) - tpy_n, hi(tyo) - lo(tyo));
      const f2 dqz = pk(lo(qz) - qz_n, hi(qz) - lo(qz)), dqy = pk(lo(qy) - qy_n, hi(qy) - lo(qy));
      const f2 aa = prod(a, a), bb = prod(b, b), cc = prod(c, c), ac = add(a, c), bc = add(b, c);
      const f2 eu = prod(add(add(add(add(aa, bb), add(cc, cc)), prod(ac, ac)), prod(bc, bc)), a1s);
      // (the reference leaves the tensor zero beyond its launch grid: eta_u = 0 there, tau / 1 = tau)
      const f2 te = step_of<PLAIN>(tau, PLAIN ? eu : pk(lo(eu) == 0.0f ? 1.0f : lo(eu), hi(eu) == 0.0f ? 1.0f : hi(eu)));
      const f2 U = u[i];
      const f2 dun = sub(add(UB, prod(te, add(sub(txo, tpw), dy))), U);
      const f2 rho = add(prod(iu, dun), *reinterpret_cast<const f2*>(&sh.iz[i][lane]));
      const f2 lt = prod(lam, te);
      const f2 up = prod(lt, prod(iu, iu)), far = prod(lt, iu);
      f2 newton;
      if (PLAIN) newton = pk(lo(rho) / lo(iu), hi(rho) / hi(iu));
      else newton = exact::quot(rho, exact::Divisor(iu, exact::recip(iu)));
      f2 un;
      {
        // |rho| <= upper: the Newton step (none where Iu = 0); beyond it a step of lambda tau Iu / eta_u
        // against the sign of rho (lambda >= 0); a NaN residual leaves u
        float t[2];
        bool num[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const float rh = k ? hi(rho) : lo(rho), upk_ = k ? hi(up) : lo(up);
          const bool in = fabsf(rh) <= upk_;
          num[k] = in || fabsf(rh) > upk_;
          const float away = __uint_as_float(__float_as_uint(k ? hi(far) : lo(far)) ^ (__float_as_uint(rh) & 0x80000000u));
          const float nk = (k ? hi(iu) : lo(iu)) == 0.0f ? 0.0f : k ? hi(newton) : lo(newton);
          t[k] = in ? nk : away;
        }
        const f2 d = sub(dun, pk(t[0], t[1]));
        un = add(U, pk(num[0] ? lo(d) : 0.0f, num[1] ? hi(d) : 0.0f));
      }
      // ---- primal step --------------------------------------------------------------
      const f2 e1 = add(prod(a1s, add(bb, cc)), a0s4), e2 = add(prod(a1s, add(aa, cc)), a0s4);
      const f2 gx = add(prod(al1, tpx), prod(al0, add(sub(qx, qxw), dqz)));
      const f2 gy = add(prod(al1, tpy), prod(al0, add(sub(qw, qww), dqy)));
      f2 t1 = step_of<PLAIN>(tau, e1);
      if (PLAIN)  // eta_v2 = 0: updatePrimalVariables.cu:103-105 writes .x again, .y keeps its value
        t1 = pk(lo(e2) == 0.0f ? lo(tau) : lo(t1), hi(e2) == 0.0f ? hi(tau) : hi(t1));
      const f2 wx = add(VX, prod(t1, gx));
      f2 wy = add(VY, prod(step_of<PLAIN>(tau, e2), gy));
      if (PLAIN) wy = pk(lo(e2) == 0.0f ? lo(VY) : lo(wy), hi(e2) == 0.0f ? hi(VY) : hi(wy));
      f2 us = add(un, prod(mu, sub(un, UB)));
      f2 vsx = add(wx, prod(mu, sub(wx, VX))), vsy = add(wy, prod(mu, sub(wy, VY)));
      if (KEEP) {  // unwritten pixels alternate between the two ping-pong buffers' values
        un = pk(o0 ? lo(un) : ub0, o1 ? hi(un) : ub1);
        us = pk(o0 ? lo(us) : lo(U), o1 ? hi(us) : hi(U));
        vsx = pk(o0 ? lo(vsx) : lo(p0.x), o1 ? hi(vsx) : hi(p0.x));
        vsy = pk(o0 ? lo(vsy) : lo(p0.y), o1 ? hi(vsy) : hi(p0.y));
        pnx = pk(o0 ? lo(px) : lo(VX), o1 ? hi(px) : hi(VX));
        pny = pk(o0 ? lo(py) : lo(VY), o1 ? hi(py) : hi(VY));
      } else if (EDGE && !MASKED) {  // outside the circle
        un = pk(o0 ? lo(un) : 0.f, o1 ? hi(un) : 0.f);
        us = pk(o0 ? lo(us) : 0.f, o1 ? hi(us) : 0.f);
        vsx = pk(o0 ? lo(vsx) : 0.f, o1 ? hi(vsx) : 0.f);
        vsy = pk(o0 ? lo(vsy) : 0.f, o1 ? hi(vsy) : 0.f);
      }
      *reinterpret_cast<ulonglong2*>(&sh.p[i][lane]) = make_ulonglong2(pnx, pny);
      u[i] = un;
      ub[i] = us;
      vx[i] = vsx;
      vy[i] = vsy;
      tpy_n = hi(tyo);
      qz_n = hi(qz);
      qy_n = hi(qy);
    }
  }
};

// Publishes a tile's border u-bar and v-bar as tag `tag` to its words `out`.
template <int R, class State>
__device__ __forceinline__ void publish(const State& st, uint4* out, int lane, unsigned tag) {
  if (lane >= 1 && lane <= kResCols) {
    st_word(out + lane, st.word(0, tag));
    st_word(out + 32 + lane, st.word(R - 1, tag));
  }
  if (lane == 1 || lane == kResCols) {
    uint4* c = out + 64 + (lane == 1 ? 0 : R);
#pragma unroll
    for (int r = 0; r < R; r++) st_word(c + r, st.word(r, tag));
  }
}

}  // namespace

// One warp's tile.
template <bool MASKED, class ST, int R>
struct ResWarp {
  typedef ResShared<ST, R> Sh;
  typedef typename Store2<ST>::T2 T2;
  typedef typename Store2<ST>::T4 T4;
  static constexpr int kSlots = 64 + 2 * R;
  static constexpr bool kPlain = std::is_same<ST, float>::value;
  // Code of its own for the tiles without edge rules.  Eight rows of the float form are 30 KB a
  // kind; with two kinds in turn on an SM the rarer one ran from the instruction cache's misses
  // (848 x 800: 5900 cycles a tile without edge rules, 8700 with, 7.1 us per iteration; one kind 6.16).
  static constexpr bool kInner = !kPlain || R < 8;
  static constexpr int kAtOnce = 3;  // rows fetched before the first is used
  typedef ResState<MASKED, ST, R> State;
  State s;

  // Loads tile t: its coefficients, codes and state before the first iteration.  All the codes are asked
  // for at once, and the values of a few rows at a time, so that a tile waits for memory four or five
  // times and not for every row anew (848 x 800 float: 2 us less a launch, 33 of a solve's 2230).
  __device__ __forceinline__ ResEdge load(Sh& sh, const ResArgs& A, int lane, int t, const ResTile& T) {
    const IterPair& P = A.P;
    const int x = T.x0 - 1 + lane, y0 = T.y0;
    const bool x_in = x >= 0 && x < P.w;
    ResEdge e{0u, 0u, 0u};
    bool plain = false;
    auto inside = [&](int r) { return x_in && y0 + r >= 0 && y0 + r < P.h; };
    unsigned codes[R + 1];
#pragma unroll
    for (int r = -1; r < R; r++) codes[r + 1] = inside(r) ? P.code[x + (y0 + r) * P.s] : 0u;
    s.clear(sh, lane);
#pragma unroll
    for (int first = -1; first < R; first += kAtOnce) {
      typename State::Pixel px[kAtOnce];
      unsigned east[kAtOnce], south[kAtOnce];
#pragma unroll
      for (int k = 0; k < kAtOnce; k++) {
        const int r = first + k, pos = x + (y0 + r) * P.s;
        if (r >= R) break;
        unsigned& code = codes[r + 1];
        const bool in = inside(r), kept = MASKED && in && !(code & kOn);
        px[k] = State::fetch(P, r, in, kept, pos);
        east[k] = kept && (code & kR) ? P.code[pos + 1] : 0u;
        south[k] = kept && (code & kD) ? P.code[pos + P.s] : 0u;
        if (!MASKED && in) {
          code &= kOn;
          code |= (x + 1 < P.w ? kR : 0) | (x >= 1 ? kL : 0) | (y0 + r + 1 < P.h ? kD : 0) | (y0 + r >= 1 ? kU : 0);
        }
      }
#pragma unroll
      for (int k = 0; k < kAtOnce; k++) {
        const int r = first + k;
        if (r >= R) break;
        const unsigned code = codes[r + 1], b = 1u << (r + 1);
        const bool in = inside(r), kept = MASKED && in && !(code & kOn);
        plain = s.set_row(sh, lane, P, r, in, kept, px[k], code, east[k], south[k]) || plain;
        if (code & kOn) {
          e.on |= b;
          if (code & kR) e.x |= b;
          if (code & kD) e.y |= b;
        }
      }
    }
    sh.k.edge[lane] = make_uint2(e.y, e.on);
    plain = __any_sync(kFull, plain);
    if (lane == 0) {
      sh.k.kind = plain ? kResPlain : T.kind;
      sh.k.t = t;
    }
    return e;
  }

  // Where this lane finds its neighbours' words.  A missing neighbour is replaced by this tile itself:
  // the tags come, the values are not used.  Lanes 0 .. R-1 fetch the west column, lanes 16 .. 16 + R-1
  // the east one.
  __device__ __forceinline__ void link(Sh& sh, int lane, const ResTile& T, const ResEdge& e) {
    const int tn = lane == 0 ? T.nb[4] : lane == 31 ? T.nb[5] : T.nb[0];
    const int ts = lane == 0 ? T.nb[6] : lane == 31 ? T.nb[7] : T.nb[1];
    const int col = lane == 0 ? kResCols : lane == 31 ? 1 : lane;
    const int side = lane >> 4, row = lane & 15;
    sh.k.at[lane] = make_uint4((unsigned)(tn * kSlots + 32 + col), (unsigned)(ts * kSlots + col),
                               (unsigned)(T.nb[side ? 3 : 2] * kSlots + 64 + (side ? 0 : R) + (row < R ? row : 0)), e.x);
    __syncwarp();
  }

  // A tile on the plain operators marks its words, and who takes a marked word changes to them as
  // well: values beyond the exact roots' range travel no faster than the words.
  __device__ __forceinline__ unsigned flag(const Sh& sh) const {
    return kPlain && sh.k.kind == kResPlain ? kResBeyond : 0u;
  }
  __device__ __forceinline__ void meet(Sh& sh, unsigned marks) {
    if (marks & kResBeyond) sh.k.kind = kResPlain;
  }

  // One iteration.  Returns false once a wait ran out.
  __device__ __forceinline__ bool step(Sh& sh, const ResArgs& A, int lane, int j,
                                       unsigned epoch, bool waiting) {
    const uint4 o = sh.k.at[lane];
    const unsigned ring = (unsigned)A.ntiles * kSlots;
    const uint4* const base = A.exch + (size_t)(j & (kResRing - 1)) * ring;
    const unsigned tag = epoch | (unsigned)j;
    uint4 wn, ws, wc;
    // The words cannot be there yet: the neighbours published them when this tile did its own.  A first
    // look too early costs a whole round trip (848 x 800 levels: 3.95 / 1.86 us with none of this pause,
    // 3.92 / 1.83 with it, 640 x 480 2.45 / 1.63 and 2.40 / 1.55).
    for (const unsigned c = clock(); (unsigned)clock() - c < 250u;) {
    }
    for (int polls = 0;; polls++) {
      wn = ld_word(base + o.x);
      ws = ld_word(base + o.y);
      wc = ld_word(base + o.z);
      const unsigned other = (wn.w ^ tag) | (ws.w ^ tag) | (wc.w ^ tag);
      if (__all_sync(kFull, (kPlain ? other & ~kResBeyond : other) == 0) || !waiting) break;
      if (polls >= kResLooks) {
        waiting = false;
        if (lane == 0) atomicAdd(&A.ctl->done, kResGaveUp);
        break;
      }
    }
    const int side = lane >> 4, row = lane & 15;
    if (row < R) s.put_col(sh, side, row, wc);
    if (kPlain) meet(sh, wn.w | ws.w | wc.w);
    __syncwarp();
    if (lane == 0 || lane == 31) s.take_col(sh.col[side]);
    __syncwarp();
    iterate(sh, A, lane, j, o.w, wn, ws);
    if (j + 1 < A.n)
      publish<R>(s, A.exch + (size_t)((j + 1) & (kResRing - 1)) * ring + (unsigned)(sh.k.t * kSlots), lane,
                 (tag + 1) | flag(sh));
    return waiting;
  }

  // The state's iteration j for the tile's kind; the halo columns are in place.
  __device__ __forceinline__ void iterate(Sh& sh, const ResArgs& A, int lane, int j, unsigned ex, uint4 wn, uint4 ws) {
    const IterPair& P = A.P;
    const bool last = j + 1 == A.n;
    const uint2 ek = sh.k.edge[lane];
    const ResEdge E{ex, ek.x, ek.y};
    const int kind = sh.k.kind;
    float2* tp_out = nullptr;
    unsigned tp_rows = 0u;
    if (last) {
      int pos0;
      tp_rows = owned(sh, A, lane, pos0);
      tp_out = P.Tp + pos0;
    }
    if (kInner && kind == kResInner) s.template iterate<kInner ? kResInner : kResEdge>(sh, A, lane, A.step[j], E, wn, ws, tp_out, P.s, tp_rows);
    else if (kind <= kResEdge) s.template iterate<kResEdge>(sh, A, lane, A.step[j], E, wn, ws, tp_out, P.s, tp_rows);
    else if (kPlain && kind == kResPlain)
      s.template iterate<kPlain ? kResPlain : kResEdge>(sh, A, lane, A.step[j], E, wn, ws, tp_out, P.s, tp_rows);
    else if constexpr (MASKED) s.template iterate<kResKeep>(sh, A, lane, A.step[j], E, wn, ws, tp_out, P.s, tp_rows);
  }

  // The rows of this lane's column that the tile owns and the iterations write (bit r), and the
  // flat position of row 0.
  __device__ __forceinline__ unsigned owned(const Sh& sh, const ResArgs& A, int lane, int& pos0) const {
    const ResTile& T = A.tiles[sh.k.t];
    const int x = T.x0 - 1 + lane;
    pos0 = x + T.y0 * A.P.s;
    const int rows = lane >= 1 && lane <= kResCols && x < A.P.w ? min(R, A.P.h - T.y0) : 0;
    const unsigned in = (1u << rows) - 1u;
    return MASKED ? in & (sh.k.edge[lane].y >> 1) : in;
  }

  // Writes the tile's u, u-bar and v-bar: the state current after n iterations (fin), or the one
  // before the last iteration into the other ping-pong buffers.
  __device__ __forceinline__ void store(const Sh& sh, const ResArgs& A, int lane,
                                        bool fin) {
    const IterPair& P = A.P;
    const bool first = (A.n & 1) ^ (fin ? 1 : 0);  // into the launch's input buffers
    float* uo = first ? const_cast<float*>(P.u) : P.us;
    float* ubo = first ? const_cast<float*>(P.u_) : P.u_s;
    T2* vo = (T2*)(first ? const_cast<void*>(P.v_) : P.v_s);
    int pos0;
    const unsigned own = owned(sh, A, lane, pos0);
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (!((own >> r) & 1u)) continue;
      const int pos = pos0 + r * P.s;
      uo[pos] = s.u_of(r);
      ubo[pos] = s.ub_of(r);
      vo[pos] = s.v_of(r);
    }
    if (fin) {
      const int plane = A.p_planes ? (A.n & 1) * P.s * P.h : 0;
      const unsigned on = own & (sh.k.edge[lane].y >> 1);
#pragma unroll
      for (int r = 0; r < R; r++)
        if ((on >> r) & 1u) s.store_pq(sh, lane, r, (T2*)P.p + plane, (T4*)P.q + plane, pos0 + r * P.s);
    }
  }
};

// The plain form's pixels outside the circle in tiles without a pixel to solve.
template <class ST, int R>
__device__ __forceinline__ void res_fill(const ResArgs& A, int warp, int lane) {
  typedef typename Store2<ST>::T2 T2;
  const IterPair& P = A.P;
  const int warps = (int)blockDim.x >> 5, nw = (int)gridDim.x * warps;
  const float2 z = make_float2(0.f, 0.f);
  for (int k = (int)blockIdx.x * warps + warp; k < A.nfill; k += nw) {
    const int2 f = A.fill[k];
    const int x = f.x - 1 + lane;
    if (lane < 1 || lane > kResCols || x >= P.w) continue;
    for (int y = f.y; y < min(f.y + R, P.h); y++) {
      const int pos = x + y * P.s;
      // the buffers current after n iterations and, from two iterations on, the others
      if ((A.n & 1) == 0 || A.n >= 2) {
        const_cast<float*>(P.u)[pos] = 0.f;
        const_cast<float*>(P.u_)[pos] = 0.f;
        Store2<ST>::st2((T2*)const_cast<void*>(P.v_), pos, z);
      }
      P.us[pos] = 0.f;
      P.u_s[pos] = 0.f;
      Store2<ST>::st2((T2*)P.v_s, pos, z);
      P.Tp[pos] = tp_math(P.a[pos], P.b[pos], P.c[pos], z);
    }
  }
}

template <bool MASKED, class ST, int R>
__global__ void __launch_bounds__(32 * kResMostWarps, 1) k_resident(const __grid_constant__ ResArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  ResShared<ST, R>& sh = reinterpret_cast<ResShared<ST, R>*>(smem)[warp];
  // Tiles go round the blocks first, then the warps of a block: every SM, and every scheduler of an
  // SM, has the same number of tiles but for one.
  const int t = (int)blockIdx.x + (int)gridDim.x * warp;
  const unsigned epoch = (*(volatile unsigned*)&A.ctl->epoch + 1u) << 8;

  if (t < A.ntiles) {
    ResWarp<MASKED, ST, R> W;
    const ResTile T = A.tiles[t];
    W.link(sh, lane, T, W.load(sh, A, lane, t, T));
    if (t != A.mute)  // iteration 0's input
      publish<R>(W.s, A.exch + (size_t)t * (64 + 2 * R), lane, epoch | W.flag(sh));
    __syncwarp();
    bool waiting = true;
#pragma unroll 1
    for (int j = 0; j < A.n; j++) {
      waiting = W.step(sh, A, lane, j, epoch, waiting);
      if (j + 2 >= A.n) W.store(sh, A, lane, j + 1 == A.n);
    }
  }
  if (!MASKED) res_fill<ST, R>(A, warp, lane);
  // ---- the last block to end renews the epoch: every block has read it by then --------------
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned done = atomicAdd(&A.ctl->done, 1u);
    if ((done & (kResGaveUp - 1u)) == gridDim.x - 1) {
      A.ctl->done = 0;
      A.ctl->epoch += 1;
      if (done >= kResGaveUp) give_up(A);
    }
  }
}

// ---- small levels: the tiles of one cluster ---------------------------------------------------
// A level of few tiles (res_cluster_tiles) runs on the blocks of one thread-block cluster, whose
// warps store their border straight into their neighbours' shared memory (st.async through
// distributed shared memory, counted on the neighbour's mbarrier).  A level that small is all
// latency: a tile computes for 650 cycles, the way through L2 takes another 1100 to 1500, this one
// about half of that (53 x 50: 1.39 -> 0.90 us per iteration).  Two inboxes, by parity of the
// iteration, for the reason the ring has two.
namespace {

constexpr int kResWaits = 1 << 16;  // after which a wait gives up: some 0.8 s

template <class ST>
struct ResWord;  // u-bar and v-bar of a border pixel
template <>
struct ResWord<__half> {
  typedef uint2 T;
  static __device__ __forceinline__ uint2 of(uint4 w) { return make_uint2(w.x, w.y); }
  static __device__ __forceinline__ uint4 wide(uint2 w) { return make_uint4(w.x, w.y, 0u, 0u); }
};
template <>
struct ResWord<float> {
  typedef uint4 T;
  static __device__ __forceinline__ uint4 of(uint4 w) { return w; }
  static __device__ __forceinline__ uint4 wide(uint4 w) { return w; }
};

template <class ST, int R>
struct ResInbox {
  typename ResWord<ST>::T n[32], s[32], c[2][R];  // the rows above and below, the west and east column
};
template <class ST, int R>
struct ResClusterTile {
  ResShared<ST, R> sh;
  ResInbox<ST, R> in[2];
  // per lane, for slot 0, address and barrier of (its words in the tile below, in the tile above),
  // (in the two diagonal tiles of its side below, above), (in the tile beside); 0: no such tile
  uint4 row[32], diag[32];
  uint2 side[32];
  unsigned long long bar[2];
  int bytes;  // that arrive in an inbox per iteration
  int pad[3];
};

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cl_addr(unsigned local, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async(unsigned to, unsigned bar, uint2 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(to), "r"(v.x),
               "r"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned to, unsigned bar, uint4 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_arm(unsigned bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(1000)  // suspended for a microsecond at most
      : "memory");
  return ok != 0;
}

// A tile's border after k iterations into its neighbours' inboxes.
template <class ST, int R, class State>
__device__ __forceinline__ void push(const State& s, const ResClusterTile<ST, R>& C, int lane, int k, unsigned flag) {
  typedef ResWord<ST> Word;
  const unsigned in = (k & 1) * (unsigned)sizeof(ResInbox<ST, R>), bar = (k & 1) * 8u;
  const auto top = Word::of(s.word(0, flag)), bottom = Word::of(s.word(R - 1, flag));
  const uint4 row = C.row[lane], diag = C.diag[lane];
  const uint2 side = C.side[lane];
  if (row.x) st_async(row.x + in, row.y + bar, bottom);
  if (row.z) st_async(row.z + in, row.w + bar, top);
  if (diag.x) st_async(diag.x + in, diag.y + bar, bottom);
  if (diag.z) st_async(diag.z + in, diag.w + bar, top);
  if (side.x) {
#pragma unroll
    for (int r = 0; r < R; r++)
      st_async(side.x + in + r * (unsigned)sizeof(typename Word::T), side.y + bar, Word::of(s.word(r, flag)));
  }
}

}  // namespace

template <bool MASKED, class ST, int R>
__global__ void __launch_bounds__(512, 1) k_resident_cluster(const __grid_constant__ ResArgs A) {
  typedef ResWord<ST> Word;
  typedef ResClusterTile<ST, R> Tile;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31, ctas = (int)gridDim.x;
  Tile& C = reinterpret_cast<Tile*>(smem)[warp];
  ResShared<ST, R>& sh = C.sh;
  const int t = (int)cl_rank() + ctas * warp;  // this warp's tile, placed as in k_resident
  const unsigned bar = (unsigned)__cvta_generic_to_shared(&C.bar[0]);
  ResWarp<MASKED, ST, R> W;
  unsigned ex = 0;
  if (t < A.ntiles) {
    const ResTile T = A.tiles[t];
    ex = W.load(sh, A, lane, t, T).x;
    auto words = [&](int k, const void* field) {  // the same field of tile k's shared memory
      const unsigned local = (unsigned)__cvta_generic_to_shared(field) + (unsigned)((k / ctas - warp) * (int)sizeof(Tile));
      return cl_addr(local, (unsigned)(k % ctas));
    };
    auto there = [&](int d) { return T.nb[d] != t; };
    const bool own = lane >= 1 && lane <= kResCols, west = lane == 1, end = west || lane == kResCols;
    uint4 row = make_uint4(0u, 0u, 0u, 0u), diag = row;
    uint2 side = make_uint2(0u, 0u);
    if (own && there(1)) row.x = words(T.nb[1], &C.in[0].n[lane]), row.y = words(T.nb[1], &C.bar[0]);
    if (own && there(0)) row.z = words(T.nb[0], &C.in[0].s[lane]), row.w = words(T.nb[0], &C.bar[0]);
    // this tile's first column is the east halo of the tiles west of it, its last the west halo of
    // those east of it
    const int sw = west ? 6 : 7, nw = west ? 4 : 5, w = west ? 2 : 3, at = west ? 31 : 0;
    if (end && there(sw)) diag.x = words(T.nb[sw], &C.in[0].n[at]), diag.y = words(T.nb[sw], &C.bar[0]);
    if (end && there(nw)) diag.z = words(T.nb[nw], &C.in[0].s[at]), diag.w = words(T.nb[nw], &C.bar[0]);
    if (end && there(w)) side = make_uint2(words(T.nb[w], &C.in[0].c[west ? 1 : 0][0]), words(T.nb[w], &C.bar[0]));
    C.row[lane] = row;
    C.diag[lane] = diag;
    C.side[lane] = side;
    // what no neighbour fills stays zero
    for (int k = 0; k < 2; k++) {
      C.in[k].n[lane] = C.in[k].s[lane] = Word::of(make_uint4(0u, 0u, 0u, 0u));
      if (lane < 2 * R) C.in[k].c[lane / R][lane % R] = Word::of(make_uint4(0u, 0u, 0u, 0u));
    }
    if (lane == 0) {
      C.bytes = (int)sizeof(typename Word::T) * (kResCols * (there(0) + there(1)) + R * (there(2) + there(3)) + there(4) +
                                                 there(5) + there(6) + there(7));
      for (int k = 0; k < 2; k++) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8u * k) : "memory");
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      for (int k = 0; k < 2; k++) bar_arm(bar + 8u * k, C.bytes);
    }
  }
  cl_barrier();  // every inbox is ready
  bool gave_up = false;
  if (t < A.ntiles) {
    if (t != A.mute) push<ST, R>(W.s, C, lane, 0, W.flag(sh));  // iteration 0's input
    bool waiting = true;
#pragma unroll 1
    for (int j = 0; j < A.n; j++) {
      const int k = j & 1;
      for (int waits = 0; waiting && !bar_wait(bar + 8u * k, (unsigned)(j >> 1) & 1u); waits++)
        if (waits >= kResWaits) waiting = false;
      __syncwarp();
      const uint4 wn = Word::wide(C.in[k].n[lane]), ws = Word::wide(C.in[k].s[lane]);
      if (lane == 0 || lane == 31) W.s.take_col(C.in[k].c[lane >> 4]);
      if constexpr (W.kPlain) W.meet(sh, wn.w | ws.w | C.in[k].c[lane >> 4][lane & (R - 1)].w);
      __syncwarp();
      // for iteration j + 2 (not once the barrier may still be armed for this one)
      if (lane == 0 && waiting && j + 2 < A.n) bar_arm(bar + 8u * k, C.bytes);
      W.iterate(sh, A, lane, j, ex, wn, ws);
      if (j + 1 < A.n) push<ST, R>(W.s, C, lane, j + 1, W.flag(sh));
      if (j + 2 >= A.n) W.store(sh, A, lane, j + 1 == A.n);
    }
    gave_up = !__all_sync(kFull, waiting);
    if (gave_up && lane == 0) give_up(A);
  }
  if (!MASKED) res_fill<ST, R>(A, warp, lane);
  cl_barrier();  // no block leaves while its neighbours may store into it
  // Words that a tile has not waited for may still be on their way when all of them have been sent; its
  // block stays until they are in (a word takes 600 cycles).
  if (gave_up)
    for (const long long c = clock64(); clock64() - c < 200000ll;) {
    }
}

namespace {

template <bool MASKED, class ST, int R>
struct Res {
  static constexpr int kThreads = 32 * kResMostWarps;
  static constexpr size_t kSmem = sizeof(ResShared<ST, R>) * kResMostWarps;
  static constexpr size_t kClusterSmem = sizeof(ResClusterTile<ST, R>) * 16;
  // What the launches ask of the kernel, set with every plan: a device that has been reset forgets it.
  static int use(bool cluster) {
    if (!cluster)
      VFS_CUDA(cudaFuncSetAttribute(k_resident<MASKED, ST, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    if constexpr (R == kResClusterRows) {
      if (cluster) {
        const auto k = k_resident_cluster<MASKED, ST, R>;
        VFS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem));
        VFS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
      }
    }
    return 0;
  }
  // tiles that a grid of one block per SM holds, all of it resident
  static int capacity() {
    int dev = 0, sms = 0, per = 0, coop = 0, smem = 0;
    VFS_CUDA(cudaGetDevice(&dev));
    VFS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    VFS_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    VFS_CUDA(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (!coop || kSmem > (size_t)smem) return 0;
    use(false);
    VFS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_resident<MASKED, ST, R>, kThreads, kSmem));
    return per >= 1 ? sms * kResMostWarps : 0;
  }
  // warps the tiles of which one cluster of `ctas` blocks holds (0: no such cluster)
  static int cluster_capacity(int ctas) {
    if constexpr (R == kResClusterRows) {
      const auto k = k_resident_cluster<MASKED, ST, R>;
      int dev = 0, smem = 0, n = 0;
      VFS_CUDA(cudaGetDevice(&dev));
      VFS_CUDA(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
      if (kClusterSmem > (size_t)smem) return 0;
      use(true);
      cudaLaunchAttribute at[1];
      cudaLaunchConfig_t cfg = cluster_config(ctas, 16, 0, at);
      if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
      }
      return n >= 1 ? ctas * 16 : 0;
    }
    return 0;
  }
  static cudaLaunchConfig_t cluster_config(int ctas, int warps, cudaStream_t st, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(32 * warps);
    cfg.dynamicSmemBytes = sizeof(ResClusterTile<ST, R>) * warps;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
  }
  // the priority that the batch sets around a part's launches, as the other iteration kernels carry it (B200, eight
  // 848 x 800 pairs, half: 7.86 ms a batch with it, 7.85 without; the lanes' streams have priorities of their own)
  static void add_priority(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {
    const int prio = launch_priority();
    if (prio == 0) return;
    at[cfg.numAttrs].id = cudaLaunchAttributePriority;
    at[cfg.numAttrs].val.priority = prio;
    cfg.numAttrs++;
  }
  static int launch_cluster(const ResArgs& A, cudaStream_t st) {
    if constexpr (R == kResClusterRows) {
      cudaLaunchAttribute at[2];
      cudaLaunchConfig_t cfg = cluster_config(A.blocks, (A.ntiles + A.blocks - 1) / A.blocks, st, at);
      add_priority(cfg, at);
      VFS_CUDA(cudaLaunchKernelEx(&cfg, k_resident_cluster<MASKED, ST, R>, A));
    }
    return 0;
  }
  static int launch(const ResArgs& A, cudaStream_t st) {
    // only the warps that have a tile: blocks of other pairs' levels share the SM
    const int warps = (A.ntiles + A.blocks - 1) / A.blocks;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(A.blocks);
    cfg.blockDim = dim3(32 * warps);
    cfg.dynamicSmemBytes = sizeof(ResShared<ST, R>) * warps;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    add_priority(cfg, at);
    VFS_CUDA(cudaLaunchKernelEx(&cfg, k_resident<MASKED, ST, R>, A));
    return 0;
  }
};

// f(Res<...>()) for the instance of `rows` rows (kResRows)
template <bool MASKED, class ST, class F>
int res_rows(int rows, F&& f) {
  if (rows == 2) return f(Res<MASKED, ST, 2>());
  if (rows == 4) return f(Res<MASKED, ST, 4>());
  if (rows == 6) return f(Res<MASKED, ST, 6>());
  if (rows == 8) return f(Res<MASKED, ST, 8>());
  if constexpr (!std::is_same<ST, float>::value) {
    if (rows == 12) return f(Res<MASKED, ST, 12>());
    if (rows == 16) return f(Res<MASKED, ST, 16>());
  }
  return 0;
}
template <class F>
int res_dispatch(bool masked, bool half, int rows, F&& f) {
  if (masked) return half ? res_rows<true, __half>(rows, f) : res_rows<true, float>(rows, f);
  return half ? res_rows<false, __half>(rows, f) : res_rows<false, float>(rows, f);
}

}  // namespace

int res_capacity(bool masked, bool half, int rows, int cluster) {
  int dev = 0;
  VFS_CUDA(cudaGetDevice(&dev));
  static std::mutex mu;
  static std::map<std::tuple<int, bool, bool, int, int>, int> known;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_tuple(dev, masked, half, rows, cluster);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  return known[key] = res_dispatch(masked, half, rows, [cluster](auto k) {
           return cluster ? decltype(k)::cluster_capacity(cluster) : decltype(k)::capacity();
         });
}

// A plan's tables travel in kernel arguments, 28 KB a launch (848 x 800: five launches).  A copy from pageable
// memory may wait for the stream, and the first solve with a mask then returned only when the work
// queued before it was done.
namespace {
struct ResUpload {
  unsigned* to;
  int n;
  unsigned w[7168];
};
__global__ void k_res_upload(const __grid_constant__ ResUpload U) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i < U.n) U.to[i] = U.w[i];
}
}  // namespace

void res_use(bool masked, bool half, int rows, bool cluster) {
  res_dispatch(masked, half, rows, [cluster](auto k) { return decltype(k)::use(cluster); });
}

void launch_res_upload(void* to, const void* from, size_t bytes, cudaStream_t st) {
  ResUpload U;
  for (size_t at = 0; at < bytes; at += sizeof(U.w)) {
    const size_t b = std::min(bytes - at, sizeof(U.w));
    U.to = (unsigned*)((char*)to + at);
    U.n = (int)(b / 4);
    std::memcpy(U.w, (const char*)from + at, b);
    k_res_upload<<<(U.n + 127) / 128, 128, 0, st>>>(U);
    VFS_LAUNCH_CHECK();
  }
}

void launch_resident(const ResArgs& A, bool masked, bool half, cudaStream_t st) {
  if (A.ntiles <= 0 || A.blocks <= 0 || A.n < 1 || A.n > kResMaxIters) throw ArgError{"resident iteration: bad launch"};
  int dev = 0, sms = 0;
  VFS_CUDA(cudaGetDevice(&dev));
  VFS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int cap = res_capacity(masked, half, A.rows, A.cluster ? A.blocks : 0);
  if (A.cluster ? A.ntiles > cap : A.blocks > sms || A.ntiles > A.blocks * (cap / sms))
    throw ArgError{"resident iteration: more tiles than can be resident"};
  res_dispatch(masked, half, A.rows, [&](auto k) {
    return A.cluster ? decltype(k)::launch_cluster(A, st) : decltype(k)::launch(A, st);
  });
  VFS_LAUNCH_CHECK();
}

std::atomic<bool>& res_muted() {
  static std::atomic<bool> on{false};
  return on;
}

int resident_status_take() {
  int v = 0;
  VFS_CUDA(cudaMemcpyFromSymbol(&v, g_res_status, sizeof(v)));
  if (v) {
    const int z = 0;
    VFS_CUDA(cudaMemcpyToSymbol(g_res_status, &z, sizeof(z)));
  }
  return v;
}

}  // namespace vfs
