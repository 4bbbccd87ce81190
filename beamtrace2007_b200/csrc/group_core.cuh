// One sub-beam worked on by a group of lanes (device code only).
//
// A beam is four corner rays, a triangle test is up to four lines against
// those corners, a clip polygon has up to six vertices: a group of lanes
// takes a corner, a line or a vertex each, so a record's step is a few short
// operations deep where one lane would loop over them.  What bounds these
// steps is the chain of dependent operations per record (a frame's records
// depend on their parents, and a warp of independent records spends most of
// its instructions on 3-4 of its 32 lanes), not bytes.
//
// Every value is computed by the same IEEE single-precision operations in
// the same order as in beam_math.cuh / engine_core.cuh, so decisions, pieces
// and counters are bitwise the same; sums over vertices run in vertex order.
//
// All lanes of a warp run these functions together (full-mask shuffles and
// ballots, no divergence between groups); `act` says whether a group takes
// part, and the values of a group that does not are never used.
#pragma once

#include "engine_core.cuh"

namespace btg {

// --------------------------------------------------------- lanes of a group

// A group: eight lanes side by side, four groups a warp.
struct Grp {
  static __device__ __forceinline__ int lane() { return threadIdx.x & 31; }
  static __device__ __forceinline__ int sub() { return threadIdx.x & 7; }
  static __device__ __forceinline__ int base() { return threadIdx.x & 24; }
  // the group's lanes for which `pred` holds, bit 0 = its first lane
  static __device__ __forceinline__ unsigned ballot(bool pred) {
    return (__ballot_sync(0xffffffffu, pred) >> base()) & 0xffu;
  }
  template <class T>
  static __device__ __forceinline__ T shfl(T v, int src) {
    return __shfl_sync(0xffffffffu, v, src, 8);
  }
};

// A record's triangle: the line this lane looks after (0-2: the edges, 3: the
// depth line against the current hit or the far plane) and what lane 0 found
// about the triangle.
enum { kTriPlain = 1, kTriFront = 2 };  // not edge-on; D > 0

// The beam's current hit (primary visibility).
struct HitPlane {
  float A[3], C;
  V3 n;
  int tri;
};

// Edge lines and the depth line of triangle t, one per lane, before they are
// normalised (BeamCtx::triSetup and closerLine, as testOne evaluates them):
// true with the coefficients in L, or false with a constant line in L (lane 3).
// That is a tie of coplanar surfaces, whose corners vote on its 1 or -1 like on
// any other distance; or no depth line at all -- primary, no hit yet --, which
// every corner is inside of: infinitely far, whatever eps is (eps grows with the
// root's extent and passes 1 in views close to 180 degrees).  `flags`: kTriPlain
// | kTriFront, the same in all lanes of the group.
template <bool Nearest>
__device__ __forceinline__ bool laneCoefs(const Query& q, const TriRec& t, const HitPlane& h, Line& L, int& flags,
                                          V3& r0, V3& r1, V3& r2) {
  const int e = threadIdx.x & 3;
  r0 = sub(t.v0, q.P.O);
  r1 = sub(t.v1, q.P.O);
  r2 = sub(t.v2, q.P.O);
  const V3 ri = e == 0 ? r0 : (e == 1 ? r1 : r2), rj = e == 0 ? r1 : (e == 1 ? r2 : r0);
  const bool fwd = e == 0 ? t.vi[0] < t.vi[1] : (e == 1 ? t.vi[1] < t.vi[2] : t.vi[2] < t.vi[0]);
  V3 m = cross(fwd ? ri : rj, fwd ? rj : ri);
  if (!fwd) m = neg(m);
  int fl = 0;
  {
    const float D = dot(r2, m);  // lane 0's is the triangle's
    if (notEdgeOn(D, m, r2)) fl |= kTriPlain;
    if (D > 0) fl |= kTriFront;
  }
  flags = Grp::shfl(fl, 0);
  if (e == 3) m = t.n;
  L.a = dot(m, q.P.u);
  L.b = dot(m, q.P.v);
  L.c = dot(m, q.P.d);
  if (e == 3) {
    constexpr bool far = !Nearest;
    if (!far && h.tri < 0) {
      L = Line{0.f, 0.f, kInf};
      return false;
    }
    TriInfo ti;
    ti.tri = t.tri;
    ti.n = t.n;
    ti.A[0] = L.a;
    ti.A[1] = L.b;
    ti.A[2] = L.c;
    ti.C = dot(t.n, r0);
    const float AF[3] = {far ? 0.f : h.A[0], far ? 0.f : h.A[1], far ? q.farCq : h.A[2]};
    const float CF = far ? q.farCq : h.C;
    return closerCoefs(ti, AF, CF, far ? q.P.n : h.n, far ? -1 : h.tri, L);
  }
  const float sg = (flags & kTriFront) ? 1.f : -1.f;
  L.a *= sg;
  L.b *= sg;
  L.c *= sg;
  return true;
}

// ------------------------------------------------------ the walk of a record

// A record's fields other than its corners, the same in every lane of the
// group that works on it.
struct GroupRec {
  unsigned long long trail;
  uint32_t node;
  int root, hit, cursor, depth, n, neg;
};

// What a group does next.
enum GroupPhase {
  kGIdle = 0,     // no record
  kGDescend = 1,  // at an inner node
  kGTest = 2,     // a triangle of the leaf is pending
  kGClimb = 3,    // the leaf (or a skipped cell) is done: pop the restart trail
  kGDone = 4,     // the beam is finished: outTri
  kGClip = 5      // the triangle at the cursor needs a clip
};

// A record being walked by a group (lane k and lane k + 4 hold corner k & 3).
// The steps are those of engine_core.cuh (descendStep,
// climbStep, testOne) with the four corners, and the up to four lines of a
// triangle, side by side; a step's corner comparisons are packed into one word
// and the lanes' words combined by two shuffles.
template <bool Nearest>
struct GroupWalk {
  using W = Grp;
  GroupRec r;
  Query q;
  float cx[4], cy[4];  // every corner (the lines' votes)
  float qx, qy;        // this lane's corner
  float aw0, aw1, aw2; // |w| there
  float farA, farC;
  HitPlane h;
  uint2 nd;            // record of r.node
  Box box;             // its cell (while descending)
  int phase, outTri;

  static __device__ __forceinline__ unsigned all4(unsigned bits) {
    bits &= __shfl_xor_sync(0xffffffffu, bits, 1);
    return bits & __shfl_xor_sync(0xffffffffu, bits, 2);
  }
  // No record yet: values that the steps of other groups may compute with.
  __device__ __forceinline__ void idle() {
    r = GroupRec{0, 0, -1, -1, 0, 0, 0, 0};
    q = Query{};
    for (int k = 0; k < 4; ++k) cx[k] = cy[k] = 0.f;
    qx = qy = aw0 = aw1 = aw2 = farA = farC = 0.f;
    h = HitPlane{};
    h.tri = -1;
    nd = make_uint2(0, 3);
    box = Box{};
    phase = kGIdle;
    outTri = -1;
  }
  __device__ __forceinline__ float aw(int a) const { return a == 0 ? aw0 : (a == 1 ? aw1 : aw2); }

  __device__ __forceinline__ void setHit(int tri, V3 n, const float* A, float C) {
    h.tri = tri;
    h.n = n;
    h.A[0] = A[0];
    h.A[1] = A[1];
    h.A[2] = A[2];
    h.C = C;
    farA = fabs_(qx * A[0] + qy * A[1] + A[2]);
    farC = C < 0 ? -C : C;
  }

  // the cell of a node just entered: an inner one is descended, a leaf's
  // triangles are next
  __device__ __forceinline__ void enter(Stats& st) {
    if (isLeaf(nd)) {
      st.leafVisits++;
      r.cursor = 0;
      phase = (nd.y >> 2) > 0 ? kGTest : kGClimb;
    } else {
      phase = kGDescend;
    }
  }

  // Takes up a record (expand, walkBegin); r, cx, cy and q are set.
  __device__ __forceinline__ void begin(const SceneDev& s, Stats& st) {
    const int c = threadIdx.x & 3;
    qx = c == 0 ? cx[0] : (c == 1 ? cx[1] : (c == 2 ? cx[2] : cx[3]));
    qy = c == 0 ? cy[0] : (c == 1 ? cy[1] : (c == 2 ? cy[2] : cy[3]));
    const float w0 = qx * q.P.u.x + qy * q.P.v.x + q.P.d.x, w1 = qx * q.P.u.y + qy * q.P.v.y + q.P.d.y,
                w2 = qx * q.P.u.z + qy * q.P.v.z + q.P.d.z;
    const float s0 = w0 * ((r.neg & 1) ? -1.f : 1.f), s1 = w1 * ((r.neg & 2) ? -1.f : 1.f),
                s2 = w2 * ((r.neg & 4) ? -1.f : 1.f);
    aw0 = 0.f > s0 ? 0.f : s0;
    aw1 = 0.f > s1 ? 0.f : s1;
    aw2 = 0.f > s2 ? 0.f : s2;
    nd = s.node[r.node];
    h.tri = -1;
    if (!Nearest) {
      const float c0 = q.farCq < 0 ? -q.farCq : q.farCq;
      farA = c0;
      farC = c0;
    } else {
      farA = farC = 0.f;
      if (r.hit >= 0) {
        V3 nT, v0;
        float A[3], C;
        triNV(s, r.hit, nT, v0);
        hitPlane(q, nT, v0, A, C);
        setHit(r.hit, nT, A, C);
      }
    }
    outTri = -1;
    if (r.cursor < 0) {
      box = loadBox(s, r.node);
      enter(st);
    } else {
      phase = r.cursor < int(nd.y >> 2) ? kGTest : kGClimb;
    }
  }

  // descendStep: into the child the beam enters first
  __device__ __forceinline__ void descend(const SceneDev& s, bool act, Stats& st) {
    const int a = int(nd.y & 3u);
    const float sp = splitOf(nd);
    const bool pos = !((r.neg >> a) & 1);
    const float Ns = (pos ? 1.f : -1.f) * (sp - comp(q.P.O, a));
    const uint32_t left = r.node + 1, right = nd.y >> 2;
    uint2 ndLeft = nd, ndRight = nd;
    if (act) {
      ndLeft = s.node[left];
      ndRight = s.node[right];
    }
    const float wa = aw(a);
    unsigned bits = 0;
#pragma unroll
    for (int k = 1; k <= 2; ++k) {
      const int c = a + k >= 3 ? a + k - 3 : a + k;
      const bool p = !((r.neg >> c) & 1);
      const float sc = p ? 1.f : -1.f, Oc = comp(q.P.O, c), lo = boxLo(box, c), hi = boxHi(box, c);
      const float Nmin = sc * ((p ? lo : hi) - Oc), Nmax = sc * ((p ? hi : lo) - Oc);
      const float lhs = aw(c) * Ns;
      const float r0 = wa * Nmin, t0 = (fabs_(lhs) + fabs_(r0)) * kKdRel;
      if (lhs < r0 - t0) bits |= 1u << (2 * k - 2);
      const float r1 = wa * Nmax, t1 = (fabs_(lhs) + fabs_(r1)) * kKdRel;
      if (lhs > r1 + t1) bits |= 1u << (2 * k - 1);
    }
    if (!Nearest || h.tri >= 0) {
      const float lhs = farA * Ns, r0 = wa * farC, t0 = (fabs_(lhs) + fabs_(r0)) * kKdRel;
      if (lhs > r0 + t0) bits |= 16u;
    }
    bits = all4(bits);
    // decide: the first comparison that all corners pass (0 and 2: far child only)
    const unsigned first = bits & (0u - bits);
    const int dec = !(Ns > 0) ? int(kFar) : (bits == 0 ? int(kBoth) : ((first & 5u) ? int(kFar) : int(kNear)));
    if (act) {
      st.kdSteps++;
      if (dec == kBoth) r.trail |= 1ull << r.depth;
      r.depth++;
      const bool goRight = dec == kFar ? pos : !pos;
      r.node = goRight ? right : left;
      nd = goRight ? ndRight : ndLeft;
      if (goRight)
        boxSetLo(box, a, sp);
      else
        boxSetHi(box, a, sp);
      enter(st);
    }
  }

  // climbStep: one pop of the restart trail
  __device__ __forceinline__ void climb(const SceneDev& s, bool act, Stats& st) {
    const bool go = act && r.trail != 0;
    const int d = highestBit64(r.trail | 1ull);
    uint32_t node = r.node, cs = r.node;
    Box cb = box;
    uint2 nc = nd;
    if (go) {
      for (int k = r.depth; k > d; --k) node = s.parent[node];
      const uint2 nn = s.node[node];
      cs = ((r.neg >> (nn.y & 3u)) & 1) ? node + 1 : (nn.y >> 2);
      cb = loadBox(s, cs);
      nc = s.node[cs];
    }
    float Nmin[3], Nmax[3];
    bool miss = false;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const bool p = !((r.neg >> c) & 1);
      const float sc = p ? 1.f : -1.f, Oc = comp(q.P.O, c);
      Nmin[c] = sc * ((p ? cb.lo[c] : cb.hi[c]) - Oc);
      Nmax[c] = sc * ((p ? cb.hi[c] : cb.lo[c]) - Oc);
      if (Nmax[c] < 0) miss = true;
    }
    const float w[3] = {aw0, aw1, aw2};
    unsigned bits = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        if (c == e) continue;
        const float lhs = w[e] * Nmax[c], r0 = w[c] * Nmin[e], t0 = (fabs_(lhs) + fabs_(r0)) * kKdRel;
        if (lhs < r0 - t0) bits |= 1u << (3 * c + e);
      }
      if (!Nearest || h.tri >= 0) {
        const float lhs = farA * Nmin[c], r0 = w[c] * farC, t0 = (fabs_(lhs) + fabs_(r0)) * kKdRel;
        if (lhs > r0 + t0) bits |= 1u << (4 * c);  // (c == e above leaves these bits free)
      }
    }
    bits = all4(bits);
    if (go) {
      st.climbs += uint32_t(r.depth - d);
      r.trail &= (1ull << d) - 1;
      if (miss || bits) {
        r.node = node;
        r.depth = d;
      } else {
        r.node = cs;
        r.depth = d + 1;
        r.cursor = -1;
        box = cb;
        nd = nc;
        enter(st);
      }
    } else if (act) {
      phase = kGDone;
      outTri = Nearest ? h.tri : -1;
    }
  }

  // testOne: the triangle at the cursor
  __device__ __forceinline__ void test(const SceneDev& s, bool act, Stats& st) {
    TriRec t;
    t.v0 = t.v1 = t.v2 = t.n = mk(0, 0, 0);
    t.vi[0] = t.vi[1] = t.vi[2] = 0;
    t.tri = -1;
    if (act) t = loadRef(s, nd.x + uint32_t(r.cursor));
    Line L;
    int flags;
    V3 r0, r1, r2;
    const bool line = laneCoefs<Nearest>(q, t, h, L, flags, r0, r1, r2);
    bool anyIn = L.c > q.eps, anyOut = L.c < -q.eps;  // (a constant line's vote)
    const bool known =
        !line || voteUnscaled(cx, cy, L.a, L.b, L.c, max4abs(cx), max4abs(cy), q.eps, q.ext, anyIn, anyOut);
    if (__any_sync(0xffffffffu, act && !known)) {
      // a corner too close to its band's edge: the line itself
      const Line N = line ? makeLine(L.a, L.b, L.c, q.ext) : L;
      anyIn = anyOut = false;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float dv = cx[k] * N.a + cy[k] * N.b + N.c;
        anyIn |= dv > q.eps;
        anyOut |= dv < -q.eps;
      }
    }
    const unsigned in = W::ballot(anyIn), out = W::ballot(anyOut);
    const bool counted = act && t.tri != q.exclude && (flags & kTriPlain) && !(Nearest && q.cull && (flags & kTriFront));
    const bool meets = counted && !(Nearest && h.tri == t.tri) && in == 0xffu;
    if (counted) st.triTests++;
    const bool inside = meets && out == 0;
    bool clip = meets && out != 0;
    if (__any_sync(0xffffffffu, clip)) {
      // separated: a side plane of the beam with all three vertices outside it
      const int c = threadIdx.x & 3;
      const float wx = qx * q.P.u.x + qy * q.P.v.x + q.P.d.x, wy = qx * q.P.u.y + qy * q.P.v.y + q.P.d.y,
                  wz = qx * q.P.u.z + qy * q.P.v.z + q.P.d.z;
      const int nx = (W::sub() & ~3) | ((c + 1) & 3);
      const float vx = W::shfl(wx, nx), vy = W::shfl(wy, nx), vz = W::shfl(wz, nx);
      const float sx = wy * vz - wz * vy, sy = wz * vx - wx * vz, sz = wx * vy - wy * vx;
      const float sl = sqrtf(sx * sx + sy * sy + sz * sz);
      bool o = r.n == 4 || c != 2;
      const float e0 = sx * r0.x + sy * r0.y + sz * r0.z, e1 = sx * r1.x + sy * r1.y + sz * r1.z,
                  e2 = sx * r2.x + sy * r2.y + sz * r2.z;
      o = o && e0 < -(sl * (length(r0) * kEpsRel)) && e1 < -(sl * (length(r1) * kEpsRel)) &&
          e2 < -(sl * (length(r2) * kEpsRel));
      if (W::ballot(o)) clip = false;
    }
    if (act) {
      if (clip) {
        phase = kGClip;
      } else if (!Nearest && inside) {
        phase = kGDone;
        outTri = t.tri;
      } else {
        if (inside) {
          const float A[3] = {dot(t.n, q.P.u), dot(t.n, q.P.v), dot(t.n, q.P.d)};
          setHit(t.tri, t.n, A, dot(t.n, r0));
          r.hit = t.tri;
        }
        r.cursor += 1;
        phase = r.cursor < int(nd.y >> 2) ? kGTest : kGClimb;
      }
    }
  }
};

// -------------------------------------------------- polygons, a vertex a lane

// Signed area (Poly::area): the terms are summed in vertex order.
__device__ __forceinline__ float groupArea(float px, float py, int n) {
  using W = Grp;
  const int nx = W::sub() + 1 == n ? 0 : W::sub() + 1;
  const float xn = W::shfl(px, nx), yn = W::shfl(py, nx);
  const float t = px * yn - xn * py;
  float a = 0;
#pragma unroll
  for (int k = 0; k < kPolyMax; ++k) {
    const float tk = W::shfl(t, k);
    if (k < n) a += tk;
  }
  return a * 0.5f;
}

// A group's polygon in registers: this lane's vertex and the vertex count.
struct LanePoly {
  float x, y;
  int n;
};

// cleanPoly, all vertices of a pass tested at once: vertices before the first
// one to go are what the pass would have found them, so dropping that one and
// going on at its place is the pass.
struct CleanState {
  bool run, changed;
  int i0;
};
__device__ __forceinline__ void cleanBegin(CleanState& s, const LanePoly& p, bool act) {
  s.run = act && p.n >= 3;
  s.changed = false;
  s.i0 = 0;
}
__device__ __forceinline__ void cleanStep(CleanState& s, LanePoly& p, float eps) {
  using W = Grp;
  const int sub = W::sub();
  const int h = sub == 0 ? p.n - 1 : sub - 1, j = sub + 1 >= p.n ? 0 : sub + 1;
  const float xh = W::shfl(p.x, h), yh = W::shfl(p.y, h), xj = W::shfl(p.x, j), yj = W::shfl(p.y, j);
  const float ex = xj - xh, ey = yj - yh, dx = p.x - xh, dy = p.y - yh;
  const float len = sqrtf(ex * ex + ey * ey);
  const float gapSq = dx * dx + dy * dy;
  const float offLine = fabs_(ex * dy - ey * dx);
  const bool goes = sub < p.n && (gapSq <= eps * eps || offLine <= eps * len);
  const unsigned b = W::ballot(goes) & (0xffu << s.i0);
  if (!__any_sync(0xffffffffu, s.run && b)) {  // no vertex goes in any group: a pass without a drop, or one more pass
    s.run = s.run && s.changed;
    s.changed = false;
    s.i0 = 0;
    return;
  }
  const float xs = W::shfl(p.x, sub + 1), ys = W::shfl(p.y, sub + 1);
  if (s.run) {
    if (b) {
      const int k = __ffs(b) - 1;
      if (sub >= k) {
        p.x = xs;
        p.y = ys;
      }
      --p.n;
      s.changed = true;
      s.i0 = k;
      if (p.n < 3) s.run = false;
    } else {
      s.run = s.changed;
      s.changed = false;
      s.i0 = 0;
    }
  }
}
__device__ __forceinline__ void groupClean(LanePoly& p, bool act, float epsSplit) {
  const float eps = epsSplit * 1e-3f;
  CleanState s;
  cleanBegin(s, p, act);
  while (__any_sync(0xffffffffu, s.run)) cleanStep(s, p, eps);
  if (act && p.n < 3) p.n = 0;
}
// two polygons of a group at once (the halves of a split)
__device__ __forceinline__ void groupClean2(LanePoly& p, LanePoly& r, bool act, float epsSplit) {
  const float eps = epsSplit * 1e-3f;
  CleanState s, t;
  cleanBegin(s, p, act);
  cleanBegin(t, r, act);
  while (__any_sync(0xffffffffu, s.run || t.run)) {
    cleanStep(s, p, eps);
    cleanStep(t, r, eps);
  }
  if (act && p.n < 3) p.n = 0;
  if (act && r.n < 3) r.n = 0;
}

// Shared memory of one clipping group: the halves of a split on their way
// from the lane that made a vertex to the lane that keeps it, the pending
// pentagon halves (three corners each; at most one per line) and the pieces
// of the first pass.
//
// Pieces: a polygon meets at most four lines (three edges and one depth
// line); at each it gives one outside piece and at most two polygons that go
// on (a pentagon in two), so f(l) = 1 + 2 f(l - 1) pieces, f(0) = 1: 31.
constexpr int kGroupPieces = 31;
struct __align__(16) ClipScratch {
  float vx[2][8], vy[2][8];
  float sx[5][3], sy[5][3];
  int sline[5];
  uint8_t level[kGroupPieces + 1], n[kGroupPieces + 1], clean[kGroupPieces + 1];
  float lx[kGroupPieces][5], ly[kGroupPieces][5];
};

// Clips the group's beam by its lines, most-cutting edge first (clipTri), and
// logs the pieces in push order.  L: the line of lanes 0-3 (nl of them used);
// corners in lanes 0..n-1 of p.  Returns false if a piece or the pending list
// overflowed.  newArea, slots0, slots1: AreaSink's sums; five: pentagons
// split inside the clip.
__device__ __forceinline__ bool groupClip(float eps, LanePoly p, const Line& L, int nl, bool act, ClipScratch& S,
                                          float& newArea, int& slots0, int& slots1, int& count, int& five) {
  using W = Grp;
  const int sub = W::sub();
  const unsigned lt = (1u << sub) - 1u;
  newArea = 0.f;
  slots0 = slots1 = count = five = 0;
  // the edges by how much of the beam lies inside, least first (stable)
  int perm;
  {
    float score = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float dv = W::shfl(p.x, i) * L.a + W::shfl(p.y, i) * L.b + L.c;
      const float pos = dv > 0.f ? dv : 0.f;
      if (i == 0)
        score = pos;
      else if (i < 3)
        score = score + pos;
      else
        score = score + (p.n == 4 ? pos : 0.f);
    }
    float s0 = W::shfl(score, 0), s1 = W::shfl(score, 1), s2 = W::shfl(score, 2);
    int p0 = 0, p1 = 1, p2 = 2;
    if (s1 < s0) {
      const float t = s0;
      s0 = s1;
      s1 = t;
      p0 = 1;
      p1 = 0;
    }
    if (s2 < s1) {
      p2 = p1;
      p1 = 2;
      s1 = s2;
      if (s1 < s0) {
        p1 = p0;
        p0 = 2;
      }
    }
    perm = p0 | (p1 << 4) | (p2 << 8) | (3 << 12);
  }
  bool ok = true, fail = false, clean = true;
  bool run = act;
  int li = 0, sp = 0;
  while (__any_sync(0xffffffffu, run)) {
    // the group's next line; past the last one the polygon is inside them all
    const bool line = li < nl;
    const int src = (perm >> (4 * (line ? li : 0))) & 15;
    const float la = W::shfl(L.a, src), lb = W::shfl(L.b, src), lc = W::shfl(L.c, src);
    const bool mine = sub < p.n;
    const float d = la * p.x + lb * p.y + lc;
    const int s = mine ? (d > eps ? 1 : (d < -eps ? -1 : 0)) : 0;
    const unsigned bPos = W::ballot(s > 0), bNeg = W::ballot(s < 0);
    const bool cut = run && line && bPos && bNeg;
    const bool next = run && line && !bNeg;  // nothing outside this line
    bool push = run && !cut && !next;
    bool pop = push;
    LanePoly o = p;           // what is pushed
    int level = line ? 0 : 1;
    bool oClean = clean;
    if (__any_sync(0xffffffffu, cut)) {
      // splitPoly: the vertices of both halves in emission order
      const int nx = sub + 1 >= p.n ? 0 : sub + 1;
      const int sn = W::shfl(s, nx);
      const float dn = W::shfl(d, nx), xn = W::shfl(p.x, nx), yn = W::shfl(p.y, nx);
      const bool cross = mine && s * sn < 0;
      const unsigned bC = W::ballot(cross);
      const unsigned all = p.n >= 8 ? 0xffu : (1u << p.n) - 1u;
      const unsigned bIn = all & ~bNeg, bOut = all & ~bPos;
      const int nIn = __popc(bIn) + __popc(bC), nOut = __popc(bOut) + __popc(bC);
      const bool over = nIn > kPolyMax || nOut > kPolyMax;
      if (cut && !over) {
        const int at0 = __popc(bIn & lt) + __popc(bC & lt), at1 = __popc(bOut & lt) + __popc(bC & lt);
        if (mine && s >= 0) {
          S.vx[0][at0] = p.x;
          S.vy[0][at0] = p.y;
        }
        if (mine && s <= 0) {
          S.vx[1][at1] = p.x;
          S.vy[1][at1] = p.y;
        }
        if (cross) {
          // the crossing from the lexicographically smaller endpoint
          const bool here = p.x < xn || (p.x == xn && p.y < yn);
          const float da = here ? d : dn, db = here ? dn : d;
          const float xa = here ? p.x : xn, xb = here ? xn : p.x;
          const float ya = here ? p.y : yn, yb = here ? yn : p.y;
          const float t = da / (da - db);
          const float X = xa + t * (xb - xa);
          const float Y = ya + t * (yb - ya);
          const int k0 = at0 + (s >= 0 ? 1 : 0), k1 = at1 + (s <= 0 ? 1 : 0);
          S.vx[0][k0] = X;
          S.vy[0][k0] = Y;
          S.vx[1][k1] = X;
          S.vy[1][k1] = Y;
        }
      }
      __syncwarp();
      LanePoly in, out;
      in.x = S.vx[0][sub];
      in.y = S.vy[0][sub];
      in.n = nIn;
      out.x = S.vx[1][sub];
      out.y = S.vy[1][sub];
      out.n = nOut;
      __syncwarp();
      groupClean2(out, in, cut && !over, eps);
      if (cut) {
        if (over) {
          fail = true;
          run = false;
        } else {
          push = out.n >= 3;
          o = out;
          level = 0;
          oClean = true;
          if (in.n < 3) {
            pop = true;
          } else if (in.n == 5) {
            // quad (0,1,2,3) goes on, triangle (0,3,4) waits
            ++five;
            if (sub == 0 || sub == 3 || sub == 4) {
              const int k = sub == 0 ? 0 : sub - 2;
              S.sx[sp][k] = in.x;
              S.sy[sp][k] = in.y;
            }
            if (sub == 0) S.sline[sp] = li + 1;
            ++sp;  // (at most one waits per line, so sp <= 4)
            p = in;
            p.n = 4;
            clean = false;
          } else {
            p = in;
            clean = true;
          }
        }
      }
    }
    if (__any_sync(0xffffffffu, push)) {
      const float area = groupArea(o.x, o.y, o.n);
      if (push) {
        if (o.n > 5) {
          ok = false;
        } else {
          const int w = o.n == 5 ? 2 : 1;
          if (level == 1) {
            newArea += area;
            slots1 += w;
          } else {
            slots0 += w;
          }
          if (sub < 5) {
            S.lx[count][sub] = o.x;
            S.ly[count][sub] = o.y;
          }
          if (sub == 0) {
            S.level[count] = uint8_t(level);
            S.n[count] = uint8_t(o.n);
            S.clean[count] = oClean ? 1 : 0;
          }
          ++count;
        }
      }
    }
    ++li;
    if (pop && run) {
      if (sp == 0) {
        run = false;
      } else {
        --sp;
        li = S.sline[sp];
        if (sub < 3) {
          p.x = S.sx[sp][sub];
          p.y = S.sy[sp][sub];
        }
        p.n = 3;
        clean = false;
      }
    }
    __syncwarp();
  }
  return ok && !fail;
}

}  // namespace btg
