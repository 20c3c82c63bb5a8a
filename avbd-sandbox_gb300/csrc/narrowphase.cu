// narrowphase.cu - contact generation, manifold merge and warm start.
//
// One thread per candidate pair; box pairs that the f32 test below leaves
// undecided take sixteen lanes each in lists that are not too long
// (pairs_per_warp). The geometry runs in IEEE f64 with the reference's operation
// order and NO fused multiply-add (this translation unit is compiled with
// --fmad=false), so that from identical inputs the contact count, feature IDs
// and SAT/clipping decisions equal the reference engine's bit for bit:
//   collide.js:612-685 box-box 15-axis SAT, face clipping (:403-472),
//                      edge contact (:475-493)
//   collide.js:496-520 sphere-sphere, :526-600 sphere-OBB
//   manifold.js:214-318 feature-ID merge, sphere basis transport,
//                      C*(x_t) + margin, warm start lambda <- gamma(alpha lambda),
//                      k <- clamp(gamma k, kmin, kmax)
// Box-box SAT runs first in f32 in a frame centred on body A, each of the 15
// axis separations with a conservative bound on its distance from the f64
// value (GB300's FP64 rate is a small fraction of its FP32 rate). A bound
// that cannot settle a decision - the sign of a separation, the skip of a
// near-degenerate edge axis, the order of near-tied best axes, the edge-vs-
// face choice - sends just those axes through the exact f64 axis test, so
// every decision equals the f64 one. The winning axis's normal, the contact
// basis and the clipping stay in exact f64.
#include "avbd_device.cuh"
#include "collider.cuh"

namespace avbd {
namespace {

// The exact geometry (collider.cuh) in f64.
using geo::kFaceA;
using geo::kFaceB;
using geo::kEdge;
using geo::kPlaneEps;
using geo::kPolyCap;
using geo::kSatEps;
using geo::kMergeDistSq;
using D3 = geo::D3T<double>;
using QD = geo::QDT<double>;
using BodyD = geo::BodyT<double>;
using OBB = geo::OBBT<double>;
using NewContact = geo::NewContactT<double>;
using Collider = geo::ColliderT<double>;
using geo::add;
using geo::adds;
using geo::clampd;
using geo::conj;
using geo::crs;
using geo::dt3;
using geo::neg;
using geo::orthonormal;
using geo::rot;
using geo::scl;
using geo::sub;
__device__ __forceinline__ D3 mk(double x, double y, double z) { return D3{x, y, z}; }



struct NewContactF {
  uint32_t feature;
  float ra[3], rb[3];
};

// The two boxes in f32 in a frame centred on A: B's centre, the box axes and
// the half sizes.
struct BoxF {
  V3<float> d, ax[3], bx[3];
  float ha[3], hb[3];
};

__device__ BoxF make_boxf(const BodyD &A, const BodyD &B) {
  BoxF F;
  const Q4<float> qa{(float)A.q.x, (float)A.q.y, (float)A.q.z, (float)A.q.w};
  const Q4<float> qb{(float)B.q.x, (float)B.q.y, (float)B.q.z, (float)B.q.w};
  F.d = V3<float>{(float)(B.p.x - A.p.x), (float)(B.p.y - A.p.y), (float)(B.p.z - A.p.z)};
  F.ha[0] = (float)A.half.x; F.ha[1] = (float)A.half.y; F.ha[2] = (float)A.half.z;
  F.hb[0] = (float)B.half.x; F.hb[1] = (float)B.half.y; F.hb[2] = (float)B.half.z;
  F.ax[0] = qrotate(qa, V3<float>{1, 0, 0});
  F.ax[1] = qrotate(qa, V3<float>{0, 1, 0});
  F.ax[2] = qrotate(qa, V3<float>{0, 0, 1});
  F.bx[0] = qrotate(qb, V3<float>{1, 0, 0});
  F.bx[1] = qrotate(qb, V3<float>{0, 1, 0});
  F.bx[2] = qrotate(qb, V3<float>{0, 0, 1});
  return F;
}

// Outcome of the f32 SAT of a box pair.
constexpr int kSeparated = 0, kFaceWin = 1, kEdgeWin = 2, kUndecided = 3, kFaceTie = 4;

// f32 SAT of a box-box pair (collide.js:612-685), certified against the f64
// evaluation: every axis separation comes with a bound err >= |sep_f32 -
// sep_f64|, derived from a per-component error of the f32 box axes of at
// most ~32 ulp(1) and the 1/len amplification of normalising an edge axis,
// with a 16x margin:
//   err = 512 u S (1 + 1/len),  u = 2^-24,  S = |d|_1 + sum(hA) + sum(hB).
// kSeparated when some axis certainly separates the boxes (the f64 test then
// finds a separating axis too and returns no contact). kFaceWin / kEdgeWin
// when no axis can separate, the best face axis (largest separation, first
// on ties) and, if it can matter, the best edge axis are certain, and so is
// the choice 0.95 sepE > sepF + 0.01 between them. kFaceTie when all of that
// holds and a face wins, but which face is not certain: tieMask (bits 0-5:
// faces 0-2 of A, 0-2 of B) lists the face axes that can be the largest,
// for an exact f64 comparison of just those. kUndecided otherwise: the exact
// f64 path decides.
__device__ int classify_f32(const BoxF &F, bool &refIsA, int &axA, int &axB, int &tieMask) {
  const float S = fabsf(F.d.x) + fabsf(F.d.y) + fabsf(F.d.z) + F.ha[0] + F.ha[1] + F.ha[2] + F.hb[0] + F.hb[1] +
                  F.hb[2];
  if (!(S == S) || S > 1e30f) return kUndecided;
  constexpr float u512 = 512.0f / 16777216.0f;
  const float eBase = u512 * S;
  bool undecided = false;
  // best of each group so far, and the largest upper bound among the others
  int fBest = -1, eBest = -1;
  float fSep = 0.f, fErr = 0.f, fOther = -INFINITY, eSep = 0.f, eErr = 0.f, eOther = -INFINITY;
  float fUp[6];  // upper bound of each face axis's separation
#pragma unroll
  for (int k = 0; k < 6; k++) fUp[k] = -INFINITY;
#pragma unroll
  for (int k = 0; k < 15; k++) {
    V3<float> a;
    const bool edge = k >= 6;
    if (k < 3) a = F.ax[k];
    else if (k < 6) a = F.bx[k - 3];
    else {
      const V3<float> p = F.ax[(k - 6) / 3], q = F.bx[(k - 6) % 3];
      a = V3<float>{p.y * q.z - p.z * q.y, p.z * q.x - p.x * q.z, p.x * q.y - p.y * q.x};
    }
    const float lenSq = a.x * a.x + a.y * a.y + a.z * a.z;
    if (edge) {
      // lenSq of the f32 cross product is within 1024 u len + 1e-9 of the f64 one
      const float eLen = (1024.0f / 16777216.0f) * sqrtf(lenSq) + 1e-9f;
      if (lenSq + eLen < (float)kSatEps) continue;  // the f64 test skips this axis too
      if (lenSq - eLen < (float)kSatEps) {
        undecided = true;
        continue;
      }
    } else if (!(lenSq >= 0.25f)) {
      undecided = true;
      continue;
    }
    const float len = sqrtf(lenSq);
    const V3<float> n{a.x / len, a.y / len, a.z / len};
    const float dist = fabsf(n.x * F.d.x + n.y * F.d.y + n.z * F.d.z);
    float rA = 0.f, rB = 0.f;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      rA += F.ha[i] * fabsf(n.x * F.ax[i].x + n.y * F.ax[i].y + n.z * F.ax[i].z);
      rB += F.hb[i] * fabsf(n.x * F.bx[i].x + n.y * F.bx[i].y + n.z * F.bx[i].z);
    }
    const float sep = dist - (rA + rB);
    const float err = eBase * (1.0f + 1.0f / len);
    if (sep - err > 0.f) return kSeparated;
    if (sep + err > 0.f) {
      undecided = true;
      continue;
    }
    if (!edge) {
      fUp[k < 6 ? k : 0] = sep + err;
      if (fBest < 0 || sep > fSep) {
        if (fBest >= 0) fOther = fmaxf(fOther, fSep + fErr);
        fBest = k; fSep = sep; fErr = err;
      } else {
        fOther = fmaxf(fOther, sep + err);
      }
    } else {
      if (eBest < 0 || sep > eSep) {
        if (eBest >= 0) eOther = fmaxf(eOther, eSep + eErr);
        eBest = k; eSep = sep; eErr = err;
      } else {
        eOther = fmaxf(eOther, sep + err);
      }
    }
  }
  if (undecided || fBest < 0) return kUndecided;
  const float fLo = fSep - fErr, fHi = fmaxf(fSep + fErr, fOther);
  bool edgeWins = false;
  if (eBest >= 0) {
    const float eLo = eSep - eErr, eHi = fmaxf(eSep + eErr, eOther);
    const float slack = 1e-6f * (fabsf(eSep) + fabsf(fSep) + 0.01f);
    if (0.95f * eLo > fHi + 0.01f + slack) edgeWins = true;
    else if (!(0.95f * eHi < fLo + 0.01f - slack)) return kUndecided;
  }
  if (edgeWins) {
    if (!(eOther < eSep - eErr)) return kUndecided;  // tied edge axes
    axA = (eBest - 6) / 3;
    axB = (eBest - 6) % 3;
    return kEdgeWin;
  }
  if (!(fOther < fSep - fErr)) {  // tied face axes: the candidates for an exact comparison
    tieMask = 0;
#pragma unroll
    for (int k = 0; k < 6; k++)
      if (fUp[k] >= fLo) tieMask |= 1 << k;
    return kFaceTie;
  }
  refIsA = fBest < 3;
  axA = refIsA ? fBest : fBest - 3;
  return kFaceWin;
}

// ---- faceManifold (collide.js:403-472) in f32, in A's frame ------------------
struct FaceF {
  const BoxF &F;
  Q4<float> qaInv, qbInv;  // conjugate orientations of A and B (f32)
  NewContactF *outF;
  int count = 0;
  __device__ FaceF(const BoxF &f, const BodyD &A, const BodyD &B, NewContactF *o)
      : F(f),
        qaInv{(float)-A.q.x, (float)-A.q.y, (float)-A.q.z, (float)A.q.w},
        qbInv{(float)-B.q.x, (float)-B.q.y, (float)-B.q.z, (float)B.q.w},
        outF(o) {}
  // Every f32 point carries a bound .w on its distance from the f64 point
  // (minus A's position). Each discrete decision - clip side, intersection
  // denominator, contact depth, merge distance - is taken only when the
  // bound settles it; otherwise the function returns -1 and the caller runs
  // the f64 builder. Returns the contact count when every decision was certain.
  static constexpr float kU = 1.0f / 16777216.0f;  // unit roundoff of f32
  static constexpr float kEA = 64.0f * kU;         // error of an f32 box axis (2-norm)
  static constexpr float kFloor = 1e-9f;           // f64 rounding at world scale, and slack
  __device__ static float nrm(V3<float> v) { return sqrtf(v.x * v.x + v.y * v.y + v.z * v.z); }
  __device__ static V3<float> fsub(V3<float> a, V3<float> b) { return V3<float>{a.x - b.x, a.y - b.y, a.z - b.z}; }
  __device__ static V3<float> fadds(V3<float> o, V3<float> a, float s) {
    return V3<float>{o.x + a.x * s, o.y + a.y * s, o.z + a.z * s};
  }
  __device__ static float fdot(V3<float> a, V3<float> b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
  // clip side of a point at signed distance dd (bound e): 1 inside, 0 outside, -1 undecided
  __device__ static int side(float dd, float e) {
    if (dd + e <= (float)kPlaneEps) return 1;
    if (dd - e > (float)kPlaneEps) return 0;
    return -1;
  }
  // clipAgainstPlane (collide.js:202-247); -1 when a decision is undecided
  __device__ static int clipF(const float4 *in, int n, V3<float> pn, float po, float ePo, float4 *o) {
    if (n <= 0) return 0;
    auto dist = [&](float4 v, float &e) {
      const V3<float> p{v.x, v.y, v.z};
      const float np = nrm(p);
      const float dd = fdot(pn, p) - po;
      e = v.w + (kEA + 3.0f * kU) * np + ePo + kU * fabsf(dd) + kFloor;
      return dd;
    };
    int oc = 0;
    float4 a = in[n - 1];
    float ea;
    float da = dist(a, ea);
    int ai = side(da, ea);
    if (ai < 0) return -1;
    for (int i = 0; i < n; i++) {
      const float4 b = in[i];
      float eb;
      const float db = dist(b, eb);
      const int bi = side(db, eb);
      if (bi < 0) return -1;
      if (ai != bi) {
        const float denom = da - db;
        const float eDen = ea + eb + kU * fabsf(denom);
        float t = 0.f, et = 0.f;
        if (fabsf(denom) - eDen > (float)kSatEps) {
          if (fabsf(denom) < 4.0f * eDen) return -1;  // keep the first-order bound valid
          const float tr = da / denom;
          et = 1.5f * (fabsf(db) * ea + fabsf(da) * eb) / (denom * denom) + 2.0f * kU * fabsf(tr);
          t = fminf(fmaxf(tr, 0.f), 1.f);  // clamp is 1-Lipschitz: no decision to certify
        } else if (!(fabsf(denom) + eDen <= (float)kSatEps)) {
          return -1;
        }
        if (oc < kPolyCap) {
          const V3<float> pa{a.x, a.y, a.z}, pb{b.x, b.y, b.z};
          const V3<float> ab = fsub(pb, pa);
          const V3<float> q = fadds(pa, ab, t);
          const float e = a.w + t * (a.w + b.w) + nrm(ab) * et + 3.0f * kU * (nrm(pa) + nrm(ab)) + kFloor;
          o[oc++] = make_float4(q.x, q.y, q.z, e);
        }
      }
      if (bi && oc < kPolyCap) o[oc++] = b;
      a = b;
      da = db;
      ea = eb;
      ai = bi;
    }
    return oc;
  }
  // addContact (collide.js:254-285) on f32 points; 1 added, 0 merged or full,
  // -1 undecided
  __device__ int addContactF(V3<float> xA, float eA, V3<float> xB, float eB, uint32_t key, float4 *midF) {
    const V3<float> m{(xA.x + xB.x) * 0.5f, (xA.y + xB.y) * 0.5f, (xA.z + xB.z) * 0.5f};
    const float eM = 0.5f * (eA + eB) + 2.0f * kU * nrm(m) + kFloor;
    for (int i = 0; i < count; i++) {
      const V3<float> dv{m.x - midF[i].x, m.y - midF[i].y, m.z - midF[i].z};
      const float d2 = fdot(dv, dv);
      const float ee = eM + midF[i].w;
      const float e2 = 2.0f * nrm(dv) * ee + ee * ee + 4.0f * kU * d2 + kFloor;
      if (d2 + e2 < (float)kMergeDistSq) return 0;
      if (d2 - e2 < (float)kMergeDistSq) return -1;
    }
    if (count >= kMaxContacts) return 0;
    const V3<float> ra = qrotate(qaInv, xA);
    const V3<float> rb = qrotate(qbInv, fsub(xB, F.d));
    NewContactF &c = outF[count];
    c.feature = key;
    c.ra[0] = ra.x; c.ra[1] = ra.y; c.ra[2] = ra.z;
    c.rb[0] = rb.x; c.rb[1] = rb.y; c.rb[2] = rb.z;
    midF[count] = make_float4(m.x, m.y, m.z, eM);
    count++;
    return 1;
  }
  // refAx: the reference face axis in f64; ibAx: the incident box's axes in
  // f64 (the orientation decisions use the reference's own f64 expressions).
  __device__ int build(bool refIsA, int refAxis, D3 nAB, D3 refAx, const D3 *ibAx) {
    const D3 outward = refIsA ? nAB : neg(nAB);
    const double s = dt3(outward, refAx) >= 0 ? 1 : -1;
    const D3 fN64 = scl(refAx, s);
    int incAxis = 0;
    double best = -INFINITY, dots[3];
    for (int i = 0; i < 3; i++) {
      dots[i] = dt3(ibAx[i], fN64);
      const double dd = fabs(dots[i]);
      if (dd > best) {
        best = dd;
        incAxis = i;
      }
    }
    const float si = dots[incAxis] > 0 ? -1.f : 1.f;
    // the geometry in f32
    const V3<float> zero{0.f, 0.f, 0.f};
    const V3<float> *rAx = refIsA ? F.ax : F.bx;
    const V3<float> *iAx = refIsA ? F.bx : F.ax;
    const float *rH = refIsA ? F.ha : F.hb;
    const float *iH = refIsA ? F.hb : F.ha;
    const V3<float> rC = refIsA ? zero : F.d, iC = refIsA ? F.d : zero;
    const float eD = kU * nrm(F.d) + kFloor;
    const float eRC = refIsA ? 0.f : eD, eIC = refIsA ? eD : 0.f;
    const V3<float> fN{rAx[refAxis].x * (float)s, rAx[refAxis].y * (float)s, rAx[refAxis].z * (float)s};
    const float hR = rH[refAxis];
    const V3<float> fC = fadds(rC, fN, hR);
    const float eFC = eRC + kEA * hR + 3.0f * kU * (nrm(rC) + hR) + kFloor;
    const int u0 = refAxis == 0 ? 1 : 0, v0 = refAxis == 2 ? 1 : 2;
    const V3<float> fU = rAx[u0], fV = rAx[v0];
    const float fEU = rH[u0], fEV = rH[v0];
    const int u1 = incAxis == 0 ? 1 : 0, v1 = incAxis == 2 ? 1 : 2;
    const V3<float> fn{iAx[incAxis].x * si, iAx[incAxis].y * si, iAx[incAxis].z * si};
    const float hI = iH[incAxis], eU = iH[u1], eV = iH[v1];
    const V3<float> fc = fadds(iC, fn, hI);
    const float eCorner = eIC + kEA * (hI + eU + eV) + 5.0f * kU * (nrm(iC) + hI + eU + eV) + kFloor;
    float4 P[kPolyCap], Q[kPolyCap];
    for (int i = 0; i < 4; i++) {
      const float su = (i == 0 || i == 3) ? 1.f : -1.f;
      const float sv = (i == 0 || i == 1) ? 1.f : -1.f;
      const V3<float> c = fadds(fadds(fc, iAx[u1], eU * su), iAx[v1], eV * sv);
      P[i] = make_float4(c.x, c.y, c.z, eCorner);
    }
    int n = 4;
    const float nFC = nrm(fC);
    for (int k = 0; k < 4; k++) {
      const V3<float> ax = k < 2 ? fU : fV;
      const float sg = (k & 1) ? -1.f : 1.f;
      const V3<float> pn{ax.x * sg, ax.y * sg, ax.z * sg};
      const float ext = k < 2 ? fEU : fEV;
      const float po = fdot(pn, fC) + ext;
      const float ePo = kEA * nFC + eFC + 3.0f * kU * nFC + kU * (fabsf(po) + ext) + kFloor;
      n = (k & 1) ? clipF(Q, n, pn, po, ePo, P) : clipF(P, n, pn, po, ePo, Q);
      if (n < 0) return -1;
      if (n == 0) return 0;
    }
    count = 0;
    uint32_t prefix = (uint32_t)(refIsA ? kFaceA : kFaceB) << 24;
    prefix |= (uint32_t)(refAxis & 0xff) << 16;
    prefix |= (uint32_t)(incAxis & 0xff) << 8;
    float4 midF[kMaxContacts];
    count = 0;
    for (int i = 0; i < n && count < kMaxContacts; i++) {
      const V3<float> p{P[i].x, P[i].y, P[i].z};
      const V3<float> pc = fsub(p, fC);
      const float dist = fdot(pc, fN);
      const float eDist = P[i].w + eFC + kEA * nrm(pc) + 4.0f * kU * (nrm(p) + nFC) + kFloor;
      if (dist - eDist > (float)kPlaneEps) continue;
      if (dist + eDist > (float)kPlaneEps) return -1;
      const V3<float> proj = fadds(p, fN, -dist);
      const float eProj = P[i].w + kEA * fabsf(dist) + eDist + 2.0f * kU * (nrm(p) + fabsf(dist)) + kFloor;
      const int r = refIsA ? addContactF(proj, eProj, p, P[i].w, prefix | (uint32_t)(i & 0xff), midF)
                           : addContactF(p, P[i].w, proj, eProj, prefix | (uint32_t)(i & 0xff), midF);
      if (r < 0) return -1;
    }
    if (!count) return -1;  // the support-point contact is built in f64
    return count;
  }
};

__device__ BodyD load_body(const World &w, int i) {
  BodyD b;
  const D4 p = w.b.pos[i];
  const float4 q = w.b.quat[i];
  const D4 s = w.b.size[i];
  b.p = mk(p.x, p.y, p.z);
  b.q = QD{(double)q.x, (double)q.y, (double)q.z, (double)q.w};
  b.half = mk(s.x * 0.5, s.y * 0.5, s.z * 0.5);
  b.sphere = (w.b.flags0[i] & kBodySphere) != 0;
  // size.w is the broad phase's reach (the bounding radius plus the contact
  // offset under AVBD_CONTACT_MATERIALS); a sphere's own radius is half its
  // diameter (Rigid.sphere, src/physics/rigid.js:105-133)
  b.radius = (w.b.contactOffset && b.sphere) ? s.x * 0.5 : s.w;
  return b;
}

// The pair's contact skin (AVBD_CONTACT_MATERIALS: the sum of the contact
// offsets; 0 for the CPU engine's collider).
__device__ __forceinline__ double pair_skin(const World &w, int ia, int ib) {
  return w.b.contactOffset ? w.b.contactOffset[ia] + w.b.contactOffset[ib] : 0.0;
}

// transportComponents / transportPenalty (manifold.js:100-162)
__device__ void transport(double *lam, double *pen, const double *ob, const double *nb) {
  const double x = lam[0], y = lam[1], z = lam[2];
  const double kx = pen[0], ky = pen[1], kz = pen[2];
  double lo[3], po[3];
  for (int r = 0; r < 3; r++) {
    const int n = r * 3;
    const double dx = nb[n] * ob[0] + nb[n + 1] * ob[1] + nb[n + 2] * ob[2];
    const double dy = nb[n] * ob[3] + nb[n + 1] * ob[4] + nb[n + 2] * ob[5];
    const double dz = nb[n] * ob[6] + nb[n + 1] * ob[7] + nb[n + 2] * ob[8];
    lo[r] = x * dx + y * dy + z * dz;
    po[r] = kx * dx * dx + ky * dy * dy + kz * dz * dz;
  }
  for (int r = 0; r < 3; r++) {
    lam[r] = lo[r];
    pen[r] = po[r];
  }
}

// ---------------------------------------------------------------------------
// Manifold output: merge with the previous step's manifold by feature ID,
// C*(x_t) + margin, warm start (manifold.js:214-318).
// ---------------------------------------------------------------------------

// Box pairs, in f32 in A's frame (xA - xB = R_A rA - R_B rB - (pB - pA)); the
// outputs are stored in f32.
__device__ void write_manifold_materials(const World &w, int c, int ia, int ib, const BodyD &A, const BodyD &B,
                                         const D3 *ncA, const D3 *ncB, const uint32_t *feat, int num,
                                         const double *basis);

// Contact i of a box pair's manifold: matched with the previous step's by
// feature ID, C*(x_t) + margin, warm start.
__device__ __forceinline__ void write_box_contact(const World &w, int c, int i, int pi, int oldNum, const BodyD &A,
                                                  const BodyD &B, const NewContactF &nc, const float *bf) {
  const SolverParams &P = w.p;
  const Q4<float> qa{(float)A.q.x, (float)A.q.y, (float)A.q.z, (float)A.q.w};
  const Q4<float> qb{(float)B.q.x, (float)B.q.y, (float)B.q.z, (float)B.q.w};
  const V3<float> dAB{(float)(B.p.x - A.p.x), (float)(B.p.y - A.p.y), (float)(B.p.z - A.p.z)};
  const float alpha = (float)P.alpha, gamma = (float)P.gamma;
  const float kmin = (float)P.penaltyMin, kmax = (float)P.penaltyMax, margin = (float)P.margin;
  V3<float> rA{nc.ra[0], nc.ra[1], nc.ra[2]};
  V3<float> rB{nc.rb[0], nc.rb[1], nc.rb[2]};
  float lam[3] = {0.f, 0.f, 0.f}, pen[3] = {0.f, 0.f, 0.f};
  bool stick = false;
  for (int j = 0; j < oldNum; j++) {
    const int os = pi * kMaxContacts + j;
    if (nc.feature == w.prev.feat[os]) {
      const float4 ok = w.prev.cK[os], ol = w.prev.cL[os];
      lam[0] = ol.x; lam[1] = ol.y; lam[2] = ol.z;
      pen[0] = ok.x; pen[1] = ok.y; pen[2] = ok.z;
      stick = ol.w != 0.0f;
      if (stick) {  // a stuck box contact keeps its anchors (manifold.js:279-282)
        const float4 oa = w.prev.rA[os], ob = w.prev.rB[os];
        rA = V3<float>{oa.x, oa.y, oa.z};
        rB = V3<float>{ob.x, ob.y, ob.z};
      }
      break;
    }
  }
  const V3<float> rAw = qrotate(qa, rA), rBw = qrotate(qb, rB);
  const V3<float> dd{rAw.x - rBw.x - dAB.x, rAw.y - rBw.y - dAB.y, rAw.z - rBw.z - dAB.z};
  float C0[3];
  for (int k = 0; k < 3; k++) C0[k] = bf[3 * k] * dd.x + bf[3 * k + 1] * dd.y + bf[3 * k + 2] * dd.z;
  C0[0] += margin;
  if (!P.postStabilize)
    for (int k = 0; k < 3; k++) lam[k] = (lam[k] * alpha) * gamma;
  for (int k = 0; k < 3; k++) {
    const float x = pen[k] * gamma;  // clamp(gamma k, kmin, kmax), NaN propagating
    pen[k] = x != x ? x : fmaxf(kmin, fminf(kmax, x));
  }
  const int s = c * kMaxContacts + i;
  w.cur.feat[s] = nc.feature;
  w.cur.rA[s] = make_float4(rA.x, rA.y, rA.z, 0.f);
  w.cur.rB[s] = make_float4(rB.x, rB.y, rB.z, 0.f);
  w.cur.cA[s] = make_float4(rAw.x, rAw.y, rAw.z, C0[0]);
  w.cur.cB[s] = make_float4(rBw.x, rBw.y, rBw.z, C0[1]);
  w.cur.cK[s] = make_float4(pen[0], pen[1], pen[2], C0[2]);
  w.cur.cL[s] = make_float4(lam[0], lam[1], lam[2], stick ? 1.f : 0.f);
}

__device__ __forceinline__ void write_box_header(const World &w, int c, int ia, int ib, const double *basis,
                                                 const float *bf) {
  const double friction = sqrt(w.b.friction[ia] * w.b.friction[ib]);
  for (int k = 0; k < 9; k++) w.cur.basisD[c * 9 + k] = basis[k];
  w.cur.basis0[c] = make_float4(bf[0], bf[1], bf[2], (float)friction);
  w.cur.basis1[c] = make_float4(bf[3], bf[4], bf[5], 0.f);
  w.cur.basis2[c] = make_float4(bf[6], bf[7], bf[8], 0.f);
}

__device__ void write_box_manifold(const World &w, int c, int ia, int ib, const BodyD &A, const BodyD &B,
                                   const NewContactF *nc, int num, const double *basis) {
  const SolverParams &P = w.p;
  if (P.contactModel) {
    D3 ra[kMaxContacts], rb[kMaxContacts];
    uint32_t ft[kMaxContacts];
    for (int i = 0; i < num; i++) {
      ra[i] = mk(nc[i].ra[0], nc[i].ra[1], nc[i].ra[2]);
      rb[i] = mk(nc[i].rb[0], nc[i].rb[1], nc[i].rb[2]);
      ft[i] = nc[i].feature;
    }
    write_manifold_materials(w, c, ia, ib, A, B, ra, rb, ft, num, basis);
    return;
  }
  w.cur.count[c] = num;
  if (num == 0) return;
  const int pi = w.g.candPrev[c];
  const int oldNum = pi >= 0 ? w.prev.count[pi] : 0;
  float bf[9];
  for (int k = 0; k < 9; k++) bf[k] = (float)basis[k];
  for (int i = 0; i < num; i++) write_box_contact(w, c, i, pi, oldNum, A, B, nc[i], bf);
  write_box_header(w, c, ia, ib, basis, bf);
}

// Pairs with a sphere, in f64: the basis-compatibility test and the
// transport of lambda and k into the new basis (manifold.js:222-270).
__device__ void write_sphere_manifold(const World &w, int c, int ia, int ib, const BodyD &A, const BodyD &B,
                                      const NewContact *nc, int num, const double *basis) {
  const SolverParams &P = w.p;
  if (P.contactModel) {
    D3 ra[kMaxContacts], rb[kMaxContacts];
    uint32_t ft[kMaxContacts];
    for (int i = 0; i < num; i++) {
      ra[i] = nc[i].rA;
      rb[i] = nc[i].rB;
      ft[i] = nc[i].feature;
    }
    write_manifold_materials(w, c, ia, ib, A, B, ra, rb, ft, num, basis);
    return;
  }
  w.cur.count[c] = num;
  if (num == 0) return;
  const int pi = w.g.candPrev[c];
  const int oldNum = pi >= 0 ? w.prev.count[pi] : 0;
  double oldBasis[9];
  if (oldNum > 0)
    for (int k = 0; k < 9; k++) oldBasis[k] = w.prev.basisD[pi * 9 + k];
  const double friction = sqrt(w.b.friction[ia] * w.b.friction[ib]);
  const bool compatible =
      oldNum == 0 || (oldBasis[0] * basis[0] + oldBasis[1] * basis[1] + oldBasis[2] * basis[2]) > 0.85;
  const QD qA = A.q, qB = B.q;
  for (int i = 0; i < num; i++) {
    const D3 rA = nc[i].rA, rB = nc[i].rB;
    double lam[3] = {0, 0, 0}, pen[3] = {0, 0, 0};
    bool stick = false;
    for (int j = 0; j < oldNum; j++) {
      const int os = pi * kMaxContacts + j;
      if (compatible && nc[i].feature == w.prev.feat[os]) {
        const float4 ok = w.prev.cK[os], ol = w.prev.cL[os];
        lam[0] = ol.x; lam[1] = ol.y; lam[2] = ol.z;
        pen[0] = ok.x; pen[1] = ok.y; pen[2] = ok.z;
        stick = ol.w != 0.0f;
        transport(lam, pen, oldBasis, basis);
        break;
      }
    }
    // C*(x_t) and warm start (manifold.js:292-315)
    const D3 xA = add(rot(qA, rA), A.p);
    const D3 xB = add(rot(qB, rB), B.p);
    const D3 d = sub(xA, xB);
    double C0[3];
    C0[0] = basis[0] * d.x + basis[1] * d.y + basis[2] * d.z;
    C0[1] = basis[3] * d.x + basis[4] * d.y + basis[5] * d.z;
    C0[2] = basis[6] * d.x + basis[7] * d.y + basis[8] * d.z;
    C0[0] += P.margin;
    if (!P.postStabilize) {
      for (int k = 0; k < 3; k++) {
        lam[k] = lam[k] * P.alpha;
        lam[k] = lam[k] * P.gamma;
      }
    }
    for (int k = 0; k < 3; k++) pen[k] = clampd(pen[k] * P.gamma, P.penaltyMin, P.penaltyMax);
    const D3 rAw = rot(qA, rA), rBw = rot(qB, rB);
    const int s = c * kMaxContacts + i;
    w.cur.feat[s] = nc[i].feature;
    w.cur.rA[s] = make_float4((float)rA.x, (float)rA.y, (float)rA.z, 0.f);
    w.cur.rB[s] = make_float4((float)rB.x, (float)rB.y, (float)rB.z, 0.f);
    w.cur.cA[s] = make_float4((float)rAw.x, (float)rAw.y, (float)rAw.z, (float)C0[0]);
    w.cur.cB[s] = make_float4((float)rBw.x, (float)rBw.y, (float)rBw.z, (float)C0[1]);
    w.cur.cK[s] = make_float4((float)pen[0], (float)pen[1], (float)pen[2], (float)C0[2]);
    w.cur.cL[s] = make_float4((float)lam[0], (float)lam[1], (float)lam[2], stick ? 1.f : 0.f);
  }
  for (int k = 0; k < 9; k++) w.cur.basisD[c * 9 + k] = basis[k];
  w.cur.basis0[c] = make_float4((float)basis[0], (float)basis[1], (float)basis[2], (float)friction);
  w.cur.basis1[c] = make_float4((float)basis[3], (float)basis[4], (float)basis[5], 1.f);  // .w: sphere pair
  w.cur.basis2[c] = make_float4((float)basis[6], (float)basis[7], (float)basis[8], 0.f);
}

// AVBD_CONTACT_MATERIALS: the WebGPU engine's manifold warm start with its
// contact extensions (src/physics/gpu/shaders.js:1105-1366), in f64 for box
// and sphere pairs alike (an opt-in model; the default path above keeps the
// f32 box merge). Pair materials: friction as the geometric mean of the
// static and of the dynamic coefficients, restitution as the max, contact
// and rest offsets summed. A new contact matches the old one with its
// feature ID, else the nearest old contact within the persistence distance
// (separation, tangential offset and midpoint distance within it), each old
// contact claimed once and only when the normals agree (dot > 0.85);
// multiplier and penalty are transported into the new basis; a matched
// static box contact keeps its anchors; a new contact starts static. C0 on
// the normal is measured to the rest distance; a new or re-armed impact
// (the old contact still outside rest and without a bias) faster than the
// restitution threshold gets a one-frame bias.
struct MaterialsPair {
  int pi, oldNum;  // the previous manifold and its contacts
  double ob[9];    // its basis
  double mus, mud, restitution, contactDistance, restDistance, persistence, psq;
  bool compatible, curved;
};

__device__ MaterialsPair materials_pair(const World &w, int c, int ia, int ib, const BodyD &A, const BodyD &B,
                                        const double *basis) {
  MaterialsPair m;
  m.pi = w.g.candPrev[c];
  m.oldNum = m.pi >= 0 ? w.prev.count[m.pi] : 0;
  for (int k = 0; k < 9; k++) m.ob[k] = m.oldNum > 0 ? w.prev.basisD[m.pi * 9 + k] : basis[k];
  const D4 ma = w.b.mat[ia], mb = w.b.mat[ib];
  m.mus = sqrt(ma.x * mb.x);
  m.mud = sqrt(ma.y * mb.y);
  m.restitution = ma.z > mb.z ? ma.z : (mb.z > ma.z ? mb.z : ma.z);
  m.contactDistance = w.b.contactOffset[ia] + w.b.contactOffset[ib];
  m.restDistance = ma.w + mb.w;
  m.compatible = m.oldNum > 0 && (m.ob[0] * basis[0] + m.ob[1] * basis[1] + m.ob[2] * basis[2]) > 0.85;
  const double minA = fmin(A.half.x, fmin(A.half.y, A.half.z)), minB = fmin(B.half.x, fmin(B.half.y, B.half.z));
  const double minExtent = 2.0 * fmin(minA, minB);
  m.persistence = fmax(w.p.contactPersistence, fmax(m.contactDistance, minExtent * 0.02));
  m.psq = m.persistence * m.persistence;
  m.curved = A.sphere || B.sphere;
  return m;
}

__device__ __forceinline__ D3 midpoint(D3 a, D3 b) {
  return mk((a.x + b.x) * 0.5, (a.y + b.y) * 0.5, (a.z + b.z) * 0.5);
}
__device__ __forceinline__ double dist_sq(D3 a, D3 b) {
  const D3 d = mk(a.x - b.x, a.y - b.y, a.z - b.z);
  return d.x * d.x + d.y * d.y + d.z * d.z;
}

// Old contact os at the new poses: its midpoint, and whether its separation
// and tangential offset along the new normal keep it a candidate.
__device__ __forceinline__ bool old_contact(const World &w, const MaterialsPair &m, int os, const BodyD &A,
                                            const BodyD &B, D3 nN, D3 &mid) {
  const float4 oa = w.prev.rA[os], obb = w.prev.rB[os];
  const D3 oxA = add(rot(A.q, mk(oa.x, oa.y, oa.z)), A.p);
  const D3 oxB = add(rot(B.q, mk(obb.x, obb.y, obb.z)), B.p);
  const D3 od = sub(oxA, oxB);
  const double sep = nN.x * od.x + nN.y * od.y + nN.z * od.z;
  const D3 td = mk(od.x - nN.x * sep, od.y - nN.y * sep, od.z - nN.z * sep);
  mid = midpoint(oxA, oxB);
  return !(sep > m.contactDistance + m.persistence) && !(td.x * td.x + td.y * td.y + td.z * td.z > m.psq);
}

// New contact i, matched with old contact `match` (-1: none).
__device__ void write_materials_contact(const World &w, int c, int i, int ia, int ib, const BodyD &A, const BodyD &B,
                                        const MaterialsPair &m, const double *basis, D3 rA, D3 rB, uint32_t feature,
                                        int match) {
  const SolverParams &P = w.p;
  const double *ob = m.ob;
  const bool found = match >= 0;
  double lam[3] = {0, 0, 0}, pen[3] = {0, 0, 0};
  bool stick = true, priorOut = false, priorBias = false;
  if (found) {
    const int os = m.pi * kMaxContacts + match;
    const float4 ok = w.prev.cK[os], ol = w.prev.cL[os];
    for (int r = 0; r < 3; r++) {  // transport into the new basis (shaders.js:1050-1085)
      const double *nr = &basis[r * 3];
      const double a = nr[0] * ob[0] + nr[1] * ob[1] + nr[2] * ob[2];
      const double b = nr[0] * ob[3] + nr[1] * ob[4] + nr[2] * ob[5];
      const double cc = nr[0] * ob[6] + nr[1] * ob[7] + nr[2] * ob[8];
      pen[r] = (double)ok.x * (a * a) + (double)ok.y * (b * b) + (double)ok.z * (cc * cc);
      lam[r] = (double)ol.x * a + (double)ol.y * b + (double)ol.z * cc;
    }
    stick = ol.w != 0.0f;
    priorOut = w.prev.cA[os].w > 0.0f;
    priorBias = w.prev.cX[os] > 0.0f;
    if (stick && !m.curved) {
      const float4 oa = w.prev.rA[os], obb = w.prev.rB[os];
      rA = mk(oa.x, oa.y, oa.z);
      rB = mk(obb.x, obb.y, obb.z);
    }
  }
  const D3 nN = mk(basis[0], basis[1], basis[2]);
  const D3 rAw = rot(A.q, rA), rBw = rot(B.q, rB);
  const D3 d = sub(add(rAw, A.p), add(rBw, B.p));
  double C0[3];
  C0[0] = basis[0] * d.x + basis[1] * d.y + basis[2] * d.z - m.restDistance;
  C0[1] = basis[3] * d.x + basis[4] * d.y + basis[5] * d.z;
  C0[2] = basis[6] * d.x + basis[7] * d.y + basis[8] * d.z;
  double bias = 0.0;
  if ((!found || (priorOut && !priorBias)) && m.restitution > 0.0) {
    const float4 vA = w.b.vel[ia], wA = w.b.omega[ia], vB = w.b.vel[ib], wB = w.b.omega[ib];
    const D3 ua = add(mk(vA.x, vA.y, vA.z), crs(mk(wA.x, wA.y, wA.z), rAw));
    const D3 ub = add(mk(vB.x, vB.y, vB.z), crs(mk(wB.x, wB.y, wB.z), rBw));
    const D3 rel = sub(ua, ub);
    const double vn = nN.x * rel.x + nN.y * rel.y + nN.z * rel.z;
    const double closing = fmax(0.0, -vn * P.dt), toRest = fmax(0.0, C0[0]);
    if (vn < -P.restitutionThreshold && closing > toRest) bias = m.restitution * (closing - toRest);
  }
  if (!P.postStabilize)
    for (int k = 0; k < 3; k++) lam[k] = lam[k] * P.alpha * P.gamma;
  for (int k = 0; k < 3; k++) pen[k] = clampd(pen[k] * P.gamma, P.penaltyMin, P.penaltyMax);
  const int s = c * kMaxContacts + i;
  w.cur.feat[s] = feature;
  w.cur.rA[s] = make_float4((float)rA.x, (float)rA.y, (float)rA.z, 0.f);
  w.cur.rB[s] = make_float4((float)rB.x, (float)rB.y, (float)rB.z, 0.f);
  w.cur.cA[s] = make_float4((float)rAw.x, (float)rAw.y, (float)rAw.z, (float)C0[0]);
  w.cur.cB[s] = make_float4((float)rBw.x, (float)rBw.y, (float)rBw.z, (float)C0[1]);
  w.cur.cK[s] = make_float4((float)pen[0], (float)pen[1], (float)pen[2], (float)C0[2]);
  w.cur.cL[s] = make_float4((float)lam[0], (float)lam[1], (float)lam[2], stick ? 1.f : 0.f);
  w.cur.cX[s] = (float)bias;
}

__device__ __forceinline__ void write_materials_header(const World &w, int c, const MaterialsPair &m,
                                                       const double *basis) {
  for (int k = 0; k < 9; k++) w.cur.basisD[c * 9 + k] = basis[k];
  const float flags = (m.curved ? 1.f : 0.f) + (m.contactDistance > 0.0 ? 2.f : 0.f);
  w.cur.basis0[c] = make_float4((float)basis[0], (float)basis[1], (float)basis[2], (float)m.mus);
  w.cur.basis1[c] = make_float4((float)basis[3], (float)basis[4], (float)basis[5], flags);
  w.cur.basis2[c] = make_float4((float)basis[6], (float)basis[7], (float)basis[8], (float)m.mud);
}

__device__ void write_manifold_materials(const World &w, int c, int ia, int ib, const BodyD &A, const BodyD &B,
                                         const D3 *ncA, const D3 *ncB, const uint32_t *feat, int num,
                                         const double *basis) {
  w.cur.count[c] = num;
  if (num == 0) return;
  const MaterialsPair m = materials_pair(w, c, ia, ib, A, B, basis);
  const D3 nN = mk(basis[0], basis[1], basis[2]);
  unsigned used = 0u;
  for (int i = 0; i < num; i++) {
    int match = -1;
    double best = m.psq;
    if (m.compatible) {
      const D3 mid = midpoint(add(rot(A.q, ncA[i]), A.p), add(rot(B.q, ncB[i]), B.p));
      for (int j = 0; j < m.oldNum; j++) {
        if (used & (1u << j)) continue;
        const int os = m.pi * kMaxContacts + j;
        const bool same = w.prev.feat[os] == feat[i];
        if (m.curved && same) {
          match = j;
          break;
        }
        D3 oldMid;
        if (!old_contact(w, m, os, A, B, nN, oldMid)) continue;
        const double mdSq = dist_sq(mid, oldMid);
        if (mdSq > m.psq) continue;
        if (same) {
          match = j;
          break;
        }
        if (match < 0 || mdSq < best) {
          match = j;
          best = mdSq;
        }
      }
    }
    if (match >= 0) used |= 1u << match;
    write_materials_contact(w, c, i, ia, ib, A, B, m, basis, ncA[i], ncB[i], feat[i], match);
  }
  write_materials_header(w, c, m, basis);
}

// Append to one of the work lists, one atomic per coalesced group of lanes.
__device__ __forceinline__ int push_slot(int *counter) {
  const unsigned m = __activemask();
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(counter, __popc(m));
  base = __shfl_sync(m, base, leader);
  return base + __popc(m & ((1u << lane) - 1u));
}

__device__ __forceinline__ void push_exact(const World &w, int c) {
  w.g.npExact[push_slot(&w.ctl->npCount[2])] = c;
}

// Lists of up to kGroupMax box pairs take sixteen lanes a pair, longer ones a
// pair a thread: that keeps every sub-partition's FP64 pipe busy either way,
// and then needs about half the warp instructions (narrow phase of a batch with
// 10,257 such pairs: 0.70 ms on lanes, 0.72 by threads; of a crushed pyramid
// with 37,825: 1.24 and 0.93).
// In a scene at rest nearly all pairs touch, and take the same path: every box
// pair is in the list under the materials model, and boxes aligned with one
// another are undecided under both. A warp of 32 pairs then hardly diverges,
// and threads are ahead from some 6,000 pairs on (materials: 4,500, 5,900 with
// the boxes turned about the vertical). 13,514 aligned pairs, materials: 463 us on
// lanes, 193 by threads; 12,706, plain: 247 and 142. Where the pairs are of
// several kinds it is the other way round up to kGroupMax (materials, a landing
// pile's 8,544: 133 us on lanes, 263 by threads; plain, a crushed pyramid's 7,649:
// 300 and 606). So the line is kGroupMaxAlike when the box pairs that stand
// `apart` are at most a third as many as the list: those decided without it, and
// those in it (pairs with a skin) that a face separates, which long lists count
// (2 us).
constexpr int kGroupMax = 16384, kGroupMaxAlike = 6144;
__device__ __forceinline__ int pairs_per_warp(int n, int apart) {
  return n > kGroupMax || (n > kGroupMaxAlike && apart <= n / 3) ? 32 : 2;
}

// Whether no face axis of two boxes separates them by more than the skin, in
// f32 and as good as that is: only what pairs_per_warp counts.
__device__ __forceinline__ bool faces_touch(const World &w, int ia, int ib, float skin) {
  const float4 qa = w.b.quat[ia], qb = w.b.quat[ib];
  const D4 pa = w.b.pos[ia], pb = w.b.pos[ib], sa = w.b.size[ia], sb = w.b.size[ib];
  const V3<float> d{(float)(pb.x - pa.x), (float)(pb.y - pa.y), (float)(pb.z - pa.z)};
  const float ha[3] = {0.5f * (float)sa.x, 0.5f * (float)sa.y, 0.5f * (float)sa.z};
  const float hb[3] = {0.5f * (float)sb.x, 0.5f * (float)sb.y, 0.5f * (float)sb.z};
  // B's centre and axes in A's frame
  const Q4<float> inv{-qa.x, -qa.y, -qa.z, qa.w}, q{qb.x, qb.y, qb.z, qb.w};
  const V3<float> c = qrotate(inv, d);
  const V3<float> bx[3] = {qrotate(inv, qrotate(q, V3<float>{1, 0, 0})), qrotate(inv, qrotate(q, V3<float>{0, 1, 0})),
                           qrotate(inv, qrotate(q, V3<float>{0, 0, 1}))};
  const float ca[3] = {c.x, c.y, c.z};
  bool touch = true;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float b[3] = {i == 0 ? bx[0].x : i == 1 ? bx[0].y : bx[0].z, i == 0 ? bx[1].x : i == 1 ? bx[1].y : bx[1].z,
                        i == 0 ? bx[2].x : i == 1 ? bx[2].y : bx[2].z};
    touch = touch && fabsf(ca[i]) <= ha[i] + hb[0] * fabsf(b[0]) + hb[1] * fabsf(b[1]) + hb[2] * fabsf(b[2]) + skin;
    const V3<float> n = bx[i];
    touch = touch && fabsf(c.x * n.x + c.y * n.y + c.z * n.z) <=
                         hb[i] + ha[0] * fabsf(n.x) + ha[1] * fabsf(n.y) + ha[2] * fabsf(n.z) + skin;
  }
  return touch;
}

// The face axis among `mask` (bits 0-5: faces of A, then of B) with the
// largest exact separation, the first on ties: the f64 expressions of
// testAxis (collide.js:291-324) for just those axes.
__device__ int exact_best_face(const BodyD &A, const BodyD &B, int mask) {
  const D3 e3[3] = {mk(1, 0, 0), mk(0, 1, 0), mk(0, 0, 1)};
  D3 ax[3], bx[3];
  for (int i = 0; i < 3; i++) {
    ax[i] = rot(A.q, e3[i]);
    bx[i] = rot(B.q, e3[i]);
  }
  const D3 delta = sub(B.p, A.p);
  int best = -1;
  double bestSep = -INFINITY;
  for (int k = 0; k < 6; k++) {
    if (!((mask >> k) & 1)) continue;
    const D3 axis = k < 3 ? ax[k] : bx[k - 3];
    const double lenSq = axis.x * axis.x + axis.y * axis.y + axis.z * axis.z;
    const double invLen = 1.0 / sqrt(lenSq);
    D3 n = scl(axis, invLen);
    if (dt3(n, delta) < 0) n = neg(n);
    const double distance = fabs(dt3(delta, n));
    const double rA = A.half.x * fabs(dt3(n, ax[0])) + A.half.y * fabs(dt3(n, ax[1])) + A.half.z * fabs(dt3(n, ax[2]));
    const double rB = B.half.x * fabs(dt3(n, bx[0])) + B.half.y * fabs(dt3(n, bx[1])) + B.half.z * fabs(dt3(n, bx[2]));
    const double separation = distance - (rA + rB);
    if (best < 0 || separation > bestSep) {
      best = k;
      bestSep = separation;
    }
  }
  return best;
}

// The candidate's slot among the previous step's manifolds, searched in its
// body A's run of them (-1: none with contacts).
__device__ __forceinline__ int previous_slot(const World &w, uint64_t key, int a) {
  if (w.ctl->prevCandidates <= 0) return -1;
  const int end = w.g.prevStart[a + 1];
  int l = w.g.prevStart[a], h = end;
  while (l < h) {
    const int m = (l + h) >> 1;
    if (w.prev.key[m] < key) l = m + 1;
    else h = m;
  }
  return l < end && w.prev.key[l] == key && w.prev.count[l] > 0 ? l : -1;
}

// 1. Every candidate: its previous manifold, and the f32 SAT. Separated pairs get count 0; box pairs
//    with a certain winning axis go to the face or edge list, undecided ones
//    to the exact list, sphere pairs to a list that fills the edge list's
//    array from its far end (a candidate is in one list only).
__global__ void __launch_bounds__(256) classify_kernel(World w) {
  await_previous();
  const int total = *((volatile int *)&w.ctl->numCandidates);
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
    const uint64_t key = w.g.candKey[c];
    const int ia = (int)(key >> 32), ib = (int)(key & 0xffffffffu);
    w.g.candPrev[c] = previous_slot(w, key, ia);
    w.cur.key[c] = key;
    const BodyD A = load_body(w, ia), B = load_body(w, ib);
    if (A.sphere || B.sphere) {
      w.g.npEdge[w.g.candCap - 1 - push_slot(&w.ctl->npCount[4])].x = c;
      continue;
    }
    // pairs with a contact skin (speculative contacts: the f32 certification
    // covers the skin-free tests) go to the exact collider
    const double skin = pair_skin(w, ia, ib);
    if (skin != 0.0) {
      push_exact(w, c);
      if (total > kGroupMaxAlike && !faces_touch(w, ia, ib, (float)skin)) push_slot(&w.ctl->npApart);
      continue;
    }
    bool refIsA = true;
    int axA = 0, axB = 0, tieMask = 0;
    const int r = classify_f32(make_boxf(A, B), refIsA, axA, axB, tieMask);
    if (r == kSeparated) {
      w.cur.count[c] = 0;
    } else if (r == kFaceWin) {
      w.g.npFace[push_slot(&w.ctl->npCount[0])] = make_int2(c, (refIsA ? 4 : 0) | axA);
    } else if (r == kFaceTie) {
      w.g.npFace[push_slot(&w.ctl->npCount[0])] = make_int2(c, tieMask << 8);
    } else if (r == kEdgeWin) {
      w.g.npEdge[push_slot(&w.ctl->npCount[1])] = make_int2(c, axA * 3 + axB);
    } else {
      push_exact(w, c);
    }
  }
}

// 2. A face manifold: the exact normal and basis in f64, the clipping in f32
//    with certified decisions; an undecided pair moves to the late list.
__device__ __noinline__ void face_pair(const World &w, int t) {
  const int2 e = w.g.npFace[t];
  const int c = e.x;
  bool refIsA = (e.y & 4) != 0;
  int refAxis = e.y & 3;
  const uint64_t key = w.g.candKey[c];
  const int ia = (int)(key >> 32), ib = (int)(key & 0xffffffffu);
  const BodyD A = load_body(w, ia), B = load_body(w, ib);
  if (e.y >> 8) {  // tied face axes: their exact separations decide (first largest wins)
    const int k = exact_best_face(A, B, e.y >> 8);
    refIsA = k < 3;
    refAxis = refIsA ? k : k - 3;
  }
  // f64: the reference axis, the incident box's axes, the exact normal
  const QD qRef = refIsA ? A.q : B.q, qInc = refIsA ? B.q : A.q;
  const D3 e3[3] = {mk(1, 0, 0), mk(0, 1, 0), mk(0, 0, 1)};
  const D3 refAx = rot(qRef, e3[refAxis]);
  const D3 ibAx[3] = {rot(qInc, e3[0]), rot(qInc, e3[1]), rot(qInc, e3[2])};
  const D3 n = Collider::axisNormal(refAx, sub(B.p, A.p));
  double basis[9];
  orthonormal(basis, neg(n));
  const BoxF F = make_boxf(A, B);
  NewContactF ncf[kMaxContacts];
  FaceF face(F, A, B, ncf);
  const int num = face.build(refIsA, refAxis, n, refAx, ibAx);
  if (num < 0) {
    w.g.npExact[w.g.candCap - 1 - push_slot(&w.ctl->npCount[3])] = c;
    return;
  }
  write_box_manifold(w, c, ia, ib, A, B, ncf, num, basis);
}

// 3. Edge-edge contacts (collide.js:475-493), exact f64.
__device__ __noinline__ void edge_pair(const World &w, int t) {
  const int2 e = w.g.npEdge[t];
  const int c = e.x, i = e.y / 3, j = e.y % 3;
  const uint64_t key = w.g.candKey[c];
  const int ia = (int)(key >> 32), ib = (int)(key & 0xffffffffu);
  const BodyD A = load_body(w, ia), B = load_body(w, ib);
  NewContact nc[2];
  Collider col(A, B, nc);
  Collider::makeOBB(col.boxA, A);
  Collider::makeOBB(col.boxB, B);
  const D3 delta = sub(col.boxB.c, col.boxA.c);
  const D3 n = Collider::axisNormal(crs(col.boxA.ax[i], col.boxB.ax[j]), delta);
  double basis[9];
  orthonormal(basis, neg(n));
  const int num = col.edgeContact(i, j, n);
  NewContactF ncf[2];
  for (int k = 0; k < num; k++) {
    ncf[k].feature = nc[k].feature;
    ncf[k].ra[0] = (float)nc[k].rA.x; ncf[k].ra[1] = (float)nc[k].rA.y; ncf[k].ra[2] = (float)nc[k].rA.z;
    ncf[k].rb[0] = (float)nc[k].rB.x; ncf[k].rb[1] = (float)nc[k].rB.y; ncf[k].rb[2] = (float)nc[k].rB.z;
  }
  write_box_manifold(w, c, ia, ib, A, B, ncf, num, basis);
}

// ---------------------------------------------------------------------------
// The exact collider of a box pair on sixteen lanes (collide.js:612-685): an
// SAT axis a lane, then a polygon vertex a lane. An FP64 warp instruction
// costs the same for one lane as for 32, and a pair decided by one thread is
// a chain of some 2,500 of them (150-230 us for a list of ten pairs); here it
// is about 500 (the list of a 200-box pile: 150 -> 39 us). Every value is
// formed by ColliderT's operations in their order, so the contacts are bitwise
// the serial collider's. Both halves of a warp run in step; `act` is false for
// a half without a box pair.
// ---------------------------------------------------------------------------
constexpr int kGroup = 16;

__device__ __forceinline__ double gshfl(double v, int src) { return __shfl_sync(0xffffffffu, v, src, kGroup); }
__device__ __forceinline__ D3 gshfl(D3 v, int src) {
  return D3{gshfl(v.x, src), gshfl(v.y, src), gshfl(v.z, src)};
}
__device__ __forceinline__ D3 pick3(bool c, D3 a, D3 b) { return D3{c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z}; }

// The lane of the group with the largest v among those with `on`, the first
// on ties (-1: none), as a loop of `v > best` over them finds it: a NaN that
// comes first stays, a later one is passed over. Compared as integers: a double
// compare is an FP64 warp instruction. (v + 0 makes -0 equal to +0.)
__device__ __forceinline__ int group_argmax(double v, bool on) {
  long long key = __double_as_longlong(v + 0.0);
  const bool nan = (key & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
  const unsigned mine = 0xffffu << (threadIdx.x & (32 - kGroup));
  const unsigned all = __ballot_sync(0xffffffffu, on) & mine, nans = __ballot_sync(0xffffffffu, on && nan);
  key ^= (key >> 63) & 0x7fffffffffffffffLL;
  int at = on && !nan ? (int)(threadIdx.x & (kGroup - 1)) : kGroup;
#pragma unroll
  for (int m = kGroup / 2; m > 0; m >>= 1) {
    const long long ok = __shfl_xor_sync(0xffffffffu, key, m, kGroup);
    const int oa = __shfl_xor_sync(0xffffffffu, at, m, kGroup);
    const bool take = oa < kGroup && (at >= kGroup || ok > key || (ok == key && oa < at));
    key = take ? ok : key;
    at = take ? oa : at;
  }
  const int first = __ffs(all) - 1;
  if (first >= 0 && ((nans >> first) & 1u)) return first & (kGroup - 1);
  return at < kGroup ? at : -1;
}

// Returns the contact count; a lane with slot >= 0 holds contact `slot` in nc.
__device__ int collide_group(const BodyD &A, const BodyD &B, double cd, bool act, D3 *poly, double *basis,
                             NewContactF &nc, int &slot) {
  const int gl = threadIdx.x & (kGroup - 1);
  const unsigned shift = threadIdx.x & (32 - kGroup);
  auto ballot = [&](bool p) { return (__ballot_sync(0xffffffffu, p) >> shift) & 0xffffu; };
  slot = -1;
  // box axes: lanes 0-2 A's, 3-5 B's
  const bool ofA = gl < 3;
  const QD q{ofA ? A.q.x : B.q.x, ofA ? A.q.y : B.q.y, ofA ? A.q.z : B.q.z, ofA ? A.q.w : B.q.w};
  const int ak = ofA ? gl : gl - 3;
  const D3 mine = rot(q, mk(ak == 0 ? 1.0 : 0.0, ak == 1 ? 1.0 : 0.0, ak == 2 ? 1.0 : 0.0));
  OBB a, b;
  a.c = A.p; a.h = A.half;
  b.c = B.p; b.h = B.half;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    a.ax[i] = gshfl(mine, i);
    b.ax[i] = gshfl(mine, 3 + i);
  }
  const D3 delta = sub(b.c, a.c);
  // testAxis (collide.js:291-324) of axis gl: faces of A, of B, then the edge pairs
  const int ek = gl < 6 ? 0 : min(gl - 6, 8);
  const D3 axis = pick3(gl < 6, mine, crs(gshfl(mine, ek / 3), gshfl(mine, 3 + ek % 3)));
  const double lenSq = axis.x * axis.x + axis.y * axis.y + axis.z * axis.z;
  const bool tested = gl < 15 && !(lenSq < geo::kSatEps);
  const double invLen = 1.0 / sqrt(lenSq);
  D3 n = scl(axis, invLen);
  if (dt3(n, delta) < 0) n = neg(n);
  const double distance = fabs(dt3(delta, n));
  const double rA = a.h.x * fabs(dt3(n, a.ax[0])) + a.h.y * fabs(dt3(n, a.ax[1])) + a.h.z * fabs(dt3(n, a.ax[2]));
  const double rB = b.h.x * fabs(dt3(n, b.ax[0])) + b.h.y * fabs(dt3(n, b.ax[1])) + b.h.z * fabs(dt3(n, b.ax[2]));
  const double sep = distance - (rA + rB);
  const bool separated = ballot(tested && sep > cd) != 0;
  const int fBest = group_argmax(sep, tested && gl < 6), eBest = group_argmax(sep, tested && gl >= 6);
  const double fSep = gshfl(sep, max(fBest, 0)), eSep = gshfl(sep, max(eBest, 0));
  const bool live = act && !separated && fBest >= 0;
  if (!__any_sync(0xffffffffu, live)) return 0;
  const bool edge = eBest >= 0 && 0.95 * eSep > fSep + 0.01;
  n = gshfl(n, max(edge ? eBest : fBest, 0));
  {  // orthonormal(basis, -n): the three quotients on three lanes
    const D3 m = neg(n);
    const bool xz = fabs(m.x) > fabs(m.z);
    const D3 t{xz ? -m.y : 0.0, xz ? m.x : -m.z, xz ? 0.0 : m.y};
    const double len = sqrt(t.x * t.x + t.y * t.y + t.z * t.z);
    const double part = (gl == 0 ? t.x : gl == 1 ? t.y : t.z) / len;
    const D3 u{gshfl(part, 0), gshfl(part, 1), gshfl(part, 2)};
    basis[0] = m.x; basis[1] = m.y; basis[2] = m.z;
    basis[3] = u.x; basis[4] = u.y; basis[5] = u.z;
    basis[6] = m.y * u.z - m.z * u.y;
    basis[7] = m.z * u.x - m.x * u.z;
    basis[8] = m.x * u.y - m.y * u.x;
  }
  int count = 0;
  if (__any_sync(0xffffffffu, live && !edge)) {  // faceManifold (collide.js:403-472)
    const bool face = live && !edge;
    const bool refIsA = fBest < 3;
    const int refAxis = refIsA ? max(fBest, 0) : fBest - 3;
    const D3 rc = pick3(refIsA, a.c, b.c), rh = pick3(refIsA, a.h, b.h);
    const D3 ic = pick3(refIsA, b.c, a.c), ih = pick3(refIsA, b.h, a.h);
    const int rBase = refIsA ? 0 : 3, iBase = 3 - rBase;
    const D3 refAx = gshfl(mine, rBase + refAxis);
    const D3 outward = pick3(refIsA, n, neg(n));
    const D3 fN = scl(refAx, dt3(outward, refAx) >= 0 ? 1.0 : -1.0);
    const D3 fC = adds(rc, fN, Collider::hcomp(rh, refAxis));
    const int u0 = refAxis == 0 ? 1 : 0, v0 = refAxis == 2 ? 1 : 2;
    const D3 fU = gshfl(mine, rBase + u0), fV = gshfl(mine, rBase + v0);
    const double fEU = Collider::hcomp(rh, u0), fEV = Collider::hcomp(rh, v0);
    // the incident face: the axis most parallel to the normal, the first on ties
    const double dot = dt3(mine, fN);
    int inc = 0;
    double best = -INFINITY;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double d = fabs(gshfl(dot, iBase + i));
      if (d > best) {
        best = d;
        inc = i;
      }
    }
    const D3 fn = scl(gshfl(mine, iBase + inc), gshfl(dot, iBase + inc) > 0 ? -1.0 : 1.0);
    const D3 fc = adds(ic, fn, Collider::hcomp(ih, inc));
    const int u1 = inc == 0 ? 1 : 0, v1 = inc == 2 ? 1 : 2;
    const D3 u = gshfl(mine, iBase + u1), v = gshfl(mine, iBase + v1);
    const double eU = Collider::hcomp(ih, u1), eV = Collider::hcomp(ih, v1);
    const double su = (gl == 0 || gl == 3) ? 1.0 : -1.0, sv = (gl == 0 || gl == 1) ? 1.0 : -1.0;
    D3 p{fc.x + u.x * (eU * su) + v.x * (eV * sv), fc.y + u.y * (eU * su) + v.y * (eV * sv),
         fc.z + u.z * (eU * su) + v.z * (eV * sv)};
    int num = face ? 4 : 0;
#pragma unroll 1
    for (int k = 0; k < 4; k++) {  // clipPlane (collide.js:202-247)
      D3 pn = pick3(k < 2, fU, fV);
      if (k & 1) pn = neg(pn);
      const double po = dt3(pn, fC) + (k < 2 ? fEU : fEV);
      const double db = pn.x * p.x + pn.y * p.y + pn.z * p.z - po;
      const int prev = gl == 0 ? max(num - 1, 0) : gl - 1;
      const D3 pa = gshfl(p, prev);
      const double da = gshfl(db, prev);
      const bool ai = da <= geo::kPlaneEps, bi = db <= geo::kPlaneEps;
      const bool cross = gl < num && ai != bi, keep = gl < num && bi;
      double t = 0;
      const double denom = da - db;
      if (fabs(denom) > geo::kSatEps) t = clampd(da / denom, 0, 1);
      const D3 x{pa.x + (p.x - pa.x) * t, pa.y + (p.y - pa.y) * t, pa.z + (p.z - pa.z) * t};
      const unsigned m1 = ballot(cross), m2 = ballot(keep), below = (1u << gl) - 1u;
      const int at = __popc(m1 & below) + __popc(m2 & below);
      if (cross && at < geo::kPolyCap) poly[at] = x;
      if (keep && at + (cross ? 1 : 0) < geo::kPolyCap) poly[at + (cross ? 1 : 0)] = p;
      num = min(__popc(m1) + __popc(m2), geo::kPolyCap);
      __syncwarp();
      if (gl < num) p = poly[gl];
      __syncwarp();
    }
    const double dist = dt3(sub(p, fC), fN);
    const bool kept = gl < num && !(dist > cd + geo::kPlaneEps);
    const D3 proj = adds(p, fN, -dist);
    D3 xA = pick3(refIsA, proj, p), xB = pick3(refIsA, p, proj);
    // addContact (collide.js:254-285): a point within 1 mm of an earlier contact merges into it
    const D3 m{(xA.x + xB.x) * 0.5, (xA.y + xB.y) * 0.5, (xA.z + xB.z) * 0.5};
    unsigned close = 0u;
#pragma unroll 1
    for (int j = 0; j < geo::kPolyCap - 1; j++) {
      const D3 mj = gshfl(m, j);
      const double dx = m.x - mj.x, dy = m.y - mj.y, dz = m.z - mj.z;
      if (j < gl && dx * dx + dy * dy + dz * dz < geo::kMergeDistSq) close |= 1u << j;
    }
    const unsigned keptMask = ballot(kept);
    unsigned taken = 0u;
#pragma unroll
    for (int i = 0; i < geo::kPolyCap; i++) {
      const unsigned ci = __shfl_sync(0xffffffffu, close, i, kGroup);
      if (((keptMask >> i) & 1u) && !(ci & taken)) taken |= 1u << i;
    }
    count = __popc(taken);
    uint32_t key = (uint32_t)(refIsA ? geo::kFaceA : geo::kFaceB) << 24;
    key |= (uint32_t)(refAxis & 0xff) << 16;
    key |= (uint32_t)(inc & 0xff) << 8;
    bool own = ((taken >> gl) & 1u) != 0;
    const bool none = face && num > 0 && count == 0;  // (clipped away whole: no contact)
    if (__any_sync(0xffffffffu, none)) {  // no vertex deep enough: the support points
      const D3 sA = Collider::support(a, n), sB = Collider::support(b, neg(n));
      if (none) {
        xA = sA;
        xB = sB;
        own = gl == 0;
        count = 1;
        taken = 1u;
      }
    }
    const D3 ra = rot(conj(A.q), sub(xA, A.p)), rb = rot(conj(B.q), sub(xB, B.p));
    if (face && own) {
      slot = __popc(taken & ((1u << gl) - 1u));
      nc.feature = key | (uint32_t)(gl & 0xff);
      nc.ra[0] = (float)ra.x; nc.ra[1] = (float)ra.y; nc.ra[2] = (float)ra.z;
      nc.rb[0] = (float)rb.x; nc.rb[1] = (float)rb.y; nc.rb[2] = (float)rb.z;
    }
    if (!face) count = 0;
  }
  if (live && edge) {  // the edge contact by the group's first lane
    count = 1;
    if (gl == 0) {
      NewContact e[1];
      Collider col(A, B, e);
      col.boxA = a;
      col.boxB = b;
      col.cd = cd;
      count = col.edgeContact((eBest - 6) / 3, (eBest - 6) % 3, n);
      slot = 0;
      nc.feature = e[0].feature;
      nc.ra[0] = (float)e[0].rA.x; nc.ra[1] = (float)e[0].rA.y; nc.ra[2] = (float)e[0].rA.z;
      nc.rb[0] = (float)e[0].rB.x; nc.rb[1] = (float)e[0].rB.y; nc.rb[2] = (float)e[0].rB.z;
    }
  }
  __syncwarp();
  return live ? count : 0;
}

// write_manifold_materials of a box pair on the sixteen lanes: an old contact
// and a new one a lane, the claims one new contact after the other (a lane for
// the pair took 162 us of the narrow phase of 1,000 such boxes, this
// 100). `slot` is the lane's new contact, nc, or -1.
__device__ void write_materials_group(const World &w, int c, int ia, int ib, const BodyD &A, const BodyD &B, bool act,
                                      const NewContactF &nc, int slot, int num, const double *basis) {
  const int gl = threadIdx.x & (kGroup - 1);
  const unsigned shift = threadIdx.x & (32 - kGroup);
  auto ballot = [&](bool p) { return (__ballot_sync(0xffffffffu, p) >> shift) & 0xffffu; };
  const bool own = act && slot >= 0;
  const MaterialsPair m = materials_pair(w, act ? c : 0, ia, ib, A, B, basis);
  const D3 rA = own ? mk(nc.ra[0], nc.ra[1], nc.ra[2]) : mk(0, 0, 0);
  const D3 rB = own ? mk(nc.rb[0], nc.rb[1], nc.rb[2]) : mk(0, 0, 0);
  const bool merge = act && num > 0 && m.compatible;
  int match = -1;
  if (__any_sync(0xffffffffu, merge)) {
    const D3 mid = midpoint(add(rot(A.q, rA), A.p), add(rot(B.q, rB), B.p));
    const bool old = merge && gl < m.oldNum;
    D3 oldMid = mk(0, 0, 0);
    bool pass = false;
    uint32_t oldFeat = 0u;
    if (old) {
      const int os = m.pi * kMaxContacts + gl;
      oldFeat = w.prev.feat[os];
      pass = old_contact(w, m, os, A, B, mk(basis[0], basis[1], basis[2]), oldMid);
    }
    unsigned used = 0u;
#pragma unroll 1
    for (int i = 0; __any_sync(0xffffffffu, merge && i < num); i++) {
      const unsigned at = ballot(own && slot == i);
      const int src = at ? __ffs(at) - 1 : 0;
      const double mdSq = dist_sq(gshfl(mid, src), oldMid);
      const uint32_t feat = __shfl_sync(0xffffffffu, own ? nc.feature : 0u, src, kGroup);
      const bool ok = pass && i < num && !((used >> gl) & 1u) && !(mdSq > m.psq);
      const unsigned sameMask = ballot(ok && oldFeat == feat);
      const int nearest = group_argmax(-mdSq, ok);
      const int j = sameMask ? __ffs(sameMask) - 1 : nearest;
      if (j >= 0) used |= 1u << j;
      if (own && slot == i) match = j;
    }
  }
  if (own) write_materials_contact(w, c, slot, ia, ib, A, B, m, basis, rA, rB, nc.feature, match);
  if (act && num > 0 && gl == 0) write_materials_header(w, c, m, basis);
}

// A lane's pair decided by the serial collider: every sphere pair, and box
// pairs of long lists.
__device__ __noinline__ void exact_pair(const World &w, int c) {
  const uint64_t key = w.g.candKey[c];
  const int ia = (int)(key >> 32), ib = (int)(key & 0xffffffffu);
  const BodyD A = load_body(w, ia), B = load_body(w, ib);
  double basis[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  NewContact nc[kMaxContacts];
  Collider col(A, B, nc);
  col.cd = pair_skin(w, ia, ib);
  const int num = col.collide(basis);
  if (A.sphere || B.sphere) {
    write_sphere_manifold(w, c, ia, ib, A, B, nc, num, basis);
    return;
  }
  NewContactF ncf[kMaxContacts];
  for (int k = 0; k < num; k++) {
    ncf[k].feature = nc[k].feature;
    ncf[k].ra[0] = (float)nc[k].rA.x; ncf[k].ra[1] = (float)nc[k].rA.y; ncf[k].ra[2] = (float)nc[k].rA.z;
    ncf[k].rb[0] = (float)nc[k].rB.x; ncf[k].rb[1] = (float)nc[k].rB.y; ncf[k].rb[2] = (float)nc[k].rB.z;
  }
  write_box_manifold(w, c, ia, ib, A, B, ncf, num, basis);
}

// 4. Sphere pairs and undecided box pairs: the whole f64 collider. Sphere pairs
//    a thread each (a short chain: in halves of warps of their own, as the box
//    pairs, they made it 113 us for 88 in a pile of 1,777 boxes and spheres), box
//    pairs on sixteen lanes or a thread each (pairs_per_warp).
struct GroupShared {
  D3 poly[geo::kPolyCap];
};

// Two pairs of one warp, a half each; c < 0: none (the first is one).
__device__ __forceinline__ void exact_groups(const World &w, int c, GroupShared &sh) {
  const int gl = threadIdx.x & (kGroup - 1);
  const int first = __shfl_sync(0xffffffffu, c, 0);
  const uint64_t key = w.g.candKey[c >= 0 ? c : first];
  const int ia = (int)(key >> 32), ib = (int)(key & 0xffffffffu);
  const BodyD A = load_body(w, ia), B = load_body(w, ib);
  const bool act = c >= 0;
  double basis[9];
  NewContactF nc;
  int slot;
  const int num = collide_group(A, B, pair_skin(w, ia, ib), act, sh.poly, basis, nc, slot);
  if (act && gl == 0) w.cur.count[c] = num;
  if (w.p.contactModel) {
    if (__any_sync(0xffffffffu, num > 0)) write_materials_group(w, c, ia, ib, A, B, act, nc, slot, num, basis);
  } else if (act && num) {
    float bf[9];
    for (int k = 0; k < 9; k++) bf[k] = (float)basis[k];
    const int pi = w.g.candPrev[c];
    const int oldNum = pi >= 0 ? w.prev.count[pi] : 0;
    if (slot >= 0) write_box_contact(w, c, slot, pi, oldNum, A, B, nc, bf);
    if (gl == 0) write_box_header(w, c, ia, ib, basis, bf);
  }
  __syncwarp();
}

// The three lists side by side, in units of a warp: two exact pairs on lanes
// (or 32, a thread each), or 32 face, sphere or edge pairs, the longest chains
// first. A short list is one pair's chain of instructions (some 55, 30 and
// 40-80 us for the face, edge and exact lists of 200-body piles), and the
// chains now overlap; a long one keeps every warp busy to the end (a kernel
// per list, each with a grid for the whole device, had a last wave apiece).
// When there are fewer units than warps they are dealt over the SMs, else a
// free warp claims the next one (claimed, not dealt, and not before the warp
// is free: both cost the crushed pyramid 5 %). Narrow phase, three kernels
// and this one: the 200-body pile 119 -> 62 us, spheres among boxes 173 ->
// 117, a 2,000-body pile 141 -> 102, a crushed 36-layer pyramid 949 -> 843,
// a batch of 163,000 bodies 704 -> 606.
__global__ void __launch_bounds__(128) collide_kernel(const __grid_constant__ World w) {
  await_previous();
  __shared__ GroupShared shared[8];
  const int lane = threadIdx.x & 31;
  const int nFace = w.ctl->npCount[0], nEdge = w.ctl->npCount[1], nExact = w.ctl->npCount[2];
  const int nSphere = w.ctl->npCount[4];
  const int per = pairs_per_warp(nExact, w.ctl->numCandidates - nSphere - nExact + w.ctl->npApart);
  const int uExact = (nExact + per - 1) / per, uFace = (nFace + 31) / 32, uEdge = (nEdge + 31) / 32;
  const int uSphere = (nSphere + 31) / 32, units = uExact + uFace + uSphere + uEdge, warps = gridDim.x * (blockDim.x >> 5);
  const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  for (bool dealt = units < warps;; dealt = false) {
    int u = warp;
    if (!dealt) {
      if (units < warps) return;
      if (lane == 0) u = atomicAdd(&w.ctl->npNext, 1);
      u = __shfl_sync(0xffffffffu, u, 0);
    }
    if (u >= units) return;
    if (u < uExact) {
      if (per == 2) {
        const int t = u * 2 + lane / kGroup;
        exact_groups(w, t < nExact ? w.g.npExact[t] : -1, shared[threadIdx.x / kGroup]);
      } else if (u * 32 + lane < nExact) {
        exact_pair(w, w.g.npExact[u * 32 + lane]);
      }
      continue;
    }
    u -= uExact;
    if (u < uFace) {
      if (u * 32 + lane < nFace) face_pair(w, u * 32 + lane);
      continue;
    }
    u -= uFace;
    if (u < uSphere) {
      if (u * 32 + lane < nSphere) exact_pair(w, w.g.npEdge[w.g.candCap - 1 - (u * 32 + lane)].x);
      continue;
    }
    u -= uSphere;
    if (u * 32 + lane < nEdge) edge_pair(w, u * 32 + lane);
  }
}

// 5. The face pairs that f32 could not decide, by the same rule (from the
//    exact list's far end down).
__global__ void __launch_bounds__(128) late_kernel(const __grid_constant__ World w) {
  await_previous();
  __shared__ GroupShared shared[8];
  const int total = w.ctl->npCount[3], lane = threadIdx.x & 31;
  const int *last = w.g.npExact + w.g.candCap - 1;
  const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps = gridDim.x * (blockDim.x >> 5);
  const int per = total > kGroupMax ? 32 : 2;
  for (int u = warp; u * per < total; u += warps) {
    if (per == 2) {
      const int t = u * 2 + lane / kGroup;
      exact_groups(w, t < total ? last[-t] : -1, shared[threadIdx.x / kGroup]);
    } else if (u * 32 + lane < total) {
      exact_pair(w, last[-(u * 32 + lane)]);
    }
  }
}

}  // namespace

void launch_narrowphase(const World &w, cudaStream_t st, int smCount) {
  launch_early(classify_kernel, smCount * 8, 256, st, w);
  launch_early(collide_kernel, smCount * 2, 128, st, w);
  launch_early(late_kernel, smCount * 2, 128, st, w);
}

}  // namespace avbd
