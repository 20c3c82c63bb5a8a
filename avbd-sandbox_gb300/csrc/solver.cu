// solver.cu - per-step preparation, constraint adjacency, integer-priority
// colouring and the launch of the persistent primal/dual solve (solve.cu) of
// one AVBD step.
//
// Reference path (src/physics/solver.js:340-489):
//   force init   manifold.js:214-318 (narrowphase.cu), joint.js:131-160,
//                spring.js:472-507                      -> prepare_forces_kernel
//   body init    solver.js:366-401 (Eq. 2 + adaptive guess) -> prepare_bodies_kernel
//   primal       solver.js:418-458, manifold.js:411-445, joint.js:162-253,
//                spring.js:509-616, maths.js:660-725    -> solve_kernel
//   dual         manifold.js:447-491, joint.js:255-317, spring.js:618-634
//   velocity     solver.js:476-488 (BDF1)
//
// GB300 design:
//   * the primal and dual iterations of a step are ONE cooperative persistent
//     kernel; colour phases are separated by a bounded grid barrier, and the
//     last, thin colours run as one dependency-driven segment per iteration
//   * a group of G lanes assembles one body's 6x6 system (each lane takes up
//     to four of the incident constraints per staging round), reduces it with
//     warp shuffles (2-4 warps: through shared memory) and every lane solves
//     the LDL^T in registers; G (4..128) is chosen per body by the colouring,
//     which lays out each colour's groups in 128-lane chunks
//   * the dual update of a constraint is fused into the primal phase of its
//     endpoint with the larger colour: both endpoints are final for the
//     iteration at that moment, so this equals the reference's separate
//     dual sweep (solver.js:466-470) without another barrier per iteration
//   * positions are iterated as delta = x - x_t in f32 (x_t in f64), so the
//     f32 rounding is relative to the step's displacement, not to |x|
//   * bodies whose constraint stiffness dwarfs their inertia (k / (m/dt^2)
//     above a threshold) are assembled and factored in f64 from f64 shadows
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include "solve.cuh"

namespace avbd {
namespace {

// ---------------------------------------------------------------------------
// Preparation
// ---------------------------------------------------------------------------
__device__ inline double jsmin(double a, double b) { return a < b ? a : (b < a ? b : a); }
__device__ inline double jsmax(double a, double b) { return a > b ? a : (b > a ? b : a); }
__device__ inline double clampd(double x, double a, double b) { return x != x ? x : jsmax(a, jsmin(b, x)); }

__device__ inline Q4<double> body_q_t(const World &w, int i) {
  const float4 q = w.b.quat[i];
  return Q4<double>{q.x, q.y, q.z, q.w};
}

// joint.js:131-160 / spring.js:472-507, plus the f64 offsets p_A(t) - p_B(t).
__global__ void prepare_forces_kernel(World w) {
  await_previous();
  if (step_skipped(w)) return;
  const SolverParams &P = w.p;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (int j = tid; j < w.j.n; j += stride) {
    const int st = w.j.state[j];
    if (st & kRemoved) continue;  // left the force list in an earlier step
    if (st & kBroken) {
      // Joint.initialize still warm-starts a joint broken in the last step
      // (lambda = alpha gamma 0, k = min(clamp(gamma 0, kmin, kmax), stiffness)),
      // then returns !broken and the joint leaves the force list
      // (solver.js:346-360)
      const D4 sf = w.j.stiff[j];
      auto warm0 = [&](float k, double cap) {
        return (float)jsmin(clampd((double)k * P.gamma, P.penaltyMin, P.penaltyMax), cap);
      };
      const float4 kl = w.j.penLin[j], ka = w.j.penAng[j];
      w.j.penLin[j] = make_float4(warm0(kl.x, sf.x), warm0(kl.y, sf.x), warm0(kl.z, sf.x), 0.f);
      w.j.penAng[j] = make_float4(warm0(ka.x, sf.y), warm0(ka.y, sf.y), warm0(ka.z, sf.y), 0.f);
      if (!P.postStabilize) {
        D4 ll = w.j.lamLin[j], la = w.j.lamAng[j];
        ll.x = ll.x * P.alpha * P.gamma; ll.y = ll.y * P.alpha * P.gamma; ll.z = ll.z * P.alpha * P.gamma;
        la.x = la.x * P.alpha * P.gamma; la.y = la.y * P.alpha * P.gamma; la.z = la.z * P.alpha * P.gamma;
        w.j.lamLin[j] = ll;
        w.j.lamAng[j] = la;
      }
      w.j.state[j] = st | kRemoved;
      continue;
    }
    const int2 ab = w.j.bodies[j];
    const D4 rA = w.j.rAD[j], rB = w.j.rBD[j], sf = w.j.stiff[j];
    const Q4<double> qB = body_q_t(w, ab.y);
    const D4 pB = w.b.pos[ab.y];
    V3<double> pa, dpt;
    Q4<double> qA{0, 0, 0, 1};
    if (ab.x >= 0) {
      qA = body_q_t(w, ab.x);
      const D4 p = w.b.pos[ab.x];
      const V3<double> r = qrotate(qA, V3<double>{rA.x, rA.y, rA.z});
      pa = V3<double>{r.x + p.x, r.y + p.y, r.z + p.z};
      dpt = V3<double>{p.x - pB.x, p.y - pB.y, p.z - pB.z};
    } else {
      pa = V3<double>{rA.x, rA.y, rA.z};
      dpt = V3<double>{rA.x - pB.x, rA.y - pB.y, rA.z - pB.z};
    }
    const V3<double> rb = qrotate(qB, V3<double>{rB.x, rB.y, rB.z});
    const V3<double> pb{rb.x + pB.x, rb.y + pB.y, rb.z + pB.z};
    const V3<double> c0l = pa - pb;
    const V3<double> c0a = qsub(qA, qB) * sf.w;
    w.j.c0Lin[j] = make_float4((float)c0l.x, (float)c0l.y, (float)c0l.z, 0.f);
    w.j.c0Ang[j] = make_float4((float)c0a.x, (float)c0a.y, (float)c0a.z, 0.f);
    w.j.dpt[j] = make_float4((float)dpt.x, (float)dpt.y, (float)dpt.z, 0.f);
    w.j.dptD[j] = mkd4(dpt.x, dpt.y, dpt.z, 0.0);
    D4 ll = w.j.lamLin[j], la = w.j.lamAng[j];
    if (!P.postStabilize) {
      ll.x = ll.x * P.alpha * P.gamma; ll.y = ll.y * P.alpha * P.gamma; ll.z = ll.z * P.alpha * P.gamma;
      la.x = la.x * P.alpha * P.gamma; la.y = la.y * P.alpha * P.gamma; la.z = la.z * P.alpha * P.gamma;
    }
    w.j.lamLin[j] = ll;
    w.j.lamAng[j] = la;
    w.j.lamLinF[j] = make_float4((float)ll.x, (float)ll.y, (float)ll.z, 0.f);
    w.j.lamAngF[j] = make_float4((float)la.x, (float)la.y, (float)la.z, 0.f);
    float4 kl = w.j.penLin[j], ka = w.j.penAng[j];
    auto warm = [&](float k, double cap) {
      return (float)jsmin(clampd((double)k * P.gamma, P.penaltyMin, P.penaltyMax), cap);
    };
    kl = make_float4(warm(kl.x, sf.x), warm(kl.y, sf.x), warm(kl.z, sf.x), 0.f);
    ka = make_float4(warm(ka.x, sf.y), warm(ka.y, sf.y), warm(ka.z, sf.y), 0.f);
    w.j.penLin[j] = kl;
    w.j.penAng[j] = ka;
  }
  for (int s = tid; s < w.s.n; s += stride) {
    int st = w.s.state[s];
    if (st & kRemoved) continue;
    const int2 ab = w.s.bodies[s];
    const D4 prm = w.s.prm[s];
    const D4 pA = w.b.pos[ab.x], pB = w.b.pos[ab.y];
    const V3<double> dpt{pA.x - pB.x, pA.y - pB.y, pA.z - pB.z};
    w.s.dpt[s] = make_float4((float)dpt.x, (float)dpt.y, (float)dpt.z, 0.f);
    w.s.dptD[s] = mkd4(dpt.x, dpt.y, dpt.z, 0.0);
    if (st & kBroken) {
      w.s.penalty[s] = 0.f;
      continue;
    }
    if (isfinite(prm.z)) {  // tear check at x_t (spring.js:484-490)
      const D4 rA = w.s.rAD[s], rB = w.s.rBD[s];
      const V3<double> ra = qrotate(body_q_t(w, ab.x), V3<double>{rA.x, rA.y, rA.z});
      const V3<double> rb = qrotate(body_q_t(w, ab.y), V3<double>{rB.x, rB.y, rB.z});
      const V3<double> d{(ra.x + pA.x) - (rb.x + pB.x), (ra.y + pA.y) - (rb.y + pB.y),
                         (ra.z + pA.z) - (rb.z + pB.z)};
      const double len = sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
      if (len > 1.0e-6 && prm.y > 1.0e-6) {
        const double strain = jsmax(0.0, (len - prm.y) / prm.y);
        w.s.peak[s] = jsmax(w.s.peak[s], strain);
        if (strain > prm.z) {
          w.s.state[s] = st | kBroken;
          w.s.penalty[s] = 0.f;
          continue;
        }
      }
    }
    if (!P.springRamp) {
      w.s.penalty[s] = (float)prm.x;
    } else {
      double k = clampd((double)w.s.penalty[s] * P.gamma, P.penaltyMin, P.penaltyMax);
      w.s.penalty[s] = (float)jsmin(k, prm.x);
    }
    if (!(prm.x > 0)) w.s.state[s] = st | kRemoved;
  }
}

// solver.js:369-401, in delta form.
__global__ void prepare_bodies_kernel(World w) {
  await_previous();
  if (step_skipped(w)) return;
  const SolverParams &P = w.p;
  const double dt = P.dt, g = P.gravity;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < w.b.n; i += gridDim.x * blockDim.x) {
    const float4 qf = w.b.quat[i], vf = w.b.vel[i], wf = w.b.omega[i], pv = w.b.prevVel[i];
    const double mass = w.b.massD[i].x;
    const Q4<double> q{qf.x, qf.y, qf.z, qf.w};
    const V3<double> wdt{(double)wf.x * dt, (double)wf.y * dt, (double)wf.z * dt};
    V3<double> y{(double)vf.x * dt, (double)vf.y * dt, (double)vf.z * dt};
    if (mass > 0) y.z += g * (dt * dt);
    const Q4<double> qy = qintegrate(q, wdt);
    const double accelZ = ((double)vf.z - (double)pv.z) / dt;
    const double sgn = g < 0 ? -1.0 : (g > 0 ? 1.0 : 0.0);
    double weight = clampd(accelZ * sgn / fabs(g), 0.0, 1.0);
    if (!isfinite(weight)) weight = 0.0;
    w.b.quatT[i] = qf;
    w.b.yLin[i] = make_float4((float)y.x, (float)y.y, (float)y.z, 0.f);
    w.b.yAng[i] = make_float4((float)qy.x, (float)qy.y, (float)qy.z, (float)qy.w);
    int fl = w.b.flags0[i];
    if (mass > 0) {
      V3<double> d{(double)vf.x * dt, (double)vf.y * dt, (double)vf.z * dt};
      d.z += g * (weight * dt * dt);
      w.b.dp[i] = make_float4((float)d.x, (float)d.y, (float)d.z, 0.f);
      w.b.dpD[i] = mkd4(d.x, d.y, d.z, 0.0);
      w.b.quat[i] = make_float4((float)qy.x, (float)qy.y, (float)qy.z, (float)qy.w);
      w.b.quatD[i] = mkd4(qy.x, qy.y, qy.z, qy.w);
    } else {
      w.b.dp[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      w.b.dpD[i] = mkd4(0.0, 0.0, 0.0, 0.0);
      w.b.quatD[i] = mkd4(q.x, q.y, q.z, q.w);
    }
    {  // the iterate's qsub(q, q_t), as load_state<float> forms it
      const float4 qn = w.b.quat[i];
      const V3<float> da = qsub(Q4<float>{qn.x, qn.y, qn.z, qn.w}, Q4<float>{qf.x, qf.y, qf.z, qf.w});
      w.b.dang[i] = make_float4(da.x, da.y, da.z, 0.f);
    }
    w.b.flags[i] = fl;
    w.a.count[i] = 0ull;
    if (i % kAdjRun == 0) w.a.runCount[i / kAdjRun] = 0ull;
    w.b.progress[i] = 0;
  }
}

// Live manifolds of this step: count the incident ones of every dynamic body.
__device__ inline bool precedes(const World &w, int j, int i) {
  const uint32_t pj = w.b.priority[j], pi = w.b.priority[i];
  return pj < pi || (pj == pi && j < i);
}

__global__ void adj_count_kernel(World w) {
  await_previous();
  const int total = w.ctl->numCandidates;
  int live = 0, contacts = 0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
    const int n = w.cur.count[c];
    if (n <= 0) continue;
    const uint64_t k = w.cur.key[c];
    const unsigned long long one = 1ull | (unsigned long long)n << 32;
    for (int side = 0; side < 2; side++) {
      const int i = side ? (int)(k & 0xffffffffu) : (int)(k >> 32);
      if (!(w.b.flags0[i] & kBodyDynamic)) continue;
      atomicAdd(&w.a.count[i], one);
      atomicAdd(&w.a.runCount[i / kAdjRun], one);
    }
    live++;
    contacts += n;
  }
  __syncwarp();
  live = __reduce_add_sync(0xffffffffu, live);
  contacts = __reduce_add_sync(0xffffffffu, contacts);
  if ((threadIdx.x & 31) == 0 && live) {
    atomicAdd(&w.ctl->liveManifolds, live);
    atomicAdd(&w.ctl->liveContacts, contacts);
  }
}

// Where each body's manifolds and contacts start: a block sums the runs
// before its bodies, then scans their counts.
__global__ void __launch_bounds__(256) adj_scan_kernel(World w) {
  await_previous();
  typedef unsigned long long U;
  typedef cub::BlockReduce<U, 256> R;
  typedef cub::BlockScan<U, 256> S;
  __shared__ union {
    typename R::TempStorage r;
    typename S::TempStorage s;
  } tmp;
  __shared__ U base;
  static_assert(256 % kAdjRun == 0, "a block's bodies begin a run");
  const int i = blockIdx.x * 256 + threadIdx.x;
  U v = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x * (256 / kAdjRun); k += 256) v += w.a.runCount[k];
  v = R(tmp.r).Sum(v);
  if (threadIdx.x == 0) base = v;
  __syncthreads();
  U at;
  S(tmp.s).ExclusiveSum(i < w.b.n ? w.a.count[i] : 0ull, at);
  at += base;
  if (i > w.b.n) return;
  w.a.start[i] = (int)(at & 0xffffffffu);
  w.a.cstart[i] = (int)(at >> 32);
  if (i < w.b.n) w.a.cursor[i] = (int)(at & 0xffffffffu);
}

__global__ void adj_fill_kernel(World w) {
  await_previous();
  const int total = w.ctl->numCandidates;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
    if (w.cur.count[c] <= 0) continue;
    const uint64_t k = w.cur.key[c];
    const int a = (int)(k >> 32), b = (int)(k & 0xffffffffu);
    if (w.b.flags0[a] & kBodyDynamic) {
      const int at = atomicAdd(&w.a.cursor[a], 1);
      if (at < w.a.cap) w.a.entry[at] = ((uint32_t)c << 1) | 0u;
      else atomicOr(&w.ctl->flags, kOvfAdj);
    }
    if (w.b.flags0[b] & kBodyDynamic) {
      const int at = atomicAdd(&w.a.cursor[b], 1);
      if (at < w.a.cap) w.a.entry[at] = ((uint32_t)c << 1) | 1u;
      else atomicOr(&w.ctl->flags, kOvfAdj);
    }
  }
}

// The three of them in one block, the counts and cursors in shared memory:
// scenes of fewer than kAdjAlone bodies, whose work is less than the launches
// (preparation of 10 / 200 / 1,000 bodies 22 / 26 / 28 -> 19 / 24 / 26 us).
__global__ void __launch_bounds__(kAdjAlone) adj_small_kernel(World w) {
  await_previous();
  typedef unsigned long long U;
  typedef cub::BlockScan<U, kAdjAlone> S;
  __shared__ typename S::TempStorage tmp;
  __shared__ U counts[kAdjAlone];
  __shared__ int cursor[kAdjAlone];
  const int total = w.ctl->numCandidates, t = threadIdx.x;
  counts[t] = 0ull;
  __syncthreads();
  int live = 0, contacts = 0;
  for (int c = t; c < total; c += kAdjAlone) {
    const int n = w.cur.count[c];
    if (n <= 0) continue;
    const uint64_t k = w.cur.key[c];
    const int a = (int)(k >> 32), b = (int)(k & 0xffffffffu);
    const U one = 1ull | (U)n << 32;
    if (w.b.flags0[a] & kBodyDynamic) atomicAdd(&counts[a], one);
    if (w.b.flags0[b] & kBodyDynamic) atomicAdd(&counts[b], one);
    live++;
    contacts += n;
  }
  __syncwarp();
  live = __reduce_add_sync(0xffffffffu, live);
  contacts = __reduce_add_sync(0xffffffffu, contacts);
  if ((t & 31) == 0 && live) {
    atomicAdd(&w.ctl->liveManifolds, live);
    atomicAdd(&w.ctl->liveContacts, contacts);
  }
  __syncthreads();
  U at;
  S(tmp).ExclusiveSum(counts[t], at);  // (none of the bodies from n on)
  if (t <= w.b.n) {
    w.a.start[t] = (int)(at & 0xffffffffu);
    w.a.cstart[t] = (int)(at >> 32);
  }
  cursor[t] = (int)(at & 0xffffffffu);
  __syncthreads();
  for (int c = t; c < total; c += kAdjAlone) {
    if (w.cur.count[c] <= 0) continue;
    const uint64_t k = w.cur.key[c];
    for (int side = 0; side < 2; side++) {
      const int i = side ? (int)(k & 0xffffffffu) : (int)(k >> 32);
      if (!(w.b.flags0[i] & kBodyDynamic)) continue;
      const int e = atomicAdd(&cursor[i], 1);
      if (e < w.a.cap) w.a.entry[e] = ((uint32_t)c << 1) | side;
      else atomicOr(&w.ctl->flags, kOvfAdj);
    }
  }
}

// Sort each body's manifold list (determinism), list its contacts and decide
// its precision: eight lanes a body (a rank sort in shared memory, the
// contacts' places by a scan over the lanes). A thread a body took 255 us of
// a crushed pyramid's step: an insertion sort of 30 to 100 entries in global
// memory each, and of some 200 for the sphere that everything waited for.
constexpr int kSortRow = 96;  // entries sorted in shared memory; more: from a copy in the body's hpEntry range
__global__ void __launch_bounds__(256) adj_sort_kernel(World w) {
  await_previous();
  if (step_skipped(w)) return;
  __shared__ uint32_t row[32][kSortRow];
  const double dt2 = w.p.dt * w.p.dt;
  const int gl = threadIdx.x & 7, group = threadIdx.x >> 3, shift = threadIdx.x & 24;
  uint32_t *e = w.a.entry;
  for (int i0 = blockIdx.x * 32; i0 < w.b.n; i0 += gridDim.x * 32) {
    const int i = i0 + group;
    int fl = i < w.b.n ? w.b.flags[i] : 0;
    const bool dyn = (fl & kBodyDynamic) != 0;
    int beg = 0, end = 0, at = 0, cend = 0;
    if (dyn) {
      beg = w.a.start[i];
      end = min(w.a.start[i + 1], w.a.cap);
      at = w.a.cstart[i];
      cend = min(w.a.cstart[i + 1], w.a.ccap);
    }
    const int n = max(end - beg, 0);
    // entries are distinct: each goes to the number of smaller ones
    if (n <= kSortRow) {
      for (int x = gl; x < n; x += 8) row[group][x] = e[beg + x];
      __syncwarp(0xffu << shift);
      for (int x = gl; x < n; x += 8) {
        const uint32_t v = row[group][x];
        int r = 0;
        for (int y = 0; y < n; y++) r += row[group][y] < v ? 1 : 0;
        e[beg + r] = v;
      }
    } else {
      uint32_t *copy = reinterpret_cast<uint32_t *>(w.a.hpEntry);  // the body's range there is written below
      for (int x = gl; x < n; x += 8) copy[beg + x] = e[beg + x];
      __syncwarp(0xffu << shift);
      for (int x = gl; x < n; x += 8) {
        const uint32_t v = copy[beg + x];
        int r = 0;
        for (int y = 0; y < n; y++) r += copy[beg + y] < v ? 1 : 0;
        e[beg + r] = v;
      }
    }
    __syncwarp();
    // per-contact adjacency, in manifold order then contact order; and the
    // dynamic neighbours of higher colouring priority (the only ones a
    // colouring round reads), stored in the body's own manifold range
    int hc = 0;
    const int most = __reduce_max_sync(0xffffffffu, n);
    for (int x0 = 0; x0 < most; x0 += 8) {
      const int x = x0 + gl;
      int m = 0, side = 0, other = 0, cnt = 0;
      bool higher = false;
      if (x < n) {
        const uint32_t v = e[beg + x];
        m = (int)(v >> 1);
        side = (int)(v & 1u);
        const uint64_t key = w.cur.key[m];
        other = side ? (int)(key >> 32) : (int)(key & 0xffffffffu);
        cnt = w.cur.count[m];
        higher = (w.b.flags0[other] & kBodyDynamic) && precedes(w, other, i);
      }
      int incl = cnt;
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d, 8);
        if (gl >= d) incl += v;
      }
      const int first = at + incl - cnt;
      for (int k = 0; k < cnt && first + k < cend; k++)
        w.a.centry[first + k] = make_int2(((m * kMaxContacts + k) << 2) | side, other);  // owner bit set after colouring
      at += __shfl_sync(0xffffffffu, incl, 7, 8);
      const unsigned hm = (__ballot_sync(0xffffffffu, higher) >> shift) & 0xffu;
      if (higher) w.a.hpEntry[beg + hc + __popc(hm & ((1u << gl) - 1u))] = other;
      hc += __popc(hm);
    }
    if (!dyn || gl != 0) continue;
    w.a.hpCount[i] = hc;
    if (!w.p.mayFp64) continue;
    double kmax = 0;
    for (int k = w.g.cStart[i]; k < w.g.cStart[i + 1]; k++) {
      const uint32_t ref = w.g.cRef[k];
      const uint32_t type = ref >> 30, idx = (ref >> 1) & 0x1fffffffu;
      if (type == kRefJoint) {
        if (w.j.state[idx]) continue;
        const float4 kl = w.j.penLin[idx];
        const double hard = isinf(w.j.stiff[idx].x) ? w.p.penaltyMax : 0.0;
        kmax = fmax(kmax, fmax(fmax((double)kl.x, (double)kl.y), fmax((double)kl.z, hard)));
      } else {
        if (w.s.state[idx]) continue;
        kmax = fmax(kmax, (double)w.s.penalty[idx]);
      }
    }
    const double inertial = w.b.massD[i].x / dt2;
    if (kmax > w.p.fp64Ratio * inertial) {
      w.b.flags[i] = fl | kBodyFp64;
      atomicAdd(&w.ctl->fp64Bodies, 1);
    }
  }
}

// ---------------------------------------------------------------------------
// Colouring: greedy in (lowbias32(local index), index) order, computed as the
// fixed point of in-place Jacobi rounds seeded with the previous step's
// colours (the reference GPU's incremental colouring,
// src/physics/gpu/shaders.js:1558-1656, run to convergence so that the result
// is exactly the sequential greedy colouring in priority order). Then a
// stable counting sort lists each colour's bodies in index order.
// ---------------------------------------------------------------------------
// The live joint and spring partners of body i that are dynamic.
template <class F>
__device__ inline void constraint_neighbors(const World &w, int i, F &&f) {
  for (int k = w.g.cStart[i]; k < w.g.cStart[i + 1]; k++) {
    const uint32_t ref = w.g.cRef[k];
    const uint32_t type = ref >> 30, idx = (ref >> 1) & 0x1fffffffu, side = ref & 1u;
    int2 ab;
    if (type == kRefJoint) {
      if (w.j.state[idx]) continue;
      ab = w.j.bodies[idx];
    } else {
      if (w.s.state[idx]) continue;
      ab = w.s.bodies[idx];
    }
    const int other = side ? ab.x : ab.y;
    if (other >= 0 && (w.b.flags0[other] & kBodyDynamic)) f(other);
  }
}

// Every block of the colouring past this point; `arrivals` counts along.
__device__ __forceinline__ bool coloring_barrier(const World &w, unsigned &arrivals) {
  if (gridDim.x == 1) {
    __syncthreads();
    return true;
  }
  arrivals += gridDim.x;
  grid_arrive(&w.ctl->colorArrivals);
  return grid_wait(w.ctl, &w.ctl->colorArrivals, arrivals, w.p.barrierLimit);
}

// log2 of the lanes of a body's group in the colour-phase solve: the fixed
// lanes parameter, else the fewest lanes (4..128) whose staging of four
// constraints per lane holds all of the body's constraints; FP64 bodies
// (register path, warp shuffles) at most 32.
__device__ __forceinline__ int lane_log2(const World &w, int4 rec) {
  int G;
  if (w.p.lanes > 0) {
    G = w.p.lanes;
  } else {
    const int i = rec.x;
    const int total = (rec.z - rec.y) + (w.g.cStart[i + 1] - w.g.cStart[i]);
    G = 4;
    while (G < kLaneMaxGroup && 4 * G < total) G <<= 1;
  }
  if ((w.b.flags[rec.x] & kBodyFp64) && G > 32) G = 32;
  return 31 - __clz(G);
}

// The lane layout of the colour-phase solve (Adjacency::laneTab), from the
// sorted colour records: groups counted per (colour, size), each colour's
// groups placed in decreasing size (so every offset is a multiple of the
// group's own size and no group crosses a chunk), chunks of all colours
// numbered in colour order. Placement within a (colour, size) class follows
// atomics and may vary between runs; a body's arithmetic depends only on its
// group size, so results do not.
__device__ void lane_layout(const World &w, unsigned &arrivals) {
  Control *ctl = w.ctl;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  volatile int *color = w.b.color;
  int *cnt = w.a.laneHist, *cur = w.a.laneHist + kMaxColors * kLaneBuckets;
  int *used = w.a.laneHist + 2 * kMaxColors * kLaneBuckets;
  const int nrec = w.a.colorStart[kMaxColors];
  const int numColors = *((volatile int *)&ctl->numColors);
  const int lane = threadIdx.x & 31;
  // warp-uniform loops (stride is a multiple of 32): the records of a warp
  // with equal (colour, size) share one atomic
  for (int r = tid; r - lane < nrec; r += stride) {
    int key = -1;
    if (r < nrec) {
      const int4 rec = w.a.colorRec[r];
      key = color[rec.x] * kLaneBuckets + lane_log2(w, rec);
    }
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && lane == __ffs(peers) - 1) atomicAdd(&cnt[key], __popc(peers));
  }
  if (!coloring_barrier(w, arrivals)) return;
  if (blockIdx.x == 0) {
    // per colour: the offsets of its size classes (largest first) and its
    // lane count; then the colours' first chunks by a block-wide scan
    __shared__ int chunkScan[256];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    int lanesTotal = 0;
    for (int c0 = 0; c0 < numColors; c0 += blockDim.x) {
      const int c = c0 + threadIdx.x;
      int chunks = 0;
      if (c < numColors) {
        int off = 0;
        for (int b = kLaneBuckets - 1; b >= 0; b--) {
          cur[c * kLaneBuckets + b] = off;
          off += cnt[c * kLaneBuckets + b] << b;
        }
        used[c] = off;
        lanesTotal += off;
        chunks = (off + kLaneMaxGroup - 1) / kLaneMaxGroup;
      }
      chunkScan[threadIdx.x] = chunks;
      __syncthreads();
      for (int d = 1; d < (int)blockDim.x; d <<= 1) {  // inclusive scan
        const int v = threadIdx.x >= d ? chunkScan[threadIdx.x - d] : 0;
        __syncthreads();
        chunkScan[threadIdx.x] += v;
        __syncthreads();
      }
      if (c < numColors) w.a.colorChunk[c] = carry + chunkScan[threadIdx.x] - chunks;
      __syncthreads();
      if (threadIdx.x == blockDim.x - 1) carry += chunkScan[threadIdx.x];
      __syncthreads();
    }
    if (threadIdx.x == 0) w.a.colorChunk[numColors] = carry;
    lanesTotal = __reduce_add_sync(0xffffffffu, lanesTotal);
    if (lane == 0 && lanesTotal) atomicAdd(&ctl->laneTotal, lanesTotal);
  }
  if (!coloring_barrier(w, arrivals)) return;
  for (int k = tid; k < numColors * kLaneBuckets; k += stride) cnt[k] = 0;  // for the next step
  for (int r = tid; r - lane < nrec; r += stride) {
    int key = -1, c = 0, b = 0, e = 0;
    if (r < nrec) {
      const int4 rec = w.a.colorRec[r];
      c = color[rec.x];
      b = lane_log2(w, rec);
      key = c * kLaneBuckets + b;
      e = (r << 4) | ((w.b.flags[rec.x] & kBodyFp64) ? 8 : 0) | b;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (key >= 0 && lane == leader) base = atomicAdd(&cur[key], __popc(peers) << b);
    base = __shfl_sync(0xffffffffu, base, leader);
    if (key < 0) continue;
    const int off = base + (__popc(peers & ((1u << lane) - 1u)) << b);
    int *dst = w.a.laneTab + (size_t)w.a.colorChunk[c] * kLaneMaxGroup + off;
    if (b >= 2) {  // off and G are multiples of 4: 16-byte stores
      const int4 e4 = make_int4(e, e, e, e);
      for (int k = 0; k < (1 << b); k += 4) *reinterpret_cast<int4 *>(dst + k) = e4;
    } else {
      for (int k = 0; k < (1 << b); k++) dst[k] = e;
    }
  }
  // the lanes past each colour's last group, up to its last chunk's end
  for (int k = tid; k < numColors * kLaneMaxGroup; k += stride) {
    const int c = k / kLaneMaxGroup;
    const size_t L = (size_t)w.a.colorChunk[c] * kLaneMaxGroup + used[c] + (k % kLaneMaxGroup);
    if (L < (size_t)w.a.colorChunk[c + 1] * kLaneMaxGroup) w.a.laneTab[L] = -1;
  }
}

// The tail of the colouring: owner bits of the contact entries, the stable
// counting sort by colour and the solve's lane layout (cooperative: grid
// barriers inside). Per-colour loops run over the colours in use only
// (Control::numColors, from the largest colour found), so a step of few
// colours pays nothing for the colour capacity.
__device__ void coloring_finish(const World &w, unsigned &arrivals) {
  Control *ctl = w.ctl;
  const int n = w.b.n;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  volatile int *color = w.b.color;
  // owner bit (bit 1) of every contact entry: the endpoint with the larger
  // colour owns the contact's dual update (a static endpoint has colour -1);
  // and the number of colours in use
  int maxColor = -1;
  for (int i = tid; i < n; i += stride) {
    if (!(w.b.flags0[i] & kBodyDynamic)) continue;
    const int ci = color[i];
    maxColor = max(maxColor, ci);
    const int e1 = min(w.a.cstart[i + 1], w.a.ccap);
    for (int e = w.a.cstart[i]; e < e1; e++) {
      int2 v = w.a.centry[e];
      const int oc = (w.b.flags0[v.y] & kBodyDynamic) ? color[v.y] : -1;
      v.x = (v.x & ~2) | (ci > oc ? 2 : 0);
      w.a.centry[e] = v;
    }
  }
  maxColor = __reduce_max_sync(0xffffffffu, maxColor);
  if ((threadIdx.x & 31) == 0 && maxColor >= 0) atomicMax(&ctl->numColors, maxColor + 1);
  if (tid == 0) ctl->laneTotal = 0;  // summed by lane_layout after the next barriers
  if (!coloring_barrier(w, arrivals)) return;
  const int numColors = *((volatile int *)&ctl->numColors);
  // --- stable counting sort by colour (per-block chunk of body indices) ---
  __shared__ int hist[kMaxColors];
  __shared__ int base[kMaxColors];
  const int chunk = (n + gridDim.x - 1) / gridDim.x;
  const int b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
  for (int c = threadIdx.x; c < numColors; c += blockDim.x) hist[c] = 0;
  __syncthreads();
  for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
    const int c = color[i];
    if (c >= 0) atomicAdd(&hist[c], 1);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < numColors; c += blockDim.x) w.a.blockHist[blockIdx.x * kMaxColors + c] = hist[c];
  if (!coloring_barrier(w, arrivals)) return;
  if (blockIdx.x == 0) {
    // per colour: the blocks' offsets (a scan over blocks), then the colours'
    // starts (a block-wide scan over colours, in rounds of blockDim colours).
    // A round's colours share the block's threads: `parts` threads a colour,
    // each summing, then offsetting, a contiguous run of blocks (the counts
    // are integers: any grouping gives the same offsets).
    __shared__ int scan[256];
    __shared__ int partSum[256];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int c0 = 0; c0 < numColors; c0 += blockDim.x) {
      const int round = min((int)blockDim.x, numColors - c0);
      const int parts = max(1, (int)blockDim.x / round);
      const int cl = (int)threadIdx.x / parts, part = (int)threadIdx.x % parts;
      const int len = ((int)gridDim.x + parts - 1) / parts, bb = part * len, be = min((int)gridDim.x, bb + len);
      const bool mine = cl < round;
      const int cc = c0 + cl;
      int sum = 0;
      if (mine)
        for (int b = bb; b < be; b++) sum += w.a.blockHist[b * kMaxColors + cc];
      partSum[threadIdx.x] = sum;
      __syncthreads();
      if (mine) {
        int run = 0;
        for (int q = 0; q < part; q++) run += partSum[cl * parts + q];
        for (int b = bb; b < be; b++) {
          const int h = w.a.blockHist[b * kMaxColors + cc];
          w.a.blockHist[b * kMaxColors + cc] = run;
          run += h;
        }
      }
      const int c = c0 + threadIdx.x;
      int run = 0;  // colour c's total
      if (threadIdx.x < round)
        for (int q = 0; q < parts; q++) run += partSum[threadIdx.x * parts + q];
      __syncthreads();
      scan[threadIdx.x] = run;
      __syncthreads();
      for (int d = 1; d < (int)blockDim.x; d <<= 1) {  // inclusive scan
        const int v = threadIdx.x >= d ? scan[threadIdx.x - d] : 0;
        __syncthreads();
        scan[threadIdx.x] += v;
        __syncthreads();
      }
      if (c < numColors) w.a.colorStart[c] = carry + scan[threadIdx.x] - run;
      __syncthreads();
      if (threadIdx.x == blockDim.x - 1) carry += scan[threadIdx.x];
      __syncthreads();
    }
    for (int c = numColors + (int)threadIdx.x; c <= kMaxColors; c += blockDim.x) w.a.colorStart[c] = carry;
  }
  if (!coloring_barrier(w, arrivals)) return;
  for (int c = threadIdx.x; c < numColors; c += blockDim.x)
    base[c] = w.a.colorStart[c] + w.a.blockHist[blockIdx.x * kMaxColors + c];
  __syncthreads();
  // within a tile of blockDim bodies: rank among the tile's bodies of the same
  // colour = rank within the warp + the counts of that colour in earlier warps
  // (each warp lists its distinct colours with their counts)
  __shared__ int2 warpList[8][32];
  __shared__ int warpLen[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t0 = b0; t0 < b1; t0 += blockDim.x) {
    const int i = t0 + threadIdx.x;
    const int c = (i < b1) ? color[i] : -1;
    const unsigned m = __match_any_sync(0xffffffffu, c);
    const int rankInWarp = __popc(m & ((1u << lane) - 1u));
    const bool leader = rankInWarp == 0 && c >= 0;
    const unsigned leaders = __ballot_sync(0xffffffffu, leader);
    if (leader) warpList[warp][__popc(leaders & ((1u << lane) - 1u))] = make_int2(c, __popc(m));
    if (lane == 0) warpLen[warp] = __popc(leaders);
    __syncthreads();
    if (c >= 0) {
      int r = base[c] + rankInWarp;
      for (int q = 0; q < warp; q++)
        for (int k = 0; k < warpLen[q]; k++)
          if (warpList[q][k].x == c) r += warpList[q][k].y;
      w.a.colorBodies[r] = i;
      w.a.colorRec[r] = make_int4(i, w.a.cstart[i], min(w.a.cstart[i + 1], w.a.ccap), 0);
    }
    __syncthreads();
    for (int q = 0; q < (int)(blockDim.x >> 5); q++)  // advance the bases past this tile
      for (int k = threadIdx.x; k < warpLen[q]; k += blockDim.x) atomicAdd(&base[warpList[q][k].x], warpList[q][k].y);
    __syncthreads();
  }
  if (!coloring_barrier(w, arrivals)) return;
  lane_layout(w, arrivals);
}

// Smallest colour no neighbour of higher priority holds, searched in windows
// of 64 colours: one pass unless all of 0..63 are taken.
template <class F>
__device__ __forceinline__ int smallest_free_color(F &&neighbors) {
  for (int base = 0; base < kMaxColors; base += 64) {
    unsigned long long used = 0ull;
    neighbors([&](int c) {
      if (c >= base && c < base + 64) used |= 1ull << (c - base);
    });
    if (~used) return base + __ffsll((long long)~used) - 1;
  }
  return -1;
}

__global__ void __launch_bounds__(256) coloring_kernel(World w) {
  if (step_skipped(w)) return;  // every block reads the same value: none waits at a barrier
  Control *ctl = w.ctl;
  const int n = w.b.n;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  volatile int *color = w.b.color;
  unsigned arrivals = 0;
  // an uploaded colouring (copied and checked by the kernels before this
  // one) is used when proper; otherwise the priority colouring is computed
  if (w.a.colorOverride) {
    if (*((volatile int *)&ctl->colorBad) == 0) {
      coloring_finish(w, arrivals);
      return;
    }
    if (tid == 0) atomicOr(&ctl->flags, kErrColoring);
  }
  // seed: previous colours (statics -1, new dynamic bodies 0)
  for (int i = tid; i < n; i += stride) {
    if (!(w.b.flags0[i] & kBodyDynamic)) color[i] = -1;
    else if (color[i] < 0 || color[i] >= kMaxColors) color[i] = 0;
  }
  // "changed" flags, triple-buffered: round r sets flag r % 3 and clears the
  // flag of round r + 1, which no block can still be reading (it was last
  // read in round r - 2, before the barriers of round r - 1).
  if (tid == 0) ctl->pad[1] = 0;
  int round = 0;
  for (;; round++) {
    if (tid == 0) ctl->pad[1 + (round + 1) % 3] = 0;
    if (!coloring_barrier(w, arrivals)) return;
    int changed = 0;
    for (int i = tid; i < n; i += stride) {
      if (!(w.b.flags0[i] & kBodyDynamic)) continue;
      const int hb = w.a.start[i], hc = w.a.hpCount[i];
      int c = smallest_free_color([&](auto &&mark) {
        for (int k = 0; k < hc; k++) mark(color[w.a.hpEntry[hb + k]]);
        if (w.g.hasConstraints)
          constraint_neighbors(w, i, [&](int j) {
            if (precedes(w, j, i)) mark(color[j]);
          });
      });
      if (c < 0) {
        c = kMaxColors - 1;
        atomicOr(&ctl->flags, kOvfColors);
      }
      if (c != color[i]) {
        color[i] = c;
        changed = 1;
      }
    }
    if (changed) atomicOr(&ctl->pad[1 + round % 3], 1);
    if (!coloring_barrier(w, arrivals)) return;
    const int any = *((volatile int *)&ctl->pad[1 + round % 3]);
    if (!any) break;
    if (round > 4096) {
      if (tid == 0) atomicOr(&ctl->flags, kOvfColors);
      break;
    }
  }
  coloring_finish(w, arrivals);
}

// x_{t+1} = x_t + delta (f64); statics: prevVel <- vel (solver.js:479).
// Also the step's bookkeeping: its candidates become the next step's previous
// manifolds, or, for a skipped step, the skip is counted and nothing moves.
__global__ void commit_kernel(World w) {
  await_previous();
  if (step_skipped(w)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) w.ctl->stepsSkipped++;
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) w.ctl->prevCandidates = w.ctl->numCandidates;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < w.b.n; i += gridDim.x * blockDim.x) {
    const int fl = w.b.flags[i];
    if (!(fl & kBodyDynamic)) {
      w.b.prevVel[i] = w.b.vel[i];
      continue;
    }
    D4 p = w.b.pos[i];
    double dx, dy, dz;
    if (fl & kBodyFp64) {
      const D4 d = w.b.dpD[i];
      dx = d.x; dy = d.y; dz = d.z;
    } else {
      const float4 d = w.b.dp[i];
      dx = d.x; dy = d.y; dz = d.z;
    }
    p.x += dx; p.y += dy; p.z += dz;
    const float4 q = w.b.quat[i];
    if (!isfinite(p.x + p.y + p.z) || !isfinite(q.x + q.y + q.z + q.w)) atomicOr(&w.ctl->flags, kErrNaN);
    w.b.pos[i] = p;
  }
}

__global__ void stats_kernel(World w, double *out) {
  // out[0] max penetration, out[1] max |lambda|, out[2] max penalty (contacts + joints + springs)
  double e = 0, l = 0, k = 0;
  const int total = w.ctl->numCandidates;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
    const int n = w.cur.count[c];
    for (int s = 0; s < n; s++) {
      const float4 kk = w.cur.cK[c * kMaxContacts + s], ll = w.cur.cL[c * kMaxContacts + s];
      l = fmax(l, fmax(fabs((double)ll.x), fmax(fabs((double)ll.y), fabs((double)ll.z))));
      k = fmax(k, fmax((double)kk.x, fmax((double)kk.y, (double)kk.z)));
    }
  }
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < w.j.n; j += gridDim.x * blockDim.x) {
    if (w.j.state[j] & kRemoved) continue;
    const D4 a = w.j.lamLin[j], b = w.j.lamAng[j];
    l = fmax(l, sqrt(fmax(a.x * a.x + a.y * a.y + a.z * a.z, b.x * b.x + b.y * b.y + b.z * b.z)));
    const float4 p = w.j.penLin[j], q = w.j.penAng[j];
    k = fmax(k, fmax(fmax((double)p.x, fmax((double)p.y, (double)p.z)), fmax((double)q.x, fmax((double)q.y, (double)q.z))));
  }
  typedef cub::BlockReduce<double, 256> R;
  __shared__ typename R::TempStorage t0, t1, t2;
  const double me = R(t0).Reduce(e, ::cuda::maximum<>{});
  const double ml = R(t1).Reduce(l, ::cuda::maximum<>{});
  const double mk = R(t2).Reduce(k, ::cuda::maximum<>{});
  if (threadIdx.x == 0) {
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long *>(&out[0]), __double_as_longlong(me));
    atomicMax(reinterpret_cast<unsigned long long *>(&out[1]), __double_as_longlong(ml));
    atomicMax(reinterpret_cast<unsigned long long *>(&out[2]), __double_as_longlong(mk));
  }
}

}  // namespace

void launch_prepare(const World &w, cudaStream_t st, int smCount) {
  const int blocks = smCount * 4;
  if (w.j.n + w.s.n > 0) launch_early(prepare_forces_kernel, blocks, 256, st, w);
  launch_early(prepare_bodies_kernel, blocks, 256, st, w);
  if (w.b.n < kAdjAlone) {
    launch_early(adj_small_kernel, 1, kAdjAlone, st, w);
  } else {
    launch_early(adj_count_kernel, blocks, 256, st, w);
    launch_early(adj_scan_kernel, w.b.n / 256 + 1, 256, st, w);
    launch_early(adj_fill_kernel, blocks, 256, st, w);
  }
  launch_early(adj_sort_kernel, blocks, 256, st, w);
}

// One block up to kColorAlone bodies, whose dozen barriers then stay in the
// block (a pile of 60 / 120 bodies: 29 -> 21 / 45 -> 27 us). Beyond, a block
// per 64 bodies, so that they wait for few blocks, at most two an SM. (One
// block would be ahead up to 500 bodies, 43 us for 49, but these barriers are
// also where the wait limit is met in steps of the wavefront schedule whose
// bodies do not wait for one another.)
constexpr int kColorAlone = 128;
int coloring_grid(int n, int smCount) {
  int perSm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, coloring_kernel, 256, 0);
  return n <= kColorAlone ? 1 : std::max(1, std::min((n + 63) / 64, std::min(perSm, 2) * smCount));
}

// An uploaded colouring: copied, then checked against this step's graph.
__global__ void color_copy_kernel(World w) {
  if (step_skipped(w)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) w.ctl->colorBad = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < w.b.n; i += gridDim.x * blockDim.x)
    w.b.color[i] = (w.b.flags0[i] & kBodyDynamic) ? w.a.colorOverride[i] : -1;
}

__global__ void color_check_kernel(World w) {
  if (step_skipped(w)) return;
  int bad = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < w.b.n && !bad; i += gridDim.x * blockDim.x) {
    if (!(w.b.flags0[i] & kBodyDynamic)) continue;
    const int ci = w.b.color[i];
    if (ci < 0 || ci >= kMaxColors) {
      bad = 1;
      break;
    }
    // a conflicting edge is in the higher-priority list of one of its ends
    const int hb = w.a.start[i], hc = w.a.hpCount[i];
    for (int k = 0; k < hc && !bad; k++) bad = w.b.color[w.a.hpEntry[hb + k]] == ci;
    if (w.g.hasConstraints) constraint_neighbors(w, i, [&](int j) { bad |= w.b.color[j] == ci ? 1 : 0; });
  }
  if (bad) atomicOr(&w.ctl->colorBad, 1);
}

cudaError_t launch_coloring(const World &w, cudaStream_t st, int blocks) {
  if (w.a.colorOverride) {
    color_copy_kernel<<<blocks * 2, 256, 0, st>>>(w);
    color_check_kernel<<<blocks * 2, 256, 0, st>>>(w);
  }
  World arg = w;
  void *args[] = {&arg};
  return cudaLaunchCooperativeKernel((void *)coloring_kernel, dim3(blocks), dim3(256), args, 0,
                                     st);
}

// The grab, set between steps (avbd_set_grab); body < 0 releases it.
static __global__ void grab_kernel(Grab *g, int body, D4 local, D4 target, double k) {
  g->body = body;
  g->target = target;
  g->localD = local;
  g->local = make_float4((float)local.x, (float)local.y, (float)local.z, 0.f);
  g->k = k;
}

cudaError_t launch_set_grab(const World &w, int body, const double *local, const double *target, double k,
                            cudaStream_t st) {
  const D4 l = local ? mkd4(local[0], local[1], local[2], 0.0) : mkd4(0, 0, 0, 0);
  const D4 t = target ? mkd4(target[0], target[1], target[2], 0.0) : mkd4(0, 0, 0, 0);
  grab_kernel<<<1, 1, 0, st>>>(w.grab, body, l, t, k);
  return cudaGetLastError();
}

// A joint's anchor on body A, set between steps (avbd_update_joint_anchor).
static __global__ void joint_anchor_kernel(World w, int j, double x, double y, double z) {
  const_cast<D4 *>(w.j.rAD)[j] = mkd4(x, y, z, 0.0);
  const_cast<float4 *>(w.j.rAF)[j] = make_float4((float)x, (float)y, (float)z, 0.f);
}

cudaError_t launch_joint_anchor(const World &w, int joint, double x, double y, double z, cudaStream_t st) {
  joint_anchor_kernel<<<1, 1, 0, st>>>(w, joint, x, y, z);
  return cudaGetLastError();
}

static const void *solve_instance(const World &w, bool wave) {
  const bool forces = w.g.hasConstraints != 0, fp64 = w.p.mayFp64 != 0;
  if (w.p.contactModel != 0)
    return (fp64 ? solve_materials_forces_fp64 : forces ? solve_materials_forces : solve_materials)(wave);
  return (fp64 ? solve_forces_fp64 : forces ? solve_forces : solve_plain)(wave);
}

// Of the two kernels that this world's steps can launch (either schedule).
int solve_max_blocks_per_sm(const World &w) {
  int best = 1 << 30;
  for (int wave = 0; wave < 2; wave++) {
    const void *f = solve_instance(w, wave != 0);
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSolveSmem);
    int a = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, f, kSolveBlock, kSolveSmem);
    best = a < best ? a : best;
  }
  return best;
}

// lanesPerBody: the wavefront schedule's lanes per body (the colour-phase
// schedule reads its layout from the colouring).
cudaError_t launch_solve(const World &w, int lanesPerBody, int blocksPerSm, cudaStream_t st, int smCount) {
  World arg = w;
  int G = lanesPerBody;
  void *args2[] = {&arg, &G};
  void *args1[] = {&arg};
  const bool wave = w.p.schedule == 1;
  return cudaLaunchCooperativeKernel(solve_instance(w, wave), dim3(blocksPerSm * smCount), dim3(kSolveBlock),
                                     wave ? args2 : args1, kSolveSmem, st);
}

void launch_commit(const World &w, cudaStream_t st, int smCount) { launch_early(commit_kernel, smCount * 4, 256, st, w); }

void launch_stats(const World &w, double *out3, cudaStream_t st, int smCount) {
  cudaMemsetAsync(out3, 0, sizeof(double) * 3, st);
  stats_kernel<<<smCount * 2, 256, 0, st>>>(w, out3);
}

}  // namespace avbd
