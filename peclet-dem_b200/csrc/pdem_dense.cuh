// Position sweeps of dense contact graphs, where the 62 colours do not hold every contact: bodies with
// more than 62 contacts (point shells in line or face contact) leave many in the saturated colour,
// which the reference runs serially in contact order, and the ones the colouring's round limit left
// uncoloured take the Jacobi correction at the end of each sweep.
//
// The saturated colour as levels: consecutive contacts of one body pair form a run, and a run's level
// is one above the latest earlier run that shares a body. Runs of a level are body-disjoint and every
// body meets its runs in contact order, so the levels in turn, each run in its own order, give the
// serial result bit for bit. Half a warp takes a run (some 15 contacts of a pair): its lanes hold 16
// contacts' records and update the two bodies' positions in registers, one contact after the other.
//
// One persistent launch runs all sweeps: the colours, the levels and the Jacobi phases, with a barrier
// after each: one block with every body's position in shared memory (a barrier costs tens of cycles), one
// cluster, or a cooperative grid on the global positions. In the latter two successive levels of few runs are
// one block's, with block barriers, and levels of one run each (the contacts of one large grain) one warp's.
// Position stage of a substep with a grain of 20 R among 50,000 spheres, FP64: 36.2 ms with a grid barrier a
// level, 7.4 so (17.4 as one thread's serial loop); of 5 R among 8,000, one cluster: 2.70, 0.93 (1.70).
#pragma once
#include "pdem_flow.cuh"

namespace pdem {

constexpr int kDenseBlock = 512;
constexpr int kDenseBodies = 8192;  // bodies whose latest levels fit the run kernel's shared memory
constexpr size_t kDenseMaxSmem = 200 * 1024;

// runs of the saturated contacts and their levels (one block)
struct DenseRuns {
  int* start;   // [runs + 1] first entry (colour order) of each run, in contact order
  int* level;   // [runs]
  int* order;   // [runs] runs by level
  int* lvOff;   // [levels + 1]
  int* group;   // [groups + 1] first level of each group: one level, or levels of 2 to kDenseNarrow runs, or of one
  int* body;    // [bodies] scratch: latest level of each body
  int* count;   // [0] runs, [1] levels, [2] groups
};
constexpr int kDenseLanes = 16;                             // lanes of a run
constexpr int kDenseNarrow = kDenseBlock / kDenseLanes;     // runs that a block takes at once
template <class R>
__global__ void __launch_bounds__(1024) kDenseRuns(Dev<R> d, const int* order, const int* coff, int nb, DenseRuns D) {
  __shared__ int sWarp[32], sTotal;
  __shared__ int sBody[kDenseBodies];
  int* body = nb <= kDenseBodies ? sBody : D.body;
  const int b = coff[kSaturatedColor], n = coff[kSaturatedColor + 1] - b;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  auto key = [&](int t) {  // unordered pair
    const int2 ab = d.cab[order[b + t]];
    return ab.y >= 0 && ab.y < ab.x ? make_int2(ab.y, ab.x) : ab;
  };
  for (int i = tid; i < nb; i += blockDim.x)
    body[i] = 0;
  int runs = 0;
  for (int t0 = 0; t0 < n; t0 += blockDim.x) {  // run heads, ranked in order
    const int t = t0 + tid;
    int head = 0;
    if (t < n) {
      const int2 k = key(t);
      head = 1;
      if (t > 0) {
        const int2 p = key(t - 1);
        head = (p.x != k.x || p.y != k.y) ? 1 : 0;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, head);
    if (lane == 0)
      sWarp[w] = __popc(m);
    __syncthreads();
    if (tid == 0) {
      int run = 0;
      for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
        const int c = sWarp[q];
        sWarp[q] = run;
        run += c;
      }
      sTotal = run;
    }
    __syncthreads();
    if (head)
      D.start[runs + sWarp[w] + __popc(m & ((1u << lane) - 1u))] = b + t;
    runs += sTotal;
    __syncthreads();
  }
  if (tid == 0)
    D.start[runs] = b + n;
  __syncthreads();
  int levels = 0;
  if (w == 0) {  // levels in run order: 32 runs' bodies at a time, then one after the other
    for (int r0 = 0; r0 < runs; r0 += 32) {
      const int r = r0 + lane;
      int A = -1, B = -1;
      if (r < runs) {
        const int2 ab = d.cab[order[D.start[r]]];
        A = ab.x;
        B = ab.y;
      }
      int lv = 0;
      const int m = min(32, runs - r0);
      for (int k = 0; k < m; ++k) {
        if (lane == k) {
          int l = body[A];
          if (B >= 0)
            l = max(l, body[B]);
          lv = l;
          body[A] = l + 1;
          if (B >= 0)
            body[B] = l + 1;
        }
        __syncwarp();
      }
      if (r < runs)
        D.level[r] = lv;
      levels = max(levels, __reduce_max_sync(0xffffffffu, r < runs ? lv + 1 : 0));
    }
    if (lane == 0) {
      sTotal = levels;
      D.count[0] = runs;
      D.count[1] = levels;
    }
  }
  __syncthreads();
  levels = sTotal;
  // counting sort by level
  for (int l = tid; l <= levels; l += blockDim.x)
    D.lvOff[l] = 0;
  __syncthreads();
  for (int r = tid; r < runs; r += blockDim.x)
    atomicAdd(&D.lvOff[D.level[r]], 1);
  __syncthreads();
  if (tid == 0) {
    int run = 0, groups = 0;
    int before = 0;  // width of the level before: 0 wide, 1 narrow, 2 one run
    for (int l = 0; l < levels; ++l) {
      const int c = D.lvOff[l];
      D.lvOff[l] = run;
      run += c;
      const int width = c > kDenseNarrow ? 0 : c > 1 ? 1 : 2;
      if (width == 0 || width != before)
        D.group[groups++] = l;
      before = width;
    }
    D.lvOff[levels] = run;
    D.group[groups] = levels;
    D.count[2] = groups;
  }
  __syncthreads();
  for (int i = tid; i < levels; i += blockDim.x)
    D.level[runs + i] = D.lvOff[i];  // running positions (the level array has room for both)
  __syncthreads();
  for (int r = tid; r < runs; r += blockDim.x)
    D.order[atomicAdd(&D.level[runs + D.level[r]], 1)] = r;  // a level's runs are independent: any order
}

// per contact in colour order: posStatic's values, [0] (n, wT), [1] (rA, imA), [2] (rB, imB), and ids
template <class R>
struct DenseRecs {
  Q4<R>* q;  // [3 * cap], slot-major
  int4* ids; // contact, body A, body B
  long cap;
};
template <class R>
__global__ void kDensePack(Dev<R> d, const int* order, int ne, DenseRecs<R> r) {
  GRID_STRIDE(t, ne) {
    const int idx = order[t];
    const int2 ab = d.cab[idx];
    const PosStatic<R> s = posStatic(d, idx, ab.x, ab.y);
    r.q[t] = Q4<R>{s.n.x, s.n.y, s.n.z, s.wT};
    r.q[r.cap + t] = Q4<R>{s.rA.x, s.rA.y, s.rA.z, s.imA};
    r.q[2 * r.cap + t] = Q4<R>{s.rB.x, s.rB.y, s.rB.z, s.imB};
    r.ids[t] = make_int4(idx, ab.x, ab.y, 0);
  }
}
// the uncoloured contacts' ends (entry l of them), for their incidence lists
template <class R>
__global__ void kDenseLeftKeys(Dev<R> d, const int* order, int first, int n, int* keys, int* vals, int none) {
  GRID_STRIDE(l, n) {
    const int2 ab = d.cab[order[first + l]];
    keys[2 * l] = ab.x;
    vals[2 * l] = (int)(l << 1);
    keys[2 * l + 1] = ab.y >= 0 ? ab.y : none;
    vals[2 * l + 1] = (int)(l << 1 | 1);
  }
}

template <class R>
struct DenseRec {
  Q4<R> n, a, b;
  int4 id;
};
template <class R>
__device__ __forceinline__ DenseRec<R> denseLoad(const DenseRecs<R>& r, long t) {
  return DenseRec<R>{r.q[t], r.q[r.cap + t], r.q[2 * r.cap + t], r.ids[t]};
}
// posGSOne's update of pA, pB; returns the impulse (0: inactive) and raises mx
template <class R>
__device__ __forceinline__ bool denseUpdate(const DenseRec<R>& c, V3<R>& pA, V3<R>& pB, R& dl, R& mx) {
  const V3<R> n = v3(c.n), rA = v3(c.a), rB = v3(c.b);
  const bool hasB = c.id.z >= 0;
  const R C = hasB ? dot(sub(add(pA, rA), add(pB, rB)), n) : dot(sub(add(pA, rA), rB), n);
  if (C >= R(0) || c.n.w < R(1e-6))
    return false;
  dl = -C / c.n.w;
  pA = add(pA, V3<R>{n.x * dl * c.a.w, n.y * dl * c.a.w, n.z * dl * c.a.w});
  if (hasB)
    pB = add(pB, V3<R>{-n.x * dl * c.b.w, -n.y * dl * c.b.w, -n.z * dl * c.b.w});
  runMax(mx, -C);
  return true;
}
template <class R>
__device__ __forceinline__ V3<R> denseShfl(unsigned mask, V3<R> v, int lane) {
  return V3<R>{__shfl_sync(mask, v.x, lane, kDenseLanes), __shfl_sync(mask, v.y, lane, kDenseLanes),
               __shfl_sync(mask, v.z, lane, kDenseLanes)};
}

// left: uncoloured contacts, their incidence lists by body (entries l << 1 | side); corr, ok: [left]
enum { kDenseGrid, kDenseOne, kDenseCluster };
template <class R, int FORM>
__global__ void __launch_bounds__(kDenseBlock) kDenseSweeps(Dev<R> d, const int* coff, int ncol, int iters, R thr,
                                                            GridBar gb, DenseRecs<R> rec, DenseRuns D, int nb, int left,
                                                            Incidence inc, Q4<R>* corr, int* ok) {
  extern __shared__ __align__(32) unsigned char denseSmem[];
  __shared__ int sOff[kSaturatedColor + 3];
  __shared__ R sMax[kDenseBlock / 32];
  constexpr bool ONE = FORM == kDenseOne;
  Counters<R>* c = d.ctr;
  Q4<R>* pos = ONE ? reinterpret_cast<Q4<R>*>(denseSmem) : d.posPred;
  const int tid = threadIdx.x, lane = tid & 31;
  const long gtid = (long)blockIdx.x * blockDim.x + tid, gstride = (long)gridDim.x * blockDim.x;
  for (int k = tid; k < kSaturatedColor + 2; k += blockDim.x)
    sOff[k] = coff[k];
  if (ONE)
    for (int i = tid; i < nb; i += blockDim.x)
      pos[i] = d.posPred[i];
  __syncthreads();
  const int cols = min(ncol, kSaturatedColor);
  const int groups = ncol > kSaturatedColor ? D.count[ONE ? 1 : 2] : 0;
  const int leftAt = sOff[kSaturatedColor + 1];
  auto barrier = [&]() -> bool {
    if (ONE) {
      __syncthreads();
      return true;
    }
    return loopBarrier<FORM == kDenseCluster>(gb);
  };
  auto at = [&](int i) { return v3(pos[i]); };
  const int sub = lane % kDenseLanes;
  const unsigned half = ((1u << kDenseLanes) - 1u) << (lane - sub);
  // the runs of a level, half a warp a run
  auto level = [&](int lv, long id, long stride, R& mx) {
    const int r1 = D.lvOff[lv + 1];
    for (long k = D.lvOff[lv] + id / kDenseLanes; k < r1; k += stride / kDenseLanes) {
      const int run = D.order[k], s = D.start[run], e = D.start[run + 1];
      V3<R> p0{0, 0, 0}, p1{0, 0, 0};  // the run's bodies, in its first contact's order
      int A = 0, B = -1;
      for (int t0 = s; t0 < e; t0 += kDenseLanes) {
        const int t = t0 + sub, m = min(kDenseLanes, e - t0);
        DenseRec<R> q{};
        R lam = R(0);
        if (t < e) {
          q = denseLoad(rec, t);
          lam = d.posLamC[q.id.x];
        }
        if (t0 == s) {
          A = __shfl_sync(half, q.id.y, 0, kDenseLanes);
          B = __shfl_sync(half, q.id.z, 0, kDenseLanes);
          p0 = at(A);
          if (B >= 0)
            p1 = at(B);
        }
        const bool swap = t < e && q.id.y != A;
        for (int j = 0; j < m; ++j) {
          V3<R> a = swap ? p1 : p0, b = swap ? p0 : p1;
          if (sub == j) {
            R dl;
            if (denseUpdate(q, a, b, dl, mx))
              d.posLamC[q.id.x] = lam + dl;
          }
          p0 = denseShfl(half, swap ? b : a, j);
          p1 = denseShfl(half, swap ? a : b, j);
        }
      }
      if (sub == 0) {
        pos[A] = q4(p0);
        if (B >= 0)
          pos[B] = q4(p1);
      }
    }
  };
  // levels of one run each, by one warp: a lane a run, 32 runs' first records at a time
  auto chain = [&](int lv0, int lv1, R& mx) {
    for (int l0 = lv0; l0 < lv1; l0 += 32) {
      int t = 0, e = 0;
      DenseRec<R> q{};
      R lam = R(0);
      if (l0 + lane < lv1) {
        const int run = D.order[D.lvOff[l0 + lane]];
        t = D.start[run];
        e = D.start[run + 1];
        q = denseLoad(rec, t);
        lam = d.posLamC[q.id.x];
      }
      for (int j = 0; j < min(32, lv1 - l0); ++j) {
        if (lane == j) {
          const int A = q.id.y, B = q.id.z;
          V3<R> p0 = at(A), p1 = B >= 0 ? at(B) : V3<R>{0, 0, 0};
          for (;;) {
            R dl;
            if (q.id.y == A ? denseUpdate(q, p0, p1, dl, mx) : denseUpdate(q, p1, p0, dl, mx))
              d.posLamC[q.id.x] = lam + dl;
            if (++t >= e)
              break;
            q = denseLoad(rec, t);
            lam = d.posLamC[q.id.x];
          }
          pos[A] = q4(p0);
          if (B >= 0)
            pos[B] = q4(p1);
        }
        __syncwarp();
      }
    }
  };
  int it = 0;
  bool stop = false;
  for (; it < iters; ++it) {
    R mx = R(0);
    DenseRec<R> next;
    long tn = sOff[0] + gtid;
    if (tn < sOff[1])
      next = denseLoad(rec, tn);
    for (int col = 0; col < cols; ++col) {
      for (long t = sOff[col] + gtid; t < sOff[col + 1]; t += gstride) {
        const DenseRec<R> q = t == tn ? next : denseLoad(rec, t);
        V3<R> pA = at(q.id.y), pB = q.id.z >= 0 ? at(q.id.z) : V3<R>{0, 0, 0};
        R dl;
        if (denseUpdate(q, pA, pB, dl, mx)) {
          d.posLamC[q.id.x] += dl;
          pos[q.id.y] = q4(pA);
          if (q.id.z >= 0)
            pos[q.id.z] = q4(pB);
        }
      }
      if (col + 1 < cols) {  // the next colour's record before the barrier
        tn = sOff[col + 1] + gtid;
        if (tn < sOff[col + 2])
          next = denseLoad(rec, tn);
      }
      if (!barrier())
        return;
    }
    for (int g = 0; g < groups; ++g) {  // the saturated colour
      if (FORM == kDenseOne) {
        level(g, gtid, gstride, mx);
      } else {
        const int lv0 = D.group[g], lv1 = D.group[g + 1], runs = D.lvOff[lv0 + 1] - D.lvOff[lv0];
        if (runs > kDenseNarrow) {
          level(lv0, gtid, gstride, mx);
        } else if (blockIdx.x == 0) {
          if (runs > 1) {
            for (int lv = lv0; lv < lv1; ++lv) {
              level(lv, tid, blockDim.x, mx);
              __syncthreads();
            }
          } else if (tid < 32) {
            chain(lv0, lv1, mx);
          }
        }
      }
      if (!barrier())
        return;
    }
    if (left > 0) {  // Jacobi correction of the uncoloured contacts (src/solver_position.hpp:34-134)
      for (long l = gtid; l < left; l += gstride) {
        const DenseRec<R> q = denseLoad(rec, leftAt + l);
        V3<R> pA = at(q.id.y), pB = q.id.z >= 0 ? at(q.id.z) : V3<R>{0, 0, 0};
        R dl = R(0);
        const bool on = denseUpdate(q, pA, pB, dl, mx);
        ok[l] = on ? 1 : 0;
        if (on)
          corr[l] = Q4<R>{q.n.x, q.n.y, q.n.z, dl};
      }
      if (!barrier())
        return;
      for (long b = gtid; b < nb; b += gstride) {
        const int s = inc.off[b], e = inc.off[b + 1];
        if (s == e)
          continue;
        V3<R> dp = v3(d.dPos[b]);
        int cnt = d.counts[b];
        const R im = d.invMass[b];
        for (int q = s; q < e; ++q) {
          const int l = inc.ent[q] >> 1, side = inc.ent[q] & 1;
          if (!__ldcg(&ok[l]))
            continue;
          const Q4<R> v{__ldcg(&corr[l].x), __ldcg(&corr[l].y), __ldcg(&corr[l].z), __ldcg(&corr[l].w)};
          const R dl = v.w;
          if (side == 0)
            dp = add(dp, V3<R>{v.x * dl * im, v.y * dl * im, v.z * dl * im});
          else
            dp = add(dp, V3<R>{-v.x * dl * im, -v.y * dl * im, -v.z * dl * im});
          cnt += 1;
        }
        if (cnt > 0) {  // kApplyUpdates
          const R f = R(1) / static_cast<R>(cnt);
          pos[b] = q4(add(at((int)b), mul(dp, f)));
          d.velPred[b] = q4(add(v3(d.velPred[b]), mul(v3(d.dVel[b]), f)));
          d.dPos[b] = Q4<R>{0, 0, 0, 0};
          d.dVel[b] = Q4<R>{0, 0, 0, 0};
          d.counts[b] = 0;
        }
      }
    }
    // END of this sweep, then BEGIN of the next one
    if (ONE) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const R w = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = w > mx ? w : mx;
      }
      if (lane == 0)
        sMax[tid >> 5] = mx;
      __syncthreads();
      if (tid == 0) {
        R m = sMax[0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k)
          m = sMax[k] > m ? sMax[k] : m;
        sMax[0] = m;
      }
      __syncthreads();
      const R m = sMax[0];
      stop = m < thr;
      if (tid == 0) {
        c->maxOverlap = m;
        if (stop)
          c->posDone = 1;
        else if (it + 1 < iters)
          c->posSweeps += 1;
      }
      __syncthreads();
    } else {
      warpMaxAtomic(&c->maxOverlap, mx);
      if (!barrier())
        return;
      if (gtid == 0) {
        const R m = *reinterpret_cast<volatile R*>(&c->maxOverlap);
        if (m < thr) {
          *reinterpret_cast<volatile int*>(&c->posDone) = 1;
        } else if (it + 1 < iters) {
          *reinterpret_cast<volatile R*>(&c->maxOverlap) = R(0);
          c->posSweeps += 1;
        }
      }
      if (!barrier())
        return;
      stop = *reinterpret_cast<volatile int*>(&c->posDone) != 0;
    }
    if (stop)
      break;
  }
  if (ONE)
    for (int i = tid; i < nb; i += blockDim.x)
      d.posPred[i] = pos[i];
}

}  // namespace pdem
