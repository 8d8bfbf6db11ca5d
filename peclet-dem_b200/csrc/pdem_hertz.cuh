// Hertz-Mindlin soft-sphere engine (src/solver_hertz.hpp:41-606, src/sim.hpp:545-750).
//
// Explicit force model on a cached Verlet pair list: a touching pair's force, torques and Mindlin history
// are computed by one thread, which notes the pair with its two bodies; each body then takes its
// pairs' contributions in pair order and its wall contributions in wall order (the reference's atomic
// order in the serial build), then a symplectic kick-drift. The pair list is rebuilt when any body moved half
// the skin; the shear history is carried across rebuilds by pair key (both lists in pair order, binary search).
#pragma once
#include <climits>

#include "pdem_common.cuh"

namespace pdem {

template <class R>
__device__ __forceinline__ R hertzBetaD(R e) {
  if (e <= R(0))
    return R(-1);
  if (e >= R(1))
    return R(0);
  const R le = log(e);
  return le / sqrt(le * le + R(9.8696044));
}
template <class R>
__device__ __forceinline__ V3<R> hertzForce(R delta, V3<R> nh, V3<R> vr, R rS, R mS, R eS, R gS, R e, R mu,
                                            R dt, V3<R>& xi) {
  const R sq = sqrt(rS * delta);
  const R sn = R(2) * eS * sq;
  const R st = R(8) * gS * sq;
  const R kn = (R(4) / R(3)) * eS * sq;
  const R bd = hertzBetaD(e);
  const R etaN = R(-2) * R(0.9128709) * bd * sqrt(sn * mS);
  const R etaT = R(-2) * R(0.9128709) * bd * sqrt(st * mS);
  const R vn = dot(vr, nh);
  const R fs = kn * delta;
  const R fn = fs - etaN * vn;
  const V3<R> vt = sub(vr, mul(nh, vn));
  xi = add(xi, mul(vt, dt));
  xi = sub(xi, mul(nh, dot(xi, nh)));
  V3<R> ft = add(mul(xi, -st), mul(vt, -etaT));
  const R fl = sqrt(dot(ft, ft));
  const R fm = mu * fabs(fs);
  if (fl > fm) {
    const R s = (fl > R(1e-20)) ? fm / fl : R(0);
    ft = mul(ft, s);
    if (st > R(1e-20))
      xi = mul(add(ft, mul(vt, etaT)), R(-1) / st);
  }
  return add(mul(nh, fn), ft);
}
template <class R>
__device__ __forceinline__ void hertzStars(const Dev<R>& d, int ma, int mb, R& eS, R& gS) {
  const R Ei = d.hzE[ma], Ej = d.hzE[mb], ni = d.hzNu[ma], nj = d.hzNu[mb];
  eS = R(1) / ((R(1) - ni * ni) / Ei + (R(1) - nj * nj) / Ej);
  gS = R(1) / (R(2) * (R(2) - ni) * (R(1) + ni) / Ei + R(2) * (R(2) - nj) * (R(1) + nj) / Ej);
}
template <class R>
__device__ __forceinline__ void hertzEMu(const Dev<R>& d, int ma, int mb, R eG, R muG, R& e, R& mu) {
  if (d.pairMat) {
    const int t = (ma * kMaxMaterials + mb) * 2;
    e = d.pairMat[t];
    mu = d.pairMat[t + 1];
  } else {
    e = eG;
    mu = muG;
  }
}

template <class R>
struct HertzP {
  R dt, eG, muG, globalScale, contactFrac;
  int numWalls;
};

// The touching pairs of each of the n bodies (2 pair + side), in any order: cnt[body] of them at slot +
// off[body], where the body has room for all its pairs of the list; sorted: the same room, for the ones of a
// body of many pairs in order; many: the blocks of kBlock bodies with one that has room for more than
// kHertzScan. A list that the XPBD step wrote in between may name its ghost slots (n and up): they exert
// forces, as in the reference, and take none.
constexpr int kHertzSort = 16, kHertzScan = 32;
struct HertzTouch {
  int* cnt;
  const int* off;
  int *slot, *sorted;
  const uint8_t* many;
  int n;
};
__device__ __forceinline__ void hertzNote(const HertzTouch& H, int pair, int i, int j) {
  if (i < H.n)
    H.slot[H.off[i] + atomicAdd(&H.cnt[i], 1)] = 2 * pair;
  if (j < H.n)
    H.slot[H.off[j] + atomicAdd(&H.cnt[j], 1)] = 2 * pair + 1;
}
// count (at most N) of a body's pairs in ascending order, sorted in registers
template <int N, class TAKE>
__device__ __forceinline__ void hertzSorted(const int* mine, int count, TAKE&& take) {
  int node[N];
#pragma unroll
  for (int k = 0; k < N; ++k)
    node[k] = k < count ? mine[k] : INT_MAX;
#pragma unroll
  for (int p = 1; p < N; ++p)
#pragma unroll
    for (int k = p; k > 0; --k) {
      const int lo = min(node[k - 1], node[k]), hi = max(node[k - 1], node[k]);
      node[k - 1] = lo;
      node[k] = hi;
    }
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (k < count)
      take(node[k]);
}
// pairs of each body in a list that the XPBD step wrote (a rebuild's kHertzCarry counts its own)
template <class R>
__global__ void kHertzCount(Dev<R> d, int np, int n, int* cnt) {
  GRID_STRIDE(idx, np) {
    const int2 ij = d.pairs[idx];
    if (ij.x < n)
      atomicAdd(&cnt[ij.x], 1);
    if (ij.y < n)
      atomicAdd(&cnt[ij.y], 1);
  }
}
// room for each body's pairs, in any order of the bodies (taken: used so far); the counts start again
static __global__ void __launch_bounds__(kBlock) kHertzRoom(int n, int* cnt, int* off, int* taken, uint8_t* many) {
  __shared__ int sWarp[kBlock / 32];
  const int tid = threadIdx.x, lane = tid & 31;
  for (long b0 = (long)blockIdx.x * kBlock; b0 < n; b0 += (long)gridDim.x * kBlock) {
    const long b = b0 + tid;
    const int want = b < n ? cnt[b] : 0;
    int x = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o)
        x += y;
    }
    if (lane == 31)
      sWarp[tid >> 5] = x;
    const int any = __syncthreads_or(want > kHertzScan);
    if (tid == 0) {
      int sum = 0;
      for (int w = 0; w < kBlock / 32; ++w)
        sum += sWarp[w];
      int at = atomicAdd(taken, sum);
      for (int w = 0; w < kBlock / 32; ++w) {
        const int c = sWarp[w];
        sWarp[w] = at;
        at += c;
      }
      many[b0 / kBlock] = any != 0;
    }
    __syncthreads();
    if (b < n) {
      off[b] = sWarp[tid >> 5] + x - want;
      cnt[b] = 0;
    }
    __syncthreads();  // the warps' places are read before the next ones
  }
}

// positions with radii of all body slots, one load a body in the pair test
template <class R>
__global__ void kHertzPosRad(Dev<R> d, int n, Q4<R>* pr) {
  GRID_STRIDE(i, n) {
    const V3<R> x = v3(d.pos[i]);
    pr[i] = Q4<R>{x.x, x.y, x.z, d.rad[i]};
  }
}

// sphere pairs (src/solver_hertz.hpp:88-144): per-pair force F on i, torques tA on i and tB on j.
// Some 7 % of the pairs of a packing's Verlet list touch. A block tests a tile, WAYS pairs a thread so that
// their loads are in flight together, then computes the touching ones with full warps. An apart pair's history
// is cleared only where the pair's bit says that it may be set: on (bit = pair) holds the pairs that touched
// last, or all after a rebuild. 1.5 million pairs of 262,144 spheres, FP32: 48 us as one thread a pair that
// cleared every history and wrote a flag for each.
// WAYS: kHertzWays from kHertzTileFrom pairs, below that one, since the touching pairs of a small list would be
// few blocks' work in turn. Calls of 100 substeps, four ways against one: 8,000 loose spheres (46,000 pairs) FP64
// 5.25 and 5.00 ms, 30,000 (174,000) 5.50 and 5.93, 262,144 14.2 and 19.2; FP32 4.96 and 4.61, 5.21 and 5.17, 9.8
// and 11.5. 8,000 spheres in a close packing, 12 contacts each (60,000): FP64 6.37 and 5.22, FP32 5.28 and 4.50.
constexpr int kHertzWays = 4, kHertzTileFrom = 100000;
template <class R, int WAYS>
__global__ void __launch_bounds__(kBlock) kHertzPairs(Dev<R> d, int np, HertzP<R> P, const Q4<R>* pr, unsigned* on,
                                                      Q4<R>* xi, Q4<R>* F, Q4<R>* TA, Q4<R>* TB, HertzTouch H) {
  constexpr int kHertzTile = WAYS * kBlock;
  __shared__ int sList[kHertzTile], sCount;
  for (long first = (long)blockIdx.x * kHertzTile; first < np; first += (long)gridDim.x * kHertzTile) {
    if (threadIdx.x == 0)
      sCount = 0;
    __syncthreads();
    bool touch[WAYS];
#pragma unroll
    for (int q = 0; q < WAYS; ++q) {
      const long idx = first + q * kBlock + threadIdx.x;
      touch[q] = false;
      if (idx < np) {
        const int2 ij = d.pairs[idx];
        const Q4<R> a = pr[ij.x], b = pr[ij.y];
        const V3<R> dx = sub(v3(a), v3(b));
        const R d2 = dot(dx, dx), rr = a.w + b.w;
        if (!(d2 > rr * rr * R(1.0001))) {  // else apart whatever the rounding
          const R dd = sqrt(d2);
          touch[q] = !(rr - dd <= R(0) || dd < R(1e-12));
        }
      }
    }
#pragma unroll
    for (int q = 0; q < WAYS; ++q) {
      const long idx = first + q * kBlock + threadIdx.x;
      const unsigned now = __ballot_sync(0xffffffffu, touch[q]);
      const long word = idx >> 5;
      const unsigned was = (idx - (threadIdx.x & 31)) < np ? on[word] : 0u;
      if (touch[q])
        sList[atomicAdd(&sCount, 1)] = (int)idx;
      else if (idx < np && (was >> (threadIdx.x & 31) & 1u))
        xi[idx] = Q4<R>{0, 0, 0, 0};
      __syncwarp();
      if ((threadIdx.x & 31) == 0 && idx < np && now != was)
        on[word] = now;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < sCount; t += kBlock) {
      const int idx = sList[t];
      const int2 ij = d.pairs[idx];
      const int i = ij.x, j = ij.y;
      const Q4<R> a = pr[i], b = pr[j];
      const V3<R> dx = sub(v3(a), v3(b));
      const R dd = sqrt(dot(dx, dx));
      const R ri = a.w, rj = b.w;
      const R delta = ri + rj - dd;
      const V3<R> nh = mul(dx, R(1) / dd);
      const V3<R> rA = mul(nh, -(ri - R(0.5) * delta));
      const V3<R> rB = mul(nh, (rj - R(0.5) * delta));
      const V3<R> vr =
          sub(add(v3(d.vel[i]), cross(v3(d.angVel[i]), rA)), add(v3(d.vel[j]), cross(v3(d.angVel[j]), rB)));
      const int ma = d.matId[i], mb = d.matId[j];
      R e, mu, eS, gS;
      hertzEMu(d, ma, mb, P.eG, P.muG, e, mu);
      hertzStars(d, ma, mb, eS, gS);
      const R rS = ri * rj / (ri + rj);
      const R imS = d.invMass[i] + d.invMass[j];
      const R mS = (imS > R(0)) ? R(1) / imS : R(0);
      V3<R> x = v3(xi[idx]);
      const V3<R> f = hertzForce(delta, nh, vr, rS, mS, eS, gS, e, mu, P.dt, x);
      xi[idx] = q4(x);
      F[idx] = q4(f);
      TA[idx] = q4(cross(rA, f));
      TB[idx] = q4(cross(rB, mul(f, R(-1))));
      hertzNote(H, idx, i, j);
    }
    __syncthreads();  // the list is read before the next tile's
  }
}

// point-shell pairs (src/solver_hertz.hpp:454-606), one thread per pair (ordered sums over points)
template <class R>
__global__ void kHertzShapePairs(Dev<R> d, int np, HertzP<R> P, Q4<R>* xi, R* snPrev, Q4<R>* F, Q4<R>* TA, Q4<R>* TB,
                                 HertzTouch H) {
  const ShapeDesc<R> dA = d.shapes[0], dB = d.shapes[0];
  GRID_STRIDE(idx, np) {
    const int2 pr = d.pairs[idx];
    const int A = pr.x, B = pr.y;
    const V3<R> pA = v3(d.pos[A]), pB = v3(d.pos[B]);
    const Q4<R> qA = d.quat[A], qB = d.quat[B];
    const R sA = d.scale[A] * P.globalScale, sB = d.scale[B] * P.globalScale;
    const int cnt = dA.numPoints;
    const bool sphA = dA.type == SHAPE_SPHERE;
    const int iter = cnt > 0 ? cnt : 1;
    const int ma = d.matId[A], mb = d.matId[B];
    R e, mu, eS, gS;
    hertzEMu(d, ma, mb, P.eG, P.muG, e, mu);
    hertzStars(d, ma, mb, eS, gS);
    const R rcA = (sphA ? R(1) : P.contactFrac) * dA.par[0] * sA;
    const R rcB = ((dB.type == SHAPE_SPHERE) ? R(1) : P.contactFrac) * dB.par[0] * sB;
    const R rS = rcA * rcB / (rcA + rcB);
    const R imS = d.invMass[A] + d.invMass[B];
    const R mS = (imS > R(0)) ? R(1) / imS : R(0);
    const R bd = hertzBetaD(e);
    const V3<R> vA = v3(d.vel[A]), wA = v3(d.angVel[A]), vB = v3(d.vel[B]), wB = v3(d.angVel[B]);
    R fnSum = 0, snSum = 0, dMax = 0;
    V3<R> cSum{0, 0, 0}, nSum{0, 0, 0}, fAcc{0, 0, 0}, tA{0, 0, 0}, tB{0, 0, 0};
    const R snP = snPrev[idx];
    const R dampC = (mS > R(0)) ? R(-2) * R(0.9128709) * bd * sqrt(mS) : R(0);
    for (int k = 0; k < iter; ++k) {
      V3<R> pl{0, 0, 0};
      R prad = 0;
      if (cnt > 0)
        pl = v3(d.shell[dA.shellOffset + k]);
      else if (sphA)
        prad = dA.par[0] * sA;
      const V3<R> pw = add(pA, rot(qA, mul(pl, sA)));
      const V3<R> pc = mul(invrot(qB, sub(pw, pB)), R(1) / sB);
      const R dist = sdfShape(pc, dB, d.sdfGrid) * sB;
      const R eff = dist - prad;
      if (eff >= R(0))
        continue;
      const R delta = -eff;
      const V3<R> nl = sdfNormal(pc, dB, d.sdfGrid, R(1e-4));
      const V3<R> nW = rot(qB, nl);
      const V3<R> ps = sub(pw, mul(nW, prad));
      const V3<R> rA = sub(ps, pA);
      const V3<R> rB = sub(add(ps, mul(nW, delta)), pB);
      const V3<R> vrP = sub(add(vA, cross(wA, rA)), add(vB, cross(wB, rB)));
      const R vnP = dot(vrP, nW);
      const R sq = sqrt(rS * delta);
      const R fs = (R(4) / R(3)) * eS * sq * delta;
      const R snI = R(2) * eS * sq;
      const R snTot = (snP > snI) ? snP : snI;
      const R eta = dampC * snI / sqrt(snTot);
      const V3<R> f = mul(nW, fs - eta * vnP);
      fAcc = add(fAcc, f);
      tA = add(tA, cross(rA, f));
      tB = add(tB, cross(rB, mul(f, R(-1))));
      fnSum += fs;
      snSum += R(2) * eS * sq;
      cSum = add(cSum, mul(ps, fs));
      nSum = add(nSum, mul(nW, fs));
      if (delta > dMax)
        dMax = delta;
    }
    if (fnSum <= R(0)) {
      xi[idx] = Q4<R>{0, 0, 0, 0};
      snPrev[idx] = R(0);
      continue;
    }
    const V3<R> cpt = mul(cSum, R(1) / fnSum);
    V3<R> nh = nSum;
    const R nl2 = vlen(nh);
    if (nl2 > R(1e-9))
      nh = mul(nh, R(1) / nl2);
    const V3<R> rA = sub(cpt, pA), rB = sub(cpt, pB);
    const V3<R> vr = sub(add(vA, cross(wA, rA)), add(vB, cross(wB, rB)));
    snPrev[idx] = snSum;
    const V3<R> vt = sub(vr, mul(nh, dot(vr, nh)));
    const R st = R(8) * gS * sqrt(rS * dMax);
    const R etaT = R(-2) * R(0.9128709) * bd * sqrt(st * mS);
    V3<R> x = v3(xi[idx]);
    x = add(x, mul(vt, P.dt));
    x = sub(x, mul(nh, dot(x, nh)));
    V3<R> ft = add(mul(x, -st), mul(vt, -etaT));
    const R fl = vlen(ft);
    const R fm = mu * fnSum;
    if (fl > fm) {
      const R s = (fl > R(1e-20)) ? fm / fl : R(0);
      ft = mul(ft, s);
      if (st > R(1e-20))
        x = mul(add(ft, mul(vt, etaT)), R(-1) / st);
    }
    xi[idx] = q4(x);
    fAcc = add(fAcc, ft);
    tA = add(tA, cross(rA, ft));
    tB = add(tB, cross(rB, mul(ft, R(-1))));
    F[idx] = q4(fAcc);
    TA[idx] = q4(tA);
    TB[idx] = q4(tB);
    hertzNote(H, (int)idx, A, B);
  }
}

// wall candidates (src/solver_hertz.hpp:343-370), counted per particle then written in (i, wall)
// order: code i * 8 + wall
template <class R, int MODE>
__global__ void kHertzWallCand(Dev<R> d, int n, int numWalls, R skin, int* cnt, const int* off, int* out, int cap) {
  GRID_STRIDE(i, n) {
    const V3<R> p = v3(d.pos[i]);
    int c = 0;
    for (int wi = 0; wi < numWalls; ++wi) {
      const R s = sampleWall(p, d.walls[wi], d.wallGrid);
      if (s < d.rad[i] + skin) {
        if (MODE) {
          const int at = off[i] + c;
          if (at < cap)
            out[at] = (int)i * 8 + wi;
        }
        ++c;
      }
    }
    if (!MODE)
      cnt[i] = c;
  }
}

// wall forces per candidate (src/solver_hertz.hpp:148-338)
template <class R>
__global__ void kHertzWalls(Dev<R> d, int ncand, HertzP<R> P, const int* cand, Q4<R>* xiWall, R* snWall,
                            int hasShapes, Q4<R>* F, Q4<R>* T, int* on) {
  GRID_STRIDE(ci, ncand) {
    on[ci] = 0;
    const int enc = cand[ci];
    const int i = enc / 8, wi = enc % 8;
    const V3<R> p = v3(d.pos[i]);
    const R r = d.rad[i];
    const WallDesc<R>& w = d.walls[wi];
    const int slot = i * kHertzMaxWalls + wi;
    const int ma = d.matId[i];
    R e, mu;
    if (w.materialId >= 0 && d.pairMat)
      hertzEMu(d, ma, w.materialId, P.eG, P.muG, e, mu);
    else {
      e = w.restitution;
      mu = w.friction;
    }
    const int mw = (w.materialId >= 0) ? w.materialId : ma;
    R eS, gS;
    hertzStars(d, ma, mw, eS, gS);
    const R mS = (d.invMass[i] > R(0)) ? R(1) / d.invMass[i] : R(0);
    const V3<R> wl{w.linVel[0], w.linVel[1], w.linVel[2]}, wa{w.angVel[0], w.angVel[1], w.angVel[2]},
        wc{w.center[0], w.center[1], w.center[2]};
    const ShapeDesc<R> dS = d.shapes[d.shapeId[i]];
    if (hasShapes && dS.numPoints > 0) {
      const Q4<R> qP = d.quat[i];
      const R es = d.scale[i] * P.globalScale;
      const R rc = P.contactFrac * dS.par[0] * es;
      const R bd = hertzBetaD(e);
      const V3<R> vP = v3(d.vel[i]), wP = v3(d.angVel[i]);
      const R snP = snWall[slot];
      const R dampC = (mS > R(0)) ? R(-2) * R(0.9128709) * bd * sqrt(mS) : R(0);
      R fnSum = 0, snSum = 0, dMax = 0;
      V3<R> cSum{0, 0, 0}, nSum{0, 0, 0}, fAcc{0, 0, 0}, tAcc{0, 0, 0};
      for (int k = 0; k < dS.numPoints; ++k) {
        const V3<R> pW = add(p, rot(qP, mul(v3(d.shell[dS.shellOffset + k]), es)));
        const R sd = sampleWall(pW, w, d.wallGrid);
        if (sd >= R(0))
          continue;
        const R delta = -sd;
        const R hx = R(0.5) / w.invSpacing[0];
        const V3<R> gr = wallGradient(pW, w, d.wallGrid, hx);
        const R gl = vlen(gr);
        if (gl < R(1e-12))
          continue;
        const V3<R> nh = mul(gr, R(1) / gl);
        const V3<R> rA = sub(pW, p);
        const V3<R> vW = add(wl, cross(wa, sub(pW, wc)));
        const V3<R> vrP = sub(add(vP, cross(wP, rA)), vW);
        const R vnP = dot(vrP, nh);
        const R sq = sqrt(rc * delta);
        const R fs = (R(4) / R(3)) * eS * sq * delta;
        const R snI = R(2) * eS * sq;
        const R snTot = (snP > snI) ? snP : snI;
        const R eta = dampC * snI / sqrt(snTot);
        const V3<R> f = mul(nh, fs - eta * vnP);
        fAcc = add(fAcc, f);
        tAcc = add(tAcc, cross(rA, f));
        fnSum += fs;
        snSum += R(2) * eS * sq;
        cSum = add(cSum, mul(pW, fs));
        nSum = add(nSum, mul(nh, fs));
        if (delta > dMax)
          dMax = delta;
      }
      if (fnSum <= R(0)) {
        xiWall[slot] = Q4<R>{0, 0, 0, 0};
        snWall[slot] = R(0);
        continue;
      }
      const V3<R> cpt = mul(cSum, R(1) / fnSum);
      V3<R> nh = nSum;
      const R nl = vlen(nh);
      if (nl > R(1e-9))
        nh = mul(nh, R(1) / nl);
      const V3<R> rA = sub(cpt, p);
      const V3<R> vW = add(wl, cross(wa, sub(cpt, wc)));
      const V3<R> vr = sub(add(vP, cross(wP, rA)), vW);
      snWall[slot] = snSum;
      const V3<R> vt = sub(vr, mul(nh, dot(vr, nh)));
      const R st = R(8) * gS * sqrt(rc * dMax);
      const R etaT = R(-2) * R(0.9128709) * bd * sqrt(st * mS);
      V3<R> x = v3(xiWall[slot]);
      x = add(x, mul(vt, P.dt));
      x = sub(x, mul(nh, dot(x, nh)));
      V3<R> ft = add(mul(x, -st), mul(vt, -etaT));
      const R fl = vlen(ft);
      const R fm = mu * fnSum;
      if (fl > fm) {
        const R s2 = (fl > R(1e-20)) ? fm / fl : R(0);
        ft = mul(ft, s2);
        if (st > R(1e-20))
          x = mul(add(ft, mul(vt, etaT)), R(-1) / st);
      }
      xiWall[slot] = q4(x);
      fAcc = add(fAcc, ft);
      tAcc = add(tAcc, cross(rA, ft));
      F[ci] = q4(fAcc);
      T[ci] = q4(tAcc);
      on[ci] = 1;
      continue;
    }
    const R sw = sampleWall(p, w, d.wallGrid);
    const R delta = r - sw;
    if (delta <= R(0)) {
      xiWall[slot] = Q4<R>{0, 0, 0, 0};
      continue;
    }
    const R hx = R(0.5) / w.invSpacing[0];
    const V3<R> gr = wallGradient(p, w, d.wallGrid, hx);
    const R gl = sqrt(dot(gr, gr));
    if (gl < R(1e-12))
      continue;
    const V3<R> nh = mul(gr, R(1) / gl);
    const V3<R> rA = mul(nh, -(r - R(0.5) * delta));
    const V3<R> cpt = add(p, rA);
    const V3<R> vW = add(wl, cross(wa, sub(cpt, wc)));
    const V3<R> vr = sub(add(v3(d.vel[i]), cross(v3(d.angVel[i]), rA)), vW);
    V3<R> x = v3(xiWall[slot]);
    const V3<R> f = hertzForce(delta, nh, vr, r, mS, eS, gS, e, mu, P.dt, x);
    xiWall[slot] = q4(x);
    F[ci] = q4(f);
    T[ci] = q4(cross(rA, f));
    on[ci] = 1;
  }
}

// per body: pair contributions in pair order, then wall contributions in wall order; then the
// symplectic kick-drift (src/solver_hertz.hpp:374-425) with the forces consumed. first: the call's first
// substep, which takes over what the delta arrays hold (normally zero) and clears them. Up to kHertzSort
// pairs of a body are sorted in registers (half of them in a smaller network), up to kHertzScan taken by repeated
// minimum; the pairs of a larger grain are ranked by its whole block and summed in that order, one component a
// thread.
// Before, a thread walked its body's whole incidence list (some 12 pairs, a flag each): 43 us of 262,144
// spheres, FP32. A call of 40 substeps with one grain of 5 R (147 touching) among 3,000, FP64: 6.3-6.7 ms by
// that walk, 4.0 so (19.7 by repeated minimum over a chain of all its pairs); eight such among 20,000: 8.2 and
// 5.5. 8,000 spheres with 12 contacts each, 100 substeps, FP64: 5.11 ms by the walk, 5.22 so, 5.6 with up to 8
// sorted in registers.
template <class R>
__global__ void __launch_bounds__(kBlock) kHertzGatherIntegrate(Dev<R> d, int n, HertzTouch H, const Q4<R>* F,
                                                                const Q4<R>* TA, const Q4<R>* TB, const int* candOff,
                                                                int ncand, const Q4<R>* FW, const Q4<R>* TW,
                                                                const int* onW, V3<R> g, R dt, int orient, int first,
                                                                Q4<R>* pr) {
  __shared__ R sVal[6][kBlock + 1], sSum[2][6];
  __shared__ int sMany[kBlock], sManys;
  const int tid = threadIdx.x;
  for (long base = (long)blockIdx.x * kBlock; base < n; base += (long)gridDim.x * kBlock) {
    const long i = base + tid;
    V3<R> f{0, 0, 0}, t{0, 0, 0};
    if (first && i < n) {
      // the reference accumulates into the (normally zero) delta arrays it uses as force/torque
      f = v3(d.dVel[i]);
      t = v3(d.dAngVel[i]);
      d.dVel[i] = Q4<R>{0, 0, 0, 0};
      d.dAngVel[i] = Q4<R>{0, 0, 0, 0};
    }
    auto take = [&](int node) {
      const int idx = node >> 1;
      if ((node & 1) == 0) {
        f = add(f, v3(F[idx]));
        t = add(t, v3(TA[idx]));
      } else {
        f = add(f, neg(v3(F[idx])));
        t = add(t, v3(TB[idx]));
      }
    };
    const bool many = H.many[base / kBlock] != 0;  // uniform over the block
    const int count = i < n ? H.cnt[i] : 0;
    if (count > 0 && count <= kHertzScan) {
      const int* mine = H.slot + H.off[i];
      if (count <= kHertzSort / 2) {
        hertzSorted<kHertzSort / 2>(mine, count, take);
      } else if (count <= kHertzSort) {
        hertzSorted<kHertzSort>(mine, count, take);
      } else {
        for (int last = -1, k = 0; k < count; ++k) {
          int best = INT_MAX;
          for (int q = 0; q < count; ++q) {
            const int v = mine[q];
            best = v > last && v < best ? v : best;
          }
          take(best);
          last = best;
        }
      }
    }
    if (many && __syncthreads_or(count > kHertzScan)) {
      if (tid == 0)
        sManys = 0;
      __syncthreads();
      if (count > kHertzScan)
        sMany[atomicAdd(&sManys, 1)] = tid;
      __syncthreads();
      for (int q = 0; q < sManys; ++q) {
        const int who = sMany[q], c = H.cnt[base + who], o = H.off[base + who];
        R* sum = sSum[q & 1];
        if (tid == who) {
          sum[0] = f.x, sum[1] = f.y, sum[2] = f.z;
          sum[3] = t.x, sum[4] = t.y, sum[5] = t.z;
        }
        for (int k = tid; k < c; k += kBlock) {
          const int v = H.slot[o + k];
          int rank = 0;
          for (int m = 0; m < c; ++m)
            rank += H.slot[o + m] < v ? 1 : 0;
          H.sorted[o + rank] = v;
        }
        __syncthreads();
        R acc = tid < 6 ? sum[tid] : R(0);
        for (int k0 = 0; k0 < c; k0 += kBlock) {
          const int m = min(kBlock, c - k0);
          if (tid < m) {
            const int node = H.sorted[o + k0 + tid], idx = node >> 1;
            const V3<R> v = (node & 1) == 0 ? v3(F[idx]) : neg(v3(F[idx]));
            const V3<R> w = v3((node & 1) == 0 ? TA[idx] : TB[idx]);
            sVal[0][tid] = v.x, sVal[1][tid] = v.y, sVal[2][tid] = v.z;
            sVal[3][tid] = w.x, sVal[4][tid] = w.y, sVal[5][tid] = w.z;
          }
          __syncthreads();
          if (tid < 6)
            for (int j = 0; j < m; ++j)
              acc = acc + sVal[tid][j];
          __syncthreads();
        }
        if (tid < 6)
          sum[tid] = acc;
        __syncthreads();
        if (tid == who) {
          f = V3<R>{sum[0], sum[1], sum[2]};
          t = V3<R>{sum[3], sum[4], sum[5]};
        }
      }
    }
    if (i >= n)
      continue;
    if (count > 0)
      H.cnt[i] = 0;
    if (candOff)
      for (int q = candOff[i]; q < candOff[i + 1] && q < ncand; ++q)
        if (onW[q]) {
          f = add(f, v3(FW[q]));
          t = add(t, v3(TW[q]));
        }
    const R im = d.invMass[i];
    if (im > R(0)) {
      const V3<R> iI = v3(d.invI[i]);
      V3<R> dw;
      if (iI.x == iI.y && iI.y == iI.z) {
        dw = V3<R>{t.x * iI.x, t.y * iI.x, t.z * iI.x};
      } else {
        const V3<R> tl = invrot(d.quat[i], t);
        dw = rot(d.quat[i], V3<R>{tl.x * iI.x, tl.y * iI.y, tl.z * iI.z});
      }
      V3<R> v = v3(d.vel[i]), w = v3(d.angVel[i]), x = v3(d.pos[i]);
      v.x += (f.x * im + g.x) * dt;
      w.x += dw.x * dt;
      x.x += v.x * dt;
      v.y += (f.y * im + g.y) * dt;
      w.y += dw.y * dt;
      x.y += v.y * dt;
      v.z += (f.z * im + g.z) * dt;
      w.z += dw.z * dt;
      x.z += v.z * dt;
      d.vel[i] = q4(v);
      d.angVel[i] = q4(w);
      d.pos[i] = q4(x);
      pr[i] = Q4<R>{x.x, x.y, x.z, pr[i].w};
      if (orient) {
        Q4<R> q = d.quat[i];
        const Q4<R> dq{R(0.5) * dt * (w.x * q.w + w.y * q.z - w.z * q.y),
                       R(0.5) * dt * (w.y * q.w + w.z * q.x - w.x * q.z),
                       R(0.5) * dt * (w.z * q.w + w.x * q.y - w.y * q.x),
                       R(0.5) * dt * (-w.x * q.x - w.y * q.y - w.z * q.z)};
        q = Q4<R>{q.x + dq.x, q.y + dq.y, q.z + dq.z, q.w + dq.w};
        const R qn = sqrt(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
        if (qn > R(1e-12))
          d.quat[i] = Q4<R>{q.x / qn, q.y / qn, q.z / qn, q.w / qn};
      }
    }
  }
}

template <class R>
__global__ void kHertzMaxDisp2(Dev<R> d, int n, const Q4<R>* ref, R* out) {
  R mx = R(0);
  GRID_STRIDE(i, n) {
    const V3<R> dd = sub(v3(d.pos[i]), v3(ref[i]));
    runMax(mx, dot(dd, dd));
  }
  blockMaxAtomic(out, mx);  // one atomic per block on the one word
}
// carry the shear history onto the rebuilt list (src/sim.hpp:558-585). Both lists are in (first, second
// body) order, so the old one is searched as it stands; its keys are (larger << 32 | smaller). cnt: the
// pairs of each body.
__device__ __forceinline__ u64 hertzOrder(u64 k) { return (k << 32) | (k >> 32); }
template <class R>
__global__ void kHertzCarry(Dev<R> d, int np, int prevCount, const u64* prevKeys, const Q4<R>* prevXi, u64* keys,
                            Q4<R>* xi, int* cnt) {
  const int lane = threadIdx.x & 31;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx - lane < np; idx += (long)gridDim.x * blockDim.x) {
    const int2 pr = idx < np ? d.pairs[idx] : make_int2(-1, -1);
    // a body's pairs as the first one are consecutive: one count for the warp's part of them
    const bool head = __shfl_up_sync(0xffffffffu, pr.x, 1) != pr.x || lane == 0;
    const unsigned after = __ballot_sync(0xffffffffu, head) >> lane >> 1;
    if (idx >= np)
      continue;
    if (head)
      atomicAdd(&cnt[pr.x], after ? __ffs(after) : 32 - lane);
    atomicAdd(&cnt[pr.y], 1);
    const unsigned a = (unsigned)pr.x, b = (unsigned)pr.y;
    const unsigned lo = a < b ? a : b, hi = a < b ? b : a;
    const u64 k = ((u64)hi << 32) | lo, o = hertzOrder(k);
    keys[idx] = k;
    int l = 0, h = prevCount;
    while (l < h) {
      const int m = (l + h) >> 1;
      if (hertzOrder(prevKeys[m]) < o)
        l = m + 1;
      else
        h = m;
    }
    const bool hit = l < prevCount && prevKeys[l] == k;
    xi[idx] = hit ? prevXi[l] : Q4<R>{0, 0, 0, 0};
  }
}

}  // namespace pdem
