// Coloured Gauss-Seidel sweeps as a flow of body states between entries.
//
// A colour step of a packed bed is bound by latency: one update a thread (its dependent loads, a
// chain of some 140 floating-point operations with divisions and square roots, its stores) and a
// barrier over all blocks. Here a sweep has no colour barrier: each entry (manifold or contact) of
// the colour order belongs to one thread and owns a mailbox a side; when an entry has updated a body
// it sends the body's new state to the mailbox of the next entry of that body (the next colour of the
// body's colour mask, cyclic over the sweeps), and an entry starts as soon as its own mailboxes hold
// this sweep's states. Every body passes through its entries in colour order, each update is the one
// of the colour-by-colour loop on the same values, so the results are the same bits. The blocks meet
// once a sweep, for the adaptive stop, and the next sweep's first update runs while they do.
//
// A state travels as 16-byte packets of three words and a tag (the sweep), each written and read as
// one 128-bit access, so no fence or flag separates data from arrival; the warps of a cluster hand the
// sweep's maximum round in the same way. Two places for the mailboxes:
//   CLUSTER  shared memory of one thread-block cluster (remote shared-memory stores), for graphs
//            whose mailboxes fit;
//   else     global memory, the blocks of one cooperative launch.
// Records: an entry's per-substep constants, one contiguous record an entry in colour order. A warp's
// next 32 records come into shared memory as one bulk copy (mbarrier) while it computes the current
// ones; what does not depend on the states is computed before they arrive, and the stop's maximum and
// the impulses' stores come after the states have been sent.
//
// Order is safe: an entry waits only for entries of lower colours of its sweep or of the previous
// sweep, a sweep that the stop rules out is known before any wait for its states, every thread takes its
// entries in colour order, and all blocks are resident. A mailbox is
// written again only after its entry has read it, since the writer's input passed through that entry.
// Every wait is bounded (GridBar::spins; kBarrierSpins for a record's copy): on time-out the error bit is
// set and the thread goes on without waiting, so the launch ends.
#pragma once
#include <cstring>

#include "pdem_persist.cuh"

namespace pdem {

// A block's entries of a colour go to one group of four warps (one a scheduler); the two groups take the
// colours in turn, so that a group stores its impulses and prepares its next entries while the other
// one computes.
constexpr int kFlowGroup = 128, kFlowGroups = 2, kFlowBlock = kFlowGroup * kFlowGroups;
constexpr size_t kFlowMaxSmem = 212 * 1024;  // dynamic shared memory of a block
constexpr int kFlowItems = 512;  // most (colour, 128-entry chunk) items of a block
// words of the global control block: [0] arrivals, [2 + 2 k] the sweeps' maxima (64-bit, k = sweep % 3)
constexpr int kFlowCtlWords = 8;

// entry flags (ids.w)
constexpr int kFlowHasB = 1, kFlowFirstA = 2, kFlowFirstB = 4, kFlowSelf = 8, kFlowSideShift = 8;

// KIND 0: velocity sweep (pgsSolve's update), 2: position sweep (posGSOne's)
template <class R, int KIND>
struct FlowShape {
  static constexpr int kValues = KIND == 0 ? 6 : 3;                        // values of a body's state
  static constexpr int kPackets = (kValues * (int)sizeof(R) / 4 + 2) / 3;  // 16-byte packets a state
  static constexpr int kSlots = KIND == 0 ? 11 : 3;                        // 4-value slots of a record
  static constexpr int kIds = kSlots * (int)sizeof(Q4<R>);                 // byte offset of the ids, then the links
  // record bytes: a multiple of 16 and, in 16-byte units, odd, so that the eight lanes of a 128-bit
  // shared load phase meet all 32 banks
  static constexpr int kStride = ((kIds + 24 + 15) / 16 | 1) * 16;
  static constexpr int kStageBytes = kFlowBlock * kStride;                 // one record a thread
  static constexpr int kSlotBytes = 2 * kPackets * 16;                     // mailboxes of one entry
};

template <class R>
struct FlowRecs {
  char* rec;    // [cap] records: slots, ids (manifold / contact, body A, body B, flags), links
  Q4<R>* var;   // KIND 0: tangential impulse and normal impulse in colour order
  R* lam;       // KIND 2: the position impulse in colour order
  uint4* box;   // global mailboxes, 2 * kPackets * cap
  unsigned* ctl;
  long cap;
  unsigned tag0;  // tags of this launch: tag0 + sweep + 1
};
// a side's link: where it sends, target << 2 | next sweep << 1 | target side

// entries of a colour per block, and the first mailbox slot of each colour in its block
__device__ __forceinline__ int flowPerBlock(int n, int nb) { return (n + nb - 1) / nb; }

// ---- 128-bit single accesses --------------------------------------------------------------------
__device__ __forceinline__ void flowStoreRemote(unsigned addr, unsigned x, unsigned y, unsigned z, unsigned w) {
  asm volatile(
      "{\n .reg .b128 q;\n .reg .b64 lo, hi;\n mov.b64 lo, {%1, %2};\n mov.b64 hi, {%3, %4};\n mov.b128 q, {lo, hi};\n"
      " st.relaxed.cluster.shared::cluster.b128 [%0], q;\n}" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ uint4 flowLoadShared(unsigned addr) {
  uint4 v;
  asm volatile(
      "{\n .reg .b128 q;\n .reg .b64 lo, hi;\n ld.relaxed.cluster.shared::cta.b128 q, [%4];\n mov.b128 {lo, hi}, q;\n"
      " mov.b64 {%0, %1}, lo;\n mov.b64 {%2, %3}, hi;\n}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "r"(addr)
      : "memory");
  return v;
}
__device__ __forceinline__ unsigned flowRemoteAddr(unsigned local, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ unsigned flowShared(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// one bulk copy of `bytes` (a multiple of 16) from global memory, completed on the mbarrier
__device__ __forceinline__ void flowBulk(unsigned smem, const void* g, unsigned bytes, unsigned mbar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem),
               "l"(g), "r"(bytes), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ bool flowBulkDone(unsigned mbar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0u;
}

// values <-> words
__device__ __forceinline__ void flowWords(const double* v, int n, unsigned* w) {
  for (int k = 0; k < n; ++k) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v[k]);
    w[2 * k] = (unsigned)u;
    w[2 * k + 1] = (unsigned)(u >> 32);
  }
}
__device__ __forceinline__ void flowWords(const float* v, int n, unsigned* w) {
  for (int k = 0; k < n; ++k)
    w[k] = __float_as_uint(v[k]);
}
__device__ __forceinline__ void flowValues(const unsigned* w, int n, double* v) {
  for (int k = 0; k < n; ++k)
    v[k] = __longlong_as_double((long long)(((unsigned long long)w[2 * k + 1] << 32) | w[2 * k]));
}
__device__ __forceinline__ void flowValues(const unsigned* w, int n, float* v) {
  for (int k = 0; k < n; ++k)
    v[k] = __uint_as_float(w[k]);
}

// ---- records -------------------------------------------------------------------------------------
// velocity records (KIND 0): slots 0 (N, lenN), 1 (TA, vn0), 2 (TB, wAn0), 3 (dc, wBn0), 4 (rAa, imA),
// 5 (rBa, imB), 6 (wvN, eAvg), 7 (iIA, muAvg), 8 (iIB, position impulse), 9 qA, 10 qB: each the
// expression the sweep evaluates (pgsStatic). position records (KIND 2): 0 (n, wT), 1 (rA, imA), 2 (rB
// or a wall's contact point, imB): posConstraint's, whose orientations do not change while the
// position loop runs. Also the table of each body's entry of a colour, tab[body * colours + colour].
template <class R>
struct PosStatic {
  V3<R> n, rA, rB;
  R wT, imA, imB;
};
template <class R>
__device__ __forceinline__ PosStatic<R> posStatic(const Dev<R>& d, int idx, int A, int B) {
  PosStatic<R> s;
  s.imA = d.invMass[A];
  s.imB = B >= 0 ? d.invMass[B] : R(0);
  const V3<R> cn = v3(d.cn[idx]), crA = v3(d.crA[idx]), crB = v3(d.crB[idx]);
  s.rA = rot(qmul(d.quatPred[A], qinv(d.quat[A])), crA);
  s.rB = crB;
  s.n = cn;
  if (B >= 0) {
    const Q4<R> qBd = qmul(d.quatPred[B], qinv(d.quat[B]));
    s.rB = rot(qBd, crB);
    s.n = rot(qBd, cn);
  }
  const V3<R> iA = v3(d.invI[A]), iB = B >= 0 ? v3(d.invI[B]) : V3<R>{0, 0, 0};
  s.wT = computeW(s.rA, s.n, s.imA, iA) + computeW(s.rB, s.n, s.imB, iB);
  return s;
}
// slot k of a record (16-byte aligned)
__device__ __forceinline__ void flowPut(char* p, int k, const Q4<double>& v) {
  *reinterpret_cast<double2*>(p + 32 * k) = make_double2(v.x, v.y);
  *reinterpret_cast<double2*>(p + 32 * k + 16) = make_double2(v.z, v.w);
}
__device__ __forceinline__ void flowPut(char* p, int k, const Q4<float>& v) {
  *reinterpret_cast<float4*>(p + 16 * k) = make_float4(v.x, v.y, v.z, v.w);
}
template <class R, int KIND>
__global__ void kFlowPack(Dev<R> d, const int* order, const int* coff, int ncol, const u64* mask, int* tab, FlowRecs<R> r) {
  using F = FlowShape<R, KIND>;
  const long n = coff[ncol];
  GRID_STRIDE(t, n) {
    char* q = r.rec + t * F::kStride;
    auto put = [&](int k, Q4<R> v) { flowPut(q, k, v); };
    const int idx = order[t];
    int A, B, col, f = 0;
    if (KIND == 0) {
      const PgsStatic<R> s = pgsStatic(d, idx);
      put(0, Q4<R>{s.N.x, s.N.y, s.N.z, s.lenN});
      put(1, Q4<R>{s.TA.x, s.TA.y, s.TA.z, d.vn0[idx]});
      put(2, Q4<R>{s.TB.x, s.TB.y, s.TB.z, s.wAn0});
      put(3, Q4<R>{s.dc.x, s.dc.y, s.dc.z, s.wBn0});
      put(4, Q4<R>{s.rAa.x, s.rAa.y, s.rAa.z, s.imA});
      put(5, Q4<R>{s.rBa.x, s.rBa.y, s.rBa.z, s.imB});
      put(6, Q4<R>{s.wvN.x, s.wvN.y, s.wvN.z, s.eAvg});
      put(7, Q4<R>{s.iIA.x, s.iIA.y, s.iIA.z, s.muAvg});
      put(8, Q4<R>{s.iIB.x, s.iIB.y, s.iIB.z, d.posImp[idx]});
      put(9, s.qA);
      put(10, s.qB);
      const Q4<R> lt = d.lambdaT[idx];
      r.var[t] = Q4<R>{lt.x, lt.y, lt.z, d.lambda[idx]};
      A = s.ra;
      B = s.hasB ? s.rb : -1;
      col = d.mColor[idx];
      f = (int)d.sideFlags[idx] << kFlowSideShift;
    } else {
      const int2 ab = d.cab[idx];
      A = ab.x;
      B = ab.y;
      const PosStatic<R> s = posStatic(d, idx, A, B);
      put(0, Q4<R>{s.n.x, s.n.y, s.n.z, s.wT});
      put(1, Q4<R>{s.rA.x, s.rA.y, s.rA.z, s.imA});
      put(2, Q4<R>{s.rB.x, s.rB.y, s.rB.z, s.imB});
      r.lam[t] = R(0);
      col = d.cColor[idx];
    }
    const u64 lower = (1ull << col) - 1ull;
    if (!(mask[A] & lower))
      f |= kFlowFirstA;
    tab[(long)A * ncol + col] = (int)(t << 1);
    if (B >= 0) {
      f |= kFlowHasB;
      if (A == B) {
        f |= kFlowSelf;  // a body and its own periodic image: one state, through side A's mailbox
      } else {
        if (!(mask[B] & lower))
          f |= kFlowFirstB;
        tab[(long)B * ncol + col] = (int)(t << 1 | 1);
      }
    }
    *reinterpret_cast<int4*>(r.rec + t * F::kStride + F::kIds) = make_int4(idx, A, B, f);
  }
}
template <class R>
__device__ __forceinline__ PgsStatic<R> flowRecord(const char* rec, long t, int& idx) {
  using F = FlowShape<R, 0>;
  const char* q = rec + t * F::kStride;
  auto slot = [&](int k) {
    Q4<R> v;
    if constexpr (sizeof(R) == 8) {
      const double2 a = *reinterpret_cast<const double2*>(q + 32 * k), b = *reinterpret_cast<const double2*>(q + 32 * k + 16);
      v = Q4<R>{a.x, a.y, b.x, b.y};
    } else {
      const float4 a = *reinterpret_cast<const float4*>(q + 16 * k);
      v = Q4<R>{a.x, a.y, a.z, a.w};
    }
    return v;
  };
  const int4 id = *reinterpret_cast<const int4*>(q + F::kIds);
  const Q4<R> q0 = slot(0), q1 = slot(1), q2 = slot(2), q3 = slot(3), q4 = slot(4), q5 = slot(5), q6 = slot(6), q7 = slot(7);
  PgsStatic<R> s;
  idx = id.x, s.ra = id.y, s.rb = id.z, s.hasB = (id.w & kFlowHasB) != 0;
  s.Nsq = R(0);  // not read by the update
  s.N = v3(q0), s.lenN = q0.w, s.TA = v3(q1), s.TB = v3(q2), s.wAn0 = q2.w, s.dc = v3(q3), s.wBn0 = q3.w;
  s.rAa = v3(q4), s.imA = q4.w, s.rBa = v3(q5), s.imB = q5.w, s.wvN = v3(q6), s.eAvg = q6.w;
  s.iIA = v3(q7), s.muAvg = q7.w, s.iIB = v3(slot(8)), s.qA = slot(9), s.qB = slot(10);
  return s;
}
// link of each entry's sides to the next entry of the body; targets are mailbox slots of `nb` blocks
// (block << 14 | slot) or, with nb = 0, entries
static __global__ void __launch_bounds__(kFlowBlock) kFlowLink(const int* coff, int ncol, const u64* mask, const int* tab,
                                                               const int* color, char* rec, int recStride, int idsAt, int nb) {
  __shared__ int sOff[64], sPer[64], sBase[64];
  for (int k = threadIdx.x; k <= ncol; k += blockDim.x)
    sOff[k] = coff[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    int base = 0;
    for (int k = 0; k < ncol; ++k) {
      sPer[k] = nb > 0 ? flowPerBlock(sOff[k + 1] - sOff[k], nb) : 0;
      sBase[k] = base;
      base += sPer[k];
    }
  }
  __syncthreads();
  GRID_STRIDE(t, sOff[ncol]) {
    const int4 id = *reinterpret_cast<const int4*>(rec + t * recStride + idsAt);
    const int col = color[id.x];
    auto next = [&](int body) {
      const u64 m = mask[body];
      const u64 higher = col < 63 ? m >> (col + 1) << (col + 1) : 0ull;
      const int wrap = higher == 0ull ? 1 : 0;
      const int nc = __ffsll((long long)(wrap ? m : higher)) - 1;
      const int code = tab[(long)body * ncol + nc];
      int target = code >> 1;
      if (nb > 0) {
        const int i = target - sOff[nc];
        const int b = i / sPer[nc];
        target = (b << 14) | (sBase[nc] + i - b * sPer[nc]);
      }
      return (target << 2) | (wrap << 1) | (code & 1);
    };
    *reinterpret_cast<int2*>(rec + t * recStride + idsAt + 16) =
        make_int2(next(id.y), ((id.w & kFlowHasB) && !(id.w & kFlowSelf)) ? next(id.z) : 0);
  }
}

// ---- the velocity update --------------------------------------------------------------------------
// Quotient a / b with the correctly rounded reciprocal y = 1 / b known beforehand: two corrections of
// a y by the exact remainder (Markstein, IBM J. Res. Dev. 34, 1990: a quotient approximation within an
// ulp, corrected once by the remainder times the correctly rounded reciprocal, is the correctly rounded
// quotient unless b's significand is all ones). That case and operands whose remainder could underflow
// or overflow take a / b itself.
__host__ __device__ __forceinline__ double flowFma(double a, double b, double c) { return fma(a, b, c); }
__host__ __device__ __forceinline__ float flowFma(float a, float b, float c) { return fmaf(a, b, c); }
template <class R>
struct FlowRecip {
  R b, y;
  bool plain;  // take a / b
};
__host__ __device__ __forceinline__ bool flowAllOnes(double b) {
  long long u;
  memcpy(&u, &b, sizeof u);
  return (u & 0xfffffffffffffLL) == 0xfffffffffffffLL;
}
__host__ __device__ __forceinline__ bool flowAllOnes(float b) {
  int u;
  memcpy(&u, &b, sizeof u);
  return (u & 0x7fffff) == 0x7fffff;
}
template <class R>
__host__ __device__ __forceinline__ FlowRecip<R> flowRecip(R b) {
  const R big = sizeof(R) == 8 ? R(1e100) : R(1e10f), small = sizeof(R) == 8 ? R(1e-100) : R(1e-10f);
  FlowRecip<R> r;
  r.b = b;
  r.plain = !(fabs(b) < big) || !(fabs(b) > small) || flowAllOnes(b);
  r.y = R(1) / (r.plain ? R(1) : b);
  return r;
}
template <class R>
__host__ __device__ __forceinline__ R flowQuot(R a, const FlowRecip<R>& r) {
  const R big = sizeof(R) == 8 ? R(1e100) : R(1e15f), small = sizeof(R) == 8 ? R(1e-100) : R(1e-25f);
  if (r.plain || !(fabs(a) < big) || !(fabs(a) > small))
    return (a == R(0) && !r.plain) ? a * r.y : a / r.b;
  const R q0 = a * r.y;
  const R q1 = flowFma(flowFma(-q0, r.b, a), r.y, q0);
  return flowFma(flowFma(-q1, r.b, a), r.y, q1);
}

// pgsSolve's update in three parts: what the states do not enter (before they arrive), the states'
// chain, and the corrections that the adaptive stop compares (after the states are sent). Every value
// is pgsSolve's expression.
template <class R>
struct FlowPgs {
  bool ok, slow, hasB, applyA, applyB, hitN, hitT;
  int sf;
  R e, sgn, target, vgn, mu, beta, posImp, lenN, wAn, wBn, wT, wTt, dA, dd2, imA, imB;
  FlowRecip<R> rW;
  V3<R> nh;
};
template <class R>
__device__ __forceinline__ FlowPgs<R> flowPgsBegin(const PgsStatic<R>& v, int sf, R vn0, R posImp, R eG, R muG,
                                                   const SolveP<R>& P) {
  FlowPgs<R> f;
  f.hasB = v.hasB;
  f.sf = sf;
  f.lenN = v.lenN;
  f.posImp = posImp;
  f.wAn = sf == 2 ? R(0) : v.wAn0;
  f.wBn = sf == 1 ? R(0) : v.wBn0;
  f.applyA = sf != 2;
  f.applyB = v.hasB && sf != 1;
  f.wT = f.wAn + f.wBn;
  f.ok = !(v.lenN < R(1e-9)) && !(f.wT <= R(0));
  f.slow = fabs(vn0) < P.vRest * v.lenN;
  R e = v.eAvg >= R(0) ? v.eAvg : eG;
  if (sf != 0 || f.slow)
    e = R(0);
  f.sgn = dot(v.N, v.dc) > R(0) ? R(1) : R(-1);
  const R v0 = f.sgn * vn0;
  f.target = (v0 > R(0)) ? -e * v0 : R(0);
  f.vgn = dot(mul(v.dc, P.growthRate), v.N);
  f.nh = mul(v.N, R(1) / v.lenN);
  f.mu = v.muAvg >= R(0) ? v.muAvg : muG;
  f.beta = P.eT;
  if (f.beta != R(0) && (sf != 0 || f.slow))
    f.beta = R(0);
  f.rW = flowRecip<R>(f.wT);
  f.hitN = f.hitT = false;
  f.dA = f.dd2 = R(0);
  f.wTt = v.imA + v.imB;
  return f;
}
// returns bit 0: lam changed, bit 1: lt changed
template <class R, class VT0>
__device__ __forceinline__ int flowPgsStates(const PgsStatic<R>& v, FlowPgs<R>& f, VT0&& vt0, PgsVars<R>& x) {
  if (!f.ok)
    return 0;
  const bool hasB = f.hasB;
  const V3<R> vB = hasB ? x.v1 : v.wvN, wB = hasB ? x.w1 : V3<R>{0, 0, 0};
  R vn = dot(x.v0, v.N) + dot(x.w0, v.TA) + dot(vB, neg(v.N)) + dot(wB, v.TB);
  vn += f.vgn;
  const R dp = flowQuot<R>(f.sgn * vn - f.target, f.rW);
  const R pOld = x.lam;
  R pNew = pOld + dp;
  if (pNew < R(0))
    pNew = R(0);
  f.dA = pNew - pOld;
  V3<R> vA2 = x.v0, wA2 = x.w0, vB2 = vB, wB2 = wB;
  int changed = 0;
  if (f.dA != R(0)) {
    f.hitN = true;
    changed = 1;
    x.lam = pNew;
    const R lam = -f.sgn * f.dA;
    const V3<R> J = mul(v.N, lam), JA = mul(v.TA, lam), JB = mul(v.TB, lam);
    if (f.applyA) {
      vA2 = add(vA2, mul(J, v.imA));
      wA2 = add(wA2, angResponse(v.qA, JA, v.iIA));
    }
    if (f.applyB) {
      vB2 = add(vB2, mul(neg(J), v.imB));
      wB2 = add(wB2, angResponse(v.qB, JB, v.iIB));
    }
  }
  // friction cone
  const V3<R> ltOld = x.lt;
  if (f.mu > R(0) || nonzero(ltOld)) {
    const V3<R> nh = f.nh;
    const V3<R> vr = sub(add(vA2, cross(wA2, v.rAa)), add(vB2, cross(wB2, v.rBa)));
    const V3<R> vtv = sub(vr, mul(nh, dot(vr, nh)));
    V3<R> err = vtv;
    if (f.beta != R(0)) {
      V3<R> w0 = vt0();
      w0 = sub(w0, mul(nh, dot(w0, nh)));
      err = add(vtv, mul(w0, f.beta));
    }
    const R vl = sqrt(dot(err, err));
    V3<R> ltNew = ltOld;
    if (vl > R(1e-9)) {
      const V3<R> th = mul(err, R(1) / vl);
      const R wAt = (f.sf == 2) ? R(0) : v.imA + genInvMass(cross(v.rAa, th), v.iIA, v.qA);
      const R wBt = (f.sf == 1 || !hasB) ? R(0) : v.imB + genInvMass(cross(v.rBa, th), v.iIB, v.qB);
      f.wTt = wAt + wBt;
      if (f.wTt > R(1e-9))
        ltNew = add(ltOld, mul(th, -vl / f.wTt));
    }
    ltNew = sub(ltNew, mul(nh, dot(ltNew, nh)));
    R nTot = fmax(x.lam, R(0)) * v.lenN;
    if (f.slow)
      nTot += fmax(f.posImp, R(0));
    const R bound = f.mu * nTot;
    const R ll = sqrt(dot(ltNew, ltNew));
    if (ll > bound)
      ltNew = (bound > R(0)) ? mul(ltNew, bound / ll) : V3<R>{0, 0, 0};
    const V3<R> dd = sub(ltNew, ltOld);
    if (nonzero(dd)) {
      x.lt = ltNew;
      changed |= 2;
      f.hitT = true;
      f.dd2 = dot(dd, dd);
      if (f.applyA) {
        vA2 = add(vA2, mul(dd, v.imA));
        wA2 = add(wA2, angResponse(v.qA, cross(v.rAa, dd), v.iIA));
      }
      if (f.applyB) {
        vB2 = add(vB2, mul(neg(dd), v.imB));
        wB2 = add(wB2, angResponse(v.qB, cross(v.rBa, mul(dd, R(-1))), v.iIB));
      }
    }
  }
  x.v0 = vA2;
  x.w0 = wA2;
  if (hasB) {
    x.v1 = vB2;
    x.w1 = wB2;
  }
  return changed;
}
template <class R>
__device__ __forceinline__ void flowPgsReport(const FlowPgs<R>& f, R& mx) {
  if (f.hitN)
    runMax(mx, fabs(f.dA) * f.wT / f.lenN);
  if (f.hitT && f.wTt > R(1e-9))
    runMax(mx, sqrt(f.dd2) * f.wTt);
}
// keeps a value's computation above this point (before the wait for the states)
__device__ __forceinline__ void flowPin(double& v) { asm volatile("" : "+d"(v)); }
__device__ __forceinline__ void flowPin(float& v) { asm volatile("" : "+f"(v)); }

// ---- the loop ------------------------------------------------------------------------------------
// max of the sweep as ordered bits of a non-negative value
__device__ __forceinline__ unsigned long long flowBits(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ unsigned long long flowBits(float v) { return (unsigned long long)__float_as_uint(v); }
__device__ __forceinline__ double flowFromBits(unsigned long long u, double) { return __longlong_as_double((long long)u); }
__device__ __forceinline__ float flowFromBits(unsigned long long u, float) { return __uint_as_float((unsigned)u); }

// LOOP: 1 main velocity loop, 2 stabilization loop, 3 position loop. stride: mailbox slots of a block
// (CLUSTER). The host has already run the first sweep's BEGIN (kCtl).
template <class R, int KIND, int LOOP, bool CLUSTER>
__global__ void __launch_bounds__(kFlowBlock, 1) kFlowSweeps(Dev<R> d, const int* coff, int ncol, int iters, SolveP<R> P,
                                                            R thr, GridBar gb, FlowRecs<R> rec, int stride) {
  using F = FlowShape<R, KIND>;
  constexpr int NV = F::kValues, NP = F::kPackets, kWarps = kFlowBlock / 32;
  extern __shared__ __align__(16) unsigned char flowSmem[];
  __shared__ int sOff[64];
  __shared__ int3 sItem[kFlowItems];  // first entry, entries, first mailbox slot
  __shared__ int sItems;
  __shared__ unsigned long long sBar[kWarps];  // the warps' record copies
  // the warps' maxima of a sweep, by parity (CLUSTER): written by every warp of the cluster
  constexpr int kPosts = CLUSTER ? 16 * kWarps : 1;
  __shared__ __align__(16) uint4 sPost[2][kPosts];
  __shared__ unsigned long long sWarp[kWarps];
  Counters<R>* c = d.ctr;
  volatile int* done = LOOP == 1 ? &c->velDone : LOOP == 2 ? &c->stabDone : &c->posDone;
  if (*done)
    return;  // uniform over the launch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = gridDim.x, blk = blockIdx.x;
  for (int k = tid; k <= ncol; k += kFlowBlock)
    sOff[k] = coff[k];
  for (int k = tid; k < 2 * kPosts; k += kFlowBlock)
    (&sPost[0][0])[k] = make_uint4(0u, 0u, 0u, 0u);
  const unsigned bar = flowShared(&sBar[warp]);
  if (lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0) {
    int items = 0, base = 0;
    for (int k = 0; k < ncol; ++k) {
      const int n = sOff[k + 1] - sOff[k], per = flowPerBlock(n, nb);
      const int cnt = min(per, n - blk * per);
      for (int o = 0; o < cnt && items < kFlowItems; o += kFlowGroup)
        sItem[items++] = make_int3(sOff[k] + blk * per + o, min(kFlowGroup, cnt - o), base + o);
      base += per;
    }
    sItems = items;
  }
  // a thread's place in its group, and a stage of 32 records a warp. The second group starts on the third
  // scheduler, so that up to 64 entries a colour keep the groups apart
  const int grp = tid / kFlowGroup, gt = (tid + grp * (kFlowGroup / 2)) % kFlowGroup, gw = gt & ~31;
  const unsigned stage = flowShared(flowSmem) + (unsigned)(warp * 32 * F::kStride);
  const unsigned char* mine = flowSmem + tid * F::kStride;  // this thread's record
  const unsigned box = flowShared(flowSmem) + F::kStageBytes;  // CLUSTER: [packet][side][slot]
  if (CLUSTER) {
    uint4* z = reinterpret_cast<uint4*>(flowSmem + F::kStageBytes);
    for (int k = tid; k < 2 * NP * stride; k += kFlowBlock)
      z[k] = make_uint4(0u, 0u, 0u, 0u);
    cg::this_cluster().sync();
  } else {
    __syncthreads();
  }
  const int items = sItems;
  const unsigned tag0 = CLUSTER ? 0u : rec.tag0;
  bool dead = false, lost = false;  // a wait timed out; a record did not arrive
  unsigned parity = 0u;

  // the warp's records of an item into its stage (lane 0), and this thread's impulses
  bool pending = false;
  Q4<R> var{};    // KIND 0: the next entry's tangential and normal impulses
  R plam = R(0);  // KIND 2: its position impulse
  auto fetch = [&](const int3& item, bool impulses) {
    const int n = min(32, item.y - gw);
    pending = n > 0;
    if (lane == 0 && pending)
      flowBulk(stage, rec.rec + (long)(item.x + gw) * F::kStride, (unsigned)(n * F::kStride), bar);
    if (impulses && gt < item.y) {
      if (KIND == 0)
        var = rec.var[item.x + gt];
      else
        plam = rec.lam[item.x + gt];
    }
  };
  // wait for this warp's copy; one that is late stays outstanding: the warp takes no more records, and waits
  // for it once more at the end. (The limit is the constant: GridBar::spins here costs 2 % of the settled
  // 4,096-sphere step, 13.54 -> 13.82 ms per ten substeps.)
  auto landed = [&] {
    long spins = 0;
    bool late = false;
    while (!late && !flowBulkDone(bar, parity))
      late = ++spins > kBarrierSpins;
    if (late) {
      atomicOr(gb.err, kErrBarrier);
      dead = true;
    }
    lost = __any_sync(0xffffffffu, late);
    if (!lost) {
      parity ^= 1u;
      pending = false;
    }
  };
  auto slot = [&](int k) {  // slot k of this thread's staged record
    Q4<R> v;
    if constexpr (sizeof(R) == 8) {
      const double2 a = *reinterpret_cast<const double2*>(mine + 32 * k);
      const double2 b = *reinterpret_cast<const double2*>(mine + 32 * k + 16);
      v = Q4<R>{a.x, a.y, b.x, b.y};
    } else {
      const float4 a = *reinterpret_cast<const float4*>(mine + 16 * k);
      v = Q4<R>{a.x, a.y, a.z, a.w};
    }
    return v;
  };
  // wait for the states with this tag in the mailboxes of (slot or entry) at: side A into a if wa, side
  // B into b if wb
  auto receive = [&](long at, bool wa, bool wb, unsigned tag, R* a, R* b) {
    uint4 m[2][NP];
    long spins = 0;
    for (;;) {
      bool ok = true;
#pragma unroll
      for (int side = 0; side < 2; ++side)
        if (side ? wb : wa) {
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            m[side][p] = CLUSTER ? flowLoadShared(box + (unsigned)((p * 2 + side) * stride + (int)at) * 16u)
                                 : flowLoadGlobal(rec.box + (long)(p * 2 + side) * rec.cap + at);
            ok = ok && m[side][p].w == tag;
          }
        }
      if (ok || dead)
        break;
      if (++spins > gb.spins) {
        atomicOr(gb.err, kErrBarrier);
        dead = true;
      }
    }
#pragma unroll
    for (int side = 0; side < 2; ++side)
      if (side ? wb : wa) {
        unsigned w[3 * NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          w[3 * p] = m[side][p].x;
          w[3 * p + 1] = m[side][p].y;
          w[3 * p + 2] = m[side][p].z;
        }
        flowValues(w, NV, side ? b : a);
      }
  };
  // address of the first packet of a link's mailbox, and the state into it
  auto target = [&](int code) -> unsigned long long {
    const int side = code & 1, to = code >> 2;
    if (CLUSTER)
      return flowRemoteAddr(box + (unsigned)(side * stride + (to & 0x3fff)) * 16u, to >> 14);
    return reinterpret_cast<unsigned long long>(rec.box + (long)side * rec.cap + to);
  };
  auto send = [&](unsigned long long to, unsigned tag, const R* v) {
    unsigned w[3 * NP];
#pragma unroll
    for (int k = 0; k < 3 * NP; ++k)
      w[k] = 0u;
    flowWords(v, NV, w);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      if (CLUSTER)
        flowStoreRemote((unsigned)to + (unsigned)(p * 2 * stride) * 16u, w[3 * p], w[3 * p + 1], w[3 * p + 2], tag);
      else
        flowStoreGlobal(reinterpret_cast<uint4*>(to) + (long)(p * 2) * rec.cap, w[3 * p], w[3 * p + 1], w[3 * p + 2], tag);
    }
  };
  auto warpMax = [&](unsigned long long m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long w = __shfl_xor_sync(0xffffffffu, m, o);
      m = w > m ? w : m;
    }
    return m;
  };
  // the sweep's maximum of this warp (block), handed to the launch
  auto arrive = [&](int it, R mx) {
    unsigned long long m = warpMax(flowBits(mx));
    if (CLUSTER) {  // to every block; a slot is written again two sweeps later, after every warp has read it
      if (lane < nb)
        flowStoreRemote(flowRemoteAddr(flowShared(&sPost[it & 1][blk * kWarps + warp]), lane), (unsigned)m,
                        (unsigned)(m >> 32), 0u, (unsigned)it + 1u);
    } else {
      if (lane == 0)
        sWarp[warp] = m;
      __syncthreads();
      if (tid == 0) {
        for (int k = 1; k < kWarps; ++k)
          m = sWarp[k] > m ? sWarp[k] : m;
        if (m > 0ull)
          atomicMax(reinterpret_cast<unsigned long long*>(rec.ctl + 2 + 2 * (it % 3)), m);
        __threadfence();
        atomicAdd(rec.ctl, 1u);
      }
    }
  };
  // every warp (block) has arrived: the sweep's maximum
  auto decide = [&](int it) -> R {
    unsigned long long m = 0ull;
    long spins = 0;
    if (CLUSTER) {
      for (int k = lane; k < nb * kWarps; k += 32) {
        uint4 w;
        for (;;) {
          w = flowLoadShared(flowShared(&sPost[it & 1][k]));
          if (w.w == (unsigned)it + 1u || dead)
            break;
          if (++spins > gb.spins) {
            atomicOr(gb.err, kErrBarrier);
            dead = true;
          }
        }
        const unsigned long long u = ((unsigned long long)w.y << 32) | w.x;
        m = u > m ? u : m;
      }
      __syncwarp();
      m = warpMax(m);
    } else {
      if (lane == 0) {
        volatile unsigned* a = rec.ctl;
        const unsigned want = (unsigned)(it + 1) * (unsigned)nb;
        while (!dead && *a < want)
          if (++spins > gb.spins) {
            atomicOr(gb.err, kErrBarrier);
            dead = true;
          }
        __threadfence();
        m = *reinterpret_cast<volatile unsigned long long*>(rec.ctl + 2 + 2 * (it % 3));
        // free since every block has arrived, so has read the sweep before's
        if (tid == 0 && blk == 0)
          *reinterpret_cast<volatile unsigned long long*>(rec.ctl + 2 + 2 * ((it + 2) % 3)) = 0ull;
      }
      m = __shfl_sync(0xffffffffu, m, 0);
    }
    return flowFromBits(m, R(0));
  };

  const bool same = items <= grp + kFlowGroups;  // the group's next entries are these again: their impulses
                                                 // are known only after the update
  if (grp < items)
    fetch(sItem[grp], true);
  int it = 0;
  R last = R(0);
  bool stop = false;
  for (; it < iters; ++it) {
    R mx = R(0);
    bool decided = it == 0;
    for (int j = grp; j < items; j += kFlowGroups) {
      const int3 item = sItem[j];
      const int3 nitem = sItem[j + kFlowGroups < items ? j + kFlowGroups : grp];
      const bool more = j + kFlowGroups < items || it + 1 < iters;
      if (gw >= item.y) {  // nothing for this warp: only the next item's records
        if (more && !lost)
          fetch(nitem, true);
        continue;
      }
      const long t = item.x + gt;
      if (!lost)
        landed();
      const bool act = gt < item.y && !lost;  // without its record an entry is left out
      // the previous sweep's stop, before anything of this one is stored: for entries of the first colour,
      // whose states come from that sweep, after their update (below); for others before they wait for
      // this sweep's states, which do not come after a stop
      if (!decided && item.x >= sOff[1]) {
        decided = true;
        last = decide(it - 1);
        stop = KIND == 2 ? (last < thr) : (last <= thr);
        if (stop)
          break;
      }
      int4 id = make_int4(0, 0, 0, 0);
      int2 lk = make_int2(0, 0);
      if (act) {
        id = *reinterpret_cast<const int4*>(mine + F::kIds);
        lk = *reinterpret_cast<const int2*>(mine + F::kIds + 16);
      }
      Q4<R> cur = var;
      const bool hasB = (id.w & kFlowHasB) != 0, self = (id.w & kFlowSelf) != 0;
      const bool sideB = hasB && !self;
      R a[NV], b[NV];
      unsigned long long toA = 0ull, toB = 0ull;
      const unsigned tag = tag0 + (unsigned)it + 1u;
      int changed = 0;
      R dl = R(0);
      FlowPgs<R> f;
      PgsStatic<R> s;
      if (act) {
        if constexpr (KIND == 0) {
          s.ra = id.y, s.rb = id.z, s.hasB = hasB;
          s.Nsq = R(0);  // not read by the update
          const Q4<R> q0 = slot(0), q1 = slot(1), q2 = slot(2), q3 = slot(3);
          s.N = v3(q0), s.lenN = q0.w, s.TA = v3(q1), s.TB = v3(q2), s.wAn0 = q2.w, s.dc = v3(q3), s.wBn0 = q3.w;
          s.imA = slot(4).w, s.imB = slot(5).w, s.eAvg = slot(6).w, s.muAvg = slot(7).w;
          f = flowPgsBegin<R>(s, LOOP == 2 ? (id.w >> kFlowSideShift) : 0, q1.w, slot(8).w, P.eN, P.mu, P);
          flowPin(f.nh.x), flowPin(f.nh.y), flowPin(f.nh.z), flowPin(f.rW.y), flowPin(f.target), flowPin(f.vgn);
        }
        toA = target(lk.x), toB = target(lk.y);
        asm volatile("" : "+l"(toA), "+l"(toB));
        auto initial = [&](int body, R* v) {
          if (KIND == 0) {
            const Q4<R> lv = d.velPred[body], lw = d.angVelPred[body];
            v[0] = lv.x, v[1] = lv.y, v[2] = lv.z;
            v[NV - 3] = lw.x, v[NV - 2] = lw.y, v[NV - 1] = lw.z;
          } else {
            const Q4<R> lp = d.posPred[body];
            v[0] = lp.x, v[1] = lp.y, v[2] = lp.z;
          }
        };
#pragma unroll
        for (int k = 0; k < NV; ++k)
          a[k] = b[k] = R(0);
        const bool firstA = it == 0 && (id.w & kFlowFirstA), firstB = it == 0 && (id.w & kFlowFirstB);
        if (firstA)
          initial(id.y, a);
        if (sideB && firstB)
          initial(id.z, b);
        receive(CLUSTER ? (long)(item.z + gt) : t, !firstA, sideB && !firstB, tag, a, b);
        if (self) {  // a body and its own image
#pragma unroll
          for (int k = 0; k < NV; ++k)
            b[k] = a[k];
        }
      }
      __syncwarp();
      // the update, in registers
      if (act) {
        if constexpr (KIND == 0) {
          s.rAa = v3(slot(4)), s.rBa = v3(slot(5)), s.wvN = v3(slot(6)), s.iIA = v3(slot(7)), s.iIB = v3(slot(8));
          s.qA = slot(9), s.qB = slot(10);
          PgsVars<R> x;
          x.v0 = V3<R>{a[0], a[1], a[2]}, x.w0 = V3<R>{a[NV - 3], a[NV - 2], a[NV - 1]};
          x.v1 = V3<R>{b[0], b[1], b[2]}, x.w1 = V3<R>{b[NV - 3], b[NV - 2], b[NV - 1]};
          x.lt = v3(cur), x.lam = cur.w;
          changed = flowPgsStates<R>(s, f, [&] { return v3(d.vt0[id.x]); }, x);
          a[0] = x.v0.x, a[1] = x.v0.y, a[2] = x.v0.z, a[NV - 3] = x.w0.x, a[NV - 2] = x.w0.y, a[NV - 1] = x.w0.z;
          b[0] = x.v1.x, b[1] = x.v1.y, b[2] = x.v1.z, b[NV - 3] = x.w1.x, b[NV - 2] = x.w1.y, b[NV - 1] = x.w1.z;
          cur = Q4<R>{x.lt.x, x.lt.y, x.lt.z, x.lam};
        } else {
          const Q4<R> q0 = slot(0), q1 = slot(1), q2 = slot(2);
          const V3<R> n = v3(q0), rA = v3(q1), rB = v3(q2);
          const R wT = q0.w, imA = q1.w, imB = q2.w;
          const V3<R> pA{a[0], a[1], a[2]}, pB{b[0], b[1], b[2]};
          const R C = hasB ? dot(sub(add(pA, rA), add(pB, rB)), n) : dot(sub(add(pA, rA), rB), n);
          if (!(C >= R(0)) && !(wT < R(1e-6))) {
            dl = -C / wT;
            changed = 1;
            a[0] = pA.x + n.x * dl * imA, a[1] = pA.y + n.y * dl * imA, a[2] = pA.z + n.z * dl * imA;
            if (hasB)
              b[0] = pB.x + -n.x * dl * imB, b[1] = pB.y + -n.y * dl * imB, b[2] = pB.z + -n.z * dl * imB;
            f.dA = -C;
          }
        }
      }
      if (!decided) {
        __syncwarp();
        last = decide(it - 1);
        decided = true;
        stop = KIND == 2 ? (last < thr) : (last <= thr);
        if (stop)
          break;
      }
      const bool wrapA = (lk.x & 2) != 0, wrapB = (lk.y & 2) != 0;
      const R* va = self ? b : a;
      if (act) {
        if (!wrapA || it + 1 < iters)
          send(toA, tag + (wrapA ? 1u : 0u), va);
        if (sideB && (!wrapB || it + 1 < iters))
          send(toB, tag + (wrapB ? 1u : 0u), b);
      }
      const R pcur = plam;
      __syncwarp();  // every lane has left the stage
      if (more && !lost)
        fetch(nitem, !same);
      if (act) {
        auto final = [&](int body, const R* v) {  // the body's state after this sweep
          if (KIND == 0) {
            d.velPred[body] = Q4<R>{v[0], v[1], v[2], R(0)};
            d.angVelPred[body] = Q4<R>{v[NV - 3], v[NV - 2], v[NV - 1], R(0)};
          } else {
            d.posPred[body] = Q4<R>{v[0], v[1], v[2], R(0)};
          }
        };
        if (wrapA)
          final(id.y, va);
        if (sideB && wrapB)
          final(id.z, b);
        if constexpr (KIND == 0) {
          if (changed)
            rec.var[t] = cur;
          if (changed & 1)
            d.lambda[id.x] = cur.w;
          if (changed & 2)
            d.lambdaT[id.x] = Q4<R>{cur.x, cur.y, cur.z, R(0)};
          if (same)
            var = cur;
          flowPgsReport(f, mx);
        } else {
          const R nl = changed ? pcur + dl : pcur;
          if (changed) {
            rec.lam[t] = nl;
            d.posLamC[id.x] = nl;
            runMax(mx, f.dA);
          }
          if (same)
            plam = nl;
        }
      }
    }
    if (!decided) {  // a warp without entries
      last = decide(it - 1);
      stop = KIND == 2 ? (last < thr) : (last <= thr);
    }
    if (stop)
      break;
    arrive(it, mx);
  }
  const int sweeps = it;  // completed
  if (!stop) {
    last = decide(iters - 1);
    stop = KIND == 2 ? (last < thr) : (last <= thr);
  }
  // the copy of the item after the stop, or a late one: it must land before this block's memory goes
  if (pending)
    landed();
  if (CLUSTER)
    cg::this_cluster().sync();  // no block leaves while another may write to its shared memory
  if (blk == 0 && tid == 0) {
    *(KIND == 2 ? &c->maxOverlap : &c->maxApproach) = last;
    (LOOP == 1 ? c->velSweeps : LOOP == 2 ? c->stabSweeps : c->posSweeps) += sweeps - 1;
    if (stop)
      *done = 1;
  }
}

}  // namespace pdem
