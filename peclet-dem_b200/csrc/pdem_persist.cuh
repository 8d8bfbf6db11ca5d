// Persistent loops: the two colourings, the coloured Gauss-Seidel sweeps by colour and the support levels,
// each as ONE launch whose blocks are all resident (a cooperative grid, one thread-block cluster, or a block a
// scene) and step through phases, colours or sweeps together behind a barrier, where separate launches would
// need one each and a host read-back. The sweeps' work per colour and its order are those of the per-colour
// kernels (pdem_solve.cuh); most velocity and position loops run as a flow without colour barriers instead
// (pdem_flow.cuh).
#pragma once
#include "pdem_contact.cuh"
#include "pdem_solve.cuh"

namespace pdem {

constexpr int kErrBarrier = 2;  // Counters::err bit: a grid barrier timed out

// word[0] = arrivals, word[1] = generation; both zero before the launch; sleepNs = the back-off
// of a waiting block between polls of the generation; spins = the polls before a wait gives up
// (kBarrierSpins unless a test shortens it to make the wait run out)
struct GridBar {
  unsigned* word;
  int* err;
  unsigned sleepNs;
  long spins;
};

// Grid-wide barrier of a cooperative launch (all blocks co-resident). Thread 0 of each block
// arrives; the last arrival resets the counter and advances the generation; the others wait for
// the generation to move, bounded. Fences on both sides order every block's writes before the
// barrier with every block's reads after it. Returns false (and sets the error bit) on time-out;
// the caller then returns.
__device__ __forceinline__ bool gridBarrier(const GridBar& gb) {
  __shared__ int sOk;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* gen = gb.word + 1;
    const unsigned g = *gen;
    __threadfence();
    int ok = 1;
    if (atomicAdd(gb.word, 1u) == gridDim.x - 1) {
      atomicExch(gb.word, 0u);
      __threadfence();
      atomicAdd(gb.word + 1, 1u);
    } else {
      long spins = 0;
      while (*gen == g) {
        if (++spins > gb.spins) {
          atomicOr(gb.err, kErrBarrier);
          ok = 0;
          break;
        }
        if (gb.sleepNs)
          __nanosleep(gb.sleepNs);
      }
    }
    __threadfence();
    sOk = ok;
  }
  __syncthreads();
  return sOk != 0;
}

// ---------------------------------------------------------------------------------------------
// Coloured sweep loop. KIND 0: projected GS velocity sweep (pgsOne), 1: one-shot GS velocity
// sweep (gsOne), 2: position sweep (posGSOne). LOOP selects the control flags: 1 main velocity
// loop, 2 stabilization loop, 3 position loop. The host has already run the first sweep's BEGIN
// (kCtl): each END here is fused with the next sweep's BEGIN. CLUSTER: the launch is one thread-block
// cluster (a small graph), and the hardware cluster barrier (arrive with release, wait with acquire
// semantics at cluster scope) replaces the grid-wide one.
template <bool CLUSTER>
__device__ __forceinline__ bool loopBarrier(const GridBar& gb) {
  if (CLUSTER) {
    cg::this_cluster().sync();
    return true;
  }
  return gridBarrier(gb);
}
// The colour offsets (at most 63 colours) are read once into shared memory. KIND 3: KIND 0 from the
// per-substep records of kFlowPack (entry t of the order is record t; flowRecord is in pdem_flow.cuh).
template <class R>
__device__ __forceinline__ PgsStatic<R> flowRecord(const char* rec, long t, int& idx);
template <class R, int KIND, int LOOP, bool CLUSTER = false>
__global__ void __launch_bounds__(kBlock) kSweepLoop(Dev<R> d, const int* order, const int* coff, int ncol, int iters,
                                                     SolveP<R> P, R thr, GridBar gb, const char* rec) {
  __shared__ int sOff[kSaturatedColor + 2];
  Counters<R>* c = d.ctr;
  volatile int* done = LOOP == 1 ? &c->velDone : LOOP == 2 ? &c->stabDone : &c->posDone;
  int* sweeps = LOOP == 1 ? &c->velSweeps : LOOP == 2 ? &c->stabSweeps : &c->posSweeps;
  R* mxp = KIND == 2 ? &c->maxOverlap : &c->maxApproach;
  const bool lead = (blockIdx.x | threadIdx.x) == 0;
  const long gtid = (long)blockIdx.x * blockDim.x + threadIdx.x, gstride = (long)gridDim.x * blockDim.x;
  if (*done)
    return;
  for (int k = threadIdx.x; k <= ncol && k < kSaturatedColor + 2; k += blockDim.x)
    sOff[k] = coff[k];
  __syncthreads();
  for (int it = 0; it < iters; ++it) {
    R mx = R(0);
    for (int col = 0; col < ncol; ++col) {
      const int b = sOff[col], n = sOff[col + 1] - b;
      // colour 62 is where the 62-colour mask saturates: not an independent set, so one thread
      // runs it in manifold order, as the reference's serial sweep does
      const bool serial = col >= kSaturatedColor;
      if (!serial || lead)
        for (long t = serial ? 0 : gtid; t < n; t += serial ? 1 : gstride) {
          if (KIND == 0) {
            pgsOne(d, order[b + t], P, mx, LOOP);
          } else if (KIND == 1) {
            gsOne(d, order[b + t], P, mx);
          } else if (KIND == 3) {
            int idx;
            const PgsStatic<R> st = flowRecord<R>(rec, b + t, idx);
            pgsCore<R>(d, idx, st, P.eN, P.mu, 0, P, mx);
          } else {
            posGSOne(d, order[b + t], mx);
          }
        }
      if (col == ncol - 1)
        warpMaxAtomic(mxp, mx);
      if (!loopBarrier<CLUSTER>(gb))
        return;
    }
    // END of this sweep, then BEGIN of the next one
    if (d.scn) {  // batched form: every scene's own END/BEGIN; done when all scenes are
      if (blockIdx.x == 0) {
        int notDone = 0;
        for (int s = threadIdx.x; s < d.numScenes; s += blockDim.x) {
          SceneCtl<R>& q = d.scn[s];
          volatile int* dn = LOOP == 1 ? &q.velDone : LOOP == 2 ? &q.stabDone : &q.posDone;
          volatile R* m = KIND == 2 ? &q.maxOverlap : &q.maxApproach;
          if (!*dn) {
            const R mv = *m;
            if (KIND == 2 ? (mv < thr) : (mv <= thr)) {
              *dn = 1;
            } else if (it + 1 < iters) {
              *m = R(0);
              (LOOP == 1 ? q.velSweeps : LOOP == 2 ? q.stabSweeps : q.posSweeps) += 1;
            }
          }
          notDone |= !*dn;
        }
        notDone = __syncthreads_or(notDone);
        if (threadIdx.x == 0 && !notDone)
          *done = 1;
      }
    } else if (lead) {
      const R m = *reinterpret_cast<volatile R*>(mxp);
      const bool stop = KIND == 2 ? (m < thr) : (m <= thr);
      if (stop) {
        *done = 1;
      } else if (it + 1 < iters) {
        *reinterpret_cast<volatile R*>(mxp) = R(0);
        *sweeps += 1;
      }
    }
    if (!loopBarrier<CLUSTER>(gb))
      return;
    if (*done)
      break;
  }
}

// ---------------------------------------------------------------------------------------------
// Batched form: the same sweep loop with ONE BLOCK PER SCENE. A scene's colour classes are
// contiguous in the (scene, colour)-sorted order (off[s * 64 + c] .. off[s * 64 + c + 1]); its
// blocks-worth of threads sweeps them in colour order with block barriers, and the block ends its
// own loop at the scene's adaptive stop. No grid-wide barrier and no cooperative launch: scenes are
// independent. Block b runs scene sceneOrder[b] (largest scenes first, so none is left to the last
// wave). The host has run the first sweep's BEGIN for every scene (kCtlScenes).
constexpr int kSceneBlock = 128;      // default block of the per-scene sweep loops
constexpr int kSceneBlockMax = 512;   // largest block the launch shape autotuner tries

template <class R, int KIND, int LOOP>
__global__ void __launch_bounds__(kSceneBlockMax) kSweepScenes(Dev<R> d, const int* sceneOrder, const int* order,
                                                            const int* off, int iters, SolveP<R> P, R thr) {
  const int s = sceneOrder[blockIdx.x];
  SceneCtl<R>& q = d.scn[s];
  volatile int* done = LOOP == 1 ? &q.velDone : LOOP == 2 ? &q.stabDone : &q.posDone;
  volatile R* mxp = KIND == 2 ? &q.maxOverlap : &q.maxApproach;
  if (*done)
    return;
  const int* so = off + (long)s * 64;
  __shared__ R sMax[kSceneBlockMax / 32];
  for (int it = 0; it < iters; ++it) {
    R mx = R(0);  // this thread's running max of the sweep; the block reduces it at the END
    for (int col = 0; col < 63; ++col) {
      const int b = so[col], n = so[col + 1] - b;
      if (n == 0)
        continue;  // uniform over the block
      const bool serial = col >= kSaturatedColor;
      if (!serial || threadIdx.x == 0)
        for (int t = serial ? 0 : threadIdx.x; t < n; t += serial ? 1 : blockDim.x) {
          if (KIND == 0)
            pgsOne<R, true>(d, order[b + t], P, mx, LOOP);
          else if (KIND == 1)
            gsOne<R, true>(d, order[b + t], P, mx);
          else
            posGSOne<R, true>(d, order[b + t], mx);
        }
      __syncthreads();
    }
    // the sweep's max over the block (the scene): no atomics on the scene's one max word
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const R w = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = w > mx ? w : mx;
    }
    if ((threadIdx.x & 31) == 0)
      sMax[threadIdx.x >> 5] = mx;
    __syncthreads();
    // END of this sweep, then BEGIN of the next one (kCtlScenes' rule for this scene)
    if (threadIdx.x == 0) {
      R m = sMax[0];
      for (int k = 1; k < (int)(blockDim.x >> 5); ++k)
        m = sMax[k] > m ? sMax[k] : m;
      *mxp = m;  // BEGIN left it 0 and only this block writes it during the loop
      if (KIND == 2 ? (m < thr) : (m <= thr)) {
        *done = 1;
      } else if (it + 1 < iters) {
        *mxp = R(0);
        (LOOP == 1 ? q.velSweeps : LOOP == 2 ? q.stabSweeps : q.posSweeps) += 1;
      }
    }
    __syncthreads();
    if (*done)
      break;
  }
}

// ---------------------------------------------------------------------------------------------
// kGroundLevels on the whole grid, for graphs whose levels, times and edges do not fit one block's
// shared memory (about 5,600 spheres in a bed): the same relaxations of the levels L and times T, in
// global memory, the passes behind the grid barrier. A pass relaxes every edge kGroundInner times, so
// that support chains advance between barriers. The one warp that ran the exact serial sweeps of such
// graphs before needs 1.4 ms a substep on 20,011 spheres (61,000 manifolds); it remains for the graphs
// that do not reach the fixed point within the serial sweeps' count.
// ctl: [0..2] a pass changed something (pass % 3), [3] some body late; zero before the launch.
constexpr int kGroundInner = 4;
static __global__ void __launch_bounds__(kGroundBlock) kGroundLevelsGrid(int nm, int nb, int sweeps, const int4* edges,
                                                                        uint8_t* grounded, int* L, u64* T, int* ctl,
                                                                        GridBar gb) {
  volatile int* VL = L;
  volatile u64* VT = T;
  volatile int* VC = ctl;
  const long gtid = (long)blockIdx.x * blockDim.x + threadIdx.x, gstride = (long)gridDim.x * blockDim.x;
  const bool lead = gtid == 0;
  const u64 kInf = ~0ull, kStart = 1ull << 32;  // (sweep << 32) | (edge + 1); 1 << 32: final before sweep 1
  for (long i = gtid; i < nb; i += gstride)
    L[i] = grounded[i];
  if (!gridBarrier(gb))
    return;
  int pass = 0;
  // passes of relax(edge index, edge) -> changed, until one changes nothing; 1: done, 0: too many
  // passes, -1: a barrier timed out
  auto settle = [&](auto relax) -> int {
    for (int k = 0; k < kGroundPassCap; ++k, ++pass) {
      int ch = 0;
      for (int q = 0; q < kGroundInner; ++q)
        for (long e = gtid; e < nm; e += gstride)
          ch |= relax(e, edges[e]) ? 1 : 0;
      if (__syncthreads_or(ch) && threadIdx.x == 0)
        VC[pass % 3] = 1;
      if (!gridBarrier(gb))
        return -1;
      const int any = VC[pass % 3];
      if (lead)
        VC[(pass + 2) % 3] = 0;  // read by every block before it arrived here
      if (!any) {
        ++pass;
        return 1;
      }
    }
    return 0;
  };
  int ok = settle([&](long, const int4& g) {  // (a) F
    const int c = g.x == 1 ? 255 : (g.x == 2 ? VL[g.y] - 1 : 0);
    if (c > 0 && c > VL[g.z]) {
      atomicMax(&L[g.z], c);
      return true;
    }
    return false;
  });
  if (ok < 0)
    return;
  for (long i = gtid; i < nb; i += gstride)
    T[i] = VL[i] == (int)grounded[i] ? kStart : kInf;
  if (!gridBarrier(gb))
    return;
  if (ok > 0)
    ok = settle([&](long e, const int4& g) {  // (b) the sweep in which each body becomes final
      u64 te = kInf;
      if (g.x == 1 && VL[g.z] == 255) {
        te = kStart | (u64)(e + 1);
      } else if (g.x == 2 && VL[g.z] > 0 && VL[g.y] - 1 == VL[g.z]) {
        const u64 tu = VT[g.y];
        if (tu != kInf)
          te = (((e > (long)(tu & 0xffffffffull) - 1 ? tu >> 32 : (tu >> 32) + 1)) << 32) | (u64)(e + 1);
      }
      if (te < VT[g.z]) {
        atomicMin(&T[g.z], te);
        return true;
      }
      return false;
    });
  if (ok < 0)
    return;
  int late = !ok;
  for (long i = gtid; i < nb && !late; i += gstride)
    late = VT[i] == kInf || (VT[i] >> 32) > (u64)sweeps;
  if (__syncthreads_or(late) && threadIdx.x == 0)
    VC[3] = 1;
  if (!gridBarrier(gb))
    return;
  if (!VC[3]) {  // (c)
    for (long i = gtid; i < nb; i += gstride)
      grounded[i] = (uint8_t)VL[i];
  } else if (blockIdx.x == 0 && threadIdx.x < 32) {
    groundSweepsWarp(nm, 0, nb, sweeps, edges, grounded, L);
  }
}

// 128-bit single-copy atomic accesses
__device__ __forceinline__ void flowStoreGlobal(uint4* p, unsigned x, unsigned y, unsigned z, unsigned w) {
  asm volatile(
      "{\n .reg .b128 q;\n .reg .b64 lo, hi;\n mov.b64 lo, {%1, %2};\n mov.b64 hi, {%3, %4};\n mov.b128 q, {lo, hi};\n"
      " st.relaxed.gpu.global.b128 [%0], q;\n}" ::"l"(p), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ uint4 flowLoadGlobal(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n .reg .b128 q;\n .reg .b64 lo, hi;\n ld.relaxed.gpu.global.b128 q, [%4];\n mov.b128 {lo, hi}, q;\n"
      " mov.b64 {%0, %1}, lo;\n mov.b64 {%2, %3}, hi;\n}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}

constexpr int kColorBlock = 1024;  // one large block per SM: fewer arrivals per grid barrier

// ---------------------------------------------------------------------------------------------
// Both colourings of a substep in ONE launch: the manifold graph (velocity solve) and the contact graph
// (position solve), each the reference's Jones-Plassmann rounds: in a round every uncoloured entry whose
// key is the largest at both ends takes the lowest colour free at both.
//
// An entry's colour and round depend only on the entries before it (larger key) at its two ends: with
// each body's entries sorted by key and a body holding its first uncoloured one, an entry that is first at
// both ends is coloured and both bodies move on. A round of the former loop cost two barriers and 64-bit
// atomics on every remaining entry (8 to 13 us a round).
//
// Graphs of one cluster whose bodies fit a block's shared memory: one block a graph runs the rounds there,
// two block barriers each (about 0.3 us a round). Larger ones: no rounds at all, every thread visits its
// bodies and colours what is ready. The round of an entry is then one above the later of its
// predecessors' rounds; entries beyond the round limit stay uncoloured, as in the rounds. A body's state is
// one 128-bit word (first uncoloured entry + 1, its place in the lists, the body's colour mask) and a
// 64-bit word (last round, the same place): each single-copy atomic, and taken together only when the
// places agree, so no fences are needed. Only the thread that colours an entry writes its two bodies'
// states.
struct ColorJob {
  int ne, nb;          // entries, bodies
  int* col;            // [ne] colours out
  u64* mask;           // [nb] colours of each body's entries out
  int* aux;            // [0] list space taken, [1] items of long lists, [2] largest round, [3] max colour,
                       // [4] left uncoloured, [5] rounds run
  int *cnt, *at;       // [nb] entries of each body, their place in the lists
  int4* list;          // [2 ne + nb] (key low, key high, entry, other body << 1 | 1 at its first end) unsorted
  int2* sorted;        // [2 ne + nb] (entry, other body (or -1) << 1 | 1 at its first end), then (-1, 0)
  uint4* state;        // [nb]
  u64* round;          // [nb]
  int2* item;          // [ne / 4 + 2] (body, first entry) of each 32 entries of a long list
  // stable order by colour, built in the same launch when order is set: order[ne] (entry indices,
  // colour-major, index order within a colour), off[65] (first position of each colour key, then
  // ne), hist[64 * gridDim] (scratch)
  int *order = nullptr, *off = nullptr, *hist = nullptr;
};
constexpr size_t kColorMaxSmem = 200 * 1024;  // bodies of a graph in one block
constexpr int kColorMaxChunks = 20;  // histogram row chunks of 32 blocks (grids up to 640 blocks)

template <class R, bool MANIFOLD>
__device__ __forceinline__ void colorInit(const Dev<R>& d, const ColorJob& J, long gtid, long gstride) {
  if (J.ne <= 0)
    return;  // a kept (or empty) graph: its colours and statistics stay as they are
  for (long b = gtid; b < J.nb; b += gstride)
    J.cnt[b] = 0;
  for (long i = gtid; i < J.ne; i += gstride) {
    if (MANIFOLD) {
      const int2 ab = d.mab[i];
      J.col[i] = (d.mnp[i] <= 0 || (ab.y >= 0 && d.realIdx[ab.x] > d.realIdx[ab.y])) ? -2 : -1;
    } else {
      J.col[i] = -1;
    }
  }
  if (gtid == 0) {
    J.aux[0] = J.aux[1] = J.aux[2] = 0;
    J.aux[3] = INT_MIN;
    J.aux[4] = 0;
  }
}
// an entry's ends; an entry of one body (a wall's, or a body and its own image) has no second
template <class R, bool MANIFOLD>
__device__ __forceinline__ void colorTwoEnds(const Dev<R>& d, int i, int& ea, int& eb) {
  colorEnds<R, MANIFOLD>(d, i, ea, eb);
  if (eb == ea)
    eb = -1;
}
template <class R, bool MANIFOLD>
__device__ __forceinline__ void colorCount(const Dev<R>& d, const ColorJob& J, long gtid, long gstride) {
  for (long i = gtid; i < J.ne; i += gstride)
    if (J.col[i] == -1) {
      int ea, eb;
      colorTwoEnds<R, MANIFOLD>(d, (int)i, ea, eb);
      atomicAdd(&J.cnt[ea], 1);
      if (eb >= 0)
        atomicAdd(&J.cnt[eb], 1);
    }
}
// room in the lists for every body, in any order, and the items of the long ones
constexpr int kColorLanes = 8, kColorShort = 16;
__device__ __forceinline__ void colorRoom(const ColorJob& J, long gtid, long gstride) {
  if (J.ne <= 0)
    return;
  const int lane = threadIdx.x & 31;
  for (long b0 = gtid - lane; b0 < J.nb; b0 += gstride) {
    const long b = b0 + lane;
    const int n = b < J.nb ? __ldcg(&J.cnt[b]) : 0;
    const int want = b < J.nb ? n + 1 : 0;  // and the end mark
    int x = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o)
        x += y;
    }
    int base = 0;
    if (lane == 31)
      base = atomicAdd(&J.aux[0], x);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (b < J.nb) {
      J.at[b] = base + x - want;
      J.cnt[b] = 0;  // now the entries filled in
      if (n > kColorShort) {
        int it = atomicAdd(&J.aux[1], (n + 31) / 32);
        for (int k = 0; k < n; k += 32)
          J.item[it++] = make_int2((int)b, k);
      }
    }
  }
}
template <class R, bool MANIFOLD>
__device__ __forceinline__ void colorFill(const Dev<R>& d, const ColorJob& J, long gtid, long gstride) {
  for (long i = gtid; i < J.ne; i += gstride)
    if (J.col[i] == -1) {
      int ea, eb;
      colorTwoEnds<R, MANIFOLD>(d, (int)i, ea, eb);
      const long long k = entryKey<R, MANIFOLD>(d, (int)i, ea);
      const int lo = (int)(k & 0xffffffffll), hi = (int)(k >> 32);
      const int pa = __ldcg(&J.at[ea]) + atomicAdd(&J.cnt[ea], 1);
      J.list[pa] = make_int4(lo, hi, (int)i, (eb << 1) | 1);
      if (eb >= 0) {
        const int pb = __ldcg(&J.at[eb]) + atomicAdd(&J.cnt[eb], 1);
        J.list[pb] = make_int4(lo, hi, (int)i, ea << 1);
      }
    }
}
// each body's list by decreasing key: an element's place is the number of larger keys. Eight lanes a body up
// to kColorShort entries; longer lists by items of 32 entries, a warp each, with the list's keys passed round
// by shuffles. The colouring stage of one grain with 3,000, 10,000 and 30,000 contacts: 4.8, 12.9 and 16.8 ms
// (26.8, 98 and 181 by rounds of contention; 69, 550 and 830 with eight lanes a body at any length); of 216
// cylinders 0.23 (0.44).
__device__ __forceinline__ void colorSort(const ColorJob& J, long gtid, long gstride) {
  if (J.ne <= 0)
    return;
  auto keyOf = [](const int4& e) { return ((u64)(unsigned)e.y << 32) | (unsigned)e.x; };
  auto put = [&](long b, int at, const int4& e, int rank) {
    J.sorted[at + rank] = make_int2(e.z, e.w);
    if (rank == 0)
      flowStoreGlobal(&J.state[b], (unsigned)e.z + 1u, (unsigned)at, 0u, 0u);
  };
  const int lane = threadIdx.x & 31, items = __ldcg(&J.aux[1]);
  for (long it = gtid >> 5; it < items; it += gstride >> 5) {
    const int2 item = __ldcg(&J.item[it]);
    const int n = __ldcg(&J.cnt[item.x]), at = __ldcg(&J.at[item.x]), k = item.y + lane;
    const int4 e = k < n ? __ldcg(&J.list[at + k]) : make_int4(0, 0, 0, 0);
    const u64 key = keyOf(e);
    int rank = 0;
    for (int q0 = 0; q0 < n; q0 += 32) {
      const u64 f = q0 + lane < n ? keyOf(__ldcg(&J.list[at + q0 + lane])) : 0ull;  // 0 is larger than no key
#pragma unroll
      for (int j = 0; j < 32; ++j)
        rank += __shfl_sync(0xffffffffu, f, j) > key ? 1 : 0;
    }
    if (k < n)
      put(item.x, at, e, rank);
  }
  const int sub = threadIdx.x % kColorLanes;
  for (long b = gtid / kColorLanes; b < J.nb; b += gstride / kColorLanes) {
    const int n = __ldcg(&J.cnt[b]), at = __ldcg(&J.at[b]);
    for (int k = sub; k < n && n <= kColorShort; k += kColorLanes) {
      const int4 e = __ldcg(&J.list[at + k]);
      const u64 key = keyOf(e);
      int rank = 0;
      for (int q = 0; q < n; ++q)
        rank += keyOf(__ldcg(&J.list[at + q])) > key ? 1 : 0;
      put(b, at, e, rank);
    }
    if (sub == 0) {
      J.sorted[at + n] = make_int2(-1, 0);
      J.round[b] = (u64)(unsigned)at;
      if (n == 0)
        flowStoreGlobal(&J.state[b], 0u, (unsigned)at, 0u, 0u);
    }
  }
}
// one visit of body b: colours its first entry if that is first at the other end too. Returns whether the
// body has entries left.
__device__ __forceinline__ bool colorVisit(const ColorJob& J, long b, int maxRounds, int& maxRound) {
  for (;;) {
    const uint4 s = flowLoadGlobal(&J.state[b]);
    if (s.x == 0u) {
      J.mask[b] = ((u64)s.w << 32) | s.z;
      return false;
    }
    const int2 el = __ldcg(&J.sorted[s.y]);
    if (!(el.y & 1))
      return true;  // its first end's thread colours it
    const int o = el.y >> 1;
    const volatile u64* vr = J.round;
    const u64 ra = vr[b];
    if ((unsigned)ra != s.y)
      return true;
    uint4 t = make_uint4(0u, 0u, 0u, 0u);
    u64 rb = 0ull;
    if (o >= 0) {
      t = flowLoadGlobal(&J.state[o]);
      rb = vr[o];
      if (t.x != s.x || (unsigned)rb != t.y)
        return true;
    }
    const u64 ma = ((u64)s.w << 32) | s.z, mb = ((u64)t.w << 32) | t.z;
    const int r = 1 + max((int)(ra >> 32), (int)(rb >> 32));
    u64 bit = 0ull;
    if (r <= maxRounds) {
      const u64 open = ~(ma | mb) & ((1ull << 62) - 1ull);
      const int cc = open ? __ffsll((long long)open) - 1 : 62;
      J.col[s.x - 1u] = cc;
      bit = 1ull << cc;
      maxRound = max(maxRound, r);
    }
    auto advance = [&](long body, unsigned place, u64 m) {
      const unsigned next = (unsigned)(__ldcg(&J.sorted[place + 1u]).x + 1);
      *reinterpret_cast<volatile u64*>(&J.round[body]) = ((u64)(unsigned)r << 32) | (place + 1u);
      flowStoreGlobal(&J.state[body], next, place + 1u, (unsigned)m, (unsigned)(m >> 32));
    };
    advance(b, s.y, ma | bit);
    if (o >= 0)
      advance(o, t.y, mb | bit);
  }
}
// the rounds of one graph in one block, its bodies in shared memory
struct ColorBody {
  u64 mask;
  int entry, other;  // first uncoloured entry (-1: none), its other body << 1 | 1 at its first end
  int2 next;         // the one after it
  int place, moved;  // place of `next` in the lists; the entry was coloured this round
};
__device__ __forceinline__ void colorRounds(const ColorJob& J, int maxRounds, ColorBody* B) {
  for (int b = threadIdx.x; b < J.nb; b += blockDim.x) {
    const int at = __ldcg(&J.at[b]);
    const int2 el = __ldcg(&J.sorted[at]);
    ColorBody c;
    c.mask = 0ull;
    c.entry = el.x;
    c.other = el.y;
    c.next = el.x >= 0 ? __ldcg(&J.sorted[at + 1]) : make_int2(-1, 0);
    c.place = at + 1;
    c.moved = 0;
    B[b] = c;
  }
  __syncthreads();
  int round = 0;
  for (; round < maxRounds; ++round) {
    int left = 0;
    for (int b = threadIdx.x; b < J.nb; b += blockDim.x) {
      const int e = B[b].entry;
      if (e < 0)
        continue;
      left = 1;
      const int ot = B[b].other, o = ot >> 1;
      if (!(ot & 1) || (o >= 0 && B[o].entry != e))
        continue;
      const u64 ma = B[b].mask, mb = o >= 0 ? B[o].mask : 0ull;
      const u64 open = ~(ma | mb) & ((1ull << 62) - 1ull);
      const int cc = open ? __ffsll((long long)open) - 1 : 62;
      J.col[e] = cc;
      B[b].mask = ma | 1ull << cc;
      B[b].moved = 1;
      if (o >= 0) {
        B[o].mask = mb | 1ull << cc;
        B[o].moved = 1;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // this thread's bodies' next entries
    if (!__syncthreads_or(left))
      break;
    for (int b = threadIdx.x; b < J.nb; b += blockDim.x)
      if (B[b].moved) {
        const int2 n = B[b].next;
        B[b].entry = n.x;
        B[b].other = n.y;
        B[b].moved = 0;
        if (n.x >= 0) {  // the end mark is the last
          B[b].place += 1;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(&B[b].next)),
                       "l"(J.sorted + B[b].place)
                       : "memory");
        }
      }
    __syncthreads();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  for (int b = threadIdx.x; b < J.nb; b += blockDim.x)
    J.mask[b] = B[b].mask;
  if (threadIdx.x == 0)
    J.aux[2] = round;
}
// all entries, in any order the states allow; false on time-out
__device__ __forceinline__ bool colorRun(const ColorJob& jm, const ColorJob& jc, int maxRounds, const GridBar& gb, long gtid,
                                         long gstride) {
  int mr[2] = {0, 0};
  long spins = 0;
  bool late = false;
  u64 open[2] = {~0ull, ~0ull};  // of the thread's first 64 bodies of a graph: those with entries left
  for (bool more = true; more && !late;) {
    more = false;
    for (int g = 0; g < 2; ++g) {
      const ColorJob& J = g ? jc : jm;
      if (J.ne <= 0)
        continue;
      int k = 0;
      for (long b = gtid; b < J.nb; b += gstride, ++k) {
        if (k < 64 && !(open[g] >> k & 1ull))
          continue;
        if (colorVisit(J, b, maxRounds, mr[g]))
          more = true;
        else if (k < 64)
          open[g] &= ~(1ull << k);
      }
    }
    late = ++spins > gb.spins;
  }
  if (late)
    atomicOr(gb.err, kErrBarrier);
  const int m = __reduce_max_sync(__activemask(), max(mr[0], mr[1]));
  if (m > 0 && (mr[0] == m || mr[1] == m)) {
    if (jm.ne > 0)
      atomicMax(&jm.aux[2], m);
    if (jc.ne > 0)
      atomicMax(&jc.aux[2], m);
  }
  return !late;
}
// ---- stable order by colour (counting sort over 64 keys: colours 0..62, 63 for uncoloured, the
// order of the reference's stable sort by colour). Block b owns the contiguous chunk
// [b * chunk, (b + 1) * chunk) of the entries; the colour-major histogram H[key * gridDim + b]
// scanned exclusively gives each (key, block) its first position. Colours are read through L2
// (__ldcg): other SMs wrote them in this launch.
__device__ __forceinline__ int colorSortKey(int c) { return c >= 0 ? c : 63; }
__device__ __forceinline__ void colorChunk(const ColorJob& J, long& b0, long& b1) {
  const long chunk = ((long)J.ne + gridDim.x - 1) / gridDim.x;
  b0 = min((long)J.ne, (long)blockIdx.x * chunk);
  b1 = min((long)J.ne, b0 + chunk);
}
__device__ __forceinline__ void colorOrderCount(const ColorJob& J) {
  __shared__ int h[64];
  if (!J.order || J.ne <= 0)
    return;  // uniform over the grid
  long b0, b1;
  colorChunk(J, b0, b1);
  __syncthreads();
  if (threadIdx.x < 64)
    h[threadIdx.x] = 0;
  __syncthreads();
  for (long i = b0 + threadIdx.x; i < b1; i += blockDim.x)
    atomicAdd(&h[colorSortKey(__ldcg(&J.col[i]))], 1);
  __syncthreads();
  if (threadIdx.x < 64)
    J.hist[(long)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}
// one block: exclusive scan of the colour-major histogram in place, and the colour offsets. Each
// warp scans whole rows (colours) with shuffles over coalesced loads, then one warp scans the 64
// row totals, and each row gets its offset.
__device__ __forceinline__ void colorOrderScan(const ColorJob& J) {
  __shared__ int rowTot[64], rowOff[64];
  if (!J.order || J.ne <= 0)
    return;
  const int G = gridDim.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();  // rowTot / rowOff free (a previous call's reads are done)
  for (int c = w; c < 64; c += nw) {
    int* row = J.hist + (long)c * G;
    int run = 0;
    int vals[kColorMaxChunks];  // the row's loads, issued together (G <= 32 * kColorMaxChunks)
#pragma unroll
    for (int k = 0; k < kColorMaxChunks; ++k)
      vals[k] = (32 * k + lane < G) ? __ldcg(&row[32 * k + lane]) : 0;
#pragma unroll
    for (int k = 0; k < kColorMaxChunks; ++k) {
      const int b0 = 32 * k;
      if (b0 >= G)
        break;
      const int b = b0 + lane;
      const int v = vals[k];
      int x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
          x += y;
      }
      if (b < G)
        row[b] = run + x - v;
      run += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0)
      rowTot[c] = run;
  }
  __syncthreads();
  if (w == 0) {
    const int a = rowTot[lane], b = rowTot[lane + 32];
    int xa = a, xb = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ya = __shfl_up_sync(0xffffffffu, xa, o), yb = __shfl_up_sync(0xffffffffu, xb, o);
      if (lane >= o) {
        xa += ya;
        xb += yb;
      }
    }
    const int totA = __shfl_sync(0xffffffffu, xa, 31);
    rowOff[lane] = xa - a;
    rowOff[lane + 32] = totA + xb - b;
  }
  __syncthreads();
  for (int c = w; c < 64; c += nw) {  // the same thread wrote these entries above
    int* row = J.hist + (long)c * G;
    for (int b = lane; b < G; b += 32)
      row[b] += rowOff[c];
  }
  if (threadIdx.x < 64)
    J.off[threadIdx.x] = rowOff[threadIdx.x];
  if (threadIdx.x == 0)
    J.off[64] = J.ne;
}
// every block: its chunk in tiles of blockDim entries; within a tile, the rank among equal keys is
// the lanes below in the warp with that key plus the earlier warps' counts of it
__device__ __forceinline__ void colorOrderScatter(const ColorJob& J) {
  __shared__ int run[64];
  __shared__ int cnt[kColorBlock / 32][64];
  if (!J.order || J.ne <= 0)
    return;
  long b0, b1;
  colorChunk(J, b0, b1);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (threadIdx.x < 64)
    run[threadIdx.x] = __ldcg(&J.hist[(long)threadIdx.x * gridDim.x + blockIdx.x]);
  for (long t0 = b0; t0 < b1; t0 += blockDim.x) {
    for (int k = threadIdx.x; k < nw * 64; k += blockDim.x)
      (&cnt[0][0])[k] = 0;
    __syncthreads();
    const long i = t0 + threadIdx.x;
    const int key = i < b1 ? colorSortKey(__ldcg(&J.col[i])) : 64;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int below = __popc(peers & ((1u << lane) - 1u));
    if (key < 64 && below == 0)
      cnt[w][key] = __popc(peers);
    __syncthreads();
    if (key < 64) {
      int pos = run[key] + below;
      for (int v = 0; v < w; ++v)
        pos += cnt[v][key];
      J.order[pos] = (int)i;
    }
    __syncthreads();
    if (threadIdx.x < 64) {
      int tot = 0;
      for (int v = 0; v < nw; ++v)
        tot += cnt[v][threadIdx.x];
      run[threadIdx.x] += tot;
    }
    __syncthreads();
  }
}
__device__ __forceinline__ void colorStats(const ColorJob& J, long gtid, long gstride) {
  int mxc = INT_MIN, left = 0;
  for (long i = gtid; i < J.ne; i += gstride) {
    const int v = __ldcg(&J.col[i]);
    mxc = v > mxc ? v : mxc;
    left += (v == -1) ? 1 : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int w = __shfl_xor_sync(0xffffffffu, mxc, o);
    mxc = w > mxc ? w : mxc;
    left += __shfl_xor_sync(0xffffffffu, left, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (mxc != INT_MIN)
      atomicMax(&J.aux[3], mxc);
    if (left)
      atomicAdd(&J.aux[4], left);
  }
}

// job 0: manifolds over real bodies (skipped when ne = 0), job 1: contacts over body slots.
// CLUSTER: the launch is one thread-block cluster (graphs of a few tens of thousands of entries)
// and the hardware cluster barrier replaces the grid-wide one, as in kSweepLoop.
// reuse: a graph equal to the previous substep's keeps its colours and statistics (differ[0]: the
// contact list changed, differ[1]: the manifold list changed; reuse = 0 forces both colourings)
template <class R, bool CLUSTER = false>
__global__ void __launch_bounds__(kColorBlock) kColorBoth(Dev<R> d, ColorJob jm, ColorJob jc, int maxRounds,
                                                          GridBar gb, const int* differ, int reuse, int inShared) {
  const long gtid = (long)blockIdx.x * blockDim.x + threadIdx.x, gstride = (long)gridDim.x * blockDim.x;
  if (reuse && !differ[1])
    jm.ne = 0;  // uniform over the grid: the flags are written before the launch
  if (reuse && !differ[0])
    jc.ne = 0;
  if (jm.ne <= 0 && jc.ne <= 0)
    return;
  // the lists of both graphs: one after the other, or side by side, half the blocks each, where an entry has
  // a thread even so (each phase is bound by latency; the stage of 1,000 spheres with 2,700 contacts takes 111 us
  // so, 121 one after the other; of 500 with one each 61 and 69)
  const long half = (long)(gridDim.x / 2) * blockDim.x;
  const bool side = jm.ne > 0 && jc.ne > 0 && max(jm.ne, jc.ne) <= half;
  const bool inM = !side || gtid < half, inC = !side || gtid >= half;
  const long idC = side ? gtid - half : gtid, strideM = side ? half : gstride, strideC = side ? gstride - half : gstride;
  if (inM)
    colorInit<R, true>(d, jm, gtid, strideM);
  if (inC)
    colorInit<R, false>(d, jc, idC, strideC);
  if (!loopBarrier<CLUSTER>(gb))
    return;
  if (inM)
    colorCount<R, true>(d, jm, gtid, strideM);
  if (inC)
    colorCount<R, false>(d, jc, idC, strideC);
  if (!loopBarrier<CLUSTER>(gb))
    return;
  if (inM)
    colorRoom(jm, gtid, strideM);
  if (inC)
    colorRoom(jc, idC, strideC);
  if (!loopBarrier<CLUSTER>(gb))
    return;
  if (inM)
    colorFill<R, true>(d, jm, gtid, strideM);
  if (inC)
    colorFill<R, false>(d, jc, idC, strideC);
  if (!loopBarrier<CLUSTER>(gb))
    return;
  if (inM)
    colorSort(jm, gtid, strideM);
  if (inC)
    colorSort(jc, idC, strideC);
  if (!loopBarrier<CLUSTER>(gb))
    return;
  if (CLUSTER && inShared) {
    extern __shared__ __align__(16) unsigned char colorSmem[];
    if (blockIdx.x < 2 && (blockIdx.x ? jc.ne : jm.ne) > 0)
      colorRounds(blockIdx.x ? jc : jm, maxRounds, reinterpret_cast<ColorBody*>(colorSmem));
  } else {
    colorRun(jm, jc, maxRounds, gb, gtid, gstride);
  }
  if (!loopBarrier<CLUSTER>(gb))  // every colour is visible
    return;
  if (gtid == 0) {
    const int rounds = max(jm.ne > 0 ? __ldcg(&jm.aux[2]) : 0, jc.ne > 0 ? __ldcg(&jc.aux[2]) : 0);
    if (jm.ne > 0)
      jm.aux[5] = rounds;
    if (jc.ne > 0)
      jc.aux[5] = rounds;
  }
  colorStats(jm, gtid, gstride);
  colorStats(jc, gtid, gstride);
  // both colour orders (unless kept or batched: then the host orders them)
  if (!jm.order && !jc.order)
    return;
  colorOrderCount(jm);
  colorOrderCount(jc);
  if (!loopBarrier<CLUSTER>(gb))
    return;
  if (blockIdx.x == 0)
    colorOrderScan(jm);
  if (blockIdx.x == (gridDim.x > 1 ? 1 : 0))
    colorOrderScan(jc);
  if (!loopBarrier<CLUSTER>(gb))
    return;
  colorOrderScatter(jm);
  colorOrderScatter(jc);
}

}  // namespace pdem
