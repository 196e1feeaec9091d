// loop2d.cuh — the 2D outer loop as one resident kernel (included by fim_device.cu
// inside its unnamed namespace).
//
// k_loop2d runs a whole 2D solve or batch: initial state, then per outer iteration the
// sweeps of the active blocks (FIMCuda, core2d/cuda/CUDA_kernels.cu:36-409, 7 sweeps)
// with the host's activation step behind each visit (meshFIM2d_eikonal.cu:734-756), a
// grid barrier, the checks (run_check_neighbor, CUDA_kernels.cu:415-799) with the
// all-vertex convergence test (meshFIM2d_eikonal.cu:801-815) of the vertices they
// write, and a second grid barrier whose last CTA closes the iteration.  The grid is
// a cooperative launch, so all of its CTAs are resident and may wait for one another.
//
// What bounds it: latency.  A 33 x 33 grid has 68 blocks, an icosphere of 10,242
// vertices 160; an iteration has a few dozen visits, less than one per SM, and each is
// a chain of dependent steps.  As four kernels of a CUDA graph per iteration (sweeps,
// activation, checks, vertex test) the iteration took 25 us, 12 of them in a sweep
// visit and 4 in a check visit.  Here:
//   * two grid barriers take the place of four kernel boundaries;
//   * a slot has three lanes, one per corner update (tri_candidate), with its corner's
//     constants in registers (the reference's cosine and products do not change with
//     the times); the other two corners come by shuffles.  Blocks of more than 320
//     slots have one lane per slot, which then runs the three updates;
//   * the owned times are kept as two sets of integer keys that swap roles every
//     sweep, the next set taking the minimum of the candidates, so a sweep has one
//     CTA barrier and no merge pass;
//   * where CTAs have several visits an iteration (k_loop2d), one warp fetches the next
//     visit's descriptor during the sweeps, three dependent reads that began every visit
//     (a batch of 256 icospheres: 11.8 -> 10.9 ms, 2560 blocks: 1.89 -> 1.80 ms);
//   * with one lane per slot the slot is turned so that its earliest corner comes last
//     and its update is nearly always left out (Slot2::turn; the batch: 10.9 -> 10.6 ms).
//     That batch is bound by latency, not by arithmetic: 8 CTAs an SM wait half of the
//     time, a fourth of it at the grid barriers.  No gain: ending the sweeps when nothing
//     changes (0.96x: a reduction in every barrier), one root at a time (0.97x), claims in
//     place of a fixed order (0.98x), slots fetched ahead into L1 (0.95x);
//   * the all-vertex test looks only at the vertices that a check wrote (all others
//     kept their values, which the test would find equal) and at a count of
//     unreached vertices.

// ---------------------------------------------------------------------------
// grid barrier
// ---------------------------------------------------------------------------
// Every CTA calls grid_arrive / grid_wait with the number of the barrier (1, 2, ...).
// The wait is bounded (about four seconds of device time): a CTA that gives up raises
// the error flag and leaves, and so do the others, which see the flag or run out too.
constexpr unsigned long long kGridWaitNs = 4000000000ull;
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// thread 0, after a CTA barrier: counts this CTA in, releasing its threads' writes; true
// for the last one of barrier `number` (of n CTAs), which then sees the others' writes
__device__ __forceinline__ bool grid_arrive(unsigned* count, unsigned want) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(count) : "memory");
  return old + 1u == want;
}
// thread 0: waits until *word reaches `want`
__device__ __forceinline__ bool grid_wait(GridBar* g, const unsigned* word, unsigned want,
                                          unsigned long long limit_ns = kGridWaitNs) {
  unsigned long long t0 = 0;
  for (unsigned i = 0;; ++i) {
    if ((int)(ld_acquire(word) - want) >= 0) return true;
    if (i > 4) __nanosleep(32);
    if ((i & 255u) == 255u) {
      if (ld_acquire(&g->fail)) return false;
      const unsigned long long t = global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > limit_ns) {
        st_release(&g->fail, 1u);
        return false;
      }
    }
  }
}

// A small grid polls the arrival count itself.  More CTAs would hold up the arrivals by
// their polling (an iteration of 320 resident blocks took 14.2 us so, against 11.6);
// there the last CTA lets the others go through kGridFlags words on lines of their own,
// each polled by every kGridFlags-th CTA.  That hop costs 1.2 us an iteration where it
// is not needed (68 resident blocks 7.0 against 8.2 us).  The lines lie between the
// measured sizes: resident blocks 68 and 160 (10.2 against 11.2 us), lists 152 (14.5
// against 15.8 us) and 304.
constexpr int kFlatBlocks = 96, kFlatList = 192;
constexpr int kGridFlags = 16;
struct __align__(128) GridFlag {
  unsigned go;
  unsigned pad[31];
};
// thread 0 of the last CTA
__device__ __forceinline__ void grid_release(GridFlag* f, unsigned number) {
  __threadfence();
#pragma unroll
  for (int i = 0; i < kGridFlags; ++i) asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(&f[i].go), "r"(number) : "memory");
}

// ---------------------------------------------------------------------------
// triangle update with explicit roundings
// ---------------------------------------------------------------------------
// The update of corner C from A and B in the roundings of the reference's kernels
// (tri_update in local_update.cuh, whose products and sums the compiler fuses as it
// does the reference's): every operation is one IEEE operation, so the bits do not
// depend on the code around it.  Which products are fused was fitted to the visit
// kernels' outputs on 340,000 single-triangle blocks per kernel (realistic and random
// shapes, speeds and times), all of which it reproduces; the sweep kernel and the
// check kernel differ in the cosine's numerator.  Everything that does not depend on
// the times is formed once per visit, in the order the reference forms it.
struct TriConst {
  float AB;   // length AB
  float F;    // inverse speed
  float X;    // ((F F) AB) AB
  float cosA, K;       // cosine at A; ((2 AB) AC) cosA
  float C4, s2;        // (4 AC) AC; 1 - cosA cosA
  float AC2, ACsq;     // 2 AC; AC AC
  float EA, EB;        // AC F, BC F: the edges' travel times
};
template <bool kCheck>
__device__ __forceinline__ TriConst tri_const(float AB, float BC, float AC, float F) {
  TriConst c;
  c.AB = AB;
  c.F = F;
  c.X = __fmul_rn(__fmul_rn(__fmul_rn(F, F), AB), AB);
  c.ACsq = __fmul_rn(AC, AC);
  c.AC2 = __fmul_rn(2.0f, AC);
  const float num = kCheck ? __fmaf_rn(-BC, BC, __fmaf_rn(AB, AB, c.ACsq))
                           : __fsub_rn(__fadd_rn(c.ACsq, __fmul_rn(AB, AB)), __fmul_rn(BC, BC));
  c.cosA = __fdiv_rn(num, __fmul_rn(c.AC2, AB));
  c.K = __fmul_rn(__fmul_rn(__fmul_rn(2.0f, AB), AC), c.cosA);
  c.C4 = __fmul_rn(__fmul_rn(4.0f, AC), AC);
  c.s2 = __fmaf_rn(-c.cosA, c.cosA, 1.0f);
  c.EA = __fmul_rn(AC, F);
  c.EB = __fmul_rn(BC, F);
  return c;
}
// the least candidate at C (a NaN one is left out, as the reference's MIN leaves it out)
__device__ __forceinline__ float tri_candidate(const TriConst& c, float TA, float TB) {
  const float TAB = __fsub_rn(TB, TA);
  const float W = __fsub_rn(c.X, __fmul_rn(TAB, TAB));
  const float a = __fmul_rn(__fmul_rn(W, c.AB), c.AB);
  float best = mn2(__fadd_rn(TA, c.EA), __fadd_rn(TB, c.EB));
  if (a > 0.0f) {
    const float nb = __fmul_rn(c.K, W);  // -b: the reference's b is K (TAB TAB - X)
    const float sd = __fsqrt_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(c.C4, a), TAB), TAB), c.s2));
    const float a2 = __fmul_rn(2.0f, a);
    // both roots at once: their quotients and square roots are independent chains (a
    // root outside [0, 1] may give a NaN, which its test keeps out)
    const float l1 = __fdiv_rn(__fadd_rn(nb, sd), a2), l2 = __fdiv_rn(__fsub_rn(nb, sd), a2);
    const float D1 = __fmul_rn(l1, c.AB), D2 = __fmul_rn(l2, c.AB);
    const float q1 = __fmaf_rn(-__fmul_rn(c.AC2, D1), c.cosA, __fmaf_rn(D1, D1, c.ACsq));
    const float q2 = __fmaf_rn(-__fmul_rn(c.AC2, D2), c.cosA, __fmaf_rn(D2, D2, c.ACsq));
    const float r1 = __fmaf_rn(__fsqrt_rn(q1), c.F, __fmaf_rn(l1, TAB, TA));
    const float r2 = __fmaf_rn(__fsqrt_rn(q2), c.F, __fmaf_rn(l2, TAB, TA));
    if (l1 >= 0.0f && l1 <= 1.0f) best = mn2(r1, best);
    if (l2 >= 0.0f && l2 <= 1.0f) best = mn2(r2, best);
  }
  return best;
}

// ---------------------------------------------------------------------------
// one visit
// ---------------------------------------------------------------------------
struct Smem2 {
  int* key[2];  // max_owned: the owned times' bits (times are never negative)
  float* halo;  // max_local: the halo's times
};
__host__ __device__ inline size_t smem_bytes_loop2d(int max_local, int max_owned, bool resident) {
  return (sizeof(int) * (resident ? 4 : 2) * (size_t)max_owned + sizeof(float) * (size_t)max_local + 15) & ~(size_t)15;
}
// slots a CTA of `threads` holds with three lanes per slot (ten slots a warp)
__host__ __device__ inline int loop2d_slots(int threads) { return threads / 32 * 10; }

// A thread's corners: one of a slot's three (kLanes = 3) or all of them (kLanes = 1).
template <int kLanes>
struct Slot2 {
  static constexpr int kC = (kLanes == 3) ? 1 : 3;
  int id[kC];       // local vertex
  bool live[kC];    // an owned vertex's refreshed copy: its value is the vertex's key
  bool dead[kC];    // a copy that the reference never refreshes: starts from dval
  float dval[kC];
  float e[3], F;    // the slot's edge lengths and inverse speed
  bool mine;
  __device__ __forceinline__ static int corner(int q) { return (kLanes == 3) ? (int)(threadIdx.x & 31) % 3 : q; }
  // the slot's constants from global memory (dval apart)
  __device__ __forceinline__ void load(const DevArgs& a, const BlockDesc& bd) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int j = (kLanes == 3) ? (tid >> 5) * 10 + lane / 3 : tid;
    mine = j < bd.nslots && (kLanes == 1 || lane < 30);
    uint2 l = make_uint2(0u, 0u);
    e[0] = e[1] = e[2] = F = 1.0f;
    if (mine) {
      l = a.lv[bd.slot_begin + j];
      const float* q = a.coef + 4 * (size_t)bd.slot_begin + j;
      e[0] = q[0];
      e[1] = q[bd.nslots_pad];
      e[2] = q[2 * (size_t)bd.nslots_pad];
      F = q[3 * (size_t)bd.nslots_pad];
    }
#pragma unroll
    for (int q = 0; q < kC; ++q) {
      const int c = corner(q);
      const int raw = c == 0 ? (int)(l.x & 0xffffu) : c == 1 ? (int)(l.x >> 16) : (int)(l.y & 0xffffu);
      id[q] = raw & 0x7fff;
      dead[q] = (raw & 0x8000) != 0;
      live[q] = mine && !dead[q] && id[q] < bd.nowned;
      dval[q] = 0.0f;
    }
  }
  __device__ __forceinline__ void load_dead(const DevArgs& a, const BlockDesc& bd) {
#pragma unroll
    for (int q = 0; q < kC; ++q)
      if (mine && dead[q])
        dval[q] = a.Tinit[id[q] < bd.nowned ? bd.vbase + id[q] : a.halo[bd.halo_begin + id[q] - bd.nowned]];
  }
  // One lane per slot, with the block's times staged: turns the slot so that its earliest
  // corner comes last.  The others' updates then nearly always leave it as it is
  // (settled2d), and the third update is not run.
  __device__ __forceinline__ void turn(const Smem2& s, int nown) {
    float t[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) t[q] = value(s, nown, q);
    const int by = (t[0] < t[1] && t[0] < t[2]) ? 1 : (t[1] < t[2]) ? 2 : 0;  // new corner q is corner q + by
    const auto pick = [by](auto& v) {
      const auto x = v[0], y = v[1], z = v[2];
      v[0] = by == 0 ? x : by == 1 ? y : z;
      v[1] = by == 0 ? y : by == 1 ? z : x;
      v[2] = by == 0 ? z : by == 1 ? x : y;
    };
    pick(id);
    pick(live);
    pick(dead);
    pick(dval);
    pick(e);
  }
  // corner q's time at the start of a visit
  __device__ __forceinline__ float value(const Smem2& s, int nown, int q) const {
    if (!mine || dead[q]) return dval[q];
    return id[q] >= nown ? s.halo[id[q] - nown] : __int_as_float(s.key[0][id[q]]);
  }
  template <bool kCheck>
  __device__ __forceinline__ TriConst corner_const(int q) const {
    return tri_const<kCheck>(e[(q + 1) % 3], e[(q + 2) % 3], e[q], F);
  }
  template <bool kCheck>
  __device__ __forceinline__ void consts(TriConst* tc) const {
#pragma unroll
    for (int q = 0; q < (kLanes == 3 ? 1 : 2); ++q) {
      const int c = corner(q);
      tc[q] = tri_const<kCheck>(c == 0 ? e[1] : c == 1 ? e[2] : e[0], c == 0 ? e[2] : c == 1 ? e[0] : e[1],
                                c == 0 ? e[0] : c == 1 ? e[1] : e[2], F);
    }
  }
};

// Whether no candidate at C (time T) from A and B can be below T: not those along the
// edges, whose travel times are known, and not one inside, which is a convex combination
// of TA and TB, off by less than 2^-22 of the larger after rounding, plus a distance.
__device__ __forceinline__ bool settled2d(float T, float TA, float TB, float EA, float EB) {
  return T <= __fadd_rn(TA, EA) && T <= __fadd_rn(TB, EB) && T <= __fmaf_rn(fmaxf(TA, TB), -0x1p-20f, fminf(TA, TB));
}

// n sweeps over the block whose owned times are in both key sets and whose halo times
// are in s.halo; leaves the final owned times in s.key[n & 1] and those before the last
// sweep in the other set.  Ends with a CTA barrier (the caller has one before).
template <bool kCheck, int kSweeps, int kLanes>
__device__ __forceinline__ void sweep2d(const Slot2<kLanes>& sl, const TriConst* tc, const Smem2& s, int nown) {
  constexpr int kC = Slot2<kLanes>::kC;
  const int lane = threadIdx.x & 31;
  float h[kC], pown[kC];
#pragma unroll
  for (int q = 0; q < kC; ++q) {
    h[q] = (sl.mine && !sl.dead[q] && sl.id[q] >= nown) ? s.halo[sl.id[q] - nown] : sl.dval[q];
    pown[q] = sl.live[q] ? __int_as_float(s.key[0][sl.id[q]]) : h[q];
  }
  float pA = 0.0f, pB = 0.0f;  // three lanes: the other corners' times in the sweep before
  const int c0 = lane % 3, base = lane - c0;
  int* cur = s.key[0];
  int* nxt = s.key[1];
#pragma unroll 1
  for (int sw = 0; sw < kSweeps; ++sw) {
    float own[kC], TA[kC], TB[kC];
#pragma unroll
    for (int q = 0; q < kC; ++q) own[q] = sl.live[q] ? __int_as_float(cur[sl.id[q]]) : h[q];
    if constexpr (kLanes == 3) {
      TA[0] = __shfl_sync(0xffffffffu, own[0], base + (c0 == 2 ? 0 : c0 + 1));
      TB[0] = __shfl_sync(0xffffffffu, own[0], base + (c0 == 0 ? 2 : c0 - 1));
    } else {
#pragma unroll
      for (int q = 0; q < kC; ++q) {
        TA[q] = own[(q + 1) % 3];
        TB[q] = own[(q + 2) % 3];
      }
    }
    // An update whose three times are unreached gives nothing, and one whose times did
    // not change since the sweep before repeats a candidate that its corner already has.
    bool run = sl.mine && !(own[0] >= kLarge2DDev && TA[0] >= kLarge2DDev && TB[0] >= kLarge2DDev);
    if (sw > 0) {
      if constexpr (kLanes == 3)
        run = run && (own[0] != pown[0] || TA[0] != pA || TB[0] != pB);
      else
        run = run && (own[0] != pown[0] || own[kC > 1 ? 1 : 0] != pown[kC > 1 ? 1 : 0] ||
                      own[kC > 2 ? 2 : 0] != pown[kC > 2 ? 2 : 0]);
    }
#pragma unroll
    for (int q = 0; q < kC; ++q) {
      float nw = own[q];
      if (kLanes == 3 || q < 2) {
        if (run) nw = mn2(own[q], tri_candidate(tc[q], TA[q], TB[q]));
      } else if (run && !settled2d(own[q], TA[q], TB[q], __fmul_rn(sl.e[q], sl.F), __fmul_rn(sl.e[(q + 2) % 3], sl.F))) {
        // (see Slot2::turn; its constants are formed here, as they are seldom needed)
        nw = mn2(own[q], tri_candidate(sl.template corner_const<kCheck>(q), TA[q], TB[q]));
      }
      // the next set still holds the value before this one (pown): a copy whose value
      // did not fall since then has nothing to add
      if (sl.live[q]) {
        if (nw < pown[q]) atomicMin(&nxt[sl.id[q]], __float_as_int(nw));
      } else {
        h[q] = nw;
      }
      pown[q] = own[q];
    }
    if constexpr (kLanes == 3) {
      pA = TA[0];
      pB = TB[0];
    }
    int* t = cur;
    cur = nxt;
    nxt = t;
    __syncthreads();
  }
}

// Loads block bd with the times of Tsrc and runs kSweeps sweeps on it.
// `aside` runs in the last warp while the sweeps do: a block's slots seldom reach it.
template <bool kCheck, int kSweeps, int kLanes, class Aside>
__device__ __forceinline__ void visit2d(const DevArgs& a, const BlockDesc& bd, const Smem2& s, const float* Tsrc,
                                        Aside aside) {
  Slot2<kLanes> sl;
  sl.load(a, bd);
  for (int k = threadIdx.x; k < bd.nowned; k += blockDim.x) {
    const int v = __float_as_int(__ldcg(Tsrc + bd.vbase + k));
    s.key[0][k] = v;
    s.key[1][k] = v;
  }
  for (int k = threadIdx.x; k < bd.nhalo; k += blockDim.x) s.halo[k] = __ldcg(Tsrc + a.halo[bd.halo_begin + k]);
  sl.load_dead(a, bd);
  TriConst tc[kLanes == 3 ? 1 : 3];
  if constexpr (kLanes == 3) sl.template consts<kCheck>(tc);
  __syncthreads();
  if (threadIdx.x >= blockDim.x - 32) aside();
  if constexpr (kLanes == 1) {
    sl.turn(s, bd.nowned);
    sl.template consts<kCheck>(tc);
  }
  sweep2d<kCheck, kSweeps, kLanes>(sl, tc, s, bd.nowned);
}

// ---------------------------------------------------------------------------
// the loop
// ---------------------------------------------------------------------------
// The meeting point of one instance's CTAs (k_blocks2d) or of a single solve's
// (k_loop2d).  next: blocks active in the next iteration, fail: some written vertex
// fails the all-vertex test, fresh: blocks queued for a check; one word per iteration in
// turn: the words of iteration i + 1 are cleared during iteration i, when the readers of
// their last use, iteration i - 2, have all passed a later barrier.
struct __align__(16) InstSync {
  unsigned count;
  int unreached;  // vertices still at LARGENUM
  int next[3], fail[3], fresh[3];
  int pad;
};

struct Start2 {  // the solve's inputs, staged by the host in one copy
  const int* done;   // per instance: nothing to do
  const int* maxit;  // per instance: iteration cap
  const int* seeds;
  const int* act;    // starting blocks
  int nseeds, nact;
  const int* bbeg;   // per instance: its first block, and the block count at the end
  InstSync* sync;    // per instance, zero
  GridFlag* flags;   // kGridFlags words, zero
  int user_prev;     // a.prev holds the caller's initial values
  int telemetry;
};

// End of an iteration, by all threads of the last CTA (finish_iteration_cta's rules;
// an instance passes the all-vertex test when no written vertex moved by more than
// EPS and none is unreached).
__device__ __forceinline__ void close2d(const DevArgs& a) {
  Ctl* c = a.ctl;
  int any = 0;
  for (int i = threadIdx.x; i < a.ninst; i += blockDim.x) {
    const int nn = __ldcg(a.inst_nnext + i);
    const int fail = __ldcg(a.inst_fail + i) | (__ldcg(a.inst_unreached + i) > 0 ? 1 : 0);
    if (__ldcg(a.inst_done + i) == 0) {
      const int own = __ldcg(a.inst_iters + i) + 1;
      a.inst_iters[i] = own;
      if (nn == 0 || own >= a.inst_maxit[i] || fail == 0) a.inst_done[i] = 1;
      else any = 1;
    }
    if (nn) a.inst_nnext[i] = 0;
    a.inst_fail[i] = 0;
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) {
    c->iter = __ldcg(&c->iter) + 1;
    c->nact = __ldcg(&c->nnext);
    c->nnext = 0;
    c->nnew = 0;
    c->stop = any ? 0 : 1;
  }
}

template <int kLanes, int kRegs>
__global__ void __maxnreg__(kRegs) k_loop2d(DevArgs a, Start2 st) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_flag;
  Smem2 s;
  s.key[0] = reinterpret_cast<int*>(sm);
  s.key[1] = s.key[0] + a.max_owned;
  s.halo = reinterpret_cast<float*>(s.key[1] + a.max_owned);
  const int tid = threadIdx.x, lane = tid & 31, NT = blockDim.x;
  GridBar* const g = &a.ctl->bar;
  const int G = gridDim.x;
  const int gtid = blockIdx.x * NT + tid, gn = G * NT;
  unsigned bar = 0;
  GridFlag* const mine = st.flags + blockIdx.x % kGridFlags;
  // barrier, the last CTA running close() before it lets the others go; without a
  // closing step a small grid polls the count
  auto sync_grid = [&](auto close, bool flat) -> bool {
    ++bar;
    __syncthreads();
    if (flat) {
      if (tid == 0) {
        (void)grid_arrive(&g->count, 0u);
        s_flag = grid_wait(g, &g->count, bar * (unsigned)G) ? 1 : 0;
      }
      __syncthreads();
      return s_flag != 0;
    }
    if (tid == 0) s_flag = grid_arrive(&g->count, bar * (unsigned)G) ? 2 : 1;
    __syncthreads();
    if (s_flag == 2) {
      close();
      __syncthreads();
      if (tid == 0) grid_release(st.flags, bar);
      return true;
    }
    if (tid == 0 && !grid_wait(g, &mine->go, bar)) s_flag = 0;
    __syncthreads();
    return s_flag != 0;
  };
  const bool flat = G <= kFlatList;
  auto nothing = [] {};
  // ---- initial state ----
  for (int v = gtid; v < a.nv; v += gn) {
    a.Ta[v] = kLarge2DDev;
    a.Tb[v] = kLarge2DDev;
    const_cast<float*>(a.Tinit)[v] = kLarge2DDev;
  }
  for (int b = gtid; b < a.nb; b += gn) {
    a.stampA[b] = 0;
    a.stampC[b] = 0;
  }
  // a single solve needs no closing step: its counters stand in turning words that every
  // CTA reads after the barrier
  InstSync* const y = st.sync;
  const bool single = a.ninst == 1;
  if (single && gtid == 0) y->unreached = a.nv;
  for (int i = gtid; i < a.ninst; i += gn) {
    a.inst_done[i] = st.done[i];
    const_cast<int*>(a.inst_maxit)[i] = st.maxit[i];
    a.inst_iters[i] = 0;
    a.inst_nnext[i] = 0;
    a.inst_fail[i] = 0;
    a.inst_unreached[i] = a.inst_vbeg[i + 1] - a.inst_vbeg[i];
  }
  if (!sync_grid(nothing, flat)) return;
  for (int i = gtid; i < st.nseeds; i += gn) {
    const int v = st.seeds[i];
    if (atomicExch(&a.Ta[v], 0.0f) != 0.0f) atomicSub(single ? &y->unreached : &a.inst_unreached[a.blk_inst[a.vblock[v]]], 1);
    a.Tb[v] = 0.0f;
    const_cast<float*>(a.Tinit)[v] = 0.0f;
  }
  for (int i = gtid; i < st.nact; i += gn) {
    a.list0[i] = st.act[i];
    a.stampA[st.act[i]] = 1;
  }
  if (!sync_grid(nothing, flat)) return;
  int iter = 0, nact = st.nact;
  bool go = nact > 0 && a.ctl->max_iters > 0;
  const int cap0 = st.maxit[0];
  // thread 0's sums, added to the solve's at the end
  __shared__ VisitSum s_swept, s_checked;
  if (tid == 0) {
    s_swept.clear();
    s_checked.clear();
  }
  // the CTA's present and next item: words 0-7 the block's descriptor, 8 and 9 its range of
  // neighbours, 10 its instance, 11 the block, 12 whether the instance is finished
  __shared__ int s_item[2][16];
  const bool last_warp = tid >= NT - 32;
  const auto stage = [&](int* to, int b) {  // by one warp
    int w = 0;
    if (lane < 8) w = reinterpret_cast<const int*>(a.blocks + b)[lane];
    else if (lane < 10) w = a.nbr_off[b + lane - 8];
    else if (lane == 10) w = single ? 0 : a.blk_inst[b];
    else if (lane == 11) w = b;
    if (lane < 12) to[lane] = w;
    if (lane == 10) to[12] = single ? 0 : __ldcg(a.inst_done + w);
  };
  const auto item_block = [](const int* d) {
    BlockDesc bd;
    bd.slot_begin = d[0];
    bd.nslots = d[1];
    bd.nslots_pad = d[2];
    bd.vbase = d[3];
    bd.nowned = d[4];
    bd.halo_begin = d[5];
    bd.nhalo = d[6];
    bd.ninside = d[7];
    return bd;
  };
  static_assert(sizeof(BlockDesc) == 32, "staged as eight words");
  while (go) {
    const int stamp = iter + 1;
    const int now = iter % 3, clear = (iter + 1) % 3;
    const int* act = act_list(a, iter);
    if (single && gtid == 0) y->next[clear] = y->fail[clear] = y->fresh[clear] = 0;
    int* const p_fresh = single ? &y->fresh[now] : &a.ctl->nnew;
    int* const p_next = single ? &y->next[now] : &a.ctl->nnext;
    // ---- sweeps of the active blocks: read Ta, write Tb ----
    if (tid == 0 && blockIdx.x == 0 && st.telemetry && iter < a.ktime_cap) a.ktime[kKStride * iter] = ~global_ns();
    int par = 0;
    if (last_warp && blockIdx.x < nact) stage(s_item[0], __ldcg(act + blockIdx.x));
    __syncthreads();
    for (int item = blockIdx.x; item < nact; item += G, par ^= 1) {
      const int bn = (last_warp && item + G < nact) ? __ldcg(act + item + G) : -1;
      const int* const d = s_item[par];
      const auto ahead = [&] {
        if (bn >= 0) stage(s_item[par ^ 1], bn);
      };
      if (d[12]) {  // uniform across the CTA
        if (last_warp) ahead();
        __syncthreads();
        continue;
      }
      const BlockDesc bd = item_block(d);
      const int e0 = d[8], e1 = d[9];
      const int nb0 = (tid < 32 && e0 + lane < e1) ? a.nbr[e0 + lane] : -1;
      visit2d<false, 7, kLanes>(a, bd, s, a.Ta, ahead);
      int myconv = 1;
      for (int k = tid; k < bd.nowned; k += NT) {
        const float nv = __int_as_float(s.key[1][k]), ov = __int_as_float(s.key[0][k]);
        if (k < kReduceCap2D) {
          float res = ov - nv;
          if (res < 0.0f) res = -res;
          myconv &= (res <= kEps2D) ? 1 : 0;
        }
        a.Tb[bd.vbase + k] = nv;
      }
      const int allc = __syncthreads_and(myconv);
      if (allc && tid < 32) {  // queue the neighbours that are not active, once each
        for (int e = e0; e < e1; e += 32) {
          const int nb = (e == e0) ? nb0 : ((e + lane < e1) ? a.nbr[e + lane] : -1);
          bool q = false;
          if (nb >= 0) {
            const int sa = __ldcg(a.stampA + nb);
            const int old = atomicExch(&a.stampC[nb], stamp);
            q = sa != stamp && old != stamp;
          }
          const unsigned bal = __ballot_sync(0xffffffffu, q);
          if (bal) {
            int pos = 0;
            if (lane == 0) pos = atomicAdd(p_fresh, __popc(bal));
            pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(bal & ((1u << lane) - 1u));
            if (q) a.list_new[pos] = nb;
          }
        }
      }
      if (tid == 0) {
        s_swept.add(bd.nslots, bd.nhalo, bd.nowned);
        if (st.telemetry) count_visit(a, iter, 0, bd.nslots, bd.nhalo, bd.nowned);
      }
    }
    // the last iteration's snapshot: its times stand until the checks below
    if (a.hist_cap > 0 && iter > 0 && iter <= a.hist_cap)
      for (int v = gtid; v < a.nv; v += gn) a.hist[(size_t)(iter - 1) * a.nv + v] = __ldcg(a.Ta + v);
    if (!sync_grid(nothing, flat)) return;
    if (tid == 0 && blockIdx.x == 0 && st.telemetry && iter < a.ktime_cap) {
      const unsigned long long t = global_ns();
      a.ktime[kKStride * iter + 1] = t;
      a.ktime[kKStride * iter + 2] = ~t;
    }
    // ---- checks of the active and the queued blocks: read Tb, write Ta ----
    const int count = nact + __ldcg(p_fresh);
    int* nxt = next_list(a, iter);
    const auto queued = [&](int item) { return __ldcg(item < nact ? act + item : a.list_new + item - nact); };
    par = 0;
    // (a CTA that had one sweep at most still holds that block's descriptor)
    if (last_warp && blockIdx.x < count && (blockIdx.x >= nact || nact > G)) stage(s_item[0], queued(blockIdx.x));
    __syncthreads();
    for (int item = blockIdx.x; item < count; item += G, par ^= 1) {
      const int bn = (last_warp && item + G < count) ? queued(item + G) : -1;
      const int* const d = s_item[par];
      const auto ahead = [&] {
        if (bn >= 0) stage(s_item[par ^ 1], bn);
      };
      if (d[12]) {
        if (last_warp) ahead();
        __syncthreads();
        continue;
      }
      const BlockDesc bd = item_block(d);
      const int inst = d[10], b = d[11];
      // what the all-vertex test compares with: the times before this check, which are
      // the values it kept, except the caller's initial values in its first iteration
      const float* before =
          (st.user_prev && (a.ninst > 1 ? __ldcg(a.inst_iters + inst) : iter) == 0) ? a.prev : a.Ta;
      const float old0 = (tid < bd.nowned) ? __ldcg(a.Ta + bd.vbase + tid) : 0.0f;
      const float was0 = (before == a.Ta || tid >= bd.nowned) ? old0 : __ldcg(before + bd.vbase + tid);
      visit2d<true, 1, kLanes>(a, bd, s, a.Tb, ahead);
      int myconv = 1, bad = 0, reached = 0;
      for (int k = tid; k < bd.nowned; k += NT) {
        const float nv = __int_as_float(s.key[1][k]), ov = __int_as_float(s.key[0][k]);
        if (k < kReduceCap2D) myconv &= ((ov - nv) < kEps2D) ? 1 : 0;
        const float old = (k == tid) ? old0 : __ldcg(a.Ta + bd.vbase + k);
        const float was = (k == tid) ? was0 : (before == a.Ta ? old : __ldcg(before + bd.vbase + k));
        float diff = was - nv;
        if (diff < 0.0f) diff = -diff;
        if (!((diff <= kEps2D) && (nv < kLarge2DDev))) bad = 1;
        reached += (nv < kLarge2DDev ? 1 : 0) - (old < kLarge2DDev ? 1 : 0);
        a.Ta[bd.vbase + k] = nv;
      }
      if (bad) *(single ? &y->fail[now] : &a.inst_fail[inst]) = 1;
      if (reached) atomicSub(single ? &y->unreached : &a.inst_unreached[inst], reached);
      const int allc = __syncthreads_and(myconv);
      if (tid == 0) {
        if (!allc) {
          nxt[atomicAdd(p_next, 1)] = b;
          if (!single) atomicAdd(&a.inst_nnext[inst], 1);
          a.stampA[b] = stamp + 1;  // member of the next iteration's active list
        }
        s_checked.add(bd.nslots, bd.nhalo, bd.nowned);
        if (st.telemetry) count_visit(a, iter, 1, bd.nslots, bd.nhalo, bd.nowned);
      }
    }
    // ---- close ----
    if (single) {
      if (!sync_grid(nothing, flat)) return;
      if (gtid == 0 && st.telemetry && iter < a.ktime_cap) a.ktime[kKStride * iter + 3] = global_ns();
      nact = __ldcg(&y->next[now]);
      const int fail = __ldcg(&y->fail[now]), far = __ldcg(&y->unreached);
      ++iter;
      go = nact > 0 && iter < cap0 && (fail != 0 || far > 0);
      continue;
    }
    if (!sync_grid([&] {
          close2d(a);
          if (tid == 0 && st.telemetry && iter < a.ktime_cap) a.ktime[kKStride * iter + 3] = global_ns();
        }, false))
      return;
    nact = __ldcg(&a.ctl->nact);
    go = __ldcg(&a.ctl->stop) == 0;
    ++iter;
  }
  if (a.hist_cap > 0 && iter > 0 && iter <= a.hist_cap)
    for (int v = gtid; v < a.nv; v += gn) a.hist[(size_t)(iter - 1) * a.nv + v] = __ldcg(a.Ta + v);
  if (tid == 0) {
    Ctl* c = a.ctl;
    if (single && blockIdx.x == 0) {
      c->iter = iter;
      a.inst_iters[0] = iter;
    }
    const VisitSum f = s_swept, h = s_checked;
    if (f.visits) {
      atomicAdd(&c->fim_visits, f.visits);
      atomicAdd(&c->fim_slots, f.slots);
      atomicAdd(&c->fim_halo, f.halo);
      atomicAdd(&c->fim_owned, f.owned);
    }
    if (h.visits) atomicAdd(&c->chk_visits, h.visits);
    if (f.visits + h.visits) {
      atomicAdd(&c->updates, 7ull * f.owned + h.owned);
      atomicAdd(&c->slot_visits, f.slots + h.slots);
      atomicAdd(&c->halo_visits, f.halo + h.halo);
      atomicAdd(&c->owned_visits, f.owned + h.owned);
    }
  }
}

// ---------------------------------------------------------------------------
// the loop with every block resident
// ---------------------------------------------------------------------------
// Where the GPU holds one CTA per block, each CTA keeps its block for the whole solve:
// slot constants, triangle constants and halo ids stay in registers and its own times
// in shared memory, so a visit reads nothing but the halo's times; no lists are kept
// (a CTA knows whether its block is active, and a converged block marks its neighbours
// for the check); and every instance of a batch has barriers and an end of its own.
// Per iteration an active block costs one round of loads, seven sweeps, a barrier, one
// round of loads, a sweep and a barrier.
template <int kRegs>
__global__ void __maxnreg__(kRegs) k_blocks2d(DevArgs a, Start2 st) {
  constexpr int kLanes = 3;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_flag, s_active;
  Smem2 s;
  s.key[0] = reinterpret_cast<int*>(sm);
  s.key[1] = s.key[0] + a.max_owned;
  s.halo = reinterpret_cast<float*>(s.key[1] + a.max_owned);
  float* const ta = s.halo + a.max_local;  // own values of a.Ta and a.Tb
  float* const tb = ta + a.max_owned;
  const int tid = threadIdx.x, NT = blockDim.x;
  const int b = blockIdx.x;
  const int inst = (a.ninst > 1) ? a.blk_inst[b] : 0;
  const BlockDesc bd = a.blocks[b];
  const int cap = st.maxit[inst];
  if (st.done[inst]) {  // nothing to do: the initial times are the result
    for (int k = tid; k < bd.nowned; k += NT) a.Ta[bd.vbase + k] = kLarge2DDev;
    __syncthreads();
    for (int i = tid; i < st.nseeds; i += NT) {
      const int v = st.seeds[i] - bd.vbase;
      if (v >= 0 && v < bd.nowned) a.Ta[bd.vbase + v] = 0.0f;
    }
    if (tid == 0 && b == st.bbeg[inst]) a.inst_iters[inst] = 0;
    return;
  }
  InstSync* const y = st.sync + inst;
  const unsigned group = (unsigned)(st.bbeg[inst + 1] - st.bbeg[inst]);
  unsigned bar = 0;
  unsigned number = 0;
  GridFlag* const mine = st.flags + b % kGridFlags;
  auto sync_group = [&]() -> bool {
    bar += group;
    ++number;
    __syncthreads();
    if (tid == 0) {
      const bool last = grid_arrive(&y->count, bar);
      bool ok = true;
      if (a.ninst > 1 || group <= (unsigned)kFlatBlocks) {
        ok = grid_wait(&a.ctl->bar, &y->count, bar);
      } else if (last) {
        grid_release(st.flags, number);
      } else {
        ok = grid_wait(&a.ctl->bar, &mine->go, number);
      }
      s_flag = ok ? 1 : 0;
    }
    __syncthreads();
    return s_flag != 0;
  };
  // ---- the block's constants and initial times ----
  Slot2<kLanes> sl;
  sl.load(a, bd);
  TriConst tc[Slot2<kLanes>::kC], tk[Slot2<kLanes>::kC];
  sl.template consts<false>(tc);
  sl.template consts<true>(tk);
  const int hid = (tid < bd.nhalo) ? a.halo[bd.halo_begin + tid] : 0;
  const int e0 = a.nbr_off[b], e1 = a.nbr_off[b + 1];
  const int nb0 = (tid < e1 - e0) ? a.nbr[e0 + tid] : -1;
  if (tid == 0) {
    s_active = 0;
    a.stampC[b] = 0;
  }
  for (int k = tid; k < bd.nowned; k += NT) ta[k] = kLarge2DDev;
  __syncthreads();
  for (int i = tid; i < st.nseeds; i += NT) {
    const int v = st.seeds[i] - bd.vbase;
    if (v >= 0 && v < bd.nowned) {
      ta[v] = 0.0f;
      s_active = 1;
    }
  }
  __syncthreads();
  int far = 0;
  for (int k = tid; k < bd.nowned; k += NT) {
    const float v = ta[k];
    tb[k] = v;
    a.Ta[bd.vbase + k] = v;
    a.Tb[bd.vbase + k] = v;
    const_cast<float*>(a.Tinit)[bd.vbase + k] = v;
    far += (v >= kLarge2DDev) ? 1 : 0;
  }
  if (far) atomicAdd(&y->unreached, far);
  bool active = s_active != 0;
  if (!sync_group()) return;
  sl.load_dead(a, bd);
  unsigned n_fim = 0, n_chk = 0;
  int iter = 0;
  for (;;) {
    const int stamp = iter + 1;
    const int now = iter % 3, clear = (iter + 1) % 3;
    if (tid == 0 && b == st.bbeg[inst]) y->next[clear] = y->fail[clear] = 0;
    if (active) {  // ---- FIMCuda ----
      if (st.telemetry) stamp_start(a, iter, 0);
      for (int k = tid; k < bd.nowned; k += NT) s.key[0][k] = s.key[1][k] = __float_as_int(ta[k]);
      if (tid < bd.nhalo) s.halo[tid] = __ldcg(a.Ta + hid);
      for (int k = tid + NT; k < bd.nhalo; k += NT) s.halo[k] = __ldcg(a.Ta + a.halo[bd.halo_begin + k]);
      __syncthreads();
      sweep2d<false, 7, kLanes>(sl, tc, s, bd.nowned);
      int myconv = 1;
      for (int k = tid; k < bd.nowned; k += NT) {
        const float nv = __int_as_float(s.key[1][k]), ov = __int_as_float(s.key[0][k]);
        if (k < kReduceCap2D) {
          float res = ov - nv;
          if (res < 0.0f) res = -res;
          myconv &= (res <= kEps2D) ? 1 : 0;
        }
        tb[k] = nv;
        a.Tb[bd.vbase + k] = nv;
      }
      if (__syncthreads_and(myconv)) {  // its neighbours are checked
        if (nb0 >= 0) a.stampC[nb0] = stamp;
        for (int e = e0 + tid + NT; e < e1; e += NT) a.stampC[a.nbr[e]] = stamp;
      }
      ++n_fim;
      if (st.telemetry) {
        stamp_end(a, iter, 0);
        if (tid == 0) count_visit(a, iter, 0, bd.nslots, bd.nhalo, bd.nowned);
      }
    }
    if (!sync_group()) return;
    // ---- run_check_neighbor: the queue mark and the halo come in one round ----
    const int queued = __ldcg(a.stampC + b);
    if (tid < bd.nhalo) s.halo[tid] = __ldcg(a.Tb + hid);
    if (active || queued == stamp) {
      if (st.telemetry) stamp_start(a, iter, 1);
      for (int k = tid + NT; k < bd.nhalo; k += NT) s.halo[k] = __ldcg(a.Tb + a.halo[bd.halo_begin + k]);
      for (int k = tid; k < bd.nowned; k += NT) s.key[0][k] = s.key[1][k] = __float_as_int(tb[k]);
      __syncthreads();
      sweep2d<true, 1, kLanes>(sl, tk, s, bd.nowned);
      int myconv = 1, bad = 0, reached = 0;
      for (int k = tid; k < bd.nowned; k += NT) {
        const float nv = __int_as_float(s.key[1][k]), ov = __int_as_float(s.key[0][k]);
        if (k < kReduceCap2D) myconv &= ((ov - nv) < kEps2D) ? 1 : 0;
        // the all-vertex test compares with the times before this check, in the first
        // iteration with the caller's initial values
        const float old = ta[k];
        const float was = (iter == 0 && st.user_prev) ? a.prev[bd.vbase + k] : old;
        float diff = was - nv;
        if (diff < 0.0f) diff = -diff;
        if (!((diff <= kEps2D) && (nv < kLarge2DDev))) bad = 1;
        reached += (nv < kLarge2DDev ? 1 : 0) - (old < kLarge2DDev ? 1 : 0);
        ta[k] = nv;
        a.Ta[bd.vbase + k] = nv;
      }
      if (bad) y->fail[now] = 1;
      if (reached) atomicSub(&y->unreached, reached);
      active = __syncthreads_and(myconv) == 0;
      if (tid == 0 && active) y->next[now] = 1;
      ++n_chk;
      if (st.telemetry) {
        stamp_end(a, iter, 1);
        if (tid == 0) count_visit(a, iter, 1, bd.nslots, bd.nhalo, bd.nowned);
      }
    } else {
      active = false;
    }
    if (iter < a.hist_cap)
      for (int k = tid; k < bd.nowned; k += NT) a.hist[(size_t)iter * a.nv + bd.vbase + k] = ta[k];
    if (!sync_group()) return;
    ++iter;
    if (__ldcg(&y->next[now]) == 0 || iter >= cap || (__ldcg(&y->fail[now]) == 0 && __ldcg(&y->unreached) <= 0)) break;
  }
  if (tid == 0) {
    Ctl* c = a.ctl;
    if (b == st.bbeg[inst]) {
      a.inst_iters[inst] = iter;
      atomicMax(&c->iter, iter);
    }
    if (n_fim) {
      atomicAdd(&c->fim_visits, (unsigned long long)n_fim);
      atomicAdd(&c->fim_slots, (unsigned long long)n_fim * bd.nslots);
      atomicAdd(&c->fim_halo, (unsigned long long)n_fim * bd.nhalo);
      atomicAdd(&c->fim_owned, (unsigned long long)n_fim * bd.nowned);
    }
    if (n_chk) atomicAdd(&c->chk_visits, (unsigned long long)n_chk);
    const unsigned long long n = n_fim + n_chk;
    if (n) {
      atomicAdd(&c->updates, (7ull * n_fim + n_chk) * bd.nowned);
      atomicAdd(&c->slot_visits, n * bd.nslots);
      atomicAdd(&c->halo_visits, n * bd.nhalo);
      atomicAdd(&c->owned_visits, n * bd.nowned);
    }
  }
}
