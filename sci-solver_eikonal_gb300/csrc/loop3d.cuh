// loop3d.cuh — the 3D outer loop as one resident kernel (included by fim_device.cu inside
// its unnamed namespace, behind loop2d.cuh and visit3d.cuh).
//
// k_loop3d runs a whole 3D solve or batch with the visits of visit3d.cuh.  As three
// kernels of a CUDA graph per iteration (visits, commit, close; 17^3 cube 775 us, 41^3
// 2.06 ms, 65^3 3.43 ms, 97^3 7.90 ms a solve, against 470 us, 1.68, 2.80 and 7.28 ms) an
// iteration spent 7-8 us between its visits' end and the next one's first loads, a quarter
// of it where a few dozen blocks are active.  Here an iteration has one grid barrier and no commit
// step:
//   * the times stand in two buffers; iteration i reads one and writes the swept blocks'
//     times to the other, so that no visit sees a neighbour's new times.  A block swept in
//     iteration i - 1 but not in i would be stale in the buffer that i writes: a check
//     that finds it settled writes its times there, and the others, which had converged
//     and were not queued, are listed and copied (meshFIM3dEikonal.cu's CopyOutBack
//     copies every swept block);
//   * a visit's tail queues its block for the next iteration, or a converged block's
//     neighbours for a check (meshFIM3dEikonal.cu:438-488).  A neighbour that this
//     iteration leaves unconverged may be queued too, before that is known; its stamp
//     tells the next iteration to pass it over;
//   * counters stand in words that take turns over three iterations, so a single solve
//     needs no closing step; a batch's instances are closed by the barrier's last CTA.
// Memos count only once a block has written them in this solve (mvalid), which spares
// clearing 32 bytes per slot before every solve.
struct __align__(32) Turn3 {
  int next, cand, conv;  // blocks queued for the next iteration, for a check, for a copy
  int work;              // items claimed
  int add;               // blocks that a check made active
  int pad[3];
};

struct Start3 {
  const int* done;   // per instance: nothing to do
  const int* maxit;  // per instance: iteration cap
  const int* seeds;
  const int* act;    // starting blocks
  int nseeds, nact;
  Turn3* turn;       // three, zero
  GridFlag* flags;   // kGridFlags, zero
  int* conv;         // two lists of a.nb converged blocks
  int* mvalid;       // per block: bit 0 its check memos are this solve's, bit 1 its sweep memos
  int* queued[2];    // per block: stamp of the even / odd iteration that queued it for a check
};

// End of a batch's iteration, by all threads of the barrier's last CTA: the rules of
// finish_iteration_cta.
__device__ __forceinline__ void finish_loop3d(const DevArgs& a, int iter) {
  int any = 0, swept = 0;
  for (int i = threadIdx.x; i < a.ninst; i += blockDim.x) {
    const int ist = __ldcg(a.inst_done + i), nsw = __ldcg(a.inst_swept + i);
    const int pend_check = __ldcg(a.inst_ncand + i), nn = __ldcg(a.inst_nnext + i);
    if (ist == 0 && nsw == 0) {
      a.inst_done[i] = 1;
    } else if (ist == 0) {
      swept = 1;
      const int own = __ldcg(a.inst_iters + i) + 1;
      a.inst_iters[i] = own;
      if (nn + pend_check > 0 && own < a.inst_maxit[i]) {
        any = 1;
      } else if (pend_check > 0) {
        a.inst_done[i] = 2;  // at its cap: the checks of this iteration still run
        any = 1;
      } else {
        a.inst_done[i] = 1;
      }
    } else if (ist == 2) {
      a.inst_done[i] = 1;
    }
    if (nn) a.inst_nnext[i] = 0;
    if (nsw) a.inst_swept[i] = 0;
    if (pend_check) a.inst_ncand[i] = 0;
  }
  any = __syncthreads_or(any);
  swept = __syncthreads_or(swept);
  if (threadIdx.x == 0) {
    a.ctl->iter = iter + 1;
    if (!swept) a.ctl->idle_iters = __ldcg(&a.ctl->idle_iters) + 1;
    a.ctl->stop = any ? 0 : 1;
  }
}

// copies of the times of the blocks listed by the last iteration that no visit of this
// one writes: one warp each, from the grid's end, where CTAs without a visit are
__device__ __forceinline__ void copy_settled(const DevArgs& a, const int* list, int n, const int* queued,
                                             int stamp, const float* Tsrc, float* Tdst) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int w0 = (int)(gridDim.x - 1 - blockIdx.x) * nw + (int)(threadIdx.x >> 5);
  for (int e = w0; e < n; e += (int)gridDim.x * nw) {
    const int b = __ldcg(list + e);
    const BlockDesc bd = a.blocks[b];
    if (__ldcg(queued + b) == stamp) continue;  // queued: its check writes the times
    for (int k = lane; k < bd.nowned; k += 32) Tdst[bd.vbase + k] = __ldcg(Tsrc + bd.vbase + k);
  }
}

// iteration i's times as it finds them, and as it leaves them
__device__ __forceinline__ const float* buf_in(const DevArgs& a, int i) { return (i & 1) ? a.Tb : a.Ta; }
__device__ __forceinline__ float* buf_out(const DevArgs& a, int i) { return (i & 1) ? a.Ta : a.Tb; }

// The times behind an iteration into row `row` of the history; the reference's result of
// blocks that no iteration has swept is 0 (stamp: the present iteration's, whose first
// sweeps of a block do not count yet).
__device__ __forceinline__ void snapshot3d(const DevArgs& a, int row, int stamp, const float* T) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nv; i += gridDim.x * blockDim.x) {
    const int first = __ldcg(a.conv + a.vblock[i]);
    a.hist[(size_t)row * a.nv + i] = (first && 0x7fffffff - first < stamp) ? __ldcg(T + i) : 0.0f;
  }
}

struct Loop3 {
  int iter, iters;          // loop passes, and those that the reference counts
  int nact, ncand, nconv;   // this pass's active blocks, check candidates and copies
  int snap;                 // history row of the last pass's times, or -1
  int state;                // a single solve's: 0 running, 2 at its cap with checks left
  int go;
};

// A pass ends when its last visits do, so its order matters: a sweep takes about 25,000
// cycles, a check 7,000, and one check in five goes on to a sweep.  So the check candidates
// come first, the sweeps, all alike, fill the CTAs that they leave, and an item is claimed
// only when its CTA is free.  (65^3 cube: mean visits per CTA and pass 37,000 cycles, mean
// wait at the barrier 37,700 with the sweeps first while they are fewer than the CTAs and
// the next item claimed during a visit, which hides its chain of four loads but holds it;
// solve 3.14 -> 2.80 ms, 41^3 1.82 -> 1.68, 97^3 7.53 -> 7.28.)

// One item of a pass: a block, whether it is a check candidate (flags 1), which of its
// memos are this solve's (2 check, 4 sweep), whether its instance does not run (16), and
// if so whether it is at its cap (32: its checks still run).
struct Item3 {
  int b, flags;
  BlockDesc bd;
};
// The CTA's next item (b = -1: none), by one thread: the CTA's index first, then from the
// counter.  A candidate that the last iteration left unconverged stands in the active list
// (and may have been swept from there in this one by now): passed over.
__device__ __forceinline__ void next_item(const DevArgs& a, const Start3& st, const volatile Loop3& v, bool first,
                                          volatile Item3& o) {
  const int iter = v.iter, count = v.nact + v.ncand, G = (int)gridDim.x;
  for (;; first = false) {
    const int i = first ? (int)blockIdx.x : count <= G ? count : G + atomicAdd(&st.turn[iter % 3].work, 1);
    if (i >= count) {
      o.b = -1;
      return;
    }
    const int ncand = v.ncand;
    const bool chk = i < ncand;
    const int b = __ldcg(chk ? a.cand + (size_t)((iter + 1) & 1) * a.nb + i : act_list(a, iter) + i - ncand);
    const BlockDesc bd = a.blocks[b];
    const int sa = __ldcg(a.stampA + b), valid = __ldcg(st.mvalid + b);
    const int ist = a.ninst == 1 ? v.state : __ldcg(a.inst_done + a.blk_inst[b]);
    if (chk && sa >= iter) continue;
    o.flags = (chk ? 1 : 0) | (valid << 1) | (ist ? 16 : 0) | (ist == 2 ? 32 : 0);
    o.bd.slot_begin = bd.slot_begin;
    o.bd.nslots = bd.nslots;
    o.bd.nslots_pad = bd.nslots_pad;
    o.bd.vbase = bd.vbase;
    o.bd.nowned = bd.nowned;
    o.bd.halo_begin = bd.halo_begin;
    o.bd.nhalo = bd.nhalo;
    o.b = b;
    return;
  }
}

template <int kRegs>
__global__ void __maxnreg__(kRegs) k_loop3d(const __grid_constant__ DevArgs a,
                                                                 const __grid_constant__ Start3 st) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int s_flag;
  __shared__ volatile Item3 s_it[2];
  __shared__ int s_n[2];
  __shared__ volatile int s_moved;
  __shared__ PassSum s_swept, s_checked, s_both;  // s_both: sweeps behind a check
  __shared__ VisitSum s_sum[3];                   // the same over the solve
  const SmemV s = carve_visit3d<false>(sm, a);
  GridBar* const g = &a.ctl->bar;
  const int tid = threadIdx.x, lane = tid & 31, NT = blockDim.x;
  const int G = gridDim.x, gtid = blockIdx.x * NT + tid, gn = G * NT;
  const bool single = a.ninst == 1;
  unsigned number = 0;
  auto sync_grid = [&](auto close, bool flat) -> bool {
    ++number;
    __syncthreads();
    if (tid == 0) s_flag = grid_arrive(&g->count, number * (unsigned)G) ? 2 : 1;
    if (flat) {
      if (tid == 0) s_flag = grid_wait(g, &g->count, number * (unsigned)G) ? 1 : 0;
      __syncthreads();
      return s_flag != 0;
    }
    __syncthreads();
    if (s_flag == 2) {
      close();
      __syncthreads();
      if (tid == 0) grid_release(st.flags, number);
      return true;
    }
    if (tid == 0 && !grid_wait(g, &st.flags[blockIdx.x % kGridFlags].go, number)) s_flag = 0;
    __syncthreads();
    return s_flag != 0;
  };
  auto nothing = [] {};
  const bool flat = G <= kFlatList;
  const int cap0 = st.maxit[0];
  // ---- initial state ----
  if (tid == 0) mbar_init(&bar, 1);
  if (tid < 2) s_n[tid] = 0;
  if (tid == 0) {
    s_swept.clear();
    s_checked.clear();
    s_both.clear();
    for (VisitSum& x : s_sum) x.clear();
  }
  for (int i = gtid; i < a.nv; i += gn) a.Ta[i] = a.Tb[i] = kLarge3DDev;
  for (int b = gtid; b < a.nb; b += gn) {
    a.stampA[b] = st.queued[0][b] = st.queued[1][b] = 0;
    a.conv[b] = 0;  // the first iteration that swept the block, as 0x7fffffff - (iteration + 1)
    a.visited[b] = 0;
    st.mvalid[b] = 0;
  }
  for (int i = gtid; i < a.ninst; i += gn) {
    a.inst_done[i] = st.done[i];
    const_cast<int*>(a.inst_maxit)[i] = st.maxit[i];
    a.inst_iters[i] = 0;
    a.inst_nnext[i] = 0;
    a.inst_fail[i] = 0;
    a.inst_swept[i] = 0;
    a.inst_ncand[i] = 0;
  }
  if (!sync_grid(nothing, flat)) return;
  for (int i = gtid; i < st.nseeds; i += gn) a.Ta[st.seeds[i]] = a.Tb[st.seeds[i]] = 0.0f;
  for (int i = gtid; i < st.nact; i += gn) a.list0[i] = st.act[i];
  if (!sync_grid(nothing, flat)) return;
  // The loop's state stands in shared memory: it is uniform and read a few times per
  // visit, while the visits' own values fill the registers (held there, it cost 260 bytes
  // of spills and a quarter of the speed).
  __shared__ volatile Loop3 v;
  if (tid == 0) {
    v.iter = v.iters = v.ncand = v.nconv = v.state = 0;
    v.nact = st.nact;
    v.snap = -1;
    v.go = st.nact > 0 && a.ctl->max_iters > 0;
  }
  __syncthreads();
  unsigned parity = 0;
  while (v.go) {
    if (gtid == 0) {
      Turn3* c = st.turn + (v.iter + 1) % 3;
      c->next = c->cand = c->conv = c->work = c->add = 0;
      if (a.ktime && v.iter < a.ktime_cap) a.ktime[kKStride * v.iter] = ~global_ns();
    }
    if (tid == NT - 32) next_item(a, st, v, true, s_it[0]);
    __syncthreads();
    for (int cur = 0; s_it[cur].b >= 0; cur ^= 1) {
      const volatile Item3& it = s_it[cur];
      const bool chk = (it.flags & 1) != 0, run = (it.flags & 16) == 0;  // run: the instance runs
      bool sweep = false, kept = !run && !(chk && (it.flags & 32));
      if (!kept) {
        BlockDesc bd;
        bd.slot_begin = it.bd.slot_begin;
        bd.nslots = it.bd.nslots;
        bd.nslots_pad = it.bd.nslots_pad;
        bd.vbase = it.bd.vbase;
        bd.nowned = it.bd.nowned;
        bd.halo_begin = it.bd.halo_begin;
        bd.nhalo = it.bd.nhalo;
        const bool have = (it.flags & (chk ? 2 : 4)) != 0;
        if (!load_visit3d(a, bd, s, &bar, parity, buf_in(a, v.iter), have ? (chk ? a.chk_memo : a.fim_memo) : nullptr)) {
          if (tid == 0) atomicOr(&a.ctl->error, kErrWait);
          (void)mbar_wait(&bar, parity ^ 1u);
        } else {
          if (!have)
            for (int j = tid; j < bd.nslots; j += NT)
              reinterpret_cast<uint4*>(s.h0)[j] = make_uint4(~0u, ~0u, ~0u, ~0u);
          __syncthreads();
          sweep = run;
          if (chk) {
            const bool moved = check_visit3d(a, bd, s, s_n, &s_moved);
            sweep = sweep && moved;
            if (tid == 0 && !moved) st.mvalid[it.b] = ((it.flags >> 1) & 3) | 1;
            if (!sweep)  // its times stand in the next buffer too
              for (int k = tid; k < it.bd.nowned; k += NT) buf_out(a, v.iter)[it.bd.vbase + k] = s.vt[k];
          }
          if (sweep) sweep_visit3d(a, bd, s, s_n, chk, (it.flags & 4) != 0);
        }
        if (chk && tid == 0) {
          s_checked.add(it.bd.nslots, it.bd.nhalo, it.bd.nowned);
          count_visit(a, v.iter - 1, 1, it.bd.nslots, it.bd.nhalo, it.bd.nowned);
          if (sweep) atomicAdd(&st.turn[v.iter % 3].add, 1);
        }
      } else {
        for (int k = tid; k < it.bd.nowned; k += NT)
          buf_out(a, v.iter)[it.bd.vbase + k] = __ldcg(buf_in(a, v.iter) + it.bd.vbase + k);
      }
      if (sweep) {
        const int nown = it.bd.nowned;
        float* const out = buf_out(a, v.iter) + it.bd.vbase;
        int myconv = 1;
        for (int k = tid; k < nown; k += NT) {
          const float ov = __int_as_float(s.v1[k]), nv = __int_as_float(s.v2[k]);
          float res = ov - nv;
          if (res < 0.0f) res = -res;
          myconv &= (res <= kEps3DLe) ? 1 : 0;
          out[k] = nv;
        }
        // the tail is the work of warps that have little to do in the next block's load
        const int allc = __syncthreads_and(myconv);
        const int b = it.b, iter = v.iter, stamp = iter + 1;
        Turn3* const now = st.turn + iter % 3;
        if (tid == NT - 96) {
          st.mvalid[b] = ((it.flags >> 1) & 3) | 2;
          a.visited[b] = 1;
          atomicMax(&a.conv[b], 0x7fffffff - stamp);
          if (!allc) {
            a.stampA[b] = stamp;
            next_list(a, iter)[atomicAdd(&now->next, 1)] = b;
          } else {
            st.conv[(size_t)(iter & 1) * a.nb + atomicAdd(&now->conv, 1)] = b;
          }
          if (!single) {
            atomicAdd(&a.inst_swept[a.blk_inst[b]], 1);
            if (!allc) atomicAdd(&a.inst_nnext[a.blk_inst[b]], 1);
          }
          s_swept.add(it.bd.nslots, it.bd.nhalo, nown);
          count_visit(a, iter, 0, it.bd.nslots, it.bd.nhalo, nown);
          if (chk) {  // streamed once, with the check
            s_both.add(it.bd.nslots, it.bd.nhalo, nown);
            count_visit(a, iter, 2, it.bd.nslots, it.bd.nhalo, nown);
          }
        }
        if (allc && tid >= NT - 64 && tid < NT - 32) {  // its neighbours are checked in the next iteration
          const int e0 = a.nbr_off[b], e1 = a.nbr_off[b + 1];
          for (int e = e0; e < e1; e += 32) {
            const int nb = (e + lane < e1) ? a.nbr[e + lane] : -1;
            bool q = false;
            if (nb >= 0) {
              const int sa = __ldcg(a.stampA + nb);
              const int old = atomicExch(&st.queued[iter & 1][nb], stamp);
              q = sa != stamp && old != stamp;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, q);
            if (bal) {
              int pos = 0;
              if (lane == 0) pos = atomicAdd(&now->cand, __popc(bal));
              pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(bal & ((1u << lane) - 1u));
              if (q) {
                a.cand[(size_t)(iter & 1) * a.nb + pos] = nb;
                if (!single) atomicAdd(&a.inst_ncand[a.blk_inst[b]], 1);
              }
            }
          }
        }
      }
      if (tid == NT - 32) next_item(a, st, v, false, s_it[cur ^ 1]);
      __syncthreads();
    }
    copy_settled(a, st.conv + (size_t)((v.iter + 1) & 1) * a.nb, v.nconv, st.queued[(v.iter + 1) & 1], v.iter,
                 buf_in(a, v.iter), buf_out(a, v.iter));
    if (v.snap >= 0 && v.snap < a.hist_cap) snapshot3d(a, v.snap, v.iter + 1, buf_in(a, v.iter));
    if (tid == 0 && v.iter % kTakeEvery == kTakeEvery - 1) {
      take(s_sum[0], s_swept, false);
      take(s_sum[1], s_checked, false);
      take(s_sum[2], s_both, false);
    }
    // ---- close ----
    if (!sync_grid([&] {
          if (!single) finish_loop3d(a, v.iter);
        }, single && flat))
      return;
    if (tid == 0) {
      // the memos written in the iterations so far, before the bulk copies that read them
      asm volatile("fence.proxy.async;" ::: "memory");
      const int iter = v.iter;
      const Turn3* now = st.turn + iter % 3;
      const int nn = __ldcg(&now->next), nc = __ldcg(&now->cand), add = __ldcg(&now->add);
      const int swept = v.nact + add;
      v.nconv = __ldcg(&now->conv);
      v.snap = -1;
      if (!single) {
        v.go = __ldcg(&a.ctl->stop) == 0;
      } else if (v.state == 2 || swept == 0) {
        v.go = 0;  // (checks that activated nothing: not one of the reference's iterations)
        if (gtid == 0) a.ctl->idle_iters = 1;
      } else {
        v.snap = v.iters;
        const int iters = v.iters + 1;
        v.iters = iters;
        if (nn + nc == 0) v.go = 0;
        else if (iters >= cap0) {
          v.go = nc > 0;
          v.state = 2;
        }
      }
      v.nact = nn;
      v.ncand = nc;
      v.iter = iter + 1;
      if (gtid == 0 && a.ktime && iter < a.ktime_cap) a.ktime[kKStride * iter + 1] = global_ns();
    }
    __syncthreads();
  }
  const int iter = v.iter;
  const float* Tcur = (iter & 1) ? a.Tb : a.Ta;
  if (v.snap >= 0 && v.snap < a.hist_cap) snapshot3d(a, v.snap, 0x7fffffff, Tcur);
  if (iter & 1)
    for (int i = gtid; i < a.nv; i += gn) a.Ta[i] = __ldcg(a.Tb + i);
  __syncthreads();
  if (tid == 0) {
    Ctl* c = a.ctl;
    if (single && blockIdx.x == 0) {
      c->iter = iter;
      a.inst_iters[0] = v.iters;
    }
    take(s_sum[0], s_swept, true);
    take(s_sum[1], s_checked, true);
    take(s_sum[2], s_both, true);
    const VisitSum f = s_sum[0], h = s_sum[1], x = s_sum[2];
    if (f.visits) {
      atomicAdd(&c->fim_visits, f.visits);
      atomicAdd(&c->fim_slots, f.slots);
      atomicAdd(&c->fim_halo, f.halo);
      atomicAdd(&c->fim_owned, f.owned);
    }
    if (h.visits) atomicAdd(&c->chk_visits, h.visits);
    if (f.visits + h.visits) {  // a block swept behind its check was streamed once
      atomicAdd(&c->updates, 2ull * f.owned + h.owned);
      atomicAdd(&c->slot_visits, f.slots + h.slots - x.slots);
      atomicAdd(&c->halo_visits, f.halo + h.halo - x.halo);
      atomicAdd(&c->owned_visits, f.owned + h.owned - x.owned);
    }
  }
}
