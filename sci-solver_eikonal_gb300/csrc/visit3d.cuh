// visit3d.cuh — one 3D block visit of the reference's two sweeps (FIMCuda,
// core3d/cuda/CUDA_kernels.cu:383-489) and one neighbour check (run_check_neghbor,
// :493-602) over a block staged in shared memory (included by fim_device.cu inside its
// unnamed namespace).
//
// A visit lists the apex updates that can change something and runs them 32 to a warp.
// What is left out is exact:
//   * an apex whose three other corners are all unreached, or which is at or below the
//     plane-distance bound of its update (plane_skip), keeps its time;
//   * an owned apex whose three other inputs equal, as bits, those of the last sweep of
//     the block's previous visit repeats an update its time has absorbed (sweep memo);
//   * in the second sweep only owned apexes count, and one none of whose other corners
//     changed repeats its first-sweep update;
//   * the per-slot copies of other blocks' corners are dropped after the visit, so a
//     copy's first-sweep update matters only as an input of an owned apex's second-sweep
//     update.  It is put off: the first sweep records a lower bound of the copy's new
//     value (the plane bound of its update); in the second sweep an apex that this bound
//     already settles needs no copy, and only the copies of the other slots are updated.
//     Two thirds of the first sweep's updates were copies; on a 41^3 cube 68 of 357 per
//     visit are left, and a visit runs 360 updates instead of 650.
// A check runs the first sweep's owned updates; they go into the next times, so that a
// block which moves is swept from there: its first sweep adds only the slots that the
// check memo had settled.
//
// What bounds it: instruction issue when the GPU is full (an update is about 900
// instructions, a listing pass 100-150 per slot), the latency of these chains when it is
// not.  One body serves all four apex kinds (the lanes of a warp update different ones):
// a list per kind left a third of the lanes idle and cost four counters.
struct SmemV {
  float* coef;            // 6 runs
  uint2* lv;              // corner ids
  uint2* hs;              // the apexes' distance bounds
  float4* h0;             // per slot: the visit's memos, then the copies' bounds or values
  float* vt;              // owned times, then halo times
  int* v1;                // owned: bits of the times after the first sweep
  int* v2;                // ... after the second
  unsigned short* items;  // 4 slot + apex, at most 4 per slot; precision mode: the FP64 updates from the end
  unsigned short* defer;  // slots whose copies the second sweep needs
  unsigned char* fl;      // per slot: copies of unknown value (bits 0-3), settled by the check memo (bit 7)
  int* sf;                // precision mode: per slot the FP64 products of its tet, or -1
};
// Precision mode (kPrec): the updates of flagged tets, and in the polish of all, run in
// FP64.  They are listed apart, so that every FP64 instruction of a warp works for all of
// its lanes: the FP64 unit takes 16 cycles for a warp whatever the number of lanes in
// use, and it is what bounds the mode.  A 25^3 solve with slivers took 39.5 ms with an
// update per slot, 13.0 ms with a list per apex kind, 11.2 ms with one list and body for
// all kinds, split over idle warps like the FP32 updates.
__host__ __device__ inline size_t visit3d_offsets(int np, int max_local, int max_owned, bool prec, size_t off[11]) {
  size_t o = 0;
  const size_t n = (size_t)np, bytes[11] = {24 * n, 8 * n, 8 * n, 16 * n, 4 * (size_t)max_local, 4 * (size_t)max_owned,
                                            4 * (size_t)max_owned, 8 * n, 2 * n, n, prec ? 4 * n : 0};
  for (int i = 0; i < 11; ++i) {
    off[i] = o;
    o += (bytes[i] + 15) & ~(size_t)15;
  }
  return o;
}
__host__ __device__ inline size_t smem_bytes_visit3d(int np, int max_local, int max_owned, bool prec) {
  size_t off[11];
  return visit3d_offsets(np, max_local, max_owned, prec, off);
}
template <bool kPrec>
__device__ __forceinline__ SmemV carve_visit3d(unsigned char* sm, const DevArgs& a) {
  size_t off[11];
  visit3d_offsets(a.max_slots_pad, a.max_local, a.max_owned, kPrec, off);
  SmemV s;
  s.coef = reinterpret_cast<float*>(sm + off[0]);
  s.lv = reinterpret_cast<uint2*>(sm + off[1]);
  s.hs = reinterpret_cast<uint2*>(sm + off[2]);
  s.h0 = reinterpret_cast<float4*>(sm + off[3]);
  s.vt = reinterpret_cast<float*>(sm + off[4]);
  s.v1 = reinterpret_cast<int*>(sm + off[5]);
  s.v2 = reinterpret_cast<int*>(sm + off[6]);
  s.items = reinterpret_cast<unsigned short*>(sm + off[7]);
  s.defer = reinterpret_cast<unsigned short*>(sm + off[8]);
  s.fl = sm + off[9];
  s.sf = reinterpret_cast<int*>(sm + off[10]);
  return s;
}

// What a visit of precision mode needs beyond its block: whether every update runs in
// FP64, and the polish's rule for a settled vertex.
struct PrecMode {
  int f64_all, polish;
};
// Precision mode, behind load_visit3d and a CTA barrier: the slots' FP64 products and the
// bounds that belong to their updates.
__device__ __forceinline__ void load_prec3d(const DevArgs& a, const BlockDesc& bd, const SmemV& s, PrecMode pm) {
  for (int j = threadIdx.x; j < bd.nslots; j += blockDim.x) {
    const int f = a.slot_f64[bd.slot_begin + j];
    s.sf[j] = f;
    if (f >= 0) s.hs[j] = a.hs64[f];
    else if (pm.f64_all) s.hs[j] = a.hsu64[bd.slot_begin + j];
  }
}

// Loads block bd: the bulk copies of its coefficients, corner ids, bounds and `memo`
// entries (into h0), its owned and halo times from Tsrc.  Returns false on a timeout.
__device__ __forceinline__ bool load_visit3d(const DevArgs& a, const BlockDesc& bd, const SmemV& s,
                                             unsigned long long* bar, unsigned& parity, const float* Tsrc,
                                             const uint4* memo) {
  const int tid = threadIdx.x, NT = blockDim.x;
  if (tid == 0) {
    fence_proxy_async();
    const unsigned n = (unsigned)bd.nslots_pad;
    mbar_expect_tx(bar, n * (24u + 8u + 8u + (memo ? 16u : 0u)));
    if (n > 0) {
      bulk_g2s(s.lv, a.lv + bd.slot_begin, 8u * n, bar);
      if (memo) bulk_g2s(s.h0, memo + bd.slot_begin, 16u * n, bar);
      bulk_g2s(s.hs, a.hsb + bd.slot_begin, 8u * n, bar);
      bulk_g2s(s.coef, a.coef + 6 * (size_t)bd.slot_begin, 24u * n, bar);
    }
  }
  for (int k = tid; k < bd.nowned; k += NT) {
    const float v = __ldcg(Tsrc + bd.vbase + k);
    s.vt[k] = v;
    s.v1[k] = __float_as_int(v);  // times are never negative: their bits order as integers do
  }
  for (int k = tid; k < bd.nhalo; k += NT) s.vt[bd.nowned + k] = __ldcg(Tsrc + a.halo[bd.halo_begin + k]);
  const bool ok = mbar_wait(bar, parity);
  parity ^= 1u;
  return ok;
}

__device__ __forceinline__ void slot_ids(uint2 l, int id[4]) {
  id[0] = (int)(l.x & 0xffffu);
  id[1] = (int)(l.x >> 16);
  id[2] = (int)(l.y & 0xffffu);
  id[3] = (int)(l.y >> 16);
}
__device__ __forceinline__ void slot_bounds(uint2 w, float hs[4]) {
  hs[0] = half_bits_value(w.x);
  hs[1] = half_bits_value(w.x >> 16);
  hs[2] = half_bits_value(w.y);
  hs[3] = half_bits_value(w.y >> 16);
}
// the least of the three others, per corner
__device__ __forceinline__ void others_min(const float T[4], float m[4]) {
  const float p = fminf(T[0], T[1]), q = fminf(T[2], T[3]);
  m[0] = fminf(T[1], q);
  m[1] = fminf(T[0], q);
  m[2] = fminf(p, T[3]);
  m[3] = fminf(p, T[2]);
}
// bits of corners whose values agree
__device__ __forceinline__ unsigned same_bits(const float T[4], uint4 m) {
  return (__float_as_uint(T[0]) == m.x ? 1u : 0u) | (__float_as_uint(T[1]) == m.y ? 2u : 0u) |
         (__float_as_uint(T[2]) == m.z ? 4u : 0u) | (__float_as_uint(T[3]) == m.w ? 8u : 0u);
}
// Appends slot j's apexes of `need` to the item list, which grows from `items` by kStep
// entries at a time; all lanes of a warp together.
template <int kStep = 1>
__device__ __forceinline__ void append_items(unsigned short* items, int* count, unsigned need, int j) {
  const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  unsigned bal[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) bal[k] = __ballot_sync(0xffffffffu, (need >> k) & 1u);
  const int n0 = __popc(bal[0]), n1 = n0 + __popc(bal[1]), n2 = n1 + __popc(bal[2]), n = n2 + __popc(bal[3]);
  if (n == 0) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(count, n);
  base = __shfl_sync(0xffffffffu, base, 0);
  if (need & 1u) items[kStep * (base + __popc(bal[0] & below))] = (unsigned short)(4 * j);
  if (need & 2u) items[kStep * (base + n0 + __popc(bal[1] & below))] = (unsigned short)(4 * j + 1);
  if (need & 4u) items[kStep * (base + n1 + __popc(bal[2] & below))] = (unsigned short)(4 * j + 2);
  if (need & 8u) items[kStep * (base + n2 + __popc(bal[3] & below))] = (unsigned short)(4 * j + 3);
}
template <bool kPrec>
__device__ __forceinline__ void append_updates(const DevArgs& a, const SmemV& s, int* s_n, PrecMode pm, unsigned need,
                                               int j) {
  if constexpr (kPrec) {
    // an update is in one of the lists, so the two ends of the array never meet
    const bool wide = need && (pm.f64_all || s.sf[j] >= 0);
    append_items(s.items, s_n, wide ? 0u : need, j);
    append_items<-1>(s.items + 4 * a.max_slots_pad - 1, s_n + 2, wide ? need : 0u, j);
  } else {
    append_items(s.items, s_n, need, j);
  }
}
// counters of a visit: items, deferred slots, FP64 items
template <bool kPrec>
__device__ __forceinline__ void clear_updates(int* s_n) {
  if (threadIdx.x == 0) s_n[0] = 0;
  if (kPrec && threadIdx.x == 0) s_n[2] = 0;
}

// Runs the listed updates.  kPhase 0: the first sweep's owned apexes (into v1; *moved set
// when one falls by EPS or more); 1: second-sweep owned apexes of slots whose copies are
// known to keep their values (into v2), and first-sweep copies (into h0); 2: second-sweep
// owned apexes of the slots whose copies phase 1 updated (into v2).
template <int kPhase, bool kPrec>
__device__ __forceinline__ void run_items(const DevArgs& a, const BlockDesc& bd, const SmemV& s, const int* s_n,
                                          volatile int* moved, PrecMode pm) {
  const int nown = bd.nowned, pitch = bd.nslots_pad, lane = threadIdx.x & 31;
  const int count = s_n[0], n32 = (count + 31) >> 5;
  const int count64 = kPrec ? s_n[2] : 0, n64 = (count64 + 31) >> 5;
  // Few chunks leave warps idle while each runs the long chain of a whole update: its
  // parts then run side by side in two or four warps (their least is the update).
  const int nw = blockDim.x >> 5;
  const int split = (n64 + n32) * 4 <= nw ? 2 : (n64 + n32) * 2 <= nw ? 1 : 0;  // log2 of the parts
  for (int c = threadIdx.x >> 5; c < (n64 + n32) << split; c += nw) {
    const bool wide = kPrec && (c >> split) < n64;
    const int r = (((c >> split) - (wide ? 0 : n64)) << 5) + lane;
    if (r >= (wide ? count64 : count)) continue;
    const int e = s.items[wide ? 4 * a.max_slots_pad - 1 - r : r], j = e >> 2, k = e & 3;
    const int part = c & ((1 << split) - 1);
    const unsigned parts = split == 0 ? kAllParts : split == 1 ? (part ? 24u : 7u)
                                                  : (part == 0 ? 8u : part == 1 ? 16u : part == 2 ? 4u : 3u);
    int id[4];
    slot_ids(s.lv[j], id);
    const int idk = k < 2 ? (k == 0 ? id[0] : id[1]) : (k == 2 ? id[2] : id[3]);
    const bool ownk = kPhase != 1 || idk < nown;
    float T[4];
    if constexpr (kPhase == 2) {
      const float4 h = s.h0[j];
      const float hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) T[q] = id[q] < nown ? __int_as_float(s.v1[id[q]]) : hv[q];
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        T[q] = (kPhase == 1 && ownk && id[q] < nown) ? __int_as_float(s.v1[id[q]]) : s.vt[id[q]];
    }
    const float Tk = k < 2 ? (k == 0 ? T[0] : T[1]) : (k == 2 ? T[2] : T[3]);
    const float* cf = s.coef + j;
    float u;
    if (kPrec && wide) {
      const int f = s.sf[j];
      double g[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) g[q] = (f >= 0) ? a.coef64[6 * (size_t)f + q] : (double)cf[q * pitch];
      u = apex_update64(k, T, g, parts);
    } else {
      const TetGram g = tet_gram9(cf[0], cf[pitch], cf[2 * pitch], cf[3 * pitch], cf[4 * pitch], cf[5 * pitch]);
      u = apex_update(k, T, g, parts);
    }
    if (kPhase == 1 && !ownk) {
      // (its place holds the copy's present value)
      if (u < Tk) atomicMin(reinterpret_cast<int*>(s.h0 + j) + k, __float_as_int(u));
    } else if (u < Tk) {
      atomicMin(kPhase == 0 ? &s.v1[idk] : &s.v2[idk], __float_as_int(u));
      // (double)(old - candidate) >= 1e-5 in the reference's check
      if (kPhase == 0 && moved && !((Tk - u) <= settle_eps(Tk, kPrec ? pm.polish : 0))) *moved = 1;
    }
  }
}

// One check of a loaded block (its check memos in h0): whether it moves.  s_n: two
// counters, zero on entry and on return.  All threads; ends behind a CTA barrier.
template <bool kPrec = false>
__device__ __forceinline__ bool check_visit3d(const DevArgs& a, const BlockDesc& bd, const SmemV& s, int* s_n,
                                              volatile int* s_moved, PrecMode pm = PrecMode{0, 0}) {
  const int tid = threadIdx.x, NT = blockDim.x, ns = bd.nslots, nown = bd.nowned;
  if (tid == 0) *s_moved = 0;
  for (int j0 = 0; j0 < ns; j0 += NT) {
    const int j = j0 + tid;
    unsigned need = 0;
    if (j < ns) {
      int id[4];
      slot_ids(s.lv[j], id);
      float T[4], m[4], hs[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) T[q] = s.vt[id[q]];
      const uint4 R = reinterpret_cast<const uint4*>(s.h0)[j];
      const bool memo = same_bits(T, R) == 15u;
      s.fl[j] = memo ? 0x80u : 0u;
      if (!memo) {
        others_min(T, m);
        slot_bounds(s.hs[j], hs);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          need |= (id[k] < nown && m[k] < kLarge3DDev && !plane_skip(T[k], m[k], hs[k]) ? 1u : 0u) << k;
      }
    }
    append_updates<kPrec>(a, s, s_n, pm, need, j);
  }
  __syncthreads();
  run_items<0, kPrec>(a, bd, s, s_n, s_moved, pm);
  __syncthreads();
  const bool moved = *s_moved != 0;
  clear_updates<kPrec>(s_n);
  if (!moved)  // every slot's input times lowered no owned vertex by EPS
    for (int j = tid; j < ns; j += NT) {
      if (s.fl[j]) continue;
      int id[4];
      slot_ids(s.lv[j], id);
      a.chk_memo[bd.slot_begin + j] = make_uint4(__float_as_uint(s.vt[id[0]]), __float_as_uint(s.vt[id[1]]),
                                                 __float_as_uint(s.vt[id[2]]), __float_as_uint(s.vt[id[3]]));
    }
  __syncthreads();
  return moved;
}

// The two sweeps of a loaded block (its sweep memos in h0, or behind a check read from
// memory, where `memo` says they are of this solve): the final owned times in v2, those
// after the first sweep in v1, both behind a CTA barrier.  s_n: counters that are zero
// again only behind the caller's next barrier.
template <bool kPrec = false>
__device__ __forceinline__ void sweep_visit3d(const DevArgs& a, const BlockDesc& bd, const SmemV& s, int* s_n,
                                              bool checked, bool memo, PrecMode pm = PrecMode{0, 0}) {
  const int tid = threadIdx.x, NT = blockDim.x, ns = bd.nslots, nown = bd.nowned;
  // ---- first sweep: owned apexes; bounds of the copies ----
  for (int j0 = 0; j0 < ns; j0 += NT) {
    const int j = j0 + tid;
    unsigned need = 0;
    if (j < ns) {
      int id[4];
      slot_ids(s.lv[j], id);
      float T[4], m[4], hs[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) T[q] = s.vt[id[q]];
      others_min(T, m);
      slot_bounds(s.hs[j], hs);
      unsigned same = 0, live = 0, own = 0;
      if (!checked) same = same_bits(T, reinterpret_cast<const uint4*>(s.h0)[j]);
      else if (s.fl[j] && memo) same = same_bits(T, __ldcg(a.fim_memo + bd.slot_begin + j));
      float lo[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float bound = __fmul_rn(__fadd_rn(m[q], hs[q]), 0x1.ffffep-1f);  // as in plane_skip
        const bool run = m[q] < kLarge3DDev && !(T[q] <= bound);
        live |= (run ? 1u : 0u) << q;
        own |= (id[q] < nown ? 1u : 0u) << q;
        lo[q] = (run && id[q] >= nown) ? bound : T[q];
        need |= (run && id[q] < nown && (same | (1u << q)) != 15u ? 1u : 0u) << q;
      }
      // the check ran this slot's updates already, unless its memo had settled the slot
      if (checked && !s.fl[j]) need = 0;
      s.fl[j] = (unsigned char)(live & ~own);
      s.h0[j] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
    append_updates<kPrec>(a, s, s_n, pm, need, j);
  }
  __syncthreads();
  run_items<0, kPrec>(a, bd, s, s_n, nullptr, pm);
  __syncthreads();
  // ---- second sweep: owned apexes that the copies' bounds do not settle ----
  clear_updates<kPrec>(s_n);
  __syncthreads();
  for (int k = tid; k < nown; k += NT) s.v2[k] = s.v1[k];
  for (int j0 = 0; j0 < ns; j0 += NT) {
    const int j = j0 + tid;
    unsigned need = 0;
    bool put = false;
    if (j < ns) {
      int id[4];
      slot_ids(s.lv[j], id);
      const unsigned unk = s.fl[j];
      const float4 h = s.h0[j];
      const float lo[4] = {h.x, h.y, h.z, h.w};
      float T[4], m[4], hs[4];
      unsigned chg = unk, own = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool o = id[q] < nown;
        T[q] = o ? __int_as_float(s.v1[id[q]]) : lo[q];
        own |= (o ? 1u : 0u) << q;
        chg |= (T[q] != lo[q] ? 1u : 0u) << q;  // (an owned corner's lo is its first input)
      }
      others_min(T, m);
      slot_bounds(s.hs[j], hs);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        need |= (((own >> k) & 1u) && (chg & ~(1u << k)) && m[k] < kLarge3DDev && !plane_skip(T[k], m[k], hs[k])
                     ? 1u
                     : 0u)
                << k;
      if (unk && need) {
        need = unk;  // its copies first, from their present values
        put = true;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if ((unk >> q) & 1u) reinterpret_cast<float*>(s.h0 + j)[q] = s.vt[id[q]];
      } else if (a.fim_memo) {
        a.fim_memo[bd.slot_begin + j] = make_uint4(
            (unk & 1u) ? ~0u : __float_as_uint(T[0]), (unk & 2u) ? ~0u : __float_as_uint(T[1]),
            (unk & 4u) ? ~0u : __float_as_uint(T[2]), (unk & 8u) ? ~0u : __float_as_uint(T[3]));
      }
    }
    append_updates<kPrec>(a, s, s_n, pm, need, j);
    const unsigned bal = __ballot_sync(0xffffffffu, put);
    if (bal) {
      const unsigned lane = tid & 31u;
      int base = 0;
      if (lane == 0) base = atomicAdd(s_n + 1, __popc(bal));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (put) s.defer[base + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)j;
    }
  }
  __syncthreads();
  run_items<1, kPrec>(a, bd, s, s_n, nullptr, pm);
  __syncthreads();
  const int nd = s_n[1];
  clear_updates<kPrec>(s_n);
  if (nd > 0) {  // uniform across the CTA
    __syncthreads();
    for (int i0 = 0; i0 < nd; i0 += NT) {
      const int i = i0 + tid;
      const int j = i < nd ? s.defer[i] : 0;
      unsigned need = 0;
      if (i < nd) {
        int id[4];
        slot_ids(s.lv[j], id);
        const float4 h = s.h0[j];
        const float hv[4] = {h.x, h.y, h.z, h.w};
        float T[4], m[4], hs[4];
        unsigned chg = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          T[q] = id[q] < nown ? __int_as_float(s.v1[id[q]]) : hv[q];
          chg |= (T[q] != s.vt[id[q]] ? 1u : 0u) << q;
        }
        others_min(T, m);
        slot_bounds(s.hs[j], hs);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          need |= (id[k] < nown && (chg & ~(1u << k)) && m[k] < kLarge3DDev && !plane_skip(T[k], m[k], hs[k]) ? 1u
                                                                                                              : 0u)
                  << k;
        if (a.fim_memo)
          a.fim_memo[bd.slot_begin + j] = make_uint4(__float_as_uint(T[0]), __float_as_uint(T[1]),
                                                     __float_as_uint(T[2]), __float_as_uint(T[3]));
      }
      append_updates<kPrec>(a, s, s_n, pm, need, j);
    }
    __syncthreads();
    run_items<2, kPrec>(a, bd, s, s_n, nullptr, pm);
    __syncthreads();
    clear_updates<kPrec>(s_n);
    if (tid == 0) s_n[1] = 0;
  }
}
