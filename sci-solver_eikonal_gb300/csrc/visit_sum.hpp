// visit_sum.hpp — what one CTA of a loop kernel adds up over a whole solve.
#pragma once

#ifdef __CUDACC__
#define EIK_HD __host__ __device__ __forceinline__
#else
#define EIK_HD inline
#endif

namespace eikgb {

// Block visits and the element slots, halo and owned vertices that they streamed.  In
// shared memory, added to by one thread; adding to the solve's totals at every visit met
// thousands of times at the same addresses.
template <class Word>
struct VisitCounts {
  Word visits, slots, halo, owned;
  EIK_HD void clear() { visits = slots = halo = owned = 0; }
  EIK_HD void add(int nslots, int nhalo, int nowned) {
    visits += 1;
    slots += (unsigned)nslots;
    halo += (unsigned)nhalo;
    owned += (unsigned)nowned;
  }
};

// Of a whole solve, in 64 bits as its totals are: at 3300 slots a block, 1.3 million visits
// pass 2^32.
using VisitSum = VisitCounts<unsigned long long>;

// Of some passes of the 3D loop, where 64-bit words at every visit cost 0.5% of a solve and
// a look at them after every pass as much.  Every kTakeEvery passes take() empties those
// that hold 2^28 slots into the solve's.  What is then left suffices for the passes up to
// the next: halo and owned vertices are at most four times the slots, and a CTA's sixteen
// passes would need 15,000 visits of 3300 slots each to add 3/4 of 2^30.
using PassSum = VisitCounts<unsigned>;
constexpr int kTakeEvery = 16;
EIK_HD void take(VisitSum& sum, PassSum& pass, bool all) {
  if (!all && (pass.slots >> 28) == 0u) return;
  sum.visits += pass.visits;
  sum.slots += pass.slots;
  sum.halo += pass.halo;
  sum.owned += pass.owned;
  pass.clear();
}

}  // namespace eikgb
