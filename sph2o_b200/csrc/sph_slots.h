/*
 * The walk over two ranges of slots by byte offsets, as the candidate loops of
 * the neighbour search do it (for_stretches27). Plain C++: it compiles for the
 * host as well.
 */
#ifndef SPH2O_SLOTS_H
#define SPH2O_SLOTS_H

#ifdef __CUDACC__
#define SPH_HD __host__ __device__ __forceinline__
#else
#define SPH_HD inline
#endif

namespace sph {

/* Offsets of 16-byte slots in 32 bits reach slot 2^28 - 1. A fluid of about that
   many particles fills the GPU with its lists; a boundary has no lists and can be
   larger. The searches have a form with 64-bit offsets for them, which costs more
   instructions per candidate (list build of 1M particles 295 us against 263). The
   PCISPH solver and the allocation-free densities hold fewer particles always. */
constexpr unsigned kNarrowSlots = 1u << 28;
inline bool narrow_slots(unsigned nf, unsigned nb) { return nf <= kNarrowSlots && nb <= kNarrowSlots; }

/* Byte offsets of the slots s1, s1 + 1, ... s1 + n1 - 1 and then s2, s2 + 1, ...,
   from the k-th on. Load at `at`, then advance: a next() that returned the offset
   and advanced first made the one-lane search with densities 10 % slower (174k
   particles 88 -> 98 us). */
template <typename Off>
struct SlotWalk {
    Off at, end, second;

    SPH_HD SlotWalk(unsigned s1, unsigned n1, unsigned s2, unsigned k)
        : at((Off)(k < n1 ? s1 + k : s2 + (k - n1)) * (Off)16), end((Off)(s1 + n1) * (Off)16), second((Off)s2 * (Off)16)
    {
    }
    SPH_HD void advance()
    {
        at += (Off)16;
        if (at == end) at = second;
    }
};

} // namespace sph
#endif
