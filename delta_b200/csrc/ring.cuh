// The order of a ring of mbarriers: use number n (0, 1, ...) of ``slots`` barriers completes phase n / slots of barrier n % slots.
#pragma once
#ifdef __CUDACC__
#define DK_RING __host__ __device__ __forceinline__
#else
#define DK_RING inline
#endif

DK_RING int ring_slot(int n, int slots) { return n % slots; }
DK_RING unsigned ring_parity(int n, int slots) { return (unsigned)(n / slots) & 1u; }

// Waits for what may still be under way of ``asked`` uses: the last one of every slot (a slot's earlier ones were complete when it was used
// again).  wait(slot, parity) is bounded; the first one that gives up ends the rest.  A block calls it before it leaves whatever became of
// its other warps: a copy or a product that ends later would write into memory that is another block's by then.
template <typename Wait>
DK_RING bool ring_drain(int asked, int slots, Wait&& wait) {
  for (int n = asked > slots ? asked - slots : 0; n < asked; ++n)
    if (!wait(ring_slot(n, slots), ring_parity(n, slots))) return false;
  return true;
}
