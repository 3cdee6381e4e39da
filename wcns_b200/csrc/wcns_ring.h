// wcns_ring.h -- the protocol of the rings between the CTAs of the wide sweeps
// (k_sweep_wide.cu) in counts of planes, without the kernel, so that it can be
// checked on the host.
//
// Reader.  Two warps take turns, warp T & 1 brings plane T's terms in between the
// CTA's barriers of planes T - 2 and T, which are the ones it joins; the terms of
// plane T are ring entry sf, the next plane's entry sf + 1, the other warp's.
// Writer.  Before it writes entries sf .. sf + RING_CHECK - 1, sf a multiple of
// RING_CHECK, it waits until the reader has published ring_room(sf, ringn) entries:
// those it is about to overwrite.
#pragma once
#ifdef __CUDACC__
#define WCNS_HD __host__ __device__ __forceinline__
#else
#define WCNS_HD inline
#endif

namespace wcns {

constexpr int RING_CHECK = 8;  // planes between two looks at the ring's reader

// Entries that have been read for certain once a ring warp holds entry sf: its own up
// to sf, and the other warp's up to sf - 3, which that one had before the barrier two
// planes back.  Entry sf - 1 may still be on its way to the other warp, so the count
// ends before it.
WCNS_HD constexpr int ring_read(int sf) { return sf - 1; }
// whether the reader publishes that count
WCNS_HD constexpr bool ring_publishes(int sf) { return (ring_read(sf) & (RING_CHECK - 1)) == 0; }
// entries that must have been read before entries sf .. sf + RING_CHECK - 1 are written
WCNS_HD constexpr int ring_room(int sf, int ringn) { return sf + RING_CHECK - ringn; }

}  // namespace wcns
