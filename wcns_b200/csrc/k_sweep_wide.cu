// k_sweep_wide.cu -- GS_PR_Single (LHS.f90:1559-1613) as wide cooperative
// sweeps: lusgs_l (381-478), lusgs_u (480-577), gs_pr_l (1777-1866), gs_pr_u
// (1956-2046), one cooperative launch per sweep over all blocks of the
// context.
//
// Work split.  Each block's (j,k) columns are cut into chunks of whole rows
// (all k; all j where k is the longer); one CTA owns a chunk, one thread a column, and the CTA
// walks the block's hyperplanes p = i+j+k in sweep order, the thread
// meeting its column's cell of each plane.  A cell's lower (forward) or
// upper (backward) neighbours are on the previous plane, so a cell can be
// computed once the contributions A*dq of those neighbours are known.  After
// computing its new dq a cell pushes the three contributions to its
// successors (wcns_sweep.cuh):
//   along i -- the same thread's next plane: kept in registers;
//   along k -- another thread of the CTA: shared memory, double-buffered
//              by plane parity, so one CTA barrier per plane suffices;
//   along j -- the next thread of the chunk, or, at the chunk's edge, the
//              neighbouring chunk's CTA, through a ring of planes in global
//              memory (below).
// Every CTA of the launch is resident at once (cooperative launch), so a
// wait is only ever for a running CTA.
//
// Folding.  A column is busy for ni of a block's ni+nj+nk-2 planes.  Where
// the columns would not fit the CTAs, a CTA takes several chunks of a block
// (segments), G/nseg chunks apart: a warp works through its columns of the
// first, then of the next, and each later one runs `delay` planes behind the
// one before, just enough for every warp to be done with it.
//
// What bounds a plane.  The chain from the received terms to the sent ones is
// about 15 dependent FP64 operations (8.5 cycles each), a trip through shared
// memory and a barrier, 0.5 us in all with one warp per scheduler, where every
// instruction of the loop costs about three cycles.  Everything else is taken
// off that chain:
//   - a cell's words, 22 to 27 of them from DRAM or L2 (300 to 1000 cycles),
//     are copied by a helper warp with bulk copies into shared memory, up to
//     four planes ahead.  The words of a warp's 32 slots are one record of
//     16-byte pairs, so that a warp needs one or two copies per plane, and
//     warps without a cell in a plane copy nothing.  (Loads into registers a
//     plane ahead took 1.3 us per plane: their issue alone is 800 cycles, and
//     twice unrolled the loop misses the instruction cache.)
//   - the terms that come from another CTA are fetched by two more warps, which
//     take turns, so that each has two planes' time for the trip to L2 (0.35 us;
//     with one warp a plane took 0.85 us instead of 0.65).
//   - absent neighbours are a column of zeros, and what does not change along a
//     column is computed when the thread enters it.
// Per step, prep and four sweeps (before: coefficients of 40 words, loads at
// the top of the plane, counters with fences between CTAs): the 24-block SA
// channel 4.54 -> 2.10 ms, the 64-case batch 1.50 -> 0.55 ms, the 65x33x17
// vortex 0.68 (clustered) -> 0.35 ms.  A sweep of the channel takes 0.34 to
// 0.51 ms where its records need 0.14 at the copy bandwidth (27 words of 4.16 M
// cells): the planes of little activity at both ends, which folding adds to,
// and gs_pr_u's scattered stores.  Small blocks stay on the chain.
//
// Rings.  A contribution that crosses to another CTA travels as 16-byte
// units, the two halves of one value each with a 32-bit tag, written and read
// with relaxed accesses at GPU scope: a reader that finds the tag of the plane
// it wants has the value too, so neither side needs a fence or a flag.  Tags
// never repeat: every launch counts its planes from a base that the prep
// kernel moves on (A.epoch).  The ring holds A.ringn planes; every eighth
// plane the reader publishes how many entries both of its ring warps have read,
// and the writer checks it (wcns_ring.h; a power of two of at least the fold delay
// plus 32, so that the CTA that is furthest behind can always go on).  Every wait
// is bounded.
//
// Inputs are re-laid plane-major by k_wide_prep (once per step): per cell u,
// v, w, H, the nine metrics, the inviscid radii, coed (getcoed, 602-645),
// radii plus viscous radii, and rhs = dq (store_rhs_nb, 1592-1613).
// lusgs_l stores its dq for lusgs_u; lusgs_u stores the sum of the terms it
// received from its upper neighbours without their viscous part -- evaluated
// with their final dq they are the old side of gs_pr_l; gs_pr_l stores the sum
// of the terms it received from its lower neighbours less rhs, in rhs's place,
// for gs_pr_u.  gs_pr_u writes the result to the field layout.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "wcns_launch.h"
#include "wcns_ring.h"
#include "wcns_sweep.cuh"

namespace wcns {

namespace {

// A record holds the words of 32 consecutive slots: WIDE_PAIRS pairs of words,
// the pair q of slot n at ((n / 32) * WIDE_PAIRS + q) * 32 + n % 32.
// A sweep copies one or two runs of pairs (Cell).
enum : int {
    WP_UV = 0, WP_WH, WP_G01, WP_G23, WP_G45, WP_G67, WP_G8C,  // velocity, total enthalpy, metrics, coed
    WP_R01, WP_R23, WP_RAD2R4, WP_RAD01,  // rhs (from gs_pr_l on: lower terms - rhs), inviscid radii
    WP_RS01, WP_RS2D4, WP_D01, WP_D23,    // radii plus viscous radii, dq of lusgs_l
    WP_U01, WP_U23, WP_U4,                // upper terms (lusgs_u)
    WP_N
};
static_assert(WP_N == WIDE_PAIRS, "pairs per slot");
// the record's first pair of a slot that is lane `lane` of its 32
__device__ __forceinline__ long long rec_at(int slot, int lane, int pairs) {
    return (long long)(slot >> 5) * (pairs * 32) + lane;
}
constexpr int PREP_DS = 4;        // planes per column that neighbouring lanes of a prep kernel take
constexpr int WIDE_GAP = 4;       // idle planes between a thread's columns: a new column's copies start in the first
constexpr int SA_ST = 4;          // planes of the scalar sweeps' words in shared memory

// a unit: the two halves of a value, each with the tag
struct Unit { unsigned long long lo, hi; };

__device__ __forceinline__ void st_unit(Unit *p, double v, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};\n" ::"l"(p), "l"(t | (unsigned)__double2loint(v)),
                 "l"(t | (unsigned)__double2hiint(v))
                 : "memory");
}
__device__ __forceinline__ Unit ld_unit(const Unit *p) {
    Unit u;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n" : "=l"(u.lo), "=l"(u.hi) : "l"(p) : "memory");
    return u;
}
__device__ __forceinline__ bool has_tag(const Unit &u, unsigned tag) {
    return (unsigned)(u.lo >> 32) == tag && (unsigned)(u.hi >> 32) == tag;
}
// the terms of an entry
template <int N>
__device__ __forceinline__ void send(Unit *e, const double *v, unsigned tag) {
#pragma unroll
    for (int m = 0; m < N; m++) st_unit(e + m, v[m], tag);
}
// mbarriers of a warp's bulk copies (one per stage)
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *bar, unsigned bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred pp;\n\tmbarrier.try_wait.parity.shared::cta.b64 pp, [%1], %2;\n\tselp.u32 %0, 1, 0, pp;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// waits for the phase with the given parity; false after the time limit
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, bool late) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64(), limit = late ? (1LL << 21) : (1LL << 31);
    while (!mbar_try(bar, parity))
        if (clock64() - t0 > limit) return false;
    return true;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Rows run along the shorter of j and k, chunks along the longer.  Below, j and
// k are the index along the chunks and along the rows; `swap` tells that they
// are k and j of the block.
__host__ __device__ __forceinline__ bool row_is_j(const DevBlock &B) { return B.nk > B.nj; }

// What a CTA's threads need when they enter a column, in shared memory rather
// than in everybody's registers
struct CtaInfo {
    WideCta C;
    int ni, nj, nk;  // nj: along the chunks, nk: along the rows
    bool swap;
    long long id00, sj, sk;
    // per segment: its rings, and the j of the column at the incoming edge
    int lo[WIDE_MAX_FOLD], hi[WIDE_MAX_FOLD], jin[WIDE_MAX_FOLD];
    __device__ __forceinline__ void set(const WideCta &c, const DevBlock &B, const WideSeg *__restrict__ segs, bool fwd) {
        C = c;
        for (int g = 0; g < C.nseg; g++) {
            const WideSeg &S = segs[C.seg0 + g * C.segstep];
            lo[g] = S.bnd_lo;
            hi[g] = S.bnd_hi;
            jin[g] = fwd ? S.j0 + 1 : S.j0 + S.w;
        }
        ni = B.ni;
        swap = row_is_j(B);
        nj = swap ? B.nk : B.nj;
        nk = swap ? B.nj : B.nk;
        id00 = gidx(B, 0, 0, 0);
        sj = swap ? (long long)B.gx * B.gy : B.gx;
        sk = swap ? B.gx : (long long)B.gx * B.gy;
    }
};

// The steps in which a warp (columns t0..t0+31, j + k from jklo to jkhi; none:
// jkhi < 0) has cells in segment f, and its slots: slot0 +- step * S.cols.
template <bool FWD>
__device__ __forceinline__ void window(const CtaInfo &H, const WideSeg &S, int f, int t0, int jklo, int jkhi, int &first, int &last,
                                       int &slot0) {
    const int sdel = (FWD ? f : H.C.nsegmax - 1 - f) * H.C.delay, pmax = H.ni + H.nj + H.nk;
    first = FWD ? sdel + 1 + jklo - 3 : sdel + pmax - (H.ni + jkhi);
    last = FWD ? sdel + H.ni + jkhi - 3 : sdel + pmax - (1 + jklo);
    if (jkhi < 0) first = 1, last = 0;
    // plane index (0-based) at step s: s - sdel forward, pmax - 3 - (s - sdel) backward
    slot0 = S.pmoff + t0 + (FWD ? -sdel : pmax - 3 + sdel) * S.cols;
}

// A warp's walk through the segments of its CTA, and its threads' columns
// there.  At step s a thread is at i = s + ioff (forward) or ioff - s
// (backward) of its column; the warp is in the segment as long as any of its
// columns is, steps first..last.
template <bool FWD, int NC>  // NC: terms per ring entry
struct Walk {
    int ni, nseg;
    int f, ioff, sdel;     // segment, the column's offset, the segment's delay
    int first, last;       // steps in which the warp has cells
    int cols, slot0;       // slots per plane; the warp's first slot at step 0
    bool col, jin, jout;   // the segment has the column; it is at the incoming / outgoing chunk edge
    bool hasj, hask;       // it has a predecessor along j / k (among the columns lo..n+1-lo)
    bool inner;            // it is one of those columns itself
    long long id0;         // field index of the column's position 0
    Unit *rout;

    __device__ __forceinline__ void init(const CtaInfo &H, const WideArrays &A, const WideSeg *__restrict__ segs, int t, int lo) {
        ni = H.ni;
        nseg = H.C.nseg;
        enter(FWD ? 0 : nseg - 1, H, A, segs, t, lo);
    }
    __device__ __forceinline__ void enter(int seg, const CtaInfo &H, const WideArrays &A, const WideSeg *__restrict__ segs,
                                          int t, int lo) {
        f = seg;
        const WideSeg S = segs[H.C.seg0 + f * H.C.segstep];
        const int jj = t % H.C.w, k = t / H.C.w + 1, j = S.j0 + jj + 1;
        col = k <= H.nk && jj < S.w;
        inner = col && j >= lo && j <= H.nj + 1 - lo && k >= lo && k <= H.nk + 1 - lo;
        sdel = (FWD ? f : H.C.nsegmax - 1 - f) * H.C.delay;
        const int pmax = H.ni + H.nj + H.nk;
        ioff = (FWD ? 3 - sdel : pmax + sdel) - j - k;
        cols = S.cols;
        const int jklo = __reduce_min_sync(0xffffffffu, col ? j + k : 1 << 30), jkhi = __reduce_max_sync(0xffffffffu, col ? j + k : -1);
        window<FWD>(H, S, f, t & ~31, jklo, jkhi, first, last, slot0);
        id0 = H.id00 + j * H.sj + k * H.sk;
        hasj = FWD ? j > lo : j < H.nj + 1 - lo;
        hask = FWD ? k > lo : k < H.nk + 1 - lo;
        const int bi = FWD ? S.bnd_lo : S.bnd_hi, bo = FWD ? S.bnd_hi : S.bnd_lo;
        jin = col && bi >= 0 && jj == (FWD ? 0 : S.w - 1) && hasj;
        jout = col && bo >= 0 && jj == (FWD ? S.w - 1 : 0);
        rout = (Unit *)A.ring + (long long)(bo >= 0 ? bo : 0) * A.ringn * WIDE_UNITS * A.nkmax + (k - 1) * NC;
    }
    __device__ __forceinline__ int at(int s) const { return FWD ? s + ioff : ioff - s; }
    __device__ __forceinline__ int slot(int s) const { return FWD ? slot0 + s * cols : slot0 - s * cols; }
    __device__ __forceinline__ bool busy(int s) const { return s >= first && s <= last; }
    // done with the segment and another one to come
    __device__ __forceinline__ bool past(int s) const { return s > last && (FWD ? f + 1 < nseg : f > 0); }
};

// The copies of a warp's pairs, ST planes of them in shared memory, one
// mbarrier per stage.  R0/N0, R1/N1: the two runs of pairs that a plane takes
// from a record of `pairs` pairs.
template <int ST, int R0, int N0, int R1, int N1, int PAIRS>
struct Stager {
    static constexpr int NP = N0 + N1;
    double2 *place;  // this thread's pair 0 of stage 0
    unsigned long long *bar;
    int stride;      // pairs between stages
    unsigned phase;  // parity of every stage's next wait
    __device__ __forceinline__ void init(double2 *smem, unsigned long long *bars, int t, int nt) {
        place = smem + (t >> 5) * (NP * 32) + (t & 31);
        stride = nt * NP;
        bar = bars + (t >> 5) * ST;
        phase = 0;
    }
    // the barriers of all `warps` warps, by one warp
    __device__ __forceinline__ static void init_bars(unsigned long long *bars, int warps, int lane) {
        for (int q = lane; q < warps * ST; q += 32) mbar_init(bars + q);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // starts the copy of warp w's record at `slot` into stage st (from warp 0's place and barriers)
    __device__ __forceinline__ void start(const double2 *rec, int slot, int w, int st) const {
        const double2 *r = rec + rec_at(slot, 0, PAIRS);
        double2 *d = place + st * stride + w * (NP * 32);
        unsigned long long *b = bar + w * ST + st;
        mbar_expect(b, NP * 512);
        bulk_g2s(d, r + R0 * 32, N0 * 512, b);
        if (N1 > 0) bulk_g2s(d + N0 * 32, r + R1 * 32, N1 * 512, b);
    }
    __device__ __forceinline__ bool wait(int st, bool late) {
        const bool ok = mbar_wait(bar + st, (phase >> st) & 1u, late);
        phase ^= 1u << st;
        return ok;
    }
};

// offset of plane s's entry (the block's plane counter) in a ring
__device__ __forceinline__ long long ring_at(const WideArrays &A, int s) {
    return (long long)(s & (A.ringn - 1)) * WIDE_UNITS * A.nkmax;
}

// Three more warps of the CTA take what would otherwise be on its chain.

// the barrier of plane s: the compute warps, the copy warp and one of the two
// ring warps, n threads; planes alternate between two barriers
__device__ __forceinline__ void cta_sync(int s, int n) { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + (s & 1)), "r"(n) : "memory"); }

// The first starts the bulk copies of the others (lane w those of warp w),
// ST planes ahead, and keeps the rings from overflowing.
template <bool FWD, int ST, class Stage>
__device__ __forceinline__ bool copy_warp(const CtaInfo &H, const WideArrays &A, const WideSeg *__restrict__ segs,
                                          const double2 *rec, const Stage &X0, int nt, unsigned tag0, int np, int ns) {
    const int l = threadIdx.x & 31, nseg = H.C.nseg;
    const bool copies = l < nt / 32;
    // warp l's segment, window and slots (Walk)
    int f = FWD ? 0 : nseg - 1, first = 1, last = 0, cols = 0, slot0 = 0;
    auto enter = [&]() {
        const WideSeg S = segs[H.C.seg0 + f * H.C.segstep];
        cols = S.cols;
        int jklo = 1 << 30, jkhi = -1, k = l * 32 / H.C.w + 1, jj = l * 32 - (k - 1) * H.C.w;
        for (int q = 0; q < 32 && k <= H.nk; q++) {
            if (jj < S.w) {
                jklo = min(jklo, S.j0 + jj + 1 + k);
                jkhi = max(jkhi, S.j0 + jj + 1 + k);
            }
            if (++jj == H.C.w) jj = 0, k++;
        }
        window<FWD>(H, S, f, l * 32, jklo, jkhi, first, last, slot0);
    };
    if (copies) enter();
    auto copy = [&](int s, int st) {
        if (!copies) return;
        if (s > last && (FWD ? f + 1 < nseg : f > 0)) {
            f += FWD ? 1 : -1;
            enter();
        }
        if (s >= first && s <= last) X0.start(rec, FWD ? slot0 + s * cols : slot0 - s * cols, l, st);
    };
#pragma unroll
    for (int d = 0; d < ST; d++) copy(d, d);
    int st = 0;
    bool late = false;
#pragma unroll 1
    for (int s = 0; s < ns; s++, st = st + 1 == ST ? 0 : st + 1) {
        // every RING_CHECK planes (the fold delay is a multiple of them, so that
        // the segments come due together): wait until the ring entries that the
        // CTA is about to overwrite have been read
        if ((s & (RING_CHECK - 1)) == 0 && l == 31)
            for (int g = 0; g < nseg; g++) {
                const int sf = s - (FWD ? g : H.C.nsegmax - 1 - g) * H.C.delay, bo = FWD ? H.hi[g] : H.lo[g];
                if (bo < 0 || sf < 0 || sf >= np || ring_room(sf, A.ringn) <= 0) continue;
                const unsigned want = tag0 + (unsigned)ring_room(sf, A.ringn);
                const long long t0 = clock64(), limit = late ? (1LL << 21) : (1LL << 31);
                while ((int)(ld_acquire(A.flags + bo) - want) < 0)
                    if (clock64() - t0 > limit) { late = true; break; }
            }
        __syncwarp();
        cta_sync(s, nt + 64);
        copy(s + ST, st);  // into the stage of plane s: every thread has read its words
    }
    return late;
}

// The other two bring the entries of the rings into the inboxes: `jbox` has
// three planes of them, where the columns at the incoming edge read
// their j-neighbour's terms.  They take turns, one the even and one the odd
// planes, so that each has two planes' time for the trip to L2.
template <bool FWD, int NC>
__device__ __forceinline__ bool ring_warp(const CtaInfo &H, const WideArrays &A, double *jbox, int odd, unsigned tag0, int lo, int np,
                                          int ns, int nsync) {
    constexpr int NB = NC > 5 ? 14 : 8;  // units per lane and round
    constexpr int NS = NC < 5 ? NC : 5;  // terms per part
    const int l = threadIdx.x & 31, nseg = H.C.nseg, ni = H.ni, pmax = H.ni + H.nj + H.nk;
    bool late = false;
#pragma unroll 1
    for (int s = odd - 2; s < ns; s += 2) {
        if (s >= 0) cta_sync(s, nsync);
        // the entries of plane s + 1, for plane T = s + 2
        const int T = s + 2;
        double *const box = jbox + T % 3 * H.nk * NC;
        for (int g = 0; g < nseg; g++) {
            const int sdel = (FWD ? g : H.C.nsegmax - 1 - g) * H.C.delay, sf = T - 1 - sdel;
            if (sf < 0 || sf >= np || T >= ns) continue;
            const int bi = FWD ? H.lo[g] : H.hi[g], j = H.jin[g];
            if (bi < 0) continue;
            // the edge column of row k is at i = i0 - k in plane T
            const int i0 = FWD ? T + 3 - sdel - j : pmax + sdel - j - T;
            const bool edge = FWD ? j > lo && j <= H.nj + 1 - lo : j < H.nj + 1 - lo && j >= lo;
            const int klo = max(lo, i0 - (ni + 1 - lo)), uhi = (edge ? min(H.nk + 1 - lo, i0 - lo) : 0) * NC;
            const Unit *e = (const Unit *)A.ring + ((long long)bi * A.ringn + (sf & (A.ringn - 1))) * A.nkmax * WIDE_UNITS;
            const unsigned tag = tag0 + (unsigned)sf;
            for (int u0 = (klo - 1) * NC + l; u0 < uhi; u0 += 32 * NB) {
                Unit r[NB];
                unsigned open = 0;
#pragma unroll
                for (int q = 0; q < NB; q++)
                    if (u0 + q * 32 < uhi) {
                        r[q] = ld_unit(e + u0 + q * 32);
                        open |= 1u << q;
                    }
                long long t0 = 0;
                for (;;) {
#pragma unroll
                    for (int q = 0; q < NB; q++)
                        if ((open >> q & 1) && has_tag(r[q], tag)) {
                            const int u = u0 + q * 32;
                            box[u % NC / NS * (H.nk * NS) + (u / NC) * NS + u % NS] = __hiloint2double((int)(unsigned)r[q].hi, (int)(unsigned)r[q].lo);
                            open &= ~(1u << q);
                        }
                    if (!open) break;
                    if (t0 == 0) t0 = clock64();
                    else if (clock64() - t0 > (late ? (1LL << 21) : (1LL << 31))) { late = true; break; }
#pragma unroll
                    for (int q = 0; q < NB; q++)
                        if (open >> q & 1) r[q] = ld_unit(e + u0 + q * 32);
                }
            }
            // tell the writer how far both ring warps have read
            if (ring_publishes(sf)) {
                __syncwarp();
                if (l == 0) st_release(A.flags + bi, tag0 + (unsigned)ring_read(sf));
            }
        }
    }
    return late;
}

}  // namespace

// plane-major coefficients of every cell, evaluated once per step for all
// four sweeps, and rhs = dq (set_nonconnect_boundary_dq_0 has run, so rhs
// holds the zeros of the physical faces); one thread per slot.  Also moves
// the tags of the rings on.
__global__ void __launch_bounds__(256, 4) k_wide_prep(DevParams P, DevFields F, const DevBlock *__restrict__ blocks,
                                                  const WideSeg *__restrict__ segs, WideArrays A) {
    const WideSeg C = segs[blockIdx.y];
    const DevBlock B = blocks[C.blk];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *A.epoch += 4 * A.span;
    const bool swap = row_is_j(B);
    const int ncolc = C.W * (swap ? B.nj : B.nk), np = B.ni + B.nj + B.nk - 2;
    const long long n = (long long)((np + PREP_DS - 1) / PREP_DS * PREP_DS) * ncolc;
    const double gama = P.gama;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        // PREP_DS consecutive planes of one column per group of lanes: their
        // cells are consecutive in i, so a group's gathers from the field
        // layout share sectors, while a plane's stores stay runs of columns
        const long long sb = e / ((long long)PREP_DS * ncolc);
        const int r = (int)(e - sb * PREP_DS * ncolc), t = r / PREP_DS;
        const int s = (int)sb * PREP_DS + (r - t * PREP_DS);
        if (s >= np) continue;
        const int p = s + 3, jj = t % C.W, j = C.j0 + jj + 1, k = t / C.W + 1, i = p - j - k;
        if (jj >= C.w || i < 1 || i > B.ni) continue;
        const long long id = gidx(B, i, swap ? k : j, swap ? j : k);
        double2 *o = A.rec + rec_at(C.pmoff + s * C.cols + t, t & 31, WIDE_PAIRS);
        auto put = [&](int q, double a, double b) { o[q * 32] = make_double2(a, b); };
        const double rm = F.f[F_R][id], um = F.f[F_U][id], vm = F.f[F_V][id], wm = F.f[F_W][id], pres = F.f[F_P][id];
        // total enthalpy, gettmhmgm_ns (GasModel.f90:411-426)
        const double hint = gama / (gama - 1.0) * pres / rm;
        put(WP_UV, sw_velocity(um, hint), vm);
        put(WP_WH, wm, hint + 0.5 * (um * um + vm * vm + wm * wm));
#pragma unroll
        for (int m = 0; m < 8; m += 2) put(WP_G01 + m / 2, F.f[F_KCX + m][id], F.f[F_KCX + m + 1][id]);
        double rad[3], srv[3], dq[5];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            rad[d] = F.f[F_SRA + d][id];
            srv[d] = F.f[F_SRVA + d][id];
        }
#pragma unroll
        for (int m = 0; m < 5; m++) dq[m] = F.f[F_DQ1 + m][id];
        // getcoed (LHS.f90:602-645), wmig = beta = 1, no dual time stepping
        double rad_ns = rad[0] + rad[1] + rad[2];
        if (P.nvis >= 1) rad_ns = rad_ns + srv[0] + srv[1] + srv[2];
        const double ct = 1.0 / F.f[F_DTDT][id];
        put(WP_G8C, F.f[F_KCX + 8][id], 1.0 / (ct + 1.0 * 1.0 * rad_ns));
        put(WP_RAD01, rad[0], rad[1]);
        put(WP_RAD2R4, rad[2], dq[4]);
        put(WP_R01, dq[0], dq[1]);
        put(WP_R23, dq[2], dq[3]);
        if (P.nvis > 0) {
            put(WP_RS01, rad[0] + srv[0], rad[1] + srv[1]);
            o[WP_RS2D4 * 32].x = rad[2] + srv[2];
        }
    }
}

namespace {

// One cell's words of a sweep, from the staged pairs: pairs 0..N0-1 of the
// record and a second run.
//   lusgs_l  velocity .. rhs; radii with viscous part (without: radii)
//   lusgs_u  velocity .. coed; radii .. dq of lusgs_l
//   gs_pr_l  velocity .. rhs, radii; upper terms
//   gs_pr_u  velocity .. lower terms - rhs, radii
template <int MODE, bool VIS>
struct Cell {
    static constexpr int N0 = MODE == 1 ? WP_G8C + 1 : MODE == 0 && VIS ? WP_RAD2R4 + 1 : WP_RAD01 + 1;
    static constexpr int R1 = MODE == 0 ? WP_RS01 : MODE == 1 ? WP_RAD2R4 : WP_U01;
    static constexpr int N1 = MODE == 0 ? (VIS ? 2 : 0) : MODE == 1 ? 6 : MODE == 2 ? 3 : 0;
    static constexpr int NP = N0 + N1;
    template <int ST>
    using Stage = Stager<ST, 0, N0, R1, N1, WIDE_PAIRS>;
    // where pair `q` of the record is among the staged ones
    __device__ static constexpr int at(int q) { return q < N0 ? q : N0 + q - R1; }
    double2 w[NP];
    __device__ __forceinline__ void load(const double2 *place) {
#pragma unroll
        for (int q = 0; q < NP; q++) w[q] = place[q * 32];
    }
    // waits for the words: after the plane's barrier their place is filled anew
    __device__ __forceinline__ void arrived() const {
#pragma unroll
        for (int q = 0; q < NP; q++) asm volatile("" ::"d"(w[q].x), "d"(w[q].y) : "memory");
    }
    __device__ __forceinline__ double u() const { return w[0].x; }
    __device__ __forceinline__ double v() const { return w[0].y; }
    __device__ __forceinline__ double vz() const { return w[1].x; }
    __device__ __forceinline__ double h() const { return w[1].y; }
    __device__ __forceinline__ double coed() const { return w[6].y; }
    __device__ __forceinline__ double g(int m) const { return (m & 1) ? w[WP_G01 + m / 2].y : w[WP_G01 + m / 2].x; }
    __device__ __forceinline__ double rad(int d) const {
        return d == 0 ? w[at(WP_RAD01)].x : d == 1 ? w[at(WP_RAD01)].y : w[at(WP_RAD2R4)].x;
    }
    __device__ __forceinline__ double rads(int d) const {
        if constexpr (!VIS) return rad(d);
        else return d == 0 ? w[at(WP_RS01)].x : d == 1 ? w[at(WP_RS01)].y : w[at(WP_RS2D4)].x;
    }
    __device__ __forceinline__ double base(int m) const {
        if constexpr (MODE == 1) return m == 0 ? w[at(WP_D01)].x : m == 1 ? w[at(WP_D01)].y : m == 2 ? w[at(WP_D23)].x : m == 3 ? w[at(WP_D23)].y : w[at(WP_RS2D4)].y;
        else return m == 0 ? w[WP_R01].x : m == 1 ? w[WP_R01].y : m == 2 ? w[WP_R23].x : m == 3 ? w[WP_R23].y : w[WP_RAD2R4].y;
    }
    __device__ __forceinline__ double old(int m) const {
        if constexpr (MODE == 2) return m == 0 ? w[at(WP_U01)].x : m == 1 ? w[at(WP_U01)].y : m == 2 ? w[at(WP_U23)].x : m == 3 ? w[at(WP_U23)].y : w[at(WP_U4)].x;
        else return 0.0;
    }
};

// terms sent per direction: with viscous radii lusgs_u also needs the terms
// without them (for gs_pr_l)
template <int MODE, bool VIS>
constexpr int sent() { return MODE == 1 && VIS ? 10 : 5; }

}  // namespace

// MODE 0 lusgs_l, 1 lusgs_u, 2 gs_pr_l, 3 gs_pr_u; ST planes of a cell's words
// in shared memory
template <int MODE, bool VIS, int ST>
__global__ void __launch_bounds__(WIDE_THREADS + 96, 1) k_sweep_wide(DevParams P, DevFields F, const DevBlock *__restrict__ blocks,
                                                        const WideCta *__restrict__ ctas, const WideSeg *__restrict__ segs,
                                                        WideArrays A, int *err) {
    constexpr bool FWD = MODE == 0 || MODE == 2;
    constexpr int NC = sent<MODE, VIS>();
    const int t = threadIdx.x, nt = blockDim.x - 96;
    __shared__ CtaInfo H;
    if (t == 0) H.set(ctas[blockIdx.x], blocks[ctas[blockIdx.x].blk], segs, FWD);
    const unsigned tag0 = *A.epoch + MODE * A.span;
    using Words = Cell<MODE, VIS>;
    extern __shared__ __align__(128) double2 sraw[];
    __shared__ unsigned long long bars[WIDE_THREADS / 32 * ST];
    using Stage = typename Words::template Stage<ST>;
    Stage X;
    X.init(sraw, bars, t < nt ? t : 0, nt);
    if (t >= nt && t < nt + 32) Stage::init_bars(bars, nt / 32, t - nt);
    __syncthreads();
    const int np = H.ni + H.nj + H.nk - 2, ns = np + (H.C.nsegmax - 1) * H.C.delay;
    // inbox[parity][0 = j, 1 = k][part][column, and one of zeros][5], then three
    // planes of ring entries [part][row][5]: parts of five terms, so that a
    // warp's columns fall on different banks
    constexpr int NPART = NC / 5;
    double *const smem = (double *)(sraw + ST * X.stride);
    const int part = (nt + 1) * 5, kdir = NPART * part, half = 2 * kdir, jpart = H.nk * 5, jplane = NPART * jpart;
    double *const jbox = smem + 2 * half;
    for (int q = t; q < 2 * half + 3 * jplane; q += blockDim.x) smem[q] = 0.0;
    __syncthreads();
    if (t >= nt) {
        const bool over = t < nt + 32 ? copy_warp<FWD, ST>(H, A, segs, A.rec, X, nt, tag0, np, ns)
                                      : ring_warp<FWD, NC>(H, A, jbox, t >= nt + 64 ? 1 : 0, tag0, 1, np, ns, nt + 64);
        if (over) atomicAdd(&err[ERR_TIMEOUT], 1);
        return;
    }
    Walk<FWD, NC> K;
    K.init(H, A, segs, t, 1);
    const double aeh = 0.5 * (P.gama - 1.0);
    const double *const srck = smem + kdir + (K.hask ? (FWD ? t - H.C.w : t + H.C.w) : nt) * 5;
    double *const dst = smem + t * 5;
    const int offj = H.swap ? kdir : 0, offk = H.swap ? 0 : kdir;  // where the terms along j and k go
    const double *srcj;
    double ibuf[NC];  // contribution along i from this column's previous cell
    auto entered = [&]() {
        srcj = K.jin ? jbox + t / H.C.w * 5 : smem + (K.hasj ? (FWD ? t - 1 : t + 1) : nt) * 5;
#pragma unroll
        for (int m = 0; m < NC; m++) ibuf[m] = 0.0;
    };
    entered();
    bool late = false;
    int st = 0, wr = 0;  // the plane's stage; the inbox it writes (the other one is read)
#pragma unroll 1
    for (int s = 0; s < ns; s++, wr = half - wr, st = st + 1 == ST ? 0 : st + 1) {
        if (K.past(s)) {  // on to the warp's next columns
            K.enter(FWD ? K.f + 1 : K.f - 1, H, A, segs, t, 1);
            entered();
        }
        const int i = K.at(s);
        const bool act = K.col && (unsigned)(i - 1) < (unsigned)K.ni;
        Words c;
        if (K.busy(s)) {
            late = !X.wait(st, late) || late;
            c.load(X.place + st * X.stride);
            c.arrived();
        }
        cta_sync(s, nt + 64);  // the previous plane's inbox is complete
        if (act) {
            const int rd = half - wr;
            // contributions along j and along k of the block: one comes from the
            // chunk's next column (or the ring), the other from the next row
            const double *sj = srcj + (K.jin ? s % 3 * jplane : rd), *sk = srck + rd;
            int sjp = K.jin ? jpart : part, skp = part;
            if (H.swap) {
                const double *const x = sj;
                sj = sk;
                sk = x;
                skp = sjp;
                sjp = part;
            }
            // contributions of the three neighbours on the previous plane (zero
            // outside the block: the reference's ghost dq is zero)
            double sum[NC];
#pragma unroll
            for (int m = 0; m < NC; m++) sum[m] = (ibuf[m] + sj[m / 5 * sjp + m % 5]) + sk[m / 5 * skp + m % 5];
            double nw[5];
#pragma unroll
            for (int m = 0; m < 5; m++) nw[m] = sw_new<MODE>(sum[m], c.old(m), c.base(m), c.coed());
            const double u = c.u(), v = c.v(), w = c.vz(), h = c.h();
            const double e = sw_half_dh(aeh, u, v, w, nw);
#pragma unroll
            for (int dd = 0; dd < 3; dd++) {
                const int d = dd == 0 ? 1 : dd == 1 ? 2 : 0;  // j first: it may have a long way to go
                const double gx = c.g(3 * d), gy = c.g(3 * d + 1), gz = c.g(3 * d + 2);
                const double th = sw_theta(gx, gy, gz, u, v, w);
                double tm[5], o[NC];
                sw_terms(gx, gy, gz, th, u, v, w, h, e, nw, tm);
                const double l = sw_l<FWD>(th, MODE <= 1 ? c.rads(d) : c.rad(d));
#pragma unroll
                for (int m = 0; m < 5; m++) o[m] = fma(l, nw[m], tm[m]);
                if (NC == 10) {
                    const double l0 = sw_l<FWD>(th, c.rad(d));
#pragma unroll
                    for (int m = 0; m < 5; m++) o[NC - 5 + m] = fma(l0, nw[m], tm[m]);
                }
                if (d == 0) {
#pragma unroll
                    for (int m = 0; m < NC; m++) ibuf[m] = o[m];
                } else {
#pragma unroll
                    for (int m = 0; m < NC; m++) dst[wr + (d == 2 ? offk : offj) + m / 5 * part + m % 5] = o[m];
                    if (K.jout && d == (H.swap ? 2 : 1)) send<NC>(K.rout + ring_at(A, s - K.sdel), o, tag0 + (unsigned)(s - K.sdel));
                }
            }
            // results, off the chain
            if (MODE == 3) {
                const long long id = K.id0 + i;
#pragma unroll
                for (int m = 0; m < 5; m++) F.f[F_DQ1 + m][id] = nw[m];
            } else {
                double2 *r = A.rec + rec_at(K.slot(s), t & 31, WIDE_PAIRS);
                double x[5];
#pragma unroll
                for (int m = 0; m < 5; m++) x[m] = MODE == 0 ? nw[m] : MODE == 1 ? sum[NC - 5 + m] : sum[m] - c.base(m);
                r[(MODE == 0 ? WP_D01 : MODE == 1 ? WP_U01 : WP_R01) * 32] = make_double2(x[0], x[1]);
                r[(MODE == 0 ? WP_D23 : MODE == 1 ? WP_U23 : WP_R23) * 32] = make_double2(x[2], x[3]);
                if (MODE == 0) r[WP_RS2D4 * 32].y = x[4];
                if (MODE == 1) r[WP_U4 * 32].x = x[4];
                if (MODE == 2) r[WP_RAD2R4 * 32].y = x[4];
            }
        }
    }
    if (late) atomicAdd(&err[ERR_TIMEOUT], 1);
}

template <bool FWD>
__global__ void k_sa_sweep_wide(SaFields S, const DevBlock *__restrict__ blocks, const WideCta *__restrict__ ctas,
                                const WideSeg *__restrict__ segs, WideArrays A, int *err);

static size_t sa_smem(int threads, int nk) {
    return (size_t)SA_ST * threads * WIDE_SA_PAIRS * 16 + (size_t)(4 * (threads + 1) + 3 * nk) * 8;
}
// shared memory of a sweep: the staged words, the inboxes and the ring entries
template <int MODE, bool VIS>
static size_t wide_smem_of(int threads, int nk, int stages) {
    return (size_t)stages * threads * Cell<MODE, VIS>::NP * 16 + (size_t)(4 * (threads + 1) + 3 * nk) * sent<MODE, VIS>() * 8;
}

// The kernel of a sweep: with as many planes of words in flight as fit, at
// most four, for a context with or without viscous radii.
using WideKernel = void (*)(DevParams, DevFields, const DevBlock *, const WideCta *, const WideSeg *, WideArrays, int *);
struct WidePick { WideKernel fn; size_t smem; int stages; };
constexpr size_t WIDE_SMEM = 226 * 1024;
template <int MODE, bool VIS>
static WidePick wide_pick_of(int threads, int nk, int stages) {
    static const WideKernel fn[4] = {k_sweep_wide<MODE, VIS, 1>, k_sweep_wide<MODE, VIS, 2>, k_sweep_wide<MODE, VIS, 3>, k_sweep_wide<MODE, VIS, 4>};
    while (stages > 1 && wide_smem_of<MODE, VIS>(threads, nk, stages) > WIDE_SMEM) stages--;
    return {fn[stages - 1], wide_smem_of<MODE, VIS>(threads, nk, stages), stages};
}
// stages: at most so many planes of words in flight
static WidePick wide_pick(int mode, bool vis, int threads, int nk, int stages) {
    switch (mode) {
    case 0: return vis ? wide_pick_of<0, true>(threads, nk, stages) : wide_pick_of<0, false>(threads, nk, stages);
    case 1: return vis ? wide_pick_of<1, true>(threads, nk, stages) : wide_pick_of<1, false>(threads, nk, stages);
    case 2: return wide_pick_of<2, false>(threads, nk, stages);  // the Gauss-Seidel sweeps have no viscous part
    default: return wide_pick_of<3, false>(threads, nk, stages);
    }
}

// Chunks and folding.  For every number of segments per CTA and every width
// of the chunks the time of a sweep is estimated as (planes, fold delays
// included) x (T0 + TC x columns of a CTA) + (chunks of a block) x THOP, the
// hop between neighbouring chunks' CTAs, for the slowest block; the cheapest
// split whose CTAs are all resident at once is taken.  Returns -1 when the
// blocks cannot be swept this way.
int setup_sweep_wide(LaunchCtx &c, WideSweep &W) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    int nkmax = 0, span = 0;
    for (int b = 0; b < c.nblocks; b++) {
        const DevBlock &B = c.hblocks[b];
        nkmax = std::max(nkmax, std::min(B.nj, B.nk));
        span = std::max(span, B.ni + B.nj + B.nk);
    }
    if (nkmax > WIDE_THREADS) return -1;
    const int top = WIDE_THREADS;
    const bool vis = c.P->nvis > 0;
    // tests: chunks narrower than usual, fewer planes in flight
    int min_cols = WIDE_MIN_COLS, stages = 4;
    if (const char *e = getenv("WCNS_WIDE_MIN_COLS")) min_cols = std::max(1, atoi(e));
    if (const char *e = getenv("WCNS_WIDE_ST")) stages = std::min(4, std::max(1, atoi(e)));
    struct Split { int w, G, Gc, nseg, delay; };
    auto split = [&](const DevBlock &B, int cols, int fold) {
        Split S{};
        const int nb = std::max(B.nj, B.nk), nr = std::min(B.nj, B.nk);  // along the chunks, along a row
        S.w = std::max(1, std::min(cols / nr, top / nr));
        S.w = std::min(std::max(S.w, std::min((min_cols + nr - 1) / nr, top / nr)), nb);
        S.G = (nb + S.w - 1) / S.w;
        S.Gc = (S.G + fold - 1) / fold;
        S.nseg = (S.G + S.Gc - 1) / S.Gc;
        S.delay = 0;
        if (S.nseg > 1) {
            // j + k differs by at most this over the columns of a warp, which changes over as one
            int spread = 0;
            for (int w = std::max(1, S.w - 1); w <= S.w; w++) spread = std::max(spread, w - 1 + (31 + w - 1) / w);
            // a CTA's chunks start Gc * nb / G rows apart, rounded either way
            S.delay = std::max(0, B.ni + WIDE_GAP + spread - S.Gc * nb / S.G);
        }
        S.delay = (S.delay + RING_CHECK - 1) / RING_CHECK * RING_CHECK;
        return S;
    };
    double best = 1e300;
    int best_cols = 0, best_fold = 0;
    for (int fold = 1; fold <= WIDE_MAX_FOLD; fold++)
        for (int cols = 16; cols <= top; cols += 4) {
            double worst = 0.0;
            long long n = 0;
            int warps = 1;
            for (int b = 0; b < c.nblocks; b++) {
                const Split S = split(c.hblocks[b], cols, fold);
                n += S.Gc;
                warps = std::max(warps, (S.w * std::min(c.hblocks[b].nj, c.hblocks[b].nk) + 31) / 32);
            }
            // CTAs per SM: 12 warps of 168 registers, and their shared memory
            const long long per = (n + nsm - 1) / nsm;
            size_t smem = 0;
            for (int m = 0; m < 4; m++) smem = std::max(smem, wide_pick(m, vis, warps * 32, nkmax, stages).smem);
            if (per * (warps + 3) > 12 || (per == 1 ? smem > WIDE_SMEM : per * (smem + 2048) > WIDE_SMEM)) continue;
            for (int b = 0; b < c.nblocks; b++) {
                const DevBlock &B = c.hblocks[b];
                const Split S = split(B, cols, fold);
                const int np = B.ni + B.nj + B.nk - 2 + (S.nseg - 1) * S.delay;
                worst = std::max(worst, np * (WIDE_T0 + WIDE_TC * per * S.w * std::min(B.nj, B.nk)) + S.Gc * WIDE_THOP);
            }
            if (worst < best) {
                best = worst;
                best_cols = cols;
                best_fold = fold;
            }
        }
    // tests: a given split
    if (const char *e = getenv("WCNS_WIDE_FOLD")) best_fold = std::min(WIDE_MAX_FOLD, std::max(1, atoi(e)));
    if (const char *e = getenv("WCNS_WIDE_COLS")) best_cols = std::min(top, std::max(1, atoi(e)));
    if (best_fold == 0) return -1;
    std::vector<WideSeg> segs;
    std::vector<WideCta> ctas;
    long long n = 0;
    int nbnd = 0, maxcols = 0, maxdelay = 0;
    for (int b = 0; b < c.nblocks; b++) {
        const DevBlock &B = c.hblocks[b];
        const Split S = split(B, best_cols, best_fold);
        const int nb = std::max(B.nj, B.nk), nr = std::min(B.nj, B.nk);
        const int seg0 = (int)segs.size();
        for (int q = 0; q < S.G; q++) {
            WideSeg g{};
            g.blk = b;
            g.j0 = q * nb / S.G;
            g.w = (q + 1) * nb / S.G - g.j0;
            g.bnd_lo = q > 0 ? nbnd + q - 1 : -1;
            g.bnd_hi = q < S.G - 1 ? nbnd + q : -1;
            segs.push_back(g);
        }
        for (int q = 0; q < S.Gc; q++) {
            WideCta C{};
            C.blk = b;
            C.seg0 = seg0 + q;
            C.segstep = S.Gc;
            C.nseg = (S.G - q + S.Gc - 1) / S.Gc;
            C.nsegmax = S.nseg;
            C.delay = S.delay;
            for (int f = 0; f < C.nseg; f++) C.w = std::max(C.w, segs[seg0 + q + f * S.Gc].w);
            ctas.push_back(C);
            maxcols = std::max(maxcols, C.w * nr);
            for (int f = 0; f < C.nseg; f++) {
                WideSeg &g = segs[seg0 + q + f * S.Gc];
                g.W = C.w;
                g.cols = (C.w * nr + 31) / 32 * 32;
                g.pmoff = (int)std::min<long long>(n, 0x7fffffff);
                n += (long long)(B.ni + B.nj + B.nk - 2) * g.cols;
            }
        }
        maxdelay = std::max(maxdelay, S.delay);
        nbnd += S.G - 1;
    }
    if (n > 0x7fffffffLL) return -1;  // slots are counted in 32 bits
    int ringn = 32;
    while (ringn < maxdelay + 32) ringn *= 2;
    const int threads = (maxcols + 31) / 32 * 32;
    const bool verbose = getenv("WCNS_VERBOSE") != nullptr;
    if (threads > WIDE_THREADS) return -1;
    WidePick pick[4];
    for (int m = 0; m < 4; m++) {
        pick[m] = wide_pick(m, vis, threads, nkmax, stages);
        W.stages[m] = pick[m].stages;
        if (pick[m].smem > WIDE_SMEM) {
            if (verbose) fprintf(stderr, "wide sweeps: %d threads, %zu bytes of shared memory per CTA do not fit\n", threads, pick[m].smem);
            return -1;
        }
        cudaFuncSetAttribute(pick[m].fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WIDE_SMEM);
    }
    int per_sm = 1 << 20;
    auto fits = [&](auto kern, size_t bytes) {
        int q = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, kern, threads + 96, bytes);
        if (e != cudaSuccess) {
            if (verbose) fprintf(stderr, "wide sweeps: occupancy query failed: %s\n", cudaGetErrorString(e));
            cudaGetLastError();
            q = 0;
        }
        per_sm = std::min(per_sm, q);
    };
    for (int m = 0; m < 4; m++) fits(pick[m].fn, pick[m].smem);
    cudaFuncSetAttribute(k_sa_sweep_wide<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WIDE_SMEM);
    cudaFuncSetAttribute(k_sa_sweep_wide<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WIDE_SMEM);
    fits(k_sa_sweep_wide<true>, sa_smem(threads, nkmax));
    fits(k_sa_sweep_wide<false>, sa_smem(threads, nkmax));
    if (verbose)
        fprintf(stderr, "wide sweeps: %zu chunks on %zu CTAs (%d segments at most), %d threads, fold delay %d, ring %d, %zu %zu %zu %zu bytes of shared memory, %d CTAs per SM on %d SMs\n",
                segs.size(), ctas.size(), best_fold, threads, maxdelay, ringn, pick[0].smem, pick[1].smem, pick[2].smem, pick[3].smem, per_sm, nsm);
    if ((long long)per_sm * nsm < (long long)ctas.size()) return -1;
    W.nctas = (int)ctas.size();
    W.threads = threads;
    W.hctas = ctas;
    W.hsegs = segs;
    W.A.n = n;
    W.A.nkmax = nkmax;
    W.A.nbnd = nbnd;
    W.A.ringn = ringn;
    W.A.span = (unsigned)span + 1;
    return 0;
}

// every CTA resident at once: a cooperative launch (capturable in the step graph)
static void launch_wide(const LaunchCtx &c, int mode) {
    const WideSweep &W = *c.wide;
    const WidePick pick = wide_pick(mode, c.P->nvis > 0, W.threads, W.A.nkmax, W.stages[mode]);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(W.nctas, 1, 1);
    cfg.blockDim = dim3(W.threads + 96, 1, 1);  // and the three helper warps
    cfg.dynamicSmemBytes = pick.smem;
    cfg.stream = c.stream;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, pick.fn, *c.P, *c.F, (const DevBlock *)c.blocks, (const WideCta *)W.ctas,
                       (const WideSeg *)W.segs, W.A, c.err);
}

// slots of the longest chunk, for the grids of the prep kernels
static int max_slots(const LaunchCtx &c) {
    int m = 0;
    for (const WideSeg &S : c.wide->hsegs) {
        const DevBlock &B = c.hblocks[S.blk];
        m = std::max(m, (B.ni + B.nj + B.nk - 2) * S.W * std::min(B.nj, B.nk));
    }
    return m;
}

int launch_sweeps_wide(const LaunchCtx &c) {
    const WideSweep &W = *c.wide;
    k_wide_prep<<<dim3((unsigned)std::min(4096, (max_slots(c) + 255) / 256), (unsigned)W.hsegs.size()), 256, 0, c.stream>>>(
        *c.P, *c.F, c.blocks, W.segs, W.A);
    prof_mark(c, "lhs_prep");
    launch_wide(c, 0);
    prof_mark(c, "sweep_lusgs_l");
    launch_wide(c, 1);
    prof_mark(c, "sweep_lusgs_u");
    launch_wide(c, 2);
    prof_mark(c, "sweep_gs_pr_l");
    launch_wide(c, 3);
    prof_mark(c, "sweep_gs_pr_u");
    return 5;
}


// ---------------------------------------------------------------------------
// lusgs_turbulence (turblence.f90:477-558) on the same chunks: the SA model's
// scalar forward and backward sweeps over the points 2..n-1 of every
// direction.  A point's term for a successor is mxdq_std_turbulence
// (560-583) of the point itself: 0.5*(l + npn*|l|)*dqke with l the
// contravariant velocity along the direction, so the prep keeps l for the
// three directions, 1/spec and the right-hand side per slot.

// pairs per slot: l along i and j; l along k and 1/spec; dqke (right-hand side)
// and the forward result
enum : int { WSA_L01 = 0, WSA_L2S, WSA_RF, WSA_N };
static_assert(WSA_N == WIDE_SA_PAIRS, "pairs per slot");

__global__ void __launch_bounds__(256) k_sa_wide_prep(DevFields F, SaFields S, const DevBlock *__restrict__ blocks,
                                                     const WideSeg *__restrict__ segs, WideArrays A) {
    const WideSeg C = segs[blockIdx.y];
    const DevBlock B = blocks[C.blk];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *A.epoch += 4 * A.span;
    const bool swap = row_is_j(B);
    const int ncolc = C.W * (swap ? B.nj : B.nk), np = B.ni + B.nj + B.nk - 2;
    const long long n = (long long)((np + PREP_DS - 1) / PREP_DS * PREP_DS) * ncolc;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long sb = e / ((long long)PREP_DS * ncolc);
        const int r = (int)(e - sb * PREP_DS * ncolc), t = r / PREP_DS;
        const int s = (int)sb * PREP_DS + (r - t * PREP_DS);
        if (s >= np) continue;
        const int p = s + 3, jj = t % C.W, j = C.j0 + jj + 1, k = t / C.W + 1, i = p - j - k;
        const int jb = swap ? k : j, kb = swap ? j : k;
        if (jj >= C.w || i < 2 || i > B.ni - 1 || jb < 2 || jb > B.nj - 1 || kb < 2 || kb > B.nk - 1) continue;
        const long long id = gidx(B, i, jb, kb);
        double2 *o = A.sa + rec_at(C.pmoff + s * C.cols + t, t & 31, WIDE_SA_PAIRS);
        const double u = F.f[F_U][id], v = F.f[F_V][id], w = F.f[F_W][id];
        double l[3];
#pragma unroll
        for (int d = 0; d < 3; d++)
            l[d] = F.f[F_KCX + 3 * d][id] * u + F.f[F_KCX + 3 * d + 1][id] * v + F.f[F_KCX + 3 * d + 2][id] * w;
        o[WSA_L01 * 32] = make_double2(l[0], l[1]);
        o[WSA_L2S * 32] = make_double2(l[2], S.spec[id]);
        o[WSA_RF * 32].x = S.dqke[id];
    }
}

template <bool FWD>
__global__ void __launch_bounds__(WIDE_THREADS + 96, 1) k_sa_sweep_wide(SaFields S, const DevBlock *__restrict__ blocks,
                                                                       const WideCta *__restrict__ ctas,
                                                                       const WideSeg *__restrict__ segs, WideArrays A,
                                                                       int *err) {
    const double npn = FWD ? 1.0 : -1.0;
    constexpr int NC = 1;
    const int t = threadIdx.x, nt = blockDim.x - 96;
    __shared__ CtaInfo H;
    if (t == 0) H.set(ctas[blockIdx.x], blocks[ctas[blockIdx.x].blk], segs, FWD);
    const unsigned tag0 = *A.epoch + (FWD ? 0 : 1) * A.span;
    extern __shared__ __align__(128) double2 sraw[];
    __shared__ unsigned long long bars[WIDE_THREADS / 32 * SA_ST];
    using Stage = Stager<SA_ST, 0, WSA_N, 0, 0, WSA_N>;
    Stage X;
    X.init(sraw, bars, t < nt ? t : 0, nt);
    if (t >= nt && t < nt + 32) Stage::init_bars(bars, nt / 32, t - nt);
    __syncthreads();
    const int np = H.ni + H.nj + H.nk - 2, ns = np + (H.C.nsegmax - 1) * H.C.delay;
    double *const smem = (double *)(sraw + SA_ST * X.stride);
    const int kdir = nt + 1, half = 2 * kdir, jplane = H.nk;
    double *const jbox = smem + 2 * half;
    for (int q = t; q < 2 * half + 3 * jplane; q += blockDim.x) smem[q] = 0.0;
    __syncthreads();
    // a predecessor outside 2..n-1 contributes zero (its dqke is zero)
    if (t >= nt) {
        const bool over = t < nt + 32 ? copy_warp<FWD, SA_ST>(H, A, segs, A.sa, X, nt, tag0, np, ns)
                                      : ring_warp<FWD, NC>(H, A, jbox, t >= nt + 64 ? 1 : 0, tag0, 2, np, ns, nt + 64);
        if (over) atomicAdd(&err[ERR_TIMEOUT], 1);
        return;
    }
    Walk<FWD, NC> K;
    K.init(H, A, segs, t, 2);
    const double *const srck = smem + kdir + (K.hask ? (FWD ? t - H.C.w : t + H.C.w) : nt);
    double *const dst = smem + t;
    const double *srcj;
    double ibuf;
    auto entered = [&]() {
        srcj = K.jin ? jbox + t / H.C.w : smem + (K.hasj ? (FWD ? t - 1 : t + 1) : nt);
        ibuf = 0.0;
    };
    entered();
    bool late = false;
    int st = 0, wr = 0;
#pragma unroll 1
    for (int s = 0; s < ns; s++, wr = half - wr, st = st + 1 == SA_ST ? 0 : st + 1) {
        if (K.past(s)) {
            K.enter(FWD ? K.f + 1 : K.f - 1, H, A, segs, t, 2);
            entered();
        }
        const int i = K.at(s);
        const bool act = K.inner && (unsigned)(i - 2) < (unsigned)(K.ni - 2);
        double2 l01, l2s, rf;
        if (K.busy(s)) {
            late = !X.wait(st, late) || late;
            const double2 *c = X.place + st * X.stride;
            l01 = c[WSA_L01 * 32];
            l2s = c[WSA_L2S * 32];
            rf = c[WSA_RF * 32];
            asm volatile("" ::"d"(l01.x), "d"(l2s.x), "d"(rf.x), "d"(rf.y) : "memory");
        }
        cta_sync(s, nt + 64);
        if (act) {
            const int rd = half - wr;
            const double tc = srcj[K.jin ? s % 3 * jplane : rd], tr = srck[rd];
            const double rhs0 = ibuf + (H.swap ? tr : tc) + (H.swap ? tc : tr);
            const double nw = FWD ? (rhs0 - rf.x) * l2s.y : rf.y - rhs0 * l2s.y;
            const double oj = 0.5 * (l01.y + npn * fabs(l01.y)) * nw, ok = 0.5 * (l2s.x + npn * fabs(l2s.x)) * nw;
            const double oc = H.swap ? ok : oj, orow = H.swap ? oj : ok;
            if (K.jout) send<1>(K.rout + ring_at(A, s - K.sdel), &oc, tag0 + (unsigned)(s - K.sdel));
            ibuf = 0.5 * (l01.x + npn * fabs(l01.x)) * nw;
            dst[wr] = oc;
            dst[wr + kdir] = orow;
            if (FWD) A.sa[rec_at(K.slot(s), t & 31, WIDE_SA_PAIRS) + WSA_RF * 32].y = nw;
            else S.dqke[K.id0 + i] = nw;
        }
    }
    if (late) atomicAdd(&err[ERR_TIMEOUT], 1);
}

template <bool FWD>
static void launch_sa_wide_t(const LaunchCtx &c) {
    const WideSweep &W = *c.wide;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(W.nctas, 1, 1);
    cfg.blockDim = dim3(W.threads + 96, 1, 1);  // and the three helper warps
    cfg.dynamicSmemBytes = sa_smem(W.threads, W.A.nkmax);
    cfg.stream = c.stream;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_sa_sweep_wide<FWD>, *c.SA, (const DevBlock *)c.blocks, (const WideCta *)W.ctas,
                       (const WideSeg *)W.segs, W.A, c.err);
}

// the SA model's scalar LU-SGS on the wide chunks; returns the number of launches
int launch_sa_lusgs_wide(const LaunchCtx &c) {
    const WideSweep &W = *c.wide;
    k_sa_wide_prep<<<dim3((unsigned)std::min(4096, (max_slots(c) + 255) / 256), (unsigned)W.hsegs.size()), 256, 0, c.stream>>>(
        *c.F, *c.SA, c.blocks, W.segs, W.A);
    launch_sa_wide_t<true>(c);
    launch_sa_wide_t<false>(c);
    return 3;
}

}  // namespace wcns
