// ran1_pair.cuh -- the ran1 stream by three warps (auxiliary_routines.py:324-391).
//
// The Bays-Durham shuffle is a chain: the next slot is the top five bits of the value found in
// this one.  Only those five bits ("keys") are on the chain, and the keys of the values that will
// be written into the slots are known ahead (the Park-Miller sequence does not depend on the
// slots).  So one warp walks the slots on keys alone, a second forms the Park-Miller values before
// it, and a third the stream's values from the slots walked.
//
// The walk takes two steps per shuffle latency.  Lane i holds the key a of slot i and the key e of
// the slot a points at; the walk at slot c fetches both with two shuffles issued together, p = a[c]
// (the second slot) and q = e[c] (the slot after it; the first step's key u instead where p is c
// itself).  The two writes (key u into slot c, key v into slot p) are then folded into every lane: a
// changes in lanes c and p, e in those and in the lanes whose a points at c or p.  Two more shuffles in
// the shadow of the first two (a[u], and a[v] after the first write) supply what lanes c and p point
// at.  The e of a slot that points at itself is never read, so it may hold anything.  Everything
// that involves c and u is prepared while the shuffles run: a comparison and two selects stand between
// a fetch and the next, and a double step issues 12 comparisons and selects, which run at half rate.
//
// Measured on B200, cycles a value: 27.2 in a fill of 140,000 (23 the walk alone); 29.4 with the values formed by the maker's
// warp and 18 comparisons and selects; 31.4 for one warp that shuffles values and keys step by step; the
// dependent shuffle alone is 26.
#pragma once

#include "common.cuh"
#include "umma.cuh"

namespace epsr {

constexpr int R1_NB = 16;         // batches of 32 in flight between the warps (power of two)

struct alignas(16) R1Ring {       // shared memory; rows are read 16 bytes at a time
    int keys[R1_NB][32];
    int32_t vals[R1_NB][32];
    uint4 slots[R1_NB][2];        // step t of the batch in byte t ^ 3
    int tab[32];                  // the table of the value warp
    // mbarriers: a batch's keys are there; its slots are; its values are delivered
    uint64_t made[R1_NB], walked[R1_NB], taken[R1_NB];
    int stop;                     // 1: the other warps leave
    unsigned byte;                // 256
};

__device__ __forceinline__ int r1_vol(const int *p) { return *(const volatile int *)p; }
__device__ __forceinline__ void r1_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void r1_arrive_if(uint64_t *bar, bool yes) {   // predicated, not a branch
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(bar)),
                 "r"((int)yes)
                 : "memory");
}
__device__ __forceinline__ void r1_init(R1Ring &R) {   // one thread; a barrier follows
    for (int i = 0; i < R1_NB; ++i) {
        umma::mbar_init(&R.made[i], 1);
        umma::mbar_init(&R.walked[i], 1);
        umma::mbar_init(&R.taken[i], 1);
    }
    R.stop = 0;
    R.byte = 256;
    umma::fence_mbar_init();
}

// The slot warp.  a: the key of this lane's slot; c: the first slot.  Walks batches 0 .. nb - 1
// as their keys (and the first key of the batch after) arrive; gives up when they do not, and
// leaves when R.stop is set.
__device__ __forceinline__ void r1_walk(R1Ring &R, int a, int c, int nb) {
    const int lane = threadIdx.x & 31;
    if (nb > 0 && !(umma::mbar_wait(&R.made[0], 0, nullptr) && umma::mbar_wait(&R.made[1], 0, nullptr))) return;
    int e = __shfl_sync(0xffffffffu, a, a);
    const unsigned byte = *(volatile unsigned *)&R.byte;
    int4 k = nb > 0 ? *(const int4 *)R.keys[0] : make_int4(0, 0, 0, 0);
    for (int b = 0; b < nb; ++b) {
        // the batch after the next one's keys: asked for early, waited for at the end
        bool there = true;
        int stop = 0;
        const int4 *k4 = (const int4 *)R.keys[b & (R1_NB - 1)];
        const int4 after = *(const int4 *)R.keys[(b + 1) & (R1_NB - 1)];
        uint4 *out = R.slots[b & (R1_NB - 1)];
        unsigned w[4];
#pragma unroll
        for (int s = 0; s < 16; ++s) {
            // the keys written in this double step
            const int u = (s & 1) ? k.z : k.x, v = (s & 1) ? k.w : k.y;
            if (s & 1) k = s < 15 ? k4[(s >> 1) + 1] : after;
            const int p = __shfl_sync(0xffffffffu, a, c);
            const int q = __shfl_sync(0xffffffffu, e, c);
            const int au = __shfl_sync(0xffffffffu, a, u);
            // after the first write
            const bool first = lane == c;
            const int ac = first ? u : a;
            const int av = __shfl_sync(0xffffffffu, ac, v);
            const int led = first ? au : e;
            const int ec = ac == c ? u : led;
            // after the second
            const int e1 = ac == p ? v : ec;
            const bool second = lane == p;
            e = second ? av : e1;
            a = second ? v : ac;
            // the slots walked, four to a word: on the multiplier, whose pipe is free (the factor is
            // read from memory so that it stays a product; shifts: 33 cycles a value), and stored
            // sixteen at a time under a predicate, not a branch (31)
            const unsigned wc = (s & 1) ? w[(s >> 1) & 3] * byte + (unsigned)c : (unsigned)c;
            w[(s >> 1) & 3] = wc * byte + (unsigned)p;
            if ((s & 7) == 7)
                asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %5, 0;\n\t@p st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n\t}" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(out + (s >> 3))),
                             "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(lane));
            c = p == c ? u : q;
            if (s == 8) stop = r1_vol(&R.stop);
            if (s == 8) there = umma::mbar_try(&R.made[(b + 2) & (R1_NB - 1)], (uint32_t)((b + 2) / R1_NB) & 1u);
        }
        r1_arrive_if(&R.walked[b & (R1_NB - 1)], lane == 0);
        if (!there && b + 1 < nb &&
            !umma::mbar_wait(&R.made[(b + 2) & (R1_NB - 1)], (uint32_t)((b + 2) / R1_NB) & 1u, nullptr))
            return;
        if (stop) return;
    }
}

// The maker warp: the Park-Miller values after idum and their keys, batch after batch (nb and the one
// after, which the walk looks into), as far ahead as the ring goes; leaves when R.stop is set.
__device__ __forceinline__ void r1_make(R1Ring &R, int32_t idum, uint32_t mul, int nb) {
    const int lane = threadIdx.x & 31;
    const uint32_t mul32 = (uint32_t)__shfl_sync(0xffffffffu, (int)mul, 31);   // IA^32 mod IM
    uint32_t x = r1_mulmod(mul, (uint32_t)idum);
    for (int b = 0; b - 1 < max(nb, 1); ++b) {
        const int i = b & (R1_NB - 1);
        if (b >= R1_NB && !__all_sync(0xffffffffu, umma::mbar_wait(&R.taken[i], (uint32_t)(b / R1_NB - 1) & 1u, nullptr)))
            return;
        if (r1_vol(&R.stop)) {   // no batch follows: the walk goes home
            __syncwarp();
            r1_arrive_if(&R.made[i], lane == 0);
            r1_arrive_if(&R.made[(b + 1) & (R1_NB - 1)], lane == 0);
            return;
        }
        R.keys[i][lane] = (int)(x >> 26);
        R.vals[i][lane] = (int32_t)x;
        __syncwarp();
        r1_arrive_if(&R.made[i], lane == 0);
        x = r1_mulmod(mul32, x);
    }
}

// The value warp: take() delivers the next batch's values once walked.  The table is in the ring.
struct R1Values {
    int32_t x, mine;              // the last batch's Park-Miller values and stream values
    int n;                        // batches taken

    // From a stream that is clean (common.cuh): idum in 1..IM-1, iy != 0, no zero table entry.
    __device__ __forceinline__ void begin(const Ran1Warp &g) {
        x = g.idum;
        mine = g.iy;
        n = 0;
    }
    // the state's words after the last batch taken
    __device__ __forceinline__ int32_t idum() const { return __shfl_sync(0xffffffffu, x, 31); }
    __device__ __forceinline__ int32_t iy() const { return __shfl_sync(0xffffffffu, mine, 31); }
    // Send the other warps home.  The maker waits at most for the first batch not taken (it has made
    // at least one past the last taken, so no earlier phase of that barrier is outstanding).
    __device__ __forceinline__ void leave(R1Ring &R) {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) {
            *(volatile int *)&R.stop = 1;
            r1_arrive(&R.taken[n & (R1_NB - 1)]);
        }
    }
    __device__ __forceinline__ bool walked(R1Ring &R) const {   // the next batch
        return __all_sync(0xffffffffu,
                          umma::mbar_wait(&R.walked[n & (R1_NB - 1)], (uint32_t)(n / R1_NB) & 1u, nullptr));
    }
    __device__ __forceinline__ int32_t take(R1Ring &R) {
        const int lane = threadIdx.x & 31;
        const int i = n++ & (R1_NB - 1);
        x = R.vals[i][lane];
        const int s = ((const unsigned char *)R.slots[i])[lane ^ 3];
        // the steps of the batch at this lane's slot: five ballots (match.any takes 400 cycles for
        // 32 different values)
        unsigned same = 0xffffffffu;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const bool bit = (s >> k) & 1;
            const unsigned bal = __ballot_sync(0xffffffffu, bit);
            same &= bit ? bal : ~bal;
        }
        const unsigned before = same & ((1u << lane) - 1u);
        const int32_t old = R.tab[s];
        const int32_t put = __shfl_sync(0xffffffffu, x, before ? 31 - __clz(before) : 0);
        __syncwarp();
        if ((same >> lane) == 1u) R.tab[s] = x;   // the last of the batch to write the slot
        r1_arrive_if(&R.taken[i], lane == 0);
        __syncwarp();
        mine = before ? put : old;
        return mine;
    }
};

// n values of the stream of warp-uniform `state` by the first three warps of a CTA (the other warps
// do not call; hardware barrier 7): warp 0 delivers them to put(i, value bits), lane by lane, in
// batches of 32 and less at the ends, and has the generator after them; warp 1 walks, warp 2 makes.
template <class F>
__device__ void r1_fill(R1Ring &R, int32_t *tab, const int32_t *state, int64_t n, Ran1Warp &g, F put) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ int s_batches, s_iy, s_idum;
    int64_t done = 0;
    g.load(state);
    if (w == 0) {
        // until the stream is clean: one batch as a rule (the initialisation happens inside)
        while (done < n && !(g.clean && g.idum > 0)) {
            int32_t mine;
            const int cnt = g.next(n - done > 32 ? 32 : (int)(n - done), mine, tab);
            if (lane < cnt) put(done + lane, mine);
            done += cnt;
        }
        R.tab[lane] = g.iv;
        if (lane == 0) {
            r1_init(R);
            s_batches = g.clean ? (int)((n - done) / 32) : 0;
            s_iy = g.iy;
            s_idum = g.idum;
        }
    }
    asm volatile("bar.sync 7, 96;" ::: "memory");   // the three warps of a larger CTA
    const int nb = s_batches;
    const int first_key = R.tab[lane] >> 26, first = s_iy >> 26;
    const int32_t idum = s_idum;
    asm volatile("bar.sync 7, 96;" ::: "memory");
    if (w == 1) {
        if (nb > 0) r1_walk(R, first_key, first, nb);
        return;
    }
    if (w == 2) {
        if (nb > 0) r1_make(R, idum, g.mul, nb);
        return;
    }
    if (nb > 0) {
        R1Values v;
        v.begin(g);
        for (int b = 0; b < nb; ++b) {
            if (!v.walked(R)) {   // the walk gave up: this warp goes on alone from here
                v.leave(R);
                break;
            }
            put(done + lane, v.take(R));
            done += 32;
        }
        g.idum = v.idum();
        g.iy = v.iy();
        g.iv = R.tab[lane];
        g.idl_ok = false;
    }
    while (done < n) {
        int32_t mine;
        const int cnt = g.next(n - done > 32 ? 32 : (int)(n - done), mine, tab);
        if (lane < cnt) put(done + lane, mine);
        done += cnt;
    }
}

}  // namespace epsr
