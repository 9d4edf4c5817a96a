// ran1_pair.cuh -- the ran1 stream by two warps (auxiliary_routines.py:324-391).
//
// The Bays-Durham shuffle is a chain: the next slot is the top five bits of the value found in
// this one.  Only those five bits ("keys") are on the chain, and the keys of the values that will
// be written into the slots are known ahead (the Park-Miller sequence does not depend on the
// slots).  So one warp walks the slots on keys alone, and a second warp forms the Park-Miller
// values before it and, from the slots walked, the stream's values after it.
//
// The walk takes two steps per shuffle latency.  Lane i holds the key a of slot i and the key e
// that a walk entering at slot i reads in its second step (with the first step's write taken into
// account); the walk at slot c fetches both with two shuffles issued together, p = a[c] (the
// second slot) and q = e[c] (the slot after it).  The two writes (key u into slot c, key v into
// slot p) are then folded into every lane: a changes in lanes c and p, and e in the lanes whose
// slot a points at c or p; three more shuffles in the shadow of the first two (a of a in every
// lane, a[u], a[v]) supply what the lanes read next.  Everything that involves c and u is prepared
// while the shuffles run, so a comparison and two selects stand between a fetch and the next.
//
// Measured on B200, the walk alone: 24.8 cycles a value (29 with the ring between the warps), 29.5
// step by step on keys, and 31.4 for
// one warp that shuffles values and keys step by step; the dependent shuffle alone is 26.  A branch
// for the two lanes whose e is late, instead of their selects: 26.6.
#pragma once

#include "common.cuh"
#include "umma.cuh"

namespace epsr {

constexpr int R1_NB = 16;         // batches of 32 in flight between the warps (power of two)

struct alignas(16) R1Ring {       // shared memory; rows are read 16 bytes at a time
    int keys[R1_NB][32];
    unsigned short slots[R1_NB][16];
    int tab[32];                  // the table of the value warp
    uint64_t made[R1_NB], walked[R1_NB];   // mbarriers: a batch's keys are there; its slots are
    int stop;                     // 1: the walk leaves
};

__device__ __forceinline__ int r1_vol(const int *p) { return *(const volatile int *)p; }
__device__ __forceinline__ void r1_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void r1_init(R1Ring &R) {   // one thread; a barrier follows
    for (int i = 0; i < R1_NB; ++i) {
        umma::mbar_init(&R.made[i], 1);
        umma::mbar_init(&R.walked[i], 1);
    }
    R.stop = 0;
    umma::fence_mbar_init();
}

// The slot warp.  a: the key of this lane's slot; c: the first slot.  Walks batches 0 .. nb - 1
// as their keys (and the first key of the batch after) arrive; gives up when they do not, and
// leaves when R.stop is set.
__device__ __forceinline__ void r1_walk(R1Ring &R, int a, int c, int nb) {
    const int lane = threadIdx.x & 31;
    int e = 0;
    if (nb > 0 && !(umma::mbar_wait(&R.made[0], 0, nullptr) && umma::mbar_wait(&R.made[1], 0, nullptr))) return;
    {
        const int f = __shfl_sync(0xffffffffu, a, a);
        e = a == lane ? R.keys[0][0] : f;
    }
    int4 k = nb > 0 ? *(const int4 *)R.keys[0] : make_int4(0, 0, 0, 0);
    for (int b = 0; b < nb; ++b) {
        // the batch after the next one's keys: asked for early, waited for at the end
        bool there = true;
        int stop = 0;
        const int4 *k4 = (const int4 *)R.keys[b & (R1_NB - 1)];
        const int4 after = *(const int4 *)R.keys[(b + 1) & (R1_NB - 1)];
        unsigned short *out = R.slots[b & (R1_NB - 1)];
#pragma unroll
        for (int s = 0; s < 16; ++s) {
            // the keys written in this double step, and the first of the next
            const int u = (s & 1) ? k.z : k.x, v = (s & 1) ? k.w : k.y;
            int4 kn = k;
            if (s & 1) kn = s < 15 ? k4[(s >> 1) + 1] : after;
            const int u2 = (s & 1) ? kn.x : k.z;
            const int p = __shfl_sync(0xffffffffu, a, c);
            const int q = __shfl_sync(0xffffffffu, e, c);
            const int f = __shfl_sync(0xffffffffu, a, a);
            const int au = __shfl_sync(0xffffffffu, a, u);
            const int av = __shfl_sync(0xffffffffu, a, v);
            // lanes other than p: the slot's key after the first write, and the key its key leads to
            const int ac = lane == c ? u : a;
            const bool self = ac == lane, fixed = self || ac == c;
            const int known = self ? u2 : u;
            const int led = lane == c ? au : f;
            const int ec = fixed ? known : led;
            // lane p: the second write
            const int lv = v == c ? u : av;
            const int ev = v == lane ? u2 : lv;
            const int e1 = ac == p ? v : ec;
            e = lane == p ? ev : e1;
            a = lane == p ? v : ac;
            if (lane == 0) out[s] = (unsigned short)(c | (p << 8));
            c = q;
            k = kn;
            if (s == 8) stop = r1_vol(&R.stop);
            if (s == 8) there = umma::mbar_try(&R.made[(b + 2) & (R1_NB - 1)], (uint32_t)((b + 2) / R1_NB) & 1u);
        }
        if (lane == 0) r1_arrive(&R.walked[b & (R1_NB - 1)]);
        if (!there && b + 1 < nb &&
            !umma::mbar_wait(&R.made[(b + 2) & (R1_NB - 1)], (uint32_t)((b + 2) / R1_NB) & 1u, nullptr))
            return;
        if (stop) return;
    }
}

// The value warp: make(j) puts the next batch's keys into the ring, take(b, j) delivers batch b's
// values once walked (j: the batch modulo R1_NB / 2, a constant).  idum and iy are those after the
// last batch taken, the table is in the ring.
struct R1Values {
    int32_t idum, iy;
    uint32_t mul;                 // IA^(lane + 1) mod IM
    int32_t head;                 // the last Park-Miller value made
    int32_t idl[R1_NB / 2];       // this lane's value of each batch in flight
    int made;

    // From a stream that is clean (common.cuh): idum in 1..IM-1, iy != 0, no zero table entry.
    __device__ __forceinline__ void begin(R1Ring &R, const Ran1Warp &g) {
        idum = head = g.idum;
        iy = g.iy;
        mul = g.mul;
        made = 0;
        R.tab[threadIdx.x & 31] = g.iv;
        __syncwarp();
    }
    __device__ __forceinline__ void make(R1Ring &R, int j) {
        const int lane = threadIdx.x & 31;
        idl[j] = (int32_t)r1_mulmod(mul, (uint32_t)head);
        head = __shfl_sync(0xffffffffu, idl[j], 31);
        R.keys[made & (R1_NB - 1)][lane] = idl[j] >> 26;
        __syncwarp();
        if (lane == 0) r1_arrive(&R.made[made & (R1_NB - 1)]);
        ++made;
    }
    __device__ __forceinline__ void leave(R1Ring &R) {   // no batch follows: the walk goes home
        __syncwarp();
        if ((threadIdx.x & 31) == 0) {
            *(volatile int *)&R.stop = 1;
            for (int i = 0; i < 2; ++i) r1_arrive(&R.made[(made + i) & (R1_NB - 1)]);
        }
    }
    __device__ __forceinline__ bool walked(R1Ring &R, int b) {
        return __all_sync(0xffffffffu,
                          umma::mbar_wait(&R.walked[b & (R1_NB - 1)], (uint32_t)(b / R1_NB) & 1u, nullptr));
    }
    __device__ __forceinline__ int32_t take(R1Ring &R, int b, int j) {
        const int lane = threadIdx.x & 31;
        const int32_t x = idl[j];
        const int s = ((const unsigned char *)R.slots[b & (R1_NB - 1)])[lane];
        // the steps of the batch at this lane's slot: five ballots (match.any takes 400 cycles for
        // 32 different values)
        unsigned same = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const bool bit = (s >> i) & 1;
            const unsigned bal = __ballot_sync(0xffffffffu, bit);
            same &= bit ? bal : ~bal;
        }
        const unsigned before = same & ((1u << lane) - 1u);
        const int32_t old = R.tab[s];
        const int32_t put = __shfl_sync(0xffffffffu, x, before ? 31 - __clz(before) : 0);
        __syncwarp();
        if ((same >> lane) == 1u) R.tab[s] = x;   // the last of the batch to write the slot
        __syncwarp();
        const int32_t mine = before ? put : old;
        idum = __shfl_sync(0xffffffffu, x, 31);
        iy = __shfl_sync(0xffffffffu, mine, 31);
        return mine;
    }
};

// n values of the stream of warp-uniform `state` by the first two warps of a CTA (the other warps
// do not call; hardware barrier 7): warp 0 delivers them to put(i, value bits), lane by lane, in
// batches of 32 and less at the ends, and has the generator after them; warp 1 walks.
template <class F>
__device__ void r1_fill(R1Ring &R, int32_t *tab, const int32_t *state, int64_t n, Ran1Warp &g, F put) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ int s_batches, s_first;
    int64_t done = 0;
    if (w == 0) {
        g.load(state);
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
            s_first = g.iy >> 26;
        }
    }
    asm volatile("bar.sync 7, 64;" ::: "memory");   // the two warps of a larger CTA
    const int nb = s_batches;
    const int first_key = R.tab[lane] >> 26;
    asm volatile("bar.sync 7, 64;" ::: "memory");
    if (w == 1) {
        if (nb > 0) r1_walk(R, first_key, s_first, nb);
        return;
    }
    if (nb > 0) {
        R1Values v;
        v.begin(R, g);
        constexpr int A = R1_NB / 2;   // batches made ahead
#pragma unroll
        for (int j = 0; j < A; ++j) v.make(R, j);
        bool ok = true;
        for (int b = 0; b < nb && ok; b += A) {
#pragma unroll
            for (int j = 0; j < A; ++j) {
                if (b + j < nb && ok) {
                    ok = v.walked(R, b + j);
                    if (!ok) continue;   // the walk gave up: this warp goes on alone from here
                    put(done + lane, v.take(R, b + j, j));
                    done += 32;
                    v.make(R, j);
                }
            }
        }
        g.idum = v.idum;
        g.iy = v.iy;
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
