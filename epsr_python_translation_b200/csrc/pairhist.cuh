// pairhist.cuh -- a tile of target atoms against one origin atom a thread, into a histogram of the
// distances by pair type in shared memory (the intermolecular pass of atogen,
// ato_manipulation_rev4.py:3780-3850).
//
// What bounds it: instruction issue, 55 instructions a pair of which many issue every other cycle (85%
// of the issue slots of active cycles filled), then the shared-memory adds (2.3 wavefronts a warp).  Distance and bin
// therefore avoid the conversion unit and the division, and the root is branch-free (common.cuh), the pair
// type's row comes from shared memory, four targets are in flight, a tile that counts whole is run
// without comparing molecules, and a pair's closest-contact test compares against the largest contact
// distance before it looks its own up.  The histogram leaves room for few CTAs on an SM, so a CTA is as
// wide as the SM's registers allow (hist_threads): its 256 origins times one to four parts of the tile.
// Intermolecular pass of 2,700 DMSO + 5,300 water, 1,000 origins (230 million pairs): 508 us, 2,800 us with
// one part, division and conversion.  64 boxes of 300 to 30,000 atoms (3.3 billion pairs): 6.2 ms
// against 12.5 ms.
#pragma once

#include "common.cuh"

namespace epsr {

constexpr int PH_ORIGINS = 256;   // origins of a CTA
constexpr int PH_TYPES = 16;      // atom types up to which the pair-type rows are staged

struct PairHist {
    unsigned *hist, *hpot;        // shared: [npairs*ld] bins, [npairs] close contacts
    const int *npairref;          // [ntype*ntype]
    const float *rminex;          // [npairs]
    int ld, ntype, nlim;          // bins 0 <= nint(d/stepcl) < nlim count
    float stepcl, rcp, dmax, rmax;
    Lattice L;
};

// 1/stepcl where nint_index's product is good enough for every distance of a cubic box, else NaN
__host__ __device__ inline float hist_rcp(float stepcl) {
    return stepcl >= 0.87f / 4000.0f ? 1.0f / stepcl : nanf("");
}

// nint(d / stepcl) by the product with the rounded reciprocal, which is within 7.3e-4 of the rounded
// quotient while that is at most 4096: the same integer unless it lies within 1e-3 of a half, which
// `odd` reports (as it does for a NaN)
__device__ __forceinline__ int nint_index(float d, float rcp, bool &odd) {
    const float q = __fmul_rn(d, rcp);
    const float big = __fadd_rn(q, 12582912.0f);
    odd = !(fabsf(__fsub_rn(q, __fsub_rn(big, 12582912.0f))) < 0.499f);
    return __float_as_int(big) - 0x4b400000;
}

// the largest contact distance (a warp's lanes together); NaNs never count
__device__ __forceinline__ float hist_rmax(const float *rminex, int npairs) {
    float r = 0.0f;
    for (int i = threadIdx.x & 31; i < npairs; i += 32) r = fmaxf(r, fabsf(rminex[i]));
    for (int o = 16; o; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
    return r;
}

// The pair types' row starts by (target type, origin type), all threads of the CTA; `cls` [PH_TYPES^2].
__device__ __forceinline__ void hist_stage_types(const PairHist &H, int *cls) {
    if (H.ntype <= PH_TYPES)
        for (int i = threadIdx.x; i < H.ntype * H.ntype; i += blockDim.x)
            cls[i] = H.npairref[(i % H.ntype) * H.ntype + i / H.ntype] * H.ld;
}

// The tile's copy of an atom: its type as the byte offset of its row in `cls` where that is staged.
__device__ __forceinline__ float4 hist_target(const PairHist &H, float4 p) {
    if (H.ntype <= PH_TYPES) p.w = __int_as_float(__float_as_int(p.w) * H.ntype * 4);
    return p;
}

// A tile of n targets, all threads of the CTA, with barriers around: atoms, molecules, and the first and
// last molecule.
__device__ __forceinline__ void hist_stage_tile(const PairHist &H, const float4 *pos, const int *molof, int n,
                                                float4 *tp, int *tm, int *mols) {
    __syncthreads();
    if (threadIdx.x < 2) mols[threadIdx.x] = threadIdx.x ? -1 : 0x7fffffff;
    __syncthreads();
    int lo = 0x7fffffff, hi = -1;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int m = molof[i];
        tp[i] = hist_target(H, pos[i]);
        tm[i] = m;
        lo = min(lo, m);
        hi = max(hi, m);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(mols, lo);
        atomicMax(mols + 1, hi);
    }
    __syncthreads();
}

// SOME: the group may hold targets that don't count
template <int U, bool STAGED, bool SOME>
__device__ __forceinline__ void hist_group(const PairHist &H, float4 p1, int im, bool after, const float4 *tp,
                                           const int *tm, const int *cls, int &uses) {
    float d[U];
    int n[U], base[U];
    bool use[U], odd[U], any = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const float4 p2 = tp[u];
        const int ty = __float_as_int(p2.w);
        use[u] = true;
        if (SOME) {
            const int jm = tm[u];
            use[u] = after ? jm > im : jm != im;
            uses += use[u];
        }
        base[u] = STAGED ? *(const int *)((const char *)cls + ty) : __ldg(cls + ty) * H.ld;
        // xx = x1 - x2 (ato_manipulation_rev4.py:3798); the square does not see the sign
        d[u] = sqrt_unit(dsq_cubic(p2, p1));
        n[u] = nint_index(d[u], H.rcp, odd[u]);
        any |= odd[u];
    }
    if (any) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (odd[u]) n[u] = nint_i(__fdiv_rn(d[u], H.stepcl));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (use[u] && (unsigned)n[u] < (unsigned)H.nlim) atomicAdd(H.hist + base[u] + 2 + n[u], 1u);
        const float dd = __fmul_rn(d[u], H.dmax);
        if (use[u] && dd < H.rmax) {
            const int icref = base[u] / H.ld;
            if (dd < fabsf(__ldg(H.rminex + icref))) atomicAdd(H.hpot + icref, 1u);
        }
    }
}

template <bool STAGED, bool SOME>
__device__ __forceinline__ int hist_part(const PairHist &H, float4 p1, int im, bool after, const float4 *tp,
                                         const int *tm, int q0, int q1, const int *cls) {
    int uses = 0, q = q0;
    for (; q + 4 <= q1; q += 4) hist_group<4, STAGED, SOME>(H, p1, im, after, tp + q, tm + q, cls, uses);
    for (; q < q1; ++q) hist_group<1, STAGED, SOME>(H, p1, im, after, tp + q, tm + q, cls, uses);
    return SOME ? uses : max(q1 - q0, 0);
}

// Cells that are not cubic: one target at a time, by the general distance and the division, and none for a target
// that does not count.  There the latency of three divisions and a root a pair bounds a thread, so that groups of four,
// a second loop for the lanes whose tile counts whole, and distances to targets that don't count all cost time (the
// cubic form with the general distance: sheared boxes of 200 DMSO + 400 water and 5,000 water, whole passes of 298
// and 741 us; 227 and 517 so, with a CTA for every tile).
template <bool STAGED>
__device__ __forceinline__ int hist_any_cell(const PairHist &H, float4 p1, int im, bool after, const float4 *tp,
                                             const int *tm, int q0, int q1, const int *cls) {
    int uses = 0;
    for (int q = q0; q < q1; ++q) {
        const int jm = tm[q];
        if (after ? jm <= im : jm == im) continue;
        ++uses;
        const float4 p2 = tp[q];
        const int ty = __float_as_int(p2.w);
        const int base = STAGED ? *(const int *)((const char *)cls + ty) : __ldg(cls + ty) * H.ld;
        const float d = dist_f(H.L, __fsub_rn(p1.x, p2.x), __fsub_rn(p1.y, p2.y), __fsub_rn(p1.z, p2.z));
        const int n = nint_i(__fdiv_rn(d, H.stepcl));
        if ((unsigned)n < (unsigned)H.nlim) atomicAdd(H.hist + base + 2 + n, 1u);
        const float dd = __fmul_rn(d, H.dmax);
        if (dd < H.rmax) {
            const int icref = base / H.ld;
            if (dd < fabsf(__ldg(H.rminex + icref))) atomicAdd(H.hpot + icref, 1u);
        }
    }
    return uses;
}

// Targets q0..q1-1 of a tile (its first and last molecule in `mols`) against origin p1 of molecule im:
// the molecules after im only, or all others.  Returns the number of pairs.  A tile that counts
// whole, as nearly all do, is run without the comparison of the molecules.
template <bool CUBIC, bool STAGED>
__device__ __forceinline__ int hist_tile(const PairHist &H, float4 p1, int im, bool after, const float4 *tp,
                                         const int *tm, int q0, int q1, const int *mols, const int *cls_sm) {
    const int it = __float_as_int(p1.w);
    const int *cls = STAGED ? cls_sm + it : H.npairref + it * H.ntype;
    if (!CUBIC) return hist_any_cell<STAGED>(H, p1, im, after, tp, tm, q0, q1, cls);
    if (mols[0] > im || (!after && mols[1] < im))
        return hist_part<STAGED, false>(H, p1, im, after, tp, tm, q0, q1, cls);
    return hist_part<STAGED, true>(H, p1, im, after, tp, tm, q0, q1, cls);
}

// Threads of a CTA with `shm` bytes of shared memory: 64 registers a thread let 1,024 share an SM.
inline int hist_threads(size_t shm) { return shm > 112 * 1024 ? 1024 : shm > 55 * 1024 ? 512 : 256; }

}  // namespace epsr
