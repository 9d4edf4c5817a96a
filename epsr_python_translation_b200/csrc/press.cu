// press.cu -- press (ato_manipulation_rev4.py:3903-4062): intermolecular energy and virial of
// the stored pairs, without three-body terms or coordination constraints.
//
// One CTA per molecule im (all but the last), one thread per stored partner slot: for a
// partner jm > im the thread sums, over im's atoms (outer) and jm's atoms (inner), the
// energy enwt + enpot into a float32 ergold and the virial terms into ergnew -- a float32
// add of the EP term prwt, then a double add of the reference-potential term prpot, stored
// back as float32 -- exactly as the reference (:3960-4040).  Pairs count only while the
// bin iz <= npt1.  The reduction then sums ergold in float32 and ergnew in double over
// (im, slot) in store order (:4041-4044): one thread, sequentially, for the reference's
// bits (strict); or the CTA adds its molecule's terms in double and one CTA the molecules (fast: no
// term goes through memory.  814,000 pairs: 340 us for both kernels, 777 us with one CTA over all terms).
#include <string.h>

#include "common.cuh"

namespace epsr {

constexpr int PR_THREADS = 256;
constexpr int PR_MAXAT = 64;   // atoms of a molecule held in shared memory

struct PressDev {
    Lattice L;
    const float4 *tab;         // [npairs*ld] {xavs, xavs1, ecoul, ecoul1}
    const float *xstar;        // [ld]
    float stepcl, rcp;         // and step_rcp of it
    int npt1, ld, ntype, M;
    const int32_t *naf, *nato, *npairref, *nergpairm, *molergpair;
    const float *xadd, *yadd, *zadd;
    const float4 *pos;         // absolute atom positions, type bits in .w
    float *ergold, *ergnew;    // [nmol*M]
    double *sums;              // [2] {sumc, presst}
};

// a double in two words of a float array (rows of odd length leave them unaligned)
__device__ __forceinline__ void put_double(float *p, double v) {
    p[0] = __int_as_float(__double2loint(v));
    p[1] = __int_as_float(__double2hiint(v));
}
__device__ __forceinline__ double get_double(const float *p) {
    return __hiloint2double(__float_as_int(p[1]), __float_as_int(p[0]));
}

// x - nint(x) (half away from zero) of a difference of box-fraction coordinates, on the adder
__device__ __forceinline__ float wrap_small(float x) {
    const float r = __fsub_rn(x, rint_small(x));
    return fabsf(r) == 0.5f ? copysignf(0.5f, -x) : r;
}

// one atom pair's terms; branch-free: the tables are read at iz clamped into 2..npt1 and `in` tells
// whether the pair counts, so several pairs' loads are in flight
struct PairTerms {
    float enwt, enpot, prwt, prpot;
    bool in;
};
template <bool CUBIC>
__device__ __forceinline__ PairTerms pair_terms(const PressDev &P, float4 p1, float4 p2, const int32_t *prow, float xc,
                                                float yc, float zc) {
    float xdif = __fsub_rn(p2.x, p1.x), ydif = __fsub_rn(p2.y, p1.y), zdif = __fsub_rn(p2.z, p1.z);
    if (CUBIC) {
        xdif = wrap_small(xdif);
        ydif = wrap_small(ydif);
        zdif = wrap_small(zdif);
    } else {
        minimagec(P.L, xdif, ydif, zdif);
    }
    const float dsq = __fadd_rn(__fadd_rn(__fmul_rn(xdif, xdif), __fmul_rn(ydif, ydif)), __fmul_rn(zdif, zdif));
    const float dtest = CUBIC ? sqrt_unit(dsq) : __fsqrt_rn(dsq);
    const int iz = (CUBIC ? bin_index(dtest, P.stepcl, P.rcp) : ifix(__fdiv_rn(dtest, P.stepcl))) + 2;
    const int izc = min(max(iz, 2), P.npt1);
    const int icref = __ldg(prow + __float_as_int(p2.w));
    const float4 t = __ldg(P.tab + (size_t)icref * P.ld + izc);       // bin iz
    const float4 tm = __ldg(P.tab + (size_t)icref * P.ld + izc - 1);  // bin iz-1
    const float dtdif = __fsub_rn(dtest, __ldg(P.xstar + izc));
    const float prfac = dtest > 0.0f ? __fdiv_rn(__fadd_rn(__fadd_rn(__fmul_rn(xc, xdif), __fmul_rn(yc, ydif)),
                                                           __fmul_rn(zc, zdif)),
                                                 dtest)
                                     : 0.0f;
    PairTerms r;
    r.in = iz == izc;
    r.enpot = __fadd_rn(t.z, __fmul_rn(t.w, dtdif));
    r.prpot = __fmul_rn(__fmul_rn(0.5f, __fadd_rn(t.w, tm.w)), prfac);
    r.enwt = __fadd_rn(t.x, __fmul_rn(t.y, dtdif));
    r.prwt = __fmul_rn(__fmul_rn(0.5f, __fadd_rn(t.y, tm.y)), prfac);
    return r;
}

template <bool CUBIC>
__global__ void __launch_bounds__(PR_THREADS) press_pairs_kernel(PressDev P, int fast) {
    extern __shared__ int list[];   // [M] slots with a partner jm > im, by partner atom count
    __shared__ float4 sa[PR_MAXAT];
    __shared__ int bk[PR_MAXAT + 2];
    const int im = blockIdx.x;
    const int a0 = P.naf[im], na = P.nato[im];
    const bool in_smem = na <= PR_MAXAT;   // larger molecules are read from global memory
    if (in_smem)
        for (int i = threadIdx.x; i < na; i += blockDim.x) sa[i] = P.pos[a0 + i];
    for (int i = threadIdx.x; i < PR_MAXAT + 2; i += blockDim.x) bk[i] = 0;
    __syncthreads();
    const float xc1 = P.xadd[im], yc1 = P.yadd[im], zc1 = P.zadd[im];
    const int nn = P.nergpairm[im];
    const size_t row = (size_t)im * P.M;
    // slots whose partner comes later are evaluated, listed by the partner's atom count so the
    // lanes of a warp run loops of the same length; the others hold 0
    auto nb_of = [&](int s) -> int {
        const int jm = P.molergpair[row + s];
        return jm > im ? min(P.nato[jm], PR_MAXAT) : 0;
    };
    for (int s = threadIdx.x; s < nn; s += blockDim.x) {
        const int nb = nb_of(s);
        if (nb > 0) {
            atomicAdd(&bk[nb], 1);
        } else {
            P.ergold[row + s] = 0.0f;
            P.ergnew[row + s] = 0.0f;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {   // bk[b] -> first list position of atom count b; bk[PR_MAXAT+1] = total
        int a = 0;
        for (int b = 0; b <= PR_MAXAT; ++b) {
            const int t = bk[b];
            bk[b] = a;
            a += t;
        }
        bk[PR_MAXAT + 1] = a;
    }
    __syncthreads();
    for (int s = threadIdx.x; s < nn; s += blockDim.x) {
        const int nb = nb_of(s);
        if (nb > 0) list[atomicAdd(&bk[nb], 1)] = s;
    }
    __syncthreads();
    const int total = bk[PR_MAXAT + 1];
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
        const int s = list[q];
        const int jm = P.molergpair[row + s];
        float eo = 0.0f, en = 0.0f;
        {
            // separation of the centres (the same for every atom pair of im, jm)
            float xcdif = __fsub_rn(P.xadd[jm], xc1), ycdif = __fsub_rn(P.yadd[jm], yc1),
                  zcdif = __fsub_rn(P.zadd[jm], zc1);
            minimagec(P.L, xcdif, ycdif, zcdif);
            const int b0 = P.naf[jm], nb = P.nato[jm];
            for (int ia = 0; ia < na; ++ia) {
                const float4 p1 = in_smem ? sa[ia] : __ldg(P.pos + a0 + ia);
                const int32_t *prow = P.npairref + __float_as_int(p1.w) * P.ntype;
#pragma unroll 2
                for (int j = 0; j < nb; ++j) {
                    const PairTerms t = pair_terms<CUBIC>(P, p1, __ldg(P.pos + b0 + j), prow, xcdif, ycdif, zcdif);
                    if (t.in) {
                        // the reference adds the float32 prwt and then, in double, prpot, and stores
                        // float32: a float added to a float in double and rounded to float is the
                        // float sum (exact in double unless the smaller is below 2^-29 of the larger,
                        // when both round to the larger)
                        eo = __fadd_rn(__fadd_rn(eo, t.enwt), t.enpot);
                        en = __fadd_rn(__fadd_rn(en, t.prwt), t.prpot);
                    }
                }
            }
        }
        P.ergold[row + s] = eo;
        P.ergnew[row + s] = en;
    }
    if (!fast) return;
    // the molecule's sums, by slot, so that they don't depend on the lists' order; the warps' parts lie where
    // the atoms were, since the list may take all the shared memory that is left
    __syncthreads();
    double *r0 = (double *)sa, *r1 = r0 + PR_THREADS / 32;
    double se = 0.0, sp = 0.0;
    for (int s = threadIdx.x; s < nn; s += blockDim.x) {
        se += (double)P.ergold[row + s];
        sp += (double)P.ergnew[row + s];
    }
    se = warp_sum_d(se);
    sp = warp_sum_d(sp);
    if ((threadIdx.x & 31) == 0) {
        r0[threadIdx.x >> 5] = se;
        r1[threadIdx.x >> 5] = sp;
    }
    __syncthreads();
    if (threadIdx.x == 0 && P.M >= 2) {   // into the row's first two words of each array, now read
        double a = 0.0, b = 0.0;
        for (int w = 0; w < PR_THREADS / 32; ++w) {
            a += r0[w];
            b += r1[w];
        }
        put_double(P.ergold + row, a);
        put_double(P.ergnew + row, b);
    }
}

// sumc in float32 and presst in double over (im, slot) in store order, one thread
__global__ void press_sum_strict_kernel(PressDev P, int nmol) {
    float sumc = 0.0f;
    double presst = 0.0;
    for (int im = 0; im < nmol - 1; ++im) {
        const size_t row = (size_t)im * P.M;
        const int nn = P.nergpairm[im];
        for (int s = 0; s < nn; ++s) {
            sumc = __fadd_rn(sumc, P.ergold[row + s]);
            presst = __dadd_rn(presst, (double)P.ergnew[row + s]);
        }
    }
    P.sums[0] = (double)sumc;
    P.sums[1] = presst;
}

// both sums over the molecules' in double (one CTA, a fixed order)
__global__ void __launch_bounds__(1024) press_sum_fast_kernel(PressDev P, int nmol) {
    __shared__ double r0[32], r1[32];
    double a = 0.0, b = 0.0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    for (int im = threadIdx.x; im < nmol - 1; im += blockDim.x) {
        if (P.M >= 2) {
            a += get_double(P.ergold + (size_t)im * P.M);
            b += get_double(P.ergnew + (size_t)im * P.M);
        } else if (P.nergpairm[im] > 0) {   // a row of one slot has no room for a sum, and is its sum
            a += (double)P.ergold[im];
            b += (double)P.ergnew[im];
        }
    }
    a = warp_sum_d(a);
    b = warp_sum_d(b);
    if (lane == 0) {
        r0[wid] = a;
        r1[wid] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < nwarp; ++w) {
            ta += r0[w];
            tb += r1[w];
        }
        P.sums[0] = (double)(float)ta;
        P.sums[1] = tb;
    }
}

}  // namespace epsr

using namespace epsr;

static inline size_t pr_al256(size_t x) { return (x + 255) & ~(size_t)255; }

extern "C" int64_t epsr_press_scratch_bytes(int32_t nmol, int32_t nnbrefmax) {
    return (int64_t)(2 * pr_al256(sizeof(float) * (size_t)nmol * (size_t)nnbrefmax) + pr_al256(sizeof(double) * 2));
}

extern "C" int epsr_press(const epsr_box_t *box, const epsr_store_t *store, int32_t npt1, void *scratch,
                          int64_t scratch_bytes, int32_t strict, double *sums_host, void *stream) {
    if (!box || !store || !scratch || !sums_host || !box->pos) {
        epsr_set_error("epsr_press: null pointer");
        return EPSR_ERR_ARG;
    }
    if (npt1 < 2 || npt1 >= box->ld) {
        epsr_set_error("epsr_press: npt1 %d outside 2..ld-1 (ld %d)", npt1, box->ld);
        return EPSR_ERR_ARG;
    }
    const int nmol = box->nmol, M = store->nnbrefmax;
    if (scratch_bytes < epsr_press_scratch_bytes(nmol, M)) {
        epsr_set_error("epsr_press: scratch too small");
        return EPSR_ERR_CAPACITY;
    }
    cudaStream_t s = (cudaStream_t)stream;
    PressDev P;
    memset(&P, 0, sizeof(P));
    P.L.cubic = box->cubic;
    P.L.alatx = box->lat[0];
    P.L.blatx = box->lat[1];
    P.L.clatx = box->lat[2];
    P.L.blaty = box->lat[3];
    P.L.claty = box->lat[4];
    P.L.clatz = box->lat[5];
    P.tab = (const float4 *)box->tab;
    P.xstar = box->xstar;
    P.stepcl = box->stepcl;
    P.rcp = step_rcp(box->stepcl, npt1);
    P.npt1 = npt1;
    P.ld = box->ld;
    P.ntype = box->ntype;
    P.M = M;
    P.naf = box->naf;
    P.nato = box->nato;
    P.npairref = box->npairref;
    P.nergpairm = store->nergpairm;
    P.molergpair = store->molergpair;
    P.xadd = box->xadd;
    P.yadd = box->yadd;
    P.zadd = box->zadd;
    P.pos = (const float4 *)box->pos;
    char *p = (char *)scratch;
    P.ergold = (float *)p;
    p += pr_al256(sizeof(float) * (size_t)nmol * M);
    P.ergnew = (float *)p;
    p += pr_al256(sizeof(float) * (size_t)nmol * M);
    P.sums = (double *)p;
    int rc = epsr_box_positions(box, stream);
    if (rc) return rc;
    if (nmol > 1) {
        const size_t list_bytes = sizeof(int) * (size_t)M;
        if (list_bytes > 48 * 1024) {
            EPSR_SMEM_OPTIN(press_pairs_kernel<true>);
            EPSR_SMEM_OPTIN(press_pairs_kernel<false>);
        }
        auto *pairs = box->cubic ? press_pairs_kernel<true> : press_pairs_kernel<false>;
        pairs<<<nmol - 1, PR_THREADS, list_bytes, s>>>(P, strict ? 0 : 1);
        EPSR_CUDA(cudaGetLastError());
        if (strict) press_sum_strict_kernel<<<1, 1, 0, s>>>(P, nmol);
        else press_sum_fast_kernel<<<1, 1024, 0, s>>>(P, nmol);
        EPSR_CUDA(cudaGetLastError());
        EPSR_D2H(sums_host, P.sums, sizeof(double) * 2, s);
    } else {
        sums_host[0] = 0.0;
        sums_host[1] = 0.0;
    }
    return EPSR_OK;
}
