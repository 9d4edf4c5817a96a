// fitexp.cu -- fit_expansion (epsr_standalone_rev3.py:4806-4921) on one thread-block cluster.
//
// The Monte Carlo fit is a chain of trials: perturb every coefficient (one ran1 draw each),
// evaluate chi^2 over all Q rows, Metropolis-accept (one more draw when 0 < exponent <= 20),
// smooth the coefficients every nfreq acceptances (smoop auxiliary_routines.py:744).  One
// launch fits any number of data sets in turn on the same basis, continuing one ran1
// stream, as the reference's successive calls do.
//
// Layout.  The basis rows are split over the CTAs of a cluster; a thread evaluates its row per
// trial (expand :4924, the sequential clamped sum of a row) with the row's first 128 terms in its
// registers (64 in the wide form of the CTA) and the rest in shared memory, four terms to a
// 16-byte word.  Every partial
// sum of a row is bounded by the row's L1 norm times the largest |coefficient|; when that
// bound stays below the clamp level (e^25) the clamp cannot act and the plain sequential
// sum is the reference's value, otherwise the row is summed with the clamp.  The CTAs
// exchange their chi^2 contributions through distributed shared memory: each stores its
// part (a double partial, or every residual for the reference's sequential float sum) into
// every CTA, the stores completing their bytes on that CTA's mbarrier (no release stands between a
// store and its signal).  Every warp of every CTA waits for the parts, forms the same chi^2 and
// takes the same decision, so a trial passes one barrier of the CTA, after the coefficients are
// perturbed (600 rows x 116 terms, double sums: 3,390 cycles a trial while warp 0 collected its CTA's
// sums and published the decision behind two more barriers, 3,240 now: 1,100 the row's 116 additions
// and their loads, 750 the two trees of double additions, 40 cycles each, the rest the perturbation,
// the exchange and the test, and the stream close behind).  The strict sum is one chain of additions over all
// rows, 4.7 cycles each (1,000 rows x 97 terms: 21,700 cycles a trial when every fourth row waited for
// its word, 8,340 now).
//
// ran1.  The chain is sequential and one trial's values outlast one trial's arithmetic, so it has
// an SM to itself: the cluster's last CTA generates the stream with three warps (ran1_pair.cuh) and
// stores the values into a ring in every worker CTA's shared memory, running ahead of the trials
// (bounded by the ring).  On a warp of each worker CTA, beside its rows' shared-memory reads, the
// same chain took 46 cycles a value instead of 27.  At the end the state the reference leaves after
// exactly the values the fit consumed is rebuilt from the generator's checkpoints.
//
// Every wait (ring, exchange, ring space) is bounded in time: on timeout the kernel records
// status 1, stops the fit and returns.
#include <cooperative_groups.h>

#include <algorithm>

#include "ran1_pair.cuh"

namespace cg = cooperative_groups;

namespace epsr {

constexpr int FX_MAXT = 512;                    // most threads of a worker CTA (256 when rows and terms fit)
constexpr int FX_SLOTS = FX_MAXT;               // row / coefficient slots of a worker CTA at most
constexpr int FX_ROWS = 160;                    // rows a CTA takes while the cluster has CTAs left
constexpr int FX_MAXW = 8;                      // worker CTAs of a cluster
// leading quads of a row held in its thread's registers: the narrow CTA has room for 128 terms
__host__ __device__ constexpr int fx_rq(int threads) { return threads == FX_MAXT ? 16 : 32; }
constexpr int FX_RING = 2048;                   // ran1 values held per worker CTA (power of two)
constexpr int FX_CK = 32;                       // generator checkpoints (power of two)
constexpr int FX_CKE = 8;                       // batches between checkpoints (power of two)
constexpr int FX_CKW = 36;                      // ints per checkpoint: idum, iy, iv[32], pad[2]
constexpr unsigned long long FX_WAIT_NS = 2000000000ull;  // a wait gives up after 2 s

struct FxDev {
    const float *expr;        // expr[(i-1)*nterms + m] (1-based flat, row-major by Q)
    const float *yin;         // [nprob][npt+1]
    float *yout;              // [nprob][npt+1]
    float *wt_g, *wtold_g;    // [nprob][nterms+1]
    float *scal;              // [nprob][4] {stepr, acceptr, rejrat, chisq}
    long long *trials;        // [nprob]
    int *status;              // [1]: 0 ok, 1 a bounded wait gave up
    int nprob, nmin, npt, ncfirst, nterms, nits, nfreq, strict, rpc, nw;
    int32_t *ran1;
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// a store into another CTA of the cluster that completes its bytes on that CTA's mbarrier
__device__ __forceinline__ void st_async_f32(uint32_t a, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
                 "r"(__float_as_int(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async_f64(uint32_t a, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_cl_s64(uint32_t a, long long v) {
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_cl_s64(uint32_t a, long long v) {
    asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void st_release_cl_s32(uint32_t a, int v) {
    asm volatile("st.release.cluster.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ long long ld_relaxed_s64(const long long *p) {
    long long v;
    asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];" : "=l"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ int ld_acquire_s32(const int *p) {
    int v;
    asm volatile("ld.acquire.cluster.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}
// Barrier of a worker CTA after code in which a warp may have diverged (a bounded spin, a branch
// on the thread index): the warp is reconverged first, because the barrier requires every thread
// of a warp to arrive together.
__device__ __forceinline__ void block_sync() {
    __syncwarp();
    __syncthreads();
}
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct FxShared {                 // statically sized control block (one per CTA)
    long long cons;               // generator: lowest stream index the workers may still read
    int done;                     // generator: set by the workers when the fit is over
    int abort;
    float wmx;                    // largest |wt| of the perturbed terms
};

// quads of a row, in whole groups of four (terms past nterms are zero on both sides)
__host__ __device__ inline int fx_ntq(int nt) { return (nt + 15) / 16 * 4; }
// quads of a row kept in shared memory (those after the registers')
__host__ __device__ inline int fx_nsq(int nt, int threads) {
    return fx_ntq(nt) > fx_rq(threads) ? fx_ntq(nt) - fx_rq(threads) : 0;
}
// floats per exchange buffer: every row of the cluster, padded to whole 16-byte words so the
// second buffer starts 16-byte aligned (it is read four rows at a time)
__host__ __device__ inline int fx_gstride(int nw, int rpc) { return (nw * rpc + 3) & ~3; }

size_t fx_smem_bytes(int nt, int rpc, int nw, int threads) {
    const int ntq = fx_ntq(nt);
    size_t b = 0;
    b += 16 * (size_t)fx_nsq(nt, threads) * rpc;                 // ex4
    b += sizeof(float) * (4 + 4 * ((size_t)ntq + 4));   // wt (wt + 1 16-byte aligned, a group past the end)
    b += sizeof(float) * (size_t)(nt + 1);              // wtold
    b = (b + 15) & ~(size_t)15;
    b += sizeof(unsigned long long) * FX_RING;          // ring
    b = (b + 15) & ~(size_t)15;
    b += sizeof(float) * 2 * (size_t)fx_gstride(nw, rpc);   // gat[2][gstride]
    b = (b + 15) & ~(size_t)15;
    b += sizeof(double) * 2 * (size_t)nw * ((rpc + 31) / 32);   // parts[2][nw][warps with rows]
    b += sizeof(uint64_t) * 2;                          // exchange mbarriers
    return b;
}

struct FxGen {                    // the generator CTA's shared memory
    R1Ring pair;
    int32_t tab[34];
    long long ckpos[FX_CK];
    int32_t ck[FX_CK][FX_CKW];    // idum, iy, iv[32] before a batch
    int first, idum, go;
};

// The generator CTA: values 0, 1, ... of the stream into the workers' rings until they are done,
// then the state after the values they took.  Warps 0 to 2 call.
__device__ void fx_generate(const FxDev &F, FxGen &G, FxShared &S, unsigned long long *ring) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x >= 32) {
        Ran1Warp h;
        h.load(F.ran1);   // its powers of IA
        asm volatile("bar.sync 7, 96;" ::: "memory");
        if (!*(volatile int *)&G.go) return;
        if (threadIdx.x < 64) r1_walk(G.pair, G.pair.tab[lane] >> 26, *(volatile int *)&G.first, 0x7fffffff);
        else r1_make(G.pair, *(volatile int *)&G.idum, h.mul, 0x7fffffff);
        return;
    }
    Ran1Warp g;
    g.load(F.ran1);
    const int32_t mcall0 = F.ran1[2];
    long long pos = 0, nb = 0;
    uint32_t dst[FX_MAXW];
#pragma unroll
    for (int d = 0; d < FX_MAXW; ++d) dst[d] = d < F.nw ? map_rank(smem_addr(ring), (uint32_t)d) : 0u;
    auto push = [&](int cnt, int32_t mine) {
        const long long q = pos + lane;
        const long long w = (long long)(((unsigned long long)(uint32_t)(q + 1) << 32) |
                                        (unsigned long long)__float_as_uint(ran1_out(mine)));
        if (lane < cnt)
#pragma unroll
            for (int d = 0; d < FX_MAXW; ++d)
                if (d < F.nw) st_cl_s64(dst[d] + 8u * (uint32_t)(q & (FX_RING - 1)), w);
        pos += cnt;
    };
    auto checkpoint = [&](int32_t idum, int32_t iy, int32_t iv) {   // the state before a batch
        if ((nb++ & (FX_CKE - 1)) == 0) {
            const int slot = (int)(((nb - 1) / FX_CKE) & (FX_CK - 1));
            G.ck[slot][2 + lane] = iv;
            if (lane == 0) {
                G.ck[slot][0] = idum;
                G.ck[slot][1] = iy;
                G.ckpos[slot] = pos;
            }
        }
    };
    // room for a batch in every ring; false when the workers are done (or gave up: 2 s without room).  The
    // values before the workers' cursor have been read, as the trial they decide depends on them, so
    // no fence stands between the cursor and a slot's next value (a releasing store a trial: 3% of a fit).
    long long limit = FX_RING;
    auto room = [&]() -> bool {
        unsigned long long t0 = 0;
        while (true) {
            __syncwarp();
            if (*(volatile int *)&S.done) return false;
            if (limit - pos >= 32) return true;
            limit = ld_relaxed_s64(&S.cons) + FX_RING;
            if (limit - pos >= 32) return true;
            int give_up = 0;
            if (lane == 0) {
                const unsigned long long t = now_ns();
                if (t0 == 0) t0 = t;
                else if (t - t0 > FX_WAIT_NS) {
                    atomicExch(F.status, 1);
                    give_up = 1;
                }
            }
            if (__shfl_sync(0xffffffffu, give_up, 0)) return false;
            __nanosleep(64);
        }
    };
    for (int i = lane; i < FX_CK; i += 32) G.ckpos[i] = -1;
    __syncwarp();
    bool more = true;
    // until the stream is clean: one batch as a rule (the initialisation happens inside); a
    // degenerate stream stays here
    while (more && !(g.clean && g.idum > 0)) {
        more = room();
        if (!more) break;
        checkpoint(g.idum, g.iy, g.iv);
        int32_t mine;
        const int cnt = g.next(32, mine, G.tab);
        push(cnt, mine);
    }
    G.pair.tab[lane] = g.iv;
    if (lane == 0) {
        r1_init(G.pair);
        *(volatile int *)&G.first = g.iy >> 26;
        *(volatile int *)&G.idum = g.idum;
        *(volatile int *)&G.go = more;
    }
    __syncwarp();
    asm volatile("bar.sync 7, 96;" ::: "memory");
    if (more) {
        R1Values v;
        v.begin(g);
        while (room()) {
            if (!v.walked(G.pair)) {
                if (lane == 0) atomicExch(F.status, 1);
                break;
            }
            if ((nb & (FX_CKE - 1)) == 0) checkpoint(v.idum(), v.iy(), G.pair.tab[lane]);
            else ++nb;
            push(32, v.take(G.pair));
        }
        v.leave(G.pair);
    }
    // the state after exactly the values taken, from the last checkpoint at or before it (or from
    // the launch's state when none is left)
    __syncwarp();
    if (lane == 0 && ld_acquire_s32(&S.done) == 1) {
        const long long cursor = S.cons;   // stored before done
        int best = -1;
        for (int k = 0; k < FX_CK; ++k)
            if (G.ckpos[k] >= 0 && G.ckpos[k] <= cursor && (best < 0 || G.ckpos[k] > G.ckpos[best])) best = k;
        Ran1 R;
        long long from = 0;
        ran1_load(R, F.ran1);
        if (best >= 0) {
            R.idum = G.ck[best][0];
            R.iy = G.ck[best][1];
            for (int i = 0; i < 32; ++i) R.iv[i] = G.ck[best][2 + i];
            from = G.ckpos[best];
        }
        for (long long k = from; k < cursor; ++k) ran1_next(R);
        R.mcall = (int32_t)((uint32_t)mcall0 + (uint32_t)cursor);
        ran1_store(R, F.ran1);
    }
}

template <int T>
__global__ void __launch_bounds__(T, 1) fitexp_cluster_kernel(FxDev F) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int nw = F.nw;                                // worker CTAs; rank nw generates
    extern __shared__ __align__(16) unsigned char fx_raw[];
    __shared__ FxShared S;
    __shared__ FxGen G;
    const int nt = F.nterms, rpc = F.rpc, ntq = fx_ntq(nt);
    constexpr int FX_RQ = fx_rq(T);
    const int nsq = fx_nsq(nt, T);
    // [nsq*rpc]: ex4[q*rpc + r] = terms 4(FX_RQ+q)..4(FX_RQ+q)+3 of row r
    float4 *ex4 = (float4 *)fx_raw;
    size_t off = 16 * (size_t)nsq * rpc;
    float *wt = (float *)(fx_raw + off) + 3;            // wt[0..4*ntq]; wt + 1 is 16-byte aligned
    float *wtold = wt + 1 + 4 * (ntq + 4);                    // [nt+1]
    off = ((size_t)((unsigned char *)(wtold + nt + 1) - fx_raw) + 15) & ~(size_t)15;
    // [FX_RING] stream values, each with its position + 1 in the high word, so a reader knows
    // from the one 8-byte load whether the value it wants is there yet
    unsigned long long *ring = (unsigned long long *)(fx_raw + off);
    off = ((size_t)((unsigned char *)(ring + FX_RING) - fx_raw) + 15) & ~(size_t)15;
    float *gat = (float *)(fx_raw + off);               // [2][gstride] residuals by global row
    off = ((off + sizeof(float) * 2 * (size_t)fx_gstride(nw, rpc)) + 15) & ~(size_t)15;
    const int nwr = (rpc + 31) / 32, nparts = nw * nwr; // warps of a CTA that have rows; their sums
    double *parts = (double *)(fx_raw + off);           // [2][nparts]
    uint64_t *xbar = (uint64_t *)(parts + 2 * nparts);  // [2]

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    volatile FxShared *vs = &S;
    if (rank == nw) {
        if (tid == 0) {
            S.cons = 0;
            S.done = 0;
        }
        cl.sync();
        if (tid < 96) fx_generate(F, G, S, ring);
        __syncwarp();
        cl.sync();   // no CTA leaves while others may still write into its shared memory
        return;
    }
    const int row0 = 1 + rank * rpc;                    // first (1-based) row of this CTA
    const int nrow = max(0, min(rpc, F.npt - row0 + 1));
    for (int idx = tid; idx < nsq * rpc; idx += blockDim.x) {
        const int q = idx / rpc, r = idx - q * rpc;
        float e[4];
        for (int j = 0; j < 4; ++j) {
            const int m = 4 * (FX_RQ + q) + j;          // 0-based term
            e[j] = (r < nrow && m < nt) ? F.expr[1 + (size_t)(row0 - 1 + r) * nt + m] : 0.0f;
        }
        ex4[idx] = make_float4(e[0], e[1], e[2], e[3]);
    }
    for (int i = tid; i <= 4 * (ntq + 4); i += blockDim.x) wt[i] = 0.0f;   // terms past nterms stay zero
    float e1 = 0.0f;                                    // this row's sum over terms of |basis value|
    for (int m = 0; m < nt && tid < nrow; ++m) e1 = __fadd_ru(e1, fabsf(F.expr[1 + (size_t)(row0 - 1 + tid) * nt + m]));
    for (int i = tid; i < FX_RING; i += blockDim.x) ring[i] = 0ull;   // no position yet
    if (tid == 0) {
        S.abort = 0;
        mbar_init(&xbar[0], 1);
        mbar_init(&xbar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cl.sync();
    const uint32_t gen_cons = map_rank(smem_addr(&S.cons), (uint32_t)nw), gen_done = map_rank(smem_addr(&S.done), (uint32_t)nw);

    const float summax = exp_r(25.0f);
    const int K = nt - F.ncfirst + 1;                   // draws per trial
    const int slot = tid;                               // row / coefficient slot of this thread
    const int ic = slot < K ? F.ncfirst + slot : -1;   // coefficient this thread perturbs
    // the first FX_RQ quads of this thread's row (row `slot`), in registers for the launch
    float4 rq[FX_RQ];
#pragma unroll
    for (int k = 0; k < FX_RQ; ++k) {
        float e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (slot < nrow) {
            for (int j = 0; j < 4; ++j) {
                const int m = 4 * k + j;
                if (m < nt) e[j] = F.expr[1 + (size_t)(row0 - 1 + slot) * nt + m];
            }
        }
        rq[k] = make_float4(e[0], e[1], e[2], e[3]);
    }

    // stream value idx, once the generator has written it (a bounded wait, given up at once
    // after an abort)
    auto get = [&](long long idx) -> float {
        const volatile unsigned long long *e = ring + (idx & (FX_RING - 1));
        const uint32_t want = (uint32_t)(idx + 1);
        unsigned long long v = *e;
        if ((uint32_t)(v >> 32) != want) {
            const unsigned long long t0 = now_ns();
            for (int n = 1;; ++n) {
                v = *e;
                if ((uint32_t)(v >> 32) == want) break;
                if (n & 31) continue;
                if (vs->abort) break;
                if (now_ns() - t0 > FX_WAIT_NS) {
                    atomicExch(F.status, 1);
                    vs->abort = 1;
                    break;
                }
            }
        }
        return __uint_as_float((uint32_t)v);
    };

    // state of the trial loop (the same in every worker thread)
    long long cursor = 0;
    float chisqold = 0.0f, accept = 0.0f, racc = 0.0f;
    int icount = 0;
    float yrow = 0.0f;                                  // this row's data
    float wfix = 0.0f;                                  // largest |wt| of the unperturbed terms 1..ncfirst-1

    // the largest |wt| over the perturbed terms (thread 0; a barrier follows)
    auto wmax_all = [&]() {
        float b = 0.0f;
        for (int m = F.ncfirst; m <= nt; ++m) b = fmaxf(b, fabsf(wt[m]));
        vs->wmx = b;
    };
    // smoop(ncfirst, nterms, 1, wt) (:4882-4893; thread 0; a barrier follows)
    auto smooth = [&]() {
        const int n1 = F.ncfirst, n2 = nt;
        if (!(n2 - 2 < n1)) {
            float sm_ = 0.0f, sn = wt[n1];
            float sum1 = __fmul_rn(0.25f, __fadd_rn(sm_, sn));
            for (int i = n1; i <= n2; ++i) {
                sm_ = sn;
                sn = (i + 1) <= n2 ? wt[i + 1] : 0.0f;
                const float sum2 = __fmul_rn(0.25f, __fadd_rn(sm_, sn));
                wt[i] = __fadd_rn(sum1, sum2);
                sum1 = sum2;
            }
        }
        wmax_all();
    };
    // The Metropolis test (:4871-4880) of trial chi^2 cn, u the stream's next value; draw: whether
    // the test took it.  The sign of exp(-x) - u needs neither the division nor the exponential
    // exact but near a tie.
    auto metropolis = [&](float cn, float u, bool &draw) -> bool {
        const float num = __fsub_rn(cn, chisqold);
        draw = false;
        if (num <= 0.0f && accept > 0.0f) return true;
        const float x = __fmul_rn(num, racc);
        if (x > 1.0e-30f && x < 19.9f) {
            draw = true;
            const float test = __expf(-x) - u;
            if (fabsf(test) >= 1.0e-4f) return test > 0.0f;
        }
        const float exponent = __fdiv_rn(num, accept);
        draw = exponent > 0.0f && exponent <= 20.0f;
        if (draw) return __fsub_rn(exp_r(-exponent), u) >= 0.0f;
        return !(exponent > 20.0f);
    };

    int xb = 0;                                         // exchange buffer
    uint32_t xph = 0u;                                  // mbarrier phase parity, bit b for buffer b
    // chi^2 of the current wt over rows nmin..npt, the same value in every worker thread of the
    // cluster.  Every warp sums its rows and pushes the sum into every worker CTA (lane d into CTA d),
    // the stores completing their bytes on that CTA's mbarrier; every warp waits there and forms the
    // total for itself, in one fixed order, so no barrier of the CTA and no broadcast follows.
    // strict_sum: the reference's sequential float sum over the residuals, which every row thread
    // pushes to every CTA; else a double sum.  wmax: a bound on |wt|.  u, if given, receives the
    // stream's next value while the sums travel.  yout, if given, receives this CTA's row sums.
    // A buffer is written again two sums later, when every warp of the cluster has pushed its
    // sum in between and so has read this one.
    auto chisq = [&](bool strict_sum, float wmax, float *yout, float *u) -> float {
        float *gb = gat + (size_t)xb * fx_gstride(nw, rpc);
        double mypart = 0.0;
        if (slot < nrow) {
            const int r = slot;
            float sum = 0.0f;
            const float4 *w4 = (const float4 *)(wt + 1);
            const float4 *e4 = ex4 + r;
            // every partial sum is at most e1 * wmax (times 1 + 2^-20 for rounding)
            if (__fmul_ru(__fmul_ru(e1, wmax), 1.001f) < summax) {
                // four quads at a time, the coefficients of the next four on their way: the
                // additions are a chain, 4.7 cycles each, and loads that waited in it cost 30
                float4 c[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) c[j] = w4[j];
#pragma unroll
                for (int k = 0; k < FX_RQ; k += 4) {
                    if (k < ntq) {
                        float4 n[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) n[j] = w4[k + 4 + j];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            sum = __fadd_rn(sum, __fmul_rn(rq[k + j].x, c[j].x));
                            sum = __fadd_rn(sum, __fmul_rn(rq[k + j].y, c[j].y));
                            sum = __fadd_rn(sum, __fmul_rn(rq[k + j].z, c[j].z));
                            sum = __fadd_rn(sum, __fmul_rn(rq[k + j].w, c[j].w));
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) c[j] = n[j];
                    }
                }
                for (int q = 0; q < nsq; q += 4) {
                    float4 n[4], f[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        f[j] = e4[(q + j) * rpc];
                        n[j] = w4[FX_RQ + q + 4 + j];
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        sum = __fadd_rn(sum, __fmul_rn(f[j].x, c[j].x));
                        sum = __fadd_rn(sum, __fmul_rn(f[j].y, c[j].y));
                        sum = __fadd_rn(sum, __fmul_rn(f[j].z, c[j].z));
                        sum = __fadd_rn(sum, __fmul_rn(f[j].w, c[j].w));
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) c[j] = n[j];
                }
            } else {  // the reference's clamped sum (expand :4924)
#pragma unroll
                for (int k = 0; k < FX_RQ; ++k) {
                    const float ev[4] = {rq[k].x, rq[k].y, rq[k].z, rq[k].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int m = 4 * k + j;
                        if (m < nt) {
                            sum = __fadd_rn(sum, __fmul_rn(ev[j], wt[1 + m]));
                            if (fabsf(sum) > summax) sum = fsign(summax, sum);
                        }
                    }
                }
                for (int m = 4 * FX_RQ; m < nt; ++m) {
                    const float *ee = (const float *)(e4 + ((m >> 2) - FX_RQ) * rpc);
                    sum = __fadd_rn(sum, __fmul_rn(ee[m & 3], wt[1 + m]));
                    if (fabsf(sum) > summax) sum = fsign(summax, sum);
                }
            }
            const int i = row0 + r;
            const float term = __fsub_rn(yrow, sum);
            const float q2 = __fmul_rn(term, term);
            if (yout) yout[i] = sum;
            if (strict_sum) {
                const uint32_t la = smem_addr(gb + (rank * rpc + r)), lb = smem_addr(&xbar[xb]);
                for (int d = 0; d < nw; ++d)
                    st_async_f32(map_rank(la, (uint32_t)d), q2, map_rank(lb, (uint32_t)d));
            } else if (i >= F.nmin) {
                mypart = (double)q2;
            }
        }
        __syncwarp();
        const uint32_t ba = smem_addr(&xbar[xb]);
        if (!strict_sum && wid < nwr) {
            mypart = warp_sum_d(mypart);
            if (lane < nw)
                st_async_f64(map_rank(smem_addr(parts + xb * nparts + rank * nwr + wid), (uint32_t)lane), mypart,
                             map_rank(ba, (uint32_t)lane));
        }
        // this CTA's own arrival, and the bytes that every worker sends it
        if (tid == 0) mbar_expect(&xbar[xb], strict_sum ? 4u * (uint32_t)F.npt : 8u * (uint32_t)nparts);
        if (u) *u = get(cursor);
        __syncwarp();
        const uint32_t par = (xph >> xb) & 1u;
        if (!__all_sync(0xffffffffu, mbar_test(ba, par))) {
            const unsigned long long t0 = now_ns();
            while (!__all_sync(0xffffffffu, mbar_test(ba, par))) {
                if (__any_sync(0xffffffffu, vs->abort || now_ns() - t0 > FX_WAIT_NS)) {
                    if (lane == 0) {
                        atomicExch(F.status, 1);
                        vs->abort = 1;
                    }
                    break;
                }
            }
        }
        float v;
        if (strict_sum) {
            // sequential, the words sixteen rows ahead on their way
            const int a = F.nmin - 1, b = F.npt;    // 0-based rows a..b-1
            float c = 0.0f;
            int i = a;
            for (; i < b && (i & 3); ++i) c = __fadd_rn(c, gb[i]);
            const float4 *g4 = (const float4 *)gb;
            const int q1 = b >> 2;
            int q = i >> 2;
            float4 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = g4[min(q + j, max(q1 - 1, 0))];
            for (; q + 4 <= q1; q += 4) {
                float4 n[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) n[j] = g4[min(q + 4 + j, q1 - 1)];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    c = __fadd_rn(c, w[j].x);
                    c = __fadd_rn(c, w[j].y);
                    c = __fadd_rn(c, w[j].z);
                    c = __fadd_rn(c, w[j].w);
                    w[j] = n[j];
                }
            }
            for (i = max(i, 4 * q); i < b; ++i) c = __fadd_rn(c, gb[i]);
            v = c;
        } else {
            double t = 0.0;
            for (int k = lane; k < nparts; k += 32) t += parts[xb * nparts + k];
            v = (float)warp_sum_d(t);
        }
        xph ^= 1u << xb;
        xb ^= 1;
        return v;
    };
    // A barrier of the worker CTA at which a wait that gave up in any thread ends the fit in all (a warp
    // that gave up may have taken another branch than the rest; every barrier of the trials is this
    // one, so all leave at the same one).
    bool stop = false;
    auto meet = [&]() -> bool {
        __syncwarp();
        stop = __syncthreads_or(vs->abort) != 0;
        return stop;
    };
    // the largest |coefficient| a trial can reach from at most m: a step is stepr absolute below 1, relative above
    auto reach = [&](float m, float stepr) { return fmaxf(wfix, 1.0001f * fmaxf(m + fabsf(stepr), m * (1.0f + fabsf(stepr)))); };

    const float acceptr = 0.05f;
    const int npoints = F.npt - F.nmin + 1;
    for (int pi = 0; pi < F.nprob; ++pi) {
        const float *yin = F.yin + (size_t)pi * (F.npt + 1);
        float *yout = F.yout + (size_t)pi * (F.npt + 1);
        const float *wto_g = F.wtold_g + (size_t)pi * (nt + 1);
        float *scal = F.scal + (size_t)pi * 4;
        yrow = slot < nrow ? yin[row0 + slot] : 0.0f;
        for (int i = tid; i <= nt; i += T) {
            wtold[i] = wto_g[i];
            wt[i] = wtold[i];
        }
        block_sync();
        wfix = 0.0f;
        for (int m = 1; m < F.ncfirst; ++m) wfix = fmaxf(wfix, fabsf(wt[m]));
        if (tid == 0) wmax_all();
        block_sync();
        float wmx = vs->wmx;                         // bound on |wtold| of the perturbed terms
        float stepr = scal[0];
        float rejrat = scal[2];
        float chisqnew = scal[3];
        long long trials = 0;
        float wtmax = 0.0f;
        for (int it = 1; it <= nt; ++it) {
            const float a = fabsf(wt[it]);
            wtmax = (a >= wtmax) ? a : wtmax;
        }
        if (stepr < __fmul_rn(1.0e-6f, wtmax)) stepr = __fmul_rn(2.0e-6f, wtmax);
        if (F.nits > 0 && !stop) {
            icount = 0;
            chisqnew = chisq(F.strict != 0, fmaxf(wfix, wmx), nullptr, nullptr);
            chisqold = chisqnew;
            float chisqtest = -1.0f;
            int itry = 0;
            float wo = ic > 0 ? wtold[ic] : 0.0f;       // this thread's coefficient
            while (!stop && (itry < 10 || (itry < 150 && chisqtest < 1.0e-4f))) {
                ++itry;
                accept = __fdiv_rn(__fmul_rn(acceptr, chisqold), (float)npoints);
                racc = __fdiv_rn(1.0f, accept);
                rejrat = 0.0f;
                const float chisqstart = __fdiv_rn(chisqold, (float)npoints);
                for (int st = 1; st <= 100; ++st) {
                    ++trials;
                    // perturb coefficients ncfirst..nterms with the next K values (:4856-4861),
                    // each thread waiting for its own value
                    float wn = 0.0f;
                    if (ic > 0) {
                        const float du = __fsub_rn(__fmul_rn(2.0f, get(cursor + slot)), 1.0f);
                        if (fabsf(wo) < 1.0f) wn = __fadd_rn(wo, __fmul_rn(stepr, du));
                        else wn = __fmul_rn(wo, __fadd_rn(1.0f, __fmul_rn(stepr, du)));
                        wt[ic] = wn;
                    }
                    cursor += K;
                    if (meet()) break;
                    float u;
                    const float bound = reach(wmx, stepr);
                    chisqnew = chisq(F.strict != 0, bound, nullptr, &u);
                    bool draw;
                    const bool acc = metropolis(chisqnew, u, draw);
                    // every worker has taken the values before `cursor` (its part of chi^2 is here),
                    // but the draw at `cursor` perhaps not yet
                    if (rank == 0 && tid == 0) st_relaxed_cl_s64(gen_cons, cursor);
                    cursor += draw;
                    if (acc) {
                        wo = wn;
                        wmx = bound;
                        if (++icount == F.nfreq) {
                            icount = 0;
                            if (tid == 0) smooth();
                            if (meet()) break;
                            wmx = vs->wmx;
                            if (ic > 0) wo = wt[ic];
                            chisqnew = chisq(F.strict != 0, fmaxf(wfix, wmx), nullptr, nullptr);
                        }
                        chisqold = chisqnew;
                    } else {
                        rejrat = __fadd_rn(rejrat, 1.0f);
                    }
                }
                rejrat = __fdiv_rn(rejrat, 100.0f);
                const float chisqfinish = __fdiv_rn(chisqold, (float)npoints);
                if (chisqstart > 0.0f) chisqtest = __fdiv_rn(__fsub_rn(chisqfinish, chisqstart), chisqstart);
                else chisqtest = __fsub_rn(chisqfinish, chisqstart);
                const float rejfac = rejrat > 0.0f ? __fdiv_rn(0.75f, rejrat) : 2.0f;
                stepr = __fmul_rn(stepr, rejfac);
            }
            block_sync();
            if (ic > 0) wtold[ic] = wo;   // terms below ncfirst never change
            block_sync();
            for (int k = 1 + tid; k <= nt; k += T) wt[k] = wtold[k];
            block_sync();
            if (tid == 0) wmax_all();
            block_sync();
            wmx = vs->wmx;
        }
        // final fit over rows 1..npt, chi^2 from nmin (:4908-4914), in the reference's order
        chisqnew = chisq(true, fmaxf(wfix, wmx), yout, nullptr);
        if (rank == 0) {
            float *wt_g = F.wt_g + (size_t)pi * (nt + 1);
            float *wtold_o = F.wtold_g + (size_t)pi * (nt + 1);
            for (int k = tid; k <= nt; k += T) {
                wt_g[k] = wt[k];
                wtold_o[k] = wtold[k];
            }
            if (tid == 0) {
                scal[0] = stepr;
                scal[1] = acceptr;
                scal[2] = rejrat;
                scal[3] = chisqnew;
                F.trials[pi] = trials;
            }
        }
        block_sync();
    }
    // the generator leaves, and writes the state after the values taken unless a wait gave up
    block_sync();
    if (rank == 0 && tid == 0) {
        st_relaxed_cl_s64(gen_cons, cursor);
        st_release_cl_s32(gen_done, vs->abort ? 2 : 1);
    }
    __syncwarp();
    cl.sync();  // no CTA leaves while others may still write into its shared memory
}

}  // namespace epsr

using namespace epsr;

static inline size_t al256f(size_t x) { return (x + 255) & ~(size_t)255; }

// Worker CTAs: as many as give each FX_ROWS rows (a trial's rows are summed side by side, so the
// fewer a CTA has the shorter the trial; 600 rows x 116 terms, double sums: 5,370 cycles a trial on
// two CTAs with the stream's warp among their own, 3,240 now), up to seven beside
// the generator's CTA, the portable cluster size; more only for rows that need the memory.  Rows
// and terms for 256 threads: barriers of half the warps, and registers for the whole row.
// A CTA's rows have what the static arrays leave of the 227 KB a CTA may have.
static int fx_workers(int npt, int nterms, int ncoef, int *rpc_out, int *threads_out) {
    constexpr size_t fixed = 10 * 1024, budget = 227 * 1024 - fixed;
    static_assert(sizeof(FxGen) + sizeof(FxShared) <= fixed, "the static arrays are beside the rows");
    const int want = std::min((npt + FX_ROWS - 1) / FX_ROWS, FX_MAXW - 1);
    for (int c = std::max(want, 1); c <= FX_MAXW; ++c) {
        const int rpc = (npt + c - 1) / c;
        const int threads = rpc <= 256 && ncoef <= 256 ? 256 : FX_MAXT;
        if (rpc <= threads && fx_smem_bytes(nterms, rpc, c, threads) <= budget) {
            *rpc_out = rpc;
            *threads_out = threads;
            return c;
        }
    }
    return 0;
}

// Clusters past the portable size, allowed once per device, as EPSR_SMEM_OPTIN does.  (On every launch: ten fits of
// 3,700 rows x 12 terms in each of three threads took 225 ms, and 214 ms so; 213 and 212 ms in one thread.)
static int fx_wide_cluster() {
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    EPSR_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && ((done.load() >> dev) & 1ull)) return EPSR_OK;
    EPSR_CUDA(cudaFuncSetAttribute(fitexp_cluster_kernel<256>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    EPSR_CUDA(cudaFuncSetAttribute(fitexp_cluster_kernel<FX_MAXT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (dev >= 0 && dev < 64) done.fetch_or(1ull << dev);
    return EPSR_OK;
}

extern "C" int64_t epsr_fit_expansion_batch_scratch_bytes(int32_t nprob, int32_t npt, int32_t nterms) {
    (void)npt;
    (void)nterms;
    if (nprob < 1) nprob = 1;
    return (int64_t)(al256f(sizeof(float) * 4 * (size_t)nprob) + al256f(sizeof(long long) * (size_t)nprob) +
                     al256f(sizeof(int)));
}

extern "C" int64_t epsr_fit_expansion_scratch_bytes(int32_t npt, int32_t nterms) {
    return epsr_fit_expansion_batch_scratch_bytes(1, npt, nterms);
}

extern "C" int epsr_fit_expansion_batch(int32_t nprob, const float *yin, const float *expr, float *yout, float *wt,
                                        float *wtold, float *scal_host, int32_t nmin, int32_t npt, int32_t ncfirst,
                                        int32_t nterms, int32_t nits, int32_t nfreq, int32_t *ran1, void *scratch,
                                        int64_t scratch_bytes, int32_t strict, int64_t *trials_host, void *stream) {
    if (nprob <= 0 || !yin || !expr || !yout || !wt || !wtold || !scal_host || !ran1 || !scratch || !trials_host ||
        npt <= 0 || nterms <= 0 || nmin < 1 || nmin > npt || ncfirst < 1 || ncfirst > nterms) {
        epsr_set_error("epsr_fit_expansion_batch: bad arguments");
        return EPSR_ERR_ARG;
    }
    if (scratch_bytes < epsr_fit_expansion_batch_scratch_bytes(nprob, npt, nterms)) {
        epsr_set_error("epsr_fit_expansion_batch: scratch too small");
        return EPSR_ERR_CAPACITY;
    }
    if (nterms - ncfirst + 1 > FX_SLOTS) {
        epsr_set_error("epsr_fit_expansion_batch: at most %d perturbed terms", FX_SLOTS);
        return EPSR_ERR_UNSUPPORTED;
    }
    int rpc = 0, threads = 0;
    const int nw = fx_workers(npt, nterms, nterms - ncfirst + 1, &rpc, &threads);
    if (!nw) {
        epsr_set_error("epsr_fit_expansion_batch: %d rows x %d terms exceed 8 CTAs of shared memory", npt, nterms);
        return EPSR_ERR_UNSUPPORTED;
    }
    cudaStream_t s = (cudaStream_t)stream;
    char *p = (char *)scratch;
    float *scal = (float *)p;
    p += al256f(sizeof(float) * 4 * (size_t)nprob);
    long long *trials = (long long *)p;
    p += al256f(sizeof(long long) * (size_t)nprob);
    int *status = (int *)p;
    EPSR_H2D(scal, scal_host, sizeof(float) * 4 * (size_t)nprob, s);
    EPSR_CUDA(cudaMemsetAsync(status, 0, sizeof(int), s));
    FxDev F;
    F.expr = expr;
    F.yin = yin;
    F.yout = yout;
    F.wt_g = wt;
    F.wtold_g = wtold;
    F.scal = scal;
    F.trials = trials;
    F.status = status;
    F.nprob = nprob;
    F.nmin = nmin;
    F.npt = npt;
    F.ncfirst = ncfirst;
    F.nterms = nterms;
    F.nits = nits;
    F.nfreq = nfreq;
    F.strict = strict ? 1 : 0;
    F.rpc = rpc;
    F.nw = nw;
    F.ran1 = ran1;
    const size_t shm = fx_smem_bytes(nterms, rpc, nw, threads);
    const bool small = threads != FX_MAXT;
    EPSR_SMEM_OPTIN(fitexp_cluster_kernel<256>);
    EPSR_SMEM_OPTIN(fitexp_cluster_kernel<FX_MAXT>);
    if (nw == FX_MAXW) {   // nine CTAs
        const int rc = fx_wide_cluster();
        if (rc) return rc;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nw + 1, 1, 1);
    cfg.blockDim = dim3(small ? 256 : FX_MAXT, 1, 1);
    cfg.dynamicSmemBytes = shm;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nw + 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    EPSR_TIMED("fitexp_cluster_kernel", s,
               EPSR_CUDA(small ? cudaLaunchKernelEx(&cfg, fitexp_cluster_kernel<256>, F)
                               : cudaLaunchKernelEx(&cfg, fitexp_cluster_kernel<FX_MAXT>, F)));
    int hstatus = 0;
    EPSR_D2H(scal_host, scal, sizeof(float) * 4 * (size_t)nprob, s);
    EPSR_D2H(trials_host, trials, sizeof(long long) * (size_t)nprob, s);
    EPSR_D2H(&hstatus, status, sizeof(int), s);
    if (hstatus) {
        epsr_set_error("epsr_fit_expansion: a bounded device wait gave up (results invalid)");
        return EPSR_ERR_TIMEOUT;
    }
    return EPSR_OK;
}

extern "C" int epsr_fit_expansion(const float *yin, const float *expr, float *yout, float *wt, float *wtold,
                                  float *scal_host, int32_t nmin, int32_t npt, int32_t ncfirst, int32_t nterms,
                                  int32_t nits, int32_t nfreq, int32_t *ran1, void *scratch, int64_t scratch_bytes,
                                  int32_t strict, int64_t *trials_host, void *stream) {
    return epsr_fit_expansion_batch(1, yin, expr, yout, wt, wtold, scal_host, nmin, npt, ncfirst, nterms, nits, nfreq,
                                    ran1, scratch, scratch_bytes, strict, trials_host, stream);
}
