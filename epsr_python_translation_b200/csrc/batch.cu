// batch.cu -- many independent boxes advanced together by a parallel (checkerboard) Metropolis
// scheme, with an optional delayed-acceptance first stage from the surrogate network.
//
// Scheme.  Each sweep every box draws a random shift of its grid of ncell^3 cells and a random
// colour order; its centres are binned (counting sort, members of a cell in molecule order).
// Step t moves, in every box, one randomly chosen molecule of every cell of colour
// (colour_off + t) mod stride^3.  Cells of one colour are (stride - 1) cells apart, at least the
// interaction range, and a move that would take a centre out of its cell is rejected, so the
// moves of one step never see each other: they are exact single-molecule Metropolis moves made
// in parallel.  The proposal (rotation about a uniformly random axis by an angle uniform in
// [-rotmax, rotmax], translation uniform in the cube) is symmetric.
//
// Kernels per step: propose (one CTA per slot: the molecule, the proposal, and with the
// surrogate the radial histograms of the moved molecule before and after the move, written as
// two rows of BF16 features), the network (mlp.cu) when delayed acceptance is on, and decide
// (one CTA per slot: the first-stage test on the network's antisymmetric output, then the
// exact energy change over the partners within rint -- table lookups of molfit.py:1251-1279 --
// and the Metropolis test of molfit.py:401-408 on beta*dE - s, and the commit).  A CTA whose
// move fails the first stage returns before any pair energy: that is the work the surrogate
// saves.  All random numbers come from Philox4x32-10 counted by (sweep, step, slot).
#include <cuda_bf16.h>
#include <stddef.h>
#include <string.h>

#include <type_traits>

#include "pairhist.cuh"
#include "philox.cuh"
#include "umma.cuh"

namespace epsr {

constexpr int BMC_THREADS = 256;
constexpr int BMC_MAXT = 1024;            // most threads of a CTA that works on a move
constexpr int BMC_MAXD = 512;             // and of one that decides on a molecule of a few atoms
constexpr int BMC_MAXAT = 64;
constexpr int BMC_LIST = 6144;            // partner molecules scanned per move
constexpr int FEAT_BINS = 64, FEAT_CLASSES = 10, FEAT_HALF = FEAT_BINS * FEAT_CLASSES, FEAT_IN = 2 * FEAT_HALF;
constexpr float FEAT_RMAX = 8.0f;         // A
constexpr float FEAT_SCALE = 0.25f;       // count -> feature value
constexpr uint32_t P_BIN = 0xB1u, P_MOVE = 1u, P_DECIDE = 2u;

__device__ __forceinline__ float wrap_c(float c) { return __fsub_rn(c, nint_f(c)); }

__device__ __forceinline__ int cell_coord(float x, float shift, int n) {
    int i = __float2int_rd(__fmul_rn(__fadd_rn(__fadd_rn(x, 0.5f), shift), (float)n));
    i %= n;
    return i < 0 ? i + n : i;
}

__device__ __forceinline__ Tables box_tables(const epsr_bmc_t &B, const epsr_bmc_box_t &X) {
    Tables T;
    T.tab = (const float4 *)B.tab + X.tab0;
    T.xstar = B.xstar + X.xstar0;
    T.ld = X.ld;
    T.npt2 = X.izcut;
    T.izcut = X.izcut;
    T.stepcl = X.stepcl;
    return T;
}

__device__ __forceinline__ int feat_class(int c1, int c2) {
    const int a = c1 < c2 ? c1 : c2, b = c1 < c2 ? c2 : c1;
    return (a * (7 - a)) / 2 + b;   // (0,0)=0 ... (3,3)=9
}

// ----------------------------------------------------------------- binning
__global__ void bmc_begin_kernel(epsr_bmc_t B) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B.nbox) return;
    epsr_bmc_box_t &X = B.box[b];
    const int64_t sw = *B.sweep_counter;
    X.sweep = sw;
    const U4 r = philox4x32(U4{(uint32_t)sw, (uint32_t)(sw >> 32), P_BIN, 0u}, X.key0, X.key1);
    const float a = 1.0f / (float)X.ncell;
    X.shift[0] = u01(r.x) * a;
    X.shift[1] = u01(r.y) * a;
    X.shift[2] = u01(r.z) * a;
    const int ncol = X.stride * X.stride * X.stride;
    X.colour_off = (int)(r.w % (uint32_t)ncol);
}

// The place of a box's extent, the largest distance of an atom from its molecule's centre: the word of
// the bin cursors that no cell has.
__device__ __forceinline__ int32_t *box_extent(const epsr_bmc_t &B, const epsr_bmc_box_t &X, int b) {
    return B.mol_cell + B.nmol + X.cell0 + b + X.ncell * X.ncell * X.ncell;
}

__global__ void bmc_count_kernel(epsr_bmc_t B) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= B.nmol) return;
    const int b = B.mol_box[m];
    const epsr_bmc_box_t &X = B.box[b];
    const int n = X.ncell;
    const float4 centre = make_float4(B.xadd[m], B.yadd[m], B.zadd[m], 0.0f);
    const int c = (cell_coord(centre.x, X.shift[0], n) * n + cell_coord(centre.y, X.shift[1], n)) * n +
                  cell_coord(centre.z, X.shift[2], n);
    B.mol_cell[m] = c;
    atomicAdd(B.cell_start + X.cell0 + b + c + 1, 1);
    const float4 *p = (const float4 *)B.pos + B.naf[m];
    float r2 = 0.0f;
    for (int q = 0; q < B.nato[m]; ++q) {
        const float d = dsq_cubic(centre, p[q]);
        if (!(d <= r2) && r2 == r2) r2 = d;     // a NaN stays, and makes the extent infinite
    }
    const int mine = r2 >= 0.0f ? __float_as_int(sqrtf(r2)) : 0x7f800000;   // distances order as their bits
    const unsigned same = __match_any_sync(__activemask(), b);
    const int most = __reduce_max_sync(same, mine);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicMax(box_extent(B, X, b), most);
}

// one CTA per box: inclusive scan of the counts into starts
__global__ void bmc_scan_kernel(epsr_bmc_t B) {
    const epsr_bmc_box_t &X = B.box[blockIdx.x];
    int *st = B.cell_start + X.cell0 + blockIdx.x;
    const int nc = X.ncell * X.ncell * X.ncell;
    __shared__ int carry;
    __shared__ int ws[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 1; base <= nc; base += blockDim.x) {
        const int i = base + threadIdx.x;
        int v = i <= nc ? st[i] : 0;
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) ws[w] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            int a = 0;
            for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
                const int t = ws[k];
                ws[k] = a;
                a += t;
            }
        }
        __syncthreads();
        if (i <= nc) st[i] = carry + ws[w] + v;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += ws[w] + v;
        __syncthreads();
    }
}

__global__ void bmc_scatter_kernel(epsr_bmc_t B, int32_t *cursor) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= B.nmol) return;
    const int b = B.mol_box[m];
    const epsr_bmc_box_t &X = B.box[b];
    const int idx = X.cell0 + b + B.mol_cell[m];
    const int p = atomicAdd(cursor + idx, 1);
    B.cell_mols[X.mol0 + B.cell_start[idx] + p] = m;
}

// members of each cell in ascending molecule order (the scatter's order is not deterministic), one
// warp a cell: a member's place is the number of members before it.  A thread a cell, sorting in
// memory, took 660 us a sweep for 64 boxes of 300 to 30,000 atoms; this 71 us.
__global__ void bmc_sort_kernel(epsr_bmc_t B, const int32_t *cell_box, int ncell_tot) {
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;   // packed cell index (without the +b)
    if (g >= ncell_tot) return;
    const int lane = threadIdx.x & 31;
    const int b = cell_box[g];
    const int idx = g + b;
    int *mm = B.cell_mols + B.box[b].mol0;
    const int s0 = B.cell_start[idx], n = B.cell_start[idx + 1] - s0;
    if (n <= 256) {
        int v[8], rank[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            rank[k] = 0;
            v[k] = 32 * k + lane < n ? mm[s0 + 32 * k + lane] : 0x7fffffff;
        }
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
            const int w = mm[s0 + i];
#pragma unroll
            for (int k = 0; k < 8; ++k) rank[k] += w < v[k];
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (32 * k + lane < n) mm[s0 + rank[k]] = v[k];
    } else if (lane == 0) {
        for (int i = s0 + 1; i < s0 + n; ++i) {
            const int v = mm[i];
            int j = i - 1;
            while (j >= s0 && mm[j] > v) {
                mm[j + 1] = mm[j];
                --j;
            }
            mm[j + 1] = v;
        }
    }
}

// A molecule in one word: its first atom (from the box's first) << 7 | its atom count.
__device__ __forceinline__ unsigned mol_word(const epsr_bmc_t &B, const epsr_bmc_box_t &X, int m) {
    return ((unsigned)(B.naf[m] - X.atom0) << 7) | (unsigned)B.nato[m];
}

// the molecules in cell order, centre and packed atoms
__global__ void bmc_order_kernel(epsr_bmc_t B) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.nmol) return;
    const int m = B.cell_mols[i];
    const epsr_bmc_box_t &X = B.box[B.mol_box[m]];
    ((float4 *)B.cell_mol)[i] = make_float4(B.xadd[m], B.yadd[m], B.zadd[m], __uint_as_float(mol_word(B, X, m)));
}

__global__ void bmc_end_kernel(epsr_bmc_t B) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *B.sweep_counter += 1;
}

// ----------------------------------------------------------------- partner lists
// The molecules of the cells within `nr` of cell (ix, iy, iz) (each cell once, wrapped), in
// cell order and ascending molecule order within a cell, into list[]; returns the count (or
// -1 when the list would overflow).
__device__ int gather_partners(const epsr_bmc_t &B, const epsr_bmc_box_t &X, int b, int ix, int iy, int iz, int nr,
                               int *list, int *scan_ws) {
    const int n = X.ncell;
    const int w = 2 * nr + 1 < n ? 2 * nr + 1 : n;
    const int ox = 2 * nr + 1 < n ? ix - nr : 0, oy = 2 * nr + 1 < n ? iy - nr : 0, oz = 2 * nr + 1 < n ? iz - nr : 0;
    const int ncell = w * w * w;
    const int *st = B.cell_start + X.cell0 + b;
    const int *mm = B.cell_mols + X.mol0;
    int total = 0;
    for (int base = 0; base < ncell; base += blockDim.x) {
        const int k = base + threadIdx.x;
        int cnt = 0, s0 = 0;
        if (k < ncell) {
            const int dx = k / (w * w), dy = (k / w) % w, dz = k % w;
            const int cx = ((ox + dx) % n + n) % n, cy = ((oy + dy) % n + n) % n, cz = ((oz + dz) % n + n) % n;
            const int c = (cx * n + cy) * n + cz;
            s0 = st[c];
            cnt = st[c + 1] - s0;
        }
        // block exclusive scan of cnt
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        int v = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) scan_ws[wid] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            int a = 0;
            for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
                const int t = scan_ws[q];
                scan_ws[q] = a;
                a += t;
            }
            scan_ws[32] = a;
        }
        __syncthreads();
        const int at = total + scan_ws[wid] + v - cnt;
        for (int q = 0; q < cnt; ++q)
            if (at + q < BMC_LIST) list[at + q] = mm[s0 + q];
        total += scan_ws[32];
        __syncthreads();
    }
    return total <= BMC_LIST ? total : -1;
}

__device__ __forceinline__ float4 atom_pos(const epsr_bmc_t &B, int a) { return ((const float4 *)B.pos)[a]; }

// The work of one move, found by the threads of a CTA together.  An item is a partner molecule and
// an atom of the moved molecule that can interact: of the cells within `nr` of the move's cell
// (each cell once, wrapped) the molecules other than the moved one whose centre is within sqrt(r2)
// of its centre, and of those the atoms a whose old or new position is within sqrt(ra2) of the
// partner's centre (ra: the range plus the largest extent of the box's molecules, so every atom pair in
// range belongs to an item, whatever r2 the caller gave).  process(partner, atoms, a) is called once per item, partners of more than four
// atoms first, so that the lanes of a warp loop over atom counts that are alike.  Returns the
// molecules of the cells, the same in every thread.
//
// Bound by the latency of the dependent loads (cell starts -> members -> atoms) and by the issue
// of the pair evaluations.  So: cells that follow one another along z are one run of the member
// list (two where the run wraps), cut to the sphere; members are read side by side from the
// cell-ordered copy, 16 bytes each (five arrays indexed by molecule took ten times the cache
// sectors); and near molecules and items are listed for the whole CTA before they are worked on,
// in a fixed order, so that every thread has its share: with lists of their own the busiest of 32
// warps had three times the mean, and a step waits for its slowest warp.
struct NearMol {
    float x, y, z;                 // the centre
    unsigned mol;                  // mol_word
};
constexpr int BMC_RUNS = 512;      // runs listed at a time (a grid of up to 16 cells a side: all)
template <int CAND, int ITEMS>
struct Search {
    int end[BMC_RUNS], off[BMC_RUNS];   // members before the run's end; its first member less those before it
    NearMol mol[CAND];                  // a pass's members
    unsigned short near_[CAND];         // those in range
    unsigned short item[ITEMS];         // a pass's items: the member,
    unsigned char atom[ITEMS];          // the moved molecule's atom
    unsigned bal0[ITEMS / 32], bal1[ITEMS / 32];   // kept lanes of each 32 members or items
    int ws[2][BMC_MAXT / 32];
};
struct Near {
    int ix, iy, iz, nr, na;
    unsigned self;                 // the moved molecule's word
    float cx, cy, cz, r2, ra2;
    const float4 *p_old, *p_new;   // shared memory, na positions each
};
// Exclusive prefix of the popcounts of n words (n a multiple of 32, at most 128), by a warp:
// pre(i) for the warp's own use, and the total.
struct BallotScan {
    int mine[4], base[4], total;
    __device__ __forceinline__ BallotScan(const unsigned *w, int n) {
        const int lane = threadIdx.x & 31;
        total = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            mine[j] = base[j] = 0;
            if (32 * j < n) {
                const int c = __popc(w[32 * j + lane]);
                int v = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += u;
                }
                mine[j] = total + v - c;
                total += __shfl_sync(0xffffffffu, v, 31);
            }
        }
    }
    __device__ __forceinline__ int before(int i) const {   // i warp-uniform
        int v = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if ((i >> 5) == j) v = __shfl_sync(0xffffffffu, mine[j], i & 31);
        return v;
    }
};
// the distance of a point at fraction f of its cell from the cells o further on, in cells
__device__ __forceinline__ float cell_gap(int o, float f) { return o > 0 ? (float)o - f : (o < 0 ? f - (float)(o + 1) : 0.0f); }
__device__ __forceinline__ float cell_frac(float x, float shift, int n, int i) {
    const float u = (x + 0.5f + shift) * (float)n;
    const float f = u - (float)n * floorf(u / (float)n) - (float)i;
    return fminf(fmaxf(f, 0.0f), 1.0f);
}
template <int CAND, int ITEMS, class F>
__device__ __forceinline__ int near_items(const epsr_bmc_t &B, const epsr_bmc_box_t &X, int b, const Near &P,
                                          Search<CAND, ITEMS> &Q, F process) {
    const int n = X.ncell;
    const bool full = 2 * P.nr + 1 >= n;
    const int w = full ? n : 2 * P.nr + 1;
    const int *st = B.cell_start + X.cell0 + b;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const float inv_na = 1.0f / (float)P.na;
    // the reach in cells, with slack for the roundings of the fractions
    const float reach = sqrtf(P.r2) * (float)n + 0.01f;
    const float fx = cell_frac(P.cx, X.shift[0], n, P.ix), fy = cell_frac(P.cy, X.shift[1], n, P.iy),
                fz = cell_frac(P.cz, X.shift[2], n, P.iz);
    const int ncol = w * w;
    int scanned = 0;
    for (int e0 = 0; e0 < 2 * ncol; e0 += BMC_RUNS) {
        // the runs of this pass: columns, then the wrapped parts of columns
        const int nr = min(2 * ncol - e0, BMC_RUNS);
        int carry = 0;
        for (int b0 = 0; b0 < nr; b0 += blockDim.x) {
            const int i = b0 + tid;
            int s0 = 0, len = 0, all_len = 0;
            if (i < nr) {
                const bool wrapped = e0 + i >= ncol;
                const int r = e0 + i - (wrapped ? ncol : 0);
                int gx = r / w, gy = r - gx * w, z0 = 0, z1 = n, y0 = 0, y1 = n;   // [z0, z1) of the sphere, [y0, y1) of the cube
                if (!full) {
                    const float dx = cell_gap(gx - P.nr, fx), dy = cell_gap(gy - P.nr, fy);
                    const float h2 = reach * reach - dx * dx - dy * dy, h = sqrtf(fmaxf(h2, 0.0f));
                    y0 = P.iz - P.nr;
                    y1 = P.iz + P.nr + 1;
                    z0 = max(P.iz + (int)floorf(fz - h), y0);
                    z1 = h2 > 0.0f ? min(P.iz + (int)floorf(fz + h) + 1, y1) : z0;
                    gx += P.ix - P.nr;
                    gy += P.iy - P.nr;
                    if (gx < 0) gx += n;
                    else if (gx >= n) gx -= n;
                    if (gy < 0) gy += n;
                    else if (gy >= n) gy -= n;
                    // the part inside [0, n), or the part that wraps (below 0 or from n on: never both)
                    auto part = [&](int &lo, int &hi) {
                        if (!wrapped) {
                            lo = max(lo, 0);
                            hi = min(hi, n);
                        } else if (y0 < 0) {
                            hi = min(hi, 0) + n;
                            lo += n;
                        } else {
                            lo = max(lo, n) - n;
                            hi -= n;
                        }
                        hi = max(lo, hi);
                    };
                    part(z0, z1);
                    part(y0, y1);
                } else if (wrapped) {
                    z1 = y1 = 0;
                }
                const int base = (gx * n + gy) * n;
                if (y1 > y0) all_len = st[base + y1] - st[base + y0];
                if (z1 > z0) {
                    s0 = st[base + z0];
                    len = st[base + z1] - s0;
                }
            }
            int end = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= o) end += u;
            }
            const int sum = __reduce_add_sync(0xffffffffu, all_len);
            if (lane == 31) {
                Q.ws[0][wid] = end;
                Q.ws[1][wid] = sum;
            }
            __syncthreads();
            const int v0 = lane < nw ? Q.ws[0][lane] : 0;
            end += __reduce_add_sync(0xffffffffu, lane < wid ? v0 : 0);
            scanned += __reduce_add_sync(0xffffffffu, lane < nw ? Q.ws[1][lane] : 0);
            if (i < nr) {
                Q.end[i] = carry + end;
                Q.off[i] = s0 - (carry + end - len);
            }
            carry += __reduce_add_sync(0xffffffffu, v0);
            __syncthreads();
        }
        if (scanned > BMC_LIST) return scanned;
        for (int m0 = 0; m0 < carry; m0 += CAND) {
            // members of this pass, 32 a warp, those in range kept
            const int nm = min(carry - m0, CAND);
            for (int i = tid; i < CAND / 32; i += blockDim.x) Q.bal0[i] = 0u;
            __syncthreads();
            for (int c0 = 32 * wid; c0 < nm; c0 += 32 * nw) {
                const int c = c0 + lane;
                bool in = false;
                if (c < nm) {   // the run of the member: the first whose end is past it
                    int lo = 0, hi = nr - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (Q.end[mid] > m0 + c) hi = mid;
                        else lo = mid + 1;
                    }
                    const int at = X.mol0 + Q.off[lo] + m0 + c;
                    NearMol m;
                    if (B.cell_mol) {
                        const float4 v = ((const float4 *)B.cell_mol)[at];
                        m = NearMol{v.x, v.y, v.z, __float_as_uint(v.w)};
                    } else {
                        const int jm = B.cell_mols[at];
                        m = NearMol{B.xadd[jm], B.yadd[jm], B.zadd[jm], mol_word(B, X, jm)};
                    }
                    Q.mol[c] = m;
                    in = m.mol != P.self && dsq_cubic(make_float4(P.cx, P.cy, P.cz, 0.0f),
                                                      make_float4(m.x, m.y, m.z, 0.0f)) <= P.r2;
                }
                const unsigned bal = __ballot_sync(0xffffffffu, in);
                if (lane == 0) Q.bal0[c0 >> 5] = bal;
            }
            __syncthreads();
            int nnear;
            {
                const BallotScan S(Q.bal0, CAND / 32);
                nnear = S.total;
                for (int c0 = 32 * wid; c0 < nm; c0 += 32 * nw) {
                    const unsigned bal = Q.bal0[c0 >> 5];
                    const int at = S.before(c0 >> 5);
                    if ((bal >> lane) & 1u) Q.near_[at + __popc(bal & below)] = (unsigned short)(c0 + lane);
                }
            }
            __syncthreads();
            // their items, partner by partner
            for (int i0 = 0; i0 < nnear * P.na; i0 += ITEMS) {
                const int ni = min(nnear * P.na - i0, ITEMS);
                for (int i = tid; i < ITEMS / 32; i += blockDim.x) Q.bal0[i] = Q.bal1[i] = 0u;
                __syncthreads();
                for (int c0 = 32 * wid; c0 < ni; c0 += 32 * nw) {
                    const int i = i0 + c0 + lane;
                    bool in = false, big = false;
                    if (c0 + lane < ni) {
                        const int e = (int)(((float)i + 0.5f) * inv_na), a = i - e * P.na;
                        const NearMol m = Q.mol[Q.near_[e]];
                        const float4 c = make_float4(m.x, m.y, m.z, 0.0f);
                        in = !(dsq_cubic(P.p_old[a], c) > P.ra2 && dsq_cubic(P.p_new[a], c) > P.ra2);
                        big = (m.mol & 127u) > 4u;
                    }
                    const unsigned k0 = __ballot_sync(0xffffffffu, in && !big), k1 = __ballot_sync(0xffffffffu, in && big);
                    if (lane == 0) {
                        Q.bal0[c0 >> 5] = k0;
                        Q.bal1[c0 >> 5] = k1;
                    }
                }
                __syncthreads();
                int nkept;
                {
                    const BallotScan S1(Q.bal1, ITEMS / 32), S0(Q.bal0, ITEMS / 32);
                    nkept = S0.total + S1.total;
                    for (int c0 = 32 * wid; c0 < ni; c0 += 32 * nw) {
                        const unsigned k0 = Q.bal0[c0 >> 5], k1 = Q.bal1[c0 >> 5];
                        const int at0 = S1.total + S0.before(c0 >> 5), at1 = S1.before(c0 >> 5);
                        const bool big = (k1 >> lane) & 1u;
                        if (big || ((k0 >> lane) & 1u)) {
                            const int i = i0 + c0 + lane, e = (int)(((float)i + 0.5f) * inv_na);
                            const int at = big ? at1 + __popc(k1 & below) : at0 + __popc(k0 & below);
                            Q.item[at] = Q.near_[e];
                            Q.atom[at] = (unsigned char)(i - e * P.na);
                        }
                    }
                }
                __syncthreads();
                for (int i = tid; i < nkept; i += blockDim.x) {
                    const unsigned m = Q.mol[Q.item[i]].mol;
                    process(X.atom0 + (int)(m >> 7), (int)(m & 127u), (int)Q.atom[i]);
                }
                __syncthreads();
            }
        }
    }
    return scanned;
}

using WideSearch = Search<2048, 4096>;     // CTAs of more than 256 threads (and every feature search)
using NarrowSearch = Search<1024, 2048>;

// The distance from a partner's centre within which an atom can be in `range` of its atoms, squared: the
// box's extent as the binning found it (a molecule keeps its shape but for roundings), with slack for those.
__device__ __forceinline__ float item_range2(const epsr_bmc_t &B, const epsr_bmc_box_t &X, int b, float range) {
    const float r = range + __int_as_float(*box_extent(B, X, b)) + 1e-6f;
    return r * r * 1.00001f;
}

// ----------------------------------------------------------------- propose
// The proposal of slot k (box b, cell (ix, iy, iz)) by one warp: the molecule, its new centre and
// offsets written to the slot's arrays and its old and new positions to shared memory.  Returns
// the molecule, -1 for an empty cell; `left` is set when the centre leaves the cell.
__device__ int propose_warp(const epsr_bmc_t &B, const epsr_bmc_box_t &X, int k, int b, int step, int ix, int iy, int iz,
                            float4 *p_old, float4 *p_new, int &na_out, bool &left) {
    const int lane = threadIdx.x & 31;
    const int n = X.ncell;
    const int c = (ix * n + iy) * n + iz;
    const int *st = B.cell_start + X.cell0 + b;
    const int s0 = st[c], cnt = st[c + 1] - s0;
    na_out = 0;
    left = false;
    if (cnt <= 0) return -1;
    const U4 r0 = philox4x32(U4{(uint32_t)X.sweep, (uint32_t)step, (uint32_t)k, P_MOVE}, X.key0, X.key1);
    const U4 r1 = philox4x32(U4{(uint32_t)X.sweep, (uint32_t)step, (uint32_t)k, P_MOVE + 16u}, X.key0, X.key1);
    int pick = (int)(u01(r0.x) * (float)cnt);
    pick = pick < cnt ? pick : cnt - 1;
    const int mol = B.cell_mols[X.mol0 + s0 + pick];
    const int a0 = B.naf[mol], na = B.nato[mol];
    const float ccx = B.xadd[mol], ccy = B.yadd[mol], ccz = B.zadd[mol];
    // rotation: axis from (u1, u2), angle from u3 (Rodrigues, in float); the cosines and sines of
    // the axis' azimuth and of the angle on two lanes at a time
    const float ct = __fsub_rn(__fmul_rn(2.0f, u01(r0.y)), 1.0f);
    const float st_ = __fsqrt_rn(fmaxf(__fsub_rn(1.0f, __fmul_rn(ct, ct)), 0.0f));
    const float ph = __fmul_rn(6.2831853071795864769f, u01(r0.z));
    const float al = __fmul_rn(X.rotmax, __fsub_rn(__fmul_rn(2.0f, u01(r0.w)), 1.0f));
    const float arg = (lane & 1) ? al : ph;
    const float cv = cos_r(arg), sv = sin_r(arg);
    const float ax = __fmul_rn(st_, __shfl_sync(0xffffffffu, cv, 0)), ay = __fmul_rn(st_, __shfl_sync(0xffffffffu, sv, 0)),
                az = ct;
    const float ca = __shfl_sync(0xffffffffu, cv, 1), sa = __shfl_sync(0xffffffffu, sv, 1), oc = __fsub_rn(1.0f, ca);
    const float nx = wrap_c(__fadd_rn(ccx, __fmul_rn(X.transmax, __fsub_rn(__fmul_rn(2.0f, u01(r1.x)), 1.0f))));
    const float ny = wrap_c(__fadd_rn(ccy, __fmul_rn(X.transmax, __fsub_rn(__fmul_rn(2.0f, u01(r1.y)), 1.0f))));
    const float nz = wrap_c(__fadd_rn(ccz, __fmul_rn(X.transmax, __fsub_rn(__fmul_rn(2.0f, u01(r1.z)), 1.0f))));
    left = cell_coord(nx, X.shift[0], n) != ix || cell_coord(ny, X.shift[1], n) != iy ||
           cell_coord(nz, X.shift[2], n) != iz;
    float4 *so = (float4 *)B.slot_off + (size_t)k * BMC_MAXAT;
    float4 *sn = (float4 *)B.slot_new + (size_t)k * BMC_MAXAT;
    for (int q = lane; q < na; q += 32) {
        const float vx = B.xa[a0 + q], vy = B.ya[a0 + q], vz = B.za[a0 + q];
        // v' = v cos + (n x v) sin + n (n.v)(1 - cos)
        const float dot = __fadd_rn(__fadd_rn(__fmul_rn(ax, vx), __fmul_rn(ay, vy)), __fmul_rn(az, vz));
        const float cxv = __fsub_rn(__fmul_rn(ay, vz), __fmul_rn(az, vy));
        const float cyv = __fsub_rn(__fmul_rn(az, vx), __fmul_rn(ax, vz));
        const float czv = __fsub_rn(__fmul_rn(ax, vy), __fmul_rn(ay, vx));
        const float dd = __fmul_rn(dot, oc);
        const float rx = __fadd_rn(__fadd_rn(__fmul_rn(vx, ca), __fmul_rn(cxv, sa)), __fmul_rn(ax, dd));
        const float ry = __fadd_rn(__fadd_rn(__fmul_rn(vy, ca), __fmul_rn(cyv, sa)), __fmul_rn(ay, dd));
        const float rz = __fadd_rn(__fadd_rn(__fmul_rn(vz, ca), __fmul_rn(czv, sa)), __fmul_rn(az, dd));
        const float4 po = atom_pos(B, a0 + q);
        const float4 pn = make_float4(__fadd_rn(rx, nx), __fadd_rn(ry, ny), __fadd_rn(rz, nz), po.w);
        so[q] = make_float4(rx, ry, rz, 0.0f);
        sn[q] = pn;
        p_old[q] = po;
        p_new[q] = pn;
    }
    // the centre, and where the molecule stands in its box's cell order
    if (lane == 0) ((float4 *)B.slot_centre)[k] = make_float4(nx, ny, nz, __int_as_float(s0 + pick));
    na_out = na;
    return mol;
}

// the cell of slot k in a step
__device__ __forceinline__ void slot_cell(const epsr_bmc_box_t &X, int k, int step, int &ix, int &iy, int &iz) {
    const int j = k - X.slot0;
    const int s = X.stride, na = X.ncell / s;
    const int colour = (X.colour_off + step) % (s * s * s);
    ix = colour / (s * s) + s * (j / (na * na));
    iy = (colour / s) % s + s * ((j / na) % na);
    iz = colour % s + s * (j % na);
}

// ODD: the caller's feature rows lie on no boundary for two features at once.  (A form of its own: tested in
// the kernel, the other form's step took 1.5 us longer.)
template <bool ODD>
__global__ void __launch_bounds__(BMC_MAXT) bmc_propose_kernel(epsr_bmc_t B, int step, __nv_bfloat16 *xfeat) {
    extern __shared__ __align__(16) unsigned char bmc_smem[];
    __shared__ int hist[2 * FEAT_HALF];
    __shared__ float4 p_old[BMC_MAXAT], p_new[BMC_MAXAT];
    __shared__ int s_mol, s_n, s_left;
    const int k = blockIdx.x;
    const int b = B.slot_box[k];
    const epsr_bmc_box_t &X = B.box[b];
    int ix, iy, iz;
    slot_cell(X, k, step, ix, iy, iz);
    if (threadIdx.x < 32) {
        int na;
        bool left;
        const int mol = propose_warp(B, X, k, b, step, ix, iy, iz, p_old, p_new, na, left);
        if (threadIdx.x == 0) {
            B.slot_mol[k] = mol < 0 ? -1 : (left ? -2 : mol);
            s_mol = mol;
            s_left = left;
            s_n = na;
        }
    } else {
        for (int i = threadIdx.x - 32; i < 2 * FEAT_HALF; i += blockDim.x - 32) hist[i] = 0;
    }
    if (!xfeat) return;   // one warp: nothing to wait for
    __syncthreads();
    __nv_bfloat162 *row0 = (__nv_bfloat162 *)(xfeat + (size_t)(2 * k) * FEAT_IN), *row1 = row0 + FEAT_IN / 2;
    if (s_mol < 0 || s_left) {   // nothing to screen: zero rows
        const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
        if (ODD)
            for (int i = threadIdx.x; i < 2 * FEAT_IN; i += blockDim.x) ((__nv_bfloat16 *)row0)[i] = zero.x;
        else
            for (int i = threadIdx.x; i < FEAT_IN / 2; i += blockDim.x) row0[i] = row1[i] = zero;
        return;
    }
    const int mol = s_mol, na_ = s_n;
    const float rf = X.rfeat;
    const float binf = (float)FEAT_BINS / FEAT_RMAX * X.dmax;   // bins per box unit
    const float rsq_skip = (float)((double)rf * (double)rf * (1.0 + 1e-5));   // d >= rf beyond it
    // the distances of every item's atom before and after the move to the partner's atoms, binned
    // (no atom of a partner whose centre is beyond rfeat_c is within 8 A of the moved molecule)
    const int a00 = B.naf[mol];
    const Near P{ix, iy, iz, X.nrange_feat, na_, mol_word(B, X, mol), B.xadd[mol], B.yadd[mol], B.zadd[mol],
                 __fmul_rn(X.rfeat_c, X.rfeat_c), item_range2(B, X, b, rf), p_old, p_new};
    const int scanned = near_items(B, X, b, P, *(WideSearch *)bmc_smem, [&](int b0, int nb, int a) {
        const int ca = B.fclass[a00 + a];
        const float4 po = p_old[a], pn = p_new[a];
#pragma unroll 2
        for (int j = 0; j < nb; ++j) {
            const float4 pb = atom_pos(B, b0 + j);
            const int fc = feat_class(ca, B.fclass[b0 + j]) * FEAT_BINS;
            const float q0 = dsq_cubic(po, pb), q1 = dsq_cubic(pn, pb);
            // the square root only for pairs that can be within rf
            if (q0 <= rsq_skip) {
                const float d0 = sqrt_unit(q0);
                if (d0 < rf) atomicAdd(&hist[fc + min((int)__fmul_rn(d0, binf), FEAT_BINS - 1)], 1);
            }
            if (q1 <= rsq_skip) {
                const float d1 = sqrt_unit(q1);
                if (d1 < rf) atomicAdd(&hist[FEAT_HALF + fc + min((int)__fmul_rn(d1, binf), FEAT_BINS - 1)], 1);
            }
        }
    });
    if (scanned > BMC_LIST) {
        if (threadIdx.x == 0) atomicExch(B.status, 2);
        return;
    }
    __syncthreads();
    if (ODD) {
        for (int i = threadIdx.x; i < 2 * FEAT_IN; i += blockDim.x) {
            const int h = i < FEAT_IN ? i : (i - FEAT_IN < FEAT_HALF ? i - FEAT_HALF : i - FEAT_IN - FEAT_HALF);
            ((__nv_bfloat16 *)row0)[i] = __float2bfloat16_rn((float)hist[h] * FEAT_SCALE);
        }
        return;
    }
    for (int i = threadIdx.x; i < FEAT_HALF / 2; i += blockDim.x) {
        const int2 h0 = ((const int2 *)hist)[i], h1 = ((const int2 *)(hist + FEAT_HALF))[i];
        const __nv_bfloat162 f0 = __floats2bfloat162_rn((float)h0.x * FEAT_SCALE, (float)h0.y * FEAT_SCALE);
        const __nv_bfloat162 f1 = __floats2bfloat162_rn((float)h1.x * FEAT_SCALE, (float)h1.y * FEAT_SCALE);
        row0[i] = f0;
        row0[FEAT_HALF / 2 + i] = f1;
        row1[i] = f1;
        row1[FEAT_HALF / 2 + i] = f0;
    }
}

// ----------------------------------------------------------------- decide
__device__ __forceinline__ double block_sum_d(double v, double *ws) {
    v = warp_sum_d(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) ws[w] = v;
    __syncthreads();
    if (w == 0) {
        double t = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0.0;
        t = warp_sum_d(t);
        if (lane == 0) ws[32] = t;
    }
    __syncthreads();
    return ws[32];
}

// The energy change of one item: the partner's atoms against the moved atom before and after the
// move, float sums over the partner's atoms (each pair's value that of pair_energy), the change in
// double.  Both positions of a pair are evaluated together without a branch between them, the next
// partner atom is loaded ahead, and the wrap and the table index run on the adder, not the
// conversion unit.
struct MoveChange {
    const float4 *tab, *pos;       // the first point in range of the first pair (shared memory when staged)
    const float *xs;
    const int *pr;
    float skip, stepcl, rcp;
    int izlast, ld, ntype;         // ld: points between pairs
    __device__ __forceinline__ void both(const float4 *t, float dn, float dd, float &r1, float &r0) const {
        const float d1 = sqrt_unit(dn), d0 = sqrt_unit(dd);
        const float q1 = __fmul_rn(d1, rcp), q0 = __fmul_rn(d0, rcp);   // bin_index of both at once
        const float g1 = __fadd_rz(q1, 8388608.0f), g0 = __fadd_rz(q0, 8388608.0f);
        const float f1 = __fsub_rn(q1, __fsub_rn(g1, 8388608.0f)), f0 = __fsub_rn(q0, __fsub_rn(g0, 8388608.0f));
        int n1 = __float_as_int(g1) - 0x4b000000, n0 = __float_as_int(g0) - 0x4b000000;
        if (!(fabsf(__fsub_rn(f1, 0.5f)) < 0.499f && fabsf(__fsub_rn(f0, 0.5f)) < 0.499f)) {
            n1 = ifix(__fdiv_rn(d1, stepcl));
            n0 = ifix(__fdiv_rn(d0, stepcl));
        }
        const int c1 = min(max(n1, 0), izlast), c0 = min(max(n0, 0), izlast);
        const float4 t1 = t[c1], t0 = t[c0];
        const float x1 = __fsub_rn(d1, xs[c1]), x0 = __fsub_rn(d0, xs[c0]);
        const float v1 = __fadd_rn(__fadd_rn(__fadd_rn(t1.x, __fmul_rn(t1.y, x1)), t1.z), __fmul_rn(t1.w, x1));
        const float v0 = __fadd_rn(__fadd_rn(__fadd_rn(t0.x, __fmul_rn(t0.y, x0)), t0.z), __fmul_rn(t0.w, x0));
        r1 = n1 == c1 ? v1 : 0.0f;
        r0 = n0 == c0 ? v0 : 0.0f;
    }
    __device__ __forceinline__ double item(float4 po, float4 pn, int b0, int nb) const {
        const float4 *pb = pos + b0;
        const int *row = pr + __float_as_int(po.w) * ntype;
        float e_new = 0.0f, e_old = 0.0f;
        float4 nxt = pb[0];
        for (int q = 0; q < nb; ++q) {
            const float4 p = nxt;
            if (q + 1 < nb) nxt = pb[q + 1];
            const float dn = dsq_cubic(pn, p), dd = dsq_cubic(po, p);
            if (!(dn > skip) || !(dd > skip)) {   // beyond skip_dsq the value is +0, which adds nothing
                float v1, v0;
                both(tab + (size_t)row[__float_as_int(p.w)] * ld, dn, dd, v1, v0);
                e_new = __fadd_rn(e_new, v1);
                e_old = __fadd_rn(e_old, v0);
            }
        }
        return (double)e_new - (double)e_old;
    }
};

// Metropolis test of a move whose energy change is de (thread 0: `acc` for the others) and commit
__device__ __forceinline__ void finish_move(const epsr_bmc_t &B, const epsr_bmc_box_t &X, int k, int b, int mol, int a0,
                                            int na, double de, float sg, uint32_t ry, float *target,
                                            const float4 *p_new, int *s_go) {
    if (threadIdx.x == 0) {
        const double x = (double)X.beta * de - (double)sg;
        const int acc = x <= 0.0 || (double)u01(ry) < exp(-x);
        if (target) target[k] = (float)((double)X.beta * de - (double)sg);   // beta dE (mode 2), beta dE - s (1)
        *s_go = acc;
        if (acc) {
            atomicAdd((unsigned long long *)(B.counters + 4 * b + 2), 1ull);
            atomicAdd(B.energy + b, de);
            const float4 c = ((const float4 *)B.slot_centre)[k];
            B.xadd[mol] = c.x;
            B.yadd[mol] = c.y;
            B.zadd[mol] = c.z;
            if (B.cell_mol)
                ((float4 *)B.cell_mol)[X.mol0 + __float_as_int(c.w)] =
                    make_float4(c.x, c.y, c.z, __uint_as_float(mol_word(B, X, mol)));
        }
    }
    __syncthreads();
    if (*s_go) {
        const float4 *so = (const float4 *)B.slot_off + (size_t)k * BMC_MAXAT;
        for (int q = threadIdx.x; q < na; q += blockDim.x) {
            B.xa[a0 + q] = so[q].x;
            B.ya[a0 + q] = so[q].y;
            B.za[a0 + q] = so[q].z;
            ((float4 *)B.pos)[a0 + q] = p_new[q];
        }
    }
}

// One CTA per slot.  The box's tables go into shared memory when `table_bytes` hold them: the pair
// evaluations read four table words per lane at addresses that differ from lane to lane, and every
// CTA starts on a cold L1.  The copies are bulk copies under one mbarrier that a thread waits for
// only when it has its first item.  Time of a step's decisions (one launch, exact energies for
// every move): 64 boxes of 300-30,000 atoms, 1,175 moves, 79 us before and 41 us now; four boxes
// of 2,700 DMSO + 5,300 water, 108 moves, 149 us and 31 us; the same boxes' proposals with
// features 77 us and 18.5 us.
template <int MAXT>
__global__ void __launch_bounds__(MAXT, 1024 / MAXT) bmc_decide_kernel(epsr_bmc_t B, int step, int mode, const float *y,
                                                                    float *target, int table_bytes) {
    extern __shared__ __align__(16) unsigned char bmc_smem[];
    __shared__ double dws[33];
    __shared__ float4 p_old[BMC_MAXAT], p_new[BMC_MAXAT];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int s_go, s_rows;
    const int k = blockIdx.x;
    const int mol = B.slot_mol[k];
    const int b = B.slot_box[k];
    const epsr_bmc_box_t &X = B.box[b];
    long long *cnt4 = B.counters + 4 * b;
    const float qnan = __int_as_float(0x7fc00000);
    if (mol == -1) {
        if (target && threadIdx.x == 0) target[k] = qnan;
        return;
    }
    if (mol == -2) {
        if (threadIdx.x == 0) {
            atomicAdd((unsigned long long *)cnt4, 1ull);
            atomicAdd((unsigned long long *)(cnt4 + 3), 1ull);
            if (target) target[k] = qnan;
        }
        return;
    }
    const U4 r = philox4x32(U4{(uint32_t)X.sweep, (uint32_t)step, (uint32_t)k, P_DECIDE}, X.key0, X.key1);
    const int a0 = B.naf[mol], na_ = B.nato[mol];
    const int ntype = X.ntype, ns = X.izcut - 1;   // table points in range: iz 2 .. izcut
    float sg = 0.0f;
    if (threadIdx.x == 0) {
        int go = 1;
        atomicAdd((unsigned long long *)cnt4, 1ull);
        if (mode == 1) {
            sg = 0.5f * (y[2 * k] - y[2 * k + 1]);
            sg = fminf(fmaxf(sg, -40.0f), 40.0f);
            go = sg <= 0.0f || (double)u01(r.x) < exp(-(double)sg);
        }
        if (go) atomicAdd((unsigned long long *)(cnt4 + 1), 1ull);
        else if (target) target[k] = qnan;
        s_go = go;
        umma::mbar_init(&bar, 1);
        umma::fence_mbar_init();
    } else if (threadIdx.x >= 32 && threadIdx.x < 64) {   // the pairs of the box's types: rows of its table
        int rows = 0;
        for (int i = threadIdx.x - 32; i < ntype * ntype; i += 32) rows = max(rows, B.npairref[X.npairref0 + i] + 1);
        rows = __reduce_max_sync(0xffffffffu, rows);
        if (threadIdx.x == 32) s_rows = rows;
    }
    __syncthreads();
    if (!s_go) return;   // first stage rejected: no pair energy is evaluated
    using S = std::conditional_t<(MAXT > BMC_THREADS), WideSearch, NarrowSearch>;
    float4 *s_tab = (float4 *)(bmc_smem + sizeof(S));
    const int rows = s_rows;
    const size_t row_bytes = 16 * (size_t)max(ns, 1), need = row_bytes * rows + 4 * (size_t)max(ns, 1) +
                                                             4 * (size_t)ntype * ntype;
    const bool staged = ns > 0 && need <= (size_t)table_bytes;
    float *s_xs = (float *)(s_tab + (size_t)rows * max(ns, 1));
    int *s_pr = (int *)(s_xs + max(ns, 1));
    MoveChange change;
    change.pos = (const float4 *)B.pos;
    change.stepcl = X.stepcl;
    change.izlast = X.izcut - 2;
    change.skip = skip_dsq(X.stepcl, X.izcut);
    change.rcp = step_rcp(X.stepcl, X.izcut);
    change.ntype = ntype;
    const float4 *g_tab = (const float4 *)B.tab + X.tab0 + 2;
    if (staged) {
        if (threadIdx.x == 0) {
            umma::mbar_expect_tx(&bar, (uint32_t)(row_bytes * rows));
            for (int i = 0; i < rows; ++i) umma::bulk_load(s_tab + (size_t)i * ns, g_tab + (size_t)i * X.ld, row_bytes, &bar);
        }
        for (int i = threadIdx.x; i < ns; i += blockDim.x) s_xs[i] = B.xstar[X.xstar0 + 2 + i];
        for (int i = threadIdx.x; i < ntype * ntype; i += blockDim.x) s_pr[i] = B.npairref[X.npairref0 + i];
        change.tab = s_tab;
        change.xs = s_xs;
        change.pr = s_pr;
        change.ld = ns;
    } else {
        change.tab = g_tab;
        change.xs = B.xstar + X.xstar0 + 2;
        change.pr = B.npairref + X.npairref0;
        change.ld = X.ld;
    }
    const float4 *sn = (const float4 *)B.slot_new + (size_t)k * BMC_MAXAT;
    for (int q = threadIdx.x; q < na_; q += blockDim.x) {
        p_old[q] = atom_pos(B, a0 + q);
        p_new[q] = sn[q];
    }
    // the partners whose centre is within rint of the old centre (rint covers the cutoff, both
    // molecules' extents and the largest displacement)
    int ix, iy, iz;
    slot_cell(X, k, step, ix, iy, iz);
    const Near P{ix, iy, iz, X.nrange, na_, mol_word(B, X, mol), B.xadd[mol], B.yadd[mol], B.zadd[mol],
                 __fmul_rn(X.rint, X.rint), item_range2(B, X, b, (float)(X.izcut + 1) * X.stepcl), p_old, p_new};
    double de = 0.0;
    bool here = !staged, late = false;   // the tables have arrived; they did not in time
    const int scanned = near_items(B, X, b, P, *(S *)bmc_smem, [&](int b0, int nb, int a) {
        if (!here) {
            late = !umma::mbar_wait(&bar, 0, nullptr);
            here = true;
        }
        if (!late) de += change.item(p_old[a], p_new[a], b0, nb);
    });
    if (!here) late = !umma::mbar_wait(&bar, 0, nullptr);   // no copy lands after the CTA has gone
    de = block_sum_d(de, dws);
    if (__syncthreads_or(late) || scanned > BMC_LIST) {
        if (threadIdx.x == 0) atomicExch(B.status, scanned > BMC_LIST ? 2 : 1);
        return;
    }
    finish_move(B, X, k, b, mol, a0, na_, de, sg, r.y, target, p_new, &s_go);
}

// ----------------------------------------------------------------- total energy
__global__ void __launch_bounds__(BMC_THREADS) bmc_mol_energy_kernel(epsr_bmc_t B) {
    __shared__ int list[BMC_LIST];
    __shared__ int scan_ws[33];
    __shared__ double dws[33];
    const int mol = blockIdx.x;
    const int b = B.mol_box[mol];
    const epsr_bmc_box_t &X = B.box[b];
    const int n = X.ncell;
    const int ix = cell_coord(B.xadd[mol], X.shift[0], n), iy = cell_coord(B.yadd[mol], X.shift[1], n),
              iz = cell_coord(B.zadd[mol], X.shift[2], n);
    const int cnt = gather_partners(B, X, b, ix, iy, iz, X.nrange, list, scan_ws);
    if (cnt < 0) {
        if (threadIdx.x == 0) atomicExch(B.status, 2);
        return;
    }
    Lattice L;
    L.cubic = 1;
    const Tables T = box_tables(B, X);
    const float dsq_skip = skip_dsq(T.stepcl, T.izcut);
    const int *pr = B.npairref + X.npairref0;
    const int a0 = B.naf[mol], na_ = B.nato[mol];
    double e = 0.0;
    for (int p = threadIdx.x; p < cnt; p += blockDim.x) {
        const int jm = list[p];
        if (jm <= mol) continue;   // each pair once
        const int b0 = B.naf[jm], nb = B.nato[jm];
        float s = 0.0f;
        for (int a = 0; a < na_; ++a) {
            const float4 pa = atom_pos(B, a0 + a);
            const int *row = pr + __float_as_int(pa.w) * X.ntype;
            for (int q = 0; q < nb; ++q) {
                const float4 pb = atom_pos(B, b0 + q);
                s = __fadd_rn(s, pair_energy_far(L, T, dsq_skip, pa, pb, row[__float_as_int(pb.w)]));
            }
        }
        e += (double)s;
    }
    e = block_sum_d(e, dws);
    if (threadIdx.x == 0) B.emol[mol] = e;
}

__global__ void bmc_box_energy_kernel(epsr_bmc_t B) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B.nbox) return;
    const epsr_bmc_box_t &X = B.box[b];
    double e = 0.0;
    for (int m = 0; m < X.nmol; ++m) e += B.emol[X.mol0 + m];
    B.energy[b] = e;
}

// ----------------------------------------------------------------- histograms (atogen, all origins)
__global__ void bmc_hist_intra_kernel(epsr_bmc_t B, epsr_bmc_hist_t H) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= B.nmol) return;
    const int b = B.mol_box[m];
    const epsr_bmc_box_t &X = B.box[b];
    const int a0 = B.naf[m], n = B.nato[m];
    if (n <= 1) return;
    Lattice L;
    L.cubic = 1;
    const int ld = H.ldw[b], npt1 = H.npt1[b];
    unsigned long long *cnt = H.counts + H.hist0[b];
    const int *pr = B.npairref + X.npairref0;
    long long np = 0;
    for (int ia = a0; ia < a0 + n - 1; ++ia) {
        for (int ja = ia + 1; ja < a0 + n; ++ja) {
            const int icref = pr[__float_as_int(((const float4 *)B.pos)[ia].w) * X.ntype +
                                 __float_as_int(((const float4 *)B.pos)[ja].w)];
            const float d = dist_f(L, __fsub_rn(B.xa[ia], B.xa[ja]), __fsub_rn(B.ya[ia], B.ya[ja]),
                                   __fsub_rn(B.za[ia], B.za[ja]));
            const int iz1 = nint_i(__fdiv_rn(d, X.stepcl)) + 2;
            if (iz1 > 1 && iz1 <= npt1) atomicAdd(cnt + (size_t)icref * ld + iz1, 1ull);
            ++np;
        }
    }
    atomicAdd((unsigned long long *)(H.pairs + b), (unsigned long long)np);
}

__global__ void __launch_bounds__(1024) bmc_hist_inter_kernel(epsr_bmc_t B, epsr_bmc_hist_t H) {
    extern __shared__ unsigned char sm[];
    __shared__ int cls[PH_TYPES * PH_TYPES];
    const int it = blockIdx.x;
    const int b = H.items[3 * it], t0 = H.items[3 * it + 1], o0 = H.items[3 * it + 2];
    const epsr_bmc_box_t &X = B.box[b];
    const int np = H.npairs[b];
    const int nbins = np * H.ldw[b];
    const size_t tp_off = ((sizeof(unsigned int) * ((size_t)H.max_bins)) + 15) & ~(size_t)15;
    float4 *tp = (float4 *)(sm + tp_off);
    int *tm = (int *)(tp + H.tile);
    const int tn = min(H.tile, X.natom - t0);
    const float4 *pos = (const float4 *)B.pos + X.atom0;
    const int *amol = H.atom_mol + X.atom0;
    const int parts = blockDim.x / PH_ORIGINS, part = threadIdx.x / PH_ORIGINS;
    const int o = o0 + threadIdx.x % PH_ORIGINS;
    const bool in = o < X.natom;
    const int im = in ? amol[o] : 0x7fffffff;
    __shared__ int mols[2];   // the tile's first and last molecule
    PairHist P;
    P.hist = (unsigned int *)sm;
    P.hpot = P.hist + nbins;
    P.npairref = B.npairref + X.npairref0;
    P.rminex = H.rminex + H.pair0[b];
    P.ld = H.ldw[b];
    P.ntype = X.ntype;
    P.nlim = max(H.npt1[b] - 1, 0);
    P.stepcl = X.stepcl;
    P.rcp = hist_rcp(X.stepcl);
    P.dmax = X.dmax;
    P.rmax = hist_rmax(P.rminex, np);
    hist_stage_tile(P, pos + t0, amol + t0, tn, tp, tm, mols);
    if (!__syncthreads_or(mols[1] > im)) return;   // no target's molecule comes after an origin's
    for (int i = threadIdx.x; i < nbins + np; i += blockDim.x) P.hist[i] = 0;
    hist_stage_types(P, cls);
    __syncthreads();
    int uses = 0;
    if (in) {
        const float4 p1 = pos[o];
        const int per = ((tn + parts - 1) / parts + 3) & ~3;
        const int q0 = min(part * per, tn), q1 = min(q0 + per, tn);
        uses = P.ntype <= PH_TYPES ? hist_tile<true, true>(P, p1, im, true, tp, tm, q0, q1, mols, cls)
                                   : hist_tile<true, false>(P, p1, im, true, tp, tm, q0, q1, mols, cls);
    }
    uses = __reduce_add_sync(0xffffffffu, uses);
    if ((threadIdx.x & 31) == 0 && uses) atomicAdd((unsigned long long *)(H.pairs + b), (unsigned long long)uses);
    __syncthreads();
    unsigned long long *cnt = H.counts + H.hist0[b];
    for (int i = threadIdx.x; i < nbins; i += blockDim.x)
        if (P.hist[i]) atomicAdd(cnt + (size_t)nbins + i, (unsigned long long)P.hist[i]);
    for (int i = threadIdx.x; i < np; i += blockDim.x)
        if (P.hpot[i]) atomicAdd(cnt + (size_t)2 * nbins + i, (unsigned long long)P.hpot[i]);
}

// normalisation (:3857-3897) of box blockIdx.y, pair blockIdx.x
__global__ void bmc_hist_norm_kernel(epsr_bmc_t B, epsr_bmc_hist_t H) {
    const int b = blockIdx.y, ic = blockIdx.x;
    const int np = H.npairs[b];
    if (ic >= np) return;
    const epsr_bmc_box_t &X = B.box[b];
    const int ld = H.ldw[b], npt1 = H.npt1[b];
    const int p0 = H.pair0[b], t0 = H.type0[b];
    const int it = H.n1extr[p0 + ic], jt = H.n2extr[p0 + ic];
    const float *cfrac = H.cfrac + t0, *csampled = H.csampled + t0;
    float cprod = __fmul_rn(__fmul_rn(cfrac[it], cfrac[jt]), (float)X.natom);
    float cprod2 = __fmul_rn(csampled[it], cfrac[jt]);
    if (it != jt) {
        cprod = __fmul_rn(cprod, 2.0f);
        cprod2 = __fadd_rn(cprod2, __fmul_rn(csampled[jt], cfrac[it]));
    }
    const unsigned long long *cnt = H.counts + H.hist0[b];
    float *wav = H.wav + H.wav0[b];
    float *w1 = wav + (size_t)ic * ld, *w2 = wav + (size_t)(np + ic) * ld;
    const unsigned long long *c1 = cnt + (size_t)ic * ld, *c2 = cnt + (size_t)(np + ic) * ld;
    for (int iz = 1 + threadIdx.x; iz <= npt1; iz += blockDim.x) {
        const float v1 = (float)(2ull * c1[iz]);
        const float v2 = __fmul_rn((float)c2[iz], 2.0f);
        w1[iz] = cprod > 0.0f ? __fdiv_rn(v1, cprod) : 0.0f;
        w2[iz] = cprod2 > 0.0f ? __fdiv_rn(v2, cprod2) : 0.0f;
    }
    const unsigned long long pc = cnt[(size_t)2 * np * ld + ic];
    if (threadIdx.x == 0) H.potex[p0 + ic] = cprod2 > 0.0f ? __fdiv_rn(__fmul_rn((float)pc, cfrac[jt]), cprod2)
                                                           : (float)pc;
}

}  // namespace epsr

using namespace epsr;

namespace {
int check_bmc(const epsr_bmc_t *b, const char *who) {
    if (!b || !b->box || !b->slot_box || !b->mol_box || !b->naf || !b->nato || !b->fclass || !b->xa || !b->xadd ||
        !b->pos || !b->tab || !b->xstar || !b->npairref || !b->cell_start || !b->cell_mols || !b->mol_cell ||
        !b->slot_mol || !b->slot_new || !b->slot_off || !b->slot_centre || !b->energy || !b->counters ||
        !b->sweep_counter || !b->status || b->nbox <= 0 || b->nmol <= 0 || b->nslot <= 0 ||
        ((b->threads & ~EPSR_BMC_CELL_MOL) != 64 && (b->threads & ~EPSR_BMC_CELL_MOL) != 128 &&
         (b->threads & ~EPSR_BMC_CELL_MOL) != 256) ||
        ((b->threads & EPSR_BMC_CELL_MOL) && !b->cell_mol)) {
        epsr_set_error("%s: null pointer or empty batch", who);
        return EPSR_ERR_ARG;
    }
    return EPSR_OK;
}

// The kernels' copy of a checked structure: plain threads, and no cell_mol unless the caller's
// structure has one.
epsr_bmc_t plain_bmc(const epsr_bmc_t *b) {
    epsr_bmc_t B;
    memset(&B, 0, sizeof(B));
    memcpy(&B, b, offsetof(epsr_bmc_t, cell_mol));
    if (b->threads & EPSR_BMC_CELL_MOL) B.cell_mol = b->cell_mol;
    B.threads &= ~EPSR_BMC_CELL_MOL;
    return B;
}

// Threads of a moved molecule's CTA.  A step is one wave whose time is its slowest move's, and the
// kernels' registers let 1,024 threads share an SM: the caller's count, doubled while every move's
// CTA is still resident, so a few moves run wide and many narrow.
int move_threads(const epsr_bmc_t *b, int most) {
    int t = b->threads;
    while (t < most && 2ll * t * b->nslot <= 148ll * 1024) t *= 2;
    return t;
}
template <bool ODD>
int launch_features(const epsr_bmc_t *b, int t, int step, void *x, cudaStream_t s) {
    EPSR_SMEM_OPTIN(bmc_propose_kernel<ODD>);
    EPSR_TIMED("bmc_propose_kernel", s,
               bmc_propose_kernel<ODD><<<b->nslot, t, sizeof(WideSearch), s>>>(*b, step, (__nv_bfloat16 *)x));
    return EPSR_OK;
}
template <int T>
int launch_decide(const epsr_bmc_t *b, int t, int step, int mode, const float *y, float *target, cudaStream_t s) {
    // an SM's shared memory over the CTAs that share it, one each where there are SMs for all, else as many of T
    // threads as its registers hold: what the search leaves holds tables
    const int bytes = (220 * 1024) / (b->nslot <= 148 ? 1 : 1024 / T), table = bytes - (int)(T > BMC_THREADS ? sizeof(WideSearch) : sizeof(NarrowSearch)) - 4096;
    EPSR_SMEM_OPTIN(bmc_decide_kernel<T>);
    EPSR_TIMED("bmc_decide_kernel", s, bmc_decide_kernel<T><<<b->nslot, t, bytes - 4096, s>>>(*b, step, mode, y, target, table));
    return EPSR_OK;
}
}  // namespace

extern "C" int epsr_bmc_begin_sweep(const epsr_bmc_t *b, void *stream) {
    int rc = check_bmc(b, "epsr_bmc_begin_sweep");
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const epsr_bmc_t B = plain_bmc(b);
    // the cursor and the cell -> box map live after the molecule-cell array in mol_cell's
    // allocation: mol_cell [nmol], cursor [ncell + nbox], cell_box [ncell]
    int32_t *cursor = b->mol_cell + b->nmol;
    const int32_t *cell_box = cursor + b->ncell + b->nbox;
    bmc_begin_kernel<<<(b->nbox + 127) / 128, 128, 0, s>>>(B);
    EPSR_CUDA(cudaMemsetAsync(b->cell_start, 0, sizeof(int32_t) * (size_t)(b->ncell + b->nbox), s));
    EPSR_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int32_t) * (size_t)(b->ncell + b->nbox), s));
    bmc_count_kernel<<<(b->nmol + 255) / 256, 256, 0, s>>>(B);
    bmc_scan_kernel<<<b->nbox, 1024, 0, s>>>(B);
    bmc_scatter_kernel<<<(b->nmol + 255) / 256, 256, 0, s>>>(B, cursor);
    bmc_sort_kernel<<<(b->ncell + 7) / 8, 256, 0, s>>>(B, cell_box, b->ncell);
    if (B.cell_mol) bmc_order_kernel<<<(b->nmol + 255) / 256, 256, 0, s>>>(B);
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}

extern "C" int epsr_bmc_propose(const epsr_bmc_t *b, int32_t step, void *x, void *stream) {
    int rc = check_bmc(b, "epsr_bmc_propose");
    if (rc) return rc;
    if (step < 0) {
        epsr_set_error("epsr_bmc_propose: negative step");
        return EPSR_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const epsr_bmc_t B = plain_bmc(b);
    if (!x) {   // proposals alone: one warp a slot
        EPSR_TIMED("bmc_propose_kernel", s, bmc_propose_kernel<false><<<b->nslot, 32, 0, s>>>(B, step, nullptr));
    } else {
        const int t = move_threads(&B, BMC_MAXT);
        rc = ((uintptr_t)x & 3) ? launch_features<true>(&B, t, step, x, s) : launch_features<false>(&B, t, step, x, s);
        if (rc) return rc;
    }
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}

extern "C" int epsr_bmc_decide(const epsr_bmc_t *b, int32_t step, int32_t mode, const float *y, float *target,
                               void *stream) {
    int rc = check_bmc(b, "epsr_bmc_decide");
    if (rc) return rc;
    if (mode < 0 || mode > 2 || (mode == 1 && !y) || (mode == 2 && !target)) {
        epsr_set_error("epsr_bmc_decide: mode %d needs %s", mode, mode == 1 ? "y" : "target");
        return EPSR_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const epsr_bmc_t B = plain_bmc(b);
    // The decisions of molecules of a few atoms don't fill 1,024 threads, whose barriers then cost more than they
    // bring: plain sweeps of 48 boxes of 300 atoms of water and silica take 5.74 ms so, and 4.83 at 512 threads, of 16
    // of 1,200 24.5 and 22.2, of one of 30,000 4.38 and 4.22; of four of 2,700 DMSO + 5,300 water (5.4 atoms a
    // molecule) 11.05 and 11.15.  The features' searches reach further: learned sweeps of four boxes of 500 DMSO +
    // 1,000 water take 12.6 ms, and 13.3 with features by 512 threads.
    const int t = move_threads(&B, B.natom > 4ll * B.nmol ? BMC_MAXT : BMC_MAXD);
    rc = t <= BMC_THREADS ? launch_decide<BMC_THREADS>(&B, t, step, mode, y, target, s)
         : t <= BMC_MAXD  ? launch_decide<BMC_MAXD>(&B, t, step, mode, y, target, s)
                          : launch_decide<BMC_MAXT>(&B, t, step, mode, y, target, s);
    if (rc) return rc;
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}

extern "C" int epsr_bmc_end_sweep(const epsr_bmc_t *b, void *stream) {
    int rc = check_bmc(b, "epsr_bmc_end_sweep");
    if (rc) return rc;
    bmc_end_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(plain_bmc(b));
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}

extern "C" int epsr_bmc_total_energy(const epsr_bmc_t *b, void *stream) {
    int rc = check_bmc(b, "epsr_bmc_total_energy");
    if (rc) return rc;
    if (!b->emol) {
        epsr_set_error("epsr_bmc_total_energy: emol scratch missing");
        return EPSR_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const epsr_bmc_t B = plain_bmc(b);
    bmc_mol_energy_kernel<<<b->nmol, BMC_THREADS, 0, s>>>(B);
    bmc_box_energy_kernel<<<(b->nbox + 127) / 128, 128, 0, s>>>(B);
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}

extern "C" int epsr_bmc_histograms(const epsr_bmc_t *b, const epsr_bmc_hist_t *h, int64_t counts_len, void *stream) {
    int rc = check_bmc(b, "epsr_bmc_histograms");
    if (rc) return rc;
    if (!h || !h->items || !h->hist0 || !h->wav0 || !h->npairs || !h->npt1 || !h->ldw || !h->pair0 || !h->type0 ||
        !h->n1extr || !h->n2extr || !h->atom_mol || !h->rminex || !h->cfrac || !h->csampled || !h->counts || !h->wav ||
        !h->potex || !h->pairs || h->nitems <= 0 || h->tile <= 0 || h->tile > 4096 || h->max_bins <= 0 ||
        counts_len <= 0) {
        epsr_set_error("epsr_bmc_histograms: null pointer or bad sizes");
        return EPSR_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const epsr_bmc_t B = plain_bmc(b);
    const size_t shm = (((sizeof(unsigned int) * (size_t)h->max_bins) + 15) & ~(size_t)15) +
                       (sizeof(float4) + sizeof(int)) * (size_t)h->tile;
    if (shm > 220 * 1024) {
        epsr_set_error("epsr_bmc_histograms: %zu bytes of shared histogram and tile", shm);
        return EPSR_ERR_UNSUPPORTED;
    }
    if (shm > 48 * 1024) EPSR_SMEM_OPTIN(bmc_hist_inter_kernel);
    EPSR_CUDA(cudaMemsetAsync(h->counts, 0, sizeof(unsigned long long) * (size_t)counts_len, s));
    EPSR_CUDA(cudaMemsetAsync(h->pairs, 0, sizeof(long long) * (size_t)b->nbox, s));
    bmc_hist_intra_kernel<<<(b->nmol + 127) / 128, 128, 0, s>>>(B, *h);
    EPSR_TIMED("bmc_hist_inter_kernel", s, bmc_hist_inter_kernel<<<h->nitems, hist_threads(shm), shm, s>>>(B, *h));
    bmc_hist_norm_kernel<<<dim3(64, b->nbox), 256, 0, s>>>(B, *h);
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}
