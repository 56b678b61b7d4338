// Block-per-quartet Rys ERI + J/K kernel of the f classes and the deep d
// classes: bra class at run time, ket class (LC, LD) at compile time.
//
// One thread block evaluates one contracted quartet at a time.  Items
// (primitive quartet x root, up to nb_items per batch):
//  A. a thread per (item, axis) runs the 2-D recurrence of its axis in
//     registers and writes the table G(i <= La+Lb, k <= Lc+Ld) to shared
//     memory;
//  B. a thread owns a bra row (a0| and a chunk of at most kRowCols ket columns
//     |c0) of the radial block, reads the three G rows of its exponents once
//     per item and keeps the chunk's sums in registers over all batches; the
//     blocks' spare threads take every groups-th item.
// One item and row costs 3 (Lc+Ld+1) shared loads for all its columns, where
// the entry-per-thread form (eri_generic.cuh) loads three values per entry and
// keeps the sums in shared memory: that one was bound by the shared-memory
// pipe (74% of the L1 wavefront rate, FP64 pipe 11%).
// Then X = T PK^T and V = PB X with the plan's pair projectors and the J/K
// digestion, as in eri_generic.cuh.
#pragma once

#include "eri_common.cuh"
#include "eri_fast.cuh"

namespace tlno_gpu {
namespace dev {

constexpr int kRowCols = 16;      // ket columns per thread
constexpr int kRowMaxGroups = 4;  // item groups per block

template <int LC, int LD>
struct RowsKet {
    static constexpr int LCD = LC + LD, KS = LCD + 1, KSP = (KS + 1) / 2 * 2;
    static constexpr int OFC = ce_off(LC), NCS = ce_cum(LCD) - OFC;
    static constexpr int CH = (NCS + kRowCols - 1) / kRowCols, CC = (NCS + CH - 1) / CH;
};

// The sizes the digestion needs, those of the ket at compile time (its index
// divisions then cost no division).
template <int LC, int LD>
struct RowsDims {
    static constexpr int nc = ce_nsph(LC), nd = ce_nsph(LD), nscd = nc * nd;
    int na, nb, nsab, off_P;
};

// Block shape and shared-memory layout (in elements of double) of a class.
struct RowsLayout {
    int las, lcs, ksp, gs, slot, nas, ncs, na, nb, nc, nd, nsab, nscd;
    int rpad, ch, groups, threads, nb_items;
    int off_X, off_V, off_P, off_T, words;
    __host__ __device__ void init(int la, int lb, int lc, int ld, int nbi) {
        las = la + lb;
        lcs = lc + ld;
        ksp = (lcs + 2) / 2 * 2;
        // axis stride: even (16-byte rows), its half odd (few bank conflicts
        // between the threads' tables)
        gs = (las + 1) * ksp;
        if ((gs / 2) % 2 == 0) gs += 2;
        slot = 3 * gs;
        nas = ncart_cum(las) - cart_offset(la);
        ncs = ncart_cum(lcs) - cart_offset(lc);
        na = nsph(la); nb = nsph(lb); nc = nsph(lc); nd = nsph(ld);
        nsab = na * nb;
        nscd = nc * nd;
        ch = (ncs + kRowCols - 1) / kRowCols;
        // several chunks: whole warps per chunk, so that a warp runs one chunk's code
        rpad = ch > 1 ? (nas + 31) / 32 * 32 : nas;
        threads = rpad * ch <= 128 ? 128 : (rpad * ch + 31) / 32 * 32;
        groups = threads / (rpad * ch);
        if (groups > kRowMaxGroups) groups = kRowMaxGroups;
        nb_items = nbi;
        const int g_words = nb_items * slot;
        off_X = 0;
        off_V = off_X + nas * nscd;
        off_P = off_V + nsab * nscd;
        const int tail = off_P + na * nb + nc * nd + nb * nd + nb * nc + na * nd + na * nc;
        off_T = ((g_words > tail ? g_words : tail) + 1) & ~1;
        // odd row stride: the rows' threads store to different banks (the even
        // stride of 16 was a 32-way conflict, two thirds of all wavefronts)
        words = (off_T + nas * (ncs | 1) + 1) & ~1;
    }
};

// 1/x and 1/sqrt(x) of p + q, each within the rounding of a division and a
// square root: rsqrt_pos (in FP32, the bare instruction of 2^-22.9, one Newton
// step further) and one step on its square.
template <typename R>
__device__ __forceinline__ void reciprocals(R x, R& inv, R& rs) {
    rs = rsqrt_pos(x);
    if (sizeof(R) == 4) rs = fma(R(0.5) * rs, fma(-x * rs, rs, R(1)), rs);
    inv = rs * rs;
    inv = fma(inv, fma(-x, inv, R(1)), inv);
}

// One axis table in registers, column by column:
// G(i, k+1) = d00 G(i, k) + i b00 G(i-1, k) + k b01 G(i, k-1).
template <typename R, int LAB, int LCD, int KSP>
__device__ __forceinline__ void rows_vrr(R* G, R c00, R d00, R b00, R b10, R b01, R seed) {
    R prev[LAB + 1], cur[LAB + 1];
    cur[0] = seed;
    if constexpr (LAB > 0) cur[1] = c00 * seed;
#pragma unroll
    for (int i = 1; i < LAB; ++i) cur[i + 1] = c00 * cur[i] + R(i) * b10 * cur[i - 1];
#pragma unroll
    for (int k = 0; k <= LCD; ++k) {
#pragma unroll
        for (int i = 0; i <= LAB; ++i) G[i * KSP + k] = cur[i];
        if (k == LCD) break;
        R next[LAB + 1];
#pragma unroll
        for (int i = 0; i <= LAB; ++i) {
            R v = d00 * cur[i];
            if (i > 0) v += R(i) * b00 * cur[i - 1];
            if (k > 0) v += R(k) * b01 * prev[i];
            next[i] = v;
        }
#pragma unroll
        for (int i = 0; i <= LAB; ++i) {
            prev[i] = cur[i];
            cur[i] = next[i];
        }
    }
}

// Phase B of chunk CHUNK: items s0, s0 + step, ... of a batch.
template <typename R, int LC, int LD, int CHUNK>
__device__ __forceinline__ void rows_accumulate(const R* g, int slot, int s0, int nvalid, int step, int xo, int yo,
                                                int zo, R (&acc)[RowsKet<LC, LD>::CC]) {
    using K = RowsKet<LC, LD>;
    using V2 = typename RysTab<R>::V2;
    for (int s = s0; s < nvalid; s += step) {
        const V2* px = reinterpret_cast<const V2*>(g + s * slot + xo);
        const V2* py = reinterpret_cast<const V2*>(g + s * slot + yo);
        const V2* pz = reinterpret_cast<const V2*>(g + s * slot + zo);
        R x[K::KSP], y[K::KSP], z[K::KSP];
#pragma unroll
        for (int h = 0; h < K::KSP / 2; ++h) {
            const V2 u = px[h], v = py[h], w = pz[h];
            x[2 * h] = u.x; x[2 * h + 1] = u.y;
            y[2 * h] = v.x; y[2 * h + 1] = v.y;
            z[2 * h] = w.x; z[2 * h + 1] = w.y;
        }
        sfor<K::CC>([&](auto J) {
            constexpr int ic = CHUNK * K::CC + TLNO_CI(J);
            if constexpr (ic < K::NCS) {
                constexpr int fc = K::OFC + ic;
                acc[TLNO_CI(J)] += (x[ce_x(fc)] * y[ce_y(fc)]) * z[ce_z(fc)];
            }
        });
    }
}

template <typename R, int LC, int LD, int CHUNK = 0>
__device__ __forceinline__ void rows_dispatch(int chunk, const R* g, int slot, int s0, int nvalid, int step, int xo,
                                              int yo, int zo, R (&acc)[RowsKet<LC, LD>::CC]) {
    if constexpr (CHUNK < RowsKet<LC, LD>::CH) {
        if (chunk == CHUNK)
            rows_accumulate<R, LC, LD, CHUNK>(g, slot, s0, nvalid, step, xo, yo, zo, acc);
        else
            rows_dispatch<R, LC, LD, CHUNK + 1>(chunk, g, slot, s0, nvalid, step, xo, yo, zo, acc);
    }
}

// out[row * ns + s] = sum_k A(row, k) B(k, s): TILE rows and one s per thread
// and pass, so that a B value serves TILE sums; four steps of k in flight.
template <int TILE, typename FA, typename FB>
__device__ __forceinline__ void rows_product_tile(int nrows, int ns, int nk, FA&& a, FB&& b, double* out) {
    const int blocks = (nrows + TILE - 1) / TILE;
    for (int e = threadIdx.x; e < blocks * ns; e += blockDim.x) {
        const int rb = e / ns, s = e - rb * ns, r0 = rb * TILE;
        double sum[TILE];
#pragma unroll
        for (int t = 0; t < TILE; ++t) sum[t] = 0.0;
#pragma unroll 4
        for (int k = 0; k < nk; ++k) {
            const double v = b(k, s);
#pragma unroll
            for (int t = 0; t < TILE; ++t) sum[t] += a(min(r0 + t, nrows - 1), k) * v;
        }
#pragma unroll
        for (int t = 0; t < TILE; ++t)
            if (r0 + t < nrows) out[(r0 + t) * ns + s] = sum[t];
    }
}

// The smallest tile that covers the product in one pass of the block.
template <typename FA, typename FB>
__device__ __forceinline__ void rows_product(int nrows, int ns, int nk, FA&& a, FB&& b, double* out) {
    const int nt = blockDim.x;
    if ((nrows + 1) / 2 * ns <= nt) rows_product_tile<2>(nrows, ns, nk, a, b, out);
    else if ((nrows + 3) / 4 * ns <= nt) rows_product_tile<4>(nrows, ns, nk, a, b, out);
    else rows_product_tile<6>(nrows, ns, nk, a, b, out);
}

template <typename R, int LC, int LD>
__device__ void rows_quartet(const PlanView& pv, const ClassLaunch& cl, const RowsLayout& lay, double* sm, int bra,
                             int ket, bool jon, bool kon, int group, int chunk, int row, int xo, int yo, int zo) {
    using K = RowsKet<LC, LD>;
    const int tid = threadIdx.x, nt = blockDim.x;
    const PairRec br = load_pair_rec(pv.pair_rec + bra), kr = load_pair_rec(pv.pair_rec + ket);
    const int nroots = (lay.las + lay.lcs) / 2 + 1;
    const int npb = br.nprim, npk = kr.nprim;
    const DPrimPair* pb = pv.prim + br.prim_off;
    const DPrimPair* pk = pv.prim + kr.prim_off;
    R* Gs = reinterpret_cast<R*>(sm);
    R* T = reinterpret_cast<R*>(sm + lay.off_T);
    const int n_items = npb * npk * nroots;
    const bool fs_on = cl.fs_thr2 > 0.0;
    R acc[K::CC];
#pragma unroll
    for (int k = 0; k < K::CC; ++k) acc[k] = R(0);
    for (int base = 0; base < n_items; base += lay.nb_items) {
        const int nvalid = min(lay.nb_items, n_items - base);
        for (int task = tid; task < 3 * nvalid; task += nt) {
            const int slot = task / 3, ax = task - 3 * slot;
            const int item = base + slot;
            const int r = item % nroots, pq = item / nroots;
            const int ib = pq / npk, ik = pq - ib * npk;
            const DPrimPair bp = pb[ib];
            const DPrimPair kp = pk[ik];
            const R p = R(bp.p), q = R(kp.p);
            R inv, rs;
            reciprocals(p + q, inv, rs);
            const R PQ[3] = {R(bp.Px) - R(kp.Px), R(bp.Py) - R(kp.Py), R(bp.Pz) - R(kp.Pz)};
            const R Targ = p * q * inv * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
            R t2, wt;
            if (sizeof(R) == 4 && nroots >= 4) {
                // FP64 carve-out of the FP32 pass: high-L roots and weights
                double t2d, wtd;
                rys_root<double>(nroots, double(Targ), r, t2d, wtd);
                t2 = R(t2d);
                wt = R(wtd);
            } else {
                rys_root<R>(nroots, Targ, r, t2, wt);
            }
            R pref = R(34.98683665524972497) * R(bp.w) * R(kp.w) * rs;
            if (fs_on && !(pv.prim_fs[br.prim_off + ib] * pv.prim_fs[kr.prim_off + ik] >= cl.fs_thr2)) pref = R(0);
            const R qo = q * inv, po = p * inv;
            const R b00 = R(0.5) * inv * t2;
            const R b10 = R(0.5) * R(bp.invp) * (R(1) - qo * t2);
            const R b01 = R(0.5) * R(kp.invp) * (R(1) - po * t2);
            const double bP = ax == 0 ? bp.Px : ax == 1 ? bp.Py : bp.Pz, kP = ax == 0 ? kp.Px : ax == 1 ? kp.Py : kp.Pz;
            const double bA = ax == 0 ? br.A[0] : ax == 1 ? br.A[1] : br.A[2];
            const double kC = ax == 0 ? kr.A[0] : ax == 1 ? kr.A[1] : kr.A[2];
            const R pqx = ax == 0 ? PQ[0] : ax == 1 ? PQ[1] : PQ[2];
            const R c00 = (R(bP) - R(bA)) - qo * pqx * t2;
            const R d00 = (R(kP) - R(kC)) + po * pqx * t2;
            const R seed = ax == 2 ? pref * wt : R(1);
            R* g = Gs + slot * lay.slot + ax * lay.gs;
            switch (lay.las) {
                case 2: rows_vrr<R, 2, K::LCD, K::KSP>(g, c00, d00, b00, b10, b01, seed); break;
                case 3: rows_vrr<R, 3, K::LCD, K::KSP>(g, c00, d00, b00, b10, b01, seed); break;
                case 4: rows_vrr<R, 4, K::LCD, K::KSP>(g, c00, d00, b00, b10, b01, seed); break;
                case 5: rows_vrr<R, 5, K::LCD, K::KSP>(g, c00, d00, b00, b10, b01, seed); break;
                default: rows_vrr<R, 6, K::LCD, K::KSP>(g, c00, d00, b00, b10, b01, seed); break;
            }
        }
        __syncthreads();
        if (row >= 0) rows_dispatch<R, LC, LD>(chunk, Gs, lay.slot, group, nvalid, lay.groups, xo, yo, zo, acc);
        __syncthreads();
    }
    // radial block: the item groups add up in turn
    for (int gi = 0; gi < lay.groups; ++gi) {
        if (row >= 0 && group == gi) {
#pragma unroll
            for (int k = 0; k < K::CC; ++k) {
                const int ic = chunk * K::CC + k;
                if (ic < K::NCS) {
                    R* t = T + row * (K::NCS | 1) + ic;
                    *t = gi == 0 ? acc[k] : *t + acc[k];
                }
            }
        }
        __syncthreads();
    }

    // HRR + spherical projection: X = T PK^T, V = PB X (transposed projectors,
    // consecutive threads on consecutive ket rows).
    const double* PBt = pv.proj + pv.proj_off[bra];
    const double* PKt = pv.proj + pv.proj_off[ket];
    double* X = sm + lay.off_X;
    double* V = sm + lay.off_V;
    constexpr int nscd = RowsDims<LC, LD>::nscd;
    const int nsab = lay.nsab;
    rows_product(lay.nas, nscd, K::NCS, [&](int ia, int ic) { return double(T[ia * (K::NCS | 1) + ic]); },
                 [&](int ic, int s) { return __ldg(PKt + ic * nscd + s); }, X);
    __syncthreads();
    rows_product(nsab, nscd, lay.nas, [&](int sab, int ia) { return __ldg(PBt + ia * nsab + sab); },
                 [&](int ia, int s) { return X[ia * nscd + s]; }, V);
    __syncthreads();
    const RowsDims<LC, LD> dims{lay.na, lay.nb, nsab, lay.off_P};
    block_digest(pv, cl, dims, sm, V, br, kr, bra, ket, jon, kon);
}

// Largest block of a ket class (bra (ff): 74 rows in whole warps per chunk) and
// the resident blocks its registers are capped for: the kernel waits at
// barriers and on L2, so 5 blocks of 128 threads beat 3 uncapped or 6 (f-shell
// 14 atoms, its 20 classes: 15.0, 13.3 and 14.1 ms).
__host__ __device__ constexpr int rows_max_threads(int ch) { return ch == 1 ? 128 : 96 * ch; }
__host__ __device__ constexpr int rows_min_blocks(int ch) { return ch == 1 ? 5 : ch == 2 ? 3 : ch == 3 ? 2 : 1; }

// Tiled schedule: tile = 1 bra pair x bk ket pairs, handed out by a block-wide
// dynamic counter in parts of `part` kets (eri_generic_cta_jk_kernel).
template <typename R, int LC, int LD>
__global__ void __launch_bounds__(rows_max_threads(RowsKet<LC, LD>::CH), rows_min_blocks(RowsKet<LC, LD>::CH))
    eri_rows_jk_kernel(PlanView pv, ClassLaunch cl, int nb_items, int part) {
    extern __shared__ __align__(16) double smem[];  // the G rows are read as 16-byte vectors
    RowsLayout lay;
    lay.init(cl.la, cl.lb, LC, LD, nb_items);
    __shared__ int s_tile;
    const int per = lay.rpad * lay.ch;
    const int group = threadIdx.x / per, rem = threadIdx.x - group * per;
    const int chunk = rem / lay.rpad;
    int row = rem - chunk * lay.rpad;
    if (row >= lay.nas || group >= lay.groups) row = -1;
    int xo = 0, yo = 0, zo = 0;
    if (row >= 0) {
        const signed char* e = c_cart.xyz[cart_offset(cl.la) + row];
        xo = e[0] * lay.ksp;
        yo = lay.gs + e[1] * lay.ksp;
        zo = 2 * lay.gs + e[2] * lay.ksp;
    }
    const double thr = (cl.prec_mode != 0) ? cl.tau_mix / fmax(*cl.dmax, 1e-300) : 0.0;
    const int parts = (cl.bk + part - 1) / part;
    const int nunits = (cl.tile_end - cl.tile_begin) * parts;
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(cl.counter, 1);
        __syncthreads();
        const int t = s_tile;
        __syncthreads();
        if (t >= nunits) break;
        const int tile = cl.tile_begin + t / parts;
        const int j0 = t % parts * part;
        const int b = find_block(cl.tile_prefix, cl.n_blocks, tile);
        const int kb = tile - __ldg(cl.tile_prefix + b);
        const BlockDesc bd = cl.blocks[b];
        const int bra = __ldg(cl.bra_list + bd.bra0);  // one bra per block
        const int i = bra - bd.xbeg;
        const double qi = pv.pair_Q[bra];
        for (int jj = j0; jj < min(j0 + part, cl.bk); ++jj) {
            const int j = kb * cl.bk + jj;
            if (j >= bd.nket) break;
            if (cl.same && bd.koff + j > i) break;
            const int ket = bd.ket0 + j;
            const double qq = qi * pv.pair_Q[ket];
            if (!(qq >= cl.tau)) continue;
            if (cl.prec_mode == 1 && !(qq >= thr)) continue;
            if (cl.prec_mode == 2 && qq >= thr) continue;
            bool lj = true, lk = true;
            if (cl.den.mode) {
                const int mol = pv.pair_mol ? pv.pair_mol[ket] : 0;
                density_live(cl, pv, mol, pv.pair_A[bra], pv.pair_B[bra], pv.pair_A[ket], pv.pair_B[ket], qq, lj, lk);
                if (!lj && !lk) continue;
            }
            rows_quartet<R, LC, LD>(pv, cl, lay, smem, bra, ket, lj, lk, group, chunk, row, xo, yo, zo);
        }
    }
}

}  // namespace dev
}  // namespace tlno_gpu
