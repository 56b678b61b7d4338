// Launch descriptors and J/K digestion shared by the ERI kernels.
#pragma once

#include "device_common.cuh"
#include "launch_types.hpp"

namespace tlno_gpu {
namespace dev {

enum Mode { kStore = 0, kSchwarz = 1, kJK = 2 };

__device__ __forceinline__ PairRec load_pair_rec(const PairRec* p) {
    PairRec r;
    const int4* src = reinterpret_cast<const int4*>(p);
    int4* dst = reinterpret_cast<int4*>(&r);
#pragma unroll
    for (int k = 0; k < 5; ++k) dst[k] = __ldg(src + k);
    return r;
}

// Bra-block index of a linear tile via binary search in the prefix array.
__device__ __forceinline__ int find_block(const int* prefix, int n_blocks, int tile) {
    int lo = 0, hi = n_blocks - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Density (CVHF) screen of one quartet of global shells (A B | C D) of
// molecule `mol` with pair metric product q (the plan's Schwarz test already
// passed): whether its Coulomb (lj) and exchange (lk) contributions are kept.
// Same predicate as the reference (native_quartets.ipp:499-518,
// rys_engine.ipp:1126-1167) with the raised cutoff of direct_build.ipp:229-251.
__device__ __forceinline__ void density_live(const ClassLaunch& cl, const PlanView& pv, int mol, int A, int B,
                                             int C, int D, double q, bool& lj, bool& lk) {
    const DensityScreen& ds = cl.den;
    const int so = pv.mol_shell_off ? __ldg(pv.mol_shell_off + mol) : 0;
    const int n = pv.mol_ns ? __ldg(pv.mol_ns + mol) : 0;
    const double* blk = ds.rho_blk + (ds.rho_off ? __ldg(ds.rho_off + mol) : 0);
    const int a = A - so, b = B - so, c = C - so, d = D - so;
    const int ns = pv.mol_ns ? n : cl.M_shells;
    const double rab = __ldg(blk + (long long)a * ns + b), rcd = __ldg(blk + (long long)c * ns + d);
    const double coul = 4.0 * fmax(rab, rcd);
    const double rho = __ldg(ds.rho_max + mol);
    double tj = cl.tau, tk = cl.tau;
    if (rho > 0.0) {
        tj = fmax(cl.tau, ds.thr / (rho * 4.0));
        tk = fmax(cl.tau, ds.thr / rho);
    }
    const double exch = fmax(fmax(__ldg(blk + (long long)c * ns + a), __ldg(blk + (long long)d * ns + a)),
                             fmax(__ldg(blk + (long long)c * ns + b), __ldg(blk + (long long)d * ns + b)));
    if (ds.mode == 2) {
        lj = lk = (q >= tj) && (q * fmax(coul, exch) >= ds.thr);
    } else {
        lj = (q >= tj) && (q * coul >= ds.thr);
        lk = (q >= tk) && (q * exch >= ds.thr);
    }
}

// Canonical AO pair index of (i, j): max(i,j) (max(i,j)+1) / 2 + min(i,j).
__device__ __forceinline__ long long ao_pair_index(int i, int j) {
    const long long hi = i > j ? i : j, lo = i > j ? j : i;
    return hi * (hi + 1) / 2 + lo;
}

// Whether element (a0+sa, b0+sb | c0+sc, d0+sd) of quartet (AB|CD) belongs
// to the canonical unique set of the ERI stream: i >= j inside a shell pair
// with A == B, k >= l with C == D, and kl <= ij when bra and ket are the
// same shell pair (rys_engine.ipp:690-708).
__device__ __forceinline__ bool canonical_element(bool same_ab, bool same_cd, bool same_pair, int a0, int sa,
                                                  int b0, int sb, int c0, int sc, int d0, int sd) {
    if (same_ab && sb > sa) return false;
    if (same_cd && sd > sc) return false;
    if (same_pair && ao_pair_index(c0 + sc, d0 + sd) > ao_pair_index(a0 + sa, b0 + sb)) return false;
    return true;
}

// Smallest pair metric product that can pass the density screen of molecule
// `mol` (the raised cutoff), for whole-tile skips.
__device__ __forceinline__ double density_tau_min(const ClassLaunch& cl, int mol) {
    const double rho = __ldg(cl.den.rho_max + mol);
    return rho > 0.0 ? fmax(cl.tau, cl.den.thr / (rho * 4.0)) : cl.tau;
}

// J/K digestion (or checksum) of the finished spherical block V of one quartet
// by a whole thread block; `sm` holds the density blocks at lay.off_P.  Ends
// with a block barrier.
template <typename Layout>
__device__ void block_digest(const PlanView& pv, const ClassLaunch& cl, const Layout& lay, double* sm,
                             const double* V, const PairRec& br, const PairRec& kr, int bra, int ket, bool jon,
                             bool kon) {
    const int tid = threadIdx.x, nt = blockDim.x;
    const int A = br.shA, B = br.shB, C = kr.shA, D = kr.shB;
    const int a0 = br.a0, b0 = br.b0, c0 = kr.a0, d0 = kr.b0;
    if (cl.checksum) {
        // ERI checksum stream: canonical unique elements of the block
        double s = 0.0;
        for (int e = tid; e < lay.nsab * lay.nscd; e += nt) {
            const int sab = e / lay.nscd, scd = e - sab * lay.nscd;
            if (canonical_element(A == B, C == D, bra == ket, a0, sab / lay.nb, b0, sab % lay.nb, c0,
                                  scd / lay.nd, d0, scd % lay.nd))
                s += V[e];
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((tid & 31) == 0 && s != 0.0) atomicAdd(cl.checksum, s);
        __syncthreads();
        return;
    }
    // J/K digestion with shell-level degeneracy f (consumer_policies.ipp:87-157)
    const int mol = pv.pair_mol ? pv.pair_mol[bra] : 0;
    const int M = pv.mol_M ? pv.mol_M[mol] : cl.M;
    const long long mbase = pv.mol_mat_off ? pv.mol_mat_off[mol] : 0;
    const double* Dm = cl.dens + mbase;
    double* Jm = cl.J + mbase;
    double* Km = cl.K + mbase;
    double f = 1.0;
    if (A == B) f *= 0.5;
    if (C == D) f *= 0.5;
    if (bra == ket) f *= 0.5;
    const int na = lay.na, nb = lay.nb, nc = lay.nc, nd = lay.nd;
    double* Pab = sm + lay.off_P;
    double* Pcd = Pab + na * nb;
    double* Pbd = Pcd + nc * nd;
    double* Pbc = Pbd + nb * nd;
    double* Pad = Pbc + nb * nc;
    double* Pac = Pad + na * nd;
    for (int e = tid; e < na * nb; e += nt) Pab[e] = Dm[(long long)(a0 + e / nb) * M + b0 + e % nb];
    for (int e = tid; e < nc * nd; e += nt) Pcd[e] = Dm[(long long)(c0 + e / nd) * M + d0 + e % nd];
    for (int e = tid; e < nb * nd; e += nt) Pbd[e] = Dm[(long long)(b0 + e / nd) * M + d0 + e % nd];
    for (int e = tid; e < nb * nc; e += nt) Pbc[e] = Dm[(long long)(b0 + e / nc) * M + c0 + e % nc];
    for (int e = tid; e < na * nd; e += nt) Pad[e] = Dm[(long long)(a0 + e / nd) * M + d0 + e % nd];
    for (int e = tid; e < na * nc; e += nt) Pac[e] = Dm[(long long)(a0 + e / nc) * M + c0 + e % nc];
    __syncthreads();
    const int nscd = lay.nscd;
    if (cl.want_j && jon) {
        const double fj = 4.0 * f;
        for (int sab = tid; sab < na * nb; sab += nt) {
            double s = 0.0;
            for (int t = 0; t < nscd; ++t) s += V[sab * nscd + t] * Pcd[t];
            atomicAdd(Jm + (long long)(a0 + sab / nb) * M + b0 + sab % nb, fj * s);
        }
        for (int scd = tid; scd < nscd; scd += nt) {
            double s = 0.0;
            for (int t = 0; t < na * nb; ++t) s += V[t * nscd + scd] * Pab[t];
            atomicAdd(Jm + (long long)(c0 + scd / nd) * M + d0 + scd % nd, fj * s);
        }
    }
    if (cl.want_k && kon) {
        const double fk = 2.0 * f;
        const int nac = na * nc, nad = na * nd, nbc = nb * nc, nbd = nb * nd;
        for (int e = tid; e < nac + nad + nbc + nbd; e += nt) {
            double s = 0.0;
            if (e < nac) {
                const int a = e / nc, c = e % nc;
                for (int b = 0; b < nb; ++b)
                    for (int d = 0; d < nd; ++d) s += V[(a * nb + b) * nscd + c * nd + d] * Pbd[b * nd + d];
                atomicAdd(Km + (long long)(a0 + a) * M + c0 + c, fk * s);
            } else if (e < nac + nad) {
                const int k = e - nac, a = k / nd, d = k % nd;
                for (int b = 0; b < nb; ++b)
                    for (int c = 0; c < nc; ++c) s += V[(a * nb + b) * nscd + c * nd + d] * Pbc[b * nc + c];
                atomicAdd(Km + (long long)(a0 + a) * M + d0 + d, fk * s);
            } else if (e < nac + nad + nbc) {
                const int k = e - nac - nad, b = k / nc, c = k % nc;
                for (int a = 0; a < na; ++a)
                    for (int d = 0; d < nd; ++d) s += V[(a * nb + b) * nscd + c * nd + d] * Pad[a * nd + d];
                atomicAdd(Km + (long long)(b0 + b) * M + c0 + c, fk * s);
            } else {
                const int k = e - nac - nad - nbc, b = k / nd, d = k % nd;
                for (int a = 0; a < na; ++a)
                    for (int c = 0; c < nc; ++c) s += V[(a * nb + b) * nscd + c * nd + d] * Pac[a * nc + c];
                atomicAdd(Km + (long long)(b0 + b) * M + d0 + d, fk * s);
            }
        }
    }
    __syncthreads();
}

}  // namespace dev
}  // namespace tlno_gpu
