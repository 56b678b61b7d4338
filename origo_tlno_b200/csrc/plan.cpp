// Plan construction: shell pairs (oriented higher-L left, as the reference's
// pair groups, rys_engine.ipp:2449-2468), their primitive-pair records
// (rys_engine.ipp:2244-2279), exact Schwarz bounds Q_ab = max sqrt((ab|ab))
// computed on the device by the ERI kernel itself (the reference computes
// the same diagonal blocks, rys_engine.ipp:16165-16258), screening
// Q_ab Q_cd >= tau at shell-pair level (native_quartets.ipp:556-574), and the
// quartet-class schedules.
//
// Schedule: the pairs of every class are sorted by Q descending, so for a
// block of consecutive bra pairs the surviving kets of any class form a
// prefix of that class's list; a block's tile count is
// ceil(prefix / tile_kets).  The kernels map a linear tile id back to its
// block by binary search in the tile prefix sums and re-test every quartet.
#include "plan.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <exception>
#include <functional>
#include <mutex>
#include <numeric>
#include <thread>

#include "kernels.hpp"

namespace tlno_gpu {

namespace {
// Simint's binary64 FASTSCHWARZ prefactor sqrt(2) pi^{5/2} (the literal the
// reference keeps, rys_engine.ipp:68-72).
constexpr double kFastSchwarzPrefactor = 24.739429451193148050228357586821944304008810699990039583;

// Schwarz bucket of a pair: floor(-log2 Q), so bucket k holds
// Q in (2^-(k+1), 2^-k]; larger Q first.
int Q_bucket(double q) {
    if (!(q > 0.0)) return 1 << 20;
    int e = 0;
    const double m = std::frexp(q, &e);  // q = m 2^e, m in [0.5, 1)
    return (m == 0.5) ? 1 - e : -e;      // q == 2^(e-1) belongs to bucket 1-e
}
}  // namespace

namespace {

template <class T>
void upload_vec(DeviceBuffer& buf, const std::vector<T>& v, cudaStream_t s) {
    buf.alloc(std::max<std::size_t>(v.size() * sizeof(T), 16));
    if (!v.empty())
        TLNO_CUDA(cudaMemcpyAsync(buf.ptr, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
}

void parallel_for(long long n, const std::function<void(long long, long long)>& f) {
    const int nt = static_cast<int>(std::max(1u, std::min(16u, std::thread::hardware_concurrency())));
    if (n < 4096 || nt == 1) {
        f(0, n);
        return;
    }
    std::vector<std::thread> ts;
    const long long chunk = (n + nt - 1) / nt;
    for (int t = 0; t < nt; ++t) {
        const long long b = t * chunk, e = std::min(n, b + chunk);
        if (b >= e) break;
        ts.emplace_back(f, b, e);
    }
    for (auto& t : ts) t.join();
}

// Runs f(t) on nt threads, t = 0 on this one; the first exception is rethrown
// here.  Work is to be shared by an index of f's own: fewer threads may start.
void run_threads(std::size_t nt, const std::function<void(std::size_t)>& f) {
    std::mutex mtx;
    std::exception_ptr failed;
    auto guarded = [&](std::size_t t) {
        try {
            f(t);
        } catch (...) {
            std::lock_guard<std::mutex> lock(mtx);
            if (!failed) failed = std::current_exception();
        }
    };
    std::vector<std::thread> threads;
    try {
        for (std::size_t t = 1; t < nt; ++t) threads.emplace_back(guarded, t);
    } catch (...) {
    }
    guarded(0);
    for (auto& t : threads) t.join();
    if (failed) std::rethrow_exception(failed);
}
std::size_t host_threads() { return std::max(1u, std::min(16u, std::thread::hardware_concurrency())); }

inline void oriented(const Basis& b, int i, int j, int& A, int& B) {
    A = i;
    B = j;
    if (b.shells[B].L > b.shells[A].L) std::swap(A, B);
}

// Algorithmic flop model per primitive quartet (native-route operation
// count): 30 + N [40 + 15 + 3 V_axis + 3 nc(a)nc(b)nc(c)nc(d)],
// V_axis = 5(LAB+1)(LCD+1) + 2 sum_{j=1..b}(LAB-j+1)(LCD+1)
//        + 2 sum_{l=1..d}(a+1)(b+1)(LCD-l+1).
double flops_per_prim(int a, int b, int c, int d) {
    const int LAB = a + b, LCD = c + d, N = (LAB + LCD) / 2 + 1;
    double vaxis = 5.0 * (LAB + 1) * (LCD + 1);
    for (int j = 1; j <= b; ++j) vaxis += 2.0 * (LAB - j + 1) * (LCD + 1);
    for (int l = 1; l <= d; ++l) vaxis += 2.0 * (a + 1) * (b + 1) * (LCD - l + 1);
    const double ncart4 = double(n_cart(a)) * n_cart(b) * n_cart(c) * n_cart(d);
    return 30.0 + N * (40.0 + 15.0 + 3.0 * vaxis + 3.0 * ncart4);
}
// Classes with a compile-time kernel of 4 register slices that the
// block-per-quartet kernel beats where the contraction is deep, that is where
// the primitive loop outweighs its barriers, block | compile-time: (dd|dp) 2.0 |
// 4.7 ms at 8.4 primitive quartets per quartet (f-shell 14 atoms), 0.41 | 0.33 at
// 1.8 (24-atom organic), 7.8 | 5.2 at 1.2 (91 waters); (fp|dp) 2.5 | 4.6 at 11.7.
// The projectors this needs (2-6 KB per pair) are affordable up to a million
// pairs, and only while the tables of the classes that have no other fast
// kernel fit beside them; the kernel's item index (primitive quartets x roots)
// has to fit 31 bits.
constexpr double kBlockKernelPrims = 4.0;
constexpr long long kBlockKernelPairs = 1000000;
bool block_kernel_class(int la, int lb, int lc, int ld) {
    return lc == 2 && ld == 1 && ((la == 2 && lb == 2) || (la == 3 && lb == 1));
}
// (dd|dd) has no compile-time kernel (8 slices of spilled registers): block |
// compile-time FP64 0.45 | 0.92 ms (f-shell 14 atoms), 0.083 | 0.086 (24-atom
// organic), 0.53 | 0.55 (91 waters), FP32 0.43 | 0.68, 0.083 | 0.063, 0.53 | 0.39.
bool block_only_class(int la, int lb, int lc, int ld) { return la == 2 && lb == 2 && lc == 2 && ld == 2; }

// Projector words of one pair (HRR + spherical map, eri_generic.cuh).
long long projector_words(int la, int lb) {
    const int nslice = (la + lb + 1) * (la + lb + 2) * (la + lb + 3) / 6 - la * (la + 1) * (la + 2) / 6;
    return static_cast<long long>(2 * la + 1) * (2 * lb + 1) * nslice;
}

// ---- tile shapes of the compile-time kernels ----
// Work of a tile beside its primitive loop (geometry, transfers, digestion), in
// primitive-quartet steps.
constexpr int kTileOverheadSteps = 8;

// Serial steps a tile may take.  The dynamic schedule hands the heaviest tiles
// out first, so a launch ends within one tile of the average load; a quarter of
// a resident warp group's share keeps that tail small, and below 8 steps the
// tile's own overhead outweighs a finer split.
double fast_tile_limit(double class_steps, int resident_groups) {
    return std::max(class_steps / (4.0 * std::max(resident_groups, 1)), double(kTileOverheadSteps));
}

// Bras per block and lanes per quartet (2^lk over the ket primitives, 2^lb over
// the bra primitives) that keep a tile inside `limit` steps: fewer bras per
// block first (that costs only shared sums), then lanes per quartet (that costs
// idle lanes in the digestion), never more lanes than primitives.
struct TileShape {
    int bras, lk, lb;
};
TileShape fast_tile_shape(int npb, int npk, int nbra, double limit) {
    TileShape t{nbra, 0, 0};
    const double per_bra = double(npb) * npk + kTileOverheadSteps;
    if (per_bra * nbra <= limit) return t;
    t.bras = std::max(1, static_cast<int>(limit / per_bra));
    if (t.bras > 1) return t;
    while (t.lk + t.lb < 5 && double(npb) * npk / (1 << (t.lk + t.lb)) > limit) {
        if ((2 << t.lk) <= npk) ++t.lk;
        else if ((2 << t.lb) <= npb) ++t.lb;
        else break;
    }
    return t;
}

// Reorders a schedule's blocks by falling cost (log2 of a tile's serial steps),
// the order inside a cost kept, and rebuilds the tile prefix.
void heaviest_first(std::vector<dev::BlockDesc>& blocks, std::vector<int>& prefix, const std::vector<int>& cost) {
    // counting sort over the at most 32 cost values
    std::array<std::size_t, 33> at{};
    for (int c : cost) ++at[31 - c + 1];
    for (std::size_t c = 1; c < at.size(); ++c) at[c] += at[c - 1];
    std::vector<int> order(blocks.size());
    for (std::size_t k = 0; k < blocks.size(); ++k) order[at[31 - cost[k]]++] = static_cast<int>(k);
    std::vector<dev::BlockDesc> b(blocks.size());
    std::vector<int> p(prefix.size(), 0);
    for (std::size_t k = 0; k < order.size(); ++k) {
        b[k] = blocks[order[k]];
        p[k + 1] = p[k] + prefix[order[k] + 1] - prefix[order[k]];
    }
    blocks.swap(b);
    prefix.swap(p);
}

// Per contracted quartet: 2 x projection terms + 12 per spherical ERI.
double flops_per_contracted(int a, int b, int c, int d) {
    const double ncart4 = double(n_cart(a)) * n_cart(b) * n_cart(c) * n_cart(d);
    const double nsph4 = double(n_sph(a)) * n_sph(b) * n_sph(c) * n_sph(d);
    return 2.0 * 2.0 * ncart4 + 12.0 * nsph4;
}

}  // namespace

int primitive_pair_count(const Basis& b, int A, int B) {
    const Shell& sa = b.shells[A];
    const Shell& sb = b.shells[B];
    int n = 0;
    for (int i = 0; i < sa.nprim; ++i)
        for (int j = 0; j < sb.nprim; ++j)
            if (b.c_radial[sa.prim_offset + i] * b.c_radial[sb.prim_offset + j] != 0.0) ++n;
    return n;
}

void primitive_pairs(const Basis& b, int A, int B, std::vector<dev::DPrimPair>& out) {
    const Shell& sa = b.shells[A];
    const Shell& sb = b.shells[B];
    const double* a = sa.center;
    const double* c = sb.center;
    const double ab[3] = {a[0] - c[0], a[1] - c[1], a[2] - c[2]};
    const double r2 = ab[0] * ab[0] + ab[1] * ab[1] + ab[2] * ab[2];
    for (int i = 0; i < sa.nprim; ++i) {
        const double al = b.exps[sa.prim_offset + i];
        const double ca = b.c_radial[sa.prim_offset + i];
        for (int j = 0; j < sb.nprim; ++j) {
            const double be = b.exps[sb.prim_offset + j];
            const double cab = ca * b.c_radial[sb.prim_offset + j];
            if (cab == 0.0) continue;
            const double p = al + be, invp = 1.0 / p;
            const double K = std::exp(-(al * be * invp) * r2);
            dev::DPrimPair pp;
            pp.p = p;
            pp.invp = invp;
            pp.Px = (al * a[0] + be * c[0]) * invp;
            pp.Py = (al * a[1] + be * c[1]) * invp;
            pp.Pz = (al * a[2] + be * c[2]) * invp;
            pp.w = K * cab * invp;
            out.push_back(pp);
        }
    }
}

// Decay scale of a shell (alpha_min, K = sum_i |c_i| (pi / alpha_i)^{3/4})
// and the pair indicator K_A K_B exp(-mu |AB|^2), mu from the two smallest
// exponents (rys_engine.ipp:2205-2241).
namespace {
struct DecayScale {
    double alpha_min = 0.0, K = 0.0;
};
DecayScale decay_scale(const Basis& b, int sh) {
    const Shell& s = b.shells[sh];
    DecayScale out;
    if (s.nprim == 0) return out;
    out.alpha_min = b.exps[s.prim_offset];
    for (int i = 0; i < s.nprim; ++i) {
        const double alpha = b.exps[s.prim_offset + i];
        out.alpha_min = std::min(out.alpha_min, alpha);
        out.K += std::fabs(b.c_radial[s.prim_offset + i]) * std::pow(kPi / alpha, 0.75);
    }
    return out;
}
double pair_decay_bound(const Basis& b, int A, int B, const DecayScale& a, const DecayScale& c) {
    if (!(a.alpha_min > 0.0) || !(c.alpha_min > 0.0)) return 0.0;
    const double dx = b.shells[A].center[0] - b.shells[B].center[0];
    const double dy = b.shells[A].center[1] - b.shells[B].center[1];
    const double dz = b.shells[A].center[2] - b.shells[B].center[2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double mu = a.alpha_min * c.alpha_min / (a.alpha_min + c.alpha_min);
    return a.K * c.K * std::exp(-mu * r2);
}
}  // namespace

MolPairs build_mol_pairs(const Basis& b, double tau, cudaStream_t s, double decay) {
    MolPairs mp;
    const int ns = static_cast<int>(b.shells.size());
    const long long npairs = static_cast<long long>(ns) * (ns + 1) / 2;
    mp.Q_canonical.assign(static_cast<std::size_t>(npairs), 0.0);
    if (ns == 0) return mp;
    const bool use_decay = decay > 0.0;
    if (use_decay) tau = decay;
    std::vector<DecayScale> dscale;
    if (use_decay)
        for (int i = 0; i < ns; ++i) dscale.push_back(decay_scale(b, i));

    // Device copy of the shells for the Schwarz kernel.
    std::vector<double> xyz(3 * ns);
    std::vector<int> Ls(ns), sph(ns);
    for (int i = 0; i < ns; ++i) {
        for (int k = 0; k < 3; ++k) xyz[3 * i + k] = b.shells[i].center[k];
        Ls[i] = b.shells[i].L;
        sph[i] = b.shells[i].sph_offset;
    }
    DeviceBuffer d_xyz, d_L, d_sph;
    upload_vec(d_xyz, xyz, s);
    upload_vec(d_L, Ls, s);
    upload_vec(d_sph, sph, s);

    // Chunked evaluation of the diagonal quartets (ab|ab).
    const long long chunk = 1 << 20;
    DeviceBuffer d_A, d_B, d_off, d_np, d_prim, d_list, d_Q;
    for (long long c0 = 0; c0 < npairs; c0 += chunk) {
        const long long c1 = std::min(npairs, c0 + chunk);
        const int n = static_cast<int>(c1 - c0);
        std::vector<int> A(n), B(n), np(n), off(n + 1, 0), cls(n);
        // canonical pair index t -> (i, j), i >= j
        long long i = static_cast<long long>((std::sqrt(8.0 * c0 + 1.0) - 1.0) / 2.0);
        while (i * (i + 1) / 2 > c0) --i;
        while ((i + 1) * (i + 2) / 2 <= c0) ++i;
        long long j = c0 - i * (i + 1) / 2;
        for (int t = 0; t < n; ++t) {
            int a, bb;
            oriented(b, static_cast<int>(i), static_cast<int>(j), a, bb);
            A[t] = a;
            B[t] = bb;
            np[t] = primitive_pair_count(b, a, bb);
            cls[t] = pair_class_of(b.shells[a].L, b.shells[bb].L);
            if (++j > i) { ++i; j = 0; }
        }
        for (int t = 0; t < n; ++t) off[t + 1] = off[t] + np[t];
        std::vector<dev::DPrimPair> prim(static_cast<std::size_t>(off[n]));
        parallel_for(n, [&](long long b0, long long e0) {
            std::vector<dev::DPrimPair> tmp;
            for (long long t = b0; t < e0; ++t) {
                tmp.clear();
                primitive_pairs(b, A[t], B[t], tmp);
                std::copy(tmp.begin(), tmp.end(), prim.begin() + off[t]);
            }
        });
        upload_vec(d_A, A, s);
        upload_vec(d_B, B, s);
        upload_vec(d_off, off, s);
        upload_vec(d_np, np, s);
        upload_vec(d_prim, prim, s);
        d_Q.alloc(sizeof(double) * n);
        dev::PlanView pv{};
        pv.shell_xyz = d_xyz.as<double>();
        pv.shell_L = d_L.as<int>();
        pv.shell_sph = d_sph.as<int>();
        pv.pair_A = d_A.as<int>();
        pv.pair_B = d_B.as<int>();
        pv.pair_prim_off = d_off.as<int>();
        pv.pair_nprim = d_np.as<int>();
        pv.prim = d_prim.as<dev::DPrimPair>();
        // one launch per pair class
        std::vector<std::vector<int>> by_cls(kMaxPairClasses);
        for (int t = 0; t < n; ++t) by_cls[cls[t]].push_back(t);
        std::vector<int> list;
        std::vector<int> list_off(kMaxPairClasses + 1, 0);
        for (int c = 0; c < kMaxPairClasses; ++c) {
            list_off[c + 1] = list_off[c] + static_cast<int>(by_cls[c].size());
            list.insert(list.end(), by_cls[c].begin(), by_cls[c].end());
        }
        upload_vec(d_list, list, s);
        for (int c = 0; c < kMaxPairClasses && !use_decay; ++c) {
            const int cnt = list_off[c + 1] - list_off[c];
            if (cnt == 0) continue;
            int la = 0;
            while ((la + 1) * (la + 2) / 2 <= c) ++la;
            const int lb = c - la * (la + 1) / 2;
            dev::ClassLaunch cl{};
            cl.la = la; cl.lb = lb; cl.lc = la; cl.ld = lb;
            cl.q_bra = d_list.as<int>() + list_off[c];
            cl.q_ket = cl.q_bra;
            cl.n_quartets = cnt;
            cl.out = d_Q.as<double>() + list_off[c];
            launch_eri_schwarz(pv, cl, s);
        }
        if (use_decay) {
            for (int t = 0; t < n; ++t) mp.Q_canonical[c0 + t] = pair_decay_bound(b, A[t], B[t], dscale[A[t]], dscale[B[t]]);
        } else {
            std::vector<double> qsorted(n);
            TLNO_CUDA(cudaMemcpyAsync(qsorted.data(), d_Q.ptr, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
            TLNO_CUDA(cudaStreamSynchronize(s));
            for (int pos = 0; pos < n; ++pos) mp.Q_canonical[c0 + list[pos]] = qsorted[pos];
        }
        // remember pair metadata in canonical order for the selection below
        for (int t = 0; t < n; ++t) {
            mp.A.push_back(A[t]);
            mp.B.push_back(B[t]);
            mp.nprim.push_back(np[t]);
            mp.cls.push_back(cls[t]);
        }
    }
    for (double q : mp.Q_canonical) mp.Qmax = std::max(mp.Qmax, q);
    // Keep pairs that can pass Q_ab * Q_cd >= tau for some cd; sort by
    // class then Q descending (ties by canonical index).
    std::vector<long long> keep;
    keep.reserve(static_cast<std::size_t>(npairs));
    for (long long t = 0; t < npairs; ++t) {
        if (tau > 0.0 && !(mp.Q_canonical[t] * mp.Qmax >= tau)) continue;
        keep.push_back(t);
    }
    // Inside a class, pairs are grouped by primitive count (a tile of kets
    // then runs one primitive loop length on every lane), then by Schwarz
    // bucket floor(-log2 Q) (the kets that can pass the bound for a bra form
    // a prefix of whole buckets), and inside a bucket by shell indices, so
    // that neighbouring lanes read and update neighbouring density and J/K
    // elements.
    auto bucket = [&](long long t) { return Q_bucket(mp.Q_canonical[t]); };
    std::stable_sort(keep.begin(), keep.end(), [&](long long l, long long r) {
        if (mp.cls[l] != mp.cls[r]) return mp.cls[l] < mp.cls[r];
        if (mp.nprim[l] != mp.nprim[r]) return mp.nprim[l] < mp.nprim[r];
        const int bl = bucket(l), br = bucket(r);
        if (bl != br) return bl < br;
        if (mp.A[l] != mp.A[r]) return mp.A[l] < mp.A[r];
        return mp.B[l] < mp.B[r];
    });
    MolPairs out;
    out.Q_canonical = std::move(mp.Q_canonical);
    out.Qmax = mp.Qmax;
    out.cls_begin.fill(0);
    out.cls_count.fill(0);
    for (std::size_t k = 0; k < keep.size(); ++k) {
        const long long t = keep[k];
        out.A.push_back(mp.A[t]);
        out.B.push_back(mp.B[t]);
        out.nprim.push_back(mp.nprim[t]);
        out.cls.push_back(mp.cls[t]);
        out.Q.push_back(out.Q_canonical[t]);
        out.cls_count[mp.cls[t]]++;
    }
    int acc = 0;
    for (int c = 0; c < kMaxPairClasses; ++c) {
        out.cls_begin[c] = acc;
        acc += out.cls_count[c];
    }
    return out;
}

dev::PlanView Plan2e::view() const {
    dev::PlanView pv{};
    pv.shell_xyz = d_shell_xyz.as<double>();
    pv.shell_L = d_shell_L.as<int>();
    pv.shell_sph = d_shell_sph.as<int>();
    pv.pair_A = d_pair_A.as<int>();
    pv.pair_B = d_pair_B.as<int>();
    pv.pair_prim_off = d_pair_prim_off.as<int>();
    pv.pair_nprim = d_pair_nprim.as<int>();
    pv.pair_Q = d_pair_Q.as<double>();
    pv.pair_rec = d_pair_rec.as<dev::PairRec>();
    pv.pair_mol = n_mol > 1 ? d_pair_mol.as<int>() : nullptr;
    pv.prim = d_prim.as<dev::DPrimPair>();
    pv.prim32 = d_prim32.as<dev::FPrimPair>();
    pv.mol_mat_off = n_mol > 1 ? d_mol_mat_off.as<long long>() : nullptr;
    pv.mol_M = n_mol > 1 ? d_mol_M.as<int>() : nullptr;
    pv.prim_fs = d_prim_fs.as<double>();
    pv.mol_shell_off = n_mol > 1 ? d_mol_shell_off.as<int>() : nullptr;
    pv.mol_ns = n_mol > 1 ? d_mol_ns.as<int>() : nullptr;
    pv.proj = proj_ready ? d_proj.as<double>() : nullptr;
    pv.proj_off = proj_ready ? d_proj_off.as<long long>() : nullptr;
    return pv;
}

void check_function_count(const Basis& b) {
    if (b.n_sph > 65535) throw Error(-1, "eri_ao_tensor_hgp: direct J/K pair tables assume M <= 65535.");
}

void build_plan(Plan2e& plan, const std::vector<const Basis*>& bases, std::vector<MolPairs>&& pairs,
                double tau, const Tuning& tune, cudaStream_t s) {
    for (const Basis* b : bases) check_function_count(*b);
    plan.tau = tau;
    plan.n_mol = static_cast<int>(bases.size());
    plan.mol_pairs = std::move(pairs);
    plan.mol_shell_off.assign(plan.n_mol + 1, 0);
    plan.mol_M.assign(plan.n_mol, 0);
    plan.mol_mat_off.assign(plan.n_mol + 1, 0);
    std::vector<double> xyz;
    std::vector<int> Ls, sph;
    for (int m = 0; m < plan.n_mol; ++m) {
        const Basis& b = *bases[m];
        plan.mol_shell_off[m + 1] = plan.mol_shell_off[m] + static_cast<int>(b.shells.size());
        plan.mol_M[m] = b.n_sph;
        plan.mol_mat_off[m + 1] = plan.mol_mat_off[m] + static_cast<long long>(b.n_sph) * b.n_sph;
        for (const Shell& sh : b.shells) {
            xyz.insert(xyz.end(), sh.center, sh.center + 3);
            Ls.push_back(sh.L);
            sph.push_back(sh.sph_offset);
        }
    }
    // Global sorted pair arrays: per molecule the class-sorted list; the
    // class lists of one molecule are contiguous.
    std::vector<std::array<int, kMaxPairClasses>> gbeg(plan.n_mol);
    plan.pair_A.clear(); plan.pair_B.clear(); plan.pair_nprim.clear();
    plan.pair_prim_off.clear(); plan.pair_Q.clear(); plan.pair_mol.clear();
    plan.total_pairs = 0;
    int prim_total = 0;
    for (int m = 0; m < plan.n_mol; ++m) {
        const MolPairs& mp = plan.mol_pairs[m];
        const int base = static_cast<int>(plan.pair_A.size());
        for (int c = 0; c < kMaxPairClasses; ++c) gbeg[m][c] = base + mp.cls_begin[c];
        const int so = plan.mol_shell_off[m];
        for (std::size_t k = 0; k < mp.A.size(); ++k) {
            plan.pair_A.push_back(mp.A[k] + so);
            plan.pair_B.push_back(mp.B[k] + so);
            plan.pair_nprim.push_back(mp.nprim[k]);
            plan.pair_prim_off.push_back(prim_total);
            prim_total += mp.nprim[k];
            plan.pair_Q.push_back(mp.Q[k]);
            plan.pair_mol.push_back(m);
        }
        const long long ns = bases[m]->shells.size();
        plan.total_pairs += ns * (ns + 1) / 2;
    }
    plan.kept_pairs = static_cast<long long>(plan.pair_A.size());
    std::vector<dev::DPrimPair> prim(static_cast<std::size_t>(prim_total));
    std::vector<dev::FPrimPair> prim32(static_cast<std::size_t>(prim_total));
    std::vector<double> prim_fs(static_cast<std::size_t>(prim_total));
    {
        const long long np = static_cast<long long>(plan.pair_A.size());
        parallel_for(np, [&](long long b0, long long e0) {
            std::vector<dev::DPrimPair> tmp;
            for (long long k = b0; k < e0; ++k) {
                const int m = plan.pair_mol[k];
                const int so = plan.mol_shell_off[m];
                tmp.clear();
                primitive_pairs(*bases[m], plan.pair_A[k] - so, plan.pair_B[k] - so, tmp);
                std::copy(tmp.begin(), tmp.end(), prim.begin() + plan.pair_prim_off[k]);
                const auto& ca = bases[m]->shells[plan.pair_A[k] - so].center;
                for (std::size_t t = 0; t < tmp.size(); ++t) {
                    const dev::DPrimPair& d = tmp[t];
                    // Simint's FASTSCHWARZ primitive-pair value, squared MEST
                    // estimate sqrt(2) pi^{5/2} p^{-5/2} e^{-2 mu R^2} (cA cB)^2
                    // (rys_engine.ipp:68-72, 2264-2268)
                    prim_fs[plan.pair_prim_off[k] + t] = kFastSchwarzPrefactor * d.w * d.w * std::sqrt(d.invp);
                    prim32[plan.pair_prim_off[k] + t] = {static_cast<float>(d.p), static_cast<float>(d.Px - ca[0]),
                                                         static_cast<float>(d.Py - ca[1]), static_cast<float>(d.Pz - ca[2]),
                                                         static_cast<float>(d.w), static_cast<float>(d.invp)};
                }
            }
        });
    }
    upload_vec(plan.d_shell_xyz, xyz, s);
    upload_vec(plan.d_shell_L, Ls, s);
    upload_vec(plan.d_shell_sph, sph, s);
    upload_vec(plan.d_pair_A, plan.pair_A, s);
    upload_vec(plan.d_pair_B, plan.pair_B, s);
    upload_vec(plan.d_pair_nprim, plan.pair_nprim, s);
    upload_vec(plan.d_pair_prim_off, plan.pair_prim_off, s);
    upload_vec(plan.d_pair_Q, plan.pair_Q, s);
    upload_vec(plan.d_pair_mol, plan.pair_mol, s);
    plan.d_pair_rec.alloc(sizeof(dev::PairRec) * std::max<std::size_t>(plan.pair_A.size(), 1));
    launch_pair_records(plan.view(), static_cast<int>(plan.pair_A.size()), plan.d_pair_rec.as<dev::PairRec>(), s);
    upload_vec(plan.d_prim, prim, s);
    upload_vec(plan.d_prim32, prim32, s);
    upload_vec(plan.d_mol_mat_off, plan.mol_mat_off, s);
    upload_vec(plan.d_mol_M, plan.mol_M, s);
    upload_vec(plan.d_prim_fs, prim_fs, s);
    plan.mol_ns.assign(plan.n_mol, 0);
    plan.rho_off.assign(plan.n_mol + 1, 0);
    plan.max_ns2 = 0;
    for (int m = 0; m < plan.n_mol; ++m) {
        plan.mol_ns[m] = plan.mol_shell_off[m + 1] - plan.mol_shell_off[m];
        const long long n2 = static_cast<long long>(plan.mol_ns[m]) * plan.mol_ns[m];
        plan.rho_off[m + 1] = plan.rho_off[m] + n2;
        plan.max_ns2 = std::max(plan.max_ns2, n2);
    }
    upload_vec(plan.d_mol_shell_off, plan.mol_shell_off, s);
    upload_vec(plan.d_mol_ns, plan.mol_ns, s);
    upload_vec(plan.d_rho_off, plan.rho_off, s);

    // Ket segments of every (molecule, pair class): runs of equal primitive
    // count, with Q sorted descending inside a segment (exact quartet counts)
    // and, per position, the largest Q of its bucket (non-increasing along the
    // segment) for the schedule extent.
    struct KetClass {
        std::vector<int> seg;
        std::vector<double> qsorted, bmax;
    };
    std::vector<KetClass> kets(static_cast<std::size_t>(plan.n_mol) * kMaxPairClasses);
    for (int m = 0; m < plan.n_mol; ++m)
        for (int Y = 0; Y < kMaxPairClasses; ++Y) {
            const int nY = plan.mol_pairs[m].cls_count[Y];
            if (nY == 0) continue;
            const int by0 = gbeg[m][Y];
            KetClass& kc = kets[static_cast<std::size_t>(m) * kMaxPairClasses + Y];
            kc.seg.push_back(0);
            for (int j = 1; j < nY; ++j)
                if (plan.pair_nprim[by0 + j] != plan.pair_nprim[by0 + j - 1]) kc.seg.push_back(j);
            kc.seg.push_back(nY);
            const double* qk = plan.pair_Q.data() + by0;
            kc.qsorted.assign(qk, qk + nY);
            kc.bmax.resize(nY);
            for (std::size_t sg = 0; sg + 1 < kc.seg.size(); ++sg) {
                const int s0 = kc.seg[sg], s1 = kc.seg[sg + 1];
                std::sort(kc.qsorted.begin() + s0, kc.qsorted.begin() + s1, std::greater<double>());
                for (int j = s0; j < s1;) {
                    int e = j;
                    double mx = 0.0;
                    const int bk = Q_bucket(qk[j]);
                    while (e < s1 && Q_bucket(qk[e]) == bk) mx = std::max(mx, qk[e++]);
                    for (int t = j; t < e; ++t) kc.bmax[t] = mx;
                    j = e;
                }
            }
        }

    // Quartet-class schedules.
    plan.combos.clear();
    plan.total_quartets = plan.total_prim_quartets = 0;
    plan.total_flops = 0.0;
    // Per pair class: kept pairs, mean and largest primitive count.
    struct ClassPrims {
        long long n = 0, sum = 0;
        int max = 0;
        double mean() const { return n > 0 ? double(sum) / n : 0.0; }
    };
    std::array<ClassPrims, kMaxPairClasses> prims{};
    for (int m = 0; m < plan.n_mol; ++m)
        for (int X = 0; X < kMaxPairClasses; ++X)
            for (int k = 0; k < plan.mol_pairs[m].cls_count[X]; ++k) {
                const int np = plan.pair_nprim[gbeg[m][X] + k];
                prims[X].n += 1;
                prims[X].sum += np;
                prims[X].max = std::max(prims[X].max, np);
            }
    // The class schedules are independent: built on host threads, uploaded in
    // class order.
    std::vector<ComboSchedule> todo;
    std::vector<int> resident;  // per class: warp groups on the device
    for (int X = 0; X < kMaxPairClasses; ++X)
        for (int Y = 0; Y <= X; ++Y) {
            bool any = false;
            for (int m = 0; m < plan.n_mol && !any; ++m)
                any = plan.mol_pairs[m].cls_count[X] > 0 && plan.mol_pairs[m].cls_count[Y] > 0;
            if (!any) continue;
            ComboSchedule cs;
            cs.X = X;
            cs.Y = Y;
            int la = 0;
            while ((la + 1) * (la + 2) / 2 <= X) ++la;
            int lc = 0;
            while ((lc + 1) * (lc + 2) / 2 <= Y) ++lc;
            cs.la = la; cs.lb = X - la * (la + 1) / 2;
            cs.lc = lc; cs.ld = Y - lc * (lc + 1) / 2;
            const int combo_id = X * kMaxPairClasses + Y;
            cs.fast = has_fast_kernel(cs.la, cs.lb, cs.lc, cs.ld) &&
                      !(combo_id < 256 && tune.force_generic[combo_id]);
            cs.block = block_only_class(cs.la, cs.lb, cs.lc, cs.ld);
            // the transfers of g shells cancel too much for FP32 ((gg|gg) of two
            // atoms: J off by 2.3e-3 of 3.3): FP64 in a mixed build
            if (cs.la == kMaxL) cs.mix_scale = 0.0;
            todo.push_back(std::move(cs));
        }
    // Projector tables: those of the classes without a compile-time kernel, the
    // smallest first while they fit, then those of the classes with a choice.
    std::array<bool, kMaxPairClasses> table{};
    {
        std::array<long long, kMaxPairClasses> bytes{};
        std::array<bool, kMaxPairClasses> wanted{};
        for (const ComboSchedule& cs : todo) {
            bytes[cs.X] = 8 * prims[cs.X].n * projector_words(cs.la, cs.lb);
            bytes[cs.Y] = 8 * prims[cs.Y].n * projector_words(cs.lc, cs.ld);
            if (!cs.fast) wanted[cs.X] = wanted[cs.Y] = true;
        }
        std::vector<int> order;
        for (int X = 0; X < kMaxPairClasses; ++X)
            if (wanted[X]) order.push_back(X);
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return bytes[a] < bytes[b]; });
        long long left = tune.max_projector_bytes;
        bool all = true;
        for (int X : order) {
            all = all && bytes[X] <= left;
            if (!all) break;
            left -= bytes[X];
            table[X] = true;
        }
        for (ComboSchedule& cs : todo) {
            if (!all || !cs.fast || !block_kernel_class(cs.la, cs.lb, cs.lc, cs.ld) || tune.generic_warps > 0) continue;
            const int nroots = (cs.la + cs.lb + cs.lc + cs.ld) / 2 + 1;
            const long long more = (table[cs.X] ? 0 : bytes[cs.X]) + (table[cs.Y] ? 0 : bytes[cs.Y]);
            if (prims[cs.X].mean() * prims[cs.Y].mean() < kBlockKernelPrims || plan.kept_pairs > kBlockKernelPairs ||
                double(prims[cs.X].max) * prims[cs.Y].max * nroots > 2147483647.0 || more > left)
                continue;
            left -= more;
            table[cs.X] = table[cs.Y] = true;
            cs.fast = false;
            cs.block = true;
        }
    }
    for (ComboSchedule& cs : todo) {
        cs.proj = !cs.fast && table[cs.X] && table[cs.Y];
        cs.bb = cs.fast ? fast_kernel_bras(cs.la, cs.lb, cs.lc, cs.ld) : 1;
        cs.bk = cs.fast ? 32 : tune.generic_bk;
        resident.push_back(cs.fast ? fast_kernel_resident_groups(cs.la, cs.lb, cs.lc, cs.ld) : 1);
    }
    auto build_schedule = [&](ComboSchedule& cs, int resident_groups) {
        const int X = cs.X, Y = cs.Y;
        const double fprim = flops_per_prim(cs.la, cs.lb, cs.lc, cs.ld);
        const double fcon = flops_per_contracted(cs.la, cs.lb, cs.lc, cs.ld);
        // Tile extent of segment [s0, s1) for a bra of bound qi: the whole
        // buckets that may hold a passing ket (on the diagonal class only
        // local index <= i).
        auto seg_extent = [&](const KetClass& kc, double qi, int s0, int s1, int i) {
            int lo = s1;
            if (tau > 0.0) {
                lo = s0;
                int hi = s1;
                while (lo < hi) {
                    const int mid = (lo + hi) / 2;
                    if (qi * kc.bmax[mid] >= tau) lo = mid + 1; else hi = mid;
                }
            }
            int e = lo - s0;
            if (X == Y) e = std::min(e, i + 1 - s0);
            return std::max(e, 0);
        };
        // Serial steps a tile may take (fast_tile_limit): from the steps of
        // the whole class with one lane per quartet, sampled over the bras.
        double limit = 1e300;
        if (cs.fast) {
            double steps = 0.0;
            for (int m = 0; m < plan.n_mol; ++m) {
                const int nX = plan.mol_pairs[m].cls_count[X];
                if (nX == 0 || plan.mol_pairs[m].cls_count[Y] == 0) continue;
                const KetClass& kc = kets[static_cast<std::size_t>(m) * kMaxPairClasses + Y];
                const int stride = std::max(1, nX / 1024);
                for (int i = 0; i < nX; i += stride)
                    for (std::size_t sg = 0; sg + 1 < kc.seg.size(); ++sg) {
                        const int ext = seg_extent(kc, plan.pair_Q[gbeg[m][X] + i], kc.seg[sg], kc.seg[sg + 1], i);
                        const int npk = plan.pair_nprim[gbeg[m][Y] + kc.seg[sg]];
                        steps += stride * double((ext + 31) / 32) *
                                 (double(plan.pair_nprim[gbeg[m][X] + i]) * npk + kTileOverheadSteps);
                    }
            }
            limit = fast_tile_limit(steps, resident_groups);
        }
        cs.prefix.push_back(0);
        std::vector<int> cost;  // per block: log2 of its tiles' serial steps
        for (int m = 0; m < plan.n_mol; ++m) {
            const MolPairs& mp = plan.mol_pairs[m];
            const int nX = mp.cls_count[X], nY = mp.cls_count[Y];
            if (nX == 0 || nY == 0) continue;
            const int bx0 = gbeg[m][X], by0 = gbeg[m][Y];
            const KetClass& kc = kets[static_cast<std::size_t>(m) * kMaxPairClasses + Y];
            const std::vector<int>& seg = kc.seg;
            // passing kets of segment [s0, s1) for a bra of bound qi
            auto seg_count = [&](double qi, int s0, int s1) {
                if (tau <= 0.0) return s1 - s0;
                int a = s0, b = s1;
                while (a < b) {
                    const int mid = (a + b) / 2;
                    if (qi * kc.qsorted[mid] >= tau) a = mid + 1; else b = mid;
                }
                return a - s0;
            };
            // Exact surviving quartets and primitive quartets.  Off the
            // diagonal every (bra, ket) pair counts; on the diagonal class
            // (one list, j <= i) a ket segment before the bra's segment
            // counts fully and the bra's own segment holds
            // (ordered pairs + self pairs) / 2.
            {
                std::vector<int> seg_of(nX);
                if (X == Y)
                    for (std::size_t sg = 0; sg + 1 < seg.size(); ++sg)
                        for (int j = seg[sg]; j < seg[sg + 1]; ++j) seg_of[j] = static_cast<int>(sg);
                std::vector<long long> own_ordered(seg.size(), 0), own_self(seg.size(), 0);
                for (int i = 0; i < nX; ++i) {
                    const double qi = plan.pair_Q[bx0 + i];
                    const long long npb = plan.pair_nprim[bx0 + i];
                    for (std::size_t sg = 0; sg + 1 < seg.size(); ++sg) {
                        if (X == Y && static_cast<int>(sg) > seg_of[i]) break;
                        const int c = seg_count(qi, seg[sg], seg[sg + 1]);
                        if (X == Y && static_cast<int>(sg) == seg_of[i]) {
                            own_ordered[sg] += c;
                            if (tau <= 0.0 || qi * qi >= tau) own_self[sg] += 1;
                            continue;
                        }
                        cs.quartets += c;
                        cs.prim_quartets += npb * plan.pair_nprim[by0 + seg[sg]] * c;
                    }
                }
                if (X == Y)
                    for (std::size_t sg = 0; sg + 1 < seg.size(); ++sg) {
                        const long long n = (own_ordered[sg] + own_self[sg]) / 2;
                        const long long np = plan.pair_nprim[by0 + seg[sg]];
                        cs.quartets += n;
                        cs.prim_quartets += np * np * n;
                    }
            }
            // Bra order: the class list order, or (bra groups) grouped by
            // first shell A inside each primitive-count group, list order
            // kept inside a group; a block holds up to cs.bb bras of one A,
            // fewer where their serial steps pass the limit.
            std::vector<int> order(nX);
            for (int i = 0; i < nX; ++i) order[i] = i;
            if (cs.bb > 1)
                std::stable_sort(order.begin(), order.end(), [&](int u, int v) {
                    const int nu = plan.pair_nprim[bx0 + u], nv = plan.pair_nprim[bx0 + v];
                    if (nu != nv) return nu < nv;
                    return plan.pair_A[bx0 + u] < plan.pair_A[bx0 + v];
                });
            for (int i0 = 0; i0 < nX;) {
                int nbra = 1, npb = plan.pair_nprim[bx0 + order[i0]];
                if (cs.bb > 1)
                    while (nbra < cs.bb && i0 + nbra < nX &&
                           plan.pair_A[bx0 + order[i0 + nbra]] == plan.pair_A[bx0 + order[i0]]) {
                        npb = std::max(npb, plan.pair_nprim[bx0 + order[i0 + nbra]]);
                        ++nbra;
                    }
                const int brabeg = static_cast<int>(cs.bra_list.size());
                bool used = false;
                for (std::size_t sg = 0; sg + 1 < seg.size(); ++sg) {
                    const int s0 = seg[sg], s1 = seg[sg + 1];
                    const int npk = plan.pair_nprim[by0 + s0];
                    const TileShape ts = cs.fast ? fast_tile_shape(npb, npk, nbra, limit) : TileShape{1, 0, 0};
                    const int bk = cs.bk >> (ts.lk + ts.lb);
                    for (int w0 = 0; w0 < nbra; w0 += ts.bras) {
                        const int w1 = std::min(nbra, w0 + ts.bras);
                        int ext = 0;
                        for (int w = w0; w < w1; ++w) {
                            const int i = order[i0 + w];
                            ext = std::max(ext, seg_extent(kc, plan.pair_Q[bx0 + i], s0, s1, i));
                        }
                        const int nt = (ext + bk - 1) / bk;
                        if (nt <= 0) continue;
                        used = true;
                        dev::BlockDesc bd{};
                        bd.bra0 = brabeg + w0;
                        bd.nbra = w1 - w0;
                        bd.ket0 = by0 + s0;
                        bd.nket = s1 - s0;
                        bd.xbeg = bx0;
                        bd.koff = s0;
                        bd.lk = ts.lk;
                        bd.lb = ts.lb;
                        cs.blocks.push_back(bd);
                        cs.prefix.push_back(cs.prefix.back() + nt);
                        // (a pair of 220-primitive shells passes 31 bits)
                        const long long tile_steps = (1LL * npb * npk * (w1 - w0)) >> (ts.lk + ts.lb);
                        int lg = 0;
                        while (lg < 31 && tile_steps >> (lg + 1)) ++lg;
                        cost.push_back(lg);
                    }
                }
                if (used)
                    for (int w = 0; w < nbra; ++w) cs.bra_list.push_back(bx0 + order[i0 + w]);
                i0 += nbra;
            }
        }
        cs.n_tiles = cs.prefix.back();
        if (cs.n_tiles == 0) return;
        heaviest_first(cs.blocks, cs.prefix, cost);
        cs.flops = fprim * cs.prim_quartets + fcon * cs.quartets;
    };
    {
        // one class at a time per thread; small plans are not worth a thread
        std::atomic<std::size_t> next{0};
        run_threads(plan.kept_pairs < 2000 ? 1 : std::min(host_threads(), todo.size()), [&](std::size_t) {
            for (std::size_t k; (k = next.fetch_add(1)) < todo.size();) build_schedule(todo[k], resident[k]);
        });
    }
    for (ComboSchedule& cs : todo) {
        if (cs.n_tiles == 0) continue;
        upload_vec(cs.d_blocks, cs.blocks, s);
        upload_vec(cs.d_prefix, cs.prefix, s);
        upload_vec(cs.d_bra_list, cs.bra_list, s);
        plan.total_quartets += cs.quartets;
        plan.total_prim_quartets += cs.prim_quartets;
        plan.total_flops += cs.flops;
        plan.combos.push_back(std::move(cs));
    }
    plan.d_counters.alloc(sizeof(int) * 2 * std::max<std::size_t>(plan.combos.size(), 1));

    // HRR + spherical projectors of the pairs of the classes that a
    // block-per-quartet combination uses, built once on the device.
    {
        std::array<bool, kMaxPairClasses> need{};
        for (const ComboSchedule& cs : plan.combos)
            if (cs.proj) need[cs.X] = need[cs.Y] = true;
        const std::size_t np = plan.pair_A.size();
        plan.proj_off.assign(np, -1);
        long long words = 0;
        for (std::size_t k = 0; k < np; ++k) {
            const int la = Ls[plan.pair_A[k]], lb = Ls[plan.pair_B[k]];
            if (!need[la * (la + 1) / 2 + lb]) continue;
            plan.proj_off[k] = words;
            words += projector_words(la, lb);
        }
        plan.proj_words = words;
        plan.proj_ready = false;
        if (words > 0) {
            try {
                plan.d_proj.alloc(sizeof(double) * words);
            } catch (const Error&) {
                // no room on the device: the classes run warp per quartet
                cudaGetLastError();
                for (ComboSchedule& cs : plan.combos) cs.proj = false;
                words = 0;
            }
        }
        if (words > 0) {
            upload_vec(plan.d_proj_off, plan.proj_off, s);
            launch_pair_projectors(plan.d_pair_A.as<int>(), plan.d_pair_B.as<int>(), plan.d_shell_xyz.as<double>(),
                                   plan.d_shell_L.as<int>(), plan.d_proj_off.as<long long>(), static_cast<int>(np),
                                   plan.d_proj.as<double>(), s);
            plan.proj_ready = true;
        }
    }
    TLNO_CUDA(cudaStreamSynchronize(s));
}

void ensure_density_tables(Plan2e& plan) {
    plan.d_rho_blk.alloc(sizeof(double) * std::max<long long>(plan.rho_off.empty() ? 1 : plan.rho_off.back(), 1));
    plan.d_rho_max.alloc(sizeof(double) * std::max(plan.n_mol, 1));
}

void build_onee_plan(OneePlan& p, const Basis& b, double decay_eps, double nuclear_eps) {
    const int ns = static_cast<int>(b.shells.size());
    p.pairs.clear();
    // Group decay scales from the representative shell of each group:
    // alpha_min and K = sum_i |c_i| (pi / alpha_i)^{3/4} with the normalised
    // coefficient of the group's first Cartesian component (x^L).
    const int ng = static_cast<int>(b.onee_group_rep.size());
    std::vector<double> amin(ng, 1e300), Kd(ng, 0.0);
    auto c_first = [&](const Shell& s, int i) {
        double df = 1.0;
        for (int k = 2 * s.L - 1; k > 0; k -= 2) df *= k;
        return b.c_radial[s.prim_offset + i] / std::sqrt(df);
    };
    for (int g = 0; g < ng; ++g) {
        const Shell& s = b.shells[b.onee_group_rep[g]];
        for (int i = 0; i < s.nprim; ++i) {
            const double a = b.exps[s.prim_offset + i];
            amin[g] = std::min(amin[g], a);
            Kd[g] += std::fabs(c_first(s, i)) * std::pow(kPi / a, 0.75);
        }
    }
    // Per-primitive max |normalised coefficient| over the group's components.
    p.maxc.assign(b.exps.size(), 0.0);
    std::vector<std::vector<double>> gmax(ng);
    for (int si = 0; si < ns; ++si) {
        const Shell& s = b.shells[si];
        const int g = b.onee_group[si];
        gmax[g].resize(s.nprim, 0.0);
        double maxang = 0.0;
        for (int x = s.L; x >= 0; --x)
            for (int y = s.L - x; y >= 0; --y) {
                const int z = s.L - x - y;
                double df = 1.0;
                for (int k = 2 * x - 1; k > 0; k -= 2) df *= k;
                for (int k = 2 * y - 1; k > 0; k -= 2) df *= k;
                for (int k = 2 * z - 1; k > 0; k -= 2) df *= k;
                maxang = std::max(maxang, 1.0 / std::sqrt(df));
            }
        for (int i = 0; i < s.nprim; ++i)
            gmax[g][i] = std::max(gmax[g][i], std::fabs(b.c_radial[s.prim_offset + i]) * maxang);
    }
    for (int si = 0; si < ns; ++si) {
        const Shell& s = b.shells[si];
        for (int i = 0; i < s.nprim; ++i) p.maxc[s.prim_offset + i] = gmax[b.onee_group[si]][i];
    }
    // Pair list, rows of shells dealt to host threads in blocks and joined in
    // order.
    constexpr int kRows = 16;
    std::vector<std::vector<dev::OneePair>> part((ns + kRows - 1) / kRows);
    auto rows = [&](int i0, std::vector<dev::OneePair>& out) {
        for (int i = i0; i < std::min(ns, i0 + kRows); ++i) {
            for (int j = 0; j <= i; ++j) {
                const int gi = b.onee_group[i], gj = b.onee_group[j];
                const Shell& si_ = b.shells[i];
                const Shell& sj_ = b.shells[j];
                const double dx = si_.center[0] - sj_.center[0], dy = si_.center[1] - sj_.center[1],
                             dz = si_.center[2] - sj_.center[2];
                const double r2 = dx * dx + dy * dy + dz * dz;
                bool keep = true;
                double bound = 0.0;
                if (decay_eps > 0.0) {
                    const double mu = amin[gi] * amin[gj] / (amin[gi] + amin[gj]);
                    if (Kd[gi] * Kd[gj] * std::exp(-mu * r2) < decay_eps) keep = false;
                    if (keep) {
                        const Shell& ri = b.shells[b.onee_group_rep[gi]];
                        const Shell& rj = b.shells[b.onee_group_rep[gj]];
                        for (int a = 0; a < ri.nprim; ++a)
                            for (int c = 0; c < rj.nprim; ++c) {
                                const double ea = b.exps[ri.prim_offset + a], ec = b.exps[rj.prim_offset + c];
                                const double pp = ea + ec, chi = ea * ec / pp;
                                bound += std::fabs(c_first(ri, a) * c_first(rj, c)) * std::pow(kPi / pp, 1.5) *
                                         std::exp(-chi * r2);
                            }
                    }
                }
                if (!keep) continue;
                dev::OneePair op{};
                op.A = i;
                op.B = j;
                if (b.shells[j].L > b.shells[i].L) std::swap(op.A, op.B);
                op.do_st = 1;
                op.do_v = (decay_eps <= 0.0 || bound >= decay_eps) ? 1 : 0;
                out.push_back(op);
            }
        }
    };
    {
        // the long rows first
        std::atomic<std::size_t> next{0};
        run_threads(ns < 64 ? 1 : std::min(host_threads(), part.size()), [&](std::size_t) {
            for (std::size_t k; (k = next.fetch_add(1)) < part.size();) {
                const std::size_t r = part.size() - 1 - k;
                rows(static_cast<int>(r) * kRows, part[r]);
            }
        });
    }
    for (const auto& v : part) p.pairs.insert(p.pairs.end(), v.begin(), v.end());
    p.nuc.clear();
    double zsum = 0.0;
    for (std::size_t a = 0; a < b.Z.size(); ++a) {
        zsum += std::fabs(static_cast<double>(b.Z[a]));
        if (b.Z[a] == 0) continue;
        p.nuc.push_back(b.atom_xyz[3 * a]);
        p.nuc.push_back(b.atom_xyz[3 * a + 1]);
        p.nuc.push_back(b.atom_xyz[3 * a + 2]);
        p.nuc.push_back(static_cast<double>(b.Z[a]));
    }
    p.screen_thr = (zsum > 0.0) ? nuclear_eps / zsum : 0.0;
}

}  // namespace tlno_gpu
