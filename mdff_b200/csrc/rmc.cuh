// Reverse Monte Carlo on the pair distribution (rmc_main, src/rmc.f90:196-640,
// with g(r) from gr_main, src/radial_distrib.f90) on the device.
//
// g(r): every ordered pair (ia, ja != ia) within cutgr adds to bin
// INT(r / resg) of the all-pairs row and of the ordered type row (ita, jta),
// r from the minimum-image fractional difference in the reference's order of
// operations; rmc_gr (src/rmc.f90:1431-1497) normalises row (it1 <= it2) by
// 4 pi (res r^2 + res^3 / 12) / V x natmi(it1) natmi(it2) (natm^2 for row 0).
//
// The Markov chain runs in one persistent CTA: a trial move changes only the
// N - 1 pairs of the moved atom, so the counts are updated from those pairs
// (old bin out, new bin in) -- exactly the integers a full recount gives --
// then chi^2, the reference's per-component Metropolis tests and the accept /
// reject all stay on the device.  Random numbers come from a stream in device
// memory (the caller's, or a counter-based generator's), consumed in the
// reference's order: particle, three displacement components, then one for
// each chi^2 component whose change is not negative.
#pragma once
#include "common.cuh"

namespace mdff {

constexpr int RMC_THREADS = 512;
constexpr int RMC_TREE = 1024;            // chi^2's fixed tree: 1024 leaves, 32 groups of 32
constexpr int RMC_VT = RMC_TREE / RMC_THREADS;   // leaves per thread
constexpr int RMC_UBUF = 1024;            // uniforms staged in shared memory
constexpr int RMC_MAX_BINS = 4096;
constexpr int RMC_NT_MAX = 4;
constexpr int RMC_SMEM_INTS = RMC_MAX_BINS * 4;   // delta counts, (1 + nt^2) rows of nbins

// the binning of one pair distance
struct RmcBin {
    double cut2, resg;
    int nbins, ntype;
};

struct RmcConst {
    int n, ntype, nbins, nrow;   // nrow = 1 + ntype^2 count rows (row 0 all pairs, 1 + ita*ntype + jta)
    int npairs;                  // ntype (ntype + 1) / 2
    RmcBin bin;
    double dmax[3];              // max_displacement / ANORM(d): the fractional displacement bound
    double temp[6];              // temp_rmc(1..5) and the total's
    double natm, natmi[RMC_NT_MAX];
    double volnorm[RMC_MAX_BINS];   // 4 pi (res rr^2 + res^3/12) / V per bin, in the reference's order
};

// bin of the pair (s_i, s_j) as gr_main forms it, or -1 beyond cutgr
__device__ __forceinline__ int rmc_bin(const CellP& c, const RmcBin& k, double s1, double s2, double s3, double t1,
                                       double t2, double t3) {
    double rx, ry, rz;
    const double rsq = pairvec_exact(c, s1, s2, s3, t1, t2, t3, rx, ry, rz);
    if (!(rsq < k.cut2)) return -1;
    const int b = (int)__ddiv_rn(__dsqrt_rn(rsq), k.resg);
    return b < k.nbins ? b : -1;
}

// The same bin for a pair from a neighbour list (FAST: the two images of a pair
// at half the cell are both beyond the list), without the reference's rounding
// steps, square root and division in FP64: r^2 to 1e-15, then r / resg in FP32
// (relative error below 3e-7), which decides the bin except within 1e-6 of its
// edges; those, and r^2 within 1e-9 of the cutoff, take the exact expression.
template <bool FAST>
__device__ __forceinline__ int rmc_bin_of(const CellP& c, const RmcBin& k, float inv_res, double s1, double s2,
                                          double s3, double t1, double t2, double t3) {
    if (FAST) {
        double d0 = s1 - t1, d1 = s2 - t2, d2 = s3 - t3;
        d0 -= (d0 + 6755399441055744.0) - 6755399441055744.0;   // d - rint(d)
        d1 -= (d1 + 6755399441055744.0) - 6755399441055744.0;
        d2 -= (d2 + 6755399441055744.0) - 6755399441055744.0;
        const double rx = fma(d2, c.A[2], fma(d1, c.A[1], d0 * c.A[0]));
        const double ry = fma(d2, c.A[5], fma(d1, c.A[4], d0 * c.A[3]));
        const double rz = fma(d2, c.A[8], fma(d1, c.A[7], d0 * c.A[6]));
        const double rsq = fma(rz, rz, fma(ry, ry, rx * rx));
        if (rsq > 1.000000001 * k.cut2) return -1;
        const float q = sqrtf((float)rsq) * inv_res;
        const int b = (int)q;
        const float f = q - (float)b, tol = fmaf(1e-6f, q, 1e-6f);
        if (rsq < 0.999999999 * k.cut2 && f > tol && f < 1.0f - tol) return b < k.nbins ? b : -1;
    }
    return rmc_bin(c, k, s1, s2, s3, t1, t2, t3);
}

// gr_main over all ordered pairs: a warp per atom ia over its neighbour row
// (LIST) or all atoms; counts in shared memory where the ntype^2 type rows fit
// (in_smem), then global integer atomics (order-free).  Row 0 is their sum.
template <bool LIST>
__global__ void __launch_bounds__(256) k_gr_rows(int n, const double* __restrict__ s, const int* __restrict__ type,
                                                 CellP c, RmcBin k, const int* __restrict__ nbr,
                                                 const int* __restrict__ cnt, int cap, int in_smem, int* hist) {
    extern __shared__ int sh[];
    const int nr = k.ntype * k.ntype * k.nbins;
    if (in_smem) {
        for (int q = threadIdx.x; q < nr; q += blockDim.x) sh[q] = 0;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const float inv_res = (float)(1.0 / k.resg);
    for (int ia = blockIdx.x * 8 + (threadIdx.x >> 5); ia < n; ia += gridDim.x * 8) {
        const double s1 = s[ia], s2 = s[(size_t)n + ia], s3 = s[2 * (size_t)n + ia];
        const int row = type[ia] * k.ntype;
        const int m = LIST ? cnt[ia] : n;
        for (int q = lane; q < m; q += 32) {
            const int ja = LIST ? nbr[(size_t)ia * cap + q] : q;
            if (!LIST && ja == ia) continue;
            const int b = rmc_bin_of<LIST>(c, k, inv_res, s1, s2, s3, s[ja], s[(size_t)n + ja], s[2 * (size_t)n + ja]);
            if (b < 0) continue;
            const int r = (row + type[ja]) * k.nbins + b;
            if (in_smem) {
                atomicAdd(&sh[r], 1);
            } else {
                atomicAdd(&hist[b], 1);
                atomicAdd(&hist[k.nbins + r], 1);
            }
        }
    }
    if (!in_smem) return;
    __syncthreads();
    for (int q = threadIdx.x; q < nr; q += blockDim.x)
        if (sh[q]) {
            atomicAdd(&hist[q % k.nbins], sh[q]);
            atomicAdd(&hist[k.nbins + q], sh[q]);
        }
}

// Chain state carried across launches (a launch ends when the neighbour
// list must be rebuilt).
struct RmcOut {
    long long kall, kacc, used;   // trial moves, accepted count (starting at 1 as the reference), uniforms consumed
    double chisq[6];              // of the last accepted configuration
    double maxd;                  // largest displacement of an atom since the list was built (A)
    int status;                   // 0 done, 1 the random stream ran out, 2 the list needs rebuilding
    int started;                  // chi^2 of the start evaluated
};

// Lists of the chain in a cell narrower than twice its reach: for each atom
// every other atom.
__global__ void k_rmc_all(int n, int cap, int* nbr, int* cnt) {
    const int i = blockIdx.x;
    for (int q = threadIdx.x; q < n - 1; q += blockDim.x) nbr[(size_t)i * cap + q] = q < i ? q : q + 1;
    if (threadIdx.x == 0) cnt[i] = n - 1;
}

// a / b correctly rounded, given y = the correctly rounded 1 / b: a step with the
// exact residual brings the quotient within one unit in the last place, and a
// second one rounds it correctly (Markstein, IBM J. Res. Dev. 34, 1990).  Not
// for a divisor near the ends of the range.
__device__ __forceinline__ double div_by(double a, double b, double y) {
    double q = __dmul_rn(a, y);
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
}

// The chain: until kacc reaches acc_max or kall reaches max_trials.  s: the
// fractional coordinates [3][n] (updated); ghist: counts [nrow][nbins]
// (updated); gexp [npairs+1][nbins]; uni: nuni uniforms in [0, 1).  In shared
// memory: the change of the counts of row 0 and the rows it1 <= it2 (the
// mirrored rows have the same counts), and, with in_smem, the counts.
//
// Bound: the latency of one trial, which the next one depends on.  Every warp
// draws the particle, forms its move and takes the Metropolis decision itself,
// so a trial has three barriers (the changed counts, the group sums of chi^2,
// the update).  The next trial starts 8 or 10 uniforms on: what it needs of
// both possible particles (position, neighbour row) is read while this one is
// decided.  32 440 ions, cut 10 A, 201 bins: 3.3 us a trial (5.0 with one thread
// drawing and deciding, the counts in global memory and six atomics per pair
// change instead of four).  512 threads: 1024 leave 64 registers each and spill.
template <bool FAST>
__global__ void __launch_bounds__(RMC_THREADS) k_rmc_chain(double* s, const int* __restrict__ type, CellP c,
                                                          const RmcConst* __restrict__ kp, int* ghist,
                                                          const double* __restrict__ gexp,
                                                          const double* __restrict__ uni, long long nuni,
                                                          long long acc_max, long long max_trials,
                                                          const int* __restrict__ nbr, const int* __restrict__ ncnt,
                                                          int cap, const double* __restrict__ sb, double dlim,
                                                          int in_smem, RmcOut* out) {
    extern __shared__ int dcnt[];
    __shared__ double wsum[RMC_TREE / 32];
    __shared__ double sh_maxd;
    __shared__ double ubuf[RMC_UBUF];
    const RmcConst& k = *kp;
    const RmcBin kb = k.bin;
    const float inv_res = (float)(1.0 / kb.resg);
    const int n = k.n, tid = threadIdx.x, np1 = k.npairs + 1, nt = kb.ntype, nbins = kb.nbins;
    const int nterm = np1 * nbins;
    const int lane = tid & 31, warp = tid >> 5;
    // row it1 <= it2 -> its place among them, 0 .. npairs - 1
    auto tri = [&](int t1, int t2) {
        const int lo = min(t1, t2), hi = max(t1, t2);
        return lo * nt - lo * (lo - 1) / 2 + hi - lo;
    };
    // counts: row 0, then the rows it1 <= it2, in shared memory; or ghist's rows
    int* hist = in_smem ? dcnt + nterm : ghist;
    auto row_of = [&](int mp) {   // ghist's row of mp = 0 (all pairs), 1 + tri
        if (mp == 0) return 0;
        int m = mp - 1, it1 = 0;
        while (m >= nt - it1) { m -= nt - it1; ++it1; }
        return 1 + it1 * nt + it1 + m;
    };
    for (int q = tid; q < nterm; q += RMC_THREADS) {
        dcnt[q] = 0;
        if (in_smem) hist[q] = ghist[row_of(q / nbins) * nbins + q % nbins];
    }
    // chi^2 (eval_chisq_rmc, src/rmc.f90:667-690) of the terms q = bin x
    // (npairs + 1) + mp by a fixed tree: leaf t sums terms t, t + 1024, ...
    // in order, then a shuffle-down tree within each 32 leaves and the same tree
    // over the 32 group sums (the oracle restates this order)
    struct Term { int at, hat; double den, inv, ge; };   // change, count, normalisation and its reciprocal, experimental value
    auto term_of = [&](int q) {
        Term t;
        const int b = q / np1, mp = q - b * np1;
        int it1 = 0, it2 = 0;
        if (mp > 0) {
            int m = mp - 1;
            while (m >= nt - it1) { m -= nt - it1; ++it1; }
            it2 = it1 + m;
        }
        t.at = mp * nbins + b;
        t.hat = (in_smem ? mp : row_of(mp)) * nbins + b;
        // vol * natm * natm and vol * natmi(it1) * natmi(it2), left to right
        t.den = mp == 0 ? __dmul_rn(__dmul_rn(k.volnorm[b], k.natm), k.natm)
                        : __dmul_rn(__dmul_rn(k.volnorm[b], k.natmi[it1]), k.natmi[it2]);
        t.inv = t.den > 1e-200 && t.den < 1e200 ? __drcp_rn(t.den) : 0.0;   // 0: divide
        t.ge = gexp[(size_t)mp * nbins + b];
        return t;
    };
    Term mine[RMC_VT];
#pragma unroll
    for (int t = 0; t < RMC_VT; ++t) mine[t] = term_of(min(tid + t * RMC_THREADS, nterm - 1));
    auto square = [&](const Term& t, double v) {
        const double cnt = (double)(hist[t.hat] + dcnt[t.at]);
        const double g = t.inv != 0.0 ? div_by(cnt, t.den, t.inv) : __ddiv_rn(cnt, t.den);
        const double dv = __dsub_rn(g, t.ge);
        return __dadd_rn(v, __dmul_rn(dv, dv));
    };
    auto chisq = [&]() -> double {   // the same value in every thread; one barrier
        double v[RMC_VT];
#pragma unroll
        for (int t = 0; t < RMC_VT; ++t) {
            v[t] = 0.0;
            if (tid + t * RMC_THREADS < nterm) v[t] = square(mine[t], v[t]);
            for (int q = tid + t * RMC_THREADS + RMC_TREE; q < nterm; q += RMC_TREE) v[t] = square(term_of(q), v[t]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int t = 0; t < RMC_VT; ++t) v[t] = __dadd_rn(v[t], __shfl_down_sync(0xffffffffu, v[t], o));
        if (lane == 0)
#pragma unroll
            for (int t = 0; t < RMC_VT; ++t) wsum[warp + t * (RMC_THREADS / 32)] = v[t];
        __syncthreads();
        double t = wsum[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t = __dadd_rn(t, __shfl_down_sync(0xffffffffu, t, o));
        return __shfl_sync(0xffffffffu, t, 0);
    };
    const int started = out->started;
    __syncthreads();
    // the g(r) components: 0 and the total (5); the others stay 0
    double chi0 = started ? out->chisq[0] : 0.0, chi5 = started ? out->chisq[5] : 0.0;
    if (!started) chi0 = chi5 = chisq();
    long long u_at = started ? out->used : 0;
    double maxd2 = 0.0;   // thread 0
    if (tid == 0) {
        sh_maxd = started ? out->maxd : 0.0;
        maxd2 = sh_maxd * sh_maxd;
    }
    int stop = 0;
    long long kall = started ? out->kall : 1, kacc = started ? out->kacc : 1;
    long long ubase = u_at;   // ubuf holds the uniforms from ubase on
    auto fill = [&]() {
        for (int q = tid; q < RMC_UBUF; q += RMC_THREADS) ubuf[q] = ubase + q < nuni ? uni[ubase + q] : 0.0;
    };
    fill();
    __syncthreads();
    // what a trial needs of its particle, read ahead for two candidates: lane d of
    // a warp the component d % 3 of its position, the thread's first neighbours
    const int dl = lane % 3;
    struct Ahead { int i, ti, nn, j[RMC_VT]; double ol; };
    auto ahead = [&](int at) {   // at: place of the trial's first uniform in ubuf
        Ahead A;
        const int i = (int)(ubuf[at] * n);
        A.i = i < n ? i : n - 1;
        A.ti = type[A.i];
        A.nn = ncnt[A.i];
        A.ol = s[(size_t)dl * n + A.i];
#pragma unroll
        for (int t = 0; t < RMC_VT; ++t) {
            const int q = tid + t * RMC_THREADS;
            A.j[t] = q < cap ? nbr[(size_t)A.i * cap + q] : 0;   // (past the row's end: not used)
        }
        return A;
    };
    Ahead cur = ahead(0), nx8, nx10;
    const double temp5 = k.temp[5], dmaxl = k.dmax[dl];
    while (kacc < acc_max && kall < max_trials) {
        if (sh_maxd > dlim) { stop = 2; break; }   // an atom moved too far for the list: rebuild first
        ++kall;
        if (u_at + 4 > nuni) { stop = 1; break; }
        const int ub = (int)(u_at - ubase);
        // rmc_move (src/rmc.f90:1366-1428): the displacement, a component per lane
        const double displ = __dmul_rn(dmaxl, __dsub_rn(__dmul_rn(2.0, ubuf[ub + 1 + dl]), 1.0));
        const double um0 = ubuf[ub + 8], um1 = ubuf[ub + 9];   // the decision's uniform, after 4 or 5 others
        double vl = __dadd_rn(cur.ol, displ);
        if (vl > 1.0 || vl < 0.0) vl = __dsub_rn(vl, round(vl));
        double o[3], snew[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            o[d] = __shfl_sync(0xffffffffu, cur.ol, d);
            snew[d] = __shfl_sync(0xffffffffu, vl, d);
        }
        const double bl = sb[(size_t)dl * n + cur.i];   // the list's position
        auto neighbour = [&](double t1, double t2, double t3, int tj) {
            const int bo = rmc_bin_of<FAST>(c, kb, inv_res, o[0], o[1], o[2], t1, t2, t3);
            const int bn = rmc_bin_of<FAST>(c, kb, inv_res, snew[0], snew[1], snew[2], t1, t2, t3);
            if (bo == bn) return;
            // the pair appears as (i, j) and (j, i): twice in row 0 and in a like-type
            // row, once in each of the two rows of unlike types
            int* d = dcnt + (1 + tri(cur.ti, tj)) * nbins;
            const int w = cur.ti == tj ? 2 : 1;
            if (bo >= 0) { atomicSub(&dcnt[bo], 2); atomicSub(&d[bo], w); }
            if (bn >= 0) { atomicAdd(&dcnt[bn], 2); atomicAdd(&d[bn], w); }
        };
        double r[RMC_VT][3];
        int tj[RMC_VT];
#pragma unroll
        for (int t = 0; t < RMC_VT; ++t) {   // every load before the first bin
            const int j = tid + t * RMC_THREADS < cur.nn ? cur.j[t] : 0;
            tj[t] = type[j];
#pragma unroll
            for (int d = 0; d < 3; ++d) r[t][d] = s[(size_t)d * n + j];
        }
#pragma unroll
        for (int t = 0; t < RMC_VT; ++t)
            if (tid + t * RMC_THREADS < cur.nn) neighbour(r[t][0], r[t][1], r[t][2], tj[t]);
        for (int q = tid + RMC_TREE; q < cur.nn; q += RMC_THREADS) {
            const int j = nbr[(size_t)cur.i * cap + q];
            neighbour(s[j], s[(size_t)n + j], s[2 * (size_t)n + j], type[j]);
        }
        nx8 = ahead(ub + 8);
        nx10 = ahead(ub + 10);
        __syncthreads();
        const double c1 = chisq();
        // Metropolis per component (src/rmc.f90:521-540): each whose change is not
        // negative takes a uniform (0, then 1 to 4, whose change is 0, then the
        // total, which decides)
        bool acc = true;
        const bool up0 = !(__dsub_rn(c1, chi0) < 0.0);
        const double dq = __dsub_rn(c1, chi5);
        const bool up5 = !(dq < 0.0);
        const int used = 8 + (up0 ? 1 : 0) + (up5 ? 1 : 0);
        if (u_at + used > nuni) {
            stop = 1;
            u_at = nuni;
        } else {
            if (up5) {   // exp(x) >= u, in FP32 where that decides it
                const double x = -__dmul_rn(dq, 0.5) / temp5, u = up0 ? um1 : um0;
                const float e = __expf((float)x), uf = (float)u;
                if (x > -80.0 && fabsf(e - uf) > (1e-5f + 1e-6f * fabsf((float)x)) * e + 1e-6f * uf + 1e-30f) acc = e > uf;
                else acc = exp(x) >= u;
            }
            u_at += used;
        }
        if (stop) { --kall; break; }
        // the rejected atom goes back by the displacement (src/rmc.f90:628-636)
        const double fl = acc ? vl : __dsub_rn(vl, displ);
        if (tid < 3) s[(size_t)tid * n + cur.i] = fl;
        double f[3], b[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            f[d] = __shfl_sync(0xffffffffu, fl, d);
            b[d] = __shfl_sync(0xffffffffu, bl, d);
        }
        if (tid == 0 && acc) {
            // displacement from the list's build position
            double rx, ry, rz;
            const double d2 = pairvec_exact(c, f[0], f[1], f[2], b[0], b[1], b[2], rx, ry, rz);
            if (d2 > maxd2) {
                maxd2 = d2;
                sh_maxd = fmax(sh_maxd, sqrt(d2));
            }
        }
        if (acc) {
            ++kacc;
            chi0 = chi5 = c1;
        }
        for (int q = tid; q < nterm; q += RMC_THREADS) {
            const int v = dcnt[q];
            if (v == 0) continue;
            if (acc) hist[in_smem ? q : row_of(q / nbins) * nbins + q % nbins] += v;
            dcnt[q] = 0;
        }
        // the next trial's particle
        const int prev = cur.i, next = (int)(u_at - ubase);
        cur = used == 10 ? nx10 : nx8;
        if (used == 9 || next + 16 > RMC_UBUF) {   // (9: the two chi^2 apart, never with g(r) alone)
            __syncthreads();
            if (next + 16 > RMC_UBUF) {
                ubase = u_at;
                fill();
                __syncthreads();
            }
            cur = ahead((int)(u_at - ubase));
        } else if (cur.i == prev) {
            cur.ol = fl;
        }
        __syncthreads();
    }
    __syncthreads();
    if (in_smem)   // back to the rows, the mirrored ones too
        for (int q = tid; q < nterm; q += RMC_THREADS) {
            const int mp = q / nbins, at = q % nbins, r = row_of(mp);
            ghist[r * nbins + at] = hist[q];
            if (mp > 0) ghist[(1 + ((r - 1) % nt) * nt + (r - 1) / nt) * nbins + at] = hist[q];
        }
    else
        for (int q = tid; q < k.npairs * nbins; q += RMC_THREADS) {
            const int r = row_of(1 + q / nbins), at = q % nbins;
            ghist[(1 + ((r - 1) % nt) * nt + (r - 1) / nt) * nbins + at] = ghist[r * nbins + at];
        }
    if (tid == 0) {
        out->kall = kall;
        out->kacc = kacc;
        out->used = u_at;
        for (int q = 0; q < 6; ++q) out->chisq[q] = q == 0 ? chi0 : (q == 5 ? chi5 : 0.0);
        out->maxd = sh_maxd;
        out->status = stop;
        out->started = 1;
    }
}

// counter-based uniforms in [0, 1): splitmix64 of (seed, index), 53 bits
__global__ void k_rmc_uniforms(long long count, unsigned long long seed, double* u) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(t + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    u[t] = (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

}  // namespace mdff
