// pair.cu -- short-range pair loop: n-m Lennard-Jones, BMH / BMHFTD with
// Tang-Toennies dispersion damping, and Morse.
//
// Replaces engforce_nmlj_pbc (src/field.f90:1181-1345), engforce_bmhftd_pbc
// (src/field.f90:2876-3026) and engforce_morse_pbc (src/field.f90:3039-3185).
// Layout: G lanes cooperate on one atom's full neighbour row (ELL); every
// lane accumulates the force on atom i only, so there are no atomics and the
// result is deterministic.  Energies, virial and stress are halved per
// ordered pair (each unordered pair is visited from both ends).
#include "common.cuh"

namespace mdff {

__device__ __forceinline__ void tt_damp(double b, double c, double r, int k, double& f, double& fd) {
    tt_damp_d(b, c, r, k, f, fd);
}

__device__ __forceinline__ double ipow_half(double x, double p) {
    // x^(p/2): repeated multiplication when p/2 is a small integer, pow otherwise.
    double h = 0.5 * p;
    int k = (int)h;
    if ((double)k == h && k >= 0 && k <= 16) {
        double r = 1.0, b = x;
        while (k) {
            if (k & 1) r *= b;
            b *= b;
            k >>= 1;
        }
        return r;
    }
    return pow(x, h);
}

// Lennard-Jones 12-6 alone, or BMH / BMHFTD alone, without the other
// potentials' registers and the exact expressions of k_pair: one rsqrt instead
// of a square root and four divisions, one e^{-BD r} and one polynomial for both
// damping orders, the virial from the stress sums.
// KIND 0: Lennard-Jones 12-6, 1: BMH, 2: BMHFTD.
template <int G, int KIND>
__global__ void __launch_bounds__(256, KIND == 0 ? 4 : 3)
    k_pair1(int n, const double4* __restrict__ rec, CellP c, const int* __restrict__ nbr, const int* __restrict__ cnt, int cap,
            const PairConst* __restrict__ pc, PairFlags fl, double* fx, double* fy, double* fz, double* part) {
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x & (G - 1);
    const bool active = gid < n;
    const int i = active ? gid : 0;
    double f0 = 0.0, f1 = 0.0, f2 = 0.0, ue = 0.0;
    double tau[6] = {0, 0, 0, 0, 0, 0};
    if (active) {
        const double4 ri = ld_rec(rec + i);
        const PairConst* Pi = pc + (int)__double_as_longlong(ri.w) * NT;
        const int m = cnt[i];
        const int* row = nbr + (size_t)i * cap;
        // the record one neighbour ahead, the index two ahead: their latency under
        // the arithmetic of this one
        double4 rn = ld_rec(rec + (sub < m ? row[sub] : i));
        int jn = sub + G < m ? row[sub + G] : i;
        for (int k = sub; k < m; k += G) {
            const double4 rj = rn;
            rn = ld_rec(rec + jn);
            jn = k + 2 * G < m ? row[k + 2 * G] : i;
            double rx, ry, rz;
            const double rsq = pairvec(fl.geom, c, ri.x, ri.y, ri.z, rj.x, rj.y, rj.z, rx, ry, rz);
            const PairConst& P = Pi[(int)__double_as_longlong(rj.w)];
            if (!(rsq < P.rcutsq)) continue;
            double w;
            if (KIND == 0) {
                const double sr2 = P.sigsq / rsq, srp = sr2 * sr2 * sr2, srq = srp * srp;
                double u = P.epsp * (P.plj * srq - P.qlj * srp);
                if (fl.trunc == 1) u -= P.uc;
                if (fl.trunc == 2) u += P.uc1 * rsq - P.uc2;
                w = P.fc * (srq - srp) * sr2;
                ue += u;
            } else {
                if (P.A == 0.0) continue;
                const double dm1 = rsqrt(rsq);
                double ub;
                w = bmh_pair(KIND == 2, P.A, P.B, P.C, P.D, P.BD, rsq * dm1, dm1, ub);
                ue += ub;
            }
            f0 = fma(w, rx, f0);
            f1 = fma(w, ry, f1);
            f2 = fma(w, rz, f2);
            const double wx = w * rx, wy = w * ry;
            tau[0] = fma(wx, rx, tau[0]);
            tau[1] = fma(wy, ry, tau[1]);
            tau[2] = fma(w * rz, rz, tau[2]);
            tau[3] = fma(wx, ry, tau[3]);
            tau[4] = fma(wx, rz, tau[4]);
            tau[5] = fma(wy, rz, tau[5]);
        }
    }
    f0 = group_sum<G>(f0);
    f1 = group_sum<G>(f1);
    f2 = group_sum<G>(f2);
    if (active && sub == 0) {
        fx[i] = f0;
        fy[i] = f1;
        fz[i] = f2;
    }
    // u and virial in the slots of the potential: u_lj vir_lj u_bmh vir_bmh u_mor vir_mor, then the stress
    const double u = 0.5 * ue, vir = 0.5 * (tau[0] + tau[1] + tau[2]);
    double v[12] = {KIND == 0 ? u : 0.0, KIND == 0 ? vir : 0.0, KIND == 0 ? 0.0 : u, KIND == 0 ? 0.0 : vir, 0.0, 0.0,
                    0.5 * tau[0], 0.5 * tau[1], 0.5 * tau[2], 0.5 * tau[3], 0.5 * tau[4], 0.5 * tau[5]};
    block_partials<12>(v, part);
}

template <int G>
__global__ void __launch_bounds__(256) k_pair(int n, const double4* __restrict__ rec, CellP c,
                                              const int* __restrict__ nbr, const int* __restrict__ cnt, int cap,
                                              const PairConst* __restrict__ pc, PairFlags fl, double* fx,
                                              double* fy, double* fz, double* part) {
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x & (G - 1);
    const bool active = gid < n;
    const int i = active ? gid : 0;
    double f0 = 0.0, f1 = 0.0, f2 = 0.0;
    double acc[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};   // u_lj vir_lj u_bmh vir_bmh u_mor vir_mor tau(6 -> 4 more below)
    double tau[6] = {0, 0, 0, 0, 0, 0};
    if (active) {
        const double4 ri = ld_rec(rec + i);
        const int ti = (int)__double_as_longlong(ri.w);
        const int m = cnt[i];
        const int* row = nbr + (size_t)i * cap;
        // the record one neighbour ahead, the index two ahead
        double4 rn = ld_rec(rec + (sub < m ? row[sub] : i));
        int jn = sub + G < m ? row[sub + G] : i;
        for (int k = sub; k < m; k += G) {
            const double4 rj = rn;
            rn = ld_rec(rec + jn);
            jn = k + 2 * G < m ? row[k + 2 * G] : i;
            double rx, ry, rz;
            const double rsq = pairvec_exact(c, ri.x, ri.y, ri.z, rj.x, rj.y, rj.z, rx, ry, rz);
            const PairConst& P = pc[ti * NT + (int)__double_as_longlong(rj.w)];
            if (!(rsq < P.rcutsq)) continue;
            double w = 0.0;
            if (fl.lj) {
                const double sr2 = P.sigsq / rsq;
                const double srp = ipow_half(sr2, P.plj);
                const double srq = ipow_half(sr2, P.qlj);
                double u = P.epsp * (P.plj * srq - P.qlj * srp);
                if (fl.trunc == 1) u -= P.uc;
                if (fl.trunc == 2) u += P.uc1 * rsq - P.uc2;
                const double wl = P.fc * (srq - srp) * sr2;
                acc[0] += 0.5 * u;
                acc[1] += 0.5 * wl * rsq;
                w += wl;
            }
            if ((fl.bmh || fl.bmhftd) && P.A != 0.0) {
                const double ir2 = 1.0 / rsq;
                const double d = sqrt(rsq);
                const double erh = P.A * exp(-P.B * d);
                double ir6 = ir2 * ir2 * ir2;
                double ir8 = ir6 * ir2;
                ir6 *= P.C;
                ir8 *= P.D;
                double ir6d = ir6, ir8d = ir8, fd6 = 0.0, fd8 = 0.0;
                if (fl.bmhftd) {
                    double f6, f8;
                    tt_damp(P.BD, 1.0, d, 6, f6, fd6);
                    tt_damp(P.BD, 1.0, d, 8, f8, fd8);
                    ir6d = ir6 * f6;
                    ir8d = ir8 * f8;
                }
                const double wb = (P.B * erh - 6.0 * ir6d / d - 8.0 * ir8d / d + ir6 * fd6 + ir8 * fd8) / d;
                acc[2] += 0.5 * (erh - ir6d - ir8d);
                acc[3] += 0.5 * wb * rsq;
                w += wb;
            }
            if (fl.morse) {
                const double d = sqrt(rsq);
                const double e = exp(-d * P.rhomor) * P.rs;
                const double em1 = e - 1.0;
                acc[4] += 0.5 * P.epsmor * (em1 * em1 - 1.0);
                const double wm = 2.0 * P.epsmor * P.rhomor * e * em1 / d;
                acc[5] += 0.5 * wm * rsq;
                w += wm;
            }
            f0 += w * rx;
            f1 += w * ry;
            f2 += w * rz;
            const double hw = 0.5 * w;
            tau[0] += hw * rx * rx;
            tau[1] += hw * ry * ry;
            tau[2] += hw * rz * rz;
            tau[3] += hw * rx * ry;
            tau[4] += hw * rx * rz;
            tau[5] += hw * ry * rz;
        }
    }
    f0 = group_sum<G>(f0);
    f1 = group_sum<G>(f1);
    f2 = group_sum<G>(f2);
    if (active && sub == 0) {
        fx[i] = f0;
        fy[i] = f1;
        fz[i] = f2;
    }
    double v[12] = {acc[0], acc[1], acc[2], acc[3], acc[4], acc[5], tau[0], tau[1], tau[2], tau[3], tau[4], tau[5]};
    block_partials<12>(v, part);
}

int launch_pair(cudaStream_t st, int n, const double4* rec, CellP c, const NList& l, const PairConst* pc, PairFlags fl,
                double* fx, double* fy, double* fz, Partials& part, DevScalars* d, bool sum) {
    const int threads = 256;
    auto grid = [&](int g) { return (int)(((size_t)n * g + threads - 1) / threads); };
    int blocks;
    const bool bm = fl.bmh || fl.bmhftd;
    const int kind = !fl.fast ? -1 : fl.lj && !bm && !fl.morse && fl.lj126 ? 0 : (bm && !fl.lj && !fl.morse ? (fl.bmhftd ? 2 : 1) : -1);
#define PAIR1(G, K) k_pair1<G, K><<<blocks, threads, 0, st>>>(n, rec, c, l.nbr, l.cnt, l.cap, pc, fl, fx, fy, fz, part.buf)
    // lanes per atom: 32 until the atoms fill the SMs with 8.  Where they cross depends on
    // the length of the rows too: at 35 to 39 times as many atoms as list neighbours, that
    // is a cell of about 150 cubes of the list radius (wide_rows).  Us at 8 and 32 lanes,
    // Lennard-Jones rc 2.5: 2 048 atoms 17.5 and 14.5, 16 384 25.7 and 36.7; rc 4.5: 6 912 45.0
    // and 36.0, 32 000 107 and 116; BMHFTD rc 6: 1 728 20.3 and 17.5, 13 824 29.9 and 38.7; rc 10:
    // 4 096 52.1 and 39.2, 32 768 181 and 194.
    const bool wide = fl.wide;
    if (kind >= 0) {
        blocks = grid(wide ? 32 : 8);
        if (kind == 0) { if (wide) PAIR1(32, 0); else PAIR1(8, 0); }
        else if (kind == 1) { if (wide) PAIR1(32, 1); else PAIR1(8, 1); }
        else { if (wide) PAIR1(32, 2); else PAIR1(8, 2); }
    } else {
        constexpr int G = 8;
        blocks = grid(G);
        k_pair<G><<<blocks, threads, 0, st>>>(n, rec, c, l.nbr, l.cnt, l.cap, pc, fl, fx, fy, fz, part.buf);
    }
#undef PAIR1
    // u_lj vir_lj u_bmh vir_bmh u_mor vir_mor, then the stress sums
    if (sum) launch_reduce_partials(st, part.buf, blocks, 12, d->nonb, 0);
    return blocks;
}

}  // namespace mdff
