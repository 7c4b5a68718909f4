// FP64-grade reciprocal space on the tensor cores: 56-bit fixed point in seven
// signed int8 digits.
//
// The phase factorises, e^{ik.r_a} = X_a[nx] Y_a[ny] Z_a[nz], so both passes of
// the FP64 path (multipole_ES_rec, src/field.f90:2646-2873) are GEMMs.  With the
// real basis cos(m t), sin(m t), t = 2 pi s_z, m = 0..kz, one GEMM row gives both
// signs of nz, half the products of the complex form:
//
//   structure factor   U_m = sum_a A0 cos(m t_a) - A1 (m/kz) sin(m t_a),
//                      V_m = sum_a A0 sin(m t_a) + A1 (m/kz) cos(m t_a),
//                      S(nx, ny, +-m) = U_m +- i V_m,
//       A0 = X Y (q + i (nx m1 + ny m2)), A1 = X Y kz m3, m_d = 2 pi b_d . mu;
//       rows = (column pair (nx, +-ny), re/im), K = (atom, A0/A1), N = (m, U/V);
//   field              F_j[i, c] = sum_m cos(m t_i) P_j[c, m] + sin(m t_i) Q_j[c, m],
//       P_j = m^j (a*_m + (-1)^j a*_-m), Q_j = i m^j (a*_m - (-1)^j a*_-m), a = A_k S;
//       rows = 128 atoms, K = (m, cos/sin), N = (column, moment j, re/im),
//   followed by the contraction over columns with X_i Y_i and the k-vectors.
//
// Every operand value, scaled to |v| <= 1, is an integer V = rn(v 127 2^48) in
// seven digits, balanced ones in [-128, 127], and for the structure factor's A
// operand, which is made anew for every evaluation, the plain bytes of V (the
// first signed, the others unsigned: nothing to carry); the 28 digit products of weight >= 2^48 (of 2^96) add
// up exactly in seven S32 levels of tensor memory and are joined in FP64.  Scales
// are per row (structure factor: a bound over the CTA's atoms and over nz) and per
// (column, moment) (field).  What is lost per term: the rounding of V, 2^-56 of the
// scale, and the dropped products, rms 2^-55.3 of it or less.  That is below one FP64
// rounding of the largest term and more of a small one: in a pass of dipoles alone
// the scale is at least kz times the largest m3, so a term at |nz| = 1 loses up to about
// kz 2^-56 of its own size (2^-51 at kz = 31), as much as a phase recurrence along nz
// does, which this form does not have.  The summation over atoms loses nothing.
//
// The MMAs of one K step: A digit i times B digits 0..6-i, which lie side by
// side along N, into levels i..6, N columns apart in tensor memory, as one MMA
// (two where the width passes 256).
#pragma once
#include "umma.cuh"

namespace mdff {
namespace tc7 {

constexpr int ND = 7;                        // int8 digits per value
constexpr double QS = 35747322042253312.0;   // 127 * 2^48
constexpr double QSH = 8323072.0;            // QS / 2^32
constexpr uint64_t WAIT_NS = 200000000ull;
constexpr int NLEV_MAX = 64;                 // widest N: seven levels fit 512 tensor-memory columns

// balanced digits of V (|V| <= 127 2^48 + 1/2): byte b of the result is the
// digit of weight 2^(8 b), b = 0..6
__device__ __forceinline__ unsigned long long digits56(long long V) {
    return ((unsigned long long)V + 0x0080808080808080ull) ^ 0x0080808080808080ull;
}

// rn(v QS) in plain two's complement for t = v QS / 2^32, |v| <= 1, on the FP64
// pipe (the conversion unit has a sixteenth of its rate): rint(t) by adding
// 1.5 2^52, the exact remainder times 2^32 the same way.  The second sum's high
// word is 0x43380000, less 1 where the remainder is negative: added to the
// first (whose constant takes the 0x43380000 off) it is the borrow.
constexpr double FIX_MH = 6755399441055744.0 - 1127743488.0;   // 1.5 2^52 - 0x43380000
__device__ __forceinline__ void fix56(double t, uint32_t& hi, uint32_t& lo) {
    const double h = t + FIX_MH;
    const double r = t - (h - FIX_MH);
    const double l = fma(r, 4294967296.0, umma::MAGIC52);
    hi = (uint32_t)__double2loint(h) + (uint32_t)__double2hiint(l);
    lo = (uint32_t)__double2loint(l);
}

// four values (consecutive K bytes) -> one word per digit, s[0] most significant
__device__ __forceinline__ void slices7(const uint32_t hi[4], const uint32_t lo[4], uint32_t s[ND]) {
    umma::slices4(hi[0], hi[1], hi[2], hi[3], s[0], s[1], s[2]);
    umma::slices4x4(lo[0], lo[1], lo[2], lo[3], s[3], s[4], s[5], s[6]);
}
__device__ __forceinline__ void slices7(unsigned long long a, unsigned long long b, unsigned long long c,
                                        unsigned long long d, uint32_t s[ND]) {
    umma::slices4((uint32_t)(a >> 32), (uint32_t)(b >> 32), (uint32_t)(c >> 32), (uint32_t)(d >> 32), s[0], s[1], s[2]);
    umma::slices4x4((uint32_t)a, (uint32_t)b, (uint32_t)c, (uint32_t)d, s[3], s[4], s[5], s[6]);
}

__device__ __forceinline__ bool wait(uint64_t* b, uint32_t parity, int* err, int code, volatile int* stop) {
    if (umma::mbar_wait_ns(b, parity, WAIT_NS, stop)) return true;
    if (!*stop) atomicOr(err, code);
    *stop = 1;
    return false;
}

// widths of the (at most two) MMAs of A digit i: multiples of 16, at most 256
__host__ __device__ __forceinline__ int first_width(int w) { return w <= 256 ? w : ((w / 2 + 15) / 16) * 16; }

// =============================================================================
// Structure factor
// =============================================================================

constexpr int SA = 16;                 // atoms per pipeline stage (one K step of 32 bytes)
constexpr int KB = 2 * SA;
constexpr int TP = 32;                 // column pairs per CTA tile: 128 rows
constexpr int AL = 4;                  // atoms per producer lane
constexpr int NG = 4;                  // producer groups, each filling every NG-th stage
constexpr int GW = TP * SA / AL / 32;  // warps per group
constexpr int NPW = NG * GW;
constexpr int THREADS = 32 * (NPW + 2);
constexpr int NA = 4;                  // A-operand buffers
constexpr int MAXIN = 8;
constexpr uint32_t A_SLICE = 128 * KB;
constexpr int AP = SA + 1;             // atoms per table entry, padded: entries 272 bytes apart, no bank conflicts
// S32 headroom: 2 K entries per atom and 7 products of 255 * 128 at the lowest level
constexpr int MAX_BLOCKS_PER_CTA = 288;

struct Layout {
    int N, ent, nin;
    uint32_t a_bytes, in_off, xy_off, p_off, in_bytes;
    __host__ __device__ static uint32_t up128(uint32_t x) { return (x + 127u) & ~127u; }
    __host__ __device__ Layout(int N_, int ent_, int nin_) : N(N_), ent(ent_), nin(nin_) {
        a_bytes = (uint32_t)ND * A_SLICE;
        in_off = NA * a_bytes;
        xy_off = up128(b_bytes());
        p_off = up128(xy_off + (uint32_t)ent * AP * 16u);
        in_bytes = up128(p_off + (uint32_t)SA * 32u);
    }
    __host__ __device__ uint32_t b_bytes() const { return (uint32_t)ND * N * KB; }
    __host__ __device__ uint32_t smem_bytes() const { return in_off + (uint32_t)nin * in_bytes + 128u; }
    __host__ static int depth(int N_, int ent_, size_t limit) {
        for (int d = MAXIN; d >= 2; --d)
            if (Layout(N_, ent_, d).smem_bytes() <= limit) return d;
        return 0;
    }
};

// Per position update: X_a[nx] (nx = 0..kx), then Y_a[ny] (ny = 0..ky), as
// [16-atom block][entry][AP]; atoms past n get 0.
__global__ void k_t7_xy(int n, int nblk, const double* __restrict__ sx, const double* __restrict__ sy, int kx, int ky,
                        double2* __restrict__ xy) {
    const int ent = kx + ky + 2;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)nblk * ent * AP) return;
    const int al = (int)(t % AP);
    const int e = (int)((t / AP) % ent), a = (int)(t / ((long)ent * AP)) * SA + al;
    double2 v = make_double2(0.0, 0.0);
    if (al < SA && a < n) {
        if (e <= kx) phase((double)e, sx[a], v.x, v.y);
        else phase((double)(e - kx - 1), sy[a], v.x, v.y);
    }
    xy[t] = v;
}

// Per position update: the B digit image of each block, rows d N + n (digit d,
// n = 2m: U_m, 2m+1: V_m), K = (atom, A0/A1), in the K-major core-matrix layout
// of one stage.  One thread per (two atoms, m).
__global__ void k_t7_bimage(int n, int nblk, const double* __restrict__ sz, int kz, int N, uint8_t* __restrict__ img) {
    const int half = N / 2;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)nblk * (SA / 2) * half) return;
    const int m = (int)(t % half), p2 = (int)((t / half) % (SA / 2)), blk = (int)(t / ((long)half * (SA / 2)));
    const double f = kz > 0 ? (double)m / (double)kz : 0.0;
    unsigned long long w[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int a = blk * SA + 2 * p2 + u;
        double c = 0.0, s = 0.0;
        if (a < n && m <= kz) phase((double)m, sz[a], c, s);
        w[0][2 * u] = digits56(__double2ll_rn(c * QS));
        w[0][2 * u + 1] = digits56(__double2ll_rn(-f * s * QS));
        w[1][2 * u] = digits56(__double2ll_rn(s * QS));
        w[1][2 * u + 1] = digits56(__double2ll_rn(f * c * QS));
    }
    uint8_t* base = img + (size_t)blk * ND * N * KB;
    const uint32_t lbo = (uint32_t)(ND * N / 8) * 128, dstep = (uint32_t)(N / 8) * 128;
    const int k = 4 * p2;
#pragma unroll
    for (int row = 0; row < 2; ++row) {
        uint32_t s[ND];
        slices7(w[row][0], w[row][1], w[row][2], w[row][3], s);
        const int r = 2 * m + row;
        const uint32_t off = (uint32_t)(k >> 4) * lbo + (uint32_t)(r >> 3) * 128 + (r & 7) * 16 + (k & 15);
#pragma unroll
        for (int d = 0; d < ND; ++d) *reinterpret_cast<uint32_t*>(base + d * dstep + off) = s[d];
    }
}

// Per evaluation: (q, m1, m2, m3) per atom and their largest magnitudes per
// block.  An integer holds no infinity or NaN: a block with a source or a
// position that is not finite gets the magnitude infinity, which makes its
// sums NaN (0 times infinity) where the rows are joined.
__global__ void k_t7_params(int n, int npad, const double* __restrict__ sx, const double* __restrict__ sy,
                            const double* __restrict__ sz, const double* __restrict__ q, const double* __restrict__ mu, CellP c,
                            int with_q, int with_mu, double4* __restrict__ prm, double4* __restrict__ bmax) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (a < n) {
        if (with_q) v[0] = q[a];
        if (with_mu) {
            const double u0 = mu[a], u1 = mu[n + a], u2 = mu[2 * n + a];
#pragma unroll
            for (int d = 0; d < 3; ++d) v[1 + d] = 2.0 * PI * (c.B[d] * u0 + c.B[3 + d] * u1 + c.B[6 + d] * u2);
        }
    }
    if (a < npad) prm[a] = make_double4(v[0], v[1], v[2], v[3]);
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    if (a < n && !(fabs(sx[a]) + fabs(sy[a]) + fabs(sz[a]) < inf)) v[0] = inf;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = fabs(v[k]) < inf ? fabs(v[k]) : inf;
        for (int o = SA / 2; o > 0; o >>= 1) v[k] = fmax(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    }
    if (a < npad && a % SA == 0) bmax[a / SA] = make_double4(v[0], v[1], v[2], v[3]);
}

// grid (tiles of TP column pairs, atom splits).  pairs: (nx, ny >= 0); trange:
// per tile the table entries it reads (first X, X count, first Y, Y count).
// Writes part[split][row kind: re+, im+, re-, im-][n][pair].
//
// Bound: the producers (27 FP64 and ~25 integer instructions per (column,
// atom), each pipe at one warp instruction per two clocks per scheduler) and
// the MMAs (28 digit products, ~800 clocks per 16-atom stage of 128 rows at N =
// 48) share the shared-memory port: 1 780 clocks per stage.  32 440 ions, kmax
// 23: 229 us against 1 374 us for the FP64 CUDA-core kernel (k_sfac); 3 000
// ions, kmax 10: 14 against 35.  12 producer warps: 234 us; two atoms a lane: 255.
__global__ void __launch_bounds__(THREADS, 1)
    k_sfac_t7(int nblk, int bps, int nin, const uint8_t* __restrict__ bimg, const double2* __restrict__ xy,
              const double4* __restrict__ prm, const double4* __restrict__ bmax, const int* __restrict__ pairs,
              const int* __restrict__ trange, int npair, int kx, int ky, int kz, int N, int entmax,
              double* __restrict__ part, int pstride, int* __restrict__ err) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t infull[MAXIN], inempty[MAXIN], afull[NA], aempty[NA], done;
    __shared__ uint32_t tslot;
    __shared__ double red[4][THREADS / 32];
    __shared__ volatile int stop;
    const Layout L(N, entmax, nin);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x, split = blockIdx.y;
    const int blk0 = split * bps, blk1 = min(nblk, blk0 + bps);
    const int nst = max(0, blk1 - blk0);
    const int x0 = trange[4 * tile], xn = trange[4 * tile + 1], y0 = trange[4 * tile + 2], yn = trange[4 * tile + 3];
    double mx[4] = {0.0, 0.0, 0.0, 0.0};
    for (int b = blk0 + tid; b < blk1; b += THREADS) {
        const double4 v = bmax[b];
        mx[0] = fmax(mx[0], v.x); mx[1] = fmax(mx[1], v.y); mx[2] = fmax(mx[2], v.z); mx[3] = fmax(mx[3], v.w);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        for (int o = 16; o > 0; o >>= 1) mx[k] = fmax(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        if (lane == 0) red[k][warp] = mx[k];
    }
    if (tid == 0) {
        for (int b = 0; b < nin; ++b) {
            umma::mbar_init(&infull[b], 1);
            umma::mbar_init(&inempty[b], 1);
        }
        for (int b = 0; b < NA; ++b) {
            umma::mbar_init(&afull[b], GW);
            umma::mbar_init(&aempty[b], 1);
        }
        umma::mbar_init(&done, 1);
        stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) umma::tmem_alloc(&tslot, 512);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tslot;
    for (int k = 0; k < 4; ++k) {
        mx[k] = 0.0;
        for (int w = 0; w < THREADS / 32; ++w) mx[k] = fmax(mx[k], red[k][w]);
    }
    const uint32_t sbase = umma::smem_u32(smem);
    // the scale of a pair's rows: a bound of |A0| and |A1| over the CTA's atoms
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    const bool finite = mx[0] < inf && mx[1] < inf && mx[2] < inf && mx[3] < inf;
    auto row_scale = [&](int nx, int ny) {
        return finite ? fmax(mx[0] + nx * mx[1] + ny * mx[2], kz * mx[3]) : inf;
    };

    if (warp < NPW) {
        // ---- producers: group warp / GW; a warp fills 16 pairs x 8 atoms of the
        // stage, a lane one pair x 4 atoms: 8 bytes of each of its 4 rows per
        // digit, so that each store of the warp is 256 contiguous bytes
        const int g = warp / GW, wg = warp % GW;
        constexpr int PW = 4 * AL;                           // pairs per warp
        const int pl = PW * (wg % (TP / PW)) + (lane % PW);  // pair within the tile
        const int a0 = 8 * (wg / (TP / PW)) + AL * (lane / PW);   // first atom within the stage
        const int pi = tile * TP + pl;
        const bool valid = pi < npair;
        const int nx = valid ? pairs[2 * pi] : x0, ny = valid ? pairs[2 * pi + 1] : y0;
        const double sg = row_scale(nx, ny);
        // rows whose sources all vanish contribute exact zeros
        const double rinv = valid && sg > 1e-280 ? QSH / sg : 0.0;
        const double fnx = (double)nx * rinv, fny = (double)ny * rinv, gk = (double)kz * rinv;
        const int ex = (nx - x0) * AP + a0, ey = (xn + ny - y0) * AP + a0;
        const int k0 = 2 * a0;
        const uint32_t off = (uint32_t)(k0 >> 4) * (16 * 128) + (uint32_t)(pl >> 3) * 128 + (pl & 7) * 16 + (k0 & 15);
        int bi = g % nin, ph = (g / nin) & 1;
        for (int s = g; s < nst; s += NG) {
            const int ba = s % NA;
            if (!wait(&infull[bi], ph, err, 1 << 8, &stop)) break;
            if (s >= NA && !wait(&aempty[ba], ((s / NA) - 1) & 1, err, 1 << 9, &stop)) break;
            const uint8_t* ib = smem + L.in_off + bi * L.in_bytes;
            const double2* sxy = reinterpret_cast<const double2*>(ib + L.xy_off);
            const double4* sp = reinterpret_cast<const double4*>(ib + L.p_off) + a0;
            uint32_t w[AL / 2][4][ND];   // [two atoms][row kind][digit]
#pragma unroll
            for (int h = 0; h < AL / 2; ++h) {
                uint32_t dh[4][4], dl[4][4];   // [row kind][A0, A1 of two atoms]
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const double2 X = sxy[ex + 2 * h + u], Y = sxy[ey + 2 * h + u];
                    const double4 P = sp[2 * h + u];
                    const double b = X.y * Y.y, dd = X.x * Y.y;
                    const double pr = fma(X.x, Y.x, -b), mr = fma(X.x, Y.x, b);
                    const double pim = fma(X.y, Y.x, dd), mi = fma(X.y, Y.x, -dd);
                    const double ar = P.x * rinv, t1 = fnx * P.y, gg = P.w * gk;
                    const double ap = fma(fny, P.z, t1), am = fma(-fny, P.z, t1);
                    fix56(fma(pr, ar, -pim * ap), dh[0][2 * u], dl[0][2 * u]);
                    fix56(fma(pr, ap, pim * ar), dh[1][2 * u], dl[1][2 * u]);
                    fix56(fma(mr, ar, -mi * am), dh[2][2 * u], dl[2][2 * u]);
                    fix56(fma(mr, am, mi * ar), dh[3][2 * u], dl[3][2 * u]);
                    fix56(pr * gg, dh[0][2 * u + 1], dl[0][2 * u + 1]);
                    fix56(pim * gg, dh[1][2 * u + 1], dl[1][2 * u + 1]);
                    fix56(mr * gg, dh[2][2 * u + 1], dl[2][2 * u + 1]);
                    fix56(mi * gg, dh[3][2 * u + 1], dl[3][2 * u + 1]);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) slices7(dh[r], dl[r], w[h][r]);
            }
            uint8_t* ab = smem + ba * L.a_bytes + off;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int q = 0; q < ND; ++q) {
                    uint8_t* o = ab + q * A_SLICE + r * (32 / 8) * 128;
                    *reinterpret_cast<uint2*>(o) = make_uint2(w[0][r][q], w[1][r][q]);
                }
            umma::fence_smem_to_async();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&afull[ba]);
            for (bi += NG; bi >= nin; bi -= nin) ph ^= 1;
        }
    } else if (warp == NPW + 1) {
        // ---- copies, up to nin stages ahead: B digit image, the tile's X and Y
        // entries, parameters
        if (lane == 0) {
            const int ent = kx + ky + 2;
            const uint32_t bytes = L.b_bytes() + (uint32_t)(xn + yn) * AP * 16u + SA * 32u;
            int last = -1, bi = 0, ph = 1;
            for (int s = 0; s < nst; ++s) {
                const size_t blk = blk0 + s;
                if (s >= nin && !wait(&inempty[bi], ph, err, 1 << 10, &stop)) break;
                uint8_t* ib = smem + L.in_off + bi * L.in_bytes;
                umma::mbar_arrive_expect_tx(&infull[bi], bytes);
                umma::bulk_g2s(ib, bimg + blk * L.b_bytes(), L.b_bytes(), &infull[bi]);
                umma::bulk_g2s(ib + L.xy_off, xy + (blk * ent + x0) * AP, (uint32_t)xn * AP * 16u, &infull[bi]);
                umma::bulk_g2s(ib + L.xy_off + (uint32_t)xn * AP * 16u, xy + (blk * ent + kx + 1 + y0) * AP,
                               (uint32_t)yn * AP * 16u, &infull[bi]);
                umma::bulk_g2s(ib + L.p_off, prm + blk * SA, SA * 32u, &infull[bi]);
                last = s;
                if (++bi == nin) { bi = 0; ph ^= 1; }
            }
            // every copy issued has landed before the CTA can exit, also when the
            // pipeline was abandoned on an error (bounded, whatever the stop flag)
            for (int k = max(0, last - nin + 1); k <= last; ++k) umma::mbar_wait_ns(&infull[k % nin], (k / nin) & 1, WAIT_NS);
        }
    } else {
        // ---- MMA issue: the whole warp on uniform descriptors, one elected lane issues
        const uint32_t lboA = 16 * 128, lboB = (uint32_t)(ND * N / 8) * 128;
        const uint64_t adesc0 = umma::desc_kmajor(sbase, lboA, 128);
        const uint64_t bdesc0 = umma::desc_kmajor(sbase + L.in_off, lboB, 128);
        const uint32_t astep = L.a_bytes >> 4, instep = L.in_bytes >> 4;
        bool ok = true;
        int bi = 0, ph = 0;
        for (int s = 0; s < nst && ok; ++s) {
            const int ba = s % NA;
            ok = __all_sync(0xffffffffu, wait(&infull[bi], ph, err, 1 << 11, &stop));
            if (ok) ok = __all_sync(0xffffffffu, wait(&afull[ba], (s / NA) & 1, err, 1 << 12, &stop));
            if (!ok) break;
            umma::fence_after_sync();
            const uint64_t ab = adesc0 + (uint64_t)(ba * astep), bb = bdesc0 + (uint64_t)(bi * instep);
#pragma unroll
            for (int i = 0; i < ND; ++i) {
                const uint64_t ad = ab + (uint64_t)(i * (A_SLICE >> 4));
                const uint32_t acc = (s > 0 || i > 0) ? 1u : 0u;
                const int w = (ND - i) * N, w1 = first_width(w);
                // A digits below the first are unsigned
                const uint32_t ty = i > 0 ? umma::IDESC_A_U8 : 0u;
                umma::mma_s8_warp(tmem + (uint32_t)(i * N), ad, bb, umma::idesc_s8(128, w1) ^ ty, acc);
                if (w1 < w)
                    umma::mma_s8_warp(tmem + (uint32_t)(i * N + w1), ad, bb + (uint64_t)(((w1 >> 3) * 128) >> 4),
                                      umma::idesc_s8(128, w - w1) ^ ty, acc);
            }
            umma::commit_warp(&inempty[bi]);
            umma::commit_warp(&aempty[ba]);
            if (++bi == nin) { bi = 0; ph ^= 1; }
        }
        umma::commit_warp(&done);
    }

    // ---- epilogue: warps 0-3, row kind = warp, pair = lane
    if (warp < 4) {
        const bool ok = wait(&done, 0, err, 1 << 13, &stop);
        umma::fence_after_sync();
        const int pi = tile * TP + lane;
        const bool valid = pi < npair;
        const double sg = valid ? row_scale(pairs[2 * pi], pairs[2 * pi + 1]) : 0.0;
        const double osc = sg * (281474976710656.0 / QS / QS);   // 2^48 / QS^2
        double* o = part + ((size_t)split * 4 + warp) * N * pstride + pi;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * warp) << 16);
        for (int j = 0; j < N / 8; ++j) {
            float d[ND][8];
            if (nst > 0) {
#pragma unroll
                for (int l = 0; l < ND; ++l) umma::tmem_ld8(lane_base + l * N + 8 * j, d[l]);
                umma::tmem_wait_ld();
            }
            if (!valid || !ok) continue;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                double v = 0.0;
                if (nst > 0) {
                    auto D = [&](int l) { return (long long)__float_as_int(d[l][e]); };
                    const long long hi = (D(0) << 24) + (D(1) << 16) + (D(2) << 8) + D(3);
                    const long long lo = (D(4) << 16) + (D(5) << 8) + D(6);
                    v = fma((double)hi, 16777216.0, (double)lo) * osc;
                }
                o[(size_t)(8 * j + e) * pstride] = v;
            }
        }
    }
    // every MMA has completed before the tensor memory is released, also when the
    // pipeline was abandoned on an error (bounded, whatever the stop flag)
    if (warp == 0 && !umma::mbar_wait_ns(&done, 0, WAIT_NS)) atomicOr(err, 1 << 13);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, 512);
    }
}

// The splits summed in order, the four vectors (+-ny, +-m) of each (pair, m),
// A_k S(k) and, with `energy`, the energy and stress sums (src/field.f90:
// 2742-2745, 2803-2815).  grid (tiles of 32 pairs, kz + 1), 256 H threads: H
// threads a sum, each taking every H-th split (H = 4 from 16 splits on, where one
// thread's chain of reads is the kernel's time: 3 000 ions, 37 splits 6.5 -> 4.6 us).
__global__ void __launch_bounds__(1024)
    k_t7_sreduce(int nsplit, int N, int npair, int pstride, const int* __restrict__ pairs, int ky, int kz, int nzl,
                 const double* __restrict__ part, const double* __restrict__ Ak, const double* __restrict__ kcoe,
                 CellP c, double* __restrict__ aks, int nrect, int energy, double* partials) {
    __shared__ double s[8][32], sh[3][8][32];
    const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 7;   // q = (row kind, U/V)
    const int h = threadIdx.x >> 8, H = blockDim.x >> 8;
    const int pi = blockIdx.x * 32 + lane, m = blockIdx.y;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    double sum = 0.0;
    if (pi < npair) {
        const double* p = part + ((size_t)(q >> 1) * N + 2 * m + (q & 1)) * pstride + pi;
        const size_t step = (size_t)4 * N * pstride;
#pragma unroll 8
        for (int k = h; k < nsplit; k += H) sum += p[k * step];
    }
    if (h > 0) sh[h - 1][q][lane] = sum;
    if (H > 1) __syncthreads();
    if (h == 0) {
        for (int w = 1; w < H; ++w) sum += sh[w - 1][q][lane];
        s[q][lane] = sum;
    }
    __syncthreads();
    const int sy = q & 1, sm = (q >> 1) & 1;   // sign of ny, of nz
    if (threadIdx.x < 128 && pi < npair) {   // q < 4 of the first group
        const int nx = pairs[2 * pi], ny = sy ? -pairs[2 * pi + 1] : pairs[2 * pi + 1], nz = sm ? -m : m;
        const double Ur = s[4 * sy][lane], Vr = s[4 * sy + 1][lane], Ui = s[4 * sy + 2][lane], Vi = s[4 * sy + 3][lane];
        const double sr = sm ? Ur + Vi : Ur - Vi, si = sm ? Ui - Vr : Ui + Vr;
        const int r = (nx * (2 * ky + 1) + ny + ky) * nzl + kz + nz;
        const bool twin = (sy && ny == 0) || (sm && nz == 0);   // the same vector again
        const double ak = Ak[r];
        if (!twin) {
            aks[r] = ak * sr;
            aks[nrect + r] = ak * si;
        }
        if (energy && !twin && ak != 0.0) {
            const double k0 = 2.0 * PI * (nx * c.B[0] + ny * c.B[1] + nz * c.B[2]);
            const double k1 = 2.0 * PI * (nx * c.B[3] + ny * c.B[4] + nz * c.B[5]);
            const double k2 = 2.0 * PI * (nx * c.B[6] + ny * c.B[7] + nz * c.B[8]);
            const double str = (sr * sr + si * si) * ak;
            const double kc = kcoe[r];
            v[0] = str;
            v[1] = (1.0 - kc * k0 * k0) * str;
            v[2] = (1.0 - kc * k1 * k1) * str;
            v[3] = (1.0 - kc * k2 * k2) * str;
            v[4] = -kc * k0 * k1 * str;
            v[5] = -kc * k0 * k2 * str;
            v[6] = -kc * k1 * k2 * str;
        }
    }
    if (energy) block_partials<7>(v, partials);
}

// =============================================================================
// Field
// =============================================================================

constexpr int NB = 32;                   // GEMM N per column block
constexpr int EPW = 16;                  // epilogue warps: 4 per tensor-memory lane quarter
constexpr int NQ = EPW / 4;
constexpr int FTHREADS = 32 * (EPW + 2);
constexpr int NBS = 4;                   // B stages
constexpr int BUFC = ND * NB;            // accumulator columns; two buffers fit 512
constexpr int NCONST = 16;
constexpr int FK_MAX = 64;               // K bytes per row: keeps two joined levels inside int32

template <int NMOM>
struct Cfg {
    static constexpr int CB = NMOM == 2 ? 8 : 4;    // columns per block
    static constexpr int HC = CB / NQ;              // columns per epilogue warp
    static constexpr int CW = NB / CB;              // accumulator columns per k column (4, or 6 padded to 8)
};

struct FLayout {
    uint32_t a_bytes, b_off, img_bytes, stage_bytes;
    __host__ __device__ FLayout(int KZ, int CB) {
        a_bytes = (uint32_t)ND * 128u * KZ;
        b_off = (a_bytes + 127u) & ~127u;
        img_bytes = (uint32_t)ND * NB * KZ + (uint32_t)CB * NCONST * 8u;
        stage_bytes = (img_bytes + 127u) & ~127u;
    }
    __host__ __device__ uint32_t smem_bytes() const { return b_off + NBS * stage_bytes + 128u; }
};

// Per position update: the A digit image of each 128-atom tile (K = (m, cos/sin), KZ bytes per row).
__global__ void k_t7f_aimage(int n, int ntile, const double* __restrict__ sz, int kz, int KZ, uint8_t* __restrict__ img) {
    const int nch = KZ / 16;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)ntile * 128 * nch) return;
    const int kc = (int)(t % nch), a = (int)(t / nch);
    const int tile = a / 128, r = a % 128;
    uint32_t s[4][ND];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        unsigned long long d[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int m = 8 * kc + 2 * g + u;
            double c = 0.0, sn = 0.0;
            if (a < n && m <= kz) phase((double)m, sz[a], c, sn);
            d[2 * u] = digits56(__double2ll_rn(c * QS));
            d[2 * u + 1] = digits56(__double2ll_rn(sn * QS));
        }
        slices7(d[0], d[1], d[2], d[3], s[g]);
    }
    uint8_t* base = img + (size_t)tile * ND * 128 * KZ + (uint32_t)kc * (16 * 128) + (uint32_t)(r >> 3) * 128 + (r & 7) * 16;
#pragma unroll
    for (int q = 0; q < ND; ++q)
        *reinterpret_cast<uint4*>(base + (size_t)q * 128 * KZ) = make_uint4(s[0][q], s[1][q], s[2][q], s[3][q]);
}

// Per evaluation: B digit image and constants of each column block.  Block =
// one column block, thread = (GEMM row, 16-byte K chunk).  Constants per column
// with s_j = (scale of moment j) 2^48 / QS^2: s0 kc (3), s1, s0 kc_d kc_e (00 11
// 22 01 02 12), s1 kc (3), s2, where kc = 2 pi (nx b_1 + ny b_2), and four ints.
template <int NMOM>
__global__ void k_t7f_bimage(int ncol, const int* __restrict__ cols, int kx, int ky, int kz, int nzl, int KZ,
                             const double* __restrict__ aks, int nrect, CellP c, uint8_t* __restrict__ img) {
    using C = Cfg<NMOM>;
    const int nch = KZ / 16;
    const FLayout L(KZ, C::CB);
    __shared__ unsigned long long smax[C::CB * NMOM];
    const int q = blockIdx.x, t = threadIdx.x;
    if (t < C::CB * NMOM) smax[t] = 0ull;
    __syncthreads();
    const int nr = t / nch, kc = t % nch;
    const int cl = nr / C::CW, j = (nr % C::CW) >> 1, part = nr & 1;
    const int li = q * C::CB + cl;
    const bool valid = nr < NB && j < NMOM && li < ncol;
    double v[16];   // (cos, sin) coefficients of the chunk's 8 m
    double mx = 0.0;
    const int col = valid ? cols[li] : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int m = 8 * kc + u;
        double pr = 0.0, pi = 0.0, qr = 0.0, qi = 0.0;
        if (valid && m <= kz) {
            const double w = j == 0 ? 1.0 : (j == 1 ? (double)m : (double)m * (double)m);
            const size_t r = (size_t)col * nzl + kz;
            const double ar = aks[r + m], ai = -aks[nrect + r + m];
            if (m == 0) {
                pr = w * ar; pi = w * ai;
            } else {
                double br = aks[r - m], bi = -aks[nrect + r - m];
                if (j == 1) { br = -br; bi = -bi; }
                pr = w * (ar + br); pi = w * (ai + bi);
                qr = -w * (ai - bi); qi = w * (ar - br);   // i (a* -+ b*)
            }
        }
        v[2 * u] = part ? pi : pr;
        v[2 * u + 1] = part ? qi : qr;
        const double big = fabs(v[2 * u]) + fabs(v[2 * u + 1]), inf = __longlong_as_double(0x7ff0000000000000ll);
        mx = big < inf ? fmax(mx, fmax(fabs(v[2 * u]), fabs(v[2 * u + 1]))) : inf;   // not finite: the sums become NaN
    }
    if (valid) atomicMax(&smax[cl * NMOM + j], (unsigned long long)__double_as_longlong(mx));
    __syncthreads();
    uint8_t* base = img + (size_t)q * L.stage_bytes;
    if (nr < NB) {
        const double sg = valid ? __longlong_as_double((long long)smax[cl * NMOM + j]) : 0.0;
        const double qs = sg > 1e-280 ? QS / sg : 0.0;
        uint32_t s[4][ND];
#pragma unroll
        for (int g = 0; g < 4; ++g)
            slices7(digits56(__double2ll_rn(v[4 * g] * qs)), digits56(__double2ll_rn(v[4 * g + 1] * qs)),
                    digits56(__double2ll_rn(v[4 * g + 2] * qs)), digits56(__double2ll_rn(v[4 * g + 3] * qs)), s[g]);
        const uint32_t lbo = (uint32_t)(ND * NB / 8) * 128, dstep = (uint32_t)(NB / 8) * 128;
        const uint32_t off = (uint32_t)kc * lbo + (uint32_t)(nr >> 3) * 128 + (nr & 7) * 16;
#pragma unroll
        for (int d = 0; d < ND; ++d)
            *reinterpret_cast<uint4*>(base + d * dstep + off) = make_uint4(s[0][d], s[1][d], s[2][d], s[3][d]);
    }
    if (t < C::CB) {
        double* k = reinterpret_cast<double*>(base + (size_t)ND * NB * KZ) + t * NCONST;
        const int l2 = q * C::CB + t;
        double cv[14];
        int4 id = make_int4(0, kx + 1, 0, 0);
#pragma unroll
        for (int e = 0; e < 14; ++e) cv[e] = 0.0;
        if (l2 < ncol) {
            const int nx = cols[l2] / (2 * ky + 1), ny = cols[l2] % (2 * ky + 1) - ky;
            const double w = 281474976710656.0 / QS / QS;
            double s[3] = {0.0, 0.0, 0.0}, kk[3];
            for (int e = 0; e < NMOM; ++e) s[e] = __longlong_as_double((long long)smax[t * NMOM + e]) * w;
            for (int d = 0; d < 3; ++d) kk[d] = 2.0 * PI * (nx * c.B[3 * d] + ny * c.B[3 * d + 1]);
            for (int d = 0; d < 3; ++d) { cv[d] = s[0] * kk[d]; cv[4 + d] = s[0] * kk[d] * kk[d]; cv[10 + d] = s[1] * kk[d]; }
            cv[3] = s[1];
            cv[7] = s[0] * kk[0] * kk[1]; cv[8] = s[0] * kk[0] * kk[2]; cv[9] = s[0] * kk[1] * kk[2];
            cv[13] = s[2];
            // table entries of X and Y, conjugate Y, and how the column follows others
            // of the list: 1: the next ny after the previous column, 2: CB after the
            // one CB places before
            const bool step1 = l2 >= 1 && cols[l2] == cols[l2 - 1] + 1 && ny > -ky;
            const bool stepb = l2 >= C::CB && cols[l2] == cols[l2 - C::CB] + C::CB && ny - C::CB >= -ky && ky >= C::CB;
            id = make_int4(nx, kx + 1 + (ny < 0 ? -ny : ny), ny < 0 ? 1 : 0, (step1 ? 1 : 0) | (stepb ? 2 : 0));
        }
#pragma unroll
        for (int e = 0; e < 14; ++e) k[e] = cv[e];
        *reinterpret_cast<int4*>(k + 14) = id;
    }
}

// an int as a double on the FP64 pipe: 2^52 + 2^31 + x has x + 2^31 as its low word
__device__ __forceinline__ double to_f64(int x) {
    return __hiloint2double(0x43300000, (int)((uint32_t)x ^ 0x80000000u)) - 4503601774854144.0;
}
// the seven levels joined: sum_l D_l 2^(48 - 8 l).  Two levels stay inside int32 up
// to FK_MAX bytes of K; half of the conversions take the conversion unit, which
// is idle otherwise (wide integer multiply-adds run at a fifth of its issue rate
// and made the field pass 6 % slower).
__device__ __forceinline__ double join7(float d0, float d1, float d2, float d3, float d4, float d5, float d6) {
    const double a = (double)(__float_as_int(d0) * 256 + __float_as_int(d1));
    const double b = to_f64(__float_as_int(d2) * 256 + __float_as_int(d3));
    const double c = to_f64(__float_as_int(d4) * 256 + __float_as_int(d5));
    return fma(fma(fma(a, 65536.0, b), 65536.0, c), 256.0, (double)__float_as_int(d6));
}

// `grid` CTAs, each an equal contiguous range of the (tile, column block) units
// (umma::unit0).  Writes
// fpart[((slot * NQ + part) * nv + component) * n + i], slot counted from the
// first CTA of the atom's tile, nv = 3 or 9.
//
// Bound: the epilogue, joining 28 levels and contracting with X Y per (atom,
// column): ~2 000 clocks per (128 atoms, 8 columns) block against ~1 350 of the
// MMAs (K = 64), overlapped through two accumulator buffers.  32 440 ions, kmax
// 23: 336 us (614 with the gradient) against 1 698 (2 900) for the FP64
// CUDA-core kernel (k_kfield); 3 000 ions, kmax 10: 11 against 20, and its
// reduction over column splits 4 against 38.  Two accumulator
// buffers.  X Y advances along a run of columns by one rotation per CB columns
// (at most (2 ky + 1) / CB of them in a row), and comes from the table where a
// run starts.
template <int NMOM>
__global__ void __launch_bounds__(FTHREADS, 1)
    k_kfield_t7(int n, int ntile, int ncol, int ncb, const uint8_t* __restrict__ aimg, const double2* __restrict__ xy,
                const uint8_t* __restrict__ bimg, int kx, int ky, int KZ, CellP c, double* __restrict__ fpart,
                int* __restrict__ err) {
    using C = Cfg<NMOM>;
    constexpr int NV = NMOM == 3 ? 9 : 3;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t afull, afree, bfull[NBS], bempty[NBS], accfull[2], accfree[2], fin;
    __shared__ uint32_t tslot;
    __shared__ volatile int stop;
    const FLayout L(KZ, C::CB);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long units = (long)ntile * ncb;
    const int grid = gridDim.x;
    const long u0 = umma::unit0(blockIdx.x, units, grid);
    const int cnt = (int)(umma::unit0(blockIdx.x + 1, units, grid) - u0), tile0 = (int)(u0 / ncb), q0 = (int)(u0 % ncb);
    if (tid == 0) {
        umma::mbar_init(&afull, 1);
        umma::mbar_init(&afree, 1);
        for (int b = 0; b < NBS; ++b) {
            umma::mbar_init(&bfull[b], 1);
            umma::mbar_init(&bempty[b], 1 + EPW);
        }
        for (int b = 0; b < 2; ++b) {
            umma::mbar_init(&accfull[b], 1);
            umma::mbar_init(&accfree[b], EPW);
        }
        umma::mbar_init(&fin, 1);
        stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) umma::tmem_alloc(&tslot, 512);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tslot;
    const uint32_t sbase = umma::smem_u32(smem);

    if (warp == EPW + 1) {
        // ---- copies: a tile's A image when the range enters it (once the last
        // tile's MMAs are done), and the B stages
        if (lane == 0) {
            int seg = 0, last = -1;
            bool a_open = false;
            int tile = tile0, q = q0;
            for (int it = 0; it < cnt; ++it) {
                const int bs = it % NBS;
                if (it == 0 || q == 0) {
                    if (seg > 0 && !wait(&afree, (seg - 1) & 1, err, 1 << 14, &stop)) break;
                    umma::mbar_arrive_expect_tx(&afull, L.a_bytes);
                    umma::bulk_g2s(smem, aimg + (size_t)tile * L.a_bytes, L.a_bytes, &afull);
                    a_open = true;
                    ++seg;
                }
                if (it >= NBS && !wait(&bempty[bs], ((it / NBS) - 1) & 1, err, 1 << 15, &stop)) break;
                umma::mbar_arrive_expect_tx(&bfull[bs], L.img_bytes);
                umma::bulk_g2s(smem + L.b_off + bs * L.stage_bytes, bimg + (size_t)q * L.stage_bytes, L.img_bytes, &bfull[bs]);
                last = it;
                if (++q == ncb) { q = 0; ++tile; }
            }
            // every copy issued has landed before the CTA can exit
            if (a_open) umma::mbar_wait_ns(&afull, (seg - 1) & 1, WAIT_NS);
            for (int k = max(0, last - NBS + 1); k <= last; ++k) umma::mbar_wait_ns(&bfull[k % NBS], (k / NBS) & 1, WAIT_NS);
        }
    } else if (warp == EPW) {
        // ---- MMA issue (the whole warp, one elected lane issues)
        const uint32_t lboA = 16 * 128, lboB = (uint32_t)(ND * NB / 8) * 128;
        const uint64_t adesc0 = umma::desc_kmajor(sbase, lboA, 128);
        const uint64_t bdesc0 = umma::desc_kmajor(sbase + L.b_off, lboB, 128);
        const uint32_t aslice = (128u * KZ) >> 4, astep = (2 * lboA) >> 4, bstep = (2 * lboB) >> 4, bstage = L.stage_bytes >> 4;
        int seg = 0, q = q0;
        bool ok = true;
        for (int it = 0; it < cnt && ok; ++it) {
            const int bs = it % NBS, tb = it & 1;
            if (it == 0 || q == 0) {
                ok = __all_sync(0xffffffffu, wait(&afull, seg & 1, err, 1 << 16, &stop));
                ++seg;
            }
            if (ok) ok = __all_sync(0xffffffffu, wait(&bfull[bs], (it / NBS) & 1, err, 1 << 17, &stop));
            if (ok && it >= 2) ok = __all_sync(0xffffffffu, wait(&accfree[tb], ((it >> 1) - 1) & 1, err, 1 << 18, &stop));
            if (!ok) break;
            umma::fence_after_sync();
            const uint64_t bq = bdesc0 + (uint64_t)(bs * bstage);
            for (int ks = 0; ks < KZ / 32; ++ks) {
#pragma unroll
                for (int i = 0; i < ND; ++i) {
                    const uint64_t ad = adesc0 + (uint64_t)(i * aslice + ks * astep);
                    const uint64_t bd = bq + (uint64_t)(ks * bstep);
                    umma::mma_s8_warp(tmem + tb * BUFC + i * NB, ad, bd, umma::idesc_s8(128, (ND - i) * NB),
                                      (ks > 0 || i > 0) ? 1u : 0u);
                }
            }
            umma::commit_warp(&accfull[tb]);
            umma::commit_warp(&bempty[bs]);
            if (++q == ncb) q = 0;
            if (q == 0 || it == cnt - 1) umma::commit_warp(&afree);
        }
        umma::commit_warp(&fin);
    } else {
        // ---- epilogue: atom row = 32 (warp % 4) + lane, columns [HC part, HC part + HC) of a block
        const int qd = warp & 3, part = warp >> 2;
        const int r = 32 * qd + lane;
        const int ent = kx + ky + 2;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * qd) << 16);
        double E[3], SI1, G[6], H[3], SR2;
        double wr = 0.0, wi = 0.0, e1r = 1.0, e1i = 0.0, esr = 1.0, esi = 0.0;
        int i = 0;
        auto table = [&](int e) {   // entry e of the lane's atom
            const int a = min(i, n - 1);
            return xy[((size_t)(a / SA) * ent + e) * AP + a % SA];
        };
        auto entry = [&](const int4& id, double& ur, double& ui) {   // X Y of a column from the table
            const double2 X = table(id.x);
            double2 Y = table(id.y);
            if (id.z) Y.y = -Y.y;
            ur = fma(X.x, Y.x, -X.y * Y.y);
            ui = fma(X.x, Y.y, X.y * Y.x);
        };
        int tile = tile0, q = q0;
        for (int it = 0; it < cnt; ++it) {
            const int bs = it % NBS, tb = it & 1;
            const bool fresh = it == 0 || q == 0;
            if (fresh) {
                i = tile * 128 + r;
#pragma unroll
                for (int e = 0; e < 3; ++e) { E[e] = 0.0; H[e] = 0.0; }
#pragma unroll
                for (int e = 0; e < 6; ++e) G[e] = 0.0;
                SI1 = SR2 = 0.0;
                if (ky >= 1) { const double2 v = table(kx + 2); e1r = v.x; e1i = v.y; }
                if (ky >= C::CB) { const double2 v = table(kx + 1 + C::CB); esr = v.x; esi = v.y; }
            }
            // the block's constants, and X Y of the warp's columns, before the MMAs are done
            if (!wait(&bfull[bs], (it / NBS) & 1, err, 1 << 19, &stop)) break;
            const double* kst = reinterpret_cast<const double*>(smem + L.b_off + bs * L.stage_bytes + (size_t)ND * NB * KZ) +
                                part * C::HC * NCONST;
            double vr[C::HC], vi[C::HC];
#pragma unroll
            for (int cc = 0; cc < C::HC; ++cc) {
                const int4 id = *reinterpret_cast<const int4*>(kst + cc * NCONST + 14);
                if (cc == 0) {
                    if ((id.w & 2) && !fresh) {   // CB columns on from this warp's last one
                        const double t = fma(wr, esr, -wi * esi);
                        wi = fma(wi, esr, wr * esi);
                        wr = t;
                    } else {
                        entry(id, wr, wi);
                    }
                    vr[0] = wr;
                    vi[0] = wi;
                } else if (id.w & 1) {            // the next column
                    vr[cc] = fma(vr[cc - 1], e1r, -vi[cc - 1] * e1i);
                    vi[cc] = fma(vi[cc - 1], e1r, vr[cc - 1] * e1i);
                } else {
                    entry(id, vr[cc], vi[cc]);
                }
            }
            if (!wait(&accfull[tb], (it >> 1) & 1, err, 1 << 20, &stop)) break;
            umma::fence_after_sync();
            float d[ND][8];
#pragma unroll
            for (int l = 0; l < ND; ++l) umma::tmem_ld8(lane_base + tb * BUFC + l * NB + part * 8, d[l]);
            umma::tmem_wait_ld();
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&accfree[tb]);
            double f[8];   // in straight line: the joins of all columns overlap
#pragma unroll
            for (int o = 0; o < 8; ++o)
                if (o % C::CW < 2 * NMOM) f[o] = join7(d[0][o], d[1][o], d[2][o], d[3][o], d[4][o], d[5][o], d[6][o]);
#pragma unroll
            for (int cc = 0; cc < C::HC; ++cc) {   // (a padding column has zero constants)
                const double* k = kst + cc * NCONST;
                const int o = cc * C::CW;
                const double i0 = fma(vr[cc], f[o + 1], vi[cc] * f[o]), i1 = fma(vr[cc], f[o + 3], vi[cc] * f[o + 2]);
                E[0] = fma(k[0], i0, E[0]);
                E[1] = fma(k[1], i0, E[1]);
                E[2] = fma(k[2], i0, E[2]);
                SI1 = fma(k[3], i1, SI1);
                if (NMOM == 3) {
                    const double r0 = fma(vr[cc], f[o], -vi[cc] * f[o + 1]), r1 = fma(vr[cc], f[o + 2], -vi[cc] * f[o + 3]);
                    const double r2 = fma(vr[cc], f[(o + 4) & 7], -vi[cc] * f[(o + 5) & 7]);
#pragma unroll
                    for (int e = 0; e < 6; ++e) G[e] = fma(k[4 + e], r0, G[e]);
#pragma unroll
                    for (int e = 0; e < 3; ++e) H[e] = fma(k[10 + e], r1, H[e]);
                    SR2 = fma(k[13], r2, SR2);
                }
            }
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&bempty[bs]);
            const bool last = q == ncb - 1 || it == cnt - 1;
            if (last && i < n) {   // the tile's segment is done
                const int slot = (int)blockIdx.x - umma::range_of((long)tile * ncb, units, grid);
                double* o = fpart + (size_t)(slot * NQ + part) * NV * n + i;
                const double b3[3] = {2.0 * PI * c.B[2], 2.0 * PI * c.B[5], 2.0 * PI * c.B[8]};
                for (int e = 0; e < 3; ++e) o[(size_t)e * n] = fma(b3[e], SI1, E[e]);
                if (NMOM == 3) {
                    const int pd[6] = {0, 1, 2, 0, 0, 1}, pe[6] = {0, 1, 2, 1, 2, 2};
                    for (int e = 0; e < 6; ++e)
                        o[(size_t)(3 + e) * n] =
                            G[e] + b3[pe[e]] * H[pd[e]] + b3[pd[e]] * H[pe[e]] + b3[pd[e]] * b3[pe[e]] * SR2;
                }
            }
            if (++q == ncb) { q = 0; ++tile; }
        }
    }
    // every MMA has completed before the tensor memory is released, also when the
    // pipeline was abandoned on an error (bounded, whatever the stop flag)
    if (warp == 0 && !umma::mbar_wait_ns(&fin, 0, WAIT_NS)) atomicOr(err, 1 << 21);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, 512);
    }
}

}  // namespace tc7
}  // namespace mdff
