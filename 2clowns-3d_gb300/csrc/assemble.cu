// assemble.cu -- static coefficients, row numbering, right-hand side, per-step
// matrix assembly and the pressure / velocity correction on the GPU.
//
// This translation unit is compiled with --fmad=false: every coefficient is
// produced with separately rounded multiplies and adds, in the reference's
// evaluation order, so the assembled matrix is bit-identical to an IEEE
// evaluation of the Fortran source (the per-row sort inside the solve compares
// these values, and ties must break the same way).
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "grid_index.cuh"
#include "trace.h"

namespace clowns {

constexpr int kAsmBlock = 256;

static inline int grid_for(long n) {
    long b = (n + kAsmBlock - 1) / kAsmBlock;
    if (b < 1) b = 1;
    if (b > 152L * 16) b = 152L * 16;
    return (int)b;
}

// ---------------------------------------------------------------------------
// mp = minval(dx, dx > 0)**2 over the axes in `axes` (bit l: axis l): every
// axis in 3D (1sub-matrix.F90:17), the two of the x-z or y-z plane in 2DV (20-21)
__global__ void k_min_dx(const double* __restrict__ dx, int count, int axes, double* mp) {
    __shared__ double s[256];
    double m = 1.0e300;
    for (int t = threadIdx.x; t < count; t += blockDim.x) {
        if (!((axes >> (t % 3)) & 1)) continue;
        double v = dx[t];
        if (v > 0.0 && v < m) m = v;
    }
    s[threadIdx.x] = m;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o && s[threadIdx.x + o] < s[threadIdx.x]) s[threadIdx.x] = s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *mp = s[0] * s[0];
}

// cal_alu_f (1sub-matrix.F90:82-87)
__device__ __forceinline__ double cal_alu_f(double dx, double dxm, double ax, double fb) {
    return 2.0 / dx / (dx + dxm) * ax / fb;
}
// cal_alu (1sub-matrix.F90:75-80)
__device__ __forceinline__ double cal_alu(double fnn, double dx, double dxm) {
    return (fnn - 0.5) * dx / (fnn * dx + dxm * 0.5) * (-1.0);
}

// init_matrix (1sub-matrix.F90:25-65), one thread per cell nnn = 1..inne;
// columns 2q, 2q+1 hold the minus and plus faces of axis col_axis(q).
//
// What bounds it: an FP64 division costs about ten FP64 operations of a pipe that
// does 1.7 lane operations per clock and SM, and cal_alu_f has three per face: the
// kernel ran at 1.60 ms for 4.9 M cells (0.6 GB of traffic, 0.09 ms).  The factors
// depend on one index of one axis, so every block forms the table of all of them in
// shared memory (TAB; one block per SM walks its cells), and a face needs only the
// products with its area and porosity where these are not 1; the six quotients by one
// porosity take its reciprocal (Markstein): 176 us, half of it FP64 and the rest the
// dependent loads of six neighbours.
// TAB = false: grids whose table exceeds shared memory form every factor, in small blocks:
// there is no table to share, and long grids of few cells (1024 / 128 threads: 45 / 29 us
// at 1500 x 1 x 45 cells, 74 / 50 at 2000 x 1 x 80, 634 / 579 at 1600 x 40 x 30) leave SMs idle
// otherwise.
constexpr int kInitBlock = 1024;
constexpr int kInitPlainBlock = 128;
template <int NL, bool TAB>
__global__ void __launch_bounds__(kInitBlock, 1) k_init_matrix(GridIdx g, int inne, int mx2, const int* __restrict__ mn,
                                                          const int* __restrict__ in_, const int* __restrict__ jn,
                                                          const int* __restrict__ kn, const int* __restrict__ nf,
                                                          const int* __restrict__ nfb, const double* __restrict__ a,
                                                          const double* __restrict__ fb, const double* __restrict__ dx,
                                                          const double* __restrict__ mp_p, double* __restrict__ alu_c,
                                                          int* __restrict__ ll_c, double* __restrict__ de_c) {
    extern __shared__ double tab[];
    const double mp = *mp_p;
    const long ld = inne;
    const int base[3] = {g.is - 1, g.js - 1, g.ks - 1};     // cells lie in ls - 1 .. le + 1
    const int len[3] = {g.ie - g.is + 3, g.je - g.js + 3, g.ke - g.ks + 3};
    const int total = len[0] + len[1] + len[2];
    const int at[3] = {-base[0], len[0] - base[1], len[0] + len[1] - base[2]};
    if (TAB) {
        for (int t = threadIdx.x; t < 2 * total; t += blockDim.x) {
            const int side = t >= total, u = t - side * total;
            const int l = u < len[0] ? 0 : u < len[0] + len[1] ? 1 : 2, i = u - at[l];
            if (i + side > mx2) continue;
            const double d = dx[g.dxo(l, i)], dm = dx[g.dxo(l, i + (side ? 1 : -1))];
            const double f = 2.0 / d / (d + dm);
            tab[t] = f;
            tab[2 * total + t] = -(mp * f);
        }
        __syncthreads();
    }
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < inne; t += (long)gridDim.x * blockDim.x) {
        const int nnn = (int)t + 1;
        const double fbn = fb[nnn];
        const int fl = nf[nnn];
        const int i = in_[nnn], j = jn[nnn], k = kn[nnn];
        if (fl == -1 || is_zero(fbn)) {
#pragma unroll
            for (int c = 0; c < NL; c++) { alu_c[c * ld + t] = 0.0; ll_c[c * ld + t] = 0; }
            de_c[t] = 0.0;
            continue;
        }
        const int lg[3] = {i, j, k};
        const int self = mn[g.mn_off(i, k, j)];
        int np[NL], fn[NL];
        double ar[NL], fbp[NL];
#pragma unroll
        for (int c = 0; c < NL; c++) np[c] = mn[g.nbr(i, j, k, g.col_axis(c / 2), c & 1 ? 1 : -1)];
#pragma unroll
        for (int c = 0; c < NL; c++) {
            fn[c] = nf[np[c]];
            ar[c] = a[3L * (c & 1 ? np[c] : self) + g.col_axis(c / 2)];
            fbp[c] = fb[np[c]];
        }
        const bool full = is_one(fbn);
        Recip rfb = {};
        if (TAB && !full) rfb = make_recip(fbn);
        double de = 0.0;
#pragma unroll
        for (int c = 0; c < NL; c++) {                      // 3D: x-, x+, y-, y+, z-, z+
            const int l = g.col_axis(c / 2), side = c & 1;
            if ((fn[c] == -1 && nfb[np[c]] != 4) || is_zero(ar[c]) || is_zero(fbp[c])) {
                ll_c[c * ld + t] = 0;
                alu_c[c * ld + t] = 0.0;
                continue;
            }
            double v;
            if (TAB) {
                const int o = side * total + at[l] + lg[l];
                if (full && is_one(ar[c])) v = tab[2 * total + o];
                else {
                    v = tab[o] * ar[c];
                    if (!full) v = div_by(v, rfb);
                    v = -(mp * v);
                }
            } else {
                v = -(mp * cal_alu_f(dx[g.dxo(l, lg[l])], dx[g.dxo(l, lg[l] + (side ? 1 : -1))], ar[c], fbn));
            }
            ll_c[c * ld + t] = np[c];
            alu_c[c * ld + t] = v;
            de = de - v;
        }
        de_c[t] = de;
    }
}

// ---------------------------------------------------------------------------
// Row numbering (1sub-momentum.F90:273-296): a fluid-list entry becomes a row
// unless it is air, solid, has zero porosity, or is a surface cell whose
// normal-side neighbour is solid.  Rows keep fluid-list order (an exclusive scan).
__device__ __forceinline__ bool row_kept(const GridIdx& g, int nnn, const int* __restrict__ mn,
                                         const int* __restrict__ in_, const int* __restrict__ jn,
                                         const int* __restrict__ kn, const int* __restrict__ nf,
                                         const int* __restrict__ nfb, const double* __restrict__ fb) {
    const int fl = nf[nnn];
    if (fl == 0 || fl == -1 || is_zero(fb[nnn])) return false;
    if (fl == 2) {
        const int b = nfb[nnn];
        const int l = (b < 0 ? -b : b) - 1;
        const int s = b >= 0 ? 1 : -1;
        // an orientation of 0 has no defined neighbour in the reference; kept
        if (l >= 0 && l <= 2 && nf[mn[g.nbr(in_[nnn], jn[nnn], kn[nnn], l, s)]] == -1) return false;
    }
    return true;
}

__global__ void __launch_bounds__(kBitThreads) k_row_flags(GridIdx g, int ifln, const int* __restrict__ fln,
                                                          const int* __restrict__ mn, const int* __restrict__ in_,
                                                          const int* __restrict__ jn, const int* __restrict__ kn,
                                                          const int* __restrict__ nf, const int* __restrict__ nfb,
                                                          const double* __restrict__ fb, unsigned* __restrict__ mask,
                                                          int* __restrict__ sums) {
    const int tile = blockIdx.x;
    int count = 0;
#pragma unroll
    for (int q = 0; q < kBitRounds; q++) {
        const long t = (long)tile * kBitTile + q * kBitThreads + threadIdx.x;
        const bool keep = t < ifln && row_kept(g, fln[t], mn, in_, jn, kn, nf, nfb, fb);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if ((threadIdx.x & 31) == 0) mask[t >> 5] = m;
        count += __popc(m);
    }
    __shared__ int s[kBitThreads / 32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kBitThreads / 32; w++) count += s[w];
        sums[tile] = count;
    }
}

// rows beyond mm2 are not written (the host reports them)
__global__ void __launch_bounds__(kBitThreads) k_row_scatter(GridIdx g, int ifln, int mm2, const int* __restrict__ fln,
                                                          const int* __restrict__ in_, const int* __restrict__ jn,
                                                          const int* __restrict__ kn, const unsigned* __restrict__ mask,
                                                          const int* __restrict__ sums, int* __restrict__ mno,
                                                          int* __restrict__ mno2mn) {
    __shared__ int pre[32];
    const int tile = blockIdx.x;
    const unsigned* words = mask + (long)tile * 32;
    if (threadIdx.x < 32) bit_prefix(words, pre);
    __syncthreads();
    const int first = sums[tile];
#pragma unroll
    for (int q = 0; q < kBitRounds; q++) {
        const int w = q * (kBitThreads / 32) + (threadIdx.x >> 5);
        const unsigned m = words[w], below = m & ((1u << (threadIdx.x & 31)) - 1);
        if (!(m >> (threadIdx.x & 31) & 1)) continue;
        const int nnn = fln[(long)tile * kBitTile + q * kBitThreads + threadIdx.x];
        const int row = first + pre[w] + __popc(below) + 1;       // 1-based row number
        if (row > mm2) continue;
        mno[g.mno_off(in_[nnn], kn[nnn], jn[nnn])] = row;
        mno2mn[row - 1] = nnn;                                    // mno2mn(row)
    }
}

// RHS of the fluid rows (1sub-momentum.F90:313-360) and dmax = max |DR1|, with renzoku_fv
// (lib/src/math_func.F90:51-54).  Nothing when there are fewer than 10 rows, or no
// room for the reference's 64 spare ones.
//
// What bounds it: seven FP64 divisions per row, on a pipe that does 1.7 lane operations
// per clock and SM, were most of its 460 us at 2.8 M rows (0.28 GB of traffic, 41 us).
// The divisors dx, dy, dz and dt are few: their reciprocals come from a table (dx: one
// per index and axis, in shared memory, TAB) and Markstein's method; 1 - f and its
// division by dt drop out where f is 1, the division by a porosity of 1 too, and the
// quotient that is only compared with 1e-15 is formed only near that bound: 199 us, the
// pipe 87 % busy, 20 of a row's 27 operations in the four exact quotients that are left.
template <bool TAB>
__global__ void __launch_bounds__(kAsmBlock, 3) k_rhs(GridIdx g, int mm2, const int* __restrict__ mnoe_p,
                                                  const int* __restrict__ mno2mn,
                                                  const int* __restrict__ mn, const int* __restrict__ in_,
                                                  const int* __restrict__ jn, const int* __restrict__ kn,
                                                  const int* __restrict__ nf, const double* __restrict__ f,
                                                  const double* __restrict__ fb, const double* __restrict__ a,
                                                  const double* __restrict__ un, const double* __restrict__ dx,
                                                  const double* __restrict__ mp_p, double dt,
                                                  double* __restrict__ b, unsigned long long* dmax_bits) {
    extern __shared__ double recip[];                   // 1 / dx(l, i), i = ls - 1 .. le + 1, axis after axis
    __shared__ long long s_max[kAsmBlock / 32];
    const int mnoe = *mnoe_p;
    if (mnoe < 10 || mnoe + 64 > mm2) return;
    const int nx = g.ie - g.is + 3, ny = g.je - g.js + 3, nz = g.ke - g.ks + 3;
    const int at[3] = {1 - g.is, nx + 1 - g.js, nx + ny + 1 - g.ks};
    if (TAB) {
        for (int t = threadIdx.x; t < nx + ny + nz; t += blockDim.x) {
            const int l = t < nx ? 0 : t < nx + ny ? 1 : 2;
            recip[t] = 1.0 / dx[g.dxo(l, t - at[l])];
        }
        __syncthreads();
    }
    const double mp = *mp_p;
    const bool forward = dt > 0.0;
    const Recip rdt = make_recip(dt);
    const long long near = __double_as_longlong(1.001e-15 * fabs(dt));
    long long local = 0;                                // bits of max |DR1|: they order like the values
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < mnoe; t += (long)gridDim.x * blockDim.x) {
        const int c = mno2mn[t];
        if (nf[c] != 1) continue;
        const int i = in_[c], j = jn[c], k = kn[c];
        const double fc = f[c], fbc = fb[c];
        double rz;
        if (!is_zero(fbc)) {
            const int ip = mn[g.mn_off(i + 1, k, j)], jp = mn[g.mn_off(i, k, j + 1)], kp = mn[g.mn_off(i, k + 1, j)];
            auto flux = [&](int cell, int l) {              // u a, with most faces fully open
                const double u = un[3L * cell + l], ar = a[3L * cell + l];
                return unless(is_one(ar), u, [&] { return u * ar; });
            };
            const double qx = flux(ip, 0) - flux(c, 0);
            const double qy = flux(jp, 1) - flux(c, 1);
            const double qz = flux(kp, 2) - flux(c, 2);
            if (TAB) {
                auto rec = [&](int l, int q) {
                    const double d = dx[g.dxo(l, q)];
                    return Recip{d, recip[at[l] + q], mid_exponent(d)};
                };
                rz = div_by(qx, rec(0, i)) + div_by(qy, rec(1, j)) + div_by(qz, rec(2, k));
            } else {
                rz = qx / dx[g.dxo(0, i)] + qy / dx[g.dxo(1, j)] + qz / dx[g.dxo(2, k)];
            }
            rz = unless(is_one(fbc), rz, [&] { return rz / fbc; });
        } else {
            rz = -10000.0;
        }
        double src = 0.0;
        if (!(is_one(fc) && forward)) src = div_by(fmax(-0.001, fmin(1.0 - fc, 0.001)), rdt);
        const double dr1 = rz + src;
        const long long ad = __double_as_longlong(fabs(dr1));
        bool put = true;
        if (!(ad > near)) {
            const double q = dr1 / dt;
            put = !(fabs(q) <= 1.0e-15 && fabs(q) != 0.0);
        }
        if (put) b[t] = div_by(mp * dr1, rdt);
        if (ad > local && ad <= 0x7ff0000000000000LL) local = ad;     // not a NaN
    }
    for (int o = 16; o > 0; o >>= 1) local = max(local, __shfl_xor_sync(0xffffffffu, local, o));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kAsmBlock / 32; w++) local = max(local, s_max[w]);
        if (local > 0) atomicMax(dmax_bits, (unsigned long long)local);
    }
}

// ---------------------------------------------------------------------------
// cal_matrix_element (1sub-momentum.F90:465-551), NORMAL build, one thread per
// fluid-list entry.  Latency-bound (three levels of dependent gathers per column), so
// the columns' loads are issued together, level by level: 229 us before, 133 now at 2.8 M rows.
template <int NL>
__global__ void __launch_bounds__(kAsmBlock, 4) k_assemble(GridIdx g, int ifln, long inne, long na, long spld,
                                                       const int* __restrict__ fln, const int* __restrict__ in_,
                                                       const int* __restrict__ jn, const int* __restrict__ kn,
                                                       const int* __restrict__ nf, const int* __restrict__ nfb,
                                                       const double* __restrict__ x, const double* __restrict__ dx,
                                                       const double* __restrict__ sp, const int* __restrict__ mno,
                                                       const double* __restrict__ alu_c, const int* __restrict__ ll_c,
                                                       const double* __restrict__ de_c, double* __restrict__ alu,
                                                       int* __restrict__ llu, double* __restrict__ de, int* err) {
    const double rate = -1.0e-20;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < ifln; t += (long)gridDim.x * blockDim.x) {
        const int nnn = fln[t];
        const int i = in_[nnn], j = jn[nnn], k = kn[nnn];
        const int fl = nf[nnn];
        int lc[NL], np[NL], fn[NL];
        double ac[NL];
#pragma unroll
        for (int c = 0; c < NL; c++) {
            lc[c] = nnn <= inne ? ll_c[c * inne + (nnn - 1)] : 0;
            ac[c] = nnn <= inne ? alu_c[c * inne + (nnn - 1)] : 0.0;
        }
        const int nn = mno[g.mno_off(i, k, j)];
        if (nn == 0) continue;
        const long r = nn - 1;
        double dd;
        if (fl == 1) {
            dd = de_c[nnn - 1];
        } else if (fl == 2) {
            dd = 1.0;
        } else {
            atomicCAS(err, 0, nnn);
            continue;
        }
#pragma unroll
        for (int c = 0; c < NL; c++) {
            fn[c] = 0;
            np[c] = 0;
            if (lc[c] != 0) {
                fn[c] = nf[lc[c]];
                np[c] = mno[g.mno_off(in_[lc[c]], kn[lc[c]], jn[lc[c]])];
            }
        }
        const int bl = nfb[nnn];
        const int axis = (bl < 0 ? -bl : bl) - 1;
#pragma unroll
        for (int c = 0; c < NL; c++) {
            const long o = c * na + r;
            if (lc[c] == 0 || fn[c] == 0 || np[c] == 0) {
                llu[o] = 0;
                alu[o] = 0.0;
                if (lc[c] != 0 && fl == 1 && fn[c] != 2) dd = dd + ac[c];
                continue;
            }
            llu[o] = np[c];
            if (fl == 1) {
                alu[o] = ac[c];
            } else {
                const int l = g.col_axis(c / 2);           // 2DV: past the collapsed axis (517-520)
                if (axis == l) {
                    const int ii = (l == 0) ? i : (l == 1) ? j : k;
                    const int md = (c + 1) % 2;
                    const double fss = (double)(1 - 2 * md) * (x[g.dxo(l, ii - md + 1)] - sp[nnn + spld * l]) / dx[g.dxo(l, ii)];
                    alu[o] = cal_alu(fss, dx[g.dxo(l, ii)], dx[g.dxo(l, ii - 2 * md + 1)]);
                } else {
                    alu[o] = rate;
                }
            }
        }
        de[r] = dd;
    }
}

// ---------------------------------------------------------------------------
// p(mno2mn(r)) -= xe(r)  (1sub-momentum.F90:53-58)
__global__ void k_pressure_update(int mnoe, const int* __restrict__ mno2mn, const double* __restrict__ xe0,
                                  double* __restrict__ p) {
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < mnoe; t += (long)gridDim.x * blockDim.x) {
        const int c = mno2mn[t];
        p[c] = p[c] - xe0[t + 1];
    }
}

// estimate_velocity2 (1sub-momentum.F90:590-651) with momentum_d
// (lib/src/math_func.F90:251-254); xe0 addresses xe(0).
__global__ void __launch_bounds__(kAsmBlock) k_velocity(GridIdx g, int inne, const int* __restrict__ mn,
                                                       const int* __restrict__ in_, const int* __restrict__ jn,
                                                       const int* __restrict__ kn, const int* __restrict__ nf,
                                                       const int* __restrict__ nfb, const double* __restrict__ a,
                                                       const double* __restrict__ dx, double dt,
                                                       const int* __restrict__ mno, const double* __restrict__ xe0,
                                                       double* __restrict__ un) {
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < inne; t += (long)gridDim.x * blockDim.x) {
        const int nn = (int)t + 1;
        const int fl = nf[nn];
        if (fl == 0) continue;
        if (fl == -1 && nfb[nn] != 4) continue;
        const int i = in_[nn], j = jn[nn], k = kn[nn];
        const int ic[3] = {i, j, k};
        const int nnn = mno[g.mno_off(i, k, j)];
        const double xec = -xe0[nnn];
        const int nno[3] = {mno[g.mno_off(i - 1, k, j)], mno[g.mno_off(i, k, j - 1)], mno[g.mno_off(i, k - 1, j)]};
        const int nnm[3] = {mn[g.mn_off(i - 1, k, j)], mn[g.mn_off(i, k, j - 1)], mn[g.mn_off(i, k - 1, j)]};
        if (fl == -1 && nfb[nn] == 4) {
            for (int l = 0; l < 3; l++) {
                if (nf[nnm[l]] >= 1) {
                    const double dxc = (dx[g.dxo(l, ic[l])] + dx[g.dxo(l, ic[l] - 1)]) * 0.5;
                    un[3L * nn + l] = un[3L * nn + l] + dt * (-xe0[nno[l]] - (-xe0[nnn])) / dxc;
                }
            }
        } else {
            for (int l = 0; l < 3; l++) {
                if (a[3L * nn + l] != 0.0) {
                    const double dxc = (dx[g.dxo(l, ic[l])] + dx[g.dxo(l, ic[l] - 1)]) * 0.5;
                    const int nfm = nf[nnm[l]];
                    if (nfm >= 1) {
                        double u = un[3L * nn + l] + dt * (-xe0[nno[l]] - xec) / dxc;
                        if (fabs(u) < 1.0e-15) u = 0.0;
                        un[3L * nn + l] = u;
                    } else if (nfm == -1 && nfb[nnm[l]] == 4) {
                        un[3L * nn + l] = un[3L * nn + l] + dt * (-xe0[nno[l]] - xec) / dxc;
                    }
                }
            }
        }
    }
}

}  // namespace clowns

using namespace clowns;

// ---------------------------------------------------------------------------
// C ABI

extern "C" int clowns_grid_nl(const int* dims) {
    if (!grid_dims_ok(dims) || !grid_has_matrix(dims)) return 0;
    return GridIdx::make(dims).nl();
}

extern "C" int clowns_init_matrix_dev(const int* dims, int inne, int mx2, const int* mn, const int* in_,
                                      const int* jn, const int* kn, const int* nf, const int* nfb,
                                      const double* a, const double* fb, const double* dx, double* mp,
                                      double* alu_c, int* ll_c, double* de_c, void* stream) {
    clowns::TraceRange trace_range_("clowns_init_matrix_dev");
    if (!grid_dims_ok(dims) || inne < 1 || mx2 < 1 || !mn || !in_ || !jn || !kn || !nf || !nfb || !a || !fb || !dx || !mp ||
        !alu_c || !ll_c || !de_c) {
        set_last_error_msg("init_matrix: invalid arguments");
        return CLOWNS_ERR_ARG;
    }
    if (!grid_has_matrix(dims)) {
        set_last_error_msg("init_matrix: a grid one cell wide in both x and y has no matrix form");
        return CLOWNS_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    GridIdx g = GridIdx::make(dims);
    // 2DV: x and z when one cell wide in y, y and z when one cell wide in x
    const int axes = g.ie == g.is + 1 ? 6 : g.je == g.js + 1 ? 5 : 7;
    k_min_dx<<<1, 256, 0, s>>>(dx, 3 * mx2, axes, mp);
    const int entries = (g.ie - g.is + 3) + (g.je - g.js + 3) + (g.ke - g.ks + 3);
    const size_t tab = sizeof(double) * 4 * (size_t)entries;
    auto launch = [&](auto kern, size_t smem) {
        const int block = smem ? kInitBlock : kInitPlainBlock;
        const int blocks = (int)std::min<long>((inne + block - 1L) / block, smem ? 152L : 152L * 16);
        kern<<<blocks, block, smem, s>>>(g, inne, mx2, mn, in_, jn, kn, nf, nfb, a, fb, dx, mp, alu_c, ll_c, de_c);
    };
    // the table fits the shared memory every launch may have up to 1536 cells in i + j + k
    if (tab <= 48 * 1024) {
        if (g.nl() == 6) launch(k_init_matrix<6, true>, tab);
        else launch(k_init_matrix<4, true>, tab);
    } else {
        if (g.nl() == 6) launch(k_init_matrix<6, false>, 0);
        else launch(k_init_matrix<4, false>, 0);
    }
    CLOWNS_CUDA_TRY(cudaGetLastError());
    return CLOWNS_OK;
}

namespace clowns {
// What the row and right-hand-side kernels hand to the host.
struct RowsOut {
    unsigned long long dmax_bits;
    int mnoe, pad;
};
}  // namespace clowns

// Workspace: the row mask (a word per 32 list entries, whole tiles), the tiles' counts
// and what goes to the host.
static size_t rows_tiles(int ifln) { return ((size_t)(ifln > 0 ? ifln : 1) + kBitTile - 1) / kBitTile; }

extern "C" size_t clowns_rows_rhs_workspace_bytes(int ifln) {
    return align_up(sizeof(unsigned) * 32 * rows_tiles(ifln), 256) + align_up(sizeof(int) * rows_tiles(ifln), 256) + 256;
}

extern "C" int clowns_rows_rhs_dev(const int* dims, int inne2, int mx2, const int* mn, const int* in_,
                                   const int* jn, const int* kn, const int* nf, const int* nfb, const double* f,
                                   const double* fb, const double* a, const double* un, const double* dx,
                                   const double* mp, double dt, int ifln, const int* fln, int mm2, int* mno,
                                   int* mno2mn, double* b, double* xe, double* de, int* mnoe_out,
                                   double* dmax_out, void* work, size_t work_bytes, void* stream) {
    clowns::TraceRange trace_range_("clowns_rows_rhs_dev");
    (void)inne2; (void)mx2;
    if (!grid_dims_ok(dims) || !mn || !in_ || !jn || !kn || !nf || !nfb || !f || !fb || !a || !un || !dx || !mp || !fln ||
        !mno || !mno2mn || !b || !xe || !de || !mnoe_out || ifln < 0 || mm2 < 1 || !work) {
        set_last_error_msg("rows_rhs: invalid arguments");
        return CLOWNS_ERR_ARG;
    }
    if (work_bytes < clowns_rows_rhs_workspace_bytes(ifln)) {
        set_last_error_msg("rows_rhs: workspace too small");
        return CLOWNS_ERR_WORKSPACE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    GridIdx g = GridIdx::make(dims);
    char* wb = (char*)work;
    unsigned* mask = (unsigned*)wb;
    wb += align_up(sizeof(unsigned) * 32 * rows_tiles(ifln), 256);
    int* sums = (int*)wb;
    wb += align_up(sizeof(int) * rows_tiles(ifln), 256);
    RowsOut* out = (RowsOut*)wb;
    // 1sub-momentum.F90:267-271 and 276
    CLOWNS_CUDA_TRY(cudaMemsetAsync(b, 0, sizeof(double) * mm2, s));
    CLOWNS_CUDA_TRY(cudaMemsetAsync(xe, 0, sizeof(double) * mm2, s));
    CLOWNS_CUDA_TRY(cudaMemsetAsync(de, 0, sizeof(double) * mm2, s));
    CLOWNS_CUDA_TRY(cudaMemsetAsync(mno, 0, sizeof(int) * (size_t)g.ie * g.ke * g.je, s));
    CLOWNS_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(RowsOut), s));
    if (ifln > 0) {
        // rows, right-hand side and their count in one pass over the stream: the kernels
        // take the count from the device, the host reads it with dmax at the end
        const int tiles = (int)rows_tiles(ifln);
        k_row_flags<<<tiles, kBitThreads, 0, s>>>(g, ifln, fln, mn, in_, jn, kn, nf, nfb, fb, mask, sums);
        int rc = scan_tiles_dev(1, sums, ifln, &out->mnoe, s);
        if (rc) return rc;
        k_row_scatter<<<tiles, kBitThreads, 0, s>>>(g, ifln, mm2, fln, in_, jn, kn, mask, sums, mno, mno2mn);
        // the reciprocals leave three blocks per SM their shared memory up to 3072 cells in i + j + k
        const int entries = (g.ie - g.is + 3) + (g.je - g.js + 3) + (g.ke - g.ks + 3);
        auto rhs = [&](auto kern, size_t smem, int nb) {
            kern<<<nb, kAsmBlock, smem, s>>>(g, mm2, &out->mnoe, mno2mn, mn, in_, jn, kn, nf, f, fb, a, un, dx, mp, dt, b,
                                             &out->dmax_bits);
        };
        if (entries <= 3072) rhs(k_rhs<true>, sizeof(double) * entries, std::min(grid_for(ifln), 152 * 3));
        else rhs(k_rhs<false>, 0, grid_for(ifln));
        CLOWNS_CUDA_TRY(cudaGetLastError());
    }
    RowsOut h = {};
    CLOWNS_CUDA_TRY(cudaMemcpyAsync(&h, out, sizeof(h), cudaMemcpyDeviceToHost, s));
    CLOWNS_CUDA_TRY(cudaStreamSynchronize(s));
    if (h.mnoe > mm2) {
        set_last_error_msg("rows_rhs: mm2 smaller than the number of rows");
        return CLOWNS_ERR_ARG;
    }
    *mnoe_out = h.mnoe;
    if (dmax_out) *dmax_out = 0.0;
    if (h.mnoe < 10) return CLOWNS_OK;              // 1sub-momentum.F90:297-300
    if (h.mnoe + 64 > mm2) {                        // the reference re-allocates (302-310)
        set_last_error_msg("rows_rhs: mm2 must exceed the number of rows by at least 64");
        return CLOWNS_ERR_ARG;
    }
    if (dmax_out) memcpy(dmax_out, &h.dmax_bits, sizeof(double));
    return CLOWNS_OK;
}

extern "C" int clowns_assemble_dev(const int* dims, int inne, int inne2, int mx2, const int* in_, const int* jn,
                                   const int* kn, const int* nf, const int* nfb, const double* x, const double* dx,
                                   const double* sp, int ifln, const int* fln, const int* mno, const double* alu_c,
                                   const int* ll_c, const double* de_c, int mm2, double* alu, int* llu, double* de,
                                   int* err_cell, void* stream) {
    clowns::TraceRange trace_range_("clowns_assemble_dev");
    (void)mx2;
    if (!grid_dims_ok(dims) || inne < 1 || !in_ || !jn || !kn || !nf || !nfb || !x || !dx || !sp || !fln || !mno || !alu_c ||
        !ll_c || !de_c || mm2 < 1 || !alu || !llu || !de || !err_cell) {
        set_last_error_msg("assemble: invalid arguments");
        return CLOWNS_ERR_ARG;
    }
    if (!grid_has_matrix(dims)) {
        set_last_error_msg("assemble: a grid one cell wide in both x and y has no matrix form");
        return CLOWNS_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    GridIdx g = GridIdx::make(dims);
    CLOWNS_CUDA_TRY(cudaMemsetAsync(err_cell, 0, sizeof(int), s));
    if (ifln > 0)
        (g.nl() == 6 ? k_assemble<6> : k_assemble<4>)<<<grid_for(ifln), kAsmBlock, 0, s>>>(
            g, ifln, inne, mm2, (long)inne2 + 2, fln, in_, jn, kn, nf, nfb, x, dx, sp, mno, alu_c, ll_c, de_c, alu, llu,
            de, err_cell);
    CLOWNS_CUDA_TRY(cudaGetLastError());
    return CLOWNS_OK;
}

extern "C" int clowns_correct_dev(const int* dims, int inne, int mx2, const int* mn, const int* in_, const int* jn,
                                  const int* kn, const int* nf, const int* nfb, const double* a, const double* dx,
                                  double dt, int mnoe, const int* mno2mn, const int* mno, const double* xe0,
                                  double* p, double* un, void* stream) {
    clowns::TraceRange trace_range_("clowns_correct_dev");
    (void)mx2;
    if (!grid_dims_ok(dims) || inne < 1 || !mn || !in_ || !jn || !kn || !nf || !nfb || !a || !dx || mnoe < 0 || !mno2mn ||
        !mno || !xe0 || !p || !un) {
        set_last_error_msg("correct: invalid arguments");
        return CLOWNS_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    GridIdx g = GridIdx::make(dims);
    if (mnoe > 0) k_pressure_update<<<grid_for(mnoe), kAsmBlock, 0, s>>>(mnoe, mno2mn, xe0, p);
    k_velocity<<<grid_for(inne), kAsmBlock, 0, s>>>(g, inne, mn, in_, jn, kn, nf, nfb, a, dx, dt, mno, xe0, un);
    CLOWNS_CUDA_TRY(cudaGetLastError());
    return CLOWNS_OK;
}
