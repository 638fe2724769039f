// nflag.cu -- cell classification set_nflag (src2LOWNS/nfd2015.F90:7-306) on the
// GPU, NORMAL + OBJECT build.
//
// The reference is a sequence of passes over the cells, restarted whenever a
// pass removes a surface cell (goto 4 / goto 3).  Three of its loops write flags
// that later iterations of the same loop read (the second pruning loop and the
// orientation loop, nfd2015.F90:133-158 and 163-244, walked in descending list
// order).  Their serial semantics are reproduced exactly here: the decision for
// list position p depends only on decisions at positions > p, so a Jacobi
// iteration over all positions reaches the serial answer after at most
// (longest dependency chain + 1) sweeps and is detected as a fixed point.
#include <cstring>

#include "common.cuh"
#include "grid_index.cuh"
#include "trace.h"

namespace clowns {

constexpr int kNfBlock = 256;

static inline int nf_grid(long n) {
    long b = (n + kNfBlock - 1) / kNfBlock;
    if (b < 1) b = 1;
    if (b > 152L * 16) b = 152L * 16;
    return (int)b;
}

struct NfArgs {
    GridIdx g;
    int inne;
    const int* mn;
    const int* in_;
    const int* jn;
    const int* kn;
    int* nf;
    int* nfb;
    const double* fb;
    const double* a;
    const double* dx;
    const int* objno;
};

// ---- nfd2015.F90:35-59 --------------------------------------------------
// imax_k: the largest i and k of a wet cell, one pair of atomics per block.
__global__ void __launch_bounds__(kNfBlock) k_vof_flags(NfArgs A, const double* __restrict__ f, int* __restrict__ dec,
                                                        int* imax_k) {
    int mi = 0, mk = 0;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < A.inne; t += (long)gridDim.x * blockDim.x) {
        const int nn = (int)t + 1;
        if (A.nf[nn] == -1) { dec[nn] = -1; continue; }
        const int i = A.in_[nn], k = A.kn[nn];
        const double fv = f[nn];
        bool air = fv <= 1.0e-12;
        if (!air && fv * A.fb[nn] < 1.0e-3) {
            const int j = A.jn[nn];
            air = A.nf[A.mn[A.g.mn_off(i, k - 1, j)]] == -1 && f[A.mn[A.g.mn_off(i, k + 1, j)]] == 0.0;
        }
        dec[nn] = air ? 0 : 1;
        if (!air) {
            mi = max(mi, i);
            mk = max(mk, k);
        }
    }
    __shared__ int s[2];
    if (threadIdx.x < 2) s[threadIdx.x] = 0;
    __syncthreads();
    mi = __reduce_max_sync(0xffffffffu, mi);
    mk = __reduce_max_sync(0xffffffffu, mk);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(s, mi);
        atomicMax(s + 1, mk);
    }
    __syncthreads();
    if (threadIdx.x < 2 && s[threadIdx.x] > 0) atomicMax(imax_k + threadIdx.x, s[threadIdx.x]);
}

__global__ void k_vof_apply(NfArgs A, double* __restrict__ f, const int* __restrict__ dec) {
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < A.inne; t += (long)gridDim.x * blockDim.x) {
        const int nn = (int)t + 1;
        const int d = dec[nn];
        if (d < 0) continue;
        A.nf[nn] = d;
        A.nfb[nn] = 0;
        if (d == 0) f[nn] = fmax(0.0, f[nn]);
    }
}

// Counters shared by the passes, on the device (zeroed before each classification).
enum { kCtrImax, kCtrKmax, kCtrWet, kCtrSurf, kCtrUnsettled, kCtrPrune, kCtrSweep, kCtrRemoved, kCtrDropped, kCtrCount };

// ---- nfd2015.F90:66-102: wet cells and surface detection over the k,j,i box, whose
// upper corner follows from the wet cells' largest i and k (kept on the device: the
// host launches for the largest box, and blocks past the box's tiles return)
struct Box {
    int is, js, ks, ni, nj;
    long total;
    __device__ __forceinline__ Box(const GridIdx& g, const int* ctr) {
        const int imax = min(ctr[kCtrImax] + 1, g.ie - 1), kmax = min(ctr[kCtrKmax] + 1, g.ke - 1);
        is = g.is; js = g.js; ks = g.ks;
        ni = max(0, imax - g.is + 1);
        nj = g.je - g.js;
        total = (long)ni * nj * max(0, kmax - g.ks + 1);
    }
    __device__ __forceinline__ void ijk(unsigned t, int& i, int& j, int& k) const {
        const unsigned r = t / (unsigned)ni;
        i = is + (int)(t - r * (unsigned)ni);
        k = ks + (int)(r / (unsigned)nj);
        j = js + (int)(r % (unsigned)nj);
    }
};

// Bit masks of the wet and the surface cells, their counts per tile (pairs).
__global__ void __launch_bounds__(kBitThreads) k_surface_flags(NfArgs A, const int* __restrict__ ctr,
                                                               unsigned* __restrict__ wet, unsigned* __restrict__ surf,
                                                               int* __restrict__ sums) {
    const Box B(A.g, ctr);
    const int tile = blockIdx.x;
    if ((long)tile * kBitTile >= B.total) {
        if (threadIdx.x < 2) sums[2 * tile + threadIdx.x] = 0;
        return;
    }
    int cw = 0, cs = 0;
#pragma unroll
    for (int q = 0; q < kBitRounds; q++) {
        const long t = (long)tile * kBitTile + q * kBitThreads + threadIdx.x;
        bool w = false, s = false;
        if (t < B.total) {
            int i, j, k;
            B.ijk((unsigned)t, i, j, k);
            const int nn = A.mn[A.g.mn_off(i, k, j)];
            w = A.nf[nn] >= 1;
            if (w) {
                for (int l = 0; l < 3 && !s; l++) {
                    const int p = A.mn[A.g.nbr(i, j, k, l, +1)];
                    if (A.nf[p] == 0 && A.a[3L * p + l] > 0.0) s = true;
                    if (!s) {
                        const int m = A.mn[A.g.nbr(i, j, k, l, -1)];
                        if (A.nf[m] == 0 && A.a[3L * nn + l] > 0.0) s = true;
                    }
                }
            }
        }
        const unsigned mw = __ballot_sync(0xffffffffu, w), ms = __ballot_sync(0xffffffffu, s);
        if ((threadIdx.x & 31) == 0) {
            wet[t >> 5] = mw;
            surf[t >> 5] = ms;
        }
        cw += __popc(mw);
        cs += __popc(ms);
    }
    __shared__ int sum[2];
    if (threadIdx.x < 2) sum[threadIdx.x] = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(sum, cw);
        atomicAdd(sum + 1, cs);
    }
    __syncthreads();
    if (threadIdx.x < 2) sums[2 * tile + threadIdx.x] = sum[threadIdx.x];
}

__global__ void __launch_bounds__(kBitThreads) k_surface_scatter(NfArgs A, const int* __restrict__ ctr,
                                                                 const unsigned* __restrict__ wet,
                                                                 const unsigned* __restrict__ surf,
                                                                 const int* __restrict__ sums, int* __restrict__ fln,
                                                                 int* __restrict__ sfn, int* __restrict__ spos_cell) {
    const Box B(A.g, ctr);
    const int tile = blockIdx.x;
    if ((long)tile * kBitTile >= B.total) return;
    __shared__ int prew[32], pres[32];
    const unsigned *ww = wet + (long)tile * 32, *sw = surf + (long)tile * 32;
    if (threadIdx.x < 32) bit_prefix(ww, prew);
    else if (threadIdx.x < 64) bit_prefix(sw, pres);
    __syncthreads();
    const int w0 = sums[2 * tile], s0 = sums[2 * tile + 1];
#pragma unroll
    for (int q = 0; q < kBitRounds; q++) {
        const int word = q * (kBitThreads / 32) + (threadIdx.x >> 5), bit = threadIdx.x & 31;
        const unsigned mw = ww[word], ms = sw[word], below = (1u << bit) - 1;
        if (!(mw >> bit & 1)) continue;
        int i, j, k;
        B.ijk((unsigned)((long)tile * kBitTile + q * kBitThreads + threadIdx.x), i, j, k);
        const int nn = A.mn[A.g.mn_off(i, k, j)];
        fln[w0 + prew[word] + __popc(mw & below)] = nn;
        if (ms >> bit & 1) {
            const int p = s0 + pres[word] + __popc(ms & below);
            sfn[p] = nn;
            spos_cell[nn] = p;
            A.nf[nn] = 2;
            A.nfb[nn] = -3;
        } else {
            A.nf[nn] = 1;
            spos_cell[nn] = -1;
        }
    }
}

// ---- nfd2015.F90:107-131: first pruning (order-independent) -------------------
__device__ __forceinline__ int prune1(const NfArgs& A, int nn) {
    const int i = A.in_[nn], j = A.jn[nn], k = A.kn[nn];
    if (A.nf[A.mn[A.g.mn_off(i, k - 1, j)]] == -1) return 0;
    int keep = 0;
    for (int l = 0; l < 3 && !keep; l++) {
        if (A.nf[A.mn[A.g.nbr(i, j, k, l, +1)]] == 1) keep = 1;
        else if (A.nf[A.mn[A.g.nbr(i, j, k, l, -1)]] == 1) keep = 1;
    }
    return !keep;
}
__global__ void k_prune1(NfArgs A, int isfn, const int* __restrict__ sfn, int* __restrict__ rem, int* count) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < isfn; p += (long)gridDim.x * blockDim.x) {
        const int r = prune1(A, sfn[p]);
        rem[p] = r;
        if (r) atomicAdd(count, 1);
    }
}

__global__ void k_remove(NfArgs A, int isfn, const int* __restrict__ sfn, const int* __restrict__ rem) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < isfn; p += (long)gridDim.x * blockDim.x) {
        if (rem[p]) {
            const int nn = sfn[p];
            A.nf[nn] = 0;
            A.nfb[nn] = 0;
        }
    }
}

// Flag of cell q as seen by list position p in a loop walked from the end of
// the list: cells later in the list (already visited) show their removal.
// state == nullptr: nothing removed.
__device__ __forceinline__ int nf_seen(const NfArgs& A, int q, long p, const int* __restrict__ spos_cell,
                                       const int* __restrict__ state) {
    const int fl = A.nf[q];
    if (fl == 2 && state) {
        const int pq = spos_cell[q];
        if (pq > p && state[pq]) return 0;
    }
    return fl;
}

// ---- nfd2015.F90:133-158: second pruning, serial semantics ---------------------
__device__ __forceinline__ int prune2(const NfArgs& A, int nn, long p, const int* __restrict__ spos_cell,
                                      const int* __restrict__ st) {
    const int i = A.in_[nn], j = A.jn[nn], k = A.kn[nn];
    const int below = nf_seen(A, A.mn[A.g.mn_off(i, k - 1, j)], p, spos_cell, st);
    const int above = nf_seen(A, A.mn[A.g.mn_off(i, k + 1, j)], p, spos_cell, st);
    if (below == -1 && above == 0) return 0;
    int keep = 0;
    for (int l = 0; l < 3 && !keep; l++) {
        const int pv = nf_seen(A, A.mn[A.g.nbr(i, j, k, l, +1)], p, spos_cell, st);
        const int mv = nf_seen(A, A.mn[A.g.nbr(i, j, k, l, -1)], p, spos_cell, st);
        if ((pv == 1 && mv == 0) || (mv == 1 && pv == 0)) keep = 1;
    }
    return !keep;
}
__global__ void k_prune2_sweep(NfArgs A, int isfn, const int* __restrict__ sfn, const int* __restrict__ spos_cell,
                               const int* __restrict__ st_in, int* __restrict__ st_out, int* changed) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < isfn; p += (long)gridDim.x * blockDim.x) {
        const int r = prune2(A, sfn[p], p, spos_cell, st_in);
        st_out[p] = r;
        if (r != st_in[p]) atomicAdd(changed, 1);
    }
}

// fxx1 (nfd2015.F90:308-332)
__device__ double fxx1_dev(const NfArgs& A, const double* __restrict__ f, int ix, int ll, int i, int j, int k) {
    const GridIdx& g = A.g;
    const int lg[3] = {i, j, k};
    double r = 0.0;
    for (int l = 0; l <= 2; l++) {
        if (l == ll) continue;
        if (g.is == g.ie - 1 && l == 0) continue;
        if (g.js == g.je - 1 && l == 1) continue;
        for (int ii = -1; ii <= 1; ii++) {
            const int ci = lg[0] + ix * (ll == 0) + ii * (l == 0);
            const int ck = lg[2] + ix * (ll == 2) + ii * (l == 2);
            const int cj = lg[1] + ix * (ll == 1) + ii * (l == 1);
            const int nnc = A.mn[g.mn_off(ci, ck, cj)];
            r = __dadd_rn(r, __dmul_rn(__dmul_rn(A.dx[g.dxo(l, lg[l] + ii)], f[nnc]), A.fb[nnc]));
        }
        for (int lll = 0; lll <= 2; lll++) {
            if (lll == l || ll == lll) continue;
            r = __dmul_rn(r, A.dx[g.dxo(lll, lg[lll])]);
        }
    }
    return __dmul_rn(r, A.dx[g.dxo(ll, lg[ll] + ix)]);
}

// ---- nfd2015.F90:163-244: orientation, serial semantics ------------------------
// Orientation b of list position p; true when the cell has none and becomes air.
__device__ __forceinline__ bool orient(const NfArgs& A, const double* __restrict__ f, int nn, long p,
                                       const int* __restrict__ spos_cell, const int* __restrict__ st_in, int& b) {
    const int i = A.in_[nn], j = A.jn[nn], k = A.kn[nn];
    int ix[3] = {0, 0, 0};
    for (int l = 0; l < 3; l++) {
        const int m = A.mn[A.g.nbr(i, j, k, l, -1)], pc = A.mn[A.g.nbr(i, j, k, l, +1)];
        const int mv = nf_seen(A, m, p, spos_cell, st_in), pv = nf_seen(A, pc, p, spos_cell, st_in);
        if (mv == 1 && pv == 0 && A.a[3L * pc + l] > 0.0) ix[l] = -1;
        else if (mv == 0 && pv == 1 && A.a[3L * nn + l] > 0.0) ix[l] = 1;
    }
    if (abs(ix[0]) + abs(ix[1]) + abs(ix[2]) == 0) {
        const int below = nf_seen(A, A.mn[A.g.mn_off(i, k - 1, j)], p, spos_cell, st_in);
        const int above = nf_seen(A, A.mn[A.g.mn_off(i, k + 1, j)], p, spos_cell, st_in);
        if (below == -1 && above == 0) {
            if (A.objno[nn] != 0 || A.fb[nn] != 0.0) {
                ix[2] = -1;
            } else {
                for (int l = 0; l <= 1; l++) {
                    const int m = A.mn[A.g.nbr(i, j, k, l, -1)], pc = A.mn[A.g.nbr(i, j, k, l, +1)];
                    const int mv = nf_seen(A, m, p, spos_cell, st_in), pv = nf_seen(A, pc, p, spos_cell, st_in);
                    if (mv > 0 && pv == 0 && A.a[3L * pc + l] > 0.0) ix[l] = -1;
                    else if (mv == 0 && pv > 0 && A.a[3L * nn + l] > 0.0) ix[l] = 1;
                }
                if (abs(ix[0]) + abs(ix[1]) == 0) ix[2] = -1;
            }
        }
    }
    const int s = abs(ix[0]) + abs(ix[1]) + abs(ix[2]);
    int g = 0;
    b = 0;
    if (s == 1) {
        int dir = 1, best = abs(ix[0]);
        for (int l = 1; l <= 2; l++)
            if (abs(ix[l]) > best) { best = abs(ix[l]); dir = l + 1; }
        b = dir * ix[dir - 1];
    } else if (s == 0) {
        g = 1;
    } else {
        double fx[3];
        for (int l = 0; l < 3; l++) fx[l] = ix[l] == 0 ? 0.0 : fxx1_dev(A, f, ix[l], l, i, j, k);
        int dir = 1;
        double best = fx[0];
        for (int l = 1; l <= 2; l++)
            if (fx[l] > best) { best = fx[l]; dir = l + 1; }
        b = dir * ix[dir - 1];
    }
    return g != 0;
}
__global__ void k_orient_sweep(NfArgs A, const double* __restrict__ f, int isfn, const int* __restrict__ sfn,
                               const int* __restrict__ spos_cell, const int* __restrict__ st_in,
                               int* __restrict__ st_out, int* __restrict__ bout, int* changed) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < isfn; p += (long)gridDim.x * blockDim.x) {
        int b;
        const int g = orient(A, f, sfn[p], p, spos_cell, st_in, b);
        st_out[p] = g;
        bout[p] = b;
        if (g != st_in[p]) atomicAdd(changed, 1);
    }
}

// The three loops at once for a surface that none of them changes, the usual case:
// the first pruning removes nothing, and a first sweep of the second and of the
// orientation from "nothing removed" finds nothing to remove either, so each has
// settled.  ctr[kCtrUnsettled] counts the positions where that fails; they leave all
// flags as they were and the loops run one by one.
__global__ void k_surface_check(NfArgs A, const double* __restrict__ f, const int* __restrict__ sfn,
                                const int* __restrict__ spos_cell, int* __restrict__ bout, int* ctr) {
    const int isfn = ctr[kCtrSurf];
    int bad = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < isfn; p += gridDim.x * blockDim.x) {
        const int nn = sfn[p];
        int b = 0;
        bad |= prune1(A, nn) || prune2(A, nn, p, spos_cell, nullptr) || orient(A, f, nn, p, spos_cell, nullptr, b);
        bout[p] = b;
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicAdd(ctr + kCtrUnsettled, 1);
}
__global__ void k_surface_settle(NfArgs A, const int* __restrict__ sfn, const int* __restrict__ bout,
                                 const int* __restrict__ ctr) {
    if (ctr[kCtrUnsettled]) return;
    const int isfn = ctr[kCtrSurf];
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < isfn; p += gridDim.x * blockDim.x) A.nfb[sfn[p]] = bout[p];
}

__global__ void k_orient_apply(NfArgs A, int isfn, const int* __restrict__ sfn, const int* __restrict__ st,
                               const int* __restrict__ b, int* count) {
    for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < isfn; p += (long)gridDim.x * blockDim.x) {
        const int nn = sfn[p];
        A.nfb[nn] = b[p];
        if (st[p]) {
            A.nf[nn] = 0;
            atomicAdd(count, 1);
        }
    }
}

__global__ void k_count_nonzero(const int* __restrict__ v, long n, int* count) {
    int c = 0;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) c += v[t] != 0;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

__global__ void k_fill(int* p, long n, int v) {
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) p[t] = v;
}

// The joint check is tried again after a pass that dropped few cells of a surface only:
// after one that dropped many the next pass seldom settles, and the loops repeat the
// check's work.  It costs about 0.15 us per 1000 positions and saves some 80 us of
// launches and read-backs where it holds.  us, checked in every pass / by this rule /
// never after a change: 225 / 225 / 315 at 402 positions in 2 passes, 755 / 760 / 835 at 67 k
// in 4, 3050 / 2710 / 2690 at 252 k in 12, 16700 / 10900 / 9700 at 937 k in 35 (the
// separate loops before there was a check: 380, 1200, 3480, 11400).
constexpr int kCheckDropped = 64;
constexpr long kCheckWork = 4000000;                 // cells dropped x positions

// Workspace: the wet and surface masks with their tiles' counts, the per-cell list
// position and the per-position states of the surface loops.
struct NfWs {
    unsigned *wet, *surf;
    int *sums, *spos_cell, *st0, *st1, *bout, *ctr;
};

static size_t nf_box(const int* dims) {
    const GridIdx g = GridIdx::make(dims);
    const long box = (long)(g.ie - g.is) * (g.je - g.js) * (g.ke - g.ks);
    return box < 1 ? 1 : (size_t)box;
}
static size_t nf_tiles(const int* dims) { return (nf_box(dims) + kBitTile - 1) / kBitTile; }

static size_t nf_layout(const int* dims, int inne2, NfWs* w, char* base) {
    const size_t box = nf_box(dims), tiles = nf_tiles(dims);
    size_t o = 0;
    auto take = [&](size_t bytes) { size_t at = o; o = align_up(o + bytes, 256); return at; };
    const size_t o_wet = take(sizeof(unsigned) * 32 * tiles);
    const size_t o_surf = take(sizeof(unsigned) * 32 * tiles);
    const size_t o_sums = take(sizeof(int) * 2 * tiles);
    const size_t o_cell = take(sizeof(int) * ((size_t)inne2 + 2));
    const size_t o_st0 = take(sizeof(int) * box);
    const size_t o_st1 = take(sizeof(int) * box);
    const size_t o_b = take(sizeof(int) * box);
    const size_t o_ctr = take(sizeof(int) * 16);
    if (w && base) {
        w->wet = (unsigned*)(base + o_wet);
        w->surf = (unsigned*)(base + o_surf);
        w->sums = (int*)(base + o_sums);
        w->spos_cell = (int*)(base + o_cell);
        w->st0 = (int*)(base + o_st0);
        w->st1 = (int*)(base + o_st1);
        w->bout = (int*)(base + o_b);
        w->ctr = (int*)(base + o_ctr);
    }
    return o;
}

static int read_int(const int* dptr, cudaStream_t s, int* out) {
    CLOWNS_CUDA_TRY(cudaMemcpyAsync(out, dptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    CLOWNS_CUDA_TRY(cudaStreamSynchronize(s));
    return CLOWNS_OK;
}

}  // namespace clowns

using namespace clowns;

extern "C" size_t clowns_set_nflag_workspace_bytes(const int* dims, int inne2) {
    if (!dims) return 0;
    return nf_layout(dims, inne2, nullptr, nullptr);
}

extern "C" int clowns_set_nflag_dev(const int* dims, int inne, int inne2, int mx2, const int* mn, const int* in_,
                                    const int* jn, const int* kn, int* nf, int* nfb, double* f, const double* fb,
                                    const double* a, const double* dx, const int* objno, int* fln, int* ifln_out,
                                    int* sfn, int* isfn_out, int* passes_out, void* work, size_t work_bytes,
                                    void* stream) {
    clowns::TraceRange trace_range_("clowns_set_nflag_dev");
    (void)mx2;
    if (!grid_dims_ok(dims) || inne < 1 || !mn || !in_ || !jn || !kn || !nf || !nfb || !f || !fb || !a || !dx || !objno ||
        !fln || !ifln_out || !sfn || !isfn_out || !work) {
        set_last_error_msg("set_nflag: invalid arguments");
        return CLOWNS_ERR_ARG;
    }
    if (work_bytes < nf_layout(dims, inne2, nullptr, nullptr)) {
        set_last_error_msg("set_nflag: workspace too small");
        return CLOWNS_ERR_WORKSPACE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    NfWs W;
    nf_layout(dims, inne2, &W, (char*)work);
    NfArgs A;
    A.g = GridIdx::make(dims);
    A.inne = inne;
    A.mn = mn; A.in_ = in_; A.jn = jn; A.kn = kn; A.nf = nf; A.nfb = nfb;
    A.fb = fb; A.a = a; A.dx = dx; A.objno = objno;

    // VOF pass (spos_cell holds the per-cell decisions until the lists are numbered)
    CLOWNS_CUDA_TRY(cudaMemsetAsync(W.ctr, 0, sizeof(int) * 16, s));
    k_vof_flags<<<nf_grid(inne), kNfBlock, 0, s>>>(A, f, W.spos_cell, W.ctr);
    k_vof_apply<<<nf_grid(inne), kNfBlock, 0, s>>>(A, f, W.spos_cell);
    const int tiles = (int)nf_tiles(dims);

    int passes = 0, ifln = 0, isfn = 0;
    int dropped = 0;                        // by the pass before
    const int kMaxPasses = 100000;
    for (;;) {
        if (++passes > kMaxPasses) {
            set_last_error_msg("set_nflag: classification did not settle");
            return CLOWNS_ERR_NOCONV;
        }
        // the lists, and the surface loops as far as they change nothing, with one read-back
        CLOWNS_CUDA_TRY(cudaMemsetAsync(W.ctr + kCtrUnsettled, 0, sizeof(int), s));
        k_surface_flags<<<tiles, kBitThreads, 0, s>>>(A, W.ctr, W.wet, W.surf, W.sums);
        int rc = scan_tiles_dev(2, W.sums, (long)nf_box(dims), W.ctr + kCtrWet, s);
        if (rc) return rc;
        k_surface_scatter<<<tiles, kBitThreads, 0, s>>>(A, W.ctr, W.wet, W.surf, W.sums, fln, sfn, W.spos_cell);
        const bool check = dropped <= kCheckDropped && (long)dropped * isfn <= kCheckWork;
        if (check) {
            k_surface_check<<<152 * 4, kNfBlock, 0, s>>>(A, f, sfn, W.spos_cell, W.bout, W.ctr);
            k_surface_settle<<<152 * 4, kNfBlock, 0, s>>>(A, sfn, W.bout, W.ctr);
        }
        int h[kCtrUnsettled + 1];
        CLOWNS_CUDA_TRY(cudaMemcpyAsync(h, W.ctr, sizeof(h), cudaMemcpyDeviceToHost, s));
        CLOWNS_CUDA_TRY(cudaStreamSynchronize(s));
        ifln = h[kCtrWet];
        isfn = h[kCtrSurf];
        if (isfn == 0 || (check && !h[kCtrUnsettled])) break;
        const int gs = nf_grid(isfn);
        // first pruning
        CLOWNS_CUDA_TRY(cudaMemsetAsync(W.ctr + kCtrPrune, 0, sizeof(int), s));
        k_prune1<<<gs, kNfBlock, 0, s>>>(A, isfn, sfn, W.st0, W.ctr + kCtrPrune);
        int removed = 0;
        rc = read_int(W.ctr + kCtrPrune, s, &removed);
        if (rc) return rc;
        dropped = removed;
        if (removed) {
            k_remove<<<gs, kNfBlock, 0, s>>>(A, isfn, sfn, W.st0);
            continue;
        }
        // second pruning: Jacobi to the serial fixed point
        k_fill<<<gs, kNfBlock, 0, s>>>(W.st0, isfn, 0);
        int* cur = W.st0;
        int* nxt = W.st1;
        bool settled = false;
        for (int sweep = 0; sweep <= isfn + 1; sweep++) {
            CLOWNS_CUDA_TRY(cudaMemsetAsync(W.ctr + kCtrSweep, 0, sizeof(int), s));
            k_prune2_sweep<<<gs, kNfBlock, 0, s>>>(A, isfn, sfn, W.spos_cell, cur, nxt, W.ctr + kCtrSweep);
            int changed = 0;
            rc = read_int(W.ctr + kCtrSweep, s, &changed);
            if (rc) return rc;
            int* tmp = cur; cur = nxt; nxt = tmp;
            if (!changed) { settled = true; break; }
        }
        if (!settled) {
            set_last_error_msg("set_nflag: second pruning did not settle");
            return CLOWNS_ERR_NOCONV;
        }
        // apply the removals of the settled state
        CLOWNS_CUDA_TRY(cudaMemsetAsync(W.ctr + kCtrRemoved, 0, sizeof(int), s));
        k_count_nonzero<<<gs, kNfBlock, 0, s>>>(cur, isfn, W.ctr + kCtrRemoved);
        k_remove<<<gs, kNfBlock, 0, s>>>(A, isfn, sfn, cur);
        int removed2 = 0;
        rc = read_int(W.ctr + kCtrRemoved, s, &removed2);
        if (rc) return rc;
        dropped = removed2;
        if (removed2) continue;
        // orientation: Jacobi to the serial fixed point
        k_fill<<<gs, kNfBlock, 0, s>>>(W.st0, isfn, 0);
        cur = W.st0;
        nxt = W.st1;
        settled = false;
        for (int sweep = 0; sweep <= isfn + 1; sweep++) {
            CLOWNS_CUDA_TRY(cudaMemsetAsync(W.ctr + kCtrSweep, 0, sizeof(int), s));
            k_orient_sweep<<<gs, kNfBlock, 0, s>>>(A, f, isfn, sfn, W.spos_cell, cur, nxt, W.bout, W.ctr + kCtrSweep);
            int changed = 0;
            rc = read_int(W.ctr + kCtrSweep, s, &changed);
            if (rc) return rc;
            int* tmp = cur; cur = nxt; nxt = tmp;
            if (!changed) { settled = true; break; }
        }
        if (!settled) {
            set_last_error_msg("set_nflag: orientation did not settle");
            return CLOWNS_ERR_NOCONV;
        }
        CLOWNS_CUDA_TRY(cudaMemsetAsync(W.ctr + kCtrDropped, 0, sizeof(int), s));
        k_orient_apply<<<gs, kNfBlock, 0, s>>>(A, isfn, sfn, cur, W.bout, W.ctr + kCtrDropped);
        int igai = 0;
        rc = read_int(W.ctr + kCtrDropped, s, &igai);
        if (rc) return rc;
        dropped = igai;
        if (igai) continue;
        break;
    }
    CLOWNS_CUDA_TRY(cudaGetLastError());
    CLOWNS_CUDA_TRY(cudaStreamSynchronize(s));
    *ifln_out = ifln;
    *isfn_out = isfn;
    if (passes_out) *passes_out = passes;
    return CLOWNS_OK;
}
