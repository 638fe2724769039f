// resident.cuh -- the iteration loop of small and medium systems as ONE resident
// kernel whose blocks exchange vectors through self-validating words.
//
// Below about half a million rows an iteration of the kernel-per-phase loop is
// bound by its kernel boundaries, not by its work: 12 kernels of about 4 us each
// at 4 k rows (0.3 us of FP64 arithmetic) and still 5-7 us each at 0.4 M rows.
// Here one cooperative launch (at most one block per SM, member rows dealt to
// the blocks in 128-row chunks) runs every iteration, and nothing in it is a
// grid-wide barrier:
//   - a vector that other rows gather (p, e, and the operator's intermediates)
//     is stored as {value, epoch} words written and read with single relaxed
//     accesses (16 bytes in FP64, 8 in FP32).  A reader polls the words it
//     gathers until they carry this step's epoch: data and signal travel
//     together, so a step costs one store-to-load trip through L2 instead of
//     stores, a fence, a flag, a wait and then the loads;
//   - chunk totals of the dot products travel the same way, and every block sums
//     them itself along the canonical tree (engine.cuh), so every block holds
//     the same scalars and takes the same stop decisions;
//   - LDUSUB's sweeps run in two steps instead of five: 1-2-3 and 4-5-6 (four
//     columns: 1-2 and 3-4).  A row re-evaluates the one or two levels of its
//     neighbours' sweeps it needs from coefficients composed once per solve
//     (k_res_compose), with the same fused multiply-adds, so the bits are those of
//     separate sweeps.  That costs 12 more operations per row and iteration and
//     saves six trips.
// A word is overwritten only after a reduction of the same iteration that every
// reader's own contribution had to precede, so no reader can miss its epoch:
// the operator's intermediates are rewritten once per reduction RQ / AMU, p and
// e once per iteration, and each of the three reductions has its own totals.
// Every poll is bounded: a warp that runs out raises the abort flag, polls of
// the other warps and blocks then give up too, and the block leaves at the next
// reduction; the host reports the failure.
#pragma once

#include <type_traits>

#include "engine.cuh"

namespace clowns {

constexpr int kResThreads = 768;                 // 24 warps: 80 registers per thread
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxGroups = 512;               // reduction groups of one member (4.2 M rows)

// Coefficients and indices of one 32-row group in the resident loop's layout:
// group-major, each a run of 32 lanes, so that one address and constant offsets
// reach all of a row's.  With c1..c6 the row's columns in sweep order:
//   slots 0..5 AL(1..6) / LL(1..6);
//   six columns   6: sweep 2 at c3   7: sweep 1 at c3   8: sweep 1 at c2
//                 9: sweep 1 at c2(c3)   10: sweep 4 at c5   11: sweep 4 at c6
//   four columns  4: sweep 1 at c2   5: sweep 3 at c4
//   last coefficient: D
template <int NL>
constexpr int kResIdx = NL == 6 ? 12 : 6;
template <int NL>
constexpr int kResCoef = kResIdx<NL> + 1;

template <typename T>
struct TagOf;
template <>
struct TagOf<double> {
    struct __align__(16) Word { unsigned long long v, tag; };
};
template <>
struct TagOf<float> {
    struct __align__(8) Word { unsigned v, tag; };
};
template <typename T>
using TagWord = typename TagOf<T>::Word;

__device__ __forceinline__ void tag_put(TagWord<double>* p, double v, unsigned tag) {
    asm volatile(
        "{\n .reg .b128 w;\n .reg .b64 t;\n cvt.u64.u32 t, %2;\n mov.b128 w, {%1, t};\n"
        " st.relaxed.gpu.global.b128 [%0], w;\n}" ::"l"(p),
        "l"(__double_as_longlong(v)), "r"(tag)
        : "memory");
}
__device__ __forceinline__ unsigned tag_get(const TagWord<double>* p, double& v) {
    unsigned long long b, t;
    asm volatile("{\n .reg .b128 w;\n ld.relaxed.gpu.global.b128 w, [%2];\n mov.b128 {%0, %1}, w;\n}"
                 : "=l"(b), "=l"(t)
                 : "l"(p));
    v = __longlong_as_double((long long)b);
    return (unsigned)t;
}
__device__ __forceinline__ void tag_put(TagWord<float>* p, float v, unsigned tag) {
    const unsigned long long w = (unsigned long long)tag << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned tag_get(const TagWord<float>* p, float& v) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p));
    v = __uint_as_float((unsigned)w);
    return (unsigned)(w >> 32);
}

// Words and composed coefficients of the resident loop (pointers into the workspace).
template <typename T>
struct ResBufs {
    TagWord<T> *p, *e, *t0, *t3;     // NV words each
    TagWord<double>* part;           // 3 reductions x 2 values x (NV / kChunk) chunk totals
    T* a;                            // kResCoef x 32 per 32-row group
    int* c;                          // kResIdx x 32 per 32-row group
    const BalBlock* tab;             // one entry per block (nullptr: a single system)
};

// The resident loop's copy of the scaled, sorted matrix with the composed
// coefficients; and no word carries an epoch yet.
template <typename T, int NL>
__global__ void __launch_bounds__(kEngBlock) k_res_compose(Eng<T> E, ResBufs<T> R) {
    const long NV = E.NV;
    const long stride = (long)gridDim.x * blockDim.x, t0 = (long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long i = t0; i < 6 * (NV / kChunk); i += stride) R.part[i].tag = 0;
    for (long i = t0; i < NV; i += stride) {
        const int m = E.blk_member[i / kTile];
        if (m < 0) continue;
        R.p[i].tag = 0;
        R.e[i].tag = 0;
        R.t0[i].tag = 0;
        R.t3[i].tag = 0;
        T* a = R.a + (i >> 5) * (32 * kResCoef<NL>) + (i & 31);
        int* c = R.c + (i >> 5) * (32 * kResIdx<NL>) + (i & 31);
        auto put = [&](int slot, int k, long j) {
            a[32 * slot] = E.al[k * NV + j];
            c[32 * slot] = E.ll[k * NV + j];
        };
#pragma unroll
        for (int k = 0; k < NL; k++) put(k, k, i);
        a[32 * kResIdx<NL>] = E.d[i];
        const int c2 = E.ll[1 * NV + i];
        if (NL == 6) {
            const int c3 = E.ll[2 * NV + i];
            put(6, 1, c3);
            put(7, 0, c3);
            put(8, 0, c2);
            put(9, 0, E.ll[1 * NV + c3]);
            put(10, 3, E.ll[4 * NV + i]);
            put(11, 3, E.ll[5 * NV + i]);
        } else {
            put(4, 0, c2);
            put(5, 2, E.ll[3 * NV + i]);
        }
    }
}

// A bounded poll: false once it ran out or anybody's did.
struct ResWait {
    long limit;
    int* abort;          // device-wide
    int* s_fail;         // this block's
    __device__ __forceinline__ bool more(long& spins) const {
        if (*(volatile int*)s_fail) return false;
        ++spins;
        if (spins > limit) {
            atomicExch(abort, 1);
            *(volatile int*)s_fail = 1;
            return false;
        }
        if ((spins & 63) == 0 && ld_relaxed_s32(abort)) {
            *(volatile int*)s_fail = 1;
            return false;
        }
        return true;
    }
};

// Gather N words written at epoch `tag` (index `pad`: the zero row, not read).
// Every lane of the warp calls it.
template <typename T, int N>
__device__ __forceinline__ void res_gather(const TagWord<T>* __restrict__ buf, const int (&c)[N], int pad,
                                           unsigned tag, T (&v)[N], const ResWait& w) {
    long spins = 0;
#pragma unroll 1
    for (;;) {
        unsigned bad = 0;
#pragma unroll
        for (int q = 0; q < N; q++) {
            v[q] = T(0);
            if (c[q] != pad)
                bad |= tag_get((const TagWord<T>*)((const char*)buf + (unsigned)c[q] * (unsigned)sizeof(TagWord<T>)),
                               v[q]) ^ tag;
        }
        if (__all_sync(0xffffffffu, bad == 0)) return;
        if (!__all_sync(0xffffffffu, w.more(spins))) return;
    }
}

// The reductions' finalisations out of line: one thread runs them, and inlined
// their divisions and square roots would raise the loop's register count.
__device__ __noinline__ void res_finish(int red, MemberScalars* S, double t0, double t1) {
    const double tot[2] = {t0, t1};
    if (red == 0) finish_sweep56<1, true>(S, tot, S);
    else if (red == 1) finish_sweep56<2, true>(S, tot, S);
    else finish_xrupdate<true>(S, tot, S);
}

// Shared state of one block of the resident loop.
template <typename T>
struct ResShared {
    MemberScalars s;
    T y[kResWarps][32], u[kResWarps][32];
    double g[2 * kResMaxGroups];
    int fail;            // a poll ran out
    int stop;            // thread 0's verdict at the last reduction: leave the loop
};

// Totals of the member's chunk totals (reduction `red`, epoch tag), summed by
// this block along the canonical tree; fin(tot) runs in thread 0, and every
// thread leaves after a block barrier.
template <int NVAL, typename T>
__device__ __forceinline__ void res_totals(const TagWord<double>* part, int nc, unsigned tag, ResShared<T>& sh,
                                           const ResWait& wt, int red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ng = (nc + kGroupChunks - 1) / kGroupChunks;
#pragma unroll 1
    for (int g = w; g < ng; g += nw) {
        const int cg = min(kGroupChunks, nc - g * kGroupChunks);
        const TagWord<double>* p = part + 2L * g * kGroupChunks;
        double a[2][NVAL];
        long spins = 0;
#pragma unroll 1
        for (;;) {
            unsigned bad = 0;
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int k = 0; k < NVAL; k++) {
                    a[h][k] = 0.0;
                    if (lane + 32 * h < cg) bad |= tag_get(p + 2 * (lane + 32 * h) + k, a[h][k]) ^ tag;
                }
            if (__all_sync(0xffffffffu, bad == 0)) break;
            if (!__all_sync(0xffffffffu, wt.more(spins))) break;
        }
        if (lane + 32 < cg)
#pragma unroll
            for (int k = 0; k < NVAL; k++) a[0][k] += a[1][k];
        if (NVAL == 1) {
            const double s = warp_sum(a[0][0]);
            if (lane == 0) sh.g[2 * g] = s;
        } else {
            const double s = warp_pair_sum(a[0][0], a[0][NVAL - 1]);
            if ((lane & 15) == 0) sh.g[2 * g + (lane >> 4)] = s;
        }
    }
    if (ng > 1) __syncthreads();
    if (w == 0) {
        __syncwarp();
        double a = 0.0, b = 0.0, tot[2];
        for (int j = lane; j < ng; j += 32) {
            a += sh.g[2 * j];
            if (NVAL == 2) b += sh.g[2 * j + 1];
        }
        if (ng > 1) {
            if (NVAL == 1) {
                tot[0] = warp_sum(a);
                tot[1] = 0.0;
            } else {
                const double s = warp_pair_sum(a, b);
                tot[0] = __shfl_sync(0xffffffffu, s, 0);
                tot[1] = __shfl_sync(0xffffffffu, s, 16);
            }
        } else {                          // one group: the butterfly adds zeros only
            tot[0] = a;
            tot[1] = b;
        }
        if (lane == 0) {
            res_finish(red, &sh.s, tot[0], tot[1]);
            sh.stop = sh.s.done || *(volatile int*)&sh.fail;
        }
    }
    __syncthreads();
}

// One block's walk over its rows: 32-row groups of its chunks, one row per
// lane, group q = w, w + nw, ... of the block.  Lanes past the member's end hold
// row numbers inside its padding (zero coefficients, indices at the zero row):
// they compute zeros and store nothing.
struct ResRow {
    unsigned i;
    bool ok;
};

template <typename T, int NL>
__global__ void __launch_bounds__(kResThreads, 1) k_res_loop(Eng<T> E, ResBufs<T> R, long limit, int absent) {
    if ((int)blockIdx.x == absent) return;
    __shared__ ResShared<T> sh;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    BalBlock bb;
    long off;
    int n, c0, c1;
    const bool go = bal_block(E, R.tab, bb, off, n, c0, c1);
    if (!go || sld(&E.S[bb.m].done)) return;            // a stopped member: none of its blocks iterates
    if (threadIdx.x == 0) sh.fail = 0;
    copy_scalars(sh.s, E.S + bb.m);
    const unsigned ep = (unsigned)sld(E.ctrl + 6);
    const ResWait wt{limit, E.abort, &sh.fail};
    __syncthreads();
    constexpr int NC = kResCoef<NL>, NI = kResIdx<NL>;
    const int nc = (n + kChunk - 1) / kChunk, nq = 4 * (c1 - c0), pad = (int)off + n;
    const int nround = (nq + nw - 1) / nw;
    const unsigned row0 = (unsigned)(off + (long)c0 * kChunk) + lane;
    TagWord<double>* part = R.part + 2 * (off / kChunk);
    const long pstride = 2 * (E.NV / kChunk);
    auto row = [&](int q) {
        unsigned i = row0 + 32u * q;
        asm volatile("" : "+r"(i));          // addresses are formed in each phase, not carried through all of them
        return ResRow{i, (int)i < pad};
    };
    auto coef = [&](const ResRow& rw) { return R.a + (size_t)(rw.i >> 5) * (32 * NC) + lane; };
    auto idx = [&](const ResRow& rw) { return R.c + (size_t)(rw.i >> 5) * (32 * NI) + lane; };
    // t0 = D in + sum_k AL_k in[LL_k] (as k_bal_axsub)
    auto axsub = [&](const TagWord<T>* in, const T* own, unsigned tag) {
#pragma unroll 1
        for (int q = w; q < nq; q += nw) {
            const ResRow rw = row(q);
            const T* a = coef(rw);
            const int* cp = idx(rw);
            T g[NL];
            int c[NL];
#pragma unroll
            for (int k = 0; k < NL; k++) c[k] = cp[32 * k];
            T s = own[rw.i] * a[32 * NI];
            res_gather<T, NL>(in, c, pad, tag, g, wt);
#pragma unroll
            for (int k = 0; k < NL; k++) s = fma_rn(a[32 * k], g[k], s);
            if (rw.ok) tag_put(R.t0 + rw.i, s, tag);
        }
    };
    // sweeps 1-2-3 (1-2 of four columns): t3 from t0
    auto sweeps_a = [&](unsigned tag) {
#pragma unroll 1
        for (int q = w; q < nq; q += nw) {
            const ResRow rw = row(q);
            const T* a = coef(rw);
            const int* cp = idx(rw);
            T o;
            if constexpr (NL == 6) {
                const int c[8] = {rw.ok ? (int)rw.i : pad, cp[0], cp[32], cp[64], cp[32 * 6], cp[32 * 7], cp[32 * 8],
                                  cp[32 * 9]};
                T g[8];
                res_gather<T, 8>(R.t0, c, pad, tag, g, wt);
                const T o1c3 = fnma(a[32 * 7], g[5], g[3]);         // sweep 1 at c3
                const T o1x = fnma(a[32 * 9], g[7], g[4]);          // at c2(c3)
                const T o2c3 = fnma(a[32 * 6], o1x, o1c3);          // sweep 2 at c3
                const T o1c2 = fnma(a[32 * 8], g[6], g[2]);         // sweep 1 at c2
                const T o2 = fnma(a[32], o1c2, fnma(a[0], g[1], g[0]));
                o = fnma(a[64], o2c3, o2);
            } else {
                const int c[4] = {rw.ok ? (int)rw.i : pad, cp[0], cp[32], cp[32 * 4]};
                T g[4];
                res_gather<T, 4>(R.t0, c, pad, tag, g, wt);
                const T o1c2 = fnma(a[32 * 4], g[3], g[2]);
                o = fnma(a[32], o1c2, fnma(a[0], g[1], g[0]));
            }
            if (rw.ok) tag_put(R.t3 + rw.i, o, tag);
        }
    };
    // sweeps 4-5-6 (3-4 of four columns) at row rw
    auto sweeps_b = [&](const ResRow& rw, unsigned tag) {
        const T* a = coef(rw);
        const int* cp = idx(rw);
        if constexpr (NL == 6) {
            const int c[6] = {rw.ok ? (int)rw.i : pad, cp[32 * 3], cp[32 * 4], cp[32 * 5], cp[32 * 10], cp[32 * 11]};
            T g[6];
            res_gather<T, 6>(R.t3, c, pad, tag, g, wt);
            const T o45 = fnma(a[32 * 10], g[4], g[2]);
            const T o46 = fnma(a[32 * 11], g[5], g[3]);
            const T o4 = fnma(a[32 * 3], g[1], g[0]);
            return fnma(a[32 * 5], o46, fnma(a[32 * 4], o45, o4));
        } else {
            const int c[4] = {rw.ok ? (int)rw.i : pad, cp[32 * 2], cp[32 * 3], cp[32 * 5]};
            T g[4];
            res_gather<T, 4>(R.t3, c, pad, tag, g, wt);
            const T o3c4 = fnma(a[32 * 5], g[3], g[2]);
            return fnma(a[32 * 3], o3c4, fnma(a[32 * 2], g[1], g[0]));
        }
    };
    // The chunk totals of one round (nw / 4 chunks): lane l of a chunk's warp folds
    // its rows 32 u + l in order, then the butterfly.  MODE 0: (u, y); 1: (u, y)
    // and (y, y); 2: (y, y) and (y, u).
    auto fold = [&](int rd, int red, unsigned tag, auto mode) {
        constexpr int MODE = decltype(mode)::value;
        constexpr int NVAL = MODE == 0 ? 1 : 2;
        __syncthreads();
        const int cc = c0 + rd * (nw / 4) + w;
        if (w < nw / 4 && cc < c1) {
            T v[NVAL];
#pragma unroll
            for (int k = 0; k < NVAL; k++) v[k] = T(0);
#pragma unroll
            for (int u = 0; u < kChunkRows; u++) {
                if ((long)cc * kChunk + 32 * u + lane >= n) continue;
                const T y = sh.y[4 * w + u][lane], b = sh.u[4 * w + u][lane];
                if (MODE == 2) {
                    v[0] = fma_rn(y, y, v[0]);
                    v[NVAL - 1] = fma_rn(y, b, v[NVAL - 1]);
                } else {
                    v[0] = fma_rn(b, y, v[0]);
                    if (MODE == 1) v[NVAL - 1] = fma_rn(y, y, v[NVAL - 1]);
                }
            }
            int idx;
            const T s = warp_tsum<T, NVAL>(v, idx);
            if ((lane & (32 / NVAL - 1)) == 0) tag_put(part + red * pstride + 2 * cc + idx, (double)s, tag);
        }
        if (rd + 1 < nround) __syncthreads();
    };
    unsigned it = 0;
#pragma unroll 1
    for (;; it++) {
        const unsigned ta = 2 * (ep + it) + 1, tb = ta + 1;
        {                                                   // p = r + BETA (p - AMU q), published
            const T BETA = T(sh.s.BETA), AMU = T(sh.s.AMU);
#pragma unroll 1
            for (int q = w; q < nq; q += nw) {
                const ResRow rw = row(q);
                T p = E.p[rw.i];
                if (it > 0) {
                    p = fma_rn(BETA, fnma(AMU, E.q[rw.i], p), E.r[rw.i]);
                    if (rw.ok) E.p[rw.i] = p;
                }
                if (rw.ok) tag_put(R.p + rw.i, p, ta);
            }
        }
        axsub(R.p, E.p, ta);                                // q = PM A p ; RQ -> ALP
        sweeps_a(ta);
#pragma unroll 1
        for (int rd = 0; rd < nround; rd++) {
            const int q = rd * nw + w;
            if (q < nq) {
                const ResRow rw = row(q);
                const T r0 = E.r0[rw.i];
                const T y = sweeps_b(rw, ta);
                if (rw.ok) E.q[rw.i] = y;
                sh.y[w][lane] = y;
                sh.u[w][lane] = r0;
            }
            fold(rd, 0, ta, std::integral_constant<int, 0>());
        }
        res_totals<1>(part, nc, ta, sh, wt, 0);
        if (sh.stop) break;
        {                                                   // e = r - ALP q, published
            const T ALP = T(sh.s.ALP);
#pragma unroll 1
            for (int q = w; q < nq; q += nw) {
                const ResRow rw = row(q);
                const T e = fnma(ALP, E.q[rw.i], E.r[rw.i]);
                if (rw.ok) {
                    E.e[rw.i] = e;
                    tag_put(R.e + rw.i, e, tb);
                }
            }
        }
        axsub(R.e, E.e, tb);                                // v = PM A e ; AMU
        sweeps_a(tb);
#pragma unroll 1
        for (int rd = 0; rd < nround; rd++) {
            const int q = rd * nw + w;
            if (q < nq) {
                const ResRow rw = row(q);
                const T e = E.e[rw.i];
                const T y = sweeps_b(rw, tb);
                if (rw.ok) E.v[rw.i] = y;
                sh.y[w][lane] = y;
                sh.u[w][lane] = e;
            }
            fold(rd, 1, tb, std::integral_constant<int, 1>());
        }
        res_totals<2>(part + pstride, nc, tb, sh, wt, 1);
        if (sh.stop) break;
        {                                                   // x, r ; RN, C1 ; stop tests
            const T ALP = T(sh.s.ALP), AMU = T(sh.s.AMU);
#pragma unroll 1
            for (int rd = 0; rd < nround; rd++) {
                const int q = rd * nw + w;
                if (q < nq) {
                    const ResRow rw = row(q);
                    const long i = rw.i;
                    const T ev = E.e[i], r0 = E.r0[i];
                    const T xn = fma_rn(AMU, ev, fma_rn(ALP, E.p[i], E.xi[i]));
                    const T rn = fnma(AMU, E.v[i], ev);
                    if (rw.ok) {
                        E.xi[i] = xn;
                        E.r[i] = rn;
                    }
                    sh.y[w][lane] = rn;
                    sh.u[w][lane] = r0;
                }
                fold(rd, 2, ta, std::integral_constant<int, 2>());
            }
        }
        res_totals<2>(part + 2 * pstride, nc, ta, sh, wt, 2);
        if (sh.stop) break;
    }
    if (bb.j == 0) {                                        // the member's scalars, for the host and later kernels
        constexpr int W = (int)(sizeof(MemberScalars) / 4);
        if (threadIdx.x < W) ((int*)(E.S + bb.m))[threadIdx.x] = ((const int*)&sh.s)[threadIdx.x];
        if (threadIdx.x == 0) atomicMax(E.ctrl + 7, (int)(ep + it + 1));
    }
}

}  // namespace clowns
