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
//   - LDUSUB's sweeps run in pairs (1-2 | 3-4 | 5-6, with four columns 1-2 | 3-4;
//     5 and 6 are one sweep).  A row re-evaluates the one neighbour value its
//     pair's second sweep needs from coefficients composed once per solve
//     (k_res_compose), with the same fused multiply-adds, so the bits are those of
//     separate sweeps.  That costs 4 more operations per row and iteration and
//     saves four trips.  (us per iteration with pairs / threes, 1-2-3 | 4-5-6, 12
//     more operations and one trip less each way / single sweeps: FP64 16.6 / 16.7 /
//     18.5 at 27 k rows, 39.8 / 43.5 / 40.7 at 239 k, 67.0 / 72.6 / 70.4 at 413 k.)
// What bounds it: a trip takes 0.3-0.5 us; a warp's FP64 operation holds its SM
// sub-partition for 64 cycles whatever its active lanes (76 with all four busy),
// so small systems are bound by the chain of dependent FP64 operations and large
// ones by their number.  Hence: rows are dealt out in groups of 32, one row per
// lane, so that a chunk's four groups use four sub-partitions; the two totals of
// a dot-product pair are folded by different warps; an extra warp per block
// finalises the scalars, and takes the square root and the stop tests of an
// iteration while the others already run the next one's first steps (after a stop
// those have only written scratch vectors); x is updated and p - AMU q formed
// while the totals travel.
// A word is overwritten only after a reduction of the same iteration that every
// reader's own contribution had to precede, so no reader can miss its epoch:
// the operator's intermediates (a vector of its own for each step) are rewritten
// once per reduction RQ / AMU, p and e once per iteration, and each of the three reductions has its own totals.
// Every poll is bounded: a warp that runs out raises the abort flag, polls of
// the other warps and blocks then give up too, and the block leaves at the next
// reduction; the host reports the failure.
#pragma once

#include <type_traits>

#include "engine.cuh"

namespace clowns {

constexpr int kResWarps = 28;                    // row warps of a block at most
constexpr int kResThreads = 32 * kResWarps + 32; // and the scalar warp: 64 registers per thread
constexpr int kResSteps = 3;                     // vectors between the operator's steps (NL / 2 of them used)

// Coefficients and indices of one 32-row group in the resident loop's layout:
// group-major, each a run of 32 lanes, so that one address and constant offsets
// reach all of a row's.  With c1..c6 the row's columns in sweep order:
//   slots 0..NL-1   AL(1..NL) / LL(1..NL)
//   slots NL, NL+1  sweep 1's coefficient and index at row c2, sweep 3's at c4
//   last coefficient: D
template <int NL>
constexpr int kResIdx = NL + 2;
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
    TagWord<T> *p, *e, *t[kResSteps];   // NV words each
    TagWord<double>* part;           // 3 reductions x 2 values x (NV / kChunk) chunk totals
    TagWord<double>* gpart;          // 3 reductions x 2 values x ngrp group totals
    int ngrp;                        // groups of all members
    T* a;                            // coefficients, kResCoef x 32 per 32-row group
    int* c;                          // indices, kResIdx x 32 per 32-row group
    const BalBlock* tab;             // one entry per block (nullptr: a single system)
};

// The resident loop's copy of the scaled, sorted matrix with the composed
// coefficients; and no word carries an epoch yet.
template <typename T, int NL>
__global__ void __launch_bounds__(kEngBlock) k_res_compose(Eng<T> E, ResBufs<T> R) {
    const long NV = E.NV;
    const long stride = (long)gridDim.x * blockDim.x, t0 = (long)blockIdx.x * blockDim.x + threadIdx.x;
    constexpr int NI = kResIdx<NL>;
    for (long i = t0; i < 6 * (NV / kChunk); i += stride) R.part[i].tag = 0;
    for (long i = t0; i < 6 * R.ngrp; i += stride) R.gpart[i].tag = 0;
    for (long i = t0; i < NV; i += stride) {
        const int m = E.blk_member[i / kTile];
        if (m < 0) continue;
        R.p[i].tag = 0;
        R.e[i].tag = 0;
#pragma unroll
        for (int k = 0; k < NL / 2; k++) R.t[k][i].tag = 0;
        T* a = R.a + (i >> 5) * (32 * (NI + 1)) + (i & 31);
        int* c = R.c + (i >> 5) * (32 * NI) + (i & 31);
        auto put = [&](int slot, int sweep, long j) {
            a[32 * slot] = E.al[(sweep - 1) * NV + j];
            c[32 * slot] = E.ll[(sweep - 1) * NV + j];
        };
#pragma unroll
        for (int k = 0; k < NL; k++) put(k, k + 1, i);
        a[32 * NI] = E.d[i];
        put(NL, 1, E.ll[1 * NV + i]);
        put(NL + 1, 3, E.ll[3 * NV + i]);
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

// Integer forms of the scalar tests: an FP64 comparison costs as much as an addition.
__device__ __forceinline__ bool f64_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ bool f64_finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// finish_xrupdate's stop tests (pcgpme_para.F90:215-254) by one thread, BETA
// already formed.  ERR = sqrt(RN / BN) takes a division and a square root, some 2000
// cycles in which the next reduction would wait; but with q = RN (1 / BN), within a
// few roundings of ERR^2, two inequalities rule both tests out in nearly every
// iteration: q above EPS^2, and |q - q_prev| above 2e-6 q (|ERR - ERRP| <= 1e-6 ERR
// gives at most that).  Otherwise ERR and ERRP are formed and compared exactly as
// finish_xrupdate does; at the loop's end ERR is formed from RN in any case.
struct ResStop {
    double invbn, eps2, q, rn_prev;
};
__device__ __noinline__ void res_stop_exact(MemberScalars* S, double RN, double rn_prev) {
    const double ERR = sqrt(RN / S->BN);                         // 215
    const double ERRP = S->K > 1 ? sqrt(rn_prev / S->BN) : S->ERRP;
    S->ERR = ERR;
    if (S->K >= 10 && fabs(ERR - ERRP) <= ERR * 1.0e-6) {        // 228
        stop_member(S, CLOWNS_STOP_STAGNATION, 0);
        S->ERRP = ERRP;
    } else if (ERR <= S->EPS) {                                  // 232
        stop_member(S, CLOWNS_STOP_TOL, 0);
        S->ERRP = ERRP;
    }
}
__device__ __forceinline__ void res_stop_tests(MemberScalars* S, ResStop& st, double RN, double C1, double BETA) {
    const double q = RN * st.invbn, dq = fabs(q - st.q);
    const int K = S->K + 1;
    S->RN = RN;
    S->C1 = C1;
    S->K = K;
    S->total_iter += 1;
    if (!f64_finite(RN) || !f64_finite(C1)) {
        S->ERR = sqrt(RN / S->BN);
        stop_member(S, CLOWNS_STOP_NONFINITE, S->mode != 1 ? CLOWNS_IER_NONFINITE : 0);
        return;
    }
    // q in (1e-290, 1e290) by its exponent; a NaN fails the comparisons
    const int ex = (__double2hiint(q) >> 20) & 0x7ff;
    const bool clear = ex > 60 && ex < 1986 && q > st.eps2 && dq > 2.1e-6 * q;
    if (!clear) res_stop_exact(S, RN, st.rn_prev);
    st.q = q;
    st.rn_prev = RN;
    if (S->done) return;
    if (f64_zero(S->AMU)) {                                      // 234
        stop_member(S, CLOWNS_STOP_AMU_ZERO, 0);
    } else if (f64_zero(C1)) {                                   // 240
        stop_member(S, CLOWNS_STOP_C1_ZERO, 0);
    } else {
        S->BETA = BETA;
        if (K >= S->ITER) {                                      // 250-254
            if (S->mode != 1) {
                stop_member(S, CLOWNS_STOP_MAXITER, CLOWNS_IER_MAXITER);
                S->K = S->ITER + 1;
            } else {
                stop_member(S, CLOWNS_STOP_MAXITER, 0);
            }
        }
    }
}

// Shared state of one block of the resident loop.
template <typename T>
struct ResShared {
    MemberScalars s;
    T y[kResWarps][32], u[kResWarps][32];
    double beta;         // of the iteration that starts (its stop tests may still run)
    ResStop st;
    int fail;            // a poll ran out
    int stop;            // the scalar warp's verdict at the last reduction: leave the loop
};

// The sum of up to 64 tagged pairs by one warp, along the canonical tree of a
// group: lane l adds words l and l + 32, then the butterfly.  NVAL = 2: value k in
// lanes 16 k .. 16 k + 15.
template <int NVAL>
__device__ __forceinline__ double res_group(const TagWord<double>* p, int cnt, unsigned tag, const ResWait& wt) {
    const int lane = threadIdx.x & 31;
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
                if (lane + 32 * h < cnt) bad |= tag_get(p + 2 * (lane + 32 * h) + k, a[h][k]) ^ tag;
            }
        if (__all_sync(0xffffffffu, bad == 0)) break;
        if (!__all_sync(0xffffffffu, wt.more(spins))) break;
    }
    if (cnt > 32) {
        if (lane + 32 < cnt)
#pragma unroll
            for (int k = 0; k < NVAL; k++) a[0][k] += a[1][k];
        __syncwarp();
    }
    return NVAL == 1 ? warp_sum(a[0][0]) : warp_pair_sum(a[0][0], a[0][NVAL - 1]);
}

// Member totals of one reduction (epoch tag), by the scalar warp of every block.
// Up to 64 chunks (one group) each block sums the chunk totals itself; otherwise
// a group is summed by one block -- the one that holds its first chunk -- and its
// total published, and every block sums the groups: 152 blocks polling every
// chunk total held up the stores they waited for (3-6 us per reduction at 27 k -
// 74 k rows).  Totals in every lane.
template <int NVAL>
__device__ __forceinline__ void res_totals(const TagWord<double>* part, TagWord<double>* gpart, int nc, int c0, int c1,
                                           unsigned tag, const ResWait& wt, double (&tot)[2]) {
    const int lane = threadIdx.x & 31;
    const int ng = (nc + kGroupChunks - 1) / kGroupChunks;
    double s;
    if (ng == 1) {
        s = res_group<NVAL>(part, nc, tag, wt);
        s += 0.0;                             // the member sum starts from 0
    } else {
#pragma unroll 1
        for (int g = (c0 + kGroupChunks - 1) / kGroupChunks; g * kGroupChunks < c1; g++) {
            const double t = res_group<NVAL>(part + 2L * g * kGroupChunks, min(kGroupChunks, nc - g * kGroupChunks),
                                             tag, wt);
            if ((lane & (32 / NVAL - 1)) == 0) tag_put(gpart + 2 * g + lane / (32 / NVAL), t, tag);
        }
        double a[NVAL];
#pragma unroll
        for (int k = 0; k < NVAL; k++) a[k] = 0.0;
        long spins = 0;
#pragma unroll 1
        for (int j = lane; j < ((ng + 31) & ~31); j += 32) {      // lane l: groups l, l + 32, ... in order
            double v[NVAL];
#pragma unroll 1
            for (;;) {
                unsigned bad = 0;
#pragma unroll
                for (int k = 0; k < NVAL; k++) {
                    v[k] = 0.0;
                    if (j < ng) bad |= tag_get(gpart + 2 * j + k, v[k]) ^ tag;
                }
                if (__all_sync(0xffffffffu, bad == 0)) break;
                if (!__all_sync(0xffffffffu, wt.more(spins))) break;
            }
            if (j < ng)
#pragma unroll
                for (int k = 0; k < NVAL; k++) a[k] += v[k];
        }
        __syncwarp();
        s = NVAL == 1 ? warp_sum(a[0]) : warp_pair_sum(a[0], a[NVAL - 1]);
    }
    tot[0] = __shfl_sync(0xffffffffu, s, 0);
    tot[1] = __shfl_sync(0xffffffffu, s, 16);
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
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nw = (blockDim.x >> 5) - 1, ws = nw;      // row warps; the scalar warp
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
    if (w == ws && lane == 0) {
        // EPS^2 with a margin far above the roundings of q (an EPS whose square underflows
        // gives 0: then q decides, and q = 0 goes to the exact tests)
        sh.st = ResStop{1.0 / sh.s.BN, sh.s.EPS * sh.s.EPS * (1.0 + 1e-9), 0.0, 0.0};
    }
    constexpr int NI = kResIdx<NL>, NC = NI + 1;
    const int nc = (n + kChunk - 1) / kChunk, pad = (int)off + n;
    const int nq = w == ws ? 0 : 4 * (c1 - c0);         // the scalar warp has no rows
    const int nround = (4 * (c1 - c0) + nw - 1) / nw;
    const unsigned row0 = (unsigned)(off + (long)c0 * kChunk) + lane;
    TagWord<double>* part = R.part + 2 * (off / kChunk);
    const long pstride = 2 * (E.NV / kChunk);
    TagWord<double>* gpart = R.gpart + 2 * E.mem_grp0[bb.m];
    const int gstride = 2 * R.ngrp;
    auto row = [&](int q) {
        unsigned i = row0 + 32u * q;
        asm volatile("" : "+r"(i));          // addresses are formed in each phase, not carried through all of them
        return ResRow{i, (int)i < pad};
    };
    auto coef = [&](const ResRow& rw) { return R.a + (size_t)(rw.i >> 5) * (32 * NC) + lane; };
    auto idx = [&](const ResRow& rw) { return R.c + (size_t)(rw.i >> 5) * (32 * NI) + lane; };
    auto self = [&](const ResRow& rw) { return rw.ok ? (int)rw.i : pad; };
    // t[0] = D in + sum_k AL_k in[LL_k] (as k_bal_axsub)
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
            if (rw.ok) tag_put(R.t[0] + rw.i, s, tag);
        }
    };
    // Sweeps S, S + 1 of LDUSUB at a row, from the words `in`; X: the slot of sweep S at
    // column S + 1.
    auto pair = [&](const ResRow& rw, const TagWord<T>* in, unsigned tag, auto S, auto X) {
        constexpr int s = decltype(S)::value - 1, x = decltype(X)::value;
        const T* a = coef(rw);
        const int* cp = idx(rw);
        const int c[4] = {self(rw), cp[32 * s], cp[32 * (s + 1)], cp[32 * x]};
        T g[4];
        res_gather<T, 4>(in, c, pad, tag, g, wt);
        const T o = fnma(a[32 * s], g[1], g[0]);
        return fnma(a[32 * (s + 1)], fnma(a[32 * x], g[3], g[2]), o);
    };
    using std::integral_constant;
#define RES_K(k) integral_constant<int, k>()
    // every step of LDUSUB but the last, from t[0]
    auto step = [&](int k, unsigned tag, auto S, auto X) {
#pragma unroll 1
        for (int q = w; q < nq; q += nw) {
            const ResRow rw = row(q);
            const T o = pair(rw, R.t[k], tag, S, X);
            if (rw.ok) tag_put(R.t[k + 1] + rw.i, o, tag);
        }
    };
    auto sweeps = [&](unsigned tag) {
        step(0, tag, RES_K(1), RES_K(NL));
        if constexpr (NL == 6) step(1, tag, RES_K(3), RES_K(NL + 1));
    };
    // the last step at one row
    auto last = [&](const ResRow& rw, unsigned tag) {
        if constexpr (NL == 4) {
            return pair(rw, R.t[1], tag, RES_K(3), RES_K(NL + 1));
        } else {
            const T* a = coef(rw);
            const int* cp = idx(rw);
            const int c[3] = {self(rw), cp[32 * 4], cp[32 * 5]};
            T g[3];
            res_gather<T, 3>(R.t[2], c, pad, tag, g, wt);
            return fnma(a[32 * 5], g[2], fnma(a[32 * 4], g[1], g[0]));
        }
    };
    // The chunk totals of one round (nw / 4 chunks, their rows' y and u in shared
    // memory): lane l of a chunk's warp folds its rows 32 u + l in order, then the
    // butterfly.  MODE 0: (u, y); 1: (u, y) and (y, y); 2: (y, y) and (y, u), each
    // total by a warp of its own.
    auto fold = [&](int rd, int red, unsigned tag, auto mode) {
        constexpr int MODE = decltype(mode)::value;
        constexpr int NVAL = MODE == 0 ? 1 : 2;
        __syncthreads();
        const int cw = w / NVAL, k = w % NVAL, cc = c0 + rd * (nw / 4) + cw;
        if (cw < nw / 4 && cc < c1) {
            const bool square = MODE == 1 ? k == 1 : MODE == 2 ? k == 0 : false;
            T v = T(0);
#pragma unroll
            for (int u = 0; u < kChunkRows; u++) {
                if ((long)cc * kChunk + 32 * u + lane >= n) continue;
                const T y = sh.y[4 * cw + u][lane], b = square ? y : sh.u[4 * cw + u][lane];
                v = fma_rn(b, y, v);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) tag_put(part + red * pstride + 2 * cc + k, (double)v, tag);
        }
        if (rd + 1 < nround) __syncthreads();
    };
    unsigned it = 0;
#pragma unroll 1
    for (;; it++) {
        const unsigned ta = 2 * (ep + it) + 1, tb = ta + 1;
        double tot[2];
        {                                                   // p = r + BETA (p - AMU q), published
            const T BETA = T(sh.beta);
#pragma unroll 1
            for (int q = w; q < nq; q += nw) {
                const ResRow rw = row(q);
                T p = E.p[rw.i];                            // p - AMU q after the first iteration
                if (it > 0) {
                    p = fma_rn(BETA, p, E.r[rw.i]);
                    if (rw.ok) E.p[rw.i] = p;
                }
                if (rw.ok) tag_put(R.p + rw.i, p, ta);
            }
        }
        axsub(R.p, E.p, ta);                                // q = PM A p ; RQ -> ALP
        sweeps(ta);
#pragma unroll 1
        for (int rd = 0; rd < nround; rd++) {
            const int q = rd * nw + w;                      // past nq in the scalar warp
            if (q < nq) {
                const ResRow rw = row(q);
                const T r0 = E.r0[rw.i];
                const T y = last(rw, ta);
                if (rw.ok) E.q[rw.i] = y;
                sh.y[w][lane] = y;
                sh.u[w][lane] = r0;
            }
            fold(rd, 0, ta, RES_K(0));
        }
        if (w == ws) {
            res_totals<1>(part, gpart, nc, c0, c1, ta, wt, tot);
            if (lane == 0) {
                if (!sh.s.done) finish_sweep56<1, true>(&sh.s, tot, &sh.s);   // done: by the last iteration's stop tests
                sh.stop = sh.s.done || *(volatile int*)&sh.fail;
            }
        }
        __syncthreads();
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
        sweeps(tb);
#pragma unroll 1
        for (int rd = 0; rd < nround; rd++) {
            const int q = rd * nw + w;                      // past nq in the scalar warp
            if (q < nq) {
                const ResRow rw = row(q);
                const T e = E.e[rw.i];
                const T y = last(rw, tb);
                if (rw.ok) E.v[rw.i] = y;
                sh.y[w][lane] = y;
                sh.u[w][lane] = e;
            }
            fold(rd, 1, tb, RES_K(1));
        }
        if (w == ws) {
            res_totals<2>(part + pstride, gpart + gstride, nc, c0, c1, tb, wt, tot);
            if (lane == 0) {
                finish_sweep56<2, true>(&sh.s, tot, &sh.s);
                sh.stop = sh.s.done || *(volatile int*)&sh.fail;
            }
        }
        __syncthreads();
        if (sh.stop) break;
        const T ALP = T(sh.s.ALP), AMU = T(sh.s.AMU);       // x, r ; RN, C1 ; stop tests
#pragma unroll 1
        for (int rd = 0; rd < nround; rd++) {
            const int q = rd * nw + w;                      // past nq in the scalar warp
            if (q < nq) {
                const ResRow rw = row(q);
                const T r0 = E.r0[rw.i];
                const T rn = fnma(AMU, E.v[rw.i], E.e[rw.i]);
                if (rw.ok) E.r[rw.i] = rn;
                sh.y[w][lane] = rn;
                sh.u[w][lane] = r0;
            }
            fold(rd, 2, ta, RES_K(2));
        }
#pragma unroll 1
        for (int q = w; q < nq; q += nw) {                  // while the totals travel
            const ResRow rw = row(q);
            if (rw.ok) {
                const T p = E.p[rw.i];
                E.xi[rw.i] = fma_rn(AMU, E.e[rw.i], fma_rn(ALP, p, E.xi[rw.i]));
                E.p[rw.i] = fnma(AMU, E.q[rw.i], p);
            }
        }
        double beta = 0.0;
        if (w == ws) {
            res_totals<2>(part + 2 * pstride, gpart + 2 * gstride, nc, c0, c1, ta, wt, tot);
            if (lane == 0) {                                // 241 (pcgpme_para.F90); pcgpme_2DH.f90:255
                beta = sh.s.mode == 2 ? tot[1] / (sh.s.AMU * sh.s.RQ) : tot[1] / sh.s.AMU / sh.s.RQ;
                sh.beta = beta;
            }
        }
        __syncthreads();
        // the stop tests, while the row warps start the next iteration; the verdict counts
        // at its first reduction
        if (w == ws && lane == 0) res_stop_tests(&sh.s, sh.st, tot[0], tot[1], beta);
    }
#undef RES_K
    if (bb.j == 0 && w == ws && lane == 0 && sh.s.K > 0 && f64_finite(sh.s.RN)) {
        // ERR of the last iteration, and ERRP where no stop test kept the older one
        sh.s.ERR = sqrt(sh.s.RN / sh.s.BN);
        if (!(sh.s.done && (sh.s.reason == CLOWNS_STOP_STAGNATION || sh.s.reason == CLOWNS_STOP_TOL)))
            sh.s.ERRP = sh.s.ERR;
    }
    __syncthreads();
    if (bb.j == 0) {                                        // the member's scalars, for the host and later kernels
        constexpr int W = (int)(sizeof(MemberScalars) / 4);
        if (threadIdx.x < W) ((int*)(E.S + bb.m))[threadIdx.x] = ((const int*)&sh.s)[threadIdx.x];
        if (threadIdx.x == 0) atomicMax(E.ctrl + 7, (int)(ep + it + 1));
    }
}

}  // namespace clowns
