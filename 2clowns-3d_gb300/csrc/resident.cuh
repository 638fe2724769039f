// resident.cuh -- solves of small and medium systems and ensembles as ONE resident
// kernel whose blocks exchange vectors through self-validating words.
//
// Below some 0.7 M rows (FP64; 1.1 M in mixed precision) an iteration of the
// kernel-per-phase loop is bound by its kernel boundaries, not by its work: 12 kernels of about 4 us each
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
//     saves four trips.  (us per iteration of the kernel's first form with pairs /
//     threes, 1-2-3 | 4-5-6, 12 more operations and one trip less each way / single
//     sweeps: FP64 16.6 / 16.7 / 18.5 at 27 k rows, 39.8 / 43.5 / 40.7 at 239 k, 67.0 /
//     72.6 / 70.4 at 413 k; the present form takes 16.6, 32 and 49 with pairs.)
// What bounds it: a trip takes 0.25 us inside a die and 0.45 us across (two words sent to
// and fro: 515-550 and 910-920 clocks each way); a warp's FP64 operation holds its SM
// sub-partition for 64 cycles whatever its active lanes (76 with all four busy),
// so small systems are bound by the chain of dependent FP64 operations and large
// ones by their number and that chain (FP64 pipe 60 % busy at 413 k rows; L2, asked for
// 1.1 KB per row and iteration, is at 31 % of its peak throughput).  Hence: rows are dealt out in groups of 32, one row per
// lane, so that a chunk's four groups use four sub-partitions; the two totals of
// a dot-product pair are folded by different warps; an extra warp per block
// finalises the scalars, and takes the square root and the stop tests of an
// iteration while the others already run the next one's first steps (after a stop
// those have only written scratch vectors); x is updated and p - AMU q formed
// while the totals travel.
// A word is overwritten only after a reduction of the same iteration that every
// reader's own contribution had to precede, so no reader can miss its epoch:
// the operator's intermediates (a vector of its own for each step) are rewritten
// once per reduction RQ / AMU, the word of p and e likewise, and each of the three
// reductions has its own totals and its own verdict.
// The vectors no other block reads (q, r / v, p, e, r0, x) live in shared memory, in 48
// (FP64) or 24 bytes per row, which leaves L2 to the matrix and the words (r0 in global
// memory where they would take the L1 cache's share).
// Every poll is bounded: a warp that runs out raises the abort flag, polls of
// the other warps and blocks then give up too, and the block leaves at the next
// reduction; the host reports the failure.
#pragma once

#include <type_traits>

#include "engine.cuh"

namespace clowns {

constexpr int kResWarps = 28;                    // row warps of a block at most
constexpr int kResThreads = 32 * kResWarps + 32; // and the scalar warp
constexpr int kResRegs = 65536 / kResThreads & ~7;  // 64 registers per thread, at any launch size
constexpr int kResReds = 5;                      // RQ, AMU, RN, and two of the mixed path's refinement: a
                                                 // reduction's words are written again only after another one
constexpr int kResVecs = 6;                      // vectors a block keeps in shared memory, five with FAR
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
    TagWord<T> *in, *t[kResSteps];   // p or e, and the operator's intermediates: NV words each
    TagWord<double> *x64, *t64[kResSteps];   // mixed path: the solution, PM's intermediates
    TagWord<double>* part;           // kResReds reductions x 2 values x (NV / kChunk) chunk totals
    TagWord<double>* gpart;          // kResReds reductions x 2 values x ngrp group totals
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
    for (long i = t0; i < 2 * kResReds * (NV / kChunk); i += stride) R.part[i].tag = 0;
    for (long i = t0; i < 2 * kResReds * R.ngrp; i += stride) R.gpart[i].tag = 0;
    for (long i = t0; i < NV; i += stride) {
        const int m = E.blk_member[i / kTile];
        if (m < 0) continue;
        R.in[i].tag = 0;
#pragma unroll
        for (int k = 0; k < NL / 2; k++) R.t[k][i].tag = 0;
        if (std::is_same<T, float>::value) {
            R.x64[i].tag = 0;
#pragma unroll
            for (int k = 0; k < NL / 2; k++) R.t64[k][i].tag = 0;
        }
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

// A coefficient's load, issued where it stands: before the poll whose wait hides it
// (the compiler leaves plain loads behind the loop that precedes their use).
__device__ __forceinline__ double ld_here(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_here(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

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

__device__ __forceinline__ bool f64_finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// finish_sweep56's finalisations.
template <int MODE>
__device__ __forceinline__ void res_finish56(MemberScalars* S, const double (&tot)[2]) {
    double ratio;
    if (MODE == 1) {
        ratio = S->C1 / tot[0];                                  // 167
        S->RQ = tot[0];
        S->ALP = ratio;
    } else {
        ratio = tot[0] / tot[1];                                 // 197
        S->SS = tot[1];
        S->AMU = ratio;
    }
    if (!f64_finite(tot[MODE - 1]) || !f64_finite(ratio)) {
        S->K += 1;
        stop_member(S, CLOWNS_STOP_NONFINITE, S->mode != 1 ? CLOWNS_IER_NONFINITE : 0);
    }
}

// finish_xrupdate's stop tests (pcgpme_para.F90:215-254) by one thread, BETA
// already formed.  ERR = sqrt(RN / BN) takes a division and a square root, some 2000
// cycles in which the next reduction would wait; but with q = RN (1 / BN), within a
// few roundings of ERR^2, two inequalities rule both tests out in nearly every
// iteration: q above EPS^2, and |q - q_prev| above 2e-6 q (|ERR - ERRP| <= 1e-6 ERR
// gives at most that).  Otherwise ERR and ERRP are formed and compared exactly as
// finish_xrupdate does; at the loop's end ERR is formed from RN in any case.
struct ResStop {
    double invbn, eps2, q, rn_prev;
    int tests;           // stop tests taken
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
    st.tests++;
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
    if (is_zero(S->AMU)) {                                      // 234
        stop_member(S, CLOWNS_STOP_AMU_ZERO, 0);
    } else if (is_zero(C1)) {                                   // 240
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

// Shared state of one block.
struct ResShared {
    MemberScalars s;
    double beta;         // of the iteration that starts (its stop tests may still run)
    ResStop st;
    Recip rq, amu;       // reciprocals for BETA, formed while others compute
    int fail;            // a poll ran out
    // The scalar warp's verdicts (leave the loop), a word for each reduction: once a poll has
    // given up, that warp no longer waits for the row warps' contributions and may reach the
    // next verdict while a row warp still has to read this one.  With one word the row
    // warps could part there, and those that went on wait for the others without a limit.
    int stop[kResReds];
};

// The butterfly over lanes of which only the first cnt hold terms: the levels that
// would add zeros are left out (no total here is -0: every sum starts from +0 or is one
// of a tree).  NVAL = 2: value k in lanes 16 k .. 16 k + 15.
template <int NVAL>
__device__ __forceinline__ double res_butterfly(const double (&a)[NVAL], int cnt) {
    double s = a[0];
    if (NVAL == 2) {
        const bool hi = (threadIdx.x & 16) != 0;
        const double other = __shfl_xor_sync(0xffffffffu, hi ? a[0] : a[NVAL - 1], 16);
        if (hi) s = a[NVAL - 1];
        if (cnt > 16) s += other;
        else if (hi) s = other;
    } else if (cnt > 16) {
        s += __shfl_xor_sync(0xffffffffu, s, 16);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
        if (cnt > o) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

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
    return res_butterfly<NVAL>(a[0], cnt);
}

// Member totals of one reduction (epoch tag), by the scalar warp of every block, in
// every lane of it.  The block that holds a group's first chunk sums the group and
// publishes its total, and every block sums the groups: 152 blocks polling every chunk
// total held up the stores they waited for (3-6 us per reduction at 27 k - 74 k rows).
template <int NVAL>
__device__ __forceinline__ void res_totals(const TagWord<double>* part, TagWord<double>* gpart, int nc, int c0, int c1,
                                           unsigned tag, const ResWait& wt, double (&tot)[2]) {
    const int lane = threadIdx.x & 31;
    const int ng = (nc + kGroupChunks - 1) / kGroupChunks;
    if (ng == 1) {                                // one group: every block sums its chunks itself
        double s = res_group<NVAL>(part, nc, tag, wt);
        s += 0.0;                                 // the member's sum starts from +0
        tot[0] = __shfl_sync(0xffffffffu, s, 0);
        tot[1] = __shfl_sync(0xffffffffu, s, 16);
        return;
    }
#pragma unroll 1
    for (int g = (c0 + kGroupChunks - 1) / kGroupChunks; g * kGroupChunks < c1; g++) {
        const double t = res_group<NVAL>(part + 2L * g * kGroupChunks, min(kGroupChunks, nc - g * kGroupChunks), tag, wt);
        if ((lane & (32 / NVAL - 1)) == 0) tag_put(gpart + 2 * g + lane / (32 / NVAL), t, tag);
    }
    double a[NVAL];
#pragma unroll
    for (int k = 0; k < NVAL; k++) a[k] = 0.0;
    long spins = 0;
#pragma unroll 1
    for (int j = lane; j < ((ng + 31) & ~31); j += 32) {          // lane l: groups l, l + 32, ... in order
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
    const double s = res_butterfly<NVAL>(a, ng);
    tot[0] = __shfl_sync(0xffffffffu, s, 0);
    tot[1] = __shfl_sync(0xffffffffu, s, 16);
}

// One block's walk over its rows: 32-row groups of its chunks, one row per
// lane, group q = w, w + nw, ... of the block.  Lanes past the member's end hold
// row numbers inside its padding (zero coefficients, indices at the zero row):
// they compute zeros and store nothing.
struct ResRow {
    unsigned i;          // row of the row space
    int l;               // of the block
    bool ok;
};

// One block's part of a member's solve.  FAR: r0, read twice an iteration, stays in
// global memory (kResL1Smem).
template <typename T, int NL, bool FAR>
struct Resident {
    static constexpr int NI = kResIdx<NL>, NC = NI + 1;
    static constexpr bool kWide = sizeof(T) == 4;     // FP64 rows take twice the registers
    const Eng<T>& E;
    const ResBufs<T>& R;
    ResShared& sh;
    T *p, *q, *e, *rv, *r0, *x;        // the block's rows of these vectors, in shared memory; rv: r from the
                                       // update of r until e is formed, v until the update of r
    ResWait wt;
    int lane, w, nw, ws;               // nw row warps; ws: the scalar warp
    BalBlock bb;
    long off, pstride;
    int n, c0, c1, nc, pad, nq, gstride;
    unsigned row0;
    TagWord<double>*part, *gpart;

    __device__ __forceinline__ Resident(const Eng<T>& E_, const ResBufs<T>& R_, ResShared& sh_, double* vecs, long limit)
        : E(E_), R(R_), sh(sh_), wt{limit, E_.abort, &sh_.fail} {
        lane = threadIdx.x & 31;
        w = threadIdx.x >> 5;
        nw = ws = (blockDim.x >> 5) - 1;
        bal_block(E, R.tab, bb, off, n, c0, c1);
        if (threadIdx.x == 0) sh.fail = 0;
        copy_scalars(sh.s, E.S + bb.m);
        __syncthreads();
        nc = (n + kChunk - 1) / kChunk;
        pad = (int)off + n;
        const int rows_b = (c1 - c0) * kChunk;
        q = (T*)vecs;
        rv = q + rows_b;
        p = rv + rows_b;
        e = p + rows_b;
        r0 = e + rows_b;
        x = r0 + rows_b;
        if constexpr (FAR) {
            x = r0;
            r0 = E.r0 + off + (long)c0 * kChunk;
        }
        nq = w == ws ? 0 : 4 * (c1 - c0);                   // the scalar warp has no rows
        row0 = (unsigned)(off + (long)c0 * kChunk) + lane;
        part = R.part + 2 * (off / kChunk);
        pstride = 2 * (E.NV / kChunk);
        gpart = R.gpart + 2 * E.mem_grp0[bb.m];
        gstride = 2 * R.ngrp;
    }
    __device__ __forceinline__ ResRow row(int q) const {
        unsigned i = row0 + 32u * q;
        asm volatile("" : "+r"(i));          // addresses are formed in each phase, not carried through all of them
        return ResRow{i, 32 * q + lane, (int)i < pad};
    }
    __device__ __forceinline__ const T* coef(const ResRow& rw) const { return R.a + (size_t)(rw.i >> 5) * (32 * NC) + lane; }
    __device__ __forceinline__ const int* idx(const ResRow& rw) const { return R.c + (size_t)(rw.i >> 5) * (32 * NI) + lane; }
    __device__ __forceinline__ int self(const ResRow& rw) const { return rw.ok ? (int)rw.i : pad; }
    // f(row) over this warp's rows
    template <typename F>
    __device__ __forceinline__ void rows(F f) const {
#pragma unroll 1
        for (int q = w; q < nq; q += nw) f(row(q));
    }
    // f(NR rows of this warp at once): NR = 1, or two where the block's rows take more than
    // one round of its warps, so that two rows' gathers are in flight per lane (a row
    // alone past the end comes twice, the second time not ok)
    template <typename F>
    __device__ __forceinline__ void rows2(F f) const {
        if (kWide && nq > nw) {
#pragma unroll 1
            for (int q = w; q < nq; q += 2 * nw) {
                const ResRow a = row(q), b = q + nw < nq ? row(q + nw) : ResRow{a.i, a.l, false};
                const ResRow rw[2] = {a, b};
                f(rw);
            }
        } else {
#pragma unroll 1
            for (int q = w; q < nq; q += nw) {
                const ResRow rw[1] = {row(q)};
                f(rw);
            }
        }
    }
    // t[0] = D in + sum_k AL_k in[LL_k] (as k_bal_axsub); own: the block's rows of `in`
    __device__ __forceinline__ void axsub(const T* own, unsigned tag) const {
        rows2([&](const auto& rw) {
            constexpr int NR = std::extent<std::remove_reference_t<decltype(rw)>>::value;
            T g[NR * NL], a[NR * NL], s[NR];
            int c[NR * NL];
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int* cp = idx(rw[r]);
                const T* ap = coef(rw[r]);
#pragma unroll
                for (int k = 0; k < NL; k++) c[r * NL + k] = cp[32 * k];
#pragma unroll
                for (int k = 0; k < NL; k++) a[r * NL + k] = ld_here(ap + 32 * k);
                s[r] = own[rw[r].l] * ap[32 * NI];
            }
            res_gather<T, NR * NL>(R.in, c, pad, tag, g, wt);
#pragma unroll
            for (int r = 0; r < NR; r++) {
#pragma unroll
                for (int k = 0; k < NL; k++) s[r] = fma_rn(a[r * NL + k], g[r * NL + k], s[r]);
                if (rw[r].ok) tag_put(R.t[0] + rw[r].i, s[r], tag);
            }
        });
    }
    // Sweeps S, S + 1 of LDUSUB at NR rows, from the words `in`; X: the slot of sweep S at
    // column S + 1.  V: the vectors' type (FP64 vectors on FP32 coefficients in the mixed
    // path's refinement).
    template <int S, int X, typename V, int NR>
    __device__ __forceinline__ void pair(const ResRow (&rw)[NR], const TagWord<V>* in, unsigned tag, V (&o)[NR]) const {
        constexpr int s = S - 1;
        V g[NR * 4];
        T a[NR * 3];
        int c[NR * 4];
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const int* cp = idx(rw[r]);
            const T* ap = coef(rw[r]);
            a[3 * r] = ld_here(ap + 32 * s);
            a[3 * r + 1] = ld_here(ap + 32 * (s + 1));
            a[3 * r + 2] = ld_here(ap + 32 * X);
            c[4 * r] = self(rw[r]);
            c[4 * r + 1] = cp[32 * s];
            c[4 * r + 2] = cp[32 * (s + 1)];
            c[4 * r + 3] = cp[32 * X];
        }
        res_gather<V, NR * 4>(in, c, pad, tag, g, wt);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const V o1 = fnma((V)a[3 * r], g[4 * r + 1], g[4 * r]);
            o[r] = fnma((V)a[3 * r + 1], fnma((V)a[3 * r + 2], g[4 * r + 3], g[4 * r + 2]), o1);
        }
    }
    template <int S, int X, typename V>
    __device__ __forceinline__ void step(const TagWord<V>* in, TagWord<V>* out, unsigned tag) const {
        auto f = [&](const auto& rw) {
            constexpr int NR = std::extent<std::remove_reference_t<decltype(rw)>>::value;
            V o[NR];
            pair<S, X, V, NR>(rw, in, tag, o);
#pragma unroll
            for (int r = 0; r < NR; r++)
                if (rw[r].ok) tag_put(out + rw[r].i, o[r], tag);
        };
        if constexpr (std::is_same<V, T>::value) rows2(f);
        else rows([&](const ResRow& r1) {
            const ResRow rw[1] = {r1};
            f(rw);
        });
    }
    // LDUSUB's steps but the last, from the words t[0]
    template <typename V>
    __device__ __forceinline__ void sweeps(TagWord<V>* const (&t)[kResSteps], unsigned tag) const {
        step<1, NL, V>(t[0], t[1], tag);
        if constexpr (NL == 6) step<3, NL + 1, V>(t[1], t[2], tag);
    }
    // the last step at NR rows
    template <typename V, int NR>
    __device__ __forceinline__ void last(TagWord<V>* const (&t)[kResSteps], const ResRow (&rw)[NR], unsigned tag,
                                         V (&o)[NR]) const {
        if constexpr (NL == 4) {
            pair<3, NL + 1, V, NR>(rw, t[1], tag, o);
        } else {
            V g[NR * 3];
            T a[NR * 2];
            int c[NR * 3];
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int* cp = idx(rw[r]);
                a[2 * r] = ld_here(coef(rw[r]) + 32 * 4);
                a[2 * r + 1] = ld_here(coef(rw[r]) + 32 * 5);
                c[3 * r] = self(rw[r]);
                c[3 * r + 1] = cp[32 * 4];
                c[3 * r + 2] = cp[32 * 5];
            }
            res_gather<V, NR * 3>(t[2], c, pad, tag, g, wt);
#pragma unroll
            for (int r = 0; r < NR; r++)
                o[r] = fnma((V)a[2 * r + 1], g[3 * r + 2], fnma((V)a[2 * r], g[3 * r + 1], g[3 * r]));
        }
    }
    template <typename V>
    __device__ __forceinline__ V last1(TagWord<V>* const (&t)[kResSteps], const ResRow& r1, unsigned tag) const {
        const ResRow rw[1] = {r1};
        V o[1];
        last<V, 1>(t, rw, tag, o);
        return o[0];
    }
    // Fold B chunk totals (numbers v0 .. v0 + B - 1; total v is value v % NVAL of the block's
    // chunk v / NVAL) in one warp: lane l folds a chunk's rows 32 h + l in order, then the
    // butterfly, in V.
    template <int MODE, int B, typename V>
    __device__ __forceinline__ void fold(const V* ys, const V* us, int v0, int red, unsigned tag) const {
        constexpr int NVAL = MODE == 1 || MODE == 2 ? 2 : 1;
        V v[B];
#pragma unroll
        for (int b = 0; b < B; b++) {
            v[b] = V(0);
            const int ch = (v0 + b) / NVAL, k = (v0 + b) % NVAL;
            if (ch >= c1 - c0) continue;
            const bool square = MODE == 3 || (MODE == 1 && k == 1) || (MODE == 2 && k == 0);
#pragma unroll
            for (int h = 0; h < kChunkRows; h++) {
                const int at = ch * kChunk + 32 * h + lane;
                if ((long)c0 * kChunk + at >= n) continue;
                const V y = ys[at], u = square ? y : us[at];
                v[b] = fma_rn(u, y, v[b]);
            }
        }
        int id;
        const V s = warp_tsum<V, B>(v, id);
        const int vv = v0 + id;
        if ((lane & (32 / B - 1)) == 0 && vv / NVAL < c1 - c0)
            tag_put(part + red * pstride + 2 * (c0 + vv / NVAL) + vv % NVAL, (double)s, tag);
    }
    // A reduction over the block's rows of y and u (in shared memory, written before the
    // barrier).  MODE 0: (u, y); 1: (u, y) and (y, y); 2: (y, y) and (y, u); 3: (y, y).
    // A warp takes one total at a time, or four by a transposed butterfly (6 additions
    // instead of 20) once there are more than five per SM sub-partition.
    template <int MODE, typename V>
    __device__ __forceinline__ void reduce(const V* ys, const V* us, int red, unsigned tag) const {
        if (w == ws) return;                                // the scalar warp has neither rows nor totals to fold
        asm volatile("bar.sync 1, %0;" ::"r"(32 * nw) : "memory");
        const int total = (c1 - c0) * (MODE == 1 || MODE == 2 ? 2 : 1);
        if (total > 20) {
#pragma unroll 1
            for (int v = 4 * w; v < total; v += 4 * nw) fold<MODE, 4, V>(ys, us, v, red, tag);
        } else {
#pragma unroll 1
            for (int v = w; v < total; v += nw) fold<MODE, 1, V>(ys, us, v, red, tag);
        }
    }
    // the operator's last step over the block's rows
    __device__ __forceinline__ void last_to(T* out, unsigned tag) const {
        rows2([&](const auto& rw) {
            constexpr int NR = std::extent<std::remove_reference_t<decltype(rw)>>::value;
            T o[NR];
            last<T, NR>(R.t, rw, tag, o);
#pragma unroll
            for (int r = 0; r < NR; r++)
                if (rw[r].ok) out[rw[r].l] = o[r];
        });
    }
    // The member's totals of reduction `red` and what follows from them: fin(totals) in
    // one thread; every thread then knows whether to go on.  A reduction never follows
    // itself, so a verdict is written over only after another reduction's barrier.
    template <int NVAL, typename F>
    __device__ __forceinline__ bool totals(int red, unsigned tag, F fin) const {
        if (w == ws) {
            double tot[2];
            res_totals<NVAL>(part + red * pstride, gpart + red * gstride, nc, c0, c1, tag, wt, tot);
            if (lane == 0) {
                fin(tot);
                sh.stop[red] = sh.s.done || *(volatile int*)&sh.fail;
            }
        }
        __syncthreads();
        return sh.stop[red] == 0;
    }
    // The iterations of one (inner) solve from r = p = r0, x, BN and C1; ep: epochs used so
    // far, each iteration takes two.
    __device__ __forceinline__ void iterate(unsigned& ep) const {
        if (w == ws && lane == 0)
            // EPS^2 with a margin far above the roundings of q (an EPS whose square underflows
            // gives 0: then q decides, and q = 0 goes to the exact tests)
            sh.st = ResStop{1.0 / sh.s.BN, sh.s.EPS * sh.s.EPS * (1.0 + 1e-9), 0.0, 0.0, 0};
#pragma unroll 1
        for (int it = 0;; it++, ep += 2) {
            const unsigned ta = ep + 1, tb = ep + 2;
            const T BETA = T(sh.beta);
            rows([&](const ResRow& rw) {                    // p = r + BETA (p - AMU q), published
                if (!rw.ok) return;
                T pn = p[rw.l];                             // p - AMU q after the first iteration
                if (it > 0) {
                    pn = fma_rn(BETA, pn, rv[rw.l]);
                    p[rw.l] = pn;
                }
                tag_put(R.in + rw.i, pn, ta);
            });
            axsub(p, ta);                                   // q = PM A p ; RQ -> ALP
            sweeps<T>(R.t, ta);
            last_to(q, ta);
            reduce<0, T>(q, r0, 0, ta);
            if (!totals<1>(0, ta, [&](const double (&tot)[2]) {
                    if (!sh.s.done) res_finish56<1>(&sh.s, tot);    // done: by the last iteration's stop tests
                }))
                break;
            if (w == ws && lane == 0) sh.rq = make_recip(sh.s.RQ);
            const T ALP = T(sh.s.ALP);
            rows([&](const ResRow& rw) {                    // e = r - ALP q, published
                if (!rw.ok) return;
                const T en = fnma(ALP, q[rw.l], rv[rw.l]);
                e[rw.l] = en;
                tag_put(R.in + rw.i, en, tb);
            });
            axsub(e, tb);                                   // v = PM A e ; AMU
            sweeps<T>(R.t, tb);
            last_to(rv, tb);
            reduce<1, T>(rv, e, 1, tb);
            if (!totals<2>(1, tb, [&](const double (&tot)[2]) { res_finish56<2>(&sh.s, tot); })) break;
            if (w == ws && lane == 0) sh.amu = make_recip(sh.s.mode == 2 ? sh.s.AMU * sh.s.RQ : sh.s.AMU);
            const T AMU = T(sh.s.AMU);                      // x, r ; RN, C1 ; stop tests
            rows([&](const ResRow& rw) {
                if (!rw.ok) return;
                const T rn = fnma(AMU, rv[rw.l], e[rw.l]);
                rv[rw.l] = rn;
                if (sh.s.mode == 2) E.r[rw.i] = rn;         // PCGPME_WILL's caller reads the residual
            });
            reduce<2, T>(rv, r0, 2, ta);
            rows([&](const ResRow& rw) {                    // while the totals travel
                if (!rw.ok) return;
                const T pn = p[rw.l];
                x[rw.l] = fma_rn(AMU, e[rw.l], fma_rn(ALP, pn, x[rw.l]));
                p[rw.l] = fnma(AMU, q[rw.l], pn);
            });
            double rn = 0.0, c1n = 0.0, beta = 0.0;
            totals<2>(2, ta, [&](const double (&tot)[2]) {  // 241 (pcgpme_para.F90); pcgpme_2DH.f90:255
                rn = tot[0];
                c1n = tot[1];
                beta = div_by(c1n, sh.amu);                 // by AMU RQ in mode 2
                if (sh.s.mode != 2) beta = div_by(beta, sh.rq);
                sh.beta = beta;
            });
            if (sh.stop[2]) break;                          // a poll ran out
            // the stop tests, while the row warps start the next iteration; the verdict counts
            // at its first reduction
            if (w == ws && lane == 0) res_stop_tests(&sh.s, sh.st, rn, c1n, beta);
        }
        ep += 2;
        if (w == ws && lane == 0 && sh.st.tests > 0 && f64_finite(sh.s.RN)) {
            // ERR of the last iteration, and ERRP where no stop test kept the older one
            sh.s.ERR = sqrt(sh.s.RN / sh.s.BN);
            if (!(sh.s.done && (sh.s.reason == CLOWNS_STOP_STAGNATION || sh.s.reason == CLOWNS_STOP_TOL)))
                sh.s.ERRP = sh.s.ERR;
        }
        __syncthreads();
    }
    // the member's scalars for the host
    __device__ __forceinline__ void finish() const {
        if (bb.j) return;
        constexpr int W = (int)(sizeof(MemberScalars) / 4);
        if (threadIdx.x < W) ((int*)(E.S + bb.m))[threadIdx.x] = ((const int*)&sh.s)[threadIdx.x];
    }
};

// A whole FP64 solve after the setup kernels: b^ = PM W b and BN, r = b^ - PM A x0
// and C1 (pcgpme_para.F90:113-145), the iterations, x to the caller.
template <int NL, bool FAR>
__global__ void __launch_bounds__(kResThreads, 1) k_res_plain(const Eng<double> E, const ResBufs<double> R, long limit,
                                                             int absent) {
    if ((int)blockIdx.x == absent) return;
    __shared__ ResShared sh;
    extern __shared__ double vecs[];
    const Resident<double, NL, FAR> S(E, R, sh, vecs, limit);
    S.rows([&](const ResRow& rw) {
        if (!rw.ok) return;
        const double x0 = E.xi[rw.i];
        S.x[rw.l] = x0;
        tag_put(R.t[0] + rw.i, E.p[rw.i], 1);               // W b
        tag_put(R.in + rw.i, x0, 2);
    });
    S.template sweeps<double>(R.t, 1);
    S.last_to(S.p, 1);
    S.template reduce<3, double>(S.p, nullptr, 0, 1);
    bool go = S.template totals<1>(0, 1, [&](const double (&tot)[2]) { sh.s.BN = tot[0]; });
    if (go) {
        S.axsub(S.x, 2);
        S.template sweeps<double>(R.t, 2);
        S.last_to(S.q, 2);
        S.rows([&](const ResRow& rw) {
            if (!rw.ok) return;
            const double r = S.p[rw.l] - S.q[rw.l];
            S.rv[rw.l] = r;
            S.p[rw.l] = r;
            S.r0[rw.l] = r;
            if (sh.s.mode == 2) E.r[rw.i] = r;
        });
        S.template reduce<3, double>(S.rv, nullptr, 1, 2);
        go = S.template totals<1>(1, 2, [&](const double (&tot)[2]) { sh.s.C1 = tot[0]; });
    }
    unsigned ep = 2;
    if (go) S.iterate(ep);
    double* out = E.in[S.bb.m].x - S.off;
    S.rows([&](const ResRow& rw) {
        if (rw.ok) out[rw.i] = S.x[rw.l];
    });
    S.finish();
}

// A whole mixed-precision solve after the setup kernels: ||PM W b|| on FP64 vectors,
// then refinement sweeps (as k_mx_residual, k_mx_sweep56, k_mx_normalize, k_mx_update)
// around the FP32 iterations until the member's outer stop test.
template <int NL, bool FAR>
__global__ void __launch_bounds__(kResThreads, 1) k_res_mixed(const Eng<float> E, const ResBufs<float> R,
                                                             double inner_tol, int inner_max, long limit, int absent) {
    if ((int)blockIdx.x == absent) return;
    __shared__ ResShared sh;
    extern __shared__ double vecs[];
    const Resident<float, NL, FAR> S(E, R, sh, vecs, limit);
    const MemberIn in = E.in[S.bb.m];
    double* y64 = vecs;                                     // FP64 operands lie over q and rv, dead between the sweeps
    S.rows([&](const ResRow& rw) {
        if (!rw.ok) return;
        tag_put(R.t64[0] + rw.i, E.r64[rw.i], 1);           // W b
        tag_put(R.x64 + rw.i, E.x64[rw.i], 1);
    });
    S.template sweeps<double>(R.t64, 1);
    S.rows([&](const ResRow& rw) { y64[rw.l] = S.template last1<double>(R.t64, rw, 1); });
    S.template reduce<3, double>(y64, nullptr, 4, 1);
    bool go = S.template totals<1>(4, 1, [&](const double (&tot)[2]) { sh.s.BN64 = tot[0]; });
    unsigned ep = 1, xtag = 1;
#pragma unroll 1
    while (go) {
        const unsigned tag = ++ep;
        S.rows([&](const ResRow& rw) {                      // r64 = W (b - A x64), the caller's matrix
            const long li = (long)rw.i - S.off;
            double g[NL];
            int c[NL];
#pragma unroll
            for (int k = 0; k < NL; k++) {
                const int cc = rw.ok && k < in.nl ? in.ll[k * (long)in.na + li] : 0;
                c[k] = cc > 0 && cc <= S.n ? (int)S.off + cc - 1 : S.pad;
            }
            double s = rw.ok ? in.d[li] * E.x64[rw.i] : 0.0;
            res_gather<double, NL>(R.x64, c, S.pad, xtag, g, S.wt);
#pragma unroll
            for (int k = 0; k < NL; k++)
                if (c[k] != S.pad) s = fma_rn(in.al[k * (long)in.na + li], g[k], s);
            if (rw.ok) tag_put(R.t64[0] + rw.i, E.W[rw.i] * (in.b[li] - s), tag);
        });
        S.template sweeps<double>(R.t64, tag);
        S.rows([&](const ResRow& rw) {
            const double y = S.template last1<double>(R.t64, rw, tag);
            y64[rw.l] = y;
            if (rw.ok) E.r64[rw.i] = y;
        });
        S.template reduce<3, double>(y64, nullptr, 3, tag);
        go = S.template totals<1>(3, tag, [&](const double (&tot)[2]) { mx_outer_test(&sh.s, tot[0], inner_tol, inner_max); });
        if (!go) break;
        const double inv = 1.0 / sh.s.SIGMA;
        S.rows([&](const ResRow& rw) {
            const float v = rw.ok ? (float)(E.r64[rw.i] * inv) : 0.f;
            S.p[rw.l] = v;
            S.r0[rw.l] = v;
            S.x[rw.l] = 0.f;
            y64[rw.l] = (double)v;
        });
        S.template reduce<3, double>(y64, nullptr, 4, tag);
        go = S.template totals<1>(4, tag, [&](const double (&tot)[2]) { sh.s.BN = sh.s.C1 = tot[0]; });
        if (!go) break;
        S.rows([&](const ResRow& rw) { S.rv[rw.l] = S.p[rw.l]; });   // r, where the operands were
        __syncthreads();
        S.iterate(ep);
        xtag = ++ep;
        const double sg = sh.s.SIGMA;
        S.rows([&](const ResRow& rw) {                      // x64 += sigma xi, published
            if (!rw.ok) return;
            const double x = fma_rn(sg, (double)S.x[rw.l], E.x64[rw.i]);
            E.x64[rw.i] = x;
            tag_put(R.x64 + rw.i, x, xtag);
        });
        go = *(volatile int*)&sh.fail == 0;
        go = __syncthreads_and(go);
    }
    S.rows([&](const ResRow& rw) {
        if (rw.ok) in.x[(long)rw.i - S.off] = E.x64[rw.i];
    });
    S.finish();
}

}  // namespace clowns
