// fvm_resident.cu -- line-resident zebra sweeps of the FP32 Poisson correction
// (mixed precision): one launch runs a whole refinement interval.
//
// The per-colour path launches one grid per zebra colour (two per sweep), and each
// launch re-reads its line factors, couplings and right-hand side from L2.  Here
// the radial lines j = 1..NJ-1 are split into blocks of B consecutive lines (B
// even); each CTA keeps its lines' FP32 factors, couplings, right-hand side and
// current correction on chip (registers and shared memory) for all refine_sweeps
// sweeps of the interval, so a sweep moves nothing but the boundary lines between
// neighbouring CTAs.
//
// Zebra order (odd lines, then even lines; lisolv.f90:18-33 reordered as in the
// per-colour kernels, neighbours through the periodic branch cut).  A CTA owning
// lines j0 .. j0+B-1 (j0 odd) also solves line j0+B, the first (odd) line of the
// next CTA, redundantly in the odd half: its even line j0+B-1 then finds both
// neighbours on chip, and the only data from other CTAs a sweep needs are the
// previous sweep's values of line j0-1 (last line of the CTA before) and of line
// j0+B+1 (second line of the CTA after).  One exchange per sweep, both directions
// at once.  The redundant line's result is bit-identical to its owner's (same
// inputs, same code).
//
// Exchange without flags or fences: every published element is one 64-bit word
// (FP32 value bits | tag << 32) written and polled with relaxed gpu-scope 64-bit
// accesses (single-copy atomic), so a word whose tag matches carries the value of
// that sweep.  Tags are the CTA's count of completed sweeps (kept in XCNT across
// launches, equal in every CTA), words alternate between two slots by sweep
// parity, and a slot is overwritten only after both readers have passed the sweep
// that read it.  Every wait is bounded (max_polls); a wait that runs out sets the
// control block's fault flag, ends the Poisson loop and returns, and the host
// reports FVM_ERR_TIMEOUT and clears the exchange state.
//
// The arithmetic of a line (right-hand side, precomputed-factor solve, correction
// added to P in FP64 with the BCP ghosts refreshed) is the per-colour kernel's,
// operation for operation, so both paths give identical bits.  Compiled with
// -ftz=true, as the per-colour sweeps are.
//
// k_pois32_resident2 (below) exchanges once per two sweeps: 4-line blocks keep an
// 11-line window and solve the neighbours' three nearest lines again; it also runs the
// whole forward iteration, residuals and decisions included, in one launch.  Launched per
// interval inside the forward Poisson loop, either kernel first takes the loop's
// convergence decision from the residual kernel's sums (resident_decide).
#include <type_traits>

#include "fvm_internal.cuh"
#include "fvm_ops.cuh"
#include "fvm_df.cuh"

namespace fvm {
namespace {

// volatile: re-executed on every poll; no memory clobber, so the loads of one poll
// can all be in flight at once
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ void st_word(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Convergence decision of the forward Poisson loop at the start of a resident
// launch (sys.decide): every block sums the partials the residual kernel
// k_mres left, in that kernel's own order (the same bits in every block), and takes
// k_mres's decision (iter_p.f90:37-50: done once the scaled residual is at the
// tolerance or the sweeps reach the cap) with the loop's sweep count from its own
// XCNT; block 0 records it.  Returns true when the loop is done: the launch then
// does nothing.  This takes the last-block reduction off the residual kernel's
// critical path.
template <int HAS_COND>
__device__ bool resident_decide(const Dev &d, const ResSys &sys, int S, double *sh, cudaGraphConditionalHandle cond)
{
    const double resip = mres_total(d.partial, (d.NJ - 1 + MRES_GROUP - 1) / MRES_GROUP, (d.NI - 1 + MRES_TI - 1) / MRES_TI, sh);
    const int it = (int)(d.XCNT[blockIdx.x] - sys.pctl->xbase);
    const bool stop = it > 0 && !(resip > d.resimax && it < d.nswpp);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sys.pctl->resip = resip;
        if (stop) {
            sys.pctl->done = 1;
            sys.pctl->capped = (resip > d.resimax) ? 1 : 0;
            sys.pctl->niter = it;
            if (HAS_COND) cudaGraphSetConditional(cond, 0);
        } else {
            sys.pctl->niter = it + S;
        }
    }
    return stop;
}

// Shared memory of a block: the block's current line values (B+1 lines, LW words
// each) and one fold buffer per line group.  Every value of the block stays in the
// chunk ownership of the line solve (thread t of a group holds elements
// t*M .. t*M+M-1); a line is stored as word k*TG + t = element t*M + k, so a
// neighbouring group reads exactly the elements its own thread t needs, bank-
// conflict free, and no transpose is needed.
template <int M, int NW>
struct ResLayout {
    // block size bound: wide chunks (M >= 6) keep their values in up to 128
    // registers per thread, so their blocks stay within 512 threads
    static constexpr int MAXT = M >= 6 ? 512 : 1024;
    static constexpr int TG = WARP * NW;
    static constexpr int LW = TG * M;   // words per line
    static size_t bytes(int B) { return sizeof(float) * size_t(B + 1) * (LW + 2 * NW); }
    // largest block of this instantiation (the dynamic shared memory allowed for it)
    static size_t max_bytes() { return bytes(MAXT / TG - 1); }
};

// Lines j0 .. j0+B-1 of block blockIdx.x and the redundant line j0+B: group g
// (32*NW threads) owns line j0+g.  S sweeps; apply != 0 adds the correction to P
// afterwards.  check_done != 0 returns at once when the loop is already done.
template <int M, int NW, int HAS_COND>
__global__ void __launch_bounds__(ResLayout<M, NW>::MAXT, 1)
    k_pois32_resident(const __grid_constant__ Dev d, const __grid_constant__ ResSys sys, int B, int S, int apply,
                      int check_done, int max_polls, unsigned tag_skew, cudaGraphConditionalHandle cond)
{
    using Lay = ResLayout<M, NW>;
    constexpr int TG = Lay::TG, LW = Lay::LW;
    extern __shared__ float shm[];
    __shared__ int s_fault, s_stop;
    __shared__ double s_sum[2 * MRES_MAX_GROUPS + 3];
    float *lines = shm;
    const int g = threadIdx.x / TG, t = threadIdx.x % TG;
    float *xch = shm + size_t(B + 1) * LW + size_t(g) * 2 * NW;
    const NamedSync<NW> bar{1 + g};
    const int L = d.NJ - 1;
    const int j0 = blockIdx.x * B + 1;
    auto wrap = [L](int j) { return j < 1 ? j + L : (j > L ? j - L : j); };
    const int j = wrap(j0 + g);
    const int n = d.sP.n;
    if (threadIdx.x == 0) {   // the loop's done flag, read once for the whole block
        s_fault = 0;
        s_stop = check_done ? sys.pctl->done : 0;
    }
    __syncthreads();
    if (s_stop) return;
    if (sys.decide && resident_decide<HAS_COND>(d, sys, S, s_sum, cond)) return;

    const size_t base = size_t(j - 1) * LW;
    float fi[M], fa[M], fb[M], an[M], as[M], rf[M], v[M], halo[M];
    load_factors<float, M, NW>(fi, fa, fb, sys.invDf + base, sys.faf + base, sys.fbf + base, t);
#pragma unroll
    for (int k = 0; k < M; k++) {
        const int e = t * M + k;   // chunk ownership
        const bool ok = e < n;
        const int c = IDX(e + 1, j);
        an[k] = ok ? sys.ANf[c] : 0.0f;
        as[k] = ok ? sys.ASf[c] : 0.0f;
        rf[k] = ok ? sys.RF[c] : 0.0f;
        halo[k] = 0.0f;   // the correction starts from zero
        v[k] = 0.0f;
        lines[g * LW + k * TG + t] = 0.0f;
    }
    const unsigned cnt0 = d.XCNT[blockIdx.x];
    const bool odd_line = (g & 1) == 0;            // j0 is odd: even g = colour 0
    const bool publish = g == 1 || g == B - 1;     // read by the blocks before / after
    const int hline = g == 0 ? wrap(j0 - 1) : (g == B ? wrap(j0 + B + 1) : 0);
    __syncthreads();

    int sw = 1;
    for (; sw <= S; sw++) {
        // odd lines (and the redundant first line of the next block)
        if (odd_line) {
            if (sw > 1 && hline) {
                const unsigned want = cnt0 + unsigned(sw - 1) + tag_skew;
                const unsigned long long *src = d.XW + (size_t((sw - 1) & 1) * L + (hline - 1)) * LW;
                unsigned pending = 0;
#pragma unroll
                for (int k = 0; k < M; k++)
                    if (t * M + k < n) pending |= 1u << k;
                for (int it = 0; pending && it < max_polls; it++) {
                    // one L2 round trip per poll: every pending word's load is issued
                    // before any is tested
                    unsigned long long w[M];
#pragma unroll
                    for (int k = 0; k < M; k++) w[k] = ((pending >> k) & 1u) ? ld_word(src + k * TG + t) : 0ull;
#pragma unroll
                    for (int k = 0; k < M; k++) {
                        if (((pending >> k) & 1u) && unsigned(w[k] >> 32) == want) {
                            halo[k] = __uint_as_float(unsigned(w[k]));
                            pending &= ~(1u << k);
                        }
                    }
                }
                if (pending) s_fault = 1;
            }
#pragma unroll
            for (int k = 0; k < M; k++) {
                const float xs = g == 0 ? halo[k] : lines[(g - 1) * LW + k * TG + t];
                const float xn = g == B ? halo[k] : lines[(g + 1) * LW + k * TG + t];
                v[k] = t * M + k < n ? pois32_rhs(an[k], xn, as[k], xs, rf[k]) : 0.0f;
            }
            group_apply_r<float, M, NW>(v, fi, fa, fb, t, xch, bar);
#pragma unroll
            for (int k = 0; k < M; k++) lines[g * LW + k * TG + t] = v[k];
        }
        __syncthreads();
        if (s_fault) break;   // read by every thread after the barrier: a uniform exit
        // even lines: both neighbours are on chip
        if (!odd_line) {
#pragma unroll
            for (int k = 0; k < M; k++) {
                const float xs = lines[(g - 1) * LW + k * TG + t];
                const float xn = lines[(g + 1) * LW + k * TG + t];
                v[k] = t * M + k < n ? pois32_rhs(an[k], xn, as[k], xs, rf[k]) : 0.0f;
            }
            group_apply_r<float, M, NW>(v, fi, fa, fb, t, xch, bar);
#pragma unroll
            for (int k = 0; k < M; k++) lines[g * LW + k * TG + t] = v[k];
            if (publish) {
                unsigned long long *dst = d.XW + (size_t(sw & 1) * L + (j - 1)) * LW;
                const unsigned long long tag = (unsigned long long)(cnt0 + unsigned(sw)) << 32;
#pragma unroll
                for (int k = 0; k < M; k++)
                    if (t * M + k < n) st_word(dst + k * TG + t, tag | __float_as_uint(v[k]));
            }
        }
        __syncthreads();
    }

    // the next residual launch (programmatic) may start its coefficient prologue;
    // it reads P only after its dependency wait, i.e. after this grid has finished
    griddep_launch();
    if (sw <= S) {   // a wait ran out: end the loop, leave P alone
        if (threadIdx.x == 0) {
            sys.pctl->fault = 1;
            sys.pctl->done = 1;
            if (HAS_COND) cudaGraphSetConditional(cond, 0);
        }
        return;
    }
    if (g < B) {
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int e = t * M + k;
            if (e < n) sys.DF[IDX(e + 1, j)] = v[k];
        }
        if (apply) {
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k;
                if (e < n) sys.X[IDX(e + 1, j)] += (double)v[k];
            }
            if (sys.bcp) {
                bar();
                if (t < WARP) refresh_row_ghosts<BCK_POISSON>(d, sys.X, sys.X, j, nullptr, nullptr, t);
            }
        }
    }
    if (threadIdx.x == 0) d.XCNT[blockIdx.x] = cnt0 + unsigned(S);
}

// Two sweeps per exchange.  A block of B = 4 lines j0 .. j0+3 keeps the window of
// lines j0-3 .. j0+B+3 on chip (rows w = 0 .. B+6, line j0-3+w; odd lines are the
// odd rows) and solves rows 1 .. B+5, one line group each.  A pair of sweeps starts
// from the previous sweep's values of the window's even lines; in the pair's first
// sweep the odd rows 1 .. B+5 and then the even rows 2 .. B+4 are solved, in the
// second the odd rows 3 .. B+3 and the even rows 4 .. B+2 (the block's own even
// lines): each half-sweep needs both neighbours, so the valid part of the window
// narrows by one row per half.  The rows beyond the block's own are the
// neighbours' lines solved again here with the same inputs and code, so their bits
// equal the owners'.  The only data from other blocks are the window's outer even
// rows 0, 2 and B+4, B+6, which are the even lines of the blocks before and after:
// every block publishes its two even lines once per pair and polls four lines at
// the start of the next, so one exchange serves two sweeps.  Tags and slots as in
// k_pois32_resident, counted per pair.
//
// LOOP: the whole forward iteration of a step in one launch.  The block also keeps the
// FP64 pressure of its lines and of lines j0-2, j0-1 and j0+4 (what the residual of
// its lines reads: rows j, j+-1 and the positional cross term's j-2) with their
// double-float split, and each interval
//   - forms the residual of its four lines in double-float, k_mres's terms in k_mres's
//     order, publishes the four lines (FP32) and its sums, polls the five other lines of
//     its window and every block's sums, and takes the decision (all blocks add the same
//     values in the same order);
//   - runs the sweeps;
//   - adds the corrections to its pressure, publishes the three lines that neighbours
//     need and adds theirs to its copies, so these stay the owners' bits.
// Ghost columns and the ghost row 0 hold the stored values in the first interval and
// BCP's of the current pressure afterwards.  The line words of an interval alternate
// between two slots of their own; a slot is rewritten two intervals later, after a
// decision that every reader has contributed to.
//
// LOOP = 2: the adjoint's transposed equation (fvm_adjoint.cu).  Its cross term reads rows j
// and j+2, columns i and i+2 (at i = 1 column 2) and no ghosts, so the pressure-like
// unknown is kept for lines j0-1 .. j0+5.
//
// Bound: the serial chain of the four half-sweeps of a pair, each a line solve (two scans
// over two warps) between block barriers, and one exchange (0.41 us one way).  The solve
// keeps its scans' constant products in registers (group_apply_c): half the shuffles.
// Measured against one launch per interval (with the steps around it): 512 x 384, two steps of
// 2048 sweeps 8.95 -> 6.59 ms; 128 x 96, four steps of 512 4.22 -> 3.17 ms; the transposed step
// at 128 x 96 1.77 -> 1.19 ms (with the later changes around it and every scan stage 6.42, 2.59, 0.85).
template <int M, int NW>
struct ResLayout2 {
    static constexpr int B = 4;
    static constexpr int TG = WARP * NW;
    static constexpr int LW = TG * M;
    static constexpr int NL = B + 7;   // window rows
    static constexpr int NG = B + 5;   // line groups (rows 1 .. B+5)
    static constexpr int NT = NG * TG;
    // Row of group gi.  A warp's quarter of the SM is its index mod 4: rows in group order
    // put every odd row of a two-warp layout on two quarters and every even row on the
    // other two; these orders spread the rows of each half-sweep over all four (512 x 384:
    // 1.39 -> 1.26 us per sweep; one-warp rows unchanged).
    __device__ static constexpr int row(int gi)
    {
        return int(((NW == 1 ? 0x864297531ull : 0x982756431ull) >> (4 * gi)) & 15u);
    }
    static constexpr size_t sweep_floats() { return (size_t(NL) * LW + size_t(NG) * 2 + 3) & ~size_t(3); }
    // LOOP: pressure of 7 lines (FP64), its split and that of the ghost row 0, the own
    // lines' residual
    static constexpr int PL = 7;
    static size_t bytes(int n, bool loop)
    {
        size_t b = sizeof(float) * sweep_floats();
        if (loop) b += sizeof(double) * size_t(PL) * (n + 1) + sizeof(float2) * size_t(PL + 1) * (n + 1) + sizeof(float) * size_t(B) * LW;
        return b;
    }
};

// Line words of the loop behind the sweeps' two slots: final corrections, residuals.
__device__ __forceinline__ unsigned long long *loop_words(const Dev &d, int what, int slot, int L, int LW)
{
    return d.XW + size_t(2 + 2 * what + slot) * L * LW;
}

template <int M, int NW, int HAS_COND, int LOOP>
__global__ void __launch_bounds__(ResLayout2<M, NW>::NT, 1)
    k_pois32_resident2(const __grid_constant__ Dev d, const __grid_constant__ ResSys sys, int S, int apply,
                       int check_done, const __grid_constant__ Waits waits, cudaGraphConditionalHandle cond)
{
    using Lay = ResLayout2<M, NW>;
    constexpr int TG = Lay::TG, LW = Lay::LW, B = Lay::B, NL = Lay::NL, PL = Lay::PL;
    static_assert(B == MRES_GROUP, "a block's lines are one group of the residual sums");
    extern __shared__ float shm[];
    __shared__ int s_fault, s_stop;
    __shared__ double s_sum[2 * MRES_MAX_GROUPS + 3], s_w[LOOP ? 2 * B * 16 : 1];
    float *rows = shm;
    const int gi = threadIdx.x / TG, t = threadIdx.x % TG;
    const int w = Lay::row(gi);   // the window row this group solves
    float *fold = shm + size_t(NL) * LW + 2 * gi;
    const NamedSync<NW> bar{1 + gi};
    const int L = d.NJ - 1;
    const int j0 = blockIdx.x * B + 1;
    auto wrap = [L](int j) { return j < 1 ? j + L : (j > L ? j - L : j); };
    const int j = wrap(j0 - 3 + w);
    const int n = d.sP.n;
    const bool own = w >= 3 && w <= B + 2;   // the block's own lines
    if (threadIdx.x == 0) {
        s_fault = 0;
        s_stop = check_done ? sys.pctl->done : 0;
    }
    __syncthreads();
    if (s_stop) return;
    if (!LOOP && sys.decide && resident_decide<HAS_COND>(d, sys, S, s_sum, cond)) return;

    const size_t base = size_t(j - 1) * LW;
    float fi[M], fa[M], fb[M], an[M], as[M], rf[M], v[M];
    load_factors<float, M, NW>(fi, fa, fb, sys.invDf + base, sys.faf + base, sys.fbf + base, t);
#pragma unroll
    for (int k = 0; k < M; k++) {
        const int e = t * M + k;
        const bool ok = e < n;
        const int c = IDX(e + 1, j);
        an[k] = ok ? sys.ANf[c] : 0.0f;
        as[k] = ok ? sys.ASf[c] : 0.0f;
        rf[k] = !LOOP && ok ? sys.RF[c] : 0.0f;
        v[k] = 0.0f;
    }
    const ScanConst<float> sc = scan_constants<float, M>(fa, fb, t);
    const unsigned cnt0 = d.XCNT[blockIdx.x];
    const bool odd = (w & 1) != 0;
    // the outer even rows, each polled by the group next to it
    const int hrow = w == 1 ? 0 : (w == 3 ? 2 : (w == B + 3 ? B + 4 : (w == B + 5 ? B + 6 : -1)));
    const int hline = hrow >= 0 ? wrap(j0 - 3 + hrow) : 0;
    const bool publish = !odd && w >= 4 && w <= B + 2;

    // poll the words of line q (chunk ownership) until they carry the tag
    auto poll = [&](const unsigned long long *src, unsigned want, auto &&take) {
        unsigned pending = 0;
#pragma unroll
        for (int k = 0; k < M; k++)
            if (t * M + k < n) pending |= 1u << k;
        for (int it = 0; pending && it < waits.max_polls; it++) {
            unsigned long long wd[M];
#pragma unroll
            for (int k = 0; k < M; k++) wd[k] = ((pending >> k) & 1u) ? ld_word(src + k * TG + t) : 0ull;
#pragma unroll
            for (int k = 0; k < M; k++) {
                if (((pending >> k) & 1u) && unsigned(wd[k] >> 32) == want) {
                    take(k, __uint_as_float(unsigned(wd[k])));
                    pending &= ~(1u << k);
                }
            }
        }
        if (pending) s_fault = 1;
    };
    auto post = [&](unsigned long long *dst, unsigned tag32) {
        const unsigned long long tag = (unsigned long long)tag32 << 32;
#pragma unroll
        for (int k = 0; k < M; k++)
            if (t * M + k < n) st_word(dst + k * TG + t, tag | __float_as_uint(v[k]));
    };
    auto solve = [&]() {
#pragma unroll
        for (int k = 0; k < M; k++) {
            const float xs = rows[(w - 1) * LW + k * TG + t];
            const float xn = rows[(w + 1) * LW + k * TG + t];
            v[k] = t * M + k < n ? pois32_rhs(an[k], xn, as[k], xs, rf[k]) : 0.0f;
        }
        group_apply_c<float, M, NW>(v, fi, fa, fb, sc, fold, t, bar);
#pragma unroll
        for (int k = 0; k < M; k++) rows[w * LW + k * TG + t] = v[k];
    };
    // S sweeps from a zero correction; false (in every thread) when a wait ran out
    auto sweeps = [&](unsigned cnt) {
        for (int q = threadIdx.x; q < NL * LW; q += Lay::NT) rows[q] = 0.0f;
        __syncthreads();
        for (int sw = 1; sw <= S; sw += 2) {   // sweeps sw and sw+1
            if (sw > 1 && hrow >= 0)
                poll(d.XW + (size_t(((sw - 1) >> 1) & 1) * L + (hline - 1)) * LW,
                     cnt + unsigned(sw - 1) + waits.skew[WAIT_SWEEP - 1],
                     [&](int k, float x) { rows[hrow * LW + k * TG + t] = x; });
            __syncthreads();
            if (s_fault) return false;   // uniform: read by every thread after the barrier
            if (odd) solve();                                  // sweep sw, odd rows 1 .. B+5
            __syncthreads();
            if (!odd) solve();                                 // sweep sw, even rows 2 .. B+4
            __syncthreads();
            if (odd && w >= 3 && w <= B + 3) solve();          // sweep sw+1, odd rows 3 .. B+3
            __syncthreads();
            if (publish) {                                     // sweep sw+1, the block's even lines
                solve();
                post(d.XW + (size_t(((sw + 1) >> 1) & 1) * L + (j - 1)) * LW, cnt + unsigned(sw + 1));
            }
            __syncthreads();
        }
        return true;
    };

    if constexpr (LOOP) {
        const int PW = n + 1, nt = (n + WARP - 1) / WARP, nb = gridDim.x;
        double *P = reinterpret_cast<double *>(shm + Lay::sweep_floats());   // [PL][PW]: lines j0-2 .. j0+4, columns 0 .. n
        float2 *ps = reinterpret_cast<float2 *>(P + size_t(PL) * PW);        // [PL + 1][PW]: split, and ghost row 0
        float *rfs = reinterpret_cast<float *>(ps + size_t(PL + 1) * PW);    // [B][LW]: own residual, words as in rows
        double *s_ab = s_sum + 2 * MRES_MAX_GROUPS;
        constexpr int ADJ = LOOP == 2 ? 1 : 0;
        const int pl = w - 1 - ADJ;   // P line of the group (rows 1 .. 7; ADJ: 2 .. 8)
        unsigned long long *psum = d.XW + size_t(6) * L * LW;
        auto split = [](double x) {
            const dd q = dd_split(x);
            return make_float2(q.hi, q.lo);
        };
        if (pl >= 0 && pl < PL) {
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k;
                if (e < n) {
                    const double x = sys.X[IDX(e + 1, j)];
                    P[pl * PW + e + 1] = x;
                    ps[pl * PW + e + 1] = split(x);
                }
            }
            if (t == 0) ps[pl * PW] = split(sys.X[IDX(0, j)]);
        } else if (!ADJ && pl == PL && j0 == 1) {
            for (int i = t; i < PW; i += TG) ps[PL * PW + i] = split(sys.X[IDX(i, 0)]);
        }
        __syncthreads();
        const int wid = threadIdx.x / WARP, lane = threadIdx.x & (WARP - 1);
        unsigned cnt = cnt0;
        int it = 0;
        double resip = 0.0;
        bool bad = false;
        for (int round = 0;; round++) {
            // residual of the own lines: one warp per line and 32 cells
            for (int task = wid; task < B * nt; task += Lay::NT / WARP) {
                const int q = task & (B - 1), col = task / B, i = col * WARP + lane + 1, jq = j0 + q;
                const bool inside = i <= n, has_cross = ADJ ? inside : inside && i > 1 && jq > 1;
                const int c = inside ? IDX(i, jq) : 0, cc = ADJ ? c : (has_cross ? IDX(i - 1, jq - 1) : 0);
                float2 cf[9];
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    const bool ok = k < 5 ? inside : has_cross;
                    cf[k] = ok ? sys.PC[size_t(k) * d.n + (k < 5 ? c : cc)] : make_float2(0.0f, 0.0f);
                }
                float raf = 0.0f, paf = 0.0f;
                if (ADJ && inside) {
                    const float2 *r0 = ps + (q + 1) * PW, *rp = r0 + 2 * PW, none = make_float2(0.0f, 0.0f);
                    auto at = [](float2 x) { return dd(x.x, x.y); };
                    auto co = [&](int k) { return at(cf[k]); };
                    const int i1 = i == 1 ? 2 : i;   // the planes of cell 1 hold its column-2 weights
                    const bool in1 = i1 <= n, in2 = i + 2 <= n;
                    const dd cross = ((co(5) * at(in1 ? r0[i1] : none) + co(6) * at(in1 ? rp[i1] : none)) +
                                      co(7) * at(in2 ? r0[i + 2] : none)) + co(8) * at(in2 ? rp[i + 2] : none);
                    const dd app = co(4) * at(r0[i]);
                    const dd am = (((app - co(0) * at(i < n ? r0[i + 1] : none)) - co(1) * at(r0[i - 1])) - co(2) * at(r0[PW + i])) -
                                  co(3) * at((r0 - PW)[i]);
                    const dd r = (dd_split(sys.SRC[c]) - cross) - am;
                    raf = fabsf(r.hi);
                    paf = fabsf(app.hi);
                    const int e = i - 1;
                    rfs[q * LW + (e % M) * TG + e / M] = r.hi;
                } else if (inside) {
                    const double divdt = sys.SRC[c];
                    const float2 *r0 = ps + (q + 2) * PW, *rm = r0 - 2 * PW;
                    if (q == 1 && j0 == 1) rm = ps + PL * PW;   // line 2: the ghost row
                    auto at = [](float2 x) { return dd(x.x, x.y); };
                    auto co = [&](int k) { return at(cf[k]); };
                    dd cross = dd(0.0f, 0.0f);
                    if (has_cross)
                        cross = ((co(5) * at(r0[i]) + co(6) * at(rm[i])) + co(7) * at(r0[i - 2])) + co(8) * at(rm[i - 2]);
                    const dd su = dd_split(divdt) - cross;
                    const dd app = co(4) * at(r0[i]);
                    const dd pe = i < n ? at(r0[i + 1]) : dd(0.0f, 0.0f);   // AE(NI-1) = 0
                    const dd r = ((((co(0) * pe + co(1) * at(r0[i - 1])) + co(2) * at(r0[PW + i])) + co(3) * at((r0 - PW)[i])) + su) - app;
                    raf = fabsf(r.hi);
                    paf = fabsf(app.hi);
                    const int e = i - 1;
                    rfs[q * LW + (e % M) * TG + e / M] = r.hi;
                }
                for (int o = 16; o > 0; o >>= 1) {
                    raf += __shfl_down_sync(0xffffffffu, raf, o);
                    paf += __shfl_down_sync(0xffffffffu, paf, o);
                }
                if (lane == 0) {
                    s_w[q * 16 + col] = (double)raf;
                    s_w[(B + q) * 16 + col] = (double)paf;
                }
            }
            __syncthreads();
            const unsigned rtag = cnt + 1u;
            unsigned long long *rw = loop_words(d, 1, round & 1, L, LW);
            unsigned long long *pw = psum + size_t(round & 1) * 4 * nb;
            if (own) {
#pragma unroll
                for (int k = 0; k < M; k++) v[k] = t * M + k < n ? rfs[(w - 3) * LW + k * TG + t] : 0.0f;
                post(rw + size_t(j - 1) * LW, rtag);
#pragma unroll
                for (int k = 0; k < M; k++) rf[k] = v[k];
            }
            if (wid == Lay::NT / WARP - 1) {   // the last group's last warp: the block's sums
                const int half = lane >> 4, col = lane & 15;
                const double x = mres_columns(col < nt ? mres_lines(s_w + half * B * 16 + col, 16) : 0.0);
                if (col == 0) {
                    const unsigned long long b = (unsigned long long)__double_as_longlong(x), tag = (unsigned long long)rtag << 32;
                    st_word(pw + 4 * blockIdx.x + 2 * half, tag | (b & 0xffffffffull));
                    st_word(pw + 4 * blockIdx.x + 2 * half + 1, tag | (b >> 32));
                }
            }
            if (!own)
                poll(rw + size_t(j - 1) * LW, rtag + waits.skew[WAIT_RES - 1], [&](int k, float x) { rf[k] = x; });
            else
                for (int q = (w - 3) * TG + t; q < 2 * nb; q += B * TG) {
                    bool got = false;
                    const unsigned want = rtag + waits.skew[WAIT_SUMS - 1];
                    for (int i = 0; !got && i < waits.max_polls; i++) {
                        const unsigned long long a = ld_word(pw + 2 * q), b = ld_word(pw + 2 * q + 1);
                        got = unsigned(a >> 32) == want && unsigned(b >> 32) == want;
                        if (got) s_sum[q] = __hiloint2double((int)(unsigned)b, (int)(unsigned)a);
                    }
                    if (!got) s_fault = 1;
                }
            __syncthreads();
            mres_ratio(s_sum, nb, s_ab, s_ab + 2);
            if (s_fault) { bad = true; break; }
            resip = ADJ && !(s_ab[1] > 0.0) ? 0.0 : s_ab[2];
            if (it > 0 && !(resip > d.resimax && it < d.nswpp)) break;
            if (!sweeps(cnt)) { bad = true; break; }
            cnt += unsigned(S);
            it += S;
            // corrections: own lines, and the neighbours' three
            unsigned long long *fw = loop_words(d, 0, round & 1, L, LW);
            if (own && w != (ADJ ? 5 : 4)) post(fw + size_t(j - 1) * LW, cnt);
            if (pl >= 0 && pl < PL && !own)
                poll(fw + size_t(j - 1) * LW, cnt + waits.skew[WAIT_CORR - 1], [&](int k, float x) { v[k] = x; });
            if (pl >= 0 && pl < PL) {
#pragma unroll
                for (int k = 0; k < M; k++) {
                    const int e = t * M + k;
                    if (e < n) {
                        const double x = P[pl * PW + e + 1] + f2d_int(v[k]);
                        P[pl * PW + e + 1] = x;
                        const float2 q = split(x);
                        ps[pl * PW + e + 1] = q;
                        if (!ADJ && e == 0) ps[pl * PW] = q;
                        if (!ADJ && j0 == 1 && w == 2) {   // line NJ-1: the ghost row 0
                            ps[PL * PW + e + 1] = q;
                            if (e == 0) ps[PL * PW] = q;
                        }
                    }
                }
            }
            __syncthreads();
            if (s_fault) { bad = true; break; }
        }
        if (bad) {   // a wait ran out: end the loop, leave P alone
            if (threadIdx.x == 0) {
                sys.pctl->fault = 1;
                sys.pctl->done = 1;
            }
            return;
        }
        if (own) {
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k;
                if (e < n) sys.X[IDX(e + 1, j)] = P[pl * PW + e + 1];
            }
        }
        if (threadIdx.x == 0) {
            d.XCNT[blockIdx.x] = cnt + 2u;   // past the last residual's tag
            if (blockIdx.x == 0) {
                sys.pctl->niter = it;
                sys.pctl->resip = resip;
                sys.pctl->capped = resip > d.resimax ? 1 : 0;
                sys.pctl->done = 1;
            }
        }
        return;
    }

    const bool ok = sweeps(cnt0);
    // the next residual launch (programmatic) may start its coefficient prologue;
    // it reads P only after its dependency wait, i.e. after this grid has finished
    griddep_launch();
    if (!ok) {   // a wait ran out: end the loop, leave P alone
        if (threadIdx.x == 0) {
            sys.pctl->fault = 1;
            sys.pctl->done = 1;
            if (HAS_COND) cudaGraphSetConditional(cond, 0);
        }
        return;
    }
    if (own) {
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int e = t * M + k;
            if (e < n) sys.DF[IDX(e + 1, j)] = v[k];
        }
        if (apply) {
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k;
                if (e < n) sys.X[IDX(e + 1, j)] += (double)v[k];
            }
            if (sys.bcp) {
                bar();
                if (t < WARP) refresh_row_ghosts<BCK_POISSON>(d, sys.X, sys.X, j, nullptr, nullptr, t);
            }
        }
    }
    if (threadIdx.x == 0) d.XCNT[blockIdx.x] = cnt0 + unsigned(S);
}

template <int M, int NW, int HAS_COND, int LOOP>
cudaError_t launch_resident2(const fvm_ctx *c, const ResSys &sys, cudaStream_t st, int S, int apply, int check_done,
                             int max_polls, int skewed, cudaGraphConditionalHandle cond)
{
    using Lay = ResLayout2<M, NW>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c->res_blocks);
    cfg.blockDim = dim3(Lay::NT);
    cfg.dynamicSmemBytes = Lay::bytes(c->d.sP.n, LOOP != 0);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = c->res_coop ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_pois32_resident2<M, NW, HAS_COND, LOOP>, c->d, sys, S, apply, check_done,
                              waits_of(max_polls, skewed), cond);
}

template <int M, int NW, int HAS_COND>
cudaError_t launch_resident(const fvm_ctx *c, const ResSys &sys, cudaStream_t st, int S, int apply, int check_done,
                            int max_polls, unsigned skew, cudaGraphConditionalHandle cond)
{
    using Lay = ResLayout<M, NW>;
    auto k = k_pois32_resident<M, NW, HAS_COND>;
    const size_t smem = Lay::bytes(c->res_lines);   // allowed by resident_setup
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c->res_blocks);
    cfg.blockDim = dim3((c->res_lines + 1) * Lay::TG);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = c->res_coop ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k, c->d, sys, c->res_lines, S, apply, check_done, max_polls, skew, cond);
}

}  // namespace

// Bounded wait of one exchange: about 1 s of polling at L2 latency.
constexpr int kResidentPolls = 1 << 21;

// Lines per block for the context (0: the per-colour path).  poisson_resident = 1
// takes 4 lines per block where they fit (measured fastest on 512 x 384: 2.40 us
// per sweep against 2.57 with 2), else the smallest even B dividing NJ-1 whose
// blocks are all co-resident; k >= 2 asks for k lines per block.
int resident_setup(fvm_ctx *c)
{
    c->res_lines = c->res_blocks = 0;
    c->res_depth = 1;
    c->res_loop = c->res_coop = false;
    const int want = c->p.poisson_resident;
    if (c->p.precision != FVM_MIXED || want == 0) return FVM_OK;
    const LineSys &s = c->d.sP;
    const int L = c->NJ - 1, TG = WARP * s.NW;
    int sms = 0;
    FVM_CUDA(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->p.device));
    const int order[] = {4, 2, 6, 8, 10, 12, 14};
    for (int B : order) {
        if (want >= 2 && B != want) continue;
        if (L % B || L / B < 2) continue;
        int per_sm = 0;
        cudaError_t e = cudaSuccess;
        bool ok = dispatch_line(s, [&](auto m, auto nw) {
            constexpr int M_ = decltype(m)::value, NW_ = decltype(nw)::value;
            if ((B + 1) * TG > ResLayout<M_, NW_>::MAXT) {
                e = cudaErrorInvalidConfiguration;
                return;
            }
            auto k0 = k_pois32_resident<M_, NW_, 0>;
            auto k1 = k_pois32_resident<M_, NW_, 1>;
            const size_t smem = ResLayout<M_, NW_>::bytes(B);
            // both variants may use the shared memory of their largest block (set here,
            // outside any stream capture; the same value for every context)
            const int cap = (int)ResLayout<M_, NW_>::max_bytes();
            e = cudaFuncSetAttribute(k0, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k1, (B + 1) * TG, smem);
        });
        if (!ok || e != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (L / B <= per_sm * sms) {
            c->res_lines = B;
            c->res_blocks = L / B;
            c->res_coop = true;
            break;
        }
    }
    if (want >= 2 && !c->res_lines) {
        c->err = "poisson_resident: the requested lines per block do not divide NJ-1 into co-resident blocks";
        return FVM_ERR_ARG;
    }
    // two sweeps per exchange where the window fits: 4 lines per block, line groups
    // of one or two warps, at least three blocks around the ring, all co-resident
    if (c->res_lines == 4 && c->p.resident_depth != 1 && c->res_blocks >= 3) {
        cudaError_t e = cudaSuccess;
        dispatch_line(s, [&](auto m, auto nw) {
            constexpr int M_ = decltype(m)::value, NW_ = decltype(nw)::value;
            if constexpr (NW_ <= 2) {
                using Lay = ResLayout2<M_, NW_>;
                auto k0 = k_pois32_resident2<M_, NW_, 0, 0>;
                auto k1 = k_pois32_resident2<M_, NW_, 1, 0>;
                auto kl = k_pois32_resident2<M_, NW_, 0, 1>;
                auto ka = k_pois32_resident2<M_, NW_, 0, 2>;
                const int n = WARP * NW_ * M_, most = (int)Lay::bytes(n, false), most_l = (int)Lay::bytes(n, true);
                int per_sm = 0, per_sm_l = 0;
                e = cudaFuncSetAttribute(k0, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
                if (e == cudaSuccess) e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
                if (e == cudaSuccess) e = cudaFuncSetAttribute(kl, cudaFuncAttributeMaxDynamicSharedMemorySize, most_l);
                if (e == cudaSuccess) e = cudaFuncSetAttribute(ka, cudaFuncAttributeMaxDynamicSharedMemorySize, most_l);
                if (e == cudaSuccess)
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k1, Lay::NT, Lay::bytes(s.n, false));
                if (e == cudaSuccess)
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_l, kl, Lay::NT, Lay::bytes(s.n, true));
                if (e == cudaSuccess && c->res_blocks <= per_sm * sms) c->res_depth = 2;
                // the whole iteration in one launch: the reference's positional cross term,
                // an even interval
                c->res_loop = c->res_depth == 2 && c->d.dd_pos && c->d.refine_sweeps % 2 == 0 &&
                              c->res_blocks <= per_sm_l * sms;
            }
        });
        if (e != cudaSuccess) cudaGetLastError();
    }
    if (c->p.resident_depth == 2 && c->res_depth != 2) {
        c->err = "resident_depth 2: needs 4 lines per block, line groups of at most two warps and 12 or more lines";
        return FVM_ERR_ARG;
    }
    return FVM_OK;
}

namespace {

// The forward pressure correction of a context.
ResSys forward_sys(const fvm_ctx *c)
{
    const Dev &d = c->d;
    return ResSys{d.sP.invDf, d.sP.faf, d.sP.fbf, d.cP.ANf, d.cP.ASf, d.RF, d.DF, d.P, d.pctl, 1, 0, d.PCD, d.DIVDT};
}

int launch_sys(fvm_ctx *c, const ResSys &sys, cudaStream_t st, int sweeps, int apply, int max_polls,
               unsigned tag_skew, cudaGraphConditionalHandle cond, int has_cond, int check_done)
{
    cudaError_t e = cudaErrorInvalidValue;
    const int polls = max_polls > 0 ? max_polls : kResidentPolls;
    const bool pairs = c->res_depth == 2 && sweeps % 2 == 0;   // two sweeps per exchange
    bool ok = dispatch_line(c->d.sP, [&](auto m, auto nw) {
        constexpr int M_ = decltype(m)::value, NW_ = decltype(nw)::value;
        if constexpr (NW_ <= 2) {
            if (pairs) {
                const int skewed = tag_skew ? WAIT_SWEEP : 0;
                if (has_cond) e = launch_resident2<M_, NW_, 1, 0>(c, sys, st, sweeps, apply, check_done, polls, skewed, cond);
                else e = launch_resident2<M_, NW_, 0, 0>(c, sys, st, sweeps, apply, check_done, polls, skewed, cond);
                return;
            }
        }
        if (has_cond) e = launch_resident<M_, NW_, 1>(c, sys, st, sweeps, apply, check_done, polls, tag_skew, cond);
        else e = launch_resident<M_, NW_, 0>(c, sys, st, sweeps, apply, check_done, polls, tag_skew, cond);
    });
    if (!ok) {
        c->err = "line length above 512 cells is not supported";
        return FVM_ERR_ARG;
    }
    if (e != cudaSuccess) {
        c->err = std::string("resident sweep launch: ") + cudaGetErrorString(e);
        return FVM_ERR_CUDA;
    }
    KCOUNT(c);
    return FVM_OK;
}

}  // namespace

// One launch of the resident sweeps for a single context (batches use the
// per-colour path).  max_polls <= 0 takes the default bound.
int resident_sweeps(const Tgt &t, int sweeps, int apply, int max_polls, unsigned tag_skew,
                    cudaGraphConditionalHandle cond, int has_cond, int check_done, int decide)
{
    ResSys sys = forward_sys(t.c);
    sys.decide = decide;
    return launch_sys(t.c, sys, t.st, sweeps, apply, max_polls, tag_skew, cond, has_cond, check_done);
}

namespace {
template <int LOOP>
int launch_loop(fvm_ctx *c, const ResSys &sys, int max_polls, int skewed)
{
    cudaError_t e = cudaErrorInvalidValue;
    dispatch_line(c->d.sP, [&](auto m, auto nw) {
        constexpr int M_ = decltype(m)::value, NW_ = decltype(nw)::value;
        if constexpr (NW_ <= 2)
            e = launch_resident2<M_, NW_, 0, LOOP>(c, sys, c->stream, c->d.refine_sweeps, 0, 0,
                                                  max_polls > 0 ? max_polls : kResidentPolls, skewed, 0);
    });
    if (e != cudaSuccess) {
        if (launch_refused(e)) {   // nor would the per-interval launch of as many blocks fit
            c->res_loop = false;
            c->res_lines = 0;
        }
        c->err = std::string("resident Poisson loop launch: ") + cudaGetErrorString(e);
        return FVM_ERR_CUDA;
    }
    KCOUNT(c);
    return FVM_OK;
}
}  // namespace

// The whole iteration whose source is in place: the forward pressure, and another system
// of the context's line tile with the transposed cross term.
int resident_loop(fvm_ctx *c, int max_polls, int skewed) { return launch_loop<1>(c, forward_sys(c), max_polls, skewed); }
int resident_loop_adjoint(fvm_ctx *c, const ResSys &sys, int max_polls, int skewed)
{
    return launch_loop<2>(c, sys, max_polls, skewed);
}

// The same sweeps on another system of the context's line tile (the adjoint's
// transposed Poisson equation); no graph condition, default wait bound.
int resident_sweeps_on(fvm_ctx *c, const ResSys &sys, int sweeps, int apply, int check_done)
{
    return launch_sys(c, sys, c->stream, sweeps, apply, 0, 0u, 0, 0, check_done);
}

// Exchange words of a context: two slots of every line in the largest tile (32 x 4
// warps x 4 elements) -- FP32, one word per value: sweeps, final corrections and
// residuals of the resident loop; FP64: two words per value of the ring -- and two slots
// of block sums.
size_t exchange_words(const fvm_ctx *c)
{
    const size_t line = 2 * size_t(c->NJ - 1) * WARP * 4 * 4;
    return (c->p.precision == FVM_MIXED ? 3 : 2) * line + 2 * 4 * size_t(RING_MAX_BLOCKS);
}

// The layout for a radial tile set after the context was created.  A layout that the
// parameters ask for and the new tile does not allow is given up (one sweep per exchange, or
// the per-colour kernels): the tile is the batch's, which runs none of them.  The exchange
// words have another layout and the blocks' counts may be of another number of blocks.
int resident_retile(fvm_ctx *c)
{
    const std::string err = c->err;
    const int rc = resident_setup(c);
    if (rc == FVM_ERR_ARG) c->err = err;
    else if (rc) return rc;
    if (c->pgraph) cudaGraphExecDestroy(c->pgraph);
    c->pgraph = nullptr;
    return resident_reset(c);
}

// After a wait ran out: the blocks' sweep counts may disagree, so clear the
// exchange words, the counts and the fault flag (stream-ordered).
int resident_reset(fvm_ctx *c)
{
    FVM_CUDA(c, cudaMemsetAsync(c->d.XW, 0, exchange_words(c) * sizeof(unsigned long long), c->stream));
    FVM_CUDA(c, cudaMemsetAsync(c->d.XCNT, 0, size_t(c->NJ) * sizeof(unsigned int), c->stream));
    FVM_CUDA(c, cudaMemsetAsync(&c->d.pctl->fault, 0, sizeof(int), c->stream));
    return FVM_OK;
}

}  // namespace fvm
