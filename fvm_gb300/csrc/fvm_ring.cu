// fvm_ring.cu -- the FP64 Poisson iteration of a step in one launch (iter_p.f90:22-51,
// lisolv.f90:18-33, bcp.f90:8-42).
//
// The per-colour path (k_pois64, k_pres64) launches two grids per sweep.  A colour of
// the 128 x 96 grid took as long as one of 512 x 384 (about 7 us): launch latency, the
// operands' L2 round trips and the FP64 recurrences, not the arithmetic.  Here the
// lines j = 1..NJ-1 are dealt to a ring of blocks in pairs (odd line, even line), at
// most one block per SM, and each block keeps the factors, couplings, cross-term
// weights, source and pressure of its lines on chip for the whole iteration: sweeps,
// residuals and the convergence decision.  Only boundary lines and the residual's
// block sums travel between blocks.
//
// Order of the values.  Sweep n solves the odd lines from the neighbours' P^(n-1),
// then the even lines from the odd lines' P^n.  The lagged cross term of cell (i,j)
// is dd_p of cell (i-1,j-1) (the positional pairing of the reference's whole-array
// operand) and reads rows j and j-2, columns i and i-2, of P^(n-1); ghost column 0 and
// ghost row 0 hold values one BCP older, so they are P^(n-2)(1,j) and P^(n-2)(i,NJ-1).
// A line's pressure is therefore kept in three versions.  Every operation is k_pois64's
// and k_pres64's in the same rounding order, but for scan stages whose factors are all at
// most 2^-80, which are left out (2 to 7 % of a step): both paths give the same bits unless
// a value lies 2^27 or more below another on its line, where they differ by at most 2^-80 of
// the larger one a solve and, through later roundings, by units in the last place of the
// largest.  A line with a value that is not finite is not finite throughout, as there.
//
// A block with lines j0 .. j1 needs from others: line j0-1 (even, version n-1: coupling
// of j0, cross term of j0+1), line j0-2 (odd, version n-1: cross term of j0) and line
// j1+1 (odd, version n: coupling of j1).  Each published FP64 value is two 64-bit words
// (half of the value | tag << 32) written and polled with relaxed gpu-scope accesses, so a
// matching tag carries its half with no flag or fence; tags are the blocks' sweep
// counts (XCNT), words alternate between two slots, and a slot is rewritten two sweeps
// later, which the writer can only reach after every reader has passed: line j at sweep
// n+2 needs neighbours that needed the readers' sweep n+1.  While one colour is solved
// the other colour's groups form their next cross terms.  The residual's block sums
// travel the same way and every block adds them in the same order, so all blocks take
// the same decision.  Every wait is bounded; one that runs out sets a flag (one
// per parity of the sweep, one for the residual) that the whole block reads after the
// sweep's or the residual's last barrier and that nobody writes again before another
// barrier, so that all threads leave together.  The block leaves its pressure alone, the
// others' waits for it run out in turn, and the host reports FVM_ERR_TIMEOUT.  Waits::skew lets
// the waits of one kind look for tags that no block publishes: the check of those exits.
//
// ADJ: the transposed equation of the adjoint, (A^T + G^T DD^T) mu = g (fvm_adjoint.cu).
// Its lagged cross term at (i,j) reads mu^(n-1) at rows j and j+2 (wrapped), columns i and
// i+2, at i = 1 column 2 as well, and no ghosts; the residual takes the cross term of
// the current mu.  So the halo lines are j1+1 and j1+2 instead of j0-1 and j0-2.
//
// Bound: FP64.  A warp's FP64 instruction holds its quarter of the SM's FP64 pipe for 64
// cycles (measured: a dependent chain of DFMAs, and the same chain beside three others
// on the quarter, run at 67 and 259 cycles a step), so a line costs 64 cycles times the FP64
// instructions of its warps, 11 per element beside the scans, and a block's one or two
// concurrent lines are spread over all four quarters (radial_tile).  The other part is the
// exchange, 0.41 us one way through L2, twice a sweep.  The products of the constant
// factors that the line solve's scans carry are formed once per launch and kept in
// shared memory: per sweep only the value part of the scans is left.
// Measured (step with 512 or 2048 sweeps, residual every 8): 128 x 96 FP64 7.48 -> 2.17 ms
// (14.3 -> 3.9 us per sweep), 512 x 384 39.8 -> 16.1 ms (18 -> 7.6 us; 196,608 cells x 11
// instructions at the chip's 0.63 T/s: 3.4 us).
#include <algorithm>
#include <type_traits>

#include "fvm_internal.cuh"
#include "fvm_ops.cuh"

namespace fvm {
namespace {

constexpr int STAGES = 5;   // Kogge-Stone stages of a warp
constexpr int kRingPolls = 1 << 21;   // bound of a wait: about a second of polling at L2 latency

template <int M, int NW>
struct RingLayout {
    static constexpr int TG = WARP * NW, LW = TG * M;
    static constexpr int CST = 2 * (STAGES + 1) + 2 * M;   // per-thread scan constants
    // lines (3 versions), two halo lines of the cross term (3 versions each), per line the
    // scan constants, the warps' total products and the fold buffers
    static size_t doubles(int nl) { return size_t(3) * (nl + 2) * LW + size_t(nl) * (size_t(CST) * TG + 4 * NW); }
    static size_t bytes(int nl) { return sizeof(double) * doubles(nl); }
    static constexpr int MAXT = 4 * TG;   // at most two pairs per block
};

__device__ __forceinline__ void ld_words(const ulonglong2 *p, unsigned long long &a, unsigned long long &b)
{
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p));
}
__device__ __forceinline__ void st_words(ulonglong2 *p, double v, unsigned tag)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | (b & 0xffffffffull)), "l"(t | (b >> 32))
                 : "memory");
}
__device__ __forceinline__ double of_words(unsigned long long a, unsigned long long b)
{
    return __hiloint2double((int)(unsigned)b, (int)(unsigned)a);
}

// The M elements of a line that thread t owns, once their words carry the tag; false
// when the wait ran out.  One L2 round trip per poll: all loads precede the tests.  (Not unrolled:
// 128 x 96 2.29 ms against 2.20.)
template <int M, int TG>
__device__ __forceinline__ bool poll_line(const ulonglong2 *src, int t, int n, unsigned want, int max_polls, double (&out)[M])
{
    unsigned pending = 0;
#pragma unroll
    for (int k = 0; k < M; k++)
        if (t * M + k < n) pending |= 1u << k;
#pragma unroll 4
    for (int it = 0; pending && it < max_polls; it++) {
        unsigned long long a[M], b[M];
#pragma unroll
        for (int k = 0; k < M; k++) {
            a[k] = b[k] = 0ull;
            if ((pending >> k) & 1u) ld_words(src + k * TG + t, a[k], b[k]);
        }
#pragma unroll
        for (int k = 0; k < M; k++)
            if (((pending >> k) & 1u) && unsigned(a[k] >> 32) == want && unsigned(b[k] >> 32) == want) {
                out[k] = of_words(a[k], b[k]);
                pending &= ~(1u << k);
            }
    }
    return pending == 0;
}

// mode 0: the whole iteration; mode 1: `count` sweeps without residuals, P unchanged
// (timing).
template <int M, int NW, int ADJ>
__global__ void __launch_bounds__(RingLayout<M, NW>::MAXT, 1)
    k_ring64(const __grid_constant__ Dev d, const __grid_constant__ RingSys sys, int ppb, int mode, int count,
             const __grid_constant__ Waits waits)
{
    using Lay = RingLayout<M, NW>;
    constexpr int TG = Lay::TG, LW = Lay::LW, CST = Lay::CST;
    extern __shared__ double shm[];
    __shared__ int s_fault[3], s_nf;   // a wait of an even sweep, an odd one, a residual ran out
    __shared__ double s_line[2 * 8], s_tot[2 * RING_MAX_BLOCKS], s_res;
    const int L = d.NJ - 1, n = d.sP.n;
    const int pairs = L / 2, p0 = blockIdx.x * ppb, nl = 2 * min(ppb, pairs - p0), j0 = 2 * p0 + 1;
    // group gi takes line j0 + g, the block's odd lines first: a warp's quarter of the SM is
    // its index mod 4, and the lines solved at a time then cover all four
    const int gi = threadIdx.x / TG, g = gi < ppb ? 2 * gi : 2 * (gi - ppb) + 1;
    const int t = threadIdx.x % TG, lane = t & (WARP - 1), wl = t / WARP;
    const bool act = g < nl, odd = (g & 1) == 0;   // j0 is odd
    const int j = j0 + g;
    const NamedSync<NW> bar{1 + gi};
    const int nlm = 2 * ppb;
    double *own = shm;                                  // [3][nlm][LW]
    double *hm1 = own + size_t(3) * nlm * LW;           // [3][LW]
    double *hm2 = hm1 + size_t(3) * LW;                 // [3][LW]
    double *cst = hm2 + size_t(3) * LW + size_t(gi) * (size_t(CST) * TG + 4 * NW);
    double *fold = cst + size_t(CST) * TG;              // [Gtot | Htot | forward | backward][NW]
    auto line = [&](int ver, int q) { return own + (size_t(ver) * nlm + q) * LW; };
    auto wrap = [L](int q) { return q < 1 ? q + L : (q > L ? q - L : q); };
    if (threadIdx.x == 0) s_fault[0] = s_fault[1] = s_fault[2] = s_nf = 0;

    // operands of the line, in the chunk ownership of the solve (element e = t*M + k)
    double fi[M], fa[M], fb[M], an[M], as[M], dv[M], c1[M], c2[M], c3[M], c4[M], v[M], su[M], sun[M], w5 = 0.0, w6 = 0.0;
    if (act) {
        const size_t base = size_t(j - 1) * LW;
        load_factors<double, M, NW>(fi, fa, fb, sys.invD + base, sys.fa + base, sys.fb + base, t);
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int e = t * M + k;
            const bool ok = e < n;
            const int c = IDX(e + 1, j);
            an[k] = ok ? sys.AN[c] : 0.0;
            as[k] = ok ? sys.AS[c] : 0.0;
            dv[k] = ok ? sys.SRC[c] : 0.0;
            if (ADJ) {   // weights at (i-1, j-1), (i-1, y), (i+1, j-1), (i+1, y), y = j+1 or, from line NJ-1, 1
                const int y = j == L ? 1 : j + 1;
                const bool up = ok && j != L - 1, dn = ok && j > 1, we = e > 0, ea = e + 2 < n;
                c1[k] = dn && we ? d.CNE[IDX(e, j - 1)] : 0.0;
                c2[k] = up && we ? d.CSE[IDX(e, y)] : 0.0;
                c3[k] = dn && ea ? d.CNW[IDX(e + 2, j - 1)] : 0.0;
                c4[k] = up && ea ? d.CSW[IDX(e + 2, y)] : 0.0;
                if (e == 0) {   // the wall ghost's share of cell 1: column 2
                    w5 = dn && n > 1 ? d.CNW[IDX(1, j - 1)] : 0.0;
                    w6 = up && n > 1 ? d.CSW[IDX(1, y)] : 0.0;
                }
            } else {
                const bool cr = ok && e > 0 && j > 1;
                const int cc = cr ? IDX(e, j - 1) : 0;
                c1[k] = cr ? d.CNE[cc] : 0.0;
                c2[k] = cr ? d.CSE[cc] : 0.0;
                c3[k] = cr ? d.CNW[cc] : 0.0;
                c4[k] = cr ? d.CSW[cc] : 0.0;
            }
            v[k] = ok ? sys.X[c] : 0.0;
            su[k] = 0.0;
            line(0, g)[k * TG + t] = v[k];
        }
        // version -1 of a line is only read for its ghost column, which sits in element 0
        if (!ADJ && t == 0) line(2, g)[0] = sys.X[IDX(0, j)];
        // the scans' constant factors (group_apply_r's products, formed once)
        double G = 1.0;
#pragma unroll
        for (int k = 0; k < M; k++) {
            G = G * fa[k];
            cst[(2 * STAGES + 2 + k) * TG + t] = G;
        }
#pragma unroll
        for (int s = 0; s < STAGES; s++) {
            const double Gp = shfl_up(G, 1 << s);
            cst[s * TG + t] = lane >= (1 << s) ? G : 0.0;
            if (lane >= (1 << s)) G = G * Gp;
        }
        double Gx = shfl_up(G, 1);
        cst[STAGES * TG + t] = lane == 0 ? 1.0 : Gx;
        if (lane == WARP - 1) fold[wl] = G;
        double H = 1.0;
#pragma unroll
        for (int k = M - 1; k >= 0; k--) {
            H = H * fb[k];
            cst[(2 * STAGES + 2 + M + k) * TG + t] = H;
        }
#pragma unroll
        for (int s = 0; s < STAGES; s++) {
            const double Hn = shfl_down(H, 1 << s);
            cst[(STAGES + 1 + s) * TG + t] = lane + (1 << s) < WARP ? H : 0.0;
            if (lane + (1 << s) < WARP) H = H * Hn;
        }
        double Hx = shfl_down(H, 1);
        cst[(2 * STAGES + 1) * TG + t] = lane == WARP - 1 ? 1.0 : Hx;
        if (lane == 0) fold[NW + wl] = H;
    }
    // scan stages whose factors are all at most 2^-80 are left out
    int ks = 0, hs = 0;
    if (act) {
        const double tiny = 0x1p-80;
#pragma unroll
        for (int s = 0; s < STAGES; s++) {
            if (__any_sync(0xffffffffu, fabs(cst[s * TG + t]) > tiny)) ks = s + 1;
            if (__any_sync(0xffffffffu, fabs(cst[(STAGES + 1 + s) * TG + t]) > tiny)) hs = s + 1;
        }
    }
    // halo lines: version 0, and version -1 (ghost columns; block 0: the stored ghost row 0).
    // hm1: line j0-1 (ADJ: j1+2, even), hm2: line j0-2 (ADJ: j1+1, odd)
    const int jm1 = wrap(j0 - 1), j1 = j0 + nl - 1;
    const int je = ADJ ? wrap(j1 + 2) : jm1, jo = ADJ ? wrap(j1 + 1) : j0 - 2;
    for (int q = threadIdx.x; q < 3 * LW; q += blockDim.x) hm2[q] = 0.0;
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int w = (e % M) * TG + e / M;
        hm1[w] = sys.X[IDX(e + 1, je)];
        if (!ADJ && j0 == 1) hm1[2 * LW + w] = sys.X[IDX(e + 1, 0)];
        if (jo >= 1) hm2[w] = sys.X[IDX(e + 1, jo)];
    }
    if (!ADJ && threadIdx.x == 0) {
        if (j0 != 1) hm1[2 * LW] = sys.X[IDX(0, jm1)];
        if (jo >= 1) hm2[2 * LW] = sys.X[IDX(0, jo)];
    }
    // groups that poll the halo lines of the cross term for themselves
    const int ge = ADJ ? nl - 1 : 1, go = ADJ ? nl - 2 : 0;
    double hal[M];   // group 0: line j0-1; the last group: line j1+1
#pragma unroll
    for (int k = 0; k < M; k++) hal[k] = 0.0;
    if (act && g == 0) {
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int e = t * M + k;
            if (e < n) hal[k] = sys.X[IDX(e + 1, jm1)];
        }
    }
    const double corner0 = ADJ ? 0.0 : sys.X[IDX(0, 0)];
    const unsigned cnt0 = d.XCNT[blockIdx.x];
    ulonglong2 *words = reinterpret_cast<ulonglong2 *>(d.XW);
    auto slot = [&](unsigned cnt, int q) { return words + (size_t(cnt & 1u) * L + (q - 1)) * LW; };
    ulonglong2 *psum = words + size_t(2) * L * LW;   // [2 slots][blocks][2]
    __syncthreads();

    // source of sweep m: DIVDT (g) minus the cross term of P^(m-1) (mu^(m-1))
    auto source = [&](int m, double (&out)[M]) {
        const int vr = (m + 2) % 3, vg = (m + 1) % 3;
        if (ADJ) {
            const double *self = line(vr, g);
            const double *row = g + 2 < nl ? line(vr, g + 2) : (odd ? hm2 : hm1) + size_t(vr) * LW;
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k;
                const int w = k + 2 < M ? (k + 2) * TG + t : (M >= 2 ? (k + 2 - M) * TG + t + 1 : t + 2);   // element e+2
                const double p0 = self[k * TG + t], pp = row[k * TG + t];
                const double q0 = e + 2 < n ? self[w] : 0.0, qp = e + 2 < n ? row[w] : 0.0;
                double x = e < n ? pois_source(dv[k], c1[k], p0, c2[k], pp, c3[k], q0, c4[k], qp) : 0.0;
                if (e == 0 && n > 1) {
                    const int w1 = M >= 2 ? TG : 1;   // element 1
                    x = fma_rn(-w6, row[w1], fma_rn(-w5, self[w1], x));
                }
                out[k] = x;
            }
            return;
        }
        const double *self = line(vr, g), *row;
        double gs = line(vg, g)[0], gr;
        if (g >= 2) {
            row = line(vr, g - 2);
            gr = line(vg, g - 2)[0];
        } else if (g == 0) {
            row = hm2 + size_t(vr) * LW;
            gr = hm2[size_t(vg) * LW];
        } else if (j0 == 1) {   // line 2: the ghost row 0
            row = hm1 + size_t(vg) * LW;
            gr = m == 1 ? corner0 : row[0];
        } else {
            row = hm1 + size_t(vr) * LW;
            gr = hm1[size_t(vg) * LW];
        }
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int e = t * M + k;
            const int w = k >= 2 ? (k - 2) * TG + t : (M >= 2 ? (k - 2 + M) * TG + t - 1 : t - 2);   // element e-2
            const double p0 = self[k * TG + t], pm = row[k * TG + t];
            const double q0 = e >= 2 ? self[w] : gs, qm = e >= 2 ? row[w] : gr;
            out[k] = e < n ? pois_source(dv[k], c1[k], p0, c2[k], pm, c3[k], q0, c4[k], qm) : 0.0;
        }
    };
    // the line solve of v (group_apply_r with the constant products from shared memory)
    auto solve = [&]() {
        double y = 0.0;
#pragma unroll
        for (int k = 0; k < M; k++) {
            y = fma_rn(fa[k], y, mul_rn(fi[k], v[k]));
            v[k] = y;
        }
#pragma unroll
        for (int s = 0; s < STAGES; s++)
            if (s < ks) y = fma_rn(cst[s * TG + t], shfl_up(y, 1 << s), y);
        double in = shfl_up(y, 1);
        if (lane == 0) in = 0.0;
        if (NW > 1) {
            if (lane == WARP - 1) fold[2 * NW + wl] = y;
            bar();
            double yw = 0.0;
            for (int q = 0; q < wl; q++) yw = fma_rn(fold[q], yw, fold[2 * NW + q]);
            in = fma_rn(cst[STAGES * TG + t], yw, in);
        }
#pragma unroll
        for (int k = 0; k < M; k++) v[k] = fma_rn(cst[(2 * STAGES + 2 + k) * TG + t], in, v[k]);
        double x = 0.0;
#pragma unroll
        for (int k = M - 1; k >= 0; k--) {
            x = fma_rn(fb[k], x, v[k]);
            v[k] = x;
        }
#pragma unroll
        for (int s = 0; s < STAGES; s++)
            if (s < hs) x = fma_rn(cst[(STAGES + 1 + s) * TG + t], shfl_down(x, 1 << s), x);
        in = shfl_down(x, 1);
        if (lane == WARP - 1) in = 0.0;
        if (NW > 1) {
            if (lane == 0) fold[3 * NW + wl] = x;
            bar();
            double xw = 0.0;
            for (int q = NW - 1; q > wl; q--) xw = fma_rn(fold[NW + q], xw, fold[3 * NW + q]);
            in = fma_rn(cst[(2 * STAGES + 1) * TG + t], xw, in);
        }
#pragma unroll
        for (int k = 0; k < M; k++) v[k] = fma_rn(cst[(2 * STAGES + 2 + M + k) * TG + t], in, v[k]);
    };
    auto publish = [&](int m) {
        ulonglong2 *dst = slot(cnt0 + unsigned(m), j);
#pragma unroll
        for (int k = 0; k < M; k++)
            if (t * M + k < n) st_words(dst + k * TG + t, v[k], cnt0 + unsigned(m));
    };
    // line q of sweep v; flag: what s_fault tells of the wait
    auto wait_into = [&](int kind, int flag, int q, int v, double (&x)[M]) {
        const unsigned tag = cnt0 + unsigned(v);
        if (!poll_line<M, TG>(slot(tag, q), t, n, tag + waits.skew[kind - 1], waits.max_polls, x)) s_fault[flag] = 1;
    };
    auto wait_line = [&](int kind, int flag, int q, int v) { wait_into(kind, flag, q, v, hal); };

    if (act && odd) source(1, su);
    int m = 0, have = 0;   // sweeps done; have: group 0's halo already holds version m
    const int per = mode ? count : sys.per;
    double resip = 0.0;
    bool bad = false;
    for (int round = 0;; round++) {
        for (int s = 0; s < per; s++) {
            m++;
            const int vr = (m + 2) % 3, vw = m % 3;
            if (act) {
                if (odd) {
                    if (g == 0 && m > 1 && !have) wait_line(WAIT_ODD, m & 1, jm1, m - 1);
                    const double *pn = line(vr, g + 1), *ps = g == 0 ? nullptr : line(vr, g - 1);
#pragma unroll
                    for (int k = 0; k < M; k++) {
                        const double lo = g == 0 ? hal[k] : ps[k * TG + t];
                        v[k] = t * M + k < n ? pois_rhs(an[k], pn[k * TG + t], as[k], lo, su[k]) : 0.0;
                    }
                    solve();
#pragma unroll
                    for (int k = 0; k < M; k++) line(vw, g)[k * TG + t] = v[k];
                    if (g == 0 || (!ADJ && g == nl - 2)) publish(m);
                } else {
                    if (ADJ && have) {
                        // the residual has formed this sweep's source
                    } else {
                    if (g == ge && m > 1) {
                        double x[M];
#pragma unroll
                        for (int k = 0; k < M; k++) x[k] = 0.0;
                        wait_into(WAIT_ODD, m & 1, je, m - 1, x);
#pragma unroll
                        for (int k = 0; k < M; k++) hm1[size_t(vr) * LW + k * TG + t] = x[k];
                        bar();
                    }
                    source(m, su);
                    }
                }
            }
            have = 0;
            __syncthreads();
            if (act) {
                if (!odd) {
                    if (g == nl - 1) wait_line(WAIT_EVEN, m & 1, wrap(j + 1), m);
                    const double *pn = g == nl - 1 ? nullptr : line(vw, g + 1), *ps = line(vw, g - 1);
#pragma unroll
                    for (int k = 0; k < M; k++) {
                        const double hi = g == nl - 1 ? hal[k] : pn[k * TG + t];
                        v[k] = t * M + k < n ? pois_rhs(an[k], hi, as[k], ps[k * TG + t], su[k]) : 0.0;
                    }
                    solve();
#pragma unroll
                    for (int k = 0; k < M; k++) line(vw, g)[k * TG + t] = v[k];
                    if (g == nl - 1 || (ADJ && g == 1)) publish(m);
                } else {
                    if (g == go && jo >= 1) {
                        double x[M];
#pragma unroll
                        for (int k = 0; k < M; k++) x[k] = 0.0;
                        wait_into(WAIT_EVEN, m & 1, jo, m, x);
#pragma unroll
                        for (int k = 0; k < M; k++) hm2[size_t(vw) * LW + k * TG + t] = x[k];
                        bar();
                    }
                    if (s + 1 < per) source(m + 1, su);
                    else source(m + 1, sun);
                }
            }
            __syncthreads();
            if (s_fault[m & 1]) { bad = true; break; }   // uniform: next written after another barrier
        }
        if (bad || mode) break;
        // scaled-L1 residual of P^m with the last sweep's source (of mu^m with its own)
        const int vw = m % 3;
        double ra = 0.0, pa = 0.0;
        if (act) {
            if (ADJ) {
                if (odd) {
#pragma unroll
                    for (int k = 0; k < M; k++) su[k] = sun[k];
                } else {
                    if (g == ge) {
                        double x[M];
#pragma unroll
                        for (int k = 0; k < M; k++) x[k] = 0.0;
                        wait_into(WAIT_RES, 2, je, m, x);
#pragma unroll
                        for (int k = 0; k < M; k++) hm1[size_t(vw) * LW + k * TG + t] = x[k];
                        bar();
                    }
                    source(m + 1, su);
                }
            }
            double ae[M], aw[M], ap[M];
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k, c = IDX(e + 1, j);
                ae[k] = e < n ? sys.AE[c] : 0.0;
                aw[k] = e < n ? sys.AW[c] : 0.0;
                ap[k] = e < n ? sys.AP[c] : 0.0;
            }
            if (g == 0) wait_line(WAIT_RES, 2, jm1, m);
            const double *self = line(vw, g);
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k;
                if (e >= n) continue;
                const double pe = e + 1 < n ? (k + 1 < M ? self[(k + 1) * TG + t] : self[t + 1]) : 0.0;
                const double pw = e > 0 ? (k > 0 ? self[(k - 1) * TG + t] : self[(M - 1) * TG + t - 1]) : 0.0;
                const double pn = g == nl - 1 ? hal[k] : line(vw, g + 1)[k * TG + t];
                const double ps = g == 0 ? hal[k] : line(vw, g - 1)[k * TG + t];
                pois_resid(ae[k], pe, aw[k], pw, an[k], pn, as[k], ps, su[k], ap[k], v[k], ra, pa);
            }
            if (!ADJ && odd) {
#pragma unroll
                for (int k = 0; k < M; k++) su[k] = sun[k];
            }
            line_sum2<NW>(ra, pa, fold + 2 * NW, fold + 3 * NW, t, bar);
            if (t == 0) {
                s_line[2 * g] = ra;
                s_line[2 * g + 1] = pa;
            }
        }
        have = 1;
        __syncthreads();
        const unsigned rtag = cnt0 + unsigned(m);
        ulonglong2 *ps = psum + size_t(round & 1) * 2 * gridDim.x;
        if (threadIdx.x == 0 && !s_fault[2]) {   // without its lines the block has no sums
            pairs_sum2(s_line, nl, ra, pa);
            st_words(ps + 2 * blockIdx.x, ra, rtag);
            st_words(ps + 2 * blockIdx.x + 1, pa, rtag);
        }
        for (int q = threadIdx.x; q < 2 * (int)gridDim.x; q += blockDim.x) {
            bool got = false;
            const unsigned want = rtag + waits.skew[WAIT_SUMS - 1];
            for (int it = 0; !got && it < waits.max_polls; it++) {
                unsigned long long a, b;
                ld_words(ps + q, a, b);
                got = unsigned(a >> 32) == want && unsigned(b >> 32) == want;
                if (got) s_tot[q] = of_words(a, b);
            }
            if (!got) s_fault[2] = 1;
        }
        __syncthreads();
        if (threadIdx.x < WARP) {
            blocks_sum2([&](int q) { return s_tot[q]; }, gridDim.x, ra, pa);
            if (threadIdx.x == 0) {
                s_res = ADJ && !(pa > 0.0) ? 0.0 : ra / pa;
                s_nf = !(isfinite(ra) && isfinite(pa));
            }
        }
        __syncthreads();
        if (s_fault[2]) { bad = true; break; }
        resip = s_res;
        if (!(resip > d.resimax && m < d.nswpp)) break;
    }
    if (bad) {
        if (threadIdx.x == 0) {
            sys.pctl->fault = 1;
            sys.pctl->done = 1;
        }
        return;
    }
    if (act && !mode) {
        // a value that is not finite fills its line, as in a solve with every stage
        if (s_nf) {
            bool nf = false;
#pragma unroll
            for (int k = 0; k < M; k++) nf = nf || (t * M + k < n && !isfinite(v[k]));
            nf = __any_sync(0xffffffffu, nf);
            if (NW > 1) {
                if (lane == 0) fold[2 * NW + wl] = nf ? 1.0 : 0.0;
                bar();
#pragma unroll
                for (int q = 0; q < NW; q++) nf = nf || fold[2 * NW + q] != 0.0;
            }
#pragma unroll
            for (int k = 0; k < M; k++)
                if (nf) v[k] = __longlong_as_double(0x7ff8000000000000ll);
        }
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int e = t * M + k;
            if (e < n) sys.X[IDX(e + 1, j)] = v[k];
        }
    }
    if (threadIdx.x == 0) {
        d.XCNT[blockIdx.x] = cnt0 + unsigned(m);
        if (blockIdx.x == 0 && !mode) {
            sys.pctl->niter = m;
            sys.pctl->resip = resip;
            sys.pctl->capped = resip > d.resimax ? 1 : 0;
            sys.pctl->done = 1;
        }
    }
}

}  // namespace

int ring_pairs(const fvm_ctx *c)
{
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->p.device) != cudaSuccess || sms < 1) return 1;
    const int room = std::min(sms, RING_MAX_BLOCKS);
    return ((c->NJ - 1) / 2 + room - 1) / room;
}

// Ring layout of a context: pairs of lines per block so that every block has an SM of
// its own.  d.ring_ppb (also the grouping of the residual sums in the per-colour path) is
// set for every FP64 context; c->ring_blocks != 0 where the ring runs: the reference's
// positional cross term, poisson_resident not 0, and blocks that fit.
int ring_setup(fvm_ctx *c)
{
    c->ring_blocks = 0;
    const int pairs = (c->NJ - 1) / 2;
    int sms = 0;
    FVM_CUDA(c, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->p.device));
    const int ppb = ring_pairs(c), nb = (pairs + ppb - 1) / ppb;
    c->d.ring_ppb = ppb;
    c->d.nblk_res64 = c->nblk_res64 = nb;
    if (c->p.precision != FVM_FP64 || !c->d.dd_pos || c->p.poisson_resident == 0 || ppb > 2 || nb < 2) return FVM_OK;
    const LineSys &s = c->d.sP;
    int per_sm = 0;
    cudaError_t e = cudaSuccess;
    const bool ok = dispatch_line(s, [&](auto m, auto nw) {
        constexpr int M_ = decltype(m)::value, NW_ = decltype(nw)::value;
        using Lay = RingLayout<M_, NW_>;
        auto k = k_ring64<M_, NW_, 0>;
        auto ka = k_ring64<M_, NW_, 1>;
        // set outside any capture, to the largest block's need, the same for every context
        int most = 0;
        for (int nl : {2, 4})
            if (Lay::bytes(nl) <= 220 * 1024) most = (int)Lay::bytes(nl);
        if ((int)Lay::bytes(2 * ppb) > most) return;
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(ka, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 2 * ppb * Lay::TG, Lay::bytes(2 * ppb));
    });
    if (e != cudaSuccess) cudaGetLastError();
    if (ok && e == cudaSuccess && per_sm >= 1 && nb <= sms) c->ring_blocks = nb;
    return FVM_OK;
}

namespace {
template <int ADJ>
int launch(fvm_ctx *c, const RingSys &sys, int mode, int count, int max_polls, int skewed)
{
    cudaError_t e = cudaErrorInvalidValue;
    dispatch_line(c->d.sP, [&](auto m, auto nw) {
        constexpr int M_ = decltype(m)::value, NW_ = decltype(nw)::value;
        using Lay = RingLayout<M_, NW_>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c->ring_blocks);
        cfg.blockDim = dim3(2 * c->d.ring_ppb * Lay::TG);
        cfg.dynamicSmemBytes = Lay::bytes(2 * c->d.ring_ppb);
        cfg.stream = c->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, k_ring64<M_, NW_, ADJ>, c->d, sys, c->d.ring_ppb, mode, count,
                               waits_of(max_polls > 0 ? max_polls : kRingPolls, skewed));
    });
    if (e != cudaSuccess) {
        if (launch_refused(e)) c->ring_blocks = 0;
        c->err = std::string("Poisson ring launch: ") + cudaGetErrorString(e);
        return FVM_ERR_CUDA;
    }
    KCOUNT(c);
    return FVM_OK;
}
}  // namespace

// The FP64 Poisson iteration of a context whose source term is in place (mode 0), or
// `count` sweeps on chip (mode 1).  Cooperative: all blocks resident at once.  max_polls 0: the
// default bound of a wait.
int ring_launch(fvm_ctx *c, int mode, int count, int max_polls, int skewed)
{
    const Dev &d = c->d;
    return launch<0>(c, RingSys{d.sP.invD, d.sP.fa, d.sP.fb, d.cP.AN, d.cP.AS, d.cP.AE, d.cP.AW, d.cP.AP, d.DIVDT, d.P, d.pctl,
                                d.res_every}, mode, count, max_polls, skewed);
}

// The adjoint's transposed equation, its factors in the layout of the radial tile.
int ring_launch_adjoint(fvm_ctx *c, const RingSys &sys, int max_polls, int skewed)
{
    return launch<1>(c, sys, 0, 0, max_polls, skewed);
}

}  // namespace fvm
