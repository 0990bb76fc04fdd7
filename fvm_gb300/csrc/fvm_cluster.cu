// fvm_cluster.cu -- the mixed Poisson iteration of a batch, one thread-block cluster per
// case (iter_p.f90:12-51, lisolv.f90:18-33, bcp.f90:8-42 in defect correction, as
// fvm_mixed.cu).
//
// The batched path launched one grid over all cases per zebra colour (two per sweep), and
// each launch read every operand from L2 again: 7.4 us a launch for 64 cases, most of it
// launch latency and dependent L2 round trips.  The cases are independent, so here a
// cluster of 8 or 16 blocks keeps one case's FP32 factors, couplings, residual and
// correction in shared memory for the whole iteration; boundary lines and residual sums
// travel through distributed shared memory, and the only waits are the cluster's own
// hardware barriers (about 480 cycles with 512 threads).  Clusters need not run at the
// same time; a case leaves when it has converged.
//
// A block owns nl consecutive lines j0 .. j0+nl-1 (j0 odd, whole groups of four lines, the
// groups of the residual sums).  Odd lines are solved, the first one is also stored into
// the previous block's upper halo; barrier; even lines, the last one also into the next
// block's lower halo; barrier.  After an interval the owners add the correction to P in
// global memory with the BCP ghosts; barrier; the residual is k_mres's, term for term and
// sum for sum, from a double-float split of P in shared memory.  The arithmetic of a line
// is k_pois32's, so the results are the per-colour path's bit for bit.
//
// Operands sit in shared memory rather than in registers so that two blocks of 512 threads
// fit an SM for up to 16 lines of 192 cells a block (the south coupling of a line is the north coupling
// of the line below: the operator is symmetric): one block's barrier hides behind the
// other's solves (operands in registers, one block per SM: 8 % slower).  Measured: 64 ragged
// cases of 64..256 x 48..192 cells, two steps of 512 sweeps with their transfers, 44.9 -> 27.2
// ms; 64 cases, 2048 sweeps, 35.4 -> 24.4 ms a step.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "fvm_internal.cuh"
#include "fvm_ops.cuh"
#include "fvm_df.cuh"

namespace cg = cooperative_groups;

namespace fvm {
namespace {

constexpr int CT = 512;         // threads per block
constexpr size_t CLUSTER_SMEM = 220 * 1024;

// Blocks per case of L lines -- 16 (the most a cluster takes) where 8 would own more than
// 16 lines each and no longer fit an SM twice -- and lines per block.
inline __host__ __device__ int cluster_size(int L) { return L > 128 ? 16 : 8; }
inline __host__ __device__ int cluster_lines(int L) { return 4 * (((L + 3) / 4 + cluster_size(L) - 1) / cluster_size(L)); }

// Shared memory of a block: an (nl + 1 lines), fi, fa, fb, rf, x (nl lines each), two halo
// lines; sums; the split pressure of lines j0-2 .. j0+nl and of the ghost row 0.
template <int M, int NW>
struct CluLayout {
    static constexpr int TG = WARP * NW, LW = TG * M, G = CT / TG;
    static size_t bytes(int nl, int n)
    {
        const size_t f = size_t(6 * nl + 3) * LW, s = size_t(2) * nl * 16 + 2 * MRES_MAX_GROUPS + 3;
        return sizeof(float) * f + sizeof(double) * s + sizeof(float2) * size_t(nl + 4) * (n + 1);
    }
};

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int M, int NW>
__global__ void __launch_bounds__(CT, 2) k_cluster32(DevTable tab, const int *cases, int timed)
{
    using Lay = CluLayout<M, NW>;
    constexpr int TG = Lay::TG, LW = Lay::LW, G = Lay::G;
    extern __shared__ float shm[];
    __shared__ float xch[G][2 * NW];
    const Dev &d = tab.devs[cases[blockIdx.z]];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = blockIdx.x;
    const int L = d.NJ - 1, n = d.sP.n, per = cluster_lines(L), nb = (L + per - 1) / per;
    const int j0 = rank * per + 1, nl = max(0, min(per, L - rank * per));   // nl = 0: a block beyond the case's lines
    const int prev = rank == 0 ? nb - 1 : rank - 1, next = rank + 1 < nb ? rank + 1 : 0;
    const int PW = n + 1, nt = (n + WARP - 1) / WARP, ng = (L + MRES_GROUP - 1) / MRES_GROUP;
    float *an = shm;                               // [per + 1][LW]: row 0 is line j0-1
    float *sfi = an + size_t(per + 1) * LW, *sfa = sfi + size_t(per) * LW, *sfb = sfa + size_t(per) * LW;
    float *rf = sfb + size_t(per) * LW, *x = rf + size_t(per) * LW;
    float *lo = x + size_t(per) * LW, *hi = lo + LW;   // halos: line j0-1, line j0+nl
    double *s_w = reinterpret_cast<double *>(hi + LW);   // [2][per][16]
    double *s_tot = s_w + size_t(2) * per * 16;          // group sums of the case, ratio
    float2 *ps = reinterpret_cast<float2 *>(s_tot + 2 * MRES_MAX_GROUPS + 3);   // [per + 4][PW]
    float *hi_prev = cluster.map_shared_rank(hi, prev), *lo_next = cluster.map_shared_rank(lo, next);
    const int g = threadIdx.x / TG, t = threadIdx.x % TG;
    const int wid = threadIdx.x / WARP, lane = threadIdx.x & (WARP - 1);
    const NamedSync<NW> bar{1 + g};
    auto wrap = [L](int j) { return j < 1 ? j + L : (j > L ? j - L : j); };

    for (int q = g; q <= nl && nl > 0; q += G) {   // operands
        const int jn = wrap(j0 - 1 + q);
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int e = t * M + k;
            an[size_t(q) * LW + k * TG + t] = e < n ? d.cP.ANf[IDX(e + 1, jn)] : 0.0f;
        }
        if (q == nl) break;
#pragma unroll
        for (int k = 0; k < M; k++) rf[size_t(q) * LW + k * TG + t] = 0.0f;   // the padding stays zero
        const size_t base = size_t(j0 + q - 1) * LW;
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int w = k * TG + t;
            sfi[size_t(q) * LW + w] = d.sP.invDf[base + w];
            sfa[size_t(q) * LW + w] = d.sP.faf[base + w];
            sfb[size_t(q) * LW + w] = d.sP.fbf[base + w];
        }
    }
    cluster_barrier();   // every block has started: its shared memory may be written from now on
    const int S = timed ? timed : d.refine_sweeps;   // timed: one interval of so many sweeps, nothing written
    int it = 0;
    double resip = 0.0;
    for (;;) {
        // split pressure: row r holds line j0-2+r (wrapped), row per + 3 the ghost row 0
        for (int r = wid; r < nl + 3 && nl > 0; r += CT / WARP) {
            const double *row = d.P + IDX(0, wrap(j0 - 2 + r));
            for (int i = lane; i < PW; i += WARP) {
                const dd v = dd_split(__ldcg(row + i));
                ps[size_t(r) * PW + i] = make_float2(v.hi, v.lo);
            }
        }
        if (j0 == 1 && wid == CT / WARP - 1)
            for (int i = lane; i < PW; i += WARP) {
                const dd v = dd_split(__ldcg(d.P + IDX(i, 0)));
                ps[size_t(per + 3) * PW + i] = make_float2(v.hi, v.lo);
            }
        for (int q = threadIdx.x; q < (per + 2) * LW; q += CT) x[q] = 0.0f;   // correction and halos
        __syncthreads();
        // residual: one warp per line and 32 cells (k_mres's terms and order)
        for (int task = wid; task < nl * nt; task += CT / WARP) {
            const int q = task / nt, col = task - q * nt, i = col * WARP + lane + 1, j = j0 + q;
            const bool inside = i <= n, has_cross = inside && i > 1 && j > 1;
            const int c = inside ? IDX(i, j) : 0, cc = has_cross ? IDX(i - 1, j - 1) : 0;
            float2 cf[9];
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const bool ok = k < 5 ? inside : has_cross;
                cf[k] = ok ? d.PCD[size_t(k) * d.n + (k < 5 ? c : cc)] : make_float2(0.0f, 0.0f);
            }
            float raf = 0.0f, paf = 0.0f;
            if (inside) {
                const float2 *r0 = ps + size_t(q + 2) * PW, *rm = j == 2 ? ps + size_t(per + 3) * PW : r0 - 2 * PW;
                auto at = [](float2 v) { return dd(v.x, v.y); };
                auto co = [&](int k) { return at(cf[k]); };
                dd cross = dd(0.0f, 0.0f);
                if (has_cross)
                    cross = ((co(5) * at(r0[i]) + co(6) * at(rm[i])) + co(7) * at(r0[i - 2])) + co(8) * at(rm[i - 2]);
                const dd su = dd_split(d.DIVDT[c]) - cross;
                const dd app = co(4) * at(r0[i]);
                const dd pe = i < n ? at(r0[i + 1]) : dd(0.0f, 0.0f);   // AE(NI-1) = 0
                const dd r = ((((co(0) * pe + co(1) * at(r0[i - 1])) + co(2) * at(r0[PW + i])) + co(3) * at((r0 - PW)[i])) + su) - app;
                raf = fabsf(r.hi);
                paf = fabsf(app.hi);
                const int e = i - 1;
                rf[size_t(q) * LW + (e % M) * TG + e / M] = r.hi;
            }
            for (int o = 16; o > 0; o >>= 1) {
                raf += __shfl_down_sync(0xffffffffu, raf, o);
                paf += __shfl_down_sync(0xffffffffu, paf, o);
            }
            if (lane == 0) {
                s_w[q * 16 + col] = (double)raf;
                s_w[(per + q) * 16 + col] = (double)paf;
            }
        }
        // lines beyond the case in the last group of four add nothing
        for (int q = nl * 16 + threadIdx.x; q < ((nl + 3) & ~3) * 16; q += CT) s_w[q] = s_w[per * 16 + q] = 0.0;
        __syncthreads();
        for (int q = wid; 4 * q < nl; q += CT / WARP) {   // the sums of a group to every block of the cluster
            const int half = lane >> 4, col = lane & 15;
            const double v = mres_columns(col < nt ? mres_lines(s_w + size_t(half * per + 4 * q) * 16 + col, 16) : 0.0);
            if (col == 0)
                for (int r = 0; r < (int)gridDim.x; r++)
                    *cluster.map_shared_rank(s_tot + 2 * ((j0 - 1) / MRES_GROUP + q) + half, r) = v;
        }
        cluster_barrier();
        mres_ratio(s_tot, ng, s_tot + 2 * MRES_MAX_GROUPS, s_tot + 2 * MRES_MAX_GROUPS + 2);
        resip = s_tot[2 * MRES_MAX_GROUPS + 2];
        if (it > 0 && !(resip > d.resimax && it < d.nswpp)) break;
        for (int half = 0; half < 2 * S; half++) {   // colour 0: the odd lines q = 0, 2, ...
            const int colour = half & 1;
            for (int q = 2 * g + colour; q < nl; q += 2 * G) {
                const int o = q * LW + t;
                const float *xs = q > 0 ? x + o - LW : lo + t, *xn = q + 1 < nl ? x + o + LW : hi + t;
                float v[M], fi[M], fa[M], fb[M];
#pragma unroll
                for (int k = 0; k < M; k++) {   // padding: zero couplings, residual and factors
                    v[k] = pois32_rhs(an[o + LW + k * TG], xn[k * TG], an[o + k * TG], xs[k * TG], rf[o + k * TG]);
                    fi[k] = sfi[o + k * TG];
                    fa[k] = sfa[o + k * TG];
                    fb[k] = sfb[o + k * TG];
                }
                group_apply_r<float, M, NW>(v, fi, fa, fb, t, xch[g], bar);
#pragma unroll
                for (int k = 0; k < M; k++) x[o + k * TG] = v[k];
                if (q == 0)
#pragma unroll
                    for (int k = 0; k < M; k++) hi_prev[k * TG + t] = v[k];
                if (q == nl - 1)
#pragma unroll
                    for (int k = 0; k < M; k++) lo_next[k * TG + t] = v[k];
            }
            cluster_barrier();
        }
        if (timed) return;   // uniform over the cluster; nobody writes to another block after the last barrier
        it += S;
        // the correction added to P on the own lines, BCP ghosts of each line
        for (int q = g; q < nl; q += G) {
            const int j = j0 + q;
#pragma unroll
            for (int k = 0; k < M; k++) {
                const int e = t * M + k;
                if (e < n) {
                    double *p = d.P + IDX(e + 1, j);
                    *p = __ldcg(p) + f2d_int(x[size_t(q) * LW + k * TG + t]);
                }
            }
            bar();
            if (t < WARP) refresh_row_ghosts<BCK_POISSON>(d, d.P, d.P, j, nullptr, nullptr, t);
        }
        cluster_barrier();
    }
    if (rank == 0 && threadIdx.x == 0) {
        d.pctl->niter = it;
        d.pctl->resip = resip;
        d.pctl->capped = resip > d.resimax ? 1 : 0;
        d.pctl->done = 1;
    }
}

}  // namespace

// Shared memory a case needs in the tile of the batch; 0: no cluster form (the cell's own
// cross term, or more than a block holds).
size_t cluster_bytes(const fvm_ctx *c, const LineSys &tile)
{
    if (c->p.precision != FVM_MIXED || !c->d.dd_pos) return 0;
    size_t b = 0;
    dispatch_line(tile, [&](auto m, auto nw) {
        b = CluLayout<decltype(m)::value, decltype(nw)::value>::bytes(cluster_lines(c->NJ - 1), c->NI - 1);
    });
    return b <= CLUSTER_SMEM ? b : 0;
}

int cluster_blocks(const fvm_ctx *c) { return cluster_size(c->NJ - 1); }

namespace {
// f(kernel, launch configuration) for clusters of `blocks` blocks with `smem` bytes each,
// one per case.
template <class F>
cudaError_t with_cluster(const LineSys &tile, int blocks, size_t smem, int count, cudaStream_t st, F &&f)
{
    cudaError_t e = cudaErrorInvalidValue;
    dispatch_line(tile, [&](auto m, auto nw) {
        auto k = k_cluster32<decltype(m)::value, decltype(nw)::value>;
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLUSTER_SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks, 1, count);
        cfg.blockDim = dim3(CT);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = blocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        e = f(k, cfg);
    });
    return e;
}
}  // namespace

// Whether the device can hold such a cluster (16 blocks are more than it must offer).
bool cluster_fits(const LineSys &tile, int blocks, size_t smem)
{
    int most = 0;
    const cudaError_t e = with_cluster(tile, blocks, smem, 1, nullptr, [&](auto k, const cudaLaunchConfig_t &cfg) {
        return cudaOccupancyMaxActiveClusters(&most, k, &cfg);
    });
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && most >= 1;
}

// The iteration of the `count` cases listed in device memory, `blocks` blocks a case with
// `smem` bytes each; timed: one residual and that many sweeps, on chip only.
int cluster_launch(const Tgt &t, cudaStream_t st, const int *cases, int count, int blocks, size_t smem, int timed)
{
    const cudaError_t e = with_cluster(t.tr, blocks, smem, count, st, [&](auto k, const cudaLaunchConfig_t &cfg) {
        return cudaLaunchKernelEx(&cfg, k, t.tab, cases, timed);
    });
    if (e != cudaSuccess) {
        t.c->err = std::string("batched Poisson launch: ") + cudaGetErrorString(e);
        return FVM_ERR_CUDA;
    }
    KCOUNT(t.c);
    return FVM_OK;
}

}  // namespace fvm
