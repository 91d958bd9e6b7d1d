// gmres.cuh -- one inner step's modified Gram-Schmidt of GMRES in one launch
// (included by solver.cu after the GMRES phases and persist.cuh).
//
// As phases, pass k of inner step i (GmMgs: w -= h v_{k-1}, h = w.v_k) is a
// row kernel and a finalize, i + 2 of them and a scaling per step: on a 96^3
// grid 13 and 4.5 us a pass, 28 MB through the L2 each, half of a
// GMRES(30) + ILU(0) solve.  Here a cooperative launch, one CTA per SM, holds
// w in shared memory for all passes, and v_k from its dot product to the
// update that follows it, so a pass reads one vector once, its loads issued
// before the grid barrier of the pass before.  What bounds a pass then is the
// FP64 pipe (two multiply-adds a row: 2.8 us on 96^3) and one grid barrier
// with the sum of the partials behind it (about 2.5 us).  96^3, GMRES(30) +
// ILU(0): 77 -> 57 ms (8.5 us a pass).
//
// The partial sums are the row tiles' and their orders are the phases'
// (block_reduce, then system_sum), so the results are the same bits.
#pragma once

namespace mtjg {

struct GmOrth {
    double *w;
    const double *V;   // the basis, vectors of n rows
    size_t n;
    int i;             // inner step
    bool write_w;      // w itself is read again (SSOR starts from its output's content)
    TileArgs rt;
    GmData g;
    MonPtrs m;
    double *part;
    unsigned long long *bar;  // arrivals, arrivals before this launch, abort
    int *err;
};

constexpr int kOrthBlock = 1024;  // four sub-blocks of kBlock threads, a row tile at a time each
constexpr int kOrthSub = kOrthBlock / kBlock;

namespace {

// kBlock values summed in block_reduce's order by one warp; valid in lane 0
__device__ __forceinline__ double tile_sum(const double *v, int lane)
{
    double s = v[lane];
#pragma unroll
    for (int k = 32; k < kBlock; k += 32) s += v[lane + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    return s;
}

// Q rows of a tile per thread, J tiles per sub-block
template <bool S, int Q, int J>
__global__ void __launch_bounds__(kOrthBlock, 1) k_gm_orth(GmOrth a)
{
    constexpr int R = Q * J;
    constexpr bool kKeepV = R <= 8;  // 128 KB of shared memory for w and v; with 16 rows w alone takes that
    extern __shared__ double dyn[];
    double *ws = dyn, *vs = dyn + (size_t)R * kOrthBlock;  // [R][kOrthBlock]
    __shared__ double red[J][kOrthBlock], s_sum;
    const int tid = threadIdx.x, sub = tid / kBlock, t = tid % kBlock, lane = tid & 31, warp = tid >> 5;
    const int G = (int)gridDim.x, NT = a.rt.num_tiles;
    SysState &st = a.m.st[0];
    if (st.gate != ST_RUNNING) return;
    unsigned long long target = a.bar[1];
    const GridBar gb{a.bar, reinterpret_cast<int *>(a.bar + 2)};
    const int ld = a.g.restart + 1, i = a.i;
    double *Hc = a.g.H + (size_t)i * ld;
    // this thread's rows: row[u], u = j Q + q, or none (-1)
    int row[R];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int tile = (int)blockIdx.x + G * (sub + kOrthSub * j);
        const int r0 = tile < NT ? a.rt.tile_row[tile] : 0, r1 = tile < NT ? a.rt.tile_row_end[tile] : 0;
#pragma unroll
        for (int q = 0; q < Q; ++q) row[j * Q + q] = r0 + t + q * kBlock < r1 ? r0 + t + q * kBlock : -1;
    }
    double vk[R];
#pragma unroll
    for (int u = 0; u < R; ++u) {
        ws[u * kOrthBlock + tid] = row[u] >= 0 ? a.w[row[u]] : 0.0;
        vk[u] = row[u] >= 0 ? __ldg(a.V + row[u]) : 0.0;
    }
    double h = 0.0;
    for (int k = 0; k <= i + 1; ++k) {
        const bool upd = k > 0 && -h != 0, dot = k <= i;
        const double *vp = a.V + (size_t)(k > 0 ? k - 1 : 0) * a.n;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            double acc = 0.0;
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int u = j * Q + q, at = u * kOrthBlock + tid;
                double wr = ws[at];
                if (upd) {
                    const double v = kKeepV ? vs[at] : row[u] >= 0 ? __ldg(vp + row[u]) : 0.0;
                    wr = fmac<S>(-h, v, wr);
                    ws[at] = wr;
                }
                acc = fmac<S>(wr, dot ? vk[u] : wr, acc);
                if (kKeepV) vs[at] = vk[u];
            }
            red[j][tid] = acc;
        }
        if (k + 1 <= i) {  // the next pass's vector, on its way across the barrier
            const double *vn = a.V + (size_t)(k + 1) * a.n;
#pragma unroll
            for (int u = 0; u < R; ++u) vk[u] = row[u] >= 0 ? __ldg(vn + row[u]) : 0.0;
        }
        __syncthreads();
        // the tiles' partials, in one of two places by turns (a slow CTA may
        // still read the last pass's)
        const int slot = 2 + (k & 1);
        if (warp < kOrthSub * J) {
            const int j = warp / kOrthSub, sb = warp % kOrthSub;
            const int tile = (int)blockIdx.x + G * (sb + kOrthSub * j);
            const double s = tile_sum(&red[j][sb * kBlock], lane);
            if (lane == 0 && tile < NT) a.part[(size_t)tile * kParts + slot] = s;
        }
        target += (unsigned long long)G;
        if (!grid_barrier(gb, target, a.err)) return;
        if (tid < kBlock) {  // system_sum
            double s = 0.0;
            for (int base = tid; base < NT; base += 4 * kBlock) {
                double o[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int q = base + u * kBlock;
                    o[u] = q < NT ? a.part[(size_t)q * kParts + slot] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (base + u * kBlock < NT) s += o[u];
            }
            red[0][tid] = s;
        }
        __syncthreads();
        if (warp == 0) {
            const double s = tile_sum(red[0], lane);
            if (lane == 0) s_sum = s;
        }
        __syncthreads();
        h = s_sum;
        if (dot && blockIdx.x == 0 && tid == 0) Hc[k] = h;
    }
    const double al = 1. / sqrt(h);  // v_{i+1} = w / h_{i+1,i}
    double *vn = const_cast<double *>(a.V) + (size_t)(i + 1) * a.n;
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const double wr = ws[u * kOrthBlock + tid];
        if (row[u] >= 0) {
            vn[row[u]] = al == 0 ? 0.0 : al * wr;
            if (a.write_w) a.w[row[u]] = wr;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.bar[1] = target;
        GmMgs<S> last{a.w, nullptr, nullptr, i, i + 1, a.m, a.g};
        Acc s;
        acc_zero(s);
        s.v[2] = h;
        last.scalar(0, s);
    }
}

// The launch's grid; 0 when the rows do not fit (the phases run instead).
template <bool S>
struct OrthPlan {
    void (*kernel)(GmOrth) = nullptr;
    int grid = 0;
    size_t smem = 0;
};

template <bool S>
OrthPlan<S> orth_plan(mtjg_ctx *ctx, const TileSet &rt)
{
    OrthPlan<S> p;
    int coop = 0, blocks = 0;
    if (rt.num_tiles == 0 || rt.num_groups != rt.num_tiles || rt.num_sys != 1) return p;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess || !coop) return p;
    const int G = std::min(rt.num_tiles, ctx->num_sms);
    const int J = (rt.num_tiles + G * kOrthSub - 1) / (G * kOrthSub);
    // every tile but the last is as long as the first
    const int Q = rt.h_tile_row[1] - rt.h_tile_row[0] > kRowTile ? kRowTileRows / kBlock : kRowTile / kBlock;
    static_assert(kRowTile == 4 * kBlock && kRowTileRows == 8 * kBlock, "rows of a tile per thread");
    if (J > 2) return p;
    auto k = Q == 4 ? (J == 1 ? k_gm_orth<S, 4, 1> : k_gm_orth<S, 4, 2>) : (J == 1 ? k_gm_orth<S, 8, 1> : k_gm_orth<S, 8, 2>);
    const size_t smem = sizeof(double) * (size_t)kOrthBlock * Q * J * (Q * J <= 8 ? 2 : 1);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, kOrthBlock, smem) != cudaSuccess) {
        (void)cudaGetLastError();
        return p;
    }
    if ((int64_t)blocks * ctx->num_sms < G) return p;
    p.kernel = k;
    p.grid = G;
    p.smem = smem;
    return p;
}

}  // namespace
}  // namespace mtjg
