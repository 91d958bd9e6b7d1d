// lines.cu -- triangular sweeps by tiles of lines.
//
// A level-scheduled sweep hands every level's values through the L2: about
// 950 cycles from one SM's store to another's poll, on every level, so a
// 96^3 grid's 286 levels took 273 (L) and 361 us (U).  The rows of a grid in its
// natural order form lines (runs of consecutive rows, each reading the one
// before), and the lines form planes.  Here a CTA owns a tile of lines, one
// lane per line, and walks the levels: a value read inside the tile comes
// from shared memory one block barrier later, and only the tile's edges go
// through the L2, once per tile boundary on the longest path instead of once
// per level.  What bounds a sweep then is the arithmetic of one row per
// level: a warp's FP64 instruction holds its quarter of the SM for 64 cycles
// on GB300, whatever its active lanes, so an L step of three entries takes
// 4 x 64 cycles and the barrier, and a tile has 128 lanes (a warp on each
// quarter; the diagonal's reciprocal, made once with the factor, spares the
// U step the 563 cycles of an FP64 division).
//
// The sweeps' vectors are in plan order (the rows of one step next to each
// other), so that b arrives by bulk copies, a step's x leaves in whole
// sectors and the CTAs' polls touch few lines; one launch permutes b ahead of
// the first sweep and one takes x back after the second.
//
// Each row's operations and their order are those of the ticket sweep
// (precond.cu).  A CTA takes its rows in level order, waits on rows of lower
// levels only, and all CTAs run at once (a cooperative launch), so the sweep
// cannot deadlock: the lowest unfinished level is always free to run.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "lines.cuh"
#include "spmv.cuh"
#include "sweep.cuh"

namespace mtjg {

constexpr int kRing = 8;          // steps whose x a tile keeps in shared memory
constexpr int kLineK = 4;         // entries per row a record may hold
constexpr int kMinLine = 4;       // rows per line, on average, that make lines worth it
constexpr long long kLineSpin = 1LL << 22;

// Slots of the operand pipeline (steps ahead of the arithmetic) and loader
// warps; an FP32 step is some 150 cycles, an FP64 step 350 to 550, against
// about 1000 for a record from memory or a value from another SM.
template <class V>
struct LinePipe {
    static constexpr int kSlots = sizeof(V) == 8 ? 8 : 16;
    static constexpr int kLoaders = sizeof(V) == 8 ? 4 : 8;
};

// A record: kmax entry values, the diagonal and its reciprocal, the codes.
// The pivots of ILU(0) (MODE 6) take 2 kmax entry values instead.
template <class V>
__host__ __device__ constexpr int line_record(int kmax, int lanes)
{
    return lanes * ((kmax + 2) * (int)sizeof(V) + 16);
}
template <class V, int MODE>
__host__ __device__ constexpr int mode_record(int kmax, int lanes)
{
    return MODE == 6 ? lanes * (2 * kmax * (int)sizeof(V) + 16) : line_record<V>(kmax, lanes);
}
// Shared memory: the values a lane may read after a step's barrier -- the
// ring (kRing steps of x), a zero, the entries from other CTAs (kSlots steps)
// -- then kSlots slots of a record and b each.  An entry's code is the byte
// offset of its value in there.
template <class V>
__host__ __device__ constexpr int line_zero(int lanes) { return kRing * lanes * (int)sizeof(V); }
template <class V>
__host__ __device__ constexpr int line_remote(int kmax, int lanes, int s)  // step s of the sweep
{
    return line_zero<V>(lanes) + 16 + (s % LinePipe<V>::kSlots) * kmax * lanes * (int)sizeof(V);
}
template <class V>
__host__ __device__ constexpr int line_slots(int kmax, int lanes)
{
    return line_zero<V>(lanes) + 16 + LinePipe<V>::kSlots * kmax * lanes * (int)sizeof(V);
}
// MODE 6's values are pairs (a pivot and its reciprocal): everything before
// the slots takes twice the place, and a code counts twice.
template <class V, int MODE = 0>
constexpr int line_smem(int kmax, int lanes)
{
    return (MODE == 6 ? 2 : 1) * line_slots<V>(kmax, lanes) +
           LinePipe<V>::kSlots * (mode_record<V, MODE>(kmax, lanes) + lanes * (int)sizeof(V));
}

// What fits a CTA (227 KB, of which the kernel's own variables take little):
// a plan serves both precisions, so four entries of 256 lanes (FP32: 254 KB)
// are never planned; the pivots' sweep of 256 lanes holds two entries (280 KB
// for three), and a factor of more takes the elimination by levels.
constexpr int kLineSmem = 226 * 1024;
constexpr bool line_plan_fits(int kmax, int lanes)
{
    return line_smem<double>(kmax, lanes) <= kLineSmem && line_smem<float>(kmax, lanes) <= kLineSmem;
}
template <int MODE>
constexpr bool line_fits(int kmax, int lanes)
{
    return MODE == 6 ? line_smem<double, 6>(kmax, lanes) <= kLineSmem : line_plan_fits(kmax, lanes);
}

// ------------------------------------------------------------ the plan
__device__ __forceinline__ void tri_range(const TriOp &op, int i, int &b, int &e)
{
    b = op.range == 2 ? op.diag[i] + 1 : op.rp[i];
    e = op.range == 1 ? op.diag[i] : op.rp[i + 1];
}

// An entry (i, c) of `op` and its mirror (c, i) in `other`
__device__ __forceinline__ bool mirrored(const TriOp &op, const TriOp &other, int i, int &most)
{
    int b, e;
    tri_range(op, i, b, e);
    most = max(most, e - b);
    bool all = true;
    for (int k = b; k < e && e - b <= kLineK; ++k) {
        int b2, e2;
        tri_range(other, op.ci[k], b2, e2);
        bool found = false;
        for (int q = b2; q < e2 && e2 - b2 <= kLineK; ++q) found |= other.ci[q] == i;
        all &= found;
    }
    return all;
}

// A row that begins a line: its last entry is not the row before
__device__ __forceinline__ bool begins_line(const TriOp &op, int i)
{
    int b, e;
    tri_range(op, i, b, e);
    return !(e > b && op.ci[e - 1] == i - 1);
}

// count[0]: the longest row of both triangles, over kLineK where an entry has
// no mirror in the other triangle; count[1]: the lines (0 and 0 before)
__global__ void k_line_look(TriOp op, TriOp up, int *count)
{
    int most = 0, starts = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < op.n; i += gridDim.x * blockDim.x) {
        starts += begins_line(op, i);
        const bool down = mirrored(op, up, i, most), above = mirrored(up, op, i, most);
        if (!down || !above) most = max(most, kLineK + 1);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    starts = __reduce_add_sync(0xffffffffu, starts);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(count, most);
        atomicAdd(count + 1, starts);
    }
}

__global__ void k_line_start(TriOp op, int *start)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < op.n; i += gridDim.x * blockDim.x)
        start[i] = begins_line(op, i);
}

// line_of from the scan of start; each line's first row; pstart to 1
__global__ void k_line_of(int n, const int *start, const int *scan, int *line_of, int *first, int *pstart, int lines)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int l = scan[i] + start[i] - 1;
        line_of[i] = l;
        if (start[i]) first[l] = i, pstart[l] = 1;
        if (i == 0) first[lines] = n;
    }
}

// pstart[l] = 0 when line l continues line l - 1's plane: one of its rows
// reads that line (pstart is 1 before)
__global__ void k_plane_start(TriOp op, const int *line_of, int *pstart)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < op.n; i += gridDim.x * blockDim.x) {
        int b, e;
        tri_range(op, i, b, e);
        const int l = line_of[i];
        for (int k = b; k < e; ++k)
            if (line_of[op.ci[k]] == l - 1) pstart[l] = 0;
    }
}

// each plane's first line, the planes, and the most lines of a plane (0
// before); scan[lines]: the planes
__global__ void k_plane_first(int lines, const int *pstart, const int *scan, int *pfirst, int *planes)
{
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < lines; l += gridDim.x * blockDim.x) {
        if (pstart[l]) pfirst[scan[l]] = l;
        if (l == 0) {
            pfirst[scan[lines]] = lines;
            *planes = scan[lines];
        }
    }
}

__global__ void k_plane_long(const int *planes, const int *pfirst, int *longest)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < *planes; p += gridDim.x * blockDim.x)
        atomicMax(longest, pfirst[p + 1] - pfirst[p]);
}

// tiles of tq lines of a plane by tp planes
__global__ void k_line_tile(int lines, const int *pstart, const int *scan, const int *pfirst, int tq, int tp, int ntq,
                            int *part_of, int *lane_of)
{
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < lines; l += gridDim.x * blockDim.x) {
        const int p = scan[l] + pstart[l] - 1, q = l - pfirst[p];
        part_of[l] = (p / tp) * ntq + q / tq;
        lane_of[l] = (p % tp) * tq + q % tq;
    }
}

// Lines as nodes: row j of line l (counted from its first) takes step
// off[l] + j, so line l may not start before off[m] + w for each line m that
// it reads, w the largest of (place of the entry read) - (place of the row)
// + 1 over its rows.  dep: up to kLineK such (m, w) per line, m = -1 for none;
// *bad = 1 for a line that reads more.  One warp per line.
__global__ void k_line_deps(TriOp op, int lines, const int *line_of, const int *first, int2 *dep, int *bad)
{
    const int l = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (l >= lines) return;
    const int r0 = first[l], r1 = first[l + 1];
    int m[kLineK], w[kLineK];
#pragma unroll
    for (int k = 0; k < kLineK; ++k) m[k] = -1, w[k] = -0x40000000;
    int used = 0;
    bool over = false;
    for (int base = r0; base < r1; base += 32) {
        const int i = base + lane;
        int cl[kLineK], cw[kLineK], b = 0, e = 0;
        if (i < r1) tri_range(op, i, b, e);
#pragma unroll
        for (int k = 0; k < kLineK; ++k) {
            cl[k] = -1;
            if (b + k < e) {
                const int c = op.ci[b + k], lc = line_of[c];
                if (lc != l) cl[k] = lc, cw[k] = (c - first[lc]) - (i - r0) + 1;
            }
        }
        // one line read by any lane at a time
        for (;;) {
            int mine = -1;
#pragma unroll
            for (int k = kLineK - 1; k >= 0; --k)
                if (cl[k] >= 0) mine = cl[k];
            const unsigned any = __ballot_sync(0xffffffffu, mine >= 0);
            if (!any) break;
            const int t = __shfl_sync(0xffffffffu, mine, __ffs(any) - 1);
            int most = -0x40000000;
#pragma unroll
            for (int k = 0; k < kLineK; ++k)
                if (cl[k] == t) most = max(most, cw[k]), cl[k] = -1;
            most = __reduce_max_sync(0xffffffffu, most);
            bool found = false;
#pragma unroll
            for (int k = 0; k < kLineK; ++k)
                if (m[k] == t) w[k] = max(w[k], most), found = true;
            if (!found) {
                over |= used == kLineK;
#pragma unroll
                for (int k = 0; k < kLineK; ++k)
                    if (k == used) m[k] = t, w[k] = most;
                ++used;
            }
        }
    }
    if (lane == 0) {
        if (over) *bad = 1;
#pragma unroll
        for (int k = 0; k < kLineK; ++k) dep[(size_t)l * kLineK + k] = make_int2(m[k], w[k]);
    }
}

// The lowest offsets, in one block, each part's first and last step, and the
// parts' places one behind the other.
// Plane after plane: a line starts after the plane's line before it (a scan
// of the maps t -> max(b, t + a)) and after what it reads in earlier planes.
// Then rounds over all lines until none moves, which cover what the scan left
// out (a line reading its own plane's lines beyond the one before) and check
// the rest; a line reads earlier lines only, so the rounds end (*bad = 1 if
// not within `lines` rounds).  9216 lines in 96 planes: 634 us by rounds
// alone (415 us by a level search through the L2), 141 with the scans.  Many
// short planes (more than kScanPlanes) go by rounds.
constexpr int kOffsetBlock = 1024;
constexpr int kScanPlanes = 2048;
__global__ void __launch_bounds__(kOffsetBlock) k_line_offsets(int lines, int planes, const int *pfirst,
                                                               const int2 *dep, const int *first, const int *part_of,
                                                               int *off, int parts, int *lo, int *hi, int *part_step,
                                                               int *bad)
{
    extern __shared__ int s_off[];
    __shared__ int s_a[kOffsetBlock / 32], s_b[kOffsetBlock / 32];
    constexpr int kNone = -0x20000000;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int l = tid; l < lines; l += kOffsetBlock) s_off[l] = 0;
    for (int p = tid; p < parts; p += kOffsetBlock) lo[p] = 0x7fffffff, hi[p] = -1;
    __syncthreads();
    for (int p = 0; p < planes && planes <= kScanPlanes; ++p) {
        const int l0 = pfirst[p], l1 = pfirst[p + 1];
        int carry = kNone;  // the offset of the line before the chunk
        for (int base = l0; base < l1; base += kOffsetBlock) {
            const int l = base + tid;
            int A = kNone, B = 0;  // off = max(B, offset of line l - 1 + A)
            if (l < l1) {
                const int4 *d = reinterpret_cast<const int4 *>(dep + (size_t)l * kLineK);
                int4 q[kLineK / 2];
#pragma unroll
                for (int k = 0; k < kLineK / 2; ++k) q[k] = __ldg(d + k);
#pragma unroll
                for (int k = 0; k < kLineK; ++k) {
                    const int m = k & 1 ? q[k / 2].z : q[k / 2].x, w = k & 1 ? q[k / 2].w : q[k / 2].y;
                    if (m >= 0 && m == l - 1 && l > l0) A = w;
                    else if (m >= 0 && m < l0) B = max(B, s_off[m] + w);
                }
            } else {
                A = 0, B = kNone;  // the identity
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {  // inclusive scan of the maps, earlier lines first
                const int pa = __shfl_up_sync(0xffffffffu, A, o), pb = __shfl_up_sync(0xffffffffu, B, o);
                if (lane >= o) {
                    B = max(B, pb + A);
                    A = max(pa + A, kNone);
                }
            }
            if (lane == 31) s_a[warp] = A, s_b[warp] = B;
            __syncthreads();
            int t = carry;  // the offset before this warp's first line
            for (int w = 0; w < warp; ++w) t = max(s_b[w], t + s_a[w]);
            const int v = max(B, t + A);
            if (l < l1) s_off[l] = v;
            __syncthreads();
            if (base + kOffsetBlock < l1) carry = s_off[base + kOffsetBlock - 1];
        }
    }
    int round = 0;
    for (;; ++round) {
        bool moved = false;
        for (int l = tid; l < lines; l += kOffsetBlock) {
            const int2 *d = dep + (size_t)l * kLineK;
            const int was = ((volatile int *)s_off)[l];
            int v = was;
#pragma unroll
            for (int k = 0; k < kLineK; ++k) {
                const int2 q = __ldg(d + k);
                if (q.x >= 0) v = max(v, ((volatile int *)s_off)[q.x] + q.y);
            }
            if (v != was) {
                ((volatile int *)s_off)[l] = v;
                moved = true;
            }
        }
        if (!__syncthreads_or(moved) || round > lines) break;
    }
    if (round > lines && tid == 0) *bad = 1;
    for (int l = tid; l < lines; l += kOffsetBlock) {
        const int v = s_off[l];
        off[l] = v;
        atomicMin(lo + part_of[l], v);
        atomicMax(hi + part_of[l], v + first[l + 1] - first[l] - 1);
    }
    __syncthreads();
    if (tid == 0) {  // (a plan of more steps than an int holds is refused)
        long long step = 0;
        for (int p = 0; p < parts; ++p) {
            part_step[p] = (int)step;
            const int l = __ldcg(lo + p), h = __ldcg(hi + p);
            step = min(step + max(0, h - l + 1), 0x7fffffffLL);
        }
        part_step[parts] = (int)step;
    }
}

// each row's position, the row at each position (row is -1 before), and the
// parts' steps into the plan's own array
__global__ void k_line_place(int n, int lanes, const int *line_of, const int *first, const int *part_of,
                             const int *lane_of, const int *off, const int *part_min, int parts, const int *part_step,
                             int *pos, int *row, int *plan_step)
{
    if (blockIdx.x == 0)
        for (int p = threadIdx.x; p <= parts; p += blockDim.x) plan_step[p] = part_step[p];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int l = line_of[i], p = part_of[l];
        const int at = (part_step[p] + off[l] + (i - first[l]) - part_min[p]) * lanes + lane_of[l];
        pos[i] = at;
        row[at] = i;
    }
}

// The part that holds a step: part_step is ascending (binary search).
__device__ __forceinline__ int part_at(const int *part_step, int parts, int step)
{
    int lo = 0, hi = parts - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (part_step[mid] <= step) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The entry codes of every position (without a row every code is the zero's)
// and, with `rem`, the remote entries of each step: rem_max places a step,
// (-1, 0) before; cursor counts a step's entries, and *longest is raised to
// the count of a step that has more.
template <class V>
__global__ void k_line_codes(TriOp op, TilePlan tp, unsigned char *rec, int *cursor, int2 *rem, int rem_max,
                             int *longest)
{
    const int T = tp.lanes, K = tp.kmax, bytes = line_record<V>(K, T);
    for (int at = blockIdx.x * blockDim.x + threadIdx.x; at < tp.steps * T; at += gridDim.x * blockDim.x) {
        const int i = tp.row[at], step = at / T, lane = at % T;
        int code[kLineK];
        for (int k = 0; k < kLineK; ++k) code[k] = line_zero<V>(T);
        if (i >= 0) {
            const int part = part_at(tp.part_step, tp.parts, step);
            const int first = tp.part_step[part], last = tp.part_step[part + 1];
            // the step in the sweep's order
            auto order = [&](int s) { return op.desc ? last - 1 - s : s - first; };
            int b, e;
            tri_range(op, i, b, e);
            for (int k = 0; k < e - b; ++k) {
                const int c = tp.pos[op.ci[op.mode == 3 ? e - 1 - k : b + k]], cs = c / T;
                if (cs >= first && cs < last && order(step) - order(cs) < kRing) {
                    code[k] = ((order(cs) % kRing) * T + c % T) * (int)sizeof(V);
                } else {
                    code[k] = line_remote<V>(K, T, order(step)) + (k * T + lane) * (int)sizeof(V);
                    if (rem) {
                        const int q = atomicAdd(cursor + step, 1);
                        if (q < rem_max) rem[(size_t)step * rem_max + q] = make_int2(c, k * T + lane);
                        else atomicMax(longest, q + 1);
                    }
                }
            }
        }
        reinterpret_cast<int4 *>(rec + (size_t)step * bytes + (size_t)T * (K + 2) * sizeof(V))[lane] =
            make_int4(code[0], code[1], code[2], code[3]);
    }
}

// Whether a quotient by d may use its reciprocal (else it is kept as 0 and
// the quotient takes a real division).
__device__ __forceinline__ bool line_safe(double d)  // 2^-299 <= |d| < 2^300
{
    return (((unsigned)__double2hiint(d) >> 20) & 0x7ffu) - 724u <= 598u;
}
__device__ __forceinline__ bool line_safe(float d)  // 2^-40 <= |d| < 2^41
{
    return ((__float_as_uint(d) >> 23) & 0xffu) - 87u <= 80u;
}

// The values of every position: entries in the order the sweep adds them,
// the diagonal and its reciprocal (1 and 1 without a row).  A row with fewer
// entries is filled up with ones whose product with the zero is -0, which
// leaves every sum as it is.
template <class V>
__global__ void k_line_values(TriOp op, TilePlan tp, unsigned char *rec, const V *v, const V *diagv)
{
    const int T = tp.lanes, K = tp.kmax, bytes = line_record<V>(K, T);
    for (int at = blockIdx.x * blockDim.x + threadIdx.x; at < tp.steps * T; at += gridDim.x * blockDim.x) {
        const int i = tp.row[at], lane = at % T;
        V *rv = reinterpret_cast<V *>(rec + (size_t)(at / T) * bytes);
        int b = 0, e = 0;
        V d = V(1);
        if (i >= 0) {
            tri_range(op, i, b, e);
            if (op.mode == 1) d = v[op.diag[i]];
            if (op.mode == 2) d = diagv[i];
        }
        const V fill = op.mode >= 2 ? V(0) : -V(0);  // modes 2 and 3 subtract
        for (int k = 0; k < K; ++k) rv[k * T + lane] = k < e - b ? v[op.mode == 3 ? e - 1 - k : b + k] : fill;
        rv[K * T + lane] = d;
        rv[(K + 1) * T + lane] = line_safe(d) ? V(1) / d : V(0);
    }
}

// ------------------------------------------------------------ the sweeps
// b into plan order, and the two sweeps' outputs to pending.
template <class V>
__global__ void k_tile_in(int count, const int *row, const V *b, V *bp, V *yp, V *xp, const int *status)
{
    if (status && *status != ST_RUNNING) return;
    const V p = pending_value<V>();
    for (int at = blockIdx.x * blockDim.x + threadIdx.x; at < count; at += gridDim.x * blockDim.x) {
        const int i = row[at];
        bp[at] = i >= 0 ? b[i] : V(0);
        yp[at] = p;
        xp[at] = p;
    }
}

template <class V>
__global__ void k_tile_out(int n, const int *pos, const V *xp, V *x, const int *status)
{
    if (status && *status != ST_RUNNING) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[i] = xp[pos[i]];
}

// a / d from y = RN(1 / d) by one residual correction, the rounded quotient
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34 (1990), for the method).  With
// d' in [1, 2) the significand of d, 1 - d y is at most 2^-54 d'.  Before its
// last rounding, q0 + (a - q0 d) y differs from a / d by (a / d - q0)(1 - d y).
// a / d lies at least 1 / (2 d) = 2^-53 / d' units off every midpoint between
// two doubles (d as an integer of 53 bits).  Only where it lies within 1.5 *
// 2^-53 units of one could the last rounding differ, and there a y is less than
// a whole unit off the midpoint, so q0 is one of its two neighbours, half a unit
// away: the difference is at most 2^-54 d' / 2, which is less than 2^-53 / d' for
// every d' < 2 (d = 2^53 - 1, where the bounds meet, included; the quotients
// nearest to midpoints are in tests/test_gpu_line_division.py).  STRICT and FP32
// take a second correction.  Out of the range where every intermediate is
// normal: a real division.
// a real division, kept out of line: inlined, its steps were computed ahead
// of the test on every row
__device__ __noinline__ double full_div(double a, double d) { return a / d; }
__device__ __noinline__ float full_div(float a, float d) { return a / d; }

template <bool S>
__device__ __forceinline__ double line_div(double a, double d, double y)
{
    const double q0 = a * y;
    double q = fma(fma(-d, q0, a), y, q0);
    if constexpr (S) q = fma(fma(-d, q, a), y, q);
    // tested on the bits (an FP64 compare takes as long as an FMA), after the
    // quotient: the test hides in its latency
    const unsigned hi = (unsigned)__double2hiint(a), ea = (hi >> 20) & 0x7ffu;
    if (ea - 623u > 800u || __double2hiint(y) == 0) {
        const bool zero = ((hi & 0x7fffffffu) | (unsigned)__double2loint(a)) == 0u;
        q = zero && __double2hiint(y) != 0 ? q0 : full_div(a, d);
    }
    return q;
}

template <bool S>
__device__ __forceinline__ float line_div(float a, float d, float y)
{
    const float q0 = a * y;
    float q = fmaf(fmaf(-d, q0, a), y, q0);
    q = fmaf(fmaf(-d, q, a), y, q);
    const unsigned ea = (__float_as_uint(a) >> 23) & 0xffu;
    if (ea - 87u > 80u || y == 0.0f) q = a == 0.0f && y != 0.0f ? q0 : full_div(a, d);
    return q;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Non-blocking (try_wait may suspend the thread).
__device__ __forceinline__ bool mbar_test_wait(uint64_t *bar, unsigned parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// The lanes of a part (threads 0 .. T-1) only compute: everything a step
// needs is in shared memory by then.  One thread of the last warp keeps the
// slots filled (bulk copies of the record and of b), and loader warp w takes
// steps w, w + kLoaders, ...: it brings in the entries solved by other CTAs,
// polling those still pending, so neither memory latency nor a poll's round
// trip sits in the chain of steps.  A slot's barrier completes when its
// copies have landed and its loader has arrived.  s_done: steps whose slots
// the lanes have read.
//
// With one warp on each quarter of the SM, every instruction of the lanes'
// loop is on the path: operands are read ahead of the step's barrier, and an
// entry costs one shared-memory read at a prepared offset and its
// multiply-add, with no test for where it comes from.  96^3 convection-
// diffusion, L / U sweep in us: tickets (precond.cu) 273 / 361; register
// prefetch by the computing warps 494 / 519 (a warp's few scoreboards make an
// old load wait for the newer ones); loader warps, b and x in row order 211 /
// 250 (32 sectors a warp for each); plan order, a test per entry 155 / 198;
// prepared offsets 104 / 155; operands read inside the chain 96 / 135 (552
// cycles an L step, of which the four dependent FP64 operations take 300).
// A whole apply, both permutations included: 633 -> 253 us; 128^3 Poisson
// ILU 389 -> 355 with the last step; 63^3 FP32 sweeps 248 / 239 -> 33 / 42.
template <bool S, int MODE, int K, int T, class V>
__global__ void __launch_bounds__(T + 32 * LinePipe<V>::kLoaders + 32, 1)
    k_line_sweep(const unsigned char *__restrict__ rec, const int *__restrict__ part_step,
                 const int2 *__restrict__ rem, int rem_max, const V *b, V *x, const int *status, int *err, int spin,
                 int *pivot0)
{
    constexpr int D = LinePipe<V>::kSlots, LW = LinePipe<V>::kLoaders;
    constexpr bool kDesc = MODE == 1 || MODE == 3, kDiv = MODE == 1 || MODE == 2;
    constexpr int kBytesB = T * (int)sizeof(V), kRec = mode_record<V, MODE>(K, T), kSlot = kRec + kBytesB;
    constexpr int kArrays = MODE == 6 ? 2 * K : K + 2;  // of a record
    constexpr int W = MODE == 6 ? 2 : 1;                // words of a value
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t full[D];
    __shared__ volatile int s_done, s_abort;
    if (status && *status != ST_RUNNING) return;
    const int tid = (int)threadIdx.x, lane = tid & 31;
    const int step0 = part_step[blockIdx.x], steps = part_step[blockIdx.x + 1] - step0;
    unsigned char *slots = sm + W * line_slots<V>(K, T);
    if (tid == 0) {
        for (int i = 0; i < D; ++i) mbar_init(&full[i], 2);
        mbar_fence_init();
        s_done = 0;
        s_abort = 0;
        for (int w = 0; w < W; ++w) reinterpret_cast<V *>(sm + W * line_zero<V>(T))[w] = V(MODE == 6 ? 1 : 0);
    }
    __syncthreads();
    // step s of the sweep is step plan_step(s) of the plan
    auto plan_step = [&](int s) { return step0 + (kDesc ? steps - 1 - s : s); };
    auto give_up = [&]() {
        s_abort = 1;
        atomicExch(err, 1);
    };
    auto slot_free = [&](int s) {  // the lanes are done with step s - D
        for (long long i = 0; s_done < s - D + 1; ++i) {
            if (s_abort) return false;
            if (i > kLineSpin * 4) {
                give_up();
                return false;
            }
            __nanosleep(20);
        }
        __threadfence_block();
        return true;
    };

    if (tid >= T + 32 * LW) {  // the records and b
        if (lane == 0) {
            // a few steps at a time: one look at s_done and one fence for all
            // (a step each: the 63^3 FP32 L sweep 40.5 us, 33.0 so)
            constexpr int kFew = D / 4;
            int s = 0;
            while (s < steps) {
                const int end = min(steps, s + kFew);
                if (!slot_free(end - 1)) break;
                fence_proxy_async();
                for (; s < end; ++s) {
                    const size_t ps = (size_t)plan_step(s);
                    uint64_t *bar = &full[s % D];
                    unsigned char *to = slots + (s % D) * kSlot;
                    mbar_arrive_expect_tx(bar, (unsigned)(kRec + kBytesB));
                    bulk_g2s(to, rec + ps * kRec, (unsigned)kRec, bar);
                    bulk_g2s(to + kRec, b + ps * T, (unsigned)kBytesB, bar);
                }
            }
            // every copy lands before the block leaves (after an abort the
            // loaders' arrivals may be missing: a bounded wait is enough, the
            // copies themselves take microseconds)
            for (int t = max(0, s - D); t < s; ++t)
                if (!mbar_wait_bounded(&full[t % D], (unsigned)(t / D) & 1u, s_abort ? 1LL << 16 : kWaitLimit)) give_up();
        }
    } else if (tid >= T) {  // the entries from other CTAs
        int s = (tid - T) >> 5;
        // step t's first items (position, slot), read ahead of its turn
        auto look = [&](int t) {
            return t < steps && lane < rem_max ? rem[(size_t)plan_step(t) * rem_max + lane] : make_int2(-1, 0);
        };
        int2 next = look(s);
        for (; s < steps; s += LW) {
            int2 it = next;
            next = look(s + LW);
            // the lanes read step s - D's entries after its barrier: one step more
            if (!__all_sync(0xffffffffu, slot_free(s + 1))) break;
            V *xs = reinterpret_cast<V *>(sm + W * line_remote<V>(K, T, s));
            bool bad = false;
            for (int q = lane; it.x >= 0;) {
                for (int w = 0; w < W; ++w) xs[it.y * W + w] = wait_x(x, it.x * W + w, err, spin, bad);
                q += 32;
                it = q < rem_max ? rem[(size_t)plan_step(s) * rem_max + q] : make_int2(-1, 0);
            }
            if (bad) give_up();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s % D]);
        }
    } else {
        bool bad = false;
        int slot = 0;         // of the coming step
        unsigned parity = 0;  // of its barrier
        struct Operands {
            V vv[K], ww[K], bi, d, y;
            int4 code;
        } even, odd;
        auto fetch = [&](Operands &o, int sl) {
            const unsigned char *at = slots + sl * kSlot;
            const V *cv = reinterpret_cast<const V *>(at) + tid;
            o.code = reinterpret_cast<const int4 *>(at + kArrays * kBytesB)[tid];
            o.bi = reinterpret_cast<const V *>(at + kRec)[tid];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                o.vv[k] = cv[k * T];
                if constexpr (MODE == 6) o.ww[k] = cv[(K + k) * T];
            }
            if constexpr (kDiv) {
                o.d = cv[K * T];
                o.y = cv[(K + 1) * T];
            }
        };
        auto wait_fetch = [&](Operands &o, int sl, unsigned par) {
            bool ok = false;
            for (long long i = 0; i < kWaitLimit && !ok && !bad; ++i) {
                ok = mbar_try_wait(&full[sl], par);
                if ((i & 255) == 255 && s_abort) break;
            }
            if (!ok && !bad) {
                bad = true;
                give_up();
            }
            fetch(o, sl);
            if (bad) o.code = make_int4(line_zero<V>(T), line_zero<V>(T), line_zero<V>(T), line_zero<V>(T));
        };
        int prev = 0;  // the slot before it
        V *out = x + ((size_t)plan_step(0) * T + tid) * W;
        int here = tid * (int)sizeof(V) * W;  // this step's place in the ring
        // Step s on `o`.  The next step's operands are read into `next` while
        // the sum's multiply-adds wait for each other (a straight line, for
        // the compiler to interleave), and again after this step's x is out
        // if their slot was not full: never waiting before that, since
        // another CTA may need this x to fill the slot.
        auto step = [&](int s, Operands &o, Operands &next) {
            asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");  // step s - 1 is in the ring, step s's slot is read
            const int at[4] = {o.code.x, o.code.y, o.code.z, o.code.w};
            V xv[K], xr[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                xv[k] = *reinterpret_cast<const V *>(sm + at[k] * W);
                if constexpr (W == 2) xr[k] = reinterpret_cast<const V *>(sm + at[k] * W)[1];
            }
            const int sl = slot;
            const unsigned par = parity;
            const bool early = mbar_test_wait(&full[sl], par);
            // (the address waits for the test's answer: reads must not pass it)
            fetch(next, early ? sl : prev);
            prev = sl;
            if (tid == 0) s_done = s + 1;
            slot = sl + 1 == D ? 0 : sl + 1;
            parity ^= slot == 0 ? 1u : 0u;
            V acc = MODE >= 2 ? o.bi : V(0);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if constexpr (MODE == 6) {  // a_kk -= (a_ki / d_i) a_ik (FP64 only)
                    acc = fmac<true>(-line_div<true>(o.vv[k], xv[k], xr[k]), o.ww[k], acc);
                    if ((unsigned long long)__double_as_longlong(xv[k]) << 1 == 0ull) *pivot0 = 1;
                } else {
                    acc = fmac<S>(MODE >= 2 ? -o.vv[k] : o.vv[k], xv[k], acc);
                }
            }
            if constexpr (MODE <= 1) acc = o.bi - acc;
            if constexpr (kDiv) acc = line_div<S>(acc, o.d, o.y);
            // (the result of an operation is never the pending pattern, a signalling NaN)
            *reinterpret_cast<V *>(sm + here) = acc;
            st_relaxed(out, acc);
            if constexpr (W == 2) {
                const V r = line_safe(acc) ? V(1) / acc : V(0);
                reinterpret_cast<V *>(sm + here)[1] = r;
                st_relaxed(out + 1, r);
            }
            out += (kDesc ? -T : T) * W;
            here = here + W * kBytesB >= kRing * W * kBytesB ? here + W * kBytesB - kRing * W * kBytesB : here + W * kBytesB;
            if (!early && s + 1 < steps) wait_fetch(next, sl, par);
        };
        if (steps > 0) {
            wait_fetch(even, 0, 0);
            slot = 1;
        }
#pragma unroll 1
        for (int s = 0; s < steps; s += 2) {
            step(s, even, odd);
            if (s + 1 < steps) step(s + 1, odd, even);
        }
    }
}

namespace {

template <bool S, int MODE, int K, int T, class V>
cudaError_t launch_line(mtjg_ctx *ctx, const TilePlan *tp, const TileOp &op, const V *b, V *x, const int *status,
                        int spin, int *pivot0 = nullptr)
{
    auto k = k_line_sweep<S, MODE, K, T, V>;
    const int smem = line_smem<V, MODE>(K, T);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)tp->parts);
    cfg.blockDim = dim3(T + 32 * LinePipe<V>::kLoaders + 32);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const unsigned char *rec = sizeof(V) == 8 ? op.rec64 : op.rec32;
    e = cudaLaunchKernelEx(&cfg, k, rec, (const int *)tp->part_step, (const int2 *)op.rem, op.rem_max, b, x, status,
                           ctx->d_flag, spin, pivot0);
    if (e == cudaSuccess) ctx->launches++;
    return e;
}

template <bool S, int MODE, class V>
cudaError_t launch_k(mtjg_ctx *ctx, const TilePlan *tp, const TileOp &op, const V *b, V *x, const int *status, int spin,
                     int *pivot0 = nullptr)
{
    const auto go = [&](auto kmax) {
        constexpr int K = decltype(kmax)::value;
        if constexpr (line_fits<MODE>(K, 256)) {
            if (tp->lanes == 256) return launch_line<S, MODE, K, 256, V>(ctx, tp, op, b, x, status, spin, pivot0);
        }
        if (tp->lanes != 128) return cudaErrorInvalidConfiguration;  // (tile_plan and tile_ilu ask line_fits)
        return launch_line<S, MODE, K, 128, V>(ctx, tp, op, b, x, status, spin, pivot0);
    };
    switch (tp->kmax) {
    case 2: return go(std::integral_constant<int, 2>{});
    case 3: return go(std::integral_constant<int, 3>{});
    default: return go(std::integral_constant<int, 4>{});
    }
}

template <bool S>
cudaError_t launch_mode(mtjg_ctx *ctx, const TilePlan *tp, const TileOp &op, const double *b, double *x,
                        const int *status, int spin)
{
    switch (op.mode) {
    case 0: return launch_k<S, 0, double>(ctx, tp, op, b, x, status, spin);
    case 1: return launch_k<S, 1, double>(ctx, tp, op, b, x, status, spin);
    case 2: return launch_k<S, 2, double>(ctx, tp, op, b, x, status, spin);
    default: return launch_k<S, 3, double>(ctx, tp, op, b, x, status, spin);
    }
}

cudaError_t sweep_op(mtjg_ctx *ctx, const TilePlan *tp, const TileOp &op, bool strict, const double *b, double *x,
                     const int *status, int spin)
{
    return strict ? launch_mode<true>(ctx, tp, op, b, x, status, spin)
                  : launch_mode<false>(ctx, tp, op, b, x, status, spin);
}

// the FP32 sweeps of the mixed-precision inner solves: MODE 0 and 1, FAST
cudaError_t sweep_op(mtjg_ctx *ctx, const TilePlan *tp, const TileOp &op, bool, const float *b, float *x,
                     const int *status, int spin)
{
    return op.mode == 0 ? launch_k<false, 0, float>(ctx, tp, op, b, x, status, spin)
                        : launch_k<false, 1, float>(ctx, tp, op, b, x, status, spin);
}

int grid_rows(mtjg_ctx *ctx, int64_t n)
{
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + kBlock - 1) / kBlock, ctx->num_sms * 8));
}

template <class V>
cudaError_t apply_t(mtjg_ctx *ctx, const TilePair *t, bool strict, const V *b, V *x, const int *status, int spin, V *bp,
                    V *yp, V *xp)
{
    const TilePlan *tp = t->plan;
    const int count = tp->steps * tp->lanes;
    k_tile_in<V><<<grid_rows(ctx, count), kBlock, 0, ctx->stream>>>(count, tp->row, b, bp, yp, xp, status);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = sweep_op(ctx, tp, t->op[0], strict, (const V *)bp, yp, status, spin);
    if (e == cudaSuccess) e = sweep_op(ctx, tp, t->op[1], strict, (const V *)yp, xp, status, spin);
    if (e != cudaSuccess) return e;
    k_tile_out<V><<<grid_rows(ctx, tp->n), kBlock, 0, ctx->stream>>>(tp->n, tp->pos, xp, x, status);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace

cudaError_t tile_apply(mtjg_ctx *ctx, const TilePair *t, bool strict, const double *b, double *x, const int *status,
                       int spin)
{
    return apply_t<double>(ctx, t, strict, b, x, status, spin, t->plan->b64, t->plan->y64, t->plan->x64);
}

cudaError_t tile_apply(mtjg_ctx *ctx, const TilePair *t, bool strict, const float *b, float *x, const int *status,
                       int spin)
{
    return apply_t<float>(ctx, t, strict, b, x, status, spin, t->plan->b32, t->plan->y32, t->plan->x32);
}

static void free_plan(TilePlan *&tp)
{
    if (!tp) return;
    cudaFree(tp->b64);
    cudaFree(tp->b32);
    delete tp;
    tp = nullptr;
}

void free_tiles_of(TilePair *&t)
{
    if (!t) return;
    if (t->owns_plan) free_plan(t->plan);
    cudaFree(t->mem);
    for (TileOp &op : t->op) cudaFree(op.rec32);
    delete t;
    t = nullptr;
}

void tile_drop32(TilePair *t)
{
    for (TileOp &op : t->op) {
        cudaFree(op.rec32);
        op.rec32 = nullptr;
    }
    cudaFree(t->plan->b32);
    t->plan->b32 = t->plan->y32 = t->plan->x32 = nullptr;
}

// Tiles of lines pay when rows form lines (kMinLine rows each on average), a
// record holds every row (kLineK entries), the two triangles mirror each
// other (so that one plan, walked up and down, serves both sweeps), the tiles
// fit the SMs one each (none waits for a place), and the plan has at most 2 n +
// 65536 places (so a small system's lanes may be mostly empty: 1600 rows in
// 27,648 places).  Tiles: 128 lanes, 256 when 128 give more tiles than SMs;
// among the shapes the one with the fewest tile boundaries on a path across
// the grid.  For cubes that is 128 lanes up to 128^3, 256 up to 192^3, and no
// plan beyond.  ILU apply / setMatrix: 128^3 0.37 / 2.9 ms, 129^3 0.49 / 18.6
// (256 lanes of three entries leave the pivots to the levels), 192^3 0.76 / 53,
// 193^3 by levels 2.4 / 115 ms.
static int tile_plan(mtjg_ctx *ctx, const TriOp &op, const TriOp &up, TilePlan **out)
{
    *out = nullptr;
    const int n = op.n;
    int coop = 0;
    if (n == 0 || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess || !coop)
        return MTJG_OK;
    TilePlan *tp = new TilePlan();
    tp->n = n;
    int *work = nullptr;
    auto done = [&](int st, bool keep) {
        cudaFree(work);
        if (keep) *out = tp;
        else free_plan(tp);
        return st;
    };
#define LP_CUDA(call)                                                           \
    do {                                                                        \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess) return done(cuda_fail(e_, "sweep plan"), false); \
    } while (0)
    cudaStream_t q = ctx->stream;
    const int g = grid_rows(ctx, n);
    // Planning costs allocations, launches and waits beside its kernels, and on
    // a small or refused factor they are all there is.  First the pattern by
    // itself, before anything is allocated (setMatrix of a permuted 20^3 grid,
    // refused: 943 us with levels alone, 995 with two allocations before the
    // refusal, 977 so); then one allocation of scratch, one of the plan, one of
    // both sweeps' records, and four waits in all (four rows of four, ILU: 312 us
    // with levels alone, 395 with 15 allocations and nine waits, 274 so; ICC 329,
    // 471, 390).
    int *look = ctx->d_flag + 2, sc[2] = {};
    LP_CUDA(cudaMemsetAsync(look, 0, sizeof(sc), q));
    k_line_look<<<g, kBlock, 0, q>>>(op, up, look);
    ctx->launches++;
    LP_CUDA(cudaMemcpyAsync(sc, look, sizeof(sc), cudaMemcpyDeviceToHost, q));
    LP_CUDA(cudaStreamSynchronize(q));
    const int lines = sc[1];
    tp->kmax = sc[0] == 1 ? 2 : sc[0];
    if (tp->kmax < 2 || tp->kmax > kLineK || (int64_t)lines * kMinLine > n) return done(MTJG_OK, false);
    // one allocation: what each line reads; per row the start of a line, the
    // line and the starts' scan; counts; per line its first row, the start of a
    // plane and its scan, the planes' first lines, part, lane and offset; per
    // part its first step, last step and place; the scans' scratch
    const size_t L = (size_t)lines, P0 = (size_t)ctx->num_sms;
    LP_CUDA(cudaMalloc(&work, sizeof(int) * (2 * kLineK * L + 3 * (size_t)n + 1 + 3 + 7 * L + 3 + 3 * P0 + 1 +
                                             (size_t)scan_scratch(n))));
    int2 *dep = reinterpret_cast<int2 *>(work);
    int *start = work + 2 * kLineK * L, *line_of = start + n, *scan = line_of + n;
    // planes, lines of the longest plane, 1 for lines without offsets
    int *scalars = scan + n + 1;
    int *first = scalars + 3, *pstart = first + L + 1, *pscan = pstart + L, *pfirst = pscan + L + 1;
    int *part_of = pfirst + L + 1, *lane_of = part_of + L, *off = lane_of + L;
    int *pw = off + L, *scratch = pw + 3 * P0 + 1;
    LP_CUDA(cudaMemsetAsync(scalars, 0, sizeof(int) * 3, q));
    k_line_start<<<g, kBlock, 0, q>>>(op, start);
    ctx->launches++;
    LP_CUDA(exclusive_scan_async(ctx, start, scan, n, scratch));
    const int gl = grid_rows(ctx, lines);
    k_line_of<<<g, kBlock, 0, q>>>(n, start, scan, line_of, first, pstart, lines);
    k_plane_start<<<g, kBlock, 0, q>>>(op, line_of, pstart);
    LP_CUDA(exclusive_scan_async(ctx, pstart, pscan, lines, scratch));
    k_plane_first<<<gl, kBlock, 0, q>>>(lines, pstart, pscan, pfirst, scalars);
    k_plane_long<<<gl, kBlock, 0, q>>>(scalars, pfirst, scalars + 1);
    ctx->launches += 4;
    LP_CUDA(cudaMemcpyAsync(sc, scalars, sizeof(int) * 2, cudaMemcpyDeviceToHost, q));
    LP_CUDA(cudaStreamSynchronize(q));
    const int planes = sc[0], longest = sc[1];
    int tq = 0, ntq = 0, best = 0;
    for (int T = 128; T <= 256 && !tp->parts; T *= 2)
        for (int a = 1; a <= T; a *= 2) {
            const int64_t nq = (longest + a - 1) / a, np = (planes + T / a - 1) / (T / a);
            if (nq * np > ctx->num_sms || (tp->parts && nq + np >= best)) continue;
            tp->parts = (int)(nq * np);
            tp->lanes = T;
            tq = a;
            ntq = (int)nq;
            best = (int)(nq + np);
        }
    int optin = 0;
    LP_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
    if (!tp->parts || (int64_t)lines * 4 + 1024 > optin || !line_plan_fits(tp->kmax, tp->lanes))
        return done(MTJG_OK, false);
    const int P = tp->parts, T = tp->lanes;
    // a grid's steps (a part of q by p lines of L rows takes L + q + p - 2):
    // twice too many, and the lines' offsets (27 ms for 8 x 8 x 2500) are not
    // worth finding
    const int64_t likely = (int64_t)P * (n / lines - 2) + (int64_t)(P / ntq) * longest + (int64_t)ntq * planes;
    if (likely * T > 2 * (2 * (int64_t)n + 65536)) return done(MTJG_OK, false);
    int *part_step = pw + 2 * (size_t)P;
    k_line_tile<<<gl, kBlock, 0, q>>>(lines, pstart, pscan, pfirst, tq, T / tq, ntq, part_of, lane_of);
    k_line_deps<<<(lines + 7) / 8, kBlock, 0, q>>>(op, lines, line_of, first, dep, scalars + 2);
    LP_CUDA(cudaFuncSetAttribute(k_line_offsets, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 1024));
    k_line_offsets<<<1, kOffsetBlock, sizeof(int) * (size_t)lines, q>>>(lines, planes, pfirst, dep, first, part_of, off,
                                                                        P, pw, pw + P, part_step, scalars + 2);
    ctx->launches += 3;
    LP_CUDA(cudaMemcpyAsync(sc, scalars + 2, sizeof(int), cudaMemcpyDeviceToHost, q));
    LP_CUDA(cudaMemcpyAsync(sc + 1, part_step + P, sizeof(int), cudaMemcpyDeviceToHost, q));
    LP_CUDA(cudaStreamSynchronize(q));
    tp->steps = sc[1];
    if (sc[0] || (int64_t)tp->steps * T > 2 * (int64_t)n + 65536) return done(MTJG_OK, false);
    const size_t count = (size_t)tp->steps * T;
    LP_CUDA(cudaMalloc(&tp->b64, sizeof(double) * 3 * count + sizeof(int) * (count + (size_t)n + (size_t)P + 1)));
    tp->y64 = tp->b64 + count;
    tp->x64 = tp->y64 + count;
    tp->row = reinterpret_cast<int *>(tp->x64 + count);
    tp->pos = tp->row + count;
    tp->part_step = tp->pos + n;
    LP_CUDA(cudaMemsetAsync(tp->row, 0xff, sizeof(int) * count, q));
    k_line_place<<<g, kBlock, 0, q>>>(n, T, line_of, first, part_of, lane_of, off, pw, P, part_step, tp->pos, tp->row,
                                      tp->part_step);
    ctx->launches++;
    // a launch that has nothing to do (a status other than running) tells
    // whether the device takes this cooperative grid
    static_assert(ST_RUNNING != -1, "the trial launch's status");
    LP_CUDA(cudaMemsetAsync(scalars, 0xff, sizeof(int), q));
    TileOp none;
    none.mode = 1;
    const cudaError_t e = sweep_op(ctx, tp, none, false, (const double *)nullptr, (double *)nullptr, scalars, 0);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        (void)cudaGetLastError();
        return done(MTJG_OK, false);
    }
    LP_CUDA(e);
    return done(MTJG_OK, true);
}
#undef LP_CUDA

// The sweeps' entry codes and the lists of what they read from other parts: 32
// places a step (a tile of 8 x 16 lines of a grid needs at most 24), or as
// many as the longest needs.
static int tile_ops(mtjg_ctx *ctx, TilePair *t, const TriOp &lo, const TriOp &up)
{
    const TilePlan *tp = t->plan;
    cudaStream_t q = ctx->stream;
    const size_t S = (size_t)tp->steps, rec = S * line_record<double>(tp->kmax, tp->lanes);
    const int g = grid_rows(ctx, (int64_t)S * tp->lanes);
    // the longest lists and the steps' counts, in a vector that no sweep uses now
    int *longest = reinterpret_cast<int *>(tp->y64), h[2] = {};
    int most = 32;
    do {
        const size_t rem = sizeof(int2) * S * most;
        cudaFree(t->mem);
        t->mem = nullptr;
        MTJG_CUDA(cudaMalloc(&t->mem, 2 * (rec + rem)));
        MTJG_CUDA(cudaMemsetAsync(t->mem + 2 * rec, 0xff, 2 * rem, q));
        MTJG_CUDA(cudaMemsetAsync(longest, 0, sizeof(int) * (2 * S + 2), q));
        for (int w = 0; w < 2; ++w) {
            TileOp &o = t->op[w];
            int *cursor = longest + 2 + w * S;
            o.mode = w ? up.mode : lo.mode;
            o.rec64 = t->mem + w * rec;
            o.rem = reinterpret_cast<int *>(t->mem + 2 * rec + w * rem);
            o.rem_max = most;
            k_line_codes<double><<<g, kBlock, 0, q>>>(w ? up : lo, *tp, o.rec64, cursor, (int2 *)o.rem, most,
                                                     longest + w);
            ctx->launches++;
        }
        MTJG_CUDA(cudaMemcpyAsync(h, longest, sizeof(h), cudaMemcpyDeviceToHost, q));
        MTJG_CUDA(cudaStreamSynchronize(q));
        h[0] = std::max(h[0], h[1]);
    } while (h[0] > most && (most = h[0]));
    return MTJG_OK;
}

int tile_pair(mtjg_ctx *ctx, const TriOp &lo, const TriOp &up, TilePlan *plan, TilePair **out)
{
    *out = nullptr;
    TilePair *t = new TilePair();
    t->owns_plan = plan == nullptr;
    t->plan = plan;
    int st = MTJG_OK;
    if (!plan) st = tile_plan(ctx, lo, up, &t->plan);
    if (st == MTJG_OK && t->plan) st = tile_ops(ctx, t, lo, up);
    if (st != MTJG_OK || !t->plan) free_tiles_of(t);
    else *out = t;
    if (st == MTJG_ERR_OUT_OF_MEMORY) {  // the level schedules take a tenth of the memory
        (void)cudaGetLastError();
        st = MTJG_OK;
    }
    return st;
}

// ----------------------------------------------------- ILU(0)'s pivots
// Where no elimination step finds a column of row k other than k itself
// (grids without diagonals), ILU.factor (S/ILU.java:98-121) changes only
// the pivots, in row order: d_k = a_kk - (a_ki / d_i) a_ik over ascending i,
// and its multipliers are a_ki / d_i.  So the factor is a sweep whose values
// are the pivots (each with its reciprocal, so that a row takes one division
// and not one per entry), then one pass over the entries.  96^3 convection-diffusion:
// 4.2 ms by one launch per level (after 2.4 ms to find the levels), 0.86 ms
// with a division per entry, 0.41 ms as here; setMatrix and one apply 17.6 ->
// 2.4 ms.
//
// *other = 1 when some step finds another column (MTJ's scan, its read past
// the row's end included).
__global__ void k_pivots_only(TriOp lo, int *other)
{
    const int *rp = lo.rp, *ci = lo.ci, *diag = lo.diag;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < lo.n; k += gridDim.x * blockDim.x)
        for (int i = rp[k]; i < diag[k]; ++i) {
            const int index = ci[i];
            for (int j = diag[index] + 1, l = rp[k] + 1; j < rp[index + 1]; ++j) {
                while (l < rp[k + 1] && ci[l] < ci[j]) l++;
                if (ci[l] == ci[j] && l != diag[k]) *other = 1;
            }
        }
}

// MODE 6's records, its b (the diagonal) and its output (a pivot and its
// reciprocal per position) to pending; codes: the records of the lower sweep
__global__ void k_pivot_records(TriOp lo, TilePlan tp, const unsigned char *codes, const double *data,
                                unsigned char *rec, double *b, double *x)
{
    const int T = tp.lanes, K = tp.kmax, from = line_record<double>(K, T), to = mode_record<double, 6>(K, T);
    for (int at = blockIdx.x * blockDim.x + threadIdx.x; at < tp.steps * T; at += gridDim.x * blockDim.x) {
        const int k = tp.row[at], step = at / T, lane = at % T;
        unsigned char *r = rec + (size_t)step * to;
        double *rv = reinterpret_cast<double *>(r);
        reinterpret_cast<int4 *>(r + (size_t)T * 2 * K * sizeof(double))[lane] =
            reinterpret_cast<const int4 *>(codes + (size_t)step * from + (size_t)T * (K + 2) * sizeof(double))[lane];
        const int b0 = k >= 0 ? lo.rp[k] : 0, cnt = k >= 0 ? lo.diag[k] - b0 : 0;
        for (int e = 0; e < K; ++e) {
            double low = 0.0, up = 0.0;
            if (e < cnt) {
                const int i = lo.ci[b0 + e];
                low = data[b0 + e];
                for (int j = lo.diag[i] + 1; j < lo.rp[i + 1]; ++j)
                    if (lo.ci[j] == k) up = data[j];
            }
            rv[e * T + lane] = low;
            rv[(K + e) * T + lane] = up;
        }
        b[at] = k >= 0 ? data[lo.diag[k]] : 1.0;
        x[2 * at] = x[2 * at + 1] = pending_value<double>();
    }
}

// the pivots into the diagonal, the multipliers into the lower entries
__global__ void k_pivots_out(TriOp lo, const int *pos, const double *x, double *data)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < lo.n; k += gridDim.x * blockDim.x) {
        data[lo.diag[k]] = x[2 * (size_t)pos[k]];
        for (int i = lo.rp[k]; i < lo.diag[k]; ++i) data[i] = data[i] / x[2 * (size_t)pos[lo.ci[i]]];
    }
}

int tile_ilu(mtjg_ctx *ctx, TilePair *t, const TriOp &lo, double *data, bool *factored)
{
    *factored = false;
    const TilePlan *tp = t->plan;
    const int64_t count = (int64_t)tp->steps * tp->lanes;
    if (!line_fits<6>(tp->kmax, tp->lanes) || !pivot_pairs_fit(count)) return MTJG_OK;
    cudaStream_t q = ctx->stream;
    const size_t bytes = (size_t)tp->steps * mode_record<double, 6>(tp->kmax, tp->lanes);
    unsigned char *rec = nullptr;
    if (cudaMalloc(&rec, bytes + 16) != cudaSuccess) {
        (void)cudaGetLastError();
        return MTJG_OK;
    }
    int *flags = reinterpret_cast<int *>(rec + bytes);  // another column found; zero pivot; the device's error flag
    int h[3] = {1, 1, 1};
    cudaError_t e = cudaMemsetAsync(flags, 0, sizeof(int) * 2, q);
    if (e == cudaSuccess) e = cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), q);
    k_pivots_only<<<grid_rows(ctx, tp->n), kBlock, 0, q>>>(lo, flags);
    // (y64 and x64 are one array of twice the positions)
    k_pivot_records<<<grid_rows(ctx, count), kBlock, 0, q>>>(lo, *tp, t->op[0].rec64, data, rec, tp->b64, tp->y64);
    ctx->launches += 2;
    TileOp op = t->op[0];
    op.rec64 = rec;
    if (e == cudaSuccess)
        e = launch_k<false, 6, double>(ctx, tp, op, tp->b64, tp->y64, nullptr, 1 << 20, flags + 1);
    if (e == cudaSuccess) e = cudaMemcpyAsync(flags + 2, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToDevice, q);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, flags, sizeof(h), cudaMemcpyDeviceToHost, q);
    if (e == cudaSuccess) e = cudaStreamSynchronize(q);
    cudaFree(rec);
    if (e != cudaSuccess) return cuda_fail(e, "ILU pivots");
    if (h[2]) {
        cudaMemset(ctx->d_flag, 0, sizeof(int));
        return fail(MTJG_ERR_DEVICE_TIMEOUT, "ILU pivots: a bounded wait gave up");
    }
    if (h[0] || h[1]) return MTJG_OK;  // general elimination, which also reports a zero pivot's row
    k_pivots_out<<<grid_rows(ctx, tp->n), kBlock, 0, q>>>(lo, tp->pos, tp->y64, data);
    ctx->launches++;
    MTJG_CUDA(cudaGetLastError());
    *factored = true;
    return MTJG_OK;
}

int tile_values(mtjg_ctx *ctx, TilePair *t, int which, const TriOp &op, const double *v, const double *diagv)
{
    const TilePlan *tp = t->plan;
    k_line_values<double><<<grid_rows(ctx, (int64_t)tp->steps * tp->lanes), kBlock, 0, ctx->stream>>>(
        op, *tp, t->op[which].rec64, v, diagv);
    ctx->launches++;
    MTJG_CUDA(cudaGetLastError());
    return MTJG_OK;
}

int tile_values(mtjg_ctx *ctx, TilePair *t, int which, const TriOp &op, const float *v, const float *diagv)
{
    TilePlan *tp = t->plan;
    TileOp &to = t->op[which];
    const size_t count = (size_t)tp->steps * tp->lanes;
    if (!tp->b32) {
        MTJG_CUDA(cudaMalloc(&tp->b32, sizeof(float) * 3 * count));
        tp->y32 = tp->b32 + count;
        tp->x32 = tp->y32 + count;
    }
    if (!to.rec32) {
        const size_t bytes = (size_t)tp->steps * line_record<float>(tp->kmax, tp->lanes);
        MTJG_CUDA(cudaMalloc(&to.rec32, bytes));
        k_line_codes<float><<<grid_rows(ctx, (int64_t)count), kBlock, 0, ctx->stream>>>(
            op, *tp, to.rec32, nullptr, nullptr, 0, nullptr);
        ctx->launches++;
    }
    k_line_values<float><<<grid_rows(ctx, (int64_t)count), kBlock, 0, ctx->stream>>>(op, *tp, to.rec32, v, diagv);
    ctx->launches++;
    MTJG_CUDA(cudaGetLastError());
    return MTJG_OK;
}

}  // namespace mtjg
