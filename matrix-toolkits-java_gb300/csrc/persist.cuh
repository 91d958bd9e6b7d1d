// persist.cuh -- CG (identity or Jacobi preconditioner) on one small system
// in one launch.
//
// On a system of a few hundred tiles every phase of the graph-captured loop
// (p, q = A p, its finalize, the update, its finalize) is a few dependent
// L2 round trips wide, and the iteration costs their latency plus the launch
// gaps.  Here one cooperative launch runs the iterations of the same loop
// (S/CG.java:66-87) until the monitor stops the solve.  A CTA owns one or two
// product tiles: their entries stay in shared memory and its rows' x, r, z, p
// and inverse diagonal in registers, so an iteration's traffic is p for the
// other tiles' gathers and the partial sums.  Three exchanges remain: p (once
// beta is known), the p.q partials (alpha), the partials of r (beta and the
// monitor's test).  Each travels as 16-byte packets of a value and a tag (the
// iteration or phase), stored and polled whole (b128), so nothing is fenced:
// a fence took 1100 to 3900 cycles of an iteration's 24,000, twice.  Every
// CTA sums the partials itself, in k_finalize's order and block tree, and
// applies the scalar step to its own copy of the state; CTA 0 alone writes
// the history, the running count and the state.  The systems that qualify run
// CG's row phases on their product tiles on the graph path too, so x, the
// history and the iteration count are the same on both paths bit for bit.
//
// 2D Poisson 128^2 (392 iterations): 5.44 ms with the vectors in the L2, row
// tiles of 1024 rows for the update (16 CTAs of 71) and an arrival counter
// read before the partials; 4.24 ms with fences around plain partials; 3.03
// ms as here.
//
// Waits are bounded: a CTA that gives up sets the error flag and the abort
// word, and every CTA leaves at its next wait.
#pragma once

#include "spmv.cuh"

// systems of at most this many product tiles take the one-launch CG (when
// their tiles also fit the shared memory of the co-resident CTAs).  Measured
// on GB300 (CG + Jacobi, against the graph path): 2.0-2.6 times its speed up
// to 150 tiles, 1.5 at 300 (one tile a CTA), 1.3-1.4 from 305 to 512 (two a
// CTA: 2D 340^2 24.5 -> 17.8 ms, 3D 43^3 4.02 -> 2.84 ms).  A thread collects
// the partials of two tiles for 512; with a limit of 608 (as many as two a CTA
// hold) it collects three, and while systems of 513 to 608 tiles were 1.25
// times as fast as the graph, those below lost up to a fifth (2D 340^2 20.2 ms,
// 3D 36^3 2.02 -> 2.41 ms).
#ifndef MTJG_PERSIST_MAX_TILES
#define MTJG_PERSIST_MAX_TILES 512
#endif
// resident CTAs per SM the one-launch CG is compiled for (its register cap):
// 2, which 90 to 96 registers and no spills need
#ifndef MTJG_PERSIST_MINB
#define MTJG_PERSIST_MINB 2
#endif

namespace mtjg {

constexpr int kPersistMaxTiles = MTJG_PERSIST_MAX_TILES;
constexpr long long kGridSpinLimit = 1LL << 22;
// one cached product tile: values, columns, row offsets (16-byte multiples)
constexpr int kSlotValBytes = kTileNnz * 8;
constexpr int kSlotColBytes = ((kTileNnz * 4 + 15) / 16) * 16;
constexpr int kSlotRowBytes = (((kTileRows + 1) * 4 + 15) / 16) * 16;
constexpr int kSlotBytes = kSlotValBytes + kSlotColBytes + kSlotRowBytes;

struct GridBar {
    unsigned long long *count;  // arrivals in this launch (zeroed before it)
    int *abort;                 // set by a CTA whose wait gave up
};

// What the one-launch CG reads and writes (the solver's vectors and tiles).
struct PersistCg {
    CsrArgs A;
    TileArgs pt;  // product tiles: groups of the product's and the update's sums
    const double *invdiag;
    double *x, *r, *z;
    int pc;
    // packets: p of each row [n], and the partials' two sets [2][tiles][3]
    ulonglong2 *p, *part;
    MonPtrs m;
    GridBar gb;
    int *err;
};

namespace {

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Arrive and wait until `target` arrivals (G per barrier of the launch).
// Every write of the CTA before it is seen by every CTA after it.  Returns
// false in every thread of the CTA when the wait gave up (about a second, or
// at once when another CTA has given up).
__device__ bool grid_barrier(const GridBar &gb, unsigned long long target, int *err)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(gb.count, 1ull);
        bool ok = false;
        unsigned ns = 0;
        for (long long i = 0; i < kGridSpinLimit; ++i) {
            if (ld_acquire_u64(gb.count) >= target) {
                ok = true;
                break;
            }
            if ((i & 63) == 63) {
                if (*(volatile int *)gb.abort) break;
                ns = ns < 256 ? ns + 32 : ns;
                __nanosleep(ns);
            }
        }
        if (!ok) {
            atomicExch(gb.abort, 1);
            atomicExch(err, 1);
        }
        __threadfence();
        s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}

// A packet: a value and its tag, written and read as one 128-bit access.
__device__ __forceinline__ ulonglong2 ld_packet(const ulonglong2 *p)
{
    ulonglong2 v;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(p)
                 : "memory");
    return v;
}

__device__ __forceinline__ void st_packet(ulonglong2 *p, double v, unsigned long long tag)
{
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"((unsigned long long)__double_as_longlong(v)), "l"(tag)
                 : "memory");
}

// One more round of waiting: false when the wait has to end (kGridSpinLimit
// rounds, or another wait gave up): the CTA's s_bad, the abort word and the
// error flag are set then.
__device__ __forceinline__ bool wait_on(const PersistCg &c, long long i, int *s_bad)
{
    if (i <= kGridSpinLimit && ((i & 255) != 255 || (!*(volatile int *)c.gb.abort && !*(volatile int *)s_bad)))
        return true;
    *(volatile int *)s_bad = 1;
    atomicExch(c.gb.abort, 1);
    atomicExch(c.err, 1);
    return false;
}

// The value of a packet once it carries `tag` (0 when the wait gives up).
__device__ double wait_packet(const PersistCg &c, const ulonglong2 *p, unsigned long long tag, int *s_bad)
{
    ulonglong2 v = ld_packet(p);
    for (long long i = 0; v.y != tag && wait_on(c, i, s_bad); ++i) v = ld_packet(p);
    return v.y == tag ? __longlong_as_double((long long)v.x) : 0.0;
}

// The tiles' partial sums of one phase meet in one of two sets of packets by
// turns, tagged with the phase.  Collecting a phase's partials waits for every
// CTA to be that far; a CTA publishes two phases on only after it has seen
// every partial of the phase between, which each CTA published after it had
// collected this one's, so no packet is overwritten before all have read it.
// For the same reason a row's p is overwritten only after every gather of it.
// Word w (0, 1: the norm, 2: the plain sum) of a tile's partial, a line of its
// own: every CTA polls every one, and a line that several CTAs write while
// others poll it is slow (128^2: 4.08 ms with the tiles' words side by side,
// 3.57 with 48 bytes a tile, 3.03 with 128).
constexpr int kPacketStride = 8;
__device__ __forceinline__ ulonglong2 *partial(const PersistCg &c, int phase, int w, int t)
{
    return c.part + ((size_t)(phase & 1) * c.pt.num_tiles + t) * kPacketStride + w;
}

// The kBlock computing threads' barrier (the scalar warp is not in it).
__device__ __forceinline__ void rows_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kBlock) : "memory"); }

// block_reduce over the computing threads, of which only the first `used`
// hold anything: the sums of the empty ones are one zero.  The norm by warp
// 0, the plain sum by warp 1 (each on a quarter of the SM of its own: a
// dependent FP64 addition takes 64 cycles there, twelve of them a sum);
// results in out[0..1] (norm) and out[2], seen after the next barrier.
template <int SLOTS>
__device__ __forceinline__ void rows_reduce(const Acc &a, int used, int type, double *sm, double *out)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool robust = type == MTJG_NORM_TWO_ROBUST;
    if constexpr ((SLOTS & kSlotNorm) != 0) {
        sm[tid] = a.v[0];
        if (robust) sm[kBlock + tid] = a.v[1];
    }
    if constexpr ((SLOTS & kSlotD2) != 0) sm[2 * kBlock + tid] = a.v[2];
    rows_sync();
    auto plain = [&](const double *v) {
        double s = v[lane];
        for (int i = lane + 32; i - lane < used; i += 32) s += v[i];
        if (used <= kBlock - 32) s += 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        return s;
    };
    if constexpr ((SLOTS & kSlotNorm) != 0) {
        if (warp == 0) {
            if (type == MTJG_NORM_ONE || type == MTJG_NORM_TWO) {
                const double s = plain(sm);
                if (lane == 0) out[0] = s, out[1] = 0.0;
            } else {
                Acc s, o;
                s.v[0] = sm[lane];
                s.v[1] = robust ? sm[kBlock + lane] : 0.0;
                for (int i = lane + 32; i - lane < used; i += 32) {
                    o.v[0] = sm[i];
                    o.v[1] = robust ? sm[kBlock + i] : 0.0;
                    acc_merge_m<kSlotNorm>(s, o, type);
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) acc_shfl_down<kSlotNorm>(s, off, type);
                if (lane == 0) out[0] = s.v[0], out[1] = s.v[1];
            }
        }
    }
    if constexpr ((SLOTS & kSlotD2) != 0) {
        if (warp == 1) {
            const double s = plain(sm + 2 * kBlock);
            if (lane == 0) out[2] = s;
        }
    }
}

// This CTA's partials of a phase: out[k] is slot k's (rows_reduce).  By the
// warps that summed them.
template <int SLOTS, int SL>
__device__ __forceinline__ void publish(const PersistCg &c, int phase, int t0, int G, const double (*out)[4], int type)
{
    const int tid = threadIdx.x;
#pragma unroll
    for (int k = 0; k < SL; ++k) {
        if (t0 + k * G >= c.pt.num_tiles) continue;
        const int t = t0 + k * G;
        const unsigned long long tag = (unsigned long long)phase + 1;
        if ((SLOTS & kSlotNorm) != 0 && tid == 0) {
            st_packet(partial(c, phase, 0, t), out[k][0], tag);
            if (type == MTJG_NORM_TWO_ROBUST) st_packet(partial(c, phase, 1, t), out[k][1], tag);
        }
        if ((SLOTS & kSlotD2) != 0 && tid == 32) st_packet(partial(c, phase, 2, t), out[k][2], tag);
    }
}

// system_sum over the tiles' partials of a phase, waiting for each with all
// of a thread's loads in flight; in out[0..2] after the barrier it ends with.
template <int SLOTS>
__device__ void collect(const PersistCg &c, int phase, int type, double *sm, double *out, int *s_bad)
{
    constexpr bool kN = (SLOTS & kSlotNorm) != 0;
    constexpr int kMost = (kPersistMaxTiles + kBlock - 1) / kBlock;
    const int NT = c.pt.num_tiles;
    const bool robust = type == MTJG_NORM_TWO_ROBUST;
    const unsigned long long tag = (unsigned long long)phase + 1;
    Acc s;
    acc_zero(s);
    if ((int)threadIdx.x < NT) {
        // every packet of the thread is read again until all are there: one
        // round trip a round, however many are late
        Acc o[kMost];
        for (long long i = 0;; ++i) {
            bool late = false;
#pragma unroll
            for (int u = 0; u < kMost; ++u) {
                const int i1 = (int)threadIdx.x + u * kBlock, t = i1 < NT ? i1 : (int)threadIdx.x;
                acc_zero(o[u]);
                if (kN) {
                    const ulonglong2 n = ld_packet(partial(c, phase, 0, t));
                    late |= n.y != tag;
                    o[u].v[0] = __longlong_as_double((long long)n.x);
                    if (robust) {
                        const ulonglong2 q = ld_packet(partial(c, phase, 1, t));
                        late |= q.y != tag;
                        o[u].v[1] = __longlong_as_double((long long)q.x);
                    }
                }
                const ulonglong2 d = ld_packet(partial(c, phase, 2, t));
                late |= d.y != tag;
                o[u].v[2] = __longlong_as_double((long long)d.x);
            }
            if (!late || !wait_on(c, i, s_bad)) break;
        }
#pragma unroll
        for (int u = 0; u < kMost; ++u)
            if ((int)threadIdx.x + u * kBlock < NT) acc_merge_m<SLOTS>(s, o[u], type);
    }
    rows_reduce<SLOTS>(s, NT < kBlock ? NT : kBlock, type, sm, out);
    rows_sync();
}

// SL product tiles per CTA (tile bid + k G in slot k).  The last warp runs
// the monitor's test (a square root, divisions and compares on the narrow
// FP64 pipe, 2400 cycles) beside the next product, whose p and q a solve that
// has ended leaves unused.
constexpr int kPersistBlock = kBlock + 32;

template <bool S, int SL>
__global__ void __launch_bounds__(kPersistBlock, MTJG_PERSIST_MINB) k_cg_persist(PersistCg c, int normtype)
{
    extern __shared__ __align__(16) unsigned char slots[];
    // (the collecting sums have a place of their own: the threads that poll
    // nothing reach theirs while warps 0 and 1 still sum the CTA's partial)
    __shared__ double red_sm[3 * kBlock], all_sm[3 * kBlock];
    __shared__ double s_q[SL][kBlock];
    __shared__ double s_out[SL][4], s_sum[4], s_beta, s_alpha;
    __shared__ SysState s_st;
    __shared__ int s_run, s_bad;  // s_run: the running count of CTAs other than 0 (unused)
    const int tid = threadIdx.x, G = (int)gridDim.x, bid = (int)blockIdx.x, NT = c.pt.num_tiles;
    const bool rows_thread = tid < kBlock;
    const int nt = normtype;
    if (tid == 0) {
        s_st = c.m.st[0];
        s_run = 1;
        s_bad = 0;
    }
    // this CTA's product tiles into their slots (entries and rows checked
    // against the slot: a tile that does not fit stops the solve), its rows'
    // vectors into registers: row r0 + tid of each tile
    int bad = 0, row[SL], r0s[SL], rows[SL];
    double xv[SL], rv[SL], zv[SL], iv[SL], pv[SL];
    const bool jac = c.pc == kPcJacobi;
#pragma unroll
    for (int k = 0; k < SL; ++k) {
        const int t = bid + k * G;
        row[k] = -1;
        rows[k] = r0s[k] = 0;
        xv[k] = rv[k] = zv[k] = iv[k] = pv[k] = 0.0;
        if (t >= NT) continue;
        unsigned char *slot = slots + (size_t)k * kSlotBytes;
        const int r0 = c.pt.tile_row[t], r1 = c.pt.tile_row_end[t];
        const int nz0 = __ldg(c.A.rowptr + r0), nz1 = __ldg(c.A.rowptr + r1);
        if (r1 - r0 > kTileRows || nz1 - nz0 > kTileNnz) {
            bad = 1;
            continue;
        }
        double *sv = reinterpret_cast<double *>(slot);
        int *sc = reinterpret_cast<int *>(slot + kSlotValBytes);
        int *sr = reinterpret_cast<int *>(slot + kSlotValBytes + kSlotColBytes);
        for (int i = tid; i <= r1 - r0; i += kPersistBlock) sr[i] = __ldg(c.A.rowptr + r0 + i) - nz0;
        for (int e = tid; e < nz1 - nz0; e += kPersistBlock) {
            sv[e] = __ldg(c.A.val + nz0 + e);
            sc[e] = __ldg(c.A.colind + nz0 + e);
        }
        r0s[k] = r0;
        rows[k] = r1 - r0;
        if (rows_thread && tid < r1 - r0) {
            const int r = r0 + tid;
            row[k] = r;
            xv[k] = c.x[r];
            rv[k] = c.r[r];
            zv[k] = jac ? c.z[r] : rv[k];
            iv[k] = jac ? __ldg(c.invdiag + r) : 0.0;
        }
        // tags of an earlier launch go
        if (tid < 3) st_packet(partial(c, 0, tid, t), 0.0, 0ull), st_packet(partial(c, 1, tid, t), 0.0, 0ull);
        if (rows_thread && tid < r1 - r0) st_packet(c.p + r0 + tid, 0.0, 0ull);
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) {
            atomicExch(c.err, 1);
            atomicExch(c.gb.abort, 1);  // the other CTAs leave at their first barrier
        }
        return;
    }
    // every tag is cleared before any packet is published
    if (!grid_barrier(c.gb, (unsigned long long)G, c.err)) return;
    MonPtrs m = c.m;
    m.st = &s_st;
    if (bid != 0) {
        m.mon.hist_cap = 0;
        m.num_running = &s_run;
    }
    constexpr int kSlotsQ = OpSlots<CgQ<S>>::value, kSlotsU = OpSlots<CgUpd<S>>::value;
    constexpr int kBatch = 8;  // entries whose packets are in flight at once
    int phase = 0;
    unsigned long long it = 1;  // the coming p's tag
    bool first = true;
    double rho = s_st.rho;  // thread 0's
    if (s_st.status != ST_RUNNING) return;
    for (;;) {
        if (rows_thread) {
            if (tid == 0 && !first) {  // beta = rho / rho_1, rho = r.z
                const double rz = s_sum[2];
                s_beta = rz / rho;
                rho = rz;
            }
            rows_sync();
            const double beta = s_beta;
            // p = z (first) or beta p + z, out to the tiles that gather it
#pragma unroll
            for (int k = 0; k < SL; ++k) {
                pv[k] = first ? zv[k] : fmac<S>(pv[k], beta, zv[k]);
                if (row[k] >= 0) {
                    st_packet(c.p + row[k], pv[k], it);
                    s_q[k][tid] = pv[k];
                }
            }
            // q = A p and the p.q partials
#pragma unroll
            for (int k = 0; k < SL; ++k) {
                const int t = bid + k * G;
                Acc part;
                acc_zero(part);
                bool one = true;
                if (t < NT) {
                    const unsigned char *slot = slots + (size_t)k * kSlotBytes;
                    const double *sv = reinterpret_cast<const double *>(slot);
                    const int *sc = reinterpret_cast<const int *>(slot + kSlotValBytes);
                    const int *sr = reinterpret_cast<const int *>(slot + kSlotValBytes + kSlotColBytes);
                    const int vec = S ? 1 : (c.pt.group_info[t] & 0xff);
                    one = vec == 1;
                    double sum = 0.0;
                    if (one) {
                        if (row[k] >= 0) {
                            const int b = sr[tid], e = sr[tid + 1];
                            for (int i0 = b; i0 < e; i0 += kBatch) {
                                ulonglong2 g[kBatch];
#pragma unroll
                                for (int u = 0; u < kBatch; ++u) g[u] = ld_packet(c.p + sc[i0 + u < e ? i0 + u : i0]);
#pragma unroll
                                for (int u = 0; u < kBatch; ++u)
                                    if (i0 + u < e)
                                        sum = fmac<S>(sv[i0 + u],
                                                      g[u].y == it ? __longlong_as_double((long long)g[u].x)
                                                                   : wait_packet(c, c.p + sc[i0 + u], it, &s_bad),
                                                      sum);
                            }
                            const double q = mtj_assign(sum);
                            s_q[k][tid] = q;
                            part.v[2] = fmac<S>(pv[k], q, part.v[2]);
                        }
                    } else {
                        // 4 or 32 lanes per row, strided entries and k_spmv's butterfly
                        const int gg = vec == 4 ? tid >> 2 : tid >> 5, l = vec == 4 ? tid & 3 : tid & 31;
                        const bool in = gg < rows[k];
                        rows_sync();  // the rows' p is in s_q
                        if (in)
                            for (int i = sr[gg] + l; i < sr[gg + 1]; i += vec)
                                sum = fmac<S>(sv[i], wait_packet(c, c.p + sc[i], it, &s_bad), sum);
                        for (int off = vec / 2; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off, vec);
                        if (in && l == 0) {
                            const double q = mtj_assign(sum);
                            part.v[2] = fmac<S>(s_q[k][gg], q, part.v[2]);
                            s_q[k][gg] = q;
                        }
                    }
                }
                // (rows of several lanes each are spread over the whole block)
                rows_reduce<kSlotsQ>(part, one ? rows[k] : kBlock, nt, red_sm, s_out[k]);
                if (SL > 1) rows_sync();
            }
        } else if (!first && tid == kBlock) {  // the last update's test
            s_st.rho_1 = s_st.rho;
            s_st.iter++;
            const int code = m.check(s_st, 0, norm_finish(s_sum, nt));
            if (code == ST_RUNNING) s_st.rho = s_sum[2];
            m.finish(s_st, code);
        }
        __syncthreads();
        if (s_st.status != ST_RUNNING) break;
        if (rows_thread) {
            publish<kSlotsQ, SL>(c, phase, bid, G, s_out, nt);
            collect<kSlotsQ>(c, phase, nt, all_sm, s_sum, &s_bad);
            ++phase;
            if (tid == 0) s_alpha = rho / s_sum[2];
            rows_sync();
            // x += alpha p, r -= alpha q, z = M r with the |r| and r.z partials
            const double al = s_alpha;
#pragma unroll
            for (int k = 0; k < SL; ++k) {
                Acc part;
                acc_zero(part);
                if (row[k] >= 0) {
                    double rr = rv[k];
                    if (al != 0) {
                        xv[k] = fmac<S>(al, pv[k], xv[k]);
                        rr = fmac<S>(-al, s_q[k][tid], rr);
                        rv[k] = rr;
                    }
                    norm_add<S>(part, rr, nt);
                    zv[k] = rr;
                    if (jac) zv[k] = rr * iv[k];
                    part.v[2] = fmac<S>(rr, zv[k], part.v[2]);
                }
                rows_reduce<kSlotsU>(part, rows[k], nt, red_sm, s_out[k]);
                if (SL > 1) rows_sync();
            }
            publish<kSlotsU, SL>(c, phase, bid, G, s_out, nt);
            collect<kSlotsU>(c, phase, nt, all_sm, s_sum, &s_bad);
            ++phase;
        }
        __syncthreads();
        if (s_bad) return;
        first = false;
        ++it;
    }
#pragma unroll
    for (int k = 0; k < SL; ++k)
        if (row[k] >= 0) {
            c.x[row[k]] = xv[k];
            c.r[row[k]] = rv[k];
        }
    if (bid == 0 && tid == 0) c.m.st[0] = s_st;
}

}  // namespace
}  // namespace mtjg
