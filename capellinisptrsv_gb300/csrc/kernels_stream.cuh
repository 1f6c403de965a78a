// Stream kernel: solves of wide levels, bound by throughput.
//
// On such levels almost every dependency has been published long before it is
// asked for, and the row kernels' time goes into getting hold of a chunk (a
// ticket, its metadata, its entries, its right-hand sides, each a round trip
// after the other: 5.4 us of the 7.2 us a chunk of 32 rows took on 2,048 systems
// with 93k rows per level) and into the machinery for rows that wait.  Here the
// warps take chunks of positions in turn, without a ticket, so each knows its next
// rows and loads their metadata and indices while it works on the present ones.
// (With tickets taken as far ahead: 12 % slower on the batch, 1.05 -> 1.17 ms on
// 1,000 rows per level with 16 RHS.)  Readiness is the row kernels': a value in the
// publication vector is pending or it is the value.  A warp asks for all
// dependencies of its rows at once; what has not arrived is asked for again.
//
// Turns need every block to run.  The blocks count themselves as they start, and
// where they do not all run within 20 us, the warps take tickets instead.  Either
// way the lowest unfinished position belongs to a running warp that has finished
// its earlier ones, so the solve proceeds; every wait is bounded.  (A cooperative
// launch would guarantee as much, but held up another stream's memset for the
// length of two solves.)
//
// Layout (capsp_stream_slices, launch_stream_layout): the rows of a level, those
// of more dependencies first, in slices of 8; a slice's entries are stored entry
// by entry, all rows' first ones, all rows' second ones, ..., so 8 indices fill
// a 32-byte sector and 8 values two, padded (-1) to the slice's longest row.
// Positions are numbered with the padding, and index the publication vector.
//
// G lanes share a row, R right-hand sides each, loaded together.
//
// What bounds it (GB300): in FP64 with several right-hand sides the FP64 pipe
// (1,024 systems of 11.0 M rows, 16 RHS: 3.46 ms, where its FMAs take 2.4 ms;
// the row kernel 6.52 ms); otherwise the loads in flight per SM (2,048 systems of
// 22.0 M rows, 1 RHS: 1.13 ms, 2.5 TB/s of matrix and vectors; the row kernel
// 1.64 ms; FP32, 16 RHS, 1,024 systems: 2.2 against 5.3 ms).
#pragma once

#include "capsp_internal.h"

namespace capsp {

// R consecutive values of the publication vector; each is pending or final
__device__ __forceinline__ void stream_poll(const unsigned long long *p, unsigned long long (&v)[1], unsigned long long pol)
{
    v[0] = ld_relaxed(p, pol);
}
__device__ __forceinline__ void stream_poll(const unsigned *p, unsigned (&v)[1], unsigned long long pol)
{
    v[0] = ld_relaxed(p, pol);
}
__device__ __forceinline__ void stream_poll(const unsigned long long *p, unsigned long long (&v)[2], unsigned long long pol)
{
    asm volatile("ld.relaxed.gpu.global.L2::cache_hint.v2.b64 {%0, %1}, [%2], %3;"
                 : "=l"(v[0]), "=l"(v[1])
                 : "l"(p), "l"(pol));
}
__device__ __forceinline__ void stream_poll(const unsigned *p, unsigned (&v)[2], unsigned long long pol)
{
    asm volatile("ld.relaxed.gpu.global.L2::cache_hint.v2.b32 {%0, %1}, [%2], %3;"
                 : "=r"(v[0]), "=r"(v[1])
                 : "l"(p), "l"(pol));
}
__device__ __forceinline__ void stream_publish(unsigned long long *p, const unsigned long long (&v)[1], unsigned long long pol)
{
    st_relaxed(p, v[0], pol);
}
__device__ __forceinline__ void stream_publish(unsigned *p, const unsigned (&v)[1], unsigned long long pol)
{
    st_relaxed(p, v[0], pol);
}
__device__ __forceinline__ void stream_publish(unsigned long long *p, const unsigned long long (&v)[2], unsigned long long pol)
{
    asm volatile("st.relaxed.gpu.global.L2::cache_hint.v2.b64 [%0], {%1, %2}, %3;" ::"l"(p), "l"(v[0]), "l"(v[1]), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void stream_publish(unsigned *p, const unsigned (&v)[2], unsigned long long pol)
{
    asm volatile("st.relaxed.gpu.global.L2::cache_hint.v2.b32 [%0], {%1, %2}, %3;" ::"l"(p), "r"(v[0]), "r"(v[1]), "l"(pol)
                 : "memory");
}

// Spin (capsp_device.cuh) whose clock starts anew where `it` was set back to 0: the
// budget is a single wait's, and lanes that are done never look at the clock
struct StreamSpin {
    unsigned it;
    unsigned long long t0;
    __device__ __forceinline__ StreamSpin() : it(0), t0(0) {}
    __device__ __forceinline__ bool next(int *err, const WaitCfg &w, int row)
    {
        ++it;
        if (it > 4u && w.sleep_max_ns) {
            unsigned s = 32u << (it - 5u < 6u ? it - 5u : 6u);
            __nanosleep(s < w.sleep_max_ns ? s : w.sleep_max_ns);
        }
        if ((it & 15u) == 0u) {
            if (ld_relaxed(reinterpret_cast<const unsigned *>(err)) != 0u)
                return true;
            const unsigned long long now = global_timer_ns();
            if (it == 16u) {
                t0 = now;
            } else if (now - t0 > w.timeout_ns || it > w.max_iters) {
                if (atomicCAS(err + kErrStatus, 0, kStatusTimeout) == 0) {
                    err[kErrRow] = row;
                    err[kErrWaitedOn] = -1;
                }
                return true;
            }
        }
        return false;
    }
};

// A lane's row, as far as it is loaded ahead of time
template <typename T, int TB>
struct StreamRow {
    int at;   // first entry
    int len;  // entries, with its slice's padding
    int row;  // < 0: none
    T dinv;
    int idx[TB];
};

// How the grid's warps share the chunks out, decided when the kernel starts.
// kStreamTurns: warp w of W takes chunks w, w + W, ... (every block is running;
// the last one to start says so).  kStreamTickets: a ticket per chunk, where some
// block is not running yet, say behind another stream's work, after
// kStreamStartNs.
constexpr unsigned long long kStreamStartNs = 20000;

// words[0]: tickets, [1]: blocks that run, [2]: the decision
__device__ __forceinline__ int stream_start(unsigned *words)
{
    if (atomicAdd(words + 1, 1u) == gridDim.x - 1u)
        atomicCAS(words + 2, (unsigned)kStreamUndecided, (unsigned)kStreamTurns);
    const unsigned long long t0 = global_timer_ns();
    unsigned how;
    while ((how = ld_acquire(words + 2)) == kStreamUndecided)
        if (global_timer_ns() - t0 > kStreamStartNs)
            atomicCAS(words + 2, (unsigned)kStreamUndecided, (unsigned)kStreamTickets);
    return (int)how;
}

template <typename T, int TB>
__device__ __forceinline__ void stream_load(const StreamArgs<T> &a, long long p, int2 rec, unsigned long long pol,
                                            StreamRow<T, TB> &w)
{
    w.at = rec.x + (int)(p & 7);
    w.len = rec.y;
    w.row = -1;
    w.dinv = T(0);
    if (p < a.npos) {
        w.row = ld_stream(a.row + p, pol);
        w.dinv = ld_stream(a.linv + p, pol);
    }
#pragma unroll
    for (int t = 0; t < TB; ++t)
        w.idx[t] = t < w.len ? ld_stream(a.idx + w.at + 8 * t, pol) : -1;
}

// Slots [a0, a1) of the lane's batch into acc, one slot after the other up to hi
// (the warp's largest a1).  Nested, so that the slots past hi are branched
// around: a warp-wide FP64 FMA holds its pipe for 64 cycles even when every
// lane has it predicated off.
template <int t, int END, typename T, int TB, int R>
__device__ __forceinline__ void stream_fold(int hi, int a0, int a1, const T (&val)[TB],
                                            const typename VBits<T>::U (&u)[TB][R], T (&acc)[R])
{
    if constexpr (t < END) {
        if (t < hi) {
            if (t >= a0 && t < a1) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    acc[r] = fma(val[t], VBits<T>::from(u[t][r]), acc[r]);
            }
            stream_fold<t + 1, END>(hi, a0, a1, val, u, acc);
        }
    }
}

template <typename T, int G, int R, int TB, bool TURNS>
__device__ __forceinline__ void stream_rows(const StreamArgs<T> &a)
{
    typedef VBits<T> VB;
    typedef typename VB::U U;
    constexpr int RPW = 32 / G;
    const int lane = threadIdx.x & 31;
    const int rl = lane / G, r0 = lane % G * R;
    const unsigned long long stream = l2_policy_evict_first(), keep = l2_policy_evict_last();
    U *const xp = reinterpret_cast<U *>(a.xp) + r0;
    const auto record = [&](long long p) {
        return p < a.npos ? __ldg(a.slice + (p >> 3)) : make_int2(0, 0);
    };
    // the lane's position in the warp's next chunk; in turns, neighbouring chunks
    // go to different SMs, and a ticket is asked for long before it is needed
    const long long step = (long long)(blockDim.x >> 5) * gridDim.x * RPW;
    long long next = ((long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * RPW + rl;
    unsigned ticket = !TURNS && lane == 0 ? atomicAdd(a.words, 1u) : 0u;
    const auto advance = [&]() {
        const long long at = TURNS ? next : (long long)__shfl_sync(kFullMask, ticket, 0) * RPW + rl;
        if (TURNS)
            next += step;
        else if (lane == 0)
            ticket = atomicAdd(a.words, 1u);
        return at;
    };
    StreamRow<T, TB> cur, nxt;
    long long p = advance();
    int2 rec = record(p);
    stream_load<T, TB>(a, p, rec, stream, nxt);
    long long p1 = advance();
    rec = record(p1);
    while (p - rl < a.npos) {
        cur = nxt;
        const bool mine = cur.row >= 0 && r0 < a.nrhs;
        T val[TB], acc[R], bv[R];
        U u[TB][R];
#pragma unroll
        for (int t = 0; t < TB; ++t) {
            val[t] = T(0);
#pragma unroll
            for (int r = 0; r < R; ++r)
                u[t][r] = (U)0;
            if (mine && cur.idx[t] >= 0) {
                stream_poll(xp + (size_t)cur.idx[t] * (G * R), u[t], keep);
                val[t] = ld_stream(a.val + cur.at + 8 * t, stream);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            bv[r] = mine && r0 + r < a.nrhs ? ld_stream(a.b + (size_t)cur.row * (size_t)a.ld + r0 + r, stream) : T(0);
        stream_load<T, TB>(a, p1, rec, stream, nxt);
        const long long p2 = advance();
        rec = record(p2);
#pragma unroll
        for (int r = 0; r < R; ++r)
            acc[r] = bv[r] * cur.dinv;
        // the batch's slots: cnt real entries, the first nacc of them folded
        unsigned pend = 0u;
        int cnt = 0, nacc = 0, t0 = 0;
        const auto take_stock = [&]() {
            pend = 0u;
            cnt = 0;
#pragma unroll
            for (int t = 0; t < TB; ++t) {
                bool late = false;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    late = late || u[t][r] == VB::kPending;
                pend |= late ? 1u << t : 0u;
                cnt += cur.idx[t] >= 0 ? 1 : 0;
            }
        };
        take_stock();
        bool open = mine;
        StreamSpin sp;
        for (;;) {
            // single precision folds a row when all of it has arrived; an FP64 FMA
            // takes so long that the part that has arrived is folded meanwhile
            const int ready = pend ? (sizeof(T) == 4 ? 0 : __ffs(pend) - 1) : cnt;
            const bool can = open && nacc < ready;
            const int hi = __reduce_max_sync(kFullMask, can ? ready : 0);
            if (hi > 0) {
                const int lo = __reduce_min_sync(kFullMask, can ? nacc : TB);
                const int a1 = can ? ready : 0;
                if (lo < 4)
                    stream_fold<0, 4>(hi, nacc, a1, val, u, acc);
                if (hi > 4 && lo < 8)
                    stream_fold<4, 8>(hi, nacc, a1, val, u, acc);
                if (hi > 8)
                    stream_fold<(TB > 8 ? 8 : TB), TB>(hi, nacc, a1, val, u, acc);
                nacc = can ? ready : nacc;
            }
            if (open && pend == 0u && nacc == cnt) {
                t0 += TB;
                if (t0 < cur.len) {  // a longer row: its next entries
#pragma unroll
                    for (int t = 0; t < TB; ++t) {
                        const bool in = t0 + t < cur.len;
                        cur.idx[t] = in ? ld_stream(a.idx + cur.at + 8 * (t0 + t), stream) : -1;
                        val[t] = in ? ld_stream(a.val + cur.at + 8 * (t0 + t), stream) : T(0);
                    }
#pragma unroll
                    for (int t = 0; t < TB; ++t) {
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            u[t][r] = (U)0;
                        if (cur.idx[t] >= 0)
                            stream_poll(xp + (size_t)cur.idx[t] * (G * R), u[t], keep);
                    }
                    nacc = 0;
                    take_stock();
                    sp.it = 0;
                } else {
                    U out[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        out[r] = VB::to(acc[r]);
                        if (r0 + r < a.nrhs)
                            st_stream(reinterpret_cast<U *>(a.x) + (size_t)cur.row * (size_t)a.ld + r0 + r, out[r], stream);
                    }
                    stream_publish(xp + (size_t)p * (G * R), out, keep);
                    open = false;
                }
            }
            if (!__any_sync(kFullMask, open))
                break;
            if (sp.next(a.err, a.wait, cur.row) && open) {
                // give up: a quiet NaN, so that the dependants end too
                if (a.err[kErrRow] == cur.row && a.err[kErrWaitedOn] < 0) {
                    int q = -1;
#pragma unroll
                    for (int t = TB - 1; t >= 0; --t)
                        q = (pend >> t) & 1u ? cur.idx[t] : q;
                    const int on = q >= 0 ? a.row[q] : -1;
                    a.err[kErrWaitedOn] = on < -1 ? stream_unpublished(on) : on;
                }
                U out[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    out[r] = VB::kQNaN;
                    if (r0 + r < a.nrhs)
                        st_stream(reinterpret_cast<U *>(a.x) + (size_t)cur.row * (size_t)a.ld + r0 + r, out[r], stream);
                }
                stream_publish(xp + (size_t)p * (G * R), out, keep);
                open = false;
            }
            // ask again for what has not arrived
            const unsigned ask = open ? pend : 0u;
#pragma unroll
            for (int t = 0; t < TB; ++t)
                if ((ask >> t) & 1u)
                    stream_poll(xp + (size_t)cur.idx[t] * (G * R), u[t], keep);
            unsigned got = 0u;
#pragma unroll
            for (int t = 0; t < TB; ++t) {
                bool late = false;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    late = late || u[t][r] == VB::kPending;
                got |= ((ask >> t) & 1u) && !late ? 1u << t : 0u;
            }
            pend &= ~got;
            // the budget is a single wait's, and a lane that is done has none (its
            // count stays below the first look at the clock)
            sp.it = got || !open ? 0u : sp.it;
        }
        p = p1;
        p1 = p2;
    }
}

template <typename T, int G, int R, int TB, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1) stream_solve_kernel(const StreamArgs<T> a)
{
    __shared__ int how;
    if (threadIdx.x == 0)
        how = stream_start(a.words);
    __syncthreads();
    if (how == kStreamTurns)
        stream_rows<T, G, R, TB, true>(a);
    else
        stream_rows<T, G, R, TB, false>(a);
}

template <typename T, int G, int R, int TB, int BLOCK>
static cudaError_t launch_stream_g(const StreamArgs<T> &a, int warps, int num_sms, cudaStream_t st)
{
    const int block = warps * 32 < BLOCK ? warps * 32 : BLOCK;
    const long long rows = 32 / G * (block / 32);  // per round of a block
    const long long need = (a.npos + rows - 1) / rows;
    const unsigned grid = (unsigned)(need < num_sms ? (need > 0 ? need : 1) : num_sms);
    stream_solve_kernel<T, G, R, TB, BLOCK><<<grid, block, 0, st>>>(a);
    return cudaGetLastError();
}

// One right-hand side per lane: rows of up to 8 entries in one go with up to 20
// warps per SM, of up to 12 with 16 (what the registers allow).  Launches of up to
// 12 warps take a build for as many, which has a third more registers (FP64, 1,000
// rows per level, 16 RHS: 1,009 us; 1,054 us with the build for 16).
template <typename T, int G>
static cudaError_t launch_stream_single(const StreamArgs<T> &a, bool long_rows, int warps, int num_sms, cudaStream_t st)
{
    if constexpr (G >= 4) {
        if (warps <= 12)
            return long_rows ? launch_stream_g<T, G, 1, 12, 384>(a, warps, num_sms, st)
                             : launch_stream_g<T, G, 1, 8, 384>(a, warps, num_sms, st);
    }
    return long_rows ? launch_stream_g<T, G, 1, 12, 512>(a, warps, num_sms, st)
                     : launch_stream_g<T, G, 1, 8, 640>(a, warps, num_sms, st);
}

template <typename T>
cudaError_t launch_stream_solve(const StreamArgs<T> &a, bool long_rows, bool pairs, int warps, int num_sms,
                                cudaStream_t st)
{
    const int cols = lanes_for_rhs(a.nrhs);
    if (pairs || cols == 32) {
        switch (cols) {
        case 4: return launch_stream_g<T, 2, 2, 8, 512>(a, warps, num_sms, st);
        case 8: return launch_stream_g<T, 4, 2, 8, 512>(a, warps, num_sms, st);
        case 16: return launch_stream_g<T, 8, 2, 8, 512>(a, warps, num_sms, st);
        case 32: return launch_stream_g<T, 16, 2, 8, 512>(a, warps, num_sms, st);
        default: break;
        }
    }
    switch (cols) {
    case 1: return launch_stream_single<T, 1>(a, long_rows, warps, num_sms, st);
    case 2: return launch_stream_single<T, 2>(a, long_rows, warps, num_sms, st);
    case 4: return launch_stream_single<T, 4>(a, long_rows, warps, num_sms, st);
    case 8: return launch_stream_single<T, 8>(a, long_rows, warps, num_sms, st);
    default: return launch_stream_single<T, 16>(a, long_rows, warps, num_sms, st);
    }
}

// The layout of a view whose level layout is in place, a thread per position:
// rows, entries' positions, source indices into the stored values, and the
// view's values as they stand.  `place` (a view position's position here) may
// lie in linv's memory, which is written by the last launch.
static __global__ void __launch_bounds__(256) stream_place_kernel(const int *__restrict__ pos, long long npos,
                                                           int *__restrict__ place)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += stride)
        if (pos[p] >= 0)
            place[pos[p]] = (int)p;
}

template <typename T>
__global__ void __launch_bounds__(256) stream_layout_kernel(const StreamBuild<T> a)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < a.npos; p += stride) {
        const int2 rec = a.slice[p >> 3];
        const int q = a.pos[p];
        a.row[p] = q >= 0 ? a.perm[q] : -1;
        const int j0 = q >= 0 ? a.lptr[q] : 0, j1 = q >= 0 ? a.lptr[q + 1] : 0;
        for (int t = 0; t < rec.y; ++t) {
            const int k = rec.x + 8 * t + (int)(p & 7);
            const bool in = j0 + t < j1;
            a.idx[k] = in ? a.place[a.lidx[j0 + t]] : -1;
            a.src[k] = in ? a.lsrc[j0 + t] : -1;
            a.val[k] = in ? a.lval[j0 + t] : T(0);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) stream_linv_kernel(const StreamBuild<T> a)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < a.npos; p += stride)
        a.linv[p] = a.pos[p] >= 0 ? a.view_linv[a.pos[p]] : T(0);
}

template <typename T>
cudaError_t launch_stream_layout(const StreamBuild<T> &a, cudaStream_t st)
{
    long long blocks = (a.npos + 255) / 256;
    if (blocks > 16384)
        blocks = 16384;
    if (blocks < 1)
        blocks = 1;
    stream_place_kernel<<<(unsigned)blocks, 256, 0, st>>>(a.pos, a.npos, a.place);
    stream_layout_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(a);
    stream_linv_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(a);
    return cudaGetLastError();
}

// New values for the view and its stream layout in one pass (level_values_kernel
// does the same for a view without one), a thread per position: 1/diagonal, and
// every entry's -v/d into the slices and into the view's row.
template <typename T>
__global__ void __launch_bounds__(256) stream_values_kernel(const StreamBuild<T> a, const int *__restrict__ diag_src,
                                                            const T *__restrict__ stored, T *__restrict__ view_linv,
                                                            T *__restrict__ lval, int *bad)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < a.npos; p += stride) {
        const int2 rec = a.slice[p >> 3];
        const int q = a.pos[p];
        if (q < 0)
            continue;  // padding stays zero
        const T dg = stored[diag_src[q]];
        if (!(dg != T(0)) || !isfinite(dg))
            atomicMin(bad, q);
        const T d = T(1) / dg;
        a.linv[p] = d;
        view_linv[q] = d;
        const int j0 = a.lptr[q];
        const int at = rec.x + (int)(p & 7);
        for (int t0 = 0; t0 < rec.y; t0 += 8) {
            int j[8];
            T v[8];
#pragma unroll
            for (int t = 0; t < 8; ++t)
                j[t] = t0 + t < rec.y ? __ldg(a.src + at + 8 * (t0 + t)) : -1;
#pragma unroll
            for (int t = 0; t < 8; ++t)
                v[t] = j[t] >= 0 ? __ldg(stored + j[t]) : T(0);
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (j[t] >= 0) {
                    const T out = -v[t] * d;
                    a.val[at + 8 * (t0 + t)] = out;
                    lval[j0 + t0 + t] = out;
                }
        }
    }
}

template <typename T>
cudaError_t launch_stream_values(const StreamBuild<T> &a, const int *diag_src, const T *stored, T *view_linv, T *lval,
                                 int *bad, cudaStream_t st)
{
    long long blocks = (a.npos + 255) / 256;
    if (blocks > 16384)
        blocks = 16384;
    if (blocks < 1)
        blocks = 1;
    stream_values_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(a, diag_src, stored, view_linv, lval, bad);
    return cudaGetLastError();
}

}  // namespace capsp
