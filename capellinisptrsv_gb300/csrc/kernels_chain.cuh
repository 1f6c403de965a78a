// Chain kernel: level-scheduled solves whose levels are narrow, with the
// dependency chain kept inside one SM.
//
// A solve of narrow levels is a serial chain, and the row kernels
// (kernels_row.cuh) pay a publication through L2 for every link of it.  Here
// one block of a thread-block cluster, the chain block, owns the
// chain: its warps take 32 schedule positions ("chunk") at a time, one row per
// lane, and wait for each other's values in a ring in shared memory, which
// holds the latest positions.  A link then costs a shared-memory load, one FMA
// and a shared-memory store instead of a cross-SM hop.
//
// Everything that is not on the chain is done by the other blocks of the
// cluster, the feeders, ahead of time: they read the rows' metadata,
// right-hand sides and entries from global memory, fold the dependencies that
// lie beyond the ring's reach (they poll those in the global publication
// vector, as the row kernels do), and put the partial sums and the remaining,
// near entries into the chain block's shared memory, which reads global memory
// only for rows whose entries do not fit there.
//
// What bounds it (GB300, FP64): the chain.  A link inside a warp costs a round
// of the polling loop, about 240 cycles with the FMA (117 ns; the bare loop of
// load, FMA, store and vote measures 125 cycles, and a loop that lets lanes
// diverge 300), and a row's dependencies that land together cost a round each.
// 1,048,576 Zipf rows in 126k levels: 100.9 ms with the row kernel (0.79 us per
// level), 28.3 ms here (0.22 us); 131,072 rows of 40 dependencies in 87k
// levels: 64.7 -> 10.7 ms; 2,003 rows in 153 levels: 137 -> 29 us (one launch
// instead of two); 20,000 rows in 100 levels: 92 -> 53 us.
//
// Per round a lane loads its next dependency's ring value together with that
// entry's value and the next entry's index, instead of carrying entries in
// registers: moving them along cost more than the loads (20,000 Zipf rows: four
// carried entries 338 ns per level, two 372, none 233).
//
// A cluster's blocks are resident together, so the two roles may wait for one
// another; chunks are fed and taken in schedule order, so the lowest
// unfinished chunk can always proceed.  Every wait is bounded.
//
// Each right-hand side is solved by a cluster of its own, all of them at once:
// 28 clusters of five blocks are resident on a GB300, and more right-hand sides
// get four blocks each.  Five blocks have a feeder warp for each of the up to 64
// slots, and more add nothing (8 blocks: 15 clusters resident, so that 16
// right-hand sides took two turns: 20,000 rows in 493 levels 320 us, 166 us now).
#pragma once

#include "capsp_internal.h"

namespace capsp {

constexpr int kChainThreads = (kChainWarps + 1) * 32;  // and the usher (below)
constexpr int kChainRounds = 6;  // polling rounds between votes on the end of a chunk
constexpr int kChainHeavy = 32;  // far dependencies from which a row is folded by the whole warp
constexpr unsigned kChainSpill = 0xffffffffu;

// shared-memory words of a block, by byte offset (chain block: full, done, ring, slots;
// feeder: freed, staging)
constexpr unsigned kChainFull = 0;       // mbarrier per slot: the slot has been filled
constexpr unsigned kChainDone = 512;     // per chain warp: its first unfinished chunk
constexpr unsigned kChainFreed = 576;    // per feeder warp: latest use its slots are free for
constexpr unsigned kChainRing = 1024;    // ring of values, or a feeder's staging

// A slot: 32 partial sums, rows, and (offset | count << 16) words of the near
// entries (LATE: and right-hand sides and 1/diagonals), then the entries' values and
// their ring indices.
template <typename T, bool LATE>
__host__ __device__ constexpr unsigned chain_slot_bytes(int entries)
{
    return (unsigned)chain_header_bytes(sizeof(T), LATE) + (unsigned)entries * (unsigned)(sizeof(T) + 2);
}

__device__ __forceinline__ unsigned cluster_ctarank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// address of this block's shared-memory location `a` in block `rank` of the cluster
__device__ __forceinline__ unsigned cluster_map(unsigned a, unsigned rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_store16(unsigned a, uint4 v)
{
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

__device__ __forceinline__ void cluster_store_release(unsigned a, unsigned v)
{
    asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned shared_load_acquire(unsigned a)
{
    unsigned v;
    asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

__device__ __forceinline__ void mbar_init(unsigned a, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_cluster(unsigned a)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(a) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned a, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(a), "r"(parity)
                 : "memory");
    return ok != 0u;
}

// A value another warp of the block may be writing: every load is issued
// anew, and an aligned 4- or 8-byte access is all or nothing.  No arithmetic
// result has the pending pattern's upper half (a signalling NaN's).
template <typename T>
__device__ __forceinline__ typename VBits<T>::U ring_load(unsigned at);
template <>
__device__ __forceinline__ unsigned long long ring_load<double>(unsigned at)
{
    unsigned long long v;
    asm volatile("ld.volatile.shared.b64 %0, [%1];" : "=l"(v) : "r"(at));
    return v;
}
template <>
__device__ __forceinline__ unsigned ring_load<float>(unsigned at)
{
    unsigned v;
    asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}
__device__ __forceinline__ unsigned shared_u16(unsigned at)
{
    unsigned short v;
    asm volatile("ld.volatile.shared.u16 %0, [%1];" : "=h"(v) : "r"(at));
    return v;
}
__device__ __forceinline__ bool ring_pending(unsigned long long u)
{
    return (unsigned)(u >> 32) == (unsigned)(VBits<double>::kPending >> 32);
}
__device__ __forceinline__ bool ring_pending(unsigned u) { return u == VBits<float>::kPending; }
__device__ __forceinline__ void ring_store(unsigned at, unsigned long long v)
{
    asm volatile("st.volatile.shared.b64 [%0], %1;" ::"r"(at), "l"(v));
}
__device__ __forceinline__ void ring_store(unsigned at, unsigned v)
{
    asm volatile("st.volatile.shared.b32 [%0], %1;" ::"r"(at), "r"(v));
}

// A wait of the two roles for one another (a slot to fill, a filled slot, a
// warp that lags).  It ends with the partner's progress, which is bounded by
// the partner's own waits for values; two budgets of one wait are the
// backstop.  True: the warp abandons its role (and so, in turn, do those that
// wait for it).
//
// What gives up reports its position p as chain_code(p) where it has no row at hand,
// and what it waits on as a position, or as chain_code(place in the ring); the host
// names the rows (capsp_status_sync).
__device__ __forceinline__ int chain_code(unsigned at) { return -2 - (int)at; }

struct RoleWait {
    unsigned it;
    unsigned long long t0;
    __device__ __forceinline__ RoleWait() : it(0), t0(0) {}
    __device__ __forceinline__ bool expired(const WaitCfg &w, int *err, int p)
    {
        if ((++it & 255u) != 0u)
            return false;
        const unsigned long long now = global_timer_ns();
        if (t0 == 0ull) {
            t0 = now;
            return false;
        }
        if (now - t0 <= 2ull * w.timeout_ns)
            return false;
        if (atomicCAS(err + kErrStatus, 0, kStatusTimeout) == 0) {
            err[kErrRow] = chain_code(p);
            err[kErrWaitedOn] = -1;
        }
        return true;
    }
};

// One far dependency: poll the publication vector until the value is there (a
// quiet NaN when the wait runs out of its budget).
template <typename T>
__device__ __forceinline__ T chain_far_value(const ChainArgs<T> &a, const typename VBits<T>::U *xp, int q,
                                             typename VBits<T>::U u, int p, unsigned long long pol)
{
    typedef VBits<T> VB;
    Spin sp;
    while (u == VB::kPending) {
        if (sp.next(a.err, a.wait, chain_code(p), q))
            return VB::from(VB::kQNaN);
        u = ld_relaxed(xp + q, pol);
    }
    return VB::from(u);
}

// acc + v * u.  A lane sums its row's entries one after the other; in single
// precision what rounding drops on the way is summed beside it and added at the
// end, off the chain (60,000 Zipf rows of 40 and more dependencies, 2-norm against 64
// bits: 5.0e-8, plainly 1.6e-7, the row kernel's tree of 32 lanes 3.7e-8).
__device__ __forceinline__ double chain_fold(double v, double u, double acc, double &) { return fma(v, u, acc); }
__device__ __forceinline__ float chain_fold(float v, float u, float acc, float &low)
{
    const float sum = fmaf(v, u, acc);
    low += fmaf(v, u, acc - sum);
    return sum;
}
__device__ __forceinline__ double chain_sum(double acc, double) { return acc; }
__device__ __forceinline__ float chain_sum(float acc, float low)
{
    // where a sum or a step of its remainder overflowed there is none to add
    const float sum = acc + low;
    return fabsf(sum) <= 3.402823466e38f ? sum : acc;
}

// LATE, for matrices whose rows the row kernels sum a warp at a time: a row's entries
// are summed from zero and its right-hand side joins last, as there, so that the value
// takes one rounding of its own size, not one per entry.  2-norm of the error against
// more than 64 bits, with the right-hand side first / LATE / row kernel: FP64 3.0e-16 /
// 8.4e-17 / 6.8e-17 (131,072 rows of 40 dependencies), 9.2e-17 / 7.8e-17 / 7.6e-17
// (200,000 Zipf rows), 1.36e-16 / 8.9e-17 / 8.1e-17 (2,003 rows of 3-12); FP32 5.0e-8 /
// 3.5e-8 / 3.7e-8, 4.9e-8 / 4.0e-8 / 4.1e-8, 4.6e-8 / 3.9e-8 / 4.1e-8.
//
// In single precision that is an FMA at the row's end (200,000 Zipf rows 3.36 -> 3.39
// ms).  An FP64 one there would hold up every link (1,048,576 Zipf rows 28.3 -> 37.6
// ms), so there the chain carries s = x - b/d: a row's s is the sum of v x over its far
// entries and of v b/d over its near ones, both known to the feeders ahead of time, and
// of v s over the near ones, in the chain.  x = b/d + s is formed off the chain, where it
// is stored (28.4 ms; the 2,003 rows 27.6 -> 29.0 us).
template <typename T, bool LATE>
__host__ __device__ constexpr bool chain_split()
{
    return LATE && sizeof(T) == 8;
}

// what a row hands to the chain, and the value of x
template <typename T, bool LATE>
__device__ __forceinline__ T chain_link(T acc, T low, T bv, T dinv)
{
    const T sum = chain_sum(acc, low);
    return LATE && !chain_split<T, LATE>() ? fma(bv, dinv, sum) : sum;
}
template <typename T, bool LATE>
__device__ __forceinline__ T chain_x(T link, T bv, T dinv)
{
    return chain_split<T, LATE>() ? fma(bv, dinv, link) : link;
}

// b/d of position q
template <typename T>
__device__ __forceinline__ T chain_base(const ChainArgs<T> &a, const T *b, int q)
{
    return __ldg(b + (size_t)__ldg(a.perm + q) * (size_t)a.ld) * __ldg(a.linv + q);
}

// Feeder: chunks c = s, s + step, ... of one slot.
template <typename T, bool LATE>
__device__ __forceinline__ void chain_feed(const ChainArgs<T> &a, unsigned base, unsigned char *smem, int rank,
                                           int warp, int lane, const T *b, const T *xp_r)
{
    typedef VBits<T> VB;
    typedef typename VB::U U;
    const int g = (rank - 1) * kChainWarps + warp;  // feeder number
    const int per_slot = ((a.blocks - 1) * kChainWarps) / a.slots;
    if (g >= per_slot * a.slots)
        return;
    const int s = g % a.slots;
    const unsigned slot_bytes = chain_slot_bytes<T, LATE>(a.entries);
    const unsigned hdr = (unsigned)chain_header_bytes(sizeof(T), LATE);
    unsigned char *mine = smem + kChainRing + (size_t)warp * (slot_bytes + chain_base_bytes(sizeof(T), LATE));
    T *m_acc = reinterpret_cast<T *>(mine);
    int *m_row = reinterpret_cast<int *>(mine + 32 * sizeof(T));
    unsigned *m_meta = reinterpret_cast<unsigned *>(m_row + 32);
    T *m_late = reinterpret_cast<T *>(m_meta + 32);
    T *m_base = reinterpret_cast<T *>(mine + slot_bytes);  // chain_split: b/d of a tile of entries
    T *m_val = reinterpret_cast<T *>(mine + hdr);
    unsigned short *m_idx = reinterpret_cast<unsigned short *>(m_val + a.entries);
    const unsigned dst = cluster_map(base + kChainRing + (unsigned)a.ring * (unsigned)sizeof(U) + 16u + (unsigned)s * slot_bytes, 0);
    const unsigned full = cluster_map(base + kChainFull + 8u * (unsigned)s, 0);
    const unsigned freed = base + kChainFreed + 4u * (unsigned)warp;
    const unsigned long long stream = l2_policy_evict_first(), keep = l2_policy_evict_last();
    const U *xp = reinterpret_cast<const U *>(xp_r);
    const unsigned mask = (unsigned)a.ring - 1u;
    for (int j = g / a.slots;; j += per_slot) {
        const long long c = (long long)j * a.slots + s;
        if (c >= a.nchunks)
            break;
        const int p = (int)(32 * c) + lane;
        const bool act = p < a.n;
        int row = 0, fs = 0, ns = 0, ne = 0;
        T acc = T(0), low = T(0);
        if (act) {
            row = ld_stream(a.perm + p, stream);
            fs = ld_stream(a.lptr + p, stream);
            ns = ld_stream(a.lnear + p, stream);
            ne = ld_stream(a.lptr + p + 1, stream);
            const T bv = ld_stream(b + (size_t)row * (size_t)a.ld, stream), dinv = ld_stream(a.linv + p, stream);
            if (LATE) {
                m_late[lane] = bv;
                m_late[32 + lane] = dinv;
            } else {
                acc = bv * dinv;
            }
        }
        // near entries: one after another in the slot, rows that do not fit are
        // left to the chain block (it then reads them from global memory)
        const int cnt = ne - ns;
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(kFullMask, incl, d);
            if (lane >= d)
                incl += v;
        }
        const int off = incl - cnt;
        const bool spill = incl > a.entries;
        const int whole = __shfl_sync(kFullMask, incl, 31);
        const int total = __reduce_min_sync(kFullMask, spill ? off : whole);
        m_row[lane] = row;
        m_meta[lane] = spill && cnt > 0 ? kChainSpill : ((unsigned)off & 0xffffu) | ((unsigned)cnt << 16);
        constexpr bool split = chain_split<T, LATE>();
        for (int k0 = 0; k0 < total; k0 += 128) {
            int src[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int k = k0 + 32 * t + lane;
                const int l = group_row_of(off, k, 32);
                src[t] = __shfl_sync(kFullMask, ns, l) + k - __shfl_sync(kFullMask, off, l);
            }
            int qi[4];
            T qv[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const bool in = k0 + 32 * t + lane < total;
                qi[t] = in ? ld_stream(a.lidx + src[t], stream) : 0;
                qv[t] = in ? ld_stream(a.lval + src[t], stream) : T(0);
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int k = k0 + 32 * t + lane;
                if (k < total) {
                    m_idx[k] = (unsigned short)((unsigned)qi[t] & mask);
                    m_val[k] = qv[t];
                }
            }
            if constexpr (split) {
                T base[4];
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    base[t] = k0 + 32 * t + lane < total ? chain_base(a, b, qi[t]) : T(0);
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    m_base[(k0 + 32 * t + lane) % kChainTile] = base[t];
                // a tile is there: each lane takes its row's part of it
                const int tile = k0 / kChainTile * kChainTile;
                if (k0 + 128 - tile == kChainTile || k0 + 128 >= total) {
                    __syncwarp();
                    const int k1 = spill ? 0 : min(min(off + cnt, total), tile + kChainTile);
                    for (int k = max(off, tile); k < k1; ++k)
                        acc = fma(m_val[k], m_base[k - tile], acc);
                    __syncwarp();
                }
            }
        }
        if constexpr (split) {
            for (int k = spill ? ns : ne; k < ne; k += 4) {
                T v[4], base[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    v[t] = k + t < ne ? ld_stream(a.lval + k + t, stream) : T(0);
                    base[t] = k + t < ne ? chain_base(a, b, ld_stream(a.lidx + k + t, stream)) : T(0);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (k + t < ne)
                        acc = fma(v[t], base[t], acc);
            }
        }
        // far dependencies of light rows: one row per lane, eight loads in flight
        const bool heavy = ns - fs > kChainHeavy;
        const int fe = heavy ? fs : ns;
        for (int k = fs; k < fe; k += 8) {
            int q[8];
            T v[8];
            U u[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const bool in = k + t < fe;
                q[t] = in ? ld_stream(a.lidx + k + t, stream) : 0;
                v[t] = in ? ld_stream(a.lval + k + t, stream) : T(0);
            }
#pragma unroll
            for (int t = 0; t < 8; ++t)
                u[t] = k + t < fe ? ld_relaxed(xp + q[t], keep) : (U)0;
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (k + t < fe)
                    acc = chain_fold(v[t], chain_far_value<T>(a, xp, q[t], u[t], p, keep), acc, low);
        }
        acc = chain_sum(acc, low);
        // ... of heavy rows: all lanes on one row, then a butterfly sum
        __syncwarp();
        for (unsigned m = __ballot_sync(kFullMask, heavy); m != 0u; m &= m - 1u) {
            const int l = __ffs(m) - 1;
            const int hs = __shfl_sync(kFullMask, fs, l), he = __shfl_sync(kFullMask, ns, l);
            T part = T(0);
            for (int k = hs + lane; k < he; k += 128) {
                int q[4];
                T v[4];
                U u[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const bool in = k + 32 * t < he;
                    q[t] = in ? ld_stream(a.lidx + k + 32 * t, stream) : 0;
                    v[t] = in ? ld_stream(a.lval + k + 32 * t, stream) : T(0);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    u[t] = k + 32 * t < he ? ld_relaxed(xp + q[t], keep) : (U)0;
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (k + 32 * t < he)
                        part = fma(v[t], chain_far_value<T>(a, xp, q[t], u[t], p - lane + l, keep), part);
            }
            __syncwarp();
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1)
                part += __shfl_xor_sync(kFullMask, part, d);
            if (lane == l)
                acc += part;
        }
        m_acc[lane] = acc;
        // the slot, once the chain block is done with its use before this one
        bool late = false;
        if (j > 0) {
            RoleWait rw;
            while (!late && (int)shared_load_acquire(freed) < j)
                late = rw.expired(a.wait, a.err, p);
        }
        if (__any_sync(kFullMask, late))
            return;
        __syncwarp();  // the sums above are other lanes' (a vote orders no memory)
        const unsigned nv = ((unsigned)total * (unsigned)sizeof(T) + 15u) / 16u;
        const unsigned ni = ((unsigned)total * 2u + 15u) / 16u;
        const unsigned vo = hdr / 16u, io = vo + (unsigned)a.entries * (unsigned)sizeof(T) / 16u;
        const uint4 *from = reinterpret_cast<const uint4 *>(mine);
        for (unsigned k = lane; k < vo + nv; k += 32)
            cluster_store16(dst + 16u * k, from[k]);
        for (unsigned k = lane; k < ni; k += 32)
            cluster_store16(dst + 16u * (io + k), from[io + k]);
        __syncwarp();
        if (lane == 0)
            mbar_arrive_cluster(full);
        __syncwarp();
    }
}

// Chain block: chunks c = warp, warp + W, ...
template <typename T, bool LATE>
__device__ __forceinline__ void chain_walk(const ChainArgs<T> &a, unsigned base, unsigned char *smem, int warp,
                                           int lane, T *x, T *xp_r)
{
    typedef VBits<T> VB;
    typedef typename VB::U U;
    const unsigned slot_bytes = chain_slot_bytes<T, LATE>(a.entries);
    const unsigned ring_at = base + kChainRing, never = ring_at + (unsigned)a.ring * (unsigned)sizeof(U);
    unsigned char *slots = smem + kChainRing + (size_t)a.ring * sizeof(U) + 16;
    volatile int *done = reinterpret_cast<volatile int *>(smem + kChainDone);
    const unsigned long long stream = l2_policy_evict_first(), keep = l2_policy_evict_last();
    U *xp = reinterpret_cast<U *>(xp_r);
    const unsigned mask = (unsigned)a.ring - 1u;
    for (int c = warp; c < a.nchunks; c += a.warps) {
        const int j = c / a.slots, s = c - j * a.slots;
        const int p = 32 * c + lane;
        if (a.lag > 0) {
            // The ring is shorter than the solve.  Keep the warps within `lag`
            // chunks of each other, and mark the slots `ahead` chunks on
            // pending: no unfinished chunk reads what they still hold, and no
            // chunk that will read them has started.
            RoleWait rw;
            while (__any_sync(kFullMask, lane < a.warps && done[lane] <= c - a.lag))
                if (__any_sync(kFullMask, rw.expired(a.wait, a.err, p)))
                    return;
            __threadfence_block();
            __syncwarp();  // every lane overwrites what the warps that were seen to be done have read
            ring_store(ring_at + (unsigned)sizeof(U) * (((unsigned)p + 32u * (unsigned)a.ahead) & mask), VB::kPending);
        }
        {
            RoleWait rw;
            bool late = false;
            const unsigned bar = base + kChainFull + 8u * (unsigned)s;
            while (!late && !mbar_try_wait(bar, (unsigned)j & 1u))
                late = rw.expired(a.wait, a.err, p);
            if (__any_sync(kFullMask, late))
                return;
        }
        const unsigned char *slot = slots + (size_t)s * slot_bytes;
        const unsigned slot_at = never + 16u + (unsigned)s * slot_bytes;
        const T *s_val = reinterpret_cast<const T *>(slot + (unsigned)chain_header_bytes(sizeof(T), LATE));
        const unsigned short *s_idx = reinterpret_cast<const unsigned short *>(s_val + a.entries);
        bool open = p < a.n;
        T acc = reinterpret_cast<const T *>(slot)[lane], low = T(0);
        const int row = reinterpret_cast<const int *>(slot + 32 * sizeof(T))[lane];
        const unsigned meta = reinterpret_cast<const unsigned *>(slot + 32 * sizeof(T) + 128)[lane];
        const T *late = reinterpret_cast<const T *>(slot + 32 * sizeof(T) + 256);
        const T bv = LATE && open ? late[lane] : T(0), dinv = LATE && open ? late[32 + lane] : T(0);
        int k = (int)(meta & 0xffffu), left = open && meta != kChainSpill ? (int)(meta >> 16) : 0;
        // a row that must not publish (debug) waits for itself
        const bool stuck = open && row == a.stuck_row;
        const unsigned own = ring_at + (unsigned)sizeof(U) * ((unsigned)p & mask);
        Spin sp;
        unsigned polls = 0;
        if (__any_sync(kFullMask, open && (meta == kChainSpill || stuck))) {
            // some rows' entries did not fit in the slot: these lanes walk them in
            // global memory (their dependencies may lie in this chunk, so the
            // lanes advance together)
            int j0 = 0, j1 = 0;
            if (open && meta == kChainSpill) {
                j0 = ld_stream(a.lnear + p, stream);
                j1 = ld_stream(a.lptr + p + 1, stream);
            }
            bool wait_own = stuck;
            while (__any_sync(kFullMask, open)) {
                if (open) {
                    const bool glob = j0 < j1;
                    if (glob || left > 0 || wait_own) {
                        const unsigned q = glob       ? (unsigned)ld_stream(a.lidx + j0, stream) & mask
                                           : left > 0 ? s_idx[k]
                                                      : (unsigned)p & mask;
                        const T v = glob ? ld_stream(a.lval + j0, stream) : left > 0 ? s_val[k] : T(0);
                        const U u = ring_load<T>(ring_at + (unsigned)sizeof(U) * q);
                        if (!ring_pending(u)) {
                            acc = chain_fold(v, VB::from(u), acc, low);
                            if (glob) {
                                ++j0;
                            } else {
                                ++k;
                                --left;
                            }
                        } else if ((++polls & 15u) == 0u && sp.next(a.err, a.wait, row, chain_code(q))) {
                            acc = VB::from(VB::kQNaN);
                            left = 0;
                            j0 = j1;
                            wait_own = false;
                        }
                    }
                    if (j0 >= j1 && left == 0 && !wait_own) {
                        acc = chain_link<T, LATE>(acc, low, bv, dinv);
                        ring_store(own, VB::to(acc));
                        open = false;
                    }
                }
            }
        } else {
            if (open && left == 0) {
                if (LATE)
                    acc = chain_link<T, LATE>(acc, low, bv, dinv);
                ring_store(own, VB::to(acc));
            }
            // Every round loads, side by side, the ring value of the row's next
            // dependency, that entry's value and the next entry's index; a lane
            // that is done polls the word after the ring, which stays pending.
            // Single precision looks at two dependencies a round and folds the
            // second too when both are there (200,000 Zipf rows: 4.18 -> 3.40 ms;
            // in FP64 the second FMA holds up the lanes that have one: 131,072 rows
            // of 40 dependencies 26 % slower).
            constexpr bool two = sizeof(T) == 4;
            unsigned q0 = never, q1 = never;
            unsigned at_v = slot_at + (unsigned)chain_header_bytes(sizeof(T), LATE) + (unsigned)sizeof(T) * (unsigned)k;
            unsigned at_i = slot_at + (unsigned)chain_header_bytes(sizeof(T), LATE) + (unsigned)sizeof(T) * (unsigned)a.entries + 2u * (unsigned)k;
            if (left > 0)
                q0 = ring_at + (unsigned)sizeof(U) * shared_u16(at_i);
            if (two && left > 1)
                q1 = ring_at + (unsigned)sizeof(U) * shared_u16(at_i + 2u);
            while (__any_sync(kFullMask, left > 0)) {
#pragma unroll
                for (int t = 0; t < (two ? 4 : kChainRounds); ++t) {
                    const U u0 = ring_load<T>(q0), u1 = two ? ring_load<T>(q1) : VB::kPending;
                    const T v0 = VB::from(ring_load<T>(at_v));
                    const T v1 = two ? VB::from(ring_load<T>(at_v + (unsigned)sizeof(T))) : T(0);
                    const unsigned i1 = shared_u16(at_i + (two ? 4u : 2u));
                    const unsigned i2 = two ? shared_u16(at_i + 6u) : 0u;
                    if (!ring_pending(u0)) {
                        acc = chain_fold(v0, VB::from(u0), acc, low);
                        int took = 1;
                        if (two) {
                            q0 = q1;
                            q1 = ring_at + (unsigned)sizeof(U) * i1;
                            if (!ring_pending(u1)) {
                                acc = chain_fold(v1, VB::from(u1), acc, low);
                                q0 = q1;
                                q1 = ring_at + (unsigned)sizeof(U) * i2;
                                took = 2;
                            }
                        } else {
                            q0 = ring_at + (unsigned)sizeof(U) * i1;
                        }
                        at_v += (unsigned)sizeof(T) * (unsigned)took;
                        at_i += 2u * (unsigned)took;
                        left -= took;
                        if (two && left < 2)
                            q1 = never;
                        if (left == 0) {
                            acc = chain_link<T, LATE>(acc, low, bv, dinv);
                            ring_store(own, VB::to(acc));
                            q0 = never;
                        }
                    }
                }
                if ((++polls & 255u) == 0u && left > 0 && sp.next(a.err, a.wait, row, chain_code((q0 - ring_at) / (unsigned)sizeof(U)))) {
                    acc = VB::from(VB::kQNaN);
                    left = 0;
                    q0 = q1 = never;
                    ring_store(own, VB::to(acc));
                }
            }
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0)
            done[warp] = c + a.warps;
        // the caller's x and the publication vector: off the chain
        if (p < a.n && !stuck) {
            const T out = chain_x<T, LATE>(acc, bv, dinv);
            if (xp != nullptr)
                st_relaxed(xp + p, VB::to(out), keep);
            st_stream(reinterpret_cast<U *>(x) + (size_t)row * (size_t)a.ld, VB::to(out), stream);
        }
        __syncwarp();
    }
}

// Usher (the chain block's last warp): hands the slots of finished chunks back
// to the feeders, a lane per chain warp.  A chain warp that did this itself
// would wait, at the cluster-scope release, for its stores of x to reach L2:
// 1.2 us of the 2.1 us it then took per chunk (20,000 rows in 100 levels: 82 us
// against 60 us).
template <typename T>
__device__ __forceinline__ void chain_usher(const ChainArgs<T> &a, unsigned base, unsigned char *smem, int lane)
{
    const volatile int *done = reinterpret_cast<const volatile int *>(smem + kChainDone);
    const int per_slot = ((a.blocks - 1) * kChainWarps) / a.slots;
    int c = lane < a.warps ? lane : a.nchunks;  // the chain warp's chunk to hand back next
    RoleWait rw;
    while (__any_sync(kFullMask, c < a.nchunks)) {
        const bool over = c < a.nchunks && done[lane] > c;
        if (__any_sync(kFullMask, over)) {
            __threadfence_block();
            if (over) {
                const int j = c / a.slots + 1, s = c % a.slots;  // the slot's next use ...
                const int g = (j % per_slot) * a.slots + s;      // ... and its feeder
                cluster_store_release(cluster_map(base + kChainFreed + 4u * (unsigned)(g % kChainWarps),
                                                  1u + (unsigned)(g / kChainWarps)),
                                      (unsigned)j);
                c += a.warps;
            }
            rw = RoleWait();
        } else if (__any_sync(kFullMask, rw.expired(a.wait, a.err, 32 * c))) {
            return;
        }
    }
}

template <typename T, bool LATE>
__global__ void __launch_bounds__(kChainThreads, 1) chain_solve_kernel(const ChainArgs<T> a)
{
    typedef VBits<T> VB;
    typedef typename VB::U U;
    extern __shared__ __align__(16) unsigned char chain_smem[];
    const unsigned base = (unsigned)__cvta_generic_to_shared(chain_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = (int)cluster_ctarank();
    const int rhs = (int)(blockIdx.x / (unsigned)a.blocks);
    if (rank == 0) {
        if (threadIdx.x < (unsigned)a.slots)
            mbar_init(base + kChainFull + 8u * threadIdx.x, 1u);
        if (threadIdx.x < kChainWarps)
            reinterpret_cast<volatile int *>(chain_smem + kChainDone)[threadIdx.x] = (int)threadIdx.x;
        U *ring = reinterpret_cast<U *>(chain_smem + kChainRing);
        for (int k = threadIdx.x; k < a.ring + 1; k += kChainThreads)
            ring[k] = VB::kPending;
        if (a.reset_err && rhs == 0 && threadIdx.x < 4)
            a.err[threadIdx.x] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    } else if (threadIdx.x < kChainWarps) {
        reinterpret_cast<volatile unsigned *>(chain_smem + kChainFreed)[threadIdx.x] = 0u;
    }
    T *xp = a.xp != nullptr ? a.xp + (size_t)rhs * (size_t)a.n : nullptr;
    if (a.fill) {
        // only this cluster polls and publishes here, after its barrier
        const unsigned long long keep = l2_policy_evict_last();
        for (int k = rank * kChainThreads + (int)threadIdx.x; k < a.n; k += a.blocks * kChainThreads)
            st_relaxed(reinterpret_cast<U *>(xp) + k, VB::kPending, keep);
    }
    cluster_sync_all();
    if (rank != 0) {
        if (warp < kChainWarps)
            chain_feed<T, LATE>(a, base, chain_smem, rank, warp, lane, a.b + rhs, xp);
    } else if (warp == kChainWarps)
        chain_usher<T>(a, base, chain_smem, lane);
    else if (warp < a.warps)
        chain_walk<T, LATE>(a, base, chain_smem, warp, lane, a.x + rhs, xp);
    // no block leaves while another may still write to its shared memory
    __syncwarp();
    cluster_sync_all();
}

template <typename T, bool LATE>
static cudaError_t launch_chain(const ChainArgs<T> &a, int nrhs, cudaStream_t st)
{
    const size_t staged =
        (size_t)kChainWarps * (chain_slot_bytes<T, LATE>(a.entries) + (size_t)chain_base_bytes(sizeof(T), LATE));
    const size_t chain = (size_t)a.ring * sizeof(T) + 16 + (size_t)a.slots * chain_slot_bytes<T, LATE>(a.entries);
    const size_t smem = kChainRing + (staged > chain ? staged : chain) + 16;  // the last slot's look-ahead
    // the limit is the kernel's, not the launch's: one value for all handles and threads
    cudaError_t e = cudaFuncSetAttribute(chain_solve_kernel<T, LATE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kChainSmem);
    if (e != cudaSuccess)
        return e;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)a.blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nrhs * a.blocks));
    cfg.blockDim = dim3(kChainThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, chain_solve_kernel<T, LATE>, a);
}

template <typename T>
cudaError_t launch_chain_solve(const ChainArgs<T> &a, int nrhs, cudaStream_t st)
{
    return a.late ? launch_chain<T, true>(a, nrhs, st) : launch_chain<T, false>(a, nrhs, st);
}

}  // namespace capsp
