// The Coulomb build of one cluster in one pass over the packed fitted tensor.
//
// J = sum_q c_q B_q with c_q = <B_q, D> (hafnium/scf/coulomb_exchange.py:176-182)
// needs every element of B_q twice: for c_q, which is complete only when the
// whole row has been read, and for J. Two kernels (jk.cu, still used for batches
// and past this form's sizes) therefore read B from HBM twice. Here each CTA owns
// a slice of the elements (mu <= nu) and keeps its part of the last rows on the
// SM until their c_q is known, so B is read once and the bound is one pass of HBM.
//
//   * The grid is groups of E CTAs, one CTA per SM. A group takes a range of rows
//     q, its CTAs a slice of the upper triangle each. Only elements mu <= nu < n
//     are read (16-byte pieces), not the lower half of the diagonal tiles nor the
//     padding. The slice's density and J stay in registers.
//   * 16 worker warps move their own pieces with cp.async into private shared
//     memory slots (no barrier between the copy and its use), form partial dot
//     products, put the pieces into tensor memory, which nothing else uses here,
//     and take them back when c_q is known: 256 KB per SM of waiting rows (about
//     5 us of HBM traffic) beside the 200 KB in flight.
//   * A publishing warp adds the workers' partial sums and sends them to the
//     group through global memory; collecting warps add the group's partials in
//     CTA order. A packet is 16 bytes, {low, tag, high, tag} (the layout of NCCL's
//     low-latency protocol): each 8-byte half carries its own tag, so a packet is
//     complete when both tags match and no fence or counter is needed. A tag is
//     used once between two zeroings of the workspace, which is zeroed whenever
//     something else may lie in it (PacketSpace): no value of another kernel's
//     data can pass for a packet.
//     Groups of more than 32 CTAs send to an owner of the row that hands out the
//     sum (two hops, but 2 E packets instead of E^2 reads of them).
//   * The CTAs wait on one another: a small grid is one thread-block cluster, a
//     larger one a cooperative launch. Every wait is bounded; past the limit the
//     kernel records an error and runs to its end. Waits poll device memory only
//     (polling the host's flag took up to 100 us).
//
// Measured on one B200 (kernels of one J with the timing events, two-pass ->
// one-pass): (H2O)8 153 -> 61 us, (H2O)12 240 -> 134, (H2O)16 457 -> 280,
// (H2O)32 2741 -> 1870 (8.55 GB: 4.6 TB/s; without the exchange of c it runs in
// 1600, so what is left is the latency of two hops and 130 for the long sums),
// (H2O)44 7120 -> 5120. Past four pieces per thread (n about 1100) registers spill
// and the rows that tensor memory holds no longer cover the exchange: six pieces
// measured 7.9 ms at n = 1152 without the exchange and three times that with it,
// against 8.7 in two passes.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "coulomb.cuh"
#include "integrals.cuh"


namespace hf {

namespace {

constexpr int kWorkers = 512;            // worker threads (16 warps)
constexpr int kLane = 8;     // groups up to this size: a collecting lane per row adds the partials
constexpr int kDirect = 32;  // ... up to this size: a warp per row; larger groups through an owner of each row
constexpr int kCollectors = 3;           // collecting warps (20 warps in all: five per scheduler)
constexpr int kThreads = kWorkers + 32 + 32 * kCollectors;
constexpr int kPrefetch = 2;             // row blocks in flight beyond the current one
constexpr int kTmemDoubles = 64;         // a worker thread's share of tensor memory (512 columns x 128 lanes x 4 B)
constexpr int kParts = 2;                 // shared buffers of partial sums
constexpr int kCluster = 8;               // grids up to this size are one thread-block cluster
constexpr int kFewRows = 8;               // blocks of more rows are summed over a warp by the workers
// Rows of one running sum of J; longer ones are added up in memory. One sum over all rows of a group
// erred by 6.7e-16 of J at (H2O)16 and 2.1e-15 at (H2O)32, the two-pass form's slabs by 3.7e-16 and
// 4.1e-16; sums of 128 rows err by 4.6e-16 at both, of 88 by 3.7e-16 and 3.8e-16 (of 64 by 3.1e-16 and
// 3.7e-16). One addition of all CTAs' sums takes about 6 us, all CTAs at once: at different times each
// held up the others ((H2O)32 1.93 -> 2.40 ms).
constexpr int kChain = 88;
constexpr int kBarW = 1, kBarEnd = 2;    // named barriers: workers; workers and publisher at the end

struct FusedArgs {
    const double* B;
    int64_t ldb;
    int n, nt, naux;
    const double* D;
    double scale;
    double* J;
    uint4* packets;             // [groups of CTAs][ns][qb][ge]
    uint4* sums;                // [groups of CTAs][ns][qb]
    double2* jpart;             // [gq][ge * pp]
    unsigned long long* jflag;  // [gq][ge]
    uint32_t tag;               // tags of this launch: tag + row block, and tag + blocks for J
    uint32_t sent;              // ... as the CTAs send them: `tag`, or, in the self-test, tags that none waits for
    uint32_t* stop;             // becomes `tag` when a wait has run out (device memory: polled by every wait)
    int* err;                   // ... and this becomes 1 (host memory: only ever written)
    uint64_t wait_ns;
    int ge, gq;   // CTAs per group, groups
    int pp;       // pieces per CTA
    int total;    // pieces in the upper triangle
    int tpq, ql;  // threads per row, rows side by side
    int b;        // rows per thread and block
    int lag;      // blocks between a dot product and its use
    int nr;       // shared buffers of c
    int ns;       // packet slots
    int rows;     // rows per group
    int blocks;   // row blocks per group
    int flush;    // row blocks between two additions of the sums of J to jsum
    double2* jsum;  // [gq * ge][ql][pp]
};

__device__ __forceinline__ void bar_sync(int id, int threads) {
    __syncwarp();  // bar counts whole warps
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(saddr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(saddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void put_packet(uint4* p, double v, uint32_t tag) {
    const uint64_t x = (uint64_t)__double_as_longlong(v);
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "r"((uint32_t)x), "r"(tag),
                 "r"((uint32_t)(x >> 32)), "r"(tag)
                 : "memory");
}
__device__ __forceinline__ uint4 get_packet(const uint4* p) {
    uint4 r;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p)
                 : "memory");
    return r;
}
__device__ __forceinline__ double packet_value(const uint4& r) {
    return __longlong_as_double((long long)(((uint64_t)r.z << 32) | r.x));
}

__device__ __forceinline__ bool stopped(const FusedArgs& a) { return *(volatile uint32_t*)a.stop == a.tag; }
__device__ __forceinline__ void give_up(const FusedArgs& a) {
    *(volatile uint32_t*)a.stop = a.tag;
    *(volatile int*)a.err = 1;
}

// Bounded wait for a barrier of this CTA: past the limit, or once any wait of the launch has run
// out, the caller goes on (its results are then undefined, its accesses stay in bounds). A collector
// that has given up passes through all remaining row blocks at once, and its arrivals no longer fit
// the workers' parities: a worker that waited for each of them ran out for each of them.
// The clock and the stop word are read out of line, after the waits that matter: with the clock in
// the loop (H2O)32 took 2.08 ms, with both 2.15, this way 1.83.
__device__ __noinline__ void mbar_wait_long(uint64_t* bar, uint32_t parity, const FusedArgs& a) {
    const uint64_t start = now_ns();
    for (uint32_t i = 1; !mbar_try(bar, parity); ++i)
        if ((i & 15) == 0) {
            const bool late = now_ns() - start > 4 * a.wait_ns;
            if (late) give_up(a);
            if (late || stopped(a)) return;
        }
}
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, const FusedArgs& a) {
    for (int i = 0; i < 256; ++i)
        if (mbar_try(bar, parity)) return;
    mbar_wait_long(bar, parity, a);
}

// A warp's pieces of one row to and from tensor memory: W 32-bit registers per lane, W columns.
template <int W>
__device__ __forceinline__ void tmem_put(uint32_t at, const uint32_t (&r)[W]) {
    static_assert(W == 4 || W == 8 || W == 16, "1, 2 or 4 pieces");
    if constexpr (W == 4)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(at), "r"(r[0]), "r"(r[1]),
                     "r"(r[2]), "r"(r[3])
                     : "memory");
    if constexpr (W == 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(at), "r"(r[0]),
                     "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                     : "memory");
    if constexpr (W == 16)
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::
                "r"(at),
            "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
            "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
            : "memory");
}
template <int W>
__device__ __forceinline__ void tmem_get(uint32_t at, uint32_t (&r)[W]) {
    if constexpr (W == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(at));
    if constexpr (W == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(at));
    if constexpr (W == 16)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(at));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// The value of packet p, read into r before: waits (bounded) until its tags match;
// `dead` threads no longer wait.
__device__ __forceinline__ double wait_packet(const uint4* p, uint4 r, uint32_t tag, const FusedArgs& a, bool& dead) {
    if (r.y == tag && r.w == tag) return packet_value(r);
    if (dead) return 0.0;
    const uint64_t start = now_ns();
    for (uint32_t i = 1;; ++i) {
        r = get_packet(p);
        if (r.y == tag && r.w == tag) return packet_value(r);
        if ((i & 127) == 0) {
            const bool late = now_ns() - start > a.wait_ns;
            if (late) give_up(a);
            if (late || stopped(a)) {
                dead = true;
                return 0.0;
            }
        }
    }
}

// The sums of NQ rows (nq of them wanted) over the CTAs' packets by a warp, each lane's in CTA order:
// all loads leave before the first is waited for. The sums are in every lane.
template <int NQ, int NP>
__device__ __forceinline__ void collect(const uint4* in, int nq, uint32_t tag, const FusedArgs& a, bool& dead,
                                        double (&s)[NQ]) {
    const int lane = threadIdx.x & 31;
    uint4 r[NQ][NP];
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
        for (int j = 0; j < NP; ++j) r[q][j] = get_packet(in + min(q, nq - 1) * a.ge + min(lane + 32 * j, a.ge - 1));
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        s[q] = 0.0;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const double v =
                wait_packet(in + min(q, nq - 1) * a.ge + min(lane + 32 * j, a.ge - 1), r[q][j], tag, a, dead);
            if (lane + 32 * j < a.ge) s[q] += v;
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
}

// Pieces (two neighbouring columns, the first even) of the upper triangle, tile
// by tile in storage order: diagonal tiles from the diagonal on, tiles of the
// last column up to n.
__device__ __forceinline__ void locate(int idx, int n, int nt, int& off, int& u, int& v) {
    const int last = n - 64 * (nt - 1), hl = (last + 1) >> 1;
    // tile rows: a diagonal tile (1056 pieces), nt - 2 - I full ones, the last column's
    int I = 0, left = idx, line = 1056 + 2048 * (nt - 2) + 64 * hl;
    while (I < nt - 1 && left >= line) {
        left -= line;
        line -= 2048;
        ++I;
    }
    int J = I, r, c, h = I == nt - 1 ? hl : 32;
    if (I == nt - 1 || left < 1056) {
        // rows 2k and 2k + 1 of a diagonal tile start at piece k
        int k = 0;
        while (left >= 2 * (h - k)) {
            left -= 2 * (h - k);
            ++k;
        }
        r = 2 * k;
        if (left >= h - k) {
            left -= h - k;
            ++r;
        }
        c = k + left;
    } else {
        left -= 1056;
        const int t = min(nt - 2 - I, left >> 11);
        J = I + 1 + t;
        left -= t << 11;
        h = J == nt - 1 ? hl : 32;
        r = h == 32 ? left >> 5 : left / h;
        c = left - r * h;
    }
    u = 64 * I + r;
    v = 64 * J + 2 * c;
    off = ((I * nt - I * (I - 1) / 2) + (J - I)) * 4096 + r * 64 + 2 * c;
}

// Columns of one row in a thread's tensor-memory share: its doubles, padded to a transfer of 4, 8 or
// 16 registers.
template <int EPT>
__host__ __device__ constexpr int tmem_width() {
    return EPT == 1 ? 4 : EPT == 2 ? 8 : 16;
}

// LONG: a thread's rows are more than one running sum takes. Without that code, whose registers they
// need, the small sizes are 3 % faster.
template <int EPT, bool LONG>
__global__ void __launch_bounds__(kThreads, 1) k_coulomb_fused(const __grid_constant__ FusedArgs a) {
    constexpr int TW = tmem_width<EPT>();
    extern __shared__ __align__(16) uint8_t smem[];
    const int qb = a.ql * a.b, lanes = a.ql * a.tpq;
    uint64_t* bar_a = reinterpret_cast<uint64_t*>(smem);      // [kParts] a block's partials written
    uint64_t* bar_p = bar_a + kParts;                         // [kParts] ... and read
    uint64_t* bar_b = bar_p + kParts;                         // [nr] c of a block ready
    double* part = reinterpret_cast<double*>(bar_b + a.nr);   // [kParts][qb][tpq]
    double* cbuf = part + kParts * qb * a.tpq;                // [nr][qb]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(cbuf + a.nr * qb);
    double2* slots = reinterpret_cast<double2*>((reinterpret_cast<uintptr_t>(tmem_slot) + 4 + 15) & ~uintptr_t(15));
    // [(kPrefetch + 1) * b][EPT][lanes]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int e = blockIdx.x % a.ge, grp = blockIdx.x / a.ge;
    const bool few = qb <= kFewRows;
    const int q0 = grp * a.rows, q1 = min(a.naux, q0 + a.rows);
    uint4* packets = a.packets + (int64_t)grp * a.ns * qb * a.ge;

    if (warp == kWorkers / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(saddr(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        for (int i = 0; i < kParts; ++i) {
            mbar_init(&bar_a[i], lanes >> 5);
            mbar_init(&bar_p[i], 1);
        }
        for (int i = 0; i < a.nr; ++i) {
            mbar_init(&bar_b[i], 1);
        }
    }

    const int lq = tid / a.tpq, tl = tid - lq * a.tpq;
    const bool mine = lq < a.ql;  // the same for a whole warp
    // where the thread's pieces lie in a row: in registers, or, where the long sums need those, in shared memory
    int4* kept = reinterpret_cast<int4*>(slots + (kPrefetch + 1) * a.b * EPT * lanes) + tid;
    int off[4] = {0, 0, 0, 0};
    uint32_t on = 0;
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
        const int i = k * a.tpq + tl, idx = e * a.pp + i;
        if (warp < kWorkers / 32 && mine && i < a.pp && idx < a.total) {
            int u, v;
            locate(idx, a.n, a.nt, off[k], u, v);
            on |= 1u << k;
        }
    }
    if (LONG && warp < kWorkers / 32 && mine) *kept = make_int4(off[0], off[1], off[2], off[3]);
    auto issue = [&](int g) {
        if (g < a.blocks) {
            if constexpr (LONG) {
                const int4 o = *kept;
                off[0] = o.x;
                off[1] = o.y;
                off[2] = o.z;
                off[3] = o.w;
            }
            for (int s = 0; s < a.b; ++s) {
                const int q = q0 + g * qb + s * a.ql + lq;
                if (q >= q1) break;
                const double* row = a.B + (int64_t)q * a.ldb;
                double2* dst = slots + ((g % (kPrefetch + 1)) * a.b + s) * (EPT * lanes) + tid;
#pragma unroll
                for (int k = 0; k < EPT; ++k)
                    if (on >> k & 1)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(saddr(dst + k * lanes)),
                                     "l"(row + off[k])
                                     : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (warp < kWorkers / 32 && mine)
#pragma unroll
        for (int g = 0; g < kPrefetch; ++g) issue(g);

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == kWorkers / 32) {  // publisher
        int buf = 0, par = 0, cb = 0, ps = 0;
        for (int g = 0; g < a.blocks; ++g) {
            mbar_wait(&bar_a[buf], par, a);
            __syncwarp();
            const double* p = part + buf * qb * a.tpq;
            double* c = cbuf + cb * qb;
            uint4* out = packets + (int64_t)ps * qb * a.ge + e;
            if (!few)
                for (int q = lane; q < qb; q += 32) {
                    double v = 0.0;
                    for (int i = 0; i < a.tpq; i += 32) v += p[q * a.tpq + i];
                    if (a.ge == 1) c[q] = v;
                    else put_packet(out + q * a.ge, v, a.sent + g);
                }
            for (int q = 0; few && q < qb; ++q, p += a.tpq) {
                double v = 0.0, w = 0.0;
#pragma unroll 4
                for (int i = lane; i < a.tpq; i += 64) {
                    v += p[i];
                    if (i + 32 < a.tpq) w += p[i + 32];
                }
                v += w;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) {
                    if (a.ge == 1) c[q] = v;
                    else put_packet(out + q * a.ge, v, a.sent + g);
                }
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bar_p[buf]);
                if (a.ge == 1) mbar_arrive(&bar_b[cb]);
            }
            if (++buf == kParts) {
                buf = 0;
                par ^= 1;
            }
            cb = cb == a.nr - 1 ? 0 : cb + 1;
            ps = ps == a.ns - 1 ? 0 : ps + 1;
        }
        bar_sync(kBarEnd, kWorkers + 32);  // the workers have read their last columns
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
        return;
    }
    if (warp > kWorkers / 32) {  // collectors: c_q in CTA order, the rows dealt out in turn
        if (a.ge == 1) return;
        bool dead = false;
        const int w = warp - kWorkers / 32 - 1;
        if (a.ge <= kLane) {  // a lane per row adds the CTAs' partials
            for (int g = w; g < a.blocks; g += kCollectors) {
                const uint4* in = packets + (int64_t)(g % a.ns) * qb * a.ge;
                double* c = cbuf + (g % a.nr) * qb;
                for (int q = lane; q < qb; q += 32) {
                    uint4 r[kLane];
#pragma unroll
                    for (int j = 0; j < kLane; ++j) r[j] = get_packet(in + q * a.ge + min(j, a.ge - 1));
                    double s = 0.0;
#pragma unroll
                    for (int j = 0; j < kLane; ++j)
                        if (j < a.ge) s += wait_packet(in + q * a.ge + j, r[j], a.tag + g, a, dead);
                    c[q] = s;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_b[g % a.nr]);
            }
            return;
        }
        if (a.ge <= kDirect) {  // a warp per row block
            for (int g = w; g < a.blocks; g += kCollectors) {
                const uint4* in = packets + (int64_t)(g % a.ns) * qb * a.ge;
                double* c = cbuf + (g % a.nr) * qb;
                for (int q = 0; q < qb; q += 2, in += 2 * a.ge, c += 2) {
                    double s[2];
                    collect<2, 1>(in, qb - q, a.tag + g, a, dead, s);
                    if (lane < 2 && lane < qb - q) c[lane] = lane ? s[1] : s[0];
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_b[g % a.nr]);
            }
            return;
        }
        uint4* sums = a.sums + (int64_t)grp * a.ns * qb;
        if (w == 0) {  // owner of every ge-th row: adds its partials, hands out the sum
            for (int q = e; q < a.blocks * qb; q += a.ge) {
                const int g = q / qb, r = q - g * qb, slot = g % a.ns;
                double s[1];
                collect<1, 5>(packets + ((int64_t)slot * qb + r) * a.ge, 1, a.tag + g, a, dead, s);
                if (lane == 0) put_packet(sums + slot * qb + r, s[0], a.tag + g);
            }
            return;
        }
        for (int g = w - 1; g < a.blocks; g += kCollectors - 1) {
            const uint4* in = sums + (g % a.ns) * qb;
            for (int q = lane; q < qb; q += 32)
                cbuf[(g % a.nr) * qb + q] = wait_packet(in + q, get_packet(in + q), a.tag + g, a, dead);
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_b[g % a.nr]);
        }
        return;
    }

    double2 acc[EPT];
#pragma unroll
    for (int k = 0; k < EPT; ++k) acc[k] = make_double2(0.0, 0.0);
    // this thread's own entries of jsum: nobody else touches them
    auto sums_at = [&] { return a.jsum + ((int64_t)blockIdx.x * a.ql + lq) * a.pp + tl; };
    auto add_up = [&](bool more) {
        double2* t = sums_at();
#pragma unroll
        for (int k = 0; k < EPT; ++k) {
            if (on >> k & 1) {
                if (more) {  // additions that nothing waits for
                    atomicAdd(&t[k * a.tpq].x, acc[k].x);
                    atomicAdd(&t[k * a.tpq].y, acc[k].y);
                } else {
                    __stcg(t + k * a.tpq, acc[k]);
                }
            }
            acc[k] = make_double2(0.0, 0.0);
        }
    };
    auto take_sums = [&] {
        const double2* t = sums_at();
#pragma unroll
        for (int k = 0; k < EPT; ++k)
            if (on >> k & 1) {
                const double2 v = __ldcg(t + k * a.tpq);
                acc[k].x += v.x;
                acc[k].y += v.y;
            }
    };
    if (mine) {
        // weights: D[mu][nu] + D[nu][mu] above the diagonal, D[mu][mu] on it, 0 below and past n
        double2 d[EPT];
#pragma unroll
        for (int k = 0; k < EPT; ++k) {
            d[k] = make_double2(0.0, 0.0);
            if (!(on >> k & 1)) continue;
            int o, u, v;
            locate(e * a.pp + k * a.tpq + tl, a.n, a.nt, o, u, v);
            const double* du = a.D + (int64_t)u * a.n + v;
            const double* dv = a.D + (int64_t)v * a.n + u;
            if (v >= u) d[k].x = a.scale * (v == u ? du[0] : du[0] + dv[0]);
            if (v + 1 < a.n) d[k].y = a.scale * (v + 1 == u ? du[1] : du[1] + dv[a.n]);
        }
        const uint32_t mine_tmem = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * (2 * kTmemDoubles);
        int slot = 0, buf = 0, bpar = 1, put = 0;  // g modulo the smem ring, kParts and lag
        int get = 0, hbuf = 0, hpar = 0;  // the same for the block to be used
        [[maybe_unused]] int left = a.flush;
        for (int g = 0; g < a.blocks + a.lag - 1; ++g) {
            if (g < a.blocks) {
                issue(g + kPrefetch);
                asm volatile("cp.async.wait_group %0;\n" ::"n"(kPrefetch) : "memory");
                mbar_wait(&bar_p[buf], bpar, a);  // the buffer's previous partials have been read
                __syncwarp();
                double* p = part + buf * qb * a.tpq + lq * a.tpq + tl;
                for (int s = 0; s < a.b; ++s) {
                    const bool valid = q0 + g * qb + s * a.ql + lq < q1;
                    const double2* src = slots + (slot * a.b + s) * (EPT * lanes) + tid;
                    const uint32_t at = mine_tmem + (uint32_t)((put * a.b + s) * TW);
                    double x = 0.0, y = 0.0;
                    uint32_t r[TW];
#pragma unroll
                    for (int k = 0; k < TW / 4; ++k) {
                        double2 v = make_double2(0.0, 0.0);
                        if (k < EPT) {
                            if (valid && (on >> k & 1)) v = src[k * lanes];
                            x += d[k < EPT ? k : 0].x * v.x;
                            y += d[k < EPT ? k : 0].y * v.y;
                        }
                        r[4 * k] = (uint32_t)__double2loint(v.x);
                        r[4 * k + 1] = (uint32_t)__double2hiint(v.x);
                        r[4 * k + 2] = (uint32_t)__double2loint(v.y);
                        r[4 * k + 3] = (uint32_t)__double2hiint(v.y);
                    }
                    __syncwarp();
                    tmem_put(at, r);
                    x += y;
                    if (few) {
                        p[s * lanes] = x;
                    } else {
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                        if (lane == 0) p[s * lanes] = x;
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_a[buf]);
                slot = slot == kPrefetch ? 0 : slot + 1;
                if (++buf == kParts) {
                    buf = 0;
                    bpar ^= 1;
                }
                put = put == a.lag - 1 ? 0 : put + 1;
            }
            // the block that this one's columns replace next: `lag` - 1 blocks behind
            const int h = g - a.lag + 1;
            if (h >= 0) {
                mbar_wait(&bar_b[hbuf], hpar, a);
                __syncwarp();
                const double* c = cbuf + hbuf * qb;
                for (int s = 0; s < a.b; ++s) {
                    const double cq = c[s * a.ql + lq];
                    const uint32_t at = mine_tmem + (uint32_t)((get * a.b + s) * TW);
                    uint32_t r[TW];
                    tmem_get(at, r);
#pragma unroll
                    for (int k = 0; k < EPT; ++k) {
                        acc[k].x += cq * __hiloint2double((int)r[4 * k + 1], (int)r[4 * k]);
                        acc[k].y += cq * __hiloint2double((int)r[4 * k + 3], (int)r[4 * k + 2]);
                    }
                }
                if (++hbuf == a.nr) {
                    hbuf = 0;
                    hpar ^= 1;
                }
                get = get == a.lag - 1 ? 0 : get + 1;
                if constexpr (LONG)
                    if (--left == 0) {
                        left = a.flush;
                        add_up(h >= a.flush);
                    }
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        if constexpr (LONG) take_sums();
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    bar_arrive(kBarEnd, kWorkers + 32);

    // rows side by side: the first row's threads add the others' sums in order
    if (a.ql > 1) {
        bar_sync(kBarW, kWorkers);
        if (mine && lq > 0)
#pragma unroll
            for (int k = 0; k < EPT; ++k) slots[k * lanes + tid] = acc[k];
        bar_sync(kBarW, kWorkers);
        if (lq == 0)
            for (int r = 1; r < a.ql; ++r)
#pragma unroll
                for (int k = 0; k < EPT; ++k) {
                    const double2 v = slots[k * lanes + r * a.tpq + tl];
                    acc[k].x += v.x;
                    acc[k].y += v.y;
                }
    }
    auto store = [&](int idx, double2 v) {
        int o, u, w;
        locate(idx, a.n, a.nt, o, u, w);
        if (w >= u) {
            a.J[(int64_t)u * a.n + w] = v.x;
            a.J[(int64_t)w * a.n + u] = v.x;
        }
        if (w + 1 < a.n) {
            a.J[(int64_t)u * a.n + w + 1] = v.y;
            a.J[(int64_t)(w + 1) * a.n + u] = v.y;
        }
    };
    if (a.gq == 1) {
        if (lq == 0)
#pragma unroll
            for (int k = 0; k < EPT; ++k)
                if (on >> k & 1) store(e * a.pp + k * a.tpq + tl, acc[k]);
        return;
    }
    // groups: every CTA of a slice adds its share of the slice over the groups, in order
    if (lq == 0)
#pragma unroll
        for (int k = 0; k < EPT; ++k)
            if (on >> k & 1) __stcg(a.jpart + ((int64_t)grp * a.ge + e) * a.pp + k * a.tpq + tl, acc[k]);
    auto flag = [&](uint32_t tag) { return ((unsigned long long)(tag + a.blocks) << 32) | (uint32_t)~(tag + a.blocks); };
    const unsigned long long done = flag(a.tag);
    bar_sync(kBarW, kWorkers);
    if (tid == 0) {
        __threadfence();
        *(volatile unsigned long long*)(a.jflag + grp * a.ge + e) = flag(a.sent);
    }
    if (tid < a.gq) {
        const volatile unsigned long long* f = a.jflag + tid * a.ge + e;
        const uint64_t start = now_ns();
        for (uint32_t i = 1; *f != done; ++i)
            if ((i & 127) == 0) {
                const bool late = now_ns() - start > a.wait_ns;
                if (late) give_up(a);
                if (late || stopped(a)) break;
            }
        __threadfence();
    }
    bar_sync(kBarW, kWorkers);
    const int share = (a.pp + a.gq - 1) / a.gq;
    for (int i = grp * share + tid; i < min(a.pp, (grp + 1) * share); i += kWorkers) {
        if (e * a.pp + i >= a.total) break;
        double2 v[4] = {};  // four chains: the sum errs half as much, and its loads are ahead of it
        auto add = [&](int m, int r) {
            const double2 x = __ldcg(a.jpart + ((int64_t)r * a.ge + e) * a.pp + i);
            v[m].x += x.x;
            v[m].y += x.y;
        };
        int r = 0;
#pragma unroll 4
        for (; r + 3 < a.gq; r += 4)
#pragma unroll
            for (int m = 0; m < 4; ++m) add(m, r + m);
        for (; r < a.gq; ++r) add(0, r);
        store(e * a.pp + i, make_double2((v[0].x + v[1].x) + (v[2].x + v[3].x), (v[0].y + v[1].y) + (v[2].y + v[3].y)));
    }
}

template <int EPT, bool LONG>
cudaError_t launch_fused(const FusedArgs& a, size_t smem, cudaStream_t stream) {
    const cudaError_t e = allow_shared((const void*)k_coulomb_fused<EPT, LONG>, smem);
    if (e != cudaSuccess) return e;
    // the grid's CTAs wait on one another: a cluster, or a cooperative grid
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(a.ge * a.gq);
    c.blockDim = dim3(kThreads);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    cudaLaunchAttribute at[1];
    if (a.ge * a.gq <= kCluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = a.ge * a.gq;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k_coulomb_fused<EPT, LONG>, a);
}


int64_t upper_pieces(int64_t n, int nt) {
    int64_t total = 0;
    const int last = (int)(n - 64 * (int64_t)(nt - 1));
    for (int I = 0; I < nt; ++I) {
        const int rows = I == nt - 1 ? last : 64, h = (rows + 1) / 2, k = rows / 2;
        total += rows * h - k * (k - 1) - ((rows & 1) ? k : 0);
        if (I < nt - 1) total += (int64_t)(nt - 2 - I) * 2048 + (int64_t)rows * ((last + 1) / 2);
    }
    return total;
}

// A thread's rows are more than one running sum takes.
bool long_sums(const FusedArgs& a) { return a.blocks >= a.flush; }

constexpr int kMaxPieces = 4;         // pieces of a row per thread
// Up to this many pieces (rows times pieces of a row) one cluster of 8 CTAs holds everything; past it
// the rows are spread out over groups. Whole calls, cluster against spread out: 1800 pieces (n = 7) 39.0
// and 40.8 us, 12700 (n = 14) 43.6 and 44.4, 17600 (one water, n = 24) 41.9 and 42.6, 44000 (n = 21) 46.8
// and 44.7, 95000 (n = 28) 49.8 and 44.6.
constexpr int64_t kSmallPieces = 20000;

// How the work is laid out; ept == 0 when the fused form does not apply.
struct FusedShape {
    FusedArgs a;
    int ept;
    size_t smem;
};

FusedShape plan_coulomb(const JkPlan& p, int sms) {
    FusedShape f{};
    if (p.n < 1 || p.naux < 1 || p.n > 30000) return f;
    FusedArgs& a = f.a;
    a.total = (int)upper_pieces(p.n, p.nt);
    const int most = kWorkers * kMaxPieces;
    a.ge = (a.total + most - 1) / most;
    if (a.ge > sms) return f;
    const bool small = a.ge == 1 && (int64_t)a.total * p.naux <= kSmallPieces;
    if (small) sms = kCluster;
    a.gq = small ? 1 : std::max(1, std::min(sms / a.ge, (p.naux + 1) / 2));
    a.ge = sms / a.gq;
    a.ge = std::max(1, std::min(a.ge, (a.total + 31) / 32));
    a.pp = (a.total + a.ge - 1) / a.ge;
    a.ge = (a.total + a.pp - 1) / a.pp;
    f.ept = (a.pp + kWorkers - 1) / kWorkers;
    if (f.ept > kMaxPieces) {
        f.ept = 0;
        return f;
    }
    a.tpq = ((a.pp + f.ept - 1) / f.ept + 31) / 32 * 32;
    a.rows = (p.naux + a.gq - 1) / a.gq;
    a.gq = (p.naux + a.rows - 1) / a.rows;
    a.ql = std::max(1, std::min(kWorkers / a.tpq, a.rows));
    const size_t slot = (size_t)a.ql * a.tpq * f.ept * 16;
    // rows per thread and block that shared memory holds: pieces in flight and partial sums
    const int fit = (int)(216 * 1024 / (slot * (kPrefetch + 1) + (size_t)8 * kParts * a.ql * a.tpq));
    if (fit < 1) {
        f.ept = 0;
        return f;
    }
    const int width = f.ept == 1 ? 4 : f.ept == 2 ? 8 : 16;  // tmem_width
    const int depth = 2 * kTmemDoubles / width;                                // rows of a thread held in tensor memory
    a.b = std::max(1, std::min({fit, depth / 4, (a.rows + a.ql - 1) / a.ql}));
    a.lag = depth / a.b;
    const int qb = a.ql * a.b;
    a.blocks = (a.rows + qb - 1) / qb;
    a.lag = std::min(a.lag, a.blocks);
    a.flush = std::max(1, kChain / a.b);
    a.nr = a.lag + 2;
    a.ns = 2 * a.lag + 2;
    f.smem = 8 * (size_t)(2 * kParts + a.nr) + 8 * ((size_t)kParts * qb * a.tpq + a.nr * qb) + 32 +
             slot * (kPrefetch + 1) * a.b + (long_sums(a) ? (size_t)16 * a.ql * a.tpq : 0);
    return f;
}

size_t packet_bytes(const FusedArgs& a) { return (size_t)16 * a.gq * a.ns * a.ql * a.b * a.ge; }
size_t sum_bytes(const FusedArgs& a) { return (size_t)16 * a.gq * a.ns * a.ql * a.b; }
size_t jpart_bytes(const FusedArgs& a) { return (size_t)16 * a.gq * a.ge * a.pp; }
size_t jsum_bytes(const FusedArgs& a) { return long_sums(a) ? (size_t)16 * a.gq * a.ge * a.ql * a.pp : 0; }

size_t flag_bytes(const FusedArgs& a) { return ((size_t)8 * a.gq * a.ge + 15) / 16 * 16 + 16; }  // and the stop word
// what a build tells from older contents by its tags, at the front of the workspace
size_t tagged_bytes(const FusedArgs& a) { return packet_bytes(a) + sum_bytes(a) + flag_bytes(a); }

int device_sms() {
    static std::atomic<int> sms[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int v = sms[dev].load();
    if (v == 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        sms[dev].store(v);
    }
    return v;
}

}  // namespace

size_t coulomb_fused_work_doubles(const JkPlan& p) {
    const FusedShape f = plan_coulomb(p, device_sms());
    if (!f.ept) return 0;
    return (tagged_bytes(f.a) + jpart_bytes(f.a) + jsum_bytes(f.a)) / 8 + 2;
}

bool coulomb_fused_cooperative(const JkPlan& p) {
    const FusedShape f = plan_coulomb(p, device_sms());
    return f.ept && f.a.ge * f.a.gq > kCluster;
}

namespace {
struct Turns {
    std::mutex mutex;
    uint64_t last = 0;       // number of the last turn
    bool busy = false;       // ... which has not been left
    cudaStream_t stream{};   // ... its stream
    cudaEvent_t mark{};      // ... and its event, if it has one
    cudaEvent_t event{};     // for those that have none
};
Turns g_turns[64];
Turns& turns_of(int device) { return g_turns[device >= 0 && device < 64 ? device : 0]; }
}  // namespace

std::mutex& CooperativeTurn::mutex() { return turns_of(device_).mutex; }

cudaError_t CooperativeTurn::follow(cudaStream_t stream) {
    Turns& t = turns_of(device_);
    if (!t.busy) return cudaSuccess;
    if (t.mark) return cudaStreamWaitEvent(stream, t.mark, 0);
    cudaError_t e = t.event ? cudaSuccess : cudaEventCreateWithFlags(&t.event, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(t.event, t.stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, t.event, 0);
    return e;
}

cudaError_t CooperativeTurn::take(cudaStream_t stream, cudaEvent_t mark) {
    Turns& t = turns_of(device_);
    number_ = ++t.last;
    t.busy = true;
    t.stream = stream;
    t.mark = mark;
    return mark ? cudaEventRecord(mark, stream) : cudaSuccess;
}

void CooperativeTurn::leave() {
    if (!number_) return;
    Turns& t = turns_of(device_);
    std::lock_guard<std::mutex> lock(t.mutex);
    if (t.last == number_) t.busy = false;
    number_ = 0;
}

cudaError_t coulomb_build_fused(const JkPlan& p, const double* D, double scale, double* J, double* work,
                                PacketSpace& held, int* err, uint64_t wait_ns, int stall, CooperativeTurn& turn,
                                cudaEvent_t mark, cudaStream_t stream) {
    const FusedShape f = plan_coulomb(p, device_sms());
    if (!f.ept) return cudaErrorInvalidValue;
    FusedArgs a = f.a;
    a.B = p.B;
    a.ldb = p.ldb;
    a.n = (int)p.n;
    a.nt = p.nt;
    a.naux = p.naux;
    a.D = D;
    a.scale = scale;
    a.J = J;
    a.packets = reinterpret_cast<uint4*>((reinterpret_cast<uintptr_t>(work) + 15) & ~uintptr_t(15));
    a.sums = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(a.packets) + packet_bytes(a));
    a.jflag = reinterpret_cast<unsigned long long*>(reinterpret_cast<uint8_t*>(a.sums) + sum_bytes(a));
    a.stop = reinterpret_cast<uint32_t*>(a.jflag + (size_t)a.gq * a.ge);
    a.jpart = reinterpret_cast<double2*>(reinterpret_cast<uint8_t*>(a.packets) + tagged_bytes(a));
    a.jsum = a.jpart + (size_t)a.gq * a.ge * a.pp;
    // no word of the tagged part holds a tag of this build: it holds smaller tags of builds of this shape, or zeros
    const uint32_t tags = ((uint32_t)a.blocks + 1) * (stall ? 2 : 1);
    if (held.next == 0 || held.n != p.n || held.naux != p.naux || held.next > UINT32_MAX - tags) {
        held.next = 0;
        const cudaError_t e = cudaMemsetAsync(a.packets, 0, tagged_bytes(a), stream);
        if (e != cudaSuccess) return e;
        held = PacketSpace{p.n, p.naux, 1};
    }
    a.tag = held.next;
    a.sent = a.tag + tags - ((uint32_t)a.blocks + 1);
    held.next += tags;
    a.err = err;
    a.wait_ns = wait_ns;
    auto launch = [&] {
        const bool more = long_sums(a);
        switch (f.ept) {
            case 1: return more ? launch_fused<1, true>(a, f.smem, stream) : launch_fused<1, false>(a, f.smem, stream);
            case 2: return more ? launch_fused<2, true>(a, f.smem, stream) : launch_fused<2, false>(a, f.smem, stream);
            case 3: return more ? launch_fused<3, true>(a, f.smem, stream) : launch_fused<3, false>(a, f.smem, stream);
            case 4: return more ? launch_fused<4, true>(a, f.smem, stream) : launch_fused<4, false>(a, f.smem, stream);
            default: return cudaErrorInvalidValue;
        }
    };
    return a.ge * a.gq > kCluster ? turn.enter(stream, mark, launch) : launch();
}

}  // namespace hf
