// stop_kernels.cu -- SATOSTOP pointer doubling over 32-bit entries
// (next | STOP << n, n <= 31).
//
// Round r of synchronous doubling (greedysatostop.rs:858-866 join_nexts) makes
// every entry advance 2^r evaluations: T_r[s] = T_{r-1}[T_{r-1}[s]], an entry
// with STOP staying where it is.  A round over the whole table is one random
// gather per entry, which the L1 tag stage limits to one per SM clock while
// the table lies in L2 (2^24 entries: 64 us) and random HBM sectors beyond
// (2^28 entries: 5 ms).  Three things keep the work per solve down:
//
// - distances are not gathered: every entry that has not stopped stands for
//   exactly 2^r evaluations, so only the entries that stop carry one, written
//   once in the round in which they stop.  A table with steps moves 12 bytes
//   per entry and round instead of 24 (2^24-state counter: 61 us -> 37 us a
//   round);
//
// - the domain is contracted.  A next-state function that is not a bijection
//   has an image that shrinks with every iteration (for a random function to
//   0.20 of the states after three rounds), and a later round only looks up
//   states of that image.  With I the image after round r0 and P = T_r0 on I,
//   the table after round r0 + k is Q_k o T_r0, where on I
//     P_{k+1} = P_k o P_k,   Q_{k+1} = P_k o Q_k,   Q_0 = the identity
//   (P_k makes 2^(r0+k) evaluations, Q_k makes 2^(r0+k) - 2^r0).  The same
//   contraction applies again to the image of Q_k on I.  Entries there are
//   64-bit, value | distance << 32: an entry that has not stopped holds an id
//   of its own domain, one that has stopped the halting state with STOP.
//   start[id] is the lowest unknown start that has reached the id, so each
//   round's answer is found without the table (24 rounds over 2^24 entries of
//   a register with a mixer: 1.55 ms -> 0.85 ms; 28 over 2^28: 140 -> 26 ms);
//
// - tables of up to 2^14 entries run every round in one CTA with the table in
//   shared memory (2^12 entries with distances, 12 rounds: 53 us as launches,
//   24 us);
//
// - and tables of up to 2^20 in one cooperative launch with a grid barrier per
//   round: a launch per round costs 3 us, and the rounds behind the answer
//   were launched too (a solve answered after 6 rounds of 2^16 entries with
//   distances 91 -> 35 us, after 15 rounds of 2^15 without 86 -> 55 us, after
//   5 rounds of 2^20 with 147 -> 54 us).
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"
#include "stop_kernels.h"

typedef unsigned int u32;
typedef unsigned long long u64;

namespace {

constexpr u32 kNone = 0xffffffffu;

// An odd multiplier is a bijection of the n-bit states; the states whose
// image has its top 8 bits clear are a 256th of them, spread over the table.
// Returns 1 for the first of equal ones.
__device__ __forceinline__ u32 sample_mark(u32* sample, u32 v, u32 bits) {
    const u32 h = (v * 0x9E3779B1u) & (u32)((1ull << bits) - 1ull);
    if ((h >> (bits - 8)) != 0u) return 0u;
    const u32 m = 1u << (h & 31u);
    u32* w = sample + (h >> 5);
    return !(*w & m) && !(atomicOr(w, m) & m) ? 1u : 0u;
}

// An answered round ends the loop: later rounds carry the answer forward and
// do no work.
__device__ __forceinline__ bool answered(NsatStopState* st, u32 r, u32 mode) {
    if (r <= 1) return false;
    const u32 pb = *(volatile u32*)&st->best[r - 1];
    if (pb == kNone || (mode != 0 && pb != 0)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->best[r] = pb;
        if (st->final_round == 0) st->final_round = r - 1;
    }
    return true;
}

// Whether rounds 1 .. r hold the answer (a contraction after round r is moot).
__device__ __forceinline__ bool moot(const NsatStopState* st, u32 r, u32 mode) {
    const u32 b = *(volatile const u32*)&st->best[r];
    return b != kNone && (mode == 0 || b == 0);
}

template <bool DIST, bool SAMPLE>
__global__ void __launch_bounds__(256) join32(const u32* src, u32* dst, u32* dist, u64 N, u32 n, u32 u, u32 r, u32 mode,
                                              NsatStopState* __restrict__ st, u32* __restrict__ sample) {
    pdl_wait();
    if (answered(st, r, mode)) return;
    const u32 stop = 1u << n, nmask = stop - 1u;
    const u32 smask = (u32)((1ull << (n - u)) - 1ull);
    const u32 half = 1u << (r - 1);      // evaluations an entry of src stands for
    u32 best = kNone, fresh = 0;
    const u64 S = (u64)gridDim.x * blockDim.x;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += 4 * S) {
        // four independent gathers in flight per thread
        u32 v[4], w[4];
        bool ok[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const u64 j = i + (u64)k * S;
            ok[k] = j < N;
            v[k] = ok[k] ? src[j] : stop;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = (v[k] & stop) ? v[k] : src[v[k] & nmask];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (!ok[k]) continue;
            const u64 j = i + (u64)k * S;
            __stcs(dst + j, w[k]);      // leaves the L2 to src, which the gathers reread (2^24 entries: 5 %)
            if (w[k] & stop) {
                if constexpr (DIST) {
                    // an entry of src that has stopped has its distance from the
                    // round it stopped in (round 1 writes those of the table built)
                    if (!(v[k] & stop)) dist[j] = half + (r == 1 ? 1u : dist[v[k]]);
                    else if (r == 1) dist[j] = 1u;
                }
                if (((u32)j & smask) == 0u && (u32)j < best) best = (u32)j;
            } else if constexpr (SAMPLE) {
                fresh += sample_mark(sample, w[k], n);
            }
        }
    }
    if constexpr (SAMPLE) {
        fresh = __reduce_add_sync(0xffffffffu, fresh);
        if ((threadIdx.x & 31) == 0 && fresh) atomicAdd(&st->distinct, fresh);
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if ((threadIdx.x & 31) == 0 && best != kNone) atomicMin(&st->best[r], best);
}

// All rounds in one CTA.  A thread keeps the entries tid + k * 1024 in
// registers; the table in shared memory is only read by the gathers, so a
// round is gathers, a barrier, stores, a barrier.  With STEPS the distances of
// the entries that have stopped follow the table in shared memory.
constexpr int kSmallThreads = 1024;
template <bool STEPS, int E>
__global__ void __launch_bounds__(kSmallThreads) small_solve(const u32* __restrict__ src, u32 n, u32 u, u32 mode,
                                                             u32* __restrict__ out32, u64* __restrict__ out64,
                                                             volatile u64* words, u32 seq) {
    extern __shared__ u32 sm[];
    __shared__ u32 s_best;        // lowest start that has stopped so far
    u32 t0;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t0));
    const u32 N = 1u << n, stop = N, smask = (1u << (n - u)) - 1u;
    u32* table = sm;
    u32* dist = sm + N;
    const u32 tid = threadIdx.x;
    if (tid == 0) s_best = kNone;
    __syncthreads();
    u32 v[E];
#pragma unroll
    for (int k = 0; k < E; k++) {
        const u32 i = tid + k * kSmallThreads;
        v[k] = i < N ? src[i] : stop;
        if (i < N) {
            table[i] = v[k];
            if constexpr (STEPS) dist[i] = 1u;
            if ((v[k] & stop) && (i & smask) == 0u) atomicMin(&s_best, i);
        }
    }
    __syncthreads();
    u32 r = 1, best = kNone;
    for (;; r++) {
        u32 w[E];
#pragma unroll
        for (int k = 0; k < E; k++) w[k] = (v[k] & stop) ? v[k] : table[v[k]];
#pragma unroll
        for (int k = 0; k < E; k++) {
            if ((w[k] & ~v[k]) & stop) {             // stops in this round: once per entry
                const u32 i = tid + k * kSmallThreads;
                // dist[v] belongs to an entry that stopped before this round:
                // nobody writes it now
                if constexpr (STEPS) dist[i] = (1u << (r - 1)) + dist[v[k]];
                if ((i & smask) == 0u) atomicMin(&s_best, i);
            }
        }
        __syncthreads();
        best = s_best;
#pragma unroll
        for (int k = 0; k < E; k++) {
            if (!(v[k] & stop)) table[tid + k * kSmallThreads] = w[k];
            v[k] = w[k];
        }
        __syncthreads();
        if (r == n || (best != kNone && (mode == 0 || best == 0))) break;
    }
#pragma unroll
    for (int k = 0; k < E; k++) {
        const u32 i = tid + k * kSmallThreads;
        if (i >= N) continue;
        if constexpr (STEPS) {
            if (out64) out64[i] = (u64)v[k] | ((u64)((v[k] & stop) ? dist[i] : 1u << r) << 32);
        } else {
            out32[i] = v[k];
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();          // the host may go on when it sees the words
        u32 t1;
        asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t1));
        const u64 number = (u64)seq << 32;
        words[0] = number | r;
        words[1] = number | best;
        words[2] = number | (best != kNone ? table[best] : 0u);
        words[3] = number | (STEPS && best != kNone ? dist[best] : 0u);
        words[4] = number | (t1 - t0);
    }
}

typedef void (*SmallKernel)(const u32*, u32, u32, u32, u32*, u64*, volatile u64*, u32);
template <bool STEPS>
SmallKernel small_kernel(u32 n) {
    switch (n) {
    case 11: return small_solve<STEPS, 2>;
    case 12: return small_solve<STEPS, 4>;
    case 13: return small_solve<STEPS, 8>;
    case 14: return small_solve<STEPS, 16>;
    default: return small_solve<STEPS, 1>;     // up to 2^10 entries
    }
}

// All rounds of a table of 2^15 .. 2^20 entries in one cooperative launch of
// N / (1024 E) CTAs: a thread keeps its E entries in registers, a round
// gathers from one buffer, writes the other and ends in a grid barrier.  The
// buffers and distances change while the kernel runs, so they are read through
// the L2.  The barrier counts arrivals up; its spin is bounded, and a CTA that
// gives up lets the others go too.  keep receives the table as built, so that
// the rounds can start again from it then (a third buffer in place of a in the
// rounds took 8 us more than this copy at 2^20 entries).  The last CTA to end
// reports as small_solve does (rounds ~0: given up) and leaves the state as it
// was.
constexpr u32 kGridThreads = 1024;

template <bool STEPS, int E>
__global__ void __launch_bounds__(kGridThreads) grid_solve(u32* a, u32* b, u32* __restrict__ keep, u32* dist, u32 n,
                                                           u32 u, u32 mode, u64* __restrict__ out64,
                                                           NsatGridState* st, u32 spin_limit, volatile u64* words,
                                                           u32 seq) {
    __shared__ u32 s_best, s_round;      // lowest start in this CTA, lowest of all after the round
    __shared__ bool s_failed;
    const u32 tid = threadIdx.x, S = gridDim.x * kGridThreads, i0 = blockIdx.x * kGridThreads + tid;
    const u32 stop = 1u << n, smask = (1u << (n - u)) - 1u;
    if (tid == 0) {
        s_best = kNone;
        if (blockIdx.x == 0) asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(*(volatile u32*)&st->t0));
    }
    __syncthreads();
    u32 v[E], d[E];
#pragma unroll
    for (int k = 0; k < E; k++) {
        const u32 i = i0 + k * S;
        v[k] = __ldcg(a + i);
        __stcs(keep + i, v[k]);
        d[k] = 1u;
        if (STEPS && (v[k] & stop)) __stcg(dist + i, 1u);
    }
    u32 *src = a, *dst = b;
    u32 r = 1, best = kNone;
    bool failed = false;
    for (;; r++) {
        u32 w[E], low = kNone;
#pragma unroll
        for (int k = 0; k < E; k++) w[k] = (v[k] & stop) ? v[k] : __ldcg(src + v[k]);
#pragma unroll
        for (int k = 0; k < E; k++) {
            const u32 i = i0 + k * S;
            if constexpr (STEPS) {
                if ((w[k] & ~v[k]) & stop) {
                    // dist[v] belongs to an entry that stopped before this round
                    d[k] = (1u << (r - 1)) + (r == 1 ? 1u : __ldcg(dist + v[k]));
                    __stcg(dist + i, d[k]);
                }
            }
            __stcg(dst + i, w[k]);
            if ((w[k] & stop) && (i & smask) == 0u) low = min(low, i);
            v[k] = w[k];
        }
        low = __reduce_min_sync(0xffffffffu, low);
        if ((tid & 31u) == 0 && low != kNone) atomicMin(&s_best, low);
        __syncthreads();
        if (tid == 0) {
            if (s_best != kNone) atomicMin(&st->best[r], s_best);
            __threadfence();
            atomicAdd(&st->arrived, 1u);
            const u32 all = r * gridDim.x;
            u32 spins = 0;
            while (*(volatile u32*)&st->arrived < all && !*(volatile u32*)&st->failed)
                if (++spins == spin_limit) *(volatile u32*)&st->failed = 1u;
            __threadfence();
            s_failed = *(volatile u32*)&st->failed != 0u;
            s_round = *(volatile u32*)&st->best[r];
        }
        __syncthreads();
        best = s_round;
        failed = s_failed;
        if (failed || r == n || (best != kNone && (mode == 0 || best == 0))) break;
        u32* t = src;
        src = dst;
        dst = t;
    }
    if (STEPS && out64) {
#pragma unroll
        for (int k = 0; k < E; k++) out64[i0 + k * S] = (u64)v[k] | ((u64)((v[k] & stop) ? d[k] : 1u << r) << 32);
    }
    __syncthreads();
    if (tid != 0) return;
    __threadfence();
    if (atomicAdd(&st->ended, 1u) != gridDim.x - 1u) return;
    __threadfence();
    failed |= *(volatile u32*)&st->failed != 0u;
    u32 t1;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t1));
    const u32 t = t1 - *(volatile u32*)&st->t0;
    for (u32 k = 0; k < sizeof(st->best) / 4; k++) st->best[k] = kNone;
    st->arrived = 0u;
    st->ended = 0u;
    st->failed = 0u;
    const u64 number = (u64)seq << 32;
    words[0] = number | (failed ? ~0u : r);
    words[1] = number | best;
    words[2] = number | (best != kNone ? __ldcg(dst + best) : 0u);
    words[3] = number | (STEPS && best != kNone ? __ldcg(dist + best) : 0u);
    words[4] = number | t;
}

typedef void (*GridKernel)(u32*, u32*, u32*, u32*, u32, u32, u32, u64*, NsatGridState*, u32, volatile u64*, u32);
template <bool STEPS>
GridKernel grid_kernel(u32 per_thread) {
    switch (per_thread) {
    case 1: return grid_solve<STEPS, 1>;
    case 2: return grid_solve<STEPS, 2>;
    case 4: return grid_solve<STEPS, 4>;
    default: return grid_solve<STEPS, 8>;
    }
}

// The test before the atomic may read a stale word: bits only get set, so it
// can only cost an atomic that was not needed.
template <typename E>
__global__ void __launch_bounds__(256) mark(const E* __restrict__ entries, u64 items, u32 n, u32* bits, u32 r,
                                            u32 mode, const NsatStopState* __restrict__ st) {
    if (moot(st, r, mode)) return;
    const u32 stop = 1u << n;
    const u64 S = (u64)gridDim.x * blockDim.x;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += 4 * S) {
        u32 v[4], w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = i + (u64)k * S < items ? (u32)entries[i + (u64)k * S] : stop;
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = (v[k] & stop) ? ~0u : bits[v[k] >> 5];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const u32 m = 1u << (v[k] & 31u);
            if (!(v[k] & stop) && !(w[k] & m)) atomicOr(bits + (v[k] >> 5), m);
        }
    }
}

// A block ranks 1024 words (32768 positions), four consecutive ones a thread.
constexpr u32 kRankWords = 1024;

__device__ __forceinline__ u32 block_exclusive(u32 c, u32* total) {
    __shared__ u32 s_warp[32];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    u32 x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (u32)o) x += y;
    }
    if (lane == 31u) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        u32 y = lane < (blockDim.x >> 5) ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 z = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= (u32)o) y += z;
        }
        s_warp[lane] = y;
    }
    __syncthreads();
    const u32 before = warp ? s_warp[warp - 1] : 0u;
    *total = s_warp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before + x - c;
}

__global__ void __launch_bounds__(256) rank_sums(const u32* __restrict__ bits, u64 words, u32* __restrict__ sums) {
    const u64 w0 = (u64)blockIdx.x * kRankWords + 4u * threadIdx.x;
    u32 c = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (w0 + k < words) c += __popc(bits[w0 + k]);
    u32 total;
    block_exclusive(c, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) rank_scan(u32* __restrict__ sums, u32 nblk, NsatStopState* __restrict__ st) {
    u32 base = 0;
    for (u32 i0 = 0; i0 < nblk; i0 += 1024) {
        const u32 i = i0 + threadIdx.x;
        const u32 c = i < nblk ? sums[i] : 0u;
        u32 total;
        const u32 x = block_exclusive(c, &total);
        if (i < nblk) sums[i] = base + x;
        base += total;
    }
    if (threadIdx.x == 0) st->count = base;
}

// A warp walks its 128 words one after another, a lane per position, so both
// lists are written in runs of neighbouring words (a thread per word, each
// writing its own positions: 113 us at 2^24 positions, 1.5 ms at 2^28; this
// way 22 us and 0.3 ms).
__global__ void __launch_bounds__(256) rank_list(const u32* __restrict__ bits, u64 words,
                                                 const u32* __restrict__ sums, u32* __restrict__ states,
                                                 u32* __restrict__ ids) {
    const u64 w0 = (u64)blockIdx.x * kRankWords + 4u * threadIdx.x;
    const u32 lane = threadIdx.x & 31u;
    u32 b[4], c = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        b[k] = w0 + k < words ? bits[w0 + k] : 0u;
        c += __popc(b[k]);
    }
    u32 total;
    const u32 mine = sums[blockIdx.x] + block_exclusive(c, &total);
    const u32 pos0 = (u32)((w0 - 4u * lane) << 5);      // the warp's first position
    const u32 below = (1u << lane) - 1u;
    for (u32 t = 0; t < 32u; t++) {
        u32 id = __shfl_sync(0xffffffffu, mine, t);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const u32 m = __shfl_sync(0xffffffffu, b[k], t);
            if ((m >> lane) & 1u) {
                const u32 s = pos0 + ((t * 4u + k) << 5) + lane, x = id + __popc(m & below);
                states[x] = s;
                ids[s] = x;
            }
            id += __popc(m);
        }
    }
}

__device__ __forceinline__ u64 entry64(u32 val, u32 dist) { return (u64)val | ((u64)dist << 32); }

__global__ void __launch_bounds__(256) contract32(const u32* __restrict__ table, const u32* __restrict__ dist,
                                                  const u32* __restrict__ states, const u32* __restrict__ ids,
                                                  u32 count, u32 n, u32 r, u64* __restrict__ P, u64* __restrict__ Q,
                                                  u32* __restrict__ start) {
    const u32 stop = 1u << n;
    for (u32 id = blockIdx.x * blockDim.x + threadIdx.x; id < count; id += gridDim.x * blockDim.x) {
        const u32 s = states[id];
        const u32 t = table[s];
        P[id] = (t & stop) ? entry64(t, dist ? dist[s] : 0u) : entry64(ids[t], 1u << r);
        Q[id] = entry64(id, 0u);
        start[id] = kNone;
    }
}

__global__ void __launch_bounds__(256) starts32(const u32* __restrict__ table, const u32* __restrict__ ids, u32 n,
                                                u32 u, u32* __restrict__ start) {
    const u32 stop = 1u << n;
    const u64 S = (u64)gridDim.x * blockDim.x;
    for (u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x; k < (1ull << u); k += S) {
        const u32 s = (u32)(k << (n - u));
        const u32 t = table[s];
        if (!(t & stop)) {
            const u32 id = ids[t];
            if (*(volatile u32*)&start[id] > s) atomicMin(&start[id], s);
        }
    }
}

__global__ void __launch_bounds__(256) contract64(const u64* __restrict__ upP, const u32* __restrict__ states,
                                                  const u32* __restrict__ ids, u32 count, u32 n, u64* __restrict__ P,
                                                  u64* __restrict__ Q, u32* __restrict__ start) {
    const u32 stop = 1u << n;
    for (u32 id = blockIdx.x * blockDim.x + threadIdx.x; id < count; id += gridDim.x * blockDim.x) {
        const u64 t = upP[states[id]];
        P[id] = ((u32)t & stop) ? t : entry64(ids[(u32)t], (u32)(t >> 32));
        Q[id] = entry64(id, 0u);
        start[id] = kNone;
    }
}

__global__ void __launch_bounds__(256) starts64(const u64* __restrict__ upQ, const u32* __restrict__ up_start,
                                                u32 up_count, const u32* __restrict__ ids, u32 n,
                                                u32* __restrict__ start) {
    const u32 stop = 1u << n;
    for (u32 x = blockIdx.x * blockDim.x + threadIdx.x; x < up_count; x += gridDim.x * blockDim.x) {
        const u32 q = (u32)upQ[x], s = up_start[x];
        if (s != kNone && !(q & stop)) {
            const u32 id = ids[q];
            if (*(volatile u32*)&start[id] > s) atomicMin(&start[id], s);
        }
    }
}

__global__ void __launch_bounds__(256) join_pq(const u64* P, const u64* Q, u64* P2, u64* Q2, const u32* start,
                                               u32 count, u32 n, u32 r, u32 mode, NsatStopState* __restrict__ st) {
    pdl_wait();
    if (answered(st, r, mode)) return;
    const u32 stop = 1u << n;
    u32 best = kNone;
    const u32 S = gridDim.x * blockDim.x;
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += 2 * S) {
        u64 p[2], q[2], pw[2], qw[2];
        bool ok[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            ok[k] = (u64)i + (u64)k * S < count;
            p[k] = ok[k] ? P[i + k * S] : (u64)stop;
            q[k] = ok[k] ? Q[i + k * S] : (u64)stop;
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            pw[k] = ((u32)p[k] & stop) ? 0ull : P[(u32)p[k]];
            qw[k] = ((u32)q[k] & stop) ? 0ull : P[(u32)q[k]];
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (!ok[k]) continue;
            const u32 x = i + k * S;
            P2[x] = ((u32)p[k] & stop) ? p[k] : entry64((u32)pw[k], (u32)(p[k] >> 32) + (u32)(pw[k] >> 32));
            const u64 o = ((u32)q[k] & stop) ? q[k] : entry64((u32)qw[k], (u32)(q[k] >> 32) + (u32)(qw[k] >> 32));
            Q2[x] = o;
            if ((u32)o & stop) best = min(best, start[x]);
        }
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if ((threadIdx.x & 31) == 0) {
        // a start resolved in an earlier round stays resolved
        if (blockIdx.x == 0 && threadIdx.x == 0) best = min(best, *(volatile u32*)&st->best[r - 1]);
        if (best != kNone) atomicMin(&st->best[r], best);
    }
}

__global__ void __launch_bounds__(256) expand64(u64* __restrict__ upQ, u32 up_count, const u64* __restrict__ Q,
                                                const u32* __restrict__ states, const u32* __restrict__ ids, u32 n) {
    const u32 stop = 1u << n;
    for (u32 x = blockIdx.x * blockDim.x + threadIdx.x; x < up_count; x += gridDim.x * blockDim.x) {
        const u64 q = upQ[x];
        if ((u32)q & stop) continue;
        const u64 e = Q[ids[(u32)q]];
        const u32 v = ((u32)e & stop) ? (u32)e : states[(u32)e];
        upQ[x] = entry64(v, (u32)(q >> 32) + (u32)(e >> 32));
    }
}

__global__ void __launch_bounds__(256) scatter(const u64* __restrict__ Q, const u32* __restrict__ states, u32 count,
                                               u32 n, u32* __restrict__ at, u32* __restrict__ at_dist) {
    const u32 stop = 1u << n;
    for (u32 id = blockIdx.x * blockDim.x + threadIdx.x; id < count; id += gridDim.x * blockDim.x) {
        const u64 e = Q[id];
        const u32 s = states[id];
        at[s] = ((u32)e & stop) ? (u32)e : states[(u32)e];
        if (at_dist) at_dist[s] = (u32)(e >> 32);
    }
}

__global__ void __launch_bounds__(256) finish(u32* __restrict__ table, u32* __restrict__ dist,
                                              const u32* __restrict__ at, const u32* __restrict__ at_dist, u64 items,
                                              u32 n, u32 r) {
    const u32 stop = 1u << n, all = 1u << r;
    const u64 S = (u64)gridDim.x * blockDim.x;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += 4 * S) {
        u32 v[4], w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = i + (u64)k * S < items ? table[i + (u64)k * S] : stop;
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = (v[k] & stop) ? v[k] : at[v[k]];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (v[k] & stop) continue;
            const u64 j = i + (u64)k * S;
            table[j] = w[k];
            if (dist && (w[k] & stop)) dist[j] = all + at_dist[v[k]];
        }
    }
}

__global__ void __launch_bounds__(256) widen(const u32* __restrict__ table, const u32* __restrict__ dist, u64 items,
                                             u32 n, u32 r, u64* __restrict__ out) {
    const u32 stop = 1u << n, all = 1u << r;
    const u64 S = (u64)gridDim.x * blockDim.x;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < items; i += S) {
        const u32 v = table[i];
        out[i] = entry64(v, dist && (v & stop) ? dist[i] : all);
    }
}

// Eight CTAs of 256 threads fill an SM; `per` items are in flight per thread.
unsigned blocks_for(u64 items, int sms, u32 per) {
    const u64 want = (items + 256ull * per - 1) / (256ull * per), cap = (u64)sms * 8ull;
    return (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
}

int ok() { return cudaGetLastError() == cudaSuccess ? 0 : -4; }

}  // namespace

extern "C" int nsat_stop_join(const uint32_t* src, uint32_t* dst, uint32_t* dist, uint32_t n, uint32_t u, uint32_t r,
                              uint32_t mode, NsatStopState* st, uint32_t* sample, int sms, cudaStream_t s) {
    const u64 N = 1ull << n;
    const unsigned g = blocks_for(N, sms, 4);
    const auto fn = dist ? (sample ? join32<true, true> : join32<true, false>)
                         : (sample ? join32<false, true> : join32<false, false>);
    return launch_pdl(fn, g, 256, s, src, dst, dist, N, n, u, r, mode, st, sample) == cudaSuccess ? 0 : -4;
}

extern "C" int nsat_stop_small(const uint32_t* src, uint32_t n, uint32_t u, uint32_t mode, int steps,
                               uint32_t* out32, uint64_t* out64, uint64_t* words, uint32_t seq, cudaStream_t s) {
    if (n > NSAT_STOP_SMALL_BITS) return -1;
    const size_t smem = ((size_t)(steps ? 8 : 4)) << n;
    const SmallKernel fn = steps ? small_kernel<true>(n) : small_kernel<false>(n);
    // per call: the attribute belongs to the current device (48 KB in all,
    // static words included, need none)
    if (smem >= 48 * 1024 && cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 8 << NSAT_STOP_SMALL_BITS) != cudaSuccess)
        return -4;
    fn<<<1, kSmallThreads, smem, s>>>(src, n, u, mode, out32, (u64*)out64, (volatile u64*)words, seq);
    return ok();
}

extern "C" int nsat_stop_grid(uint32_t* a, uint32_t* b, uint32_t* keep, uint32_t* dist, uint32_t n, uint32_t u,
                              uint32_t mode, int steps, uint64_t* out64, NsatGridState* st, uint32_t spin_limit,
                              uint64_t* words, uint32_t seq, cudaStream_t s) {
    if (n <= NSAT_STOP_SMALL_BITS || n > NSAT_STOP_GRID_BITS) return -1;
    // 128 CTAs from 2^17 entries on
    const u32 e = n <= 17 ? 1u : 1u << (n - 17);
    const GridKernel fn = steps ? grid_kernel<true>(e) : grid_kernel<false>(e);
    volatile u64* w = (volatile u64*)words;
    u64* o = (u64*)out64;
    void* args[] = {&a, &b, &keep, &dist, &n, &u, &mode, &o, &st, &spin_limit, &w, &seq};
    if (cudaLaunchCooperativeKernel((const void*)fn, dim3((1u << n) / (kGridThreads * e)), dim3(kGridThreads), args, 0, s) == cudaSuccess)
        return 0;
    cudaGetLastError();
    return 1;        // more CTAs than the device holds at once
}

extern "C" int nsat_stop_mark32(const uint32_t* entries, uint64_t items, uint32_t n, uint32_t* bits, uint32_t r,
                                uint32_t mode, const NsatStopState* st, int sms, cudaStream_t s) {
    mark<u32><<<blocks_for(items, sms, 4), 256, 0, s>>>(entries, items, n, bits, r, mode, st);
    return ok();
}

extern "C" int nsat_stop_mark64(const uint64_t* entries, uint64_t items, uint32_t n, uint32_t* bits, uint32_t r,
                                uint32_t mode, const NsatStopState* st, int sms, cudaStream_t s) {
    mark<u64><<<blocks_for(items, sms, 4), 256, 0, s>>>((const u64*)entries, items, n, bits, r, mode, st);
    return ok();
}

extern "C" int nsat_stop_rank(const uint32_t* bits, uint64_t items, uint32_t* block_sums, NsatStopState* st,
                              cudaStream_t s) {
    const u64 words = (items + 31) / 32;
    const u32 nblk = (u32)((words + kRankWords - 1) / kRankWords);
    rank_sums<<<nblk, 256, 0, s>>>(bits, words, block_sums);
    rank_scan<<<1, 1024, 0, s>>>(block_sums, nblk, st);
    return ok();
}

extern "C" int nsat_stop_list(const uint32_t* bits, uint64_t items, const uint32_t* block_sums, uint32_t* states,
                              uint32_t* ids, cudaStream_t s) {
    const u64 words = (items + 31) / 32;
    const u32 nblk = (u32)((words + kRankWords - 1) / kRankWords);
    rank_list<<<nblk, 256, 0, s>>>(bits, words, block_sums, states, ids);
    return ok();
}

extern "C" int nsat_stop_contract32(const uint32_t* table, const uint32_t* dist, const uint32_t* states,
                                    const uint32_t* ids, uint32_t count, uint32_t n, uint32_t u, uint32_t r,
                                    uint64_t* P, uint64_t* Q, uint32_t* start, int sms, cudaStream_t s) {
    contract32<<<blocks_for(count, sms, 1), 256, 0, s>>>(table, dist, states, ids, count, n, r, (u64*)P, (u64*)Q,
                                                         start);
    starts32<<<blocks_for(1ull << u, sms, 1), 256, 0, s>>>(table, ids, n, u, start);
    return ok();
}

extern "C" int nsat_stop_contract64(const uint64_t* upP, const uint64_t* upQ, const uint32_t* up_start,
                                    uint32_t up_count, const uint32_t* states, const uint32_t* ids, uint32_t count,
                                    uint32_t n, uint64_t* P, uint64_t* Q, uint32_t* start, int sms, cudaStream_t s) {
    contract64<<<blocks_for(count, sms, 1), 256, 0, s>>>((const u64*)upP, states, ids, count, n, (u64*)P, (u64*)Q,
                                                         start);
    starts64<<<blocks_for(up_count, sms, 1), 256, 0, s>>>((const u64*)upQ, up_start, up_count, ids, n, start);
    return ok();
}

extern "C" int nsat_stop_join_pq(const uint64_t* P, const uint64_t* Q, uint64_t* P2, uint64_t* Q2,
                                 const uint32_t* start, uint32_t count, uint32_t n, uint32_t r, uint32_t mode,
                                 NsatStopState* st, int sms, cudaStream_t s) {
    const unsigned g = blocks_for(count, sms, 2);
    return launch_pdl(join_pq, g, 256, s, (const u64*)P, (const u64*)Q, (u64*)P2, (u64*)Q2, start, count, n, r, mode,
                      st) == cudaSuccess ? 0 : -4;
}

extern "C" int nsat_stop_expand64(uint64_t* upQ, uint32_t up_count, const uint64_t* Q, const uint32_t* states,
                                  const uint32_t* ids, uint32_t n, int sms, cudaStream_t s) {
    expand64<<<blocks_for(up_count, sms, 1), 256, 0, s>>>((u64*)upQ, up_count, (const u64*)Q, states, ids, n);
    return ok();
}

extern "C" int nsat_stop_scatter(const uint64_t* Q, const uint32_t* states, uint32_t count, uint32_t n, uint32_t* at,
                                 uint32_t* at_dist, int sms, cudaStream_t s) {
    scatter<<<blocks_for(count, sms, 1), 256, 0, s>>>((const u64*)Q, states, count, n, at, at_dist);
    return ok();
}

extern "C" int nsat_stop_finish(uint32_t* table, uint32_t* dist, const uint32_t* at, const uint32_t* at_dist,
                                uint64_t items, uint32_t n, uint32_t r, int sms, cudaStream_t s) {
    finish<<<blocks_for(items, sms, 4), 256, 0, s>>>(table, dist, at, at_dist, items, n, r);
    return ok();
}

extern "C" int nsat_stop_widen(const uint32_t* table, const uint32_t* dist, uint64_t items, uint32_t n, uint32_t r,
                               uint64_t* out, int sms, cudaStream_t s) {
    widen<<<blocks_for(items, sms, 1), 256, 0, s>>>(table, dist, items, n, r, (u64*)out);
    return ok();
}
