// stop_kernels.h -- launchers of the SATOSTOP doubling over 32-bit entries
// (stop_kernels.cu); stop_join.cpp drives them.  All take a stream and return
// 0 or -4 (launch error).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define NSAT_STOP_SMALL_BITS 14     // tables of up to 2^14 entries are solved in one CTA

#define NSAT_STOP_GRID_BITS 20      // up to 2^20 in one cooperative launch

// Device state of nsat_stop_grid: best all ~0, the rest 0 before and after.
typedef struct {
    uint32_t best[28];
    uint32_t arrived, ended, failed, t0;
} NsatGridState;

// Device state of one solve.
typedef struct {
    uint32_t best[40];        // best[r]: lowest resolved start after round r (~0 = none)
    uint32_t final_round;     // round whose answer ended the loop early (0 = none)
    uint32_t distinct;        // sampled distinct successors (see the sample of nsat_stop_join)
    uint32_t count;           // distinct successors (nsat_stop_rank)
    uint32_t entry, dist;     // the answer's entry and distance
    uint32_t pad[3];
} NsatStopState;

#ifdef __cplusplus
extern "C" {
#endif

// Round r of synchronous doubling, dst = src o src.  dist (or null): distance
// of the entries that have stopped.  sample (or null): bitmap of 2^(n-8) bits,
// cleared, in which a 256th of the successors is marked; st->distinct counts
// the bits set.
int nsat_stop_join(const uint32_t* src, uint32_t* dst, uint32_t* dist, uint32_t n, uint32_t u, uint32_t r,
                   uint32_t mode, NsatStopState* st, uint32_t* sample, int sms, cudaStream_t s);
// Every round of a table of n <= NSAT_STOP_SMALL_BITS bits, with distances
// when steps is set; out32 or (with steps) out64, where not null, receive the
// table after the last one.  words (pinned host memory, 5) receive the
// rounds run, the lowest start (~0: none), its entry, its distance and the
// kernel's time in ns, each under seq << 32.
int nsat_stop_small(const uint32_t* src, uint32_t n, uint32_t u, uint32_t mode, int steps, uint32_t* out32,
                    uint64_t* out64, uint64_t* words, uint32_t seq, cudaStream_t s);

// The same for NSAT_STOP_SMALL_BITS < n <= NSAT_STOP_GRID_BITS in one cooperative
// launch between a (the table, also after an even number of rounds) and b.
// dist: 2^n words, with steps.  1: the device does not hold the grid.  A CTA
// that has polled the barrier spin_limit times in vain ends the launch: rounds
// ~0, and of the buffers only keep (2^n words), a copy of a, is of use.
#define NSAT_STOP_SPINS (1u << 22)
int nsat_stop_grid(uint32_t* a, uint32_t* b, uint32_t* keep, uint32_t* dist, uint32_t n, uint32_t u, uint32_t mode,
                   int steps, uint64_t* out64, NsatGridState* st, uint32_t spin_limit, uint64_t* words, uint32_t seq,
                   cudaStream_t s);

// Contraction to the states that a later round can still look up.
// marks in bits (cleared, items bits) the successors of items entries, unless
// the rounds up to r hold the answer
int nsat_stop_mark32(const uint32_t* entries, uint64_t items, uint32_t n, uint32_t* bits, uint32_t r, uint32_t mode,
                     const NsatStopState* st, int sms, cudaStream_t s);
int nsat_stop_mark64(const uint64_t* entries, uint64_t items, uint32_t n, uint32_t* bits, uint32_t r, uint32_t mode,
                     const NsatStopState* st, int sms, cudaStream_t s);
// block_sums: one u32 per 32768 bits; st->count = all set bits
int nsat_stop_rank(const uint32_t* bits, uint64_t items, uint32_t* block_sums, NsatStopState* st, cudaStream_t s);
// states[id] = the id-th marked position, ids[position] = id
int nsat_stop_list(const uint32_t* bits, uint64_t items, const uint32_t* block_sums, uint32_t* states, uint32_t* ids,
                   cudaStream_t s);
// P[id], Q[id] and start[id] of the marked states (see stop_kernels.cu)
int nsat_stop_contract32(const uint32_t* table, const uint32_t* dist, const uint32_t* states, const uint32_t* ids,
                         uint32_t count, uint32_t n, uint32_t u, uint32_t r, uint64_t* P, uint64_t* Q, uint32_t* start,
                         int sms, cudaStream_t s);
int nsat_stop_contract64(const uint64_t* upP, const uint64_t* upQ, const uint32_t* up_start, uint32_t up_count,
                         const uint32_t* states, const uint32_t* ids, uint32_t count, uint32_t n, uint64_t* P,
                         uint64_t* Q, uint32_t* start, int sms, cudaStream_t s);
// one round on a contracted domain
int nsat_stop_join_pq(const uint64_t* P, const uint64_t* Q, uint64_t* P2, uint64_t* Q2, const uint32_t* start,
                      uint32_t count, uint32_t n, uint32_t r, uint32_t mode, NsatStopState* st, int sms,
                      cudaStream_t s);
// back to the domain above
int nsat_stop_expand64(uint64_t* upQ, uint32_t up_count, const uint64_t* Q, const uint32_t* states,
                       const uint32_t* ids, uint32_t n, int sms, cudaStream_t s);
int nsat_stop_scatter(const uint64_t* Q, const uint32_t* states, uint32_t count, uint32_t n, uint32_t* at,
                      uint32_t* at_dist, int sms, cudaStream_t s);
// table[s] = at[table[s]] for entries that have not stopped, in place; with
// dist/at_dist the distances follow (an entry stands for 2^r evaluations)
int nsat_stop_finish(uint32_t* table, uint32_t* dist, const uint32_t* at, const uint32_t* at_dist, uint64_t items,
                     uint32_t n, uint32_t r, int sms, cudaStream_t s);
// 64-bit entries: out = entry | distance << 32, the distance of an entry that
// has not stopped being 2^r; dist null: every distance is 2^r
int nsat_stop_widen(const uint32_t* table, const uint32_t* dist, uint64_t items, uint32_t n, uint32_t r,
                    uint64_t* out, int sms, cudaStream_t s);

#ifdef __cplusplus
}
#endif
