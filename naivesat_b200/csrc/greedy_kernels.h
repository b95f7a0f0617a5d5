// greedy_kernels.h -- launchers of the partitioned greedysatostop kernels
// (greedy_kernels.cu).  All take a stream and return 0 or -4 (launch error).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// Device state of a solve over a device table (nsat_greedy_step).
typedef struct {
    unsigned long long key;    // start << 32 | entry of the lowest start found (~0 = none)
    uint32_t step;             // the step that found it
    uint32_t done;             // an earlier step has the answer
} NsatGreedyState;

extern "C" {
// Step `step`: partition i (2^lp entries, lp >= 6) of the table of 32-bit
// entries (n <= 31) joined with every partition in order and searched; does
// nothing once an earlier step has an answer.  snap: 2^lp words.
int nsat_greedy_step(uint32_t* table, uint32_t* snap, uint32_t i, uint32_t lp, uint32_t n, uint32_t unknowns,
                     uint32_t step, NsatGreedyState* state, int sms, cudaStream_t st);
// packed (bits-wide) entries -> u64 entries; count entries
int nsat_greedy_unpack(const uint64_t* packed, uint64_t count, uint32_t bits, uint64_t* out, int sms,
                       cudaStream_t st);
// u64 entries -> packed entries; count a multiple of 64
int nsat_greedy_pack(const uint64_t* in, uint64_t count, uint32_t bits, uint64_t* packed, int sms, cudaStream_t st);
// dest[i] = second[next - start2] where dest[i] has no STOP and its next lies in [start2, start2+count2)
int nsat_greedy_join(uint64_t* dest, uint64_t count, const uint64_t* second, uint64_t start2, uint64_t count2,
                     uint32_t n, int sms, cudaStream_t st);
// the same join reading `second` as packed (n+1)-bit entries
int nsat_greedy_join_packed(uint64_t* dest, uint64_t count, const uint64_t* second_packed, uint64_t start2,
                            uint64_t count2, uint32_t n, int sms, cudaStream_t st);
// atomicMin into *best of the unknown starts of [start, start+count) with STOP
int nsat_greedy_find(const uint64_t* dest, uint64_t start, uint64_t count, uint32_t n, uint32_t unknowns,
                     uint64_t* best, int sms, cudaStream_t st);
}
