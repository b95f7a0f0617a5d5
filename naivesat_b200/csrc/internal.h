// internal.h -- library-internal entry points shared between translation units.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <functional>
#include <string>

#include "nsat.h"

#include <cuda_runtime.h>

#include "circuit.h"
#include "stop_kernels.h"

namespace nsat {

// Device ordinal a context is bound to, its stream and SM count.
int ctx_device(const nsat_ctx* ctx);
cudaStream_t ctx_stream(const nsat_ctx* ctx);
int ctx_sm_count(const nsat_ctx* ctx);
bool ctx_no_optimize(const nsat_ctx* ctx);
// The options a context was created with.
nsat_opts ctx_opts(const nsat_ctx* ctx);
// Records a failure on the context (nsat_last_error) and returns `code`.
int ctx_fail(nsat_ctx* ctx, int code, const std::string& msg);
// Per-call device buffers (tables, partition images, work areas) from the
// context's stream-ordered pool: allocated and freed in order on the
// context's stream, and kept for reuse by the next call (up to a release
// threshold), so a repeated solve pays no cudaMalloc/cudaFree.  A buffer
// used on another stream needs the context's stream synchronised after the
// allocation.
cudaError_t ctx_alloc(nsat_ctx* ctx, void** p, size_t bytes);
void ctx_free(nsat_ctx* ctx, void* p);
// The context's device state of a SATOSTOP solve and its pinned host copy.
void ctx_stop_state(nsat_ctx* ctx, NsatStopState** dev, NsatStopState** host);
cudaEvent_t ctx_stop_event(nsat_ctx* ctx);
NsatGridState* ctx_grid_state(nsat_ctx* ctx);
uint32_t ctx_grid_spins(nsat_ctx* ctx);
void ctx_grid_gave_up(nsat_ctx* ctx);
// A short kernel that reports in up to 5 words of pinned memory, each with the
// launch's number (ctx_next_seq) in its upper half; ctx_poll_words waits for
// the first `words`.
uint32_t ctx_next_seq(nsat_ctx* ctx);
volatile uint64_t* ctx_words(nsat_ctx* ctx);
int ctx_poll_words(nsat_ctx* ctx, int words);
// A pair of timing events of the context, for one interval at a time.
void ctx_timing_events(nsat_ctx* ctx, cudaEvent_t* begin, cudaEvent_t* end);
// Bytes that the pool holds and no buffer uses.
uint64_t ctx_pool_unused(nsat_ctx* ctx);
// Returns the pool's unused memory to the device (after the context's
// stream finishes), for a caller about to size a buffer by free memory.
void ctx_trim(nsat_ctx* ctx);

// Circuit from the C ABI's flat description (not validated).
Circuit circuit_from_desc(const nsat_circuit_desc* d);

// nsat_qsat_solve with the scratch area (the chunk tree's nodes, cleared before
// the first launch) supplied by the caller
// instead of the context's cudaMalloc'd buffer; fails with NSAT_EUNSUPPORTED
// when a launch would need more than scratch_bytes.
int qsat_solve_with_scratch(nsat_ctx* ctx, nsat_circuit* c, const uint8_t* quants,
                            const nsat_qsat_opts* opts, nsat_qsat_result* res,
                            unsigned char* scratch, size_t scratch_bytes);

// The QSAT sub-problems under prefixes first .. first + count - 1 of
// prefix_bits fixed inputs, solved back to back through the launch ring when
// each is one launch (otherwise only count == 1 is accepted); on_block sees
// each result in prefix order and returns false to stop.
int qsat_solve_blocks(nsat_ctx* ctx, nsat_circuit* c, const uint8_t* quants, uint32_t prefix_bits,
                      uint64_t first, uint64_t count,
                      const std::function<bool(uint64_t, const nsat_qsat_result&)>& on_block);

// Next-state entries (next | STOP << n) of states first_state ..
// first_state+count-1 (both multiples of 1024, n >= 10) into device memory
// dev_out, as u64 (wide) or, for n <= 31, u32, on the context's stream
// (synchronous); any_stop reports a STOP among them.
int table_chunk(nsat_ctx* ctx, nsat_circuit* c, uint64_t first_state, uint64_t count, bool wide, void* dev_out,
                uint32_t* any_stop, float* ms);

const Circuit& circuit_of(const nsat_circuit* c);

}  // namespace nsat

// For the tests only: leaves the static area of nsat_qsat_solve_noalloc as a
// launch that was cut short might.
extern "C" int nsat_test_fill_noalloc(nsat_ctx* ctx, int byte);
// For the tests only: the number of the context's next launch.
extern "C" int nsat_test_launch_number(nsat_ctx* ctx, uint32_t next);
// For the tests only: the k-th buffer taken from the pool from now on is
// refused (0: none); returns what was left of an earlier call's k.
extern "C" int nsat_test_fail_alloc(nsat_ctx* ctx, uint32_t k);
// For the tests only: sets the polls after which grid_solve's barrier gives up;
// returns how many times it has since the last call.
extern "C" int nsat_test_grid_spins(nsat_ctx* ctx, uint32_t spins);
