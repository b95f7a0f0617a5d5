// device_template.cuh -- sm_100a kernels specialised per circuit by NVRTC.
//
// The host generator (codegen.cpp) prepends a prelude that defines:
//   constexpr ints NSAT_NIN, NSAT_NOUT, NSAT_NB (enumeration bits), NSAT_NT
//   (threads per CTA), NSAT_IT / NSAT_WB / NSAT_CB (log2 of iterations per
//   warp, warps per CTA and CTAs per launch; QSAT: chunks per launch),
//   NSAT_ONE (QSAT: a CTA per chunk), NSAT_INNER (log2 of iterations
//   evaluated together, at most IT), NSAT_BOUNDS (the kernels'
//   __launch_bounds__), NSAT_C (= 10+IT+WB+CB, log2 of
//   assignments per launch), NSAT_M (QSAT unit level), NSAT_Q0ALL,
//   NSAT_ALLBITS (bit j = quantifier of enumeration bit j is All),
//   NSAT_DATA (1 = items come from a buffer instead of the circuit),
//   NSAT_FMT (table entry format);
// and the generated device functions
//   nsat_inputs_fixed(x, lane, warp, cta, launch)  -- inputs that stay fixed
//   nsat_inputs_iter(x, it)                        -- inputs that follow `it`
//   nsat_eval(x, y)               output 0 of 2^NSAT_INNER iterations, a
//                                 32-lane word each
//   nsat_eval_all(x, o)           all outputs (table mode)
//   nsat_inputs_word(x, w)        inputs of word index w (table mode)
//   nsat_nodes_resolve(c, v, nodes), nsat_claim(...), NSAT_NODES
//                                 the tree above the chunks (QSAT, below)
//
// Assignment enumeration inside one launch (bit p of the launch-relative
// index selects circuit input IN_OF_BIT[p], baked into the functions above):
//   p 0..4   lane of the 32-bit word (constants 0xAAAAAAAA ... 0xFFFF0000)
//   p 5..9   lane of the warp
//   p 10..   iteration of the warp's loop (IT bits), warp in CTA (WB bits),
//            CTA in grid (CB bits); bits >= C come from the launch index.
// No input is ever read from memory: the kernels are pure ALU work plus a
// few bytes of results.

typedef unsigned int u32;
typedef unsigned long long u64;

struct LaunchOut {
    u64 min_idx;   // SAT: lowest satisfying launch-relative index; QSAT: lowest decisive unit
    u64 count;     // SAT: solutions in this launch
    u32 tree;      // QSAT: tree value of the launch when no unit boundary is inside it
    u32 ticket;    // CTAs finished
    u32 any;       // table build: some STOP output seen
    u32 values;    // QSAT: chunks claimed beyond the first of each CTA
    u32 t0;        // global timer at the first CTA's start (ns)
    u32 pad;
};

__device__ __forceinline__ u32 nsat_now() {
    u32 t;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    return t;
}

// First statement of a kernel.
__device__ __forceinline__ void nsat_begin(LaunchOut* out) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *(volatile u32*)&out->t0 = nsat_now();
}

// The last CTA of a launch: puts the slot back as the next launch expects it
// and writes the result to pinned host memory: min_idx, the kind's value and
// the kernel's time.  The host waits for the stream or, after one short
// launch, polls; so each 32-bit half goes in a 64-bit word with the launch's
// number, which vouches for it, and no fence orders the words.  A pair of
// timing events around a kernel and the wait for the second take 11 us of a
// small solve; a copy that set the slot and one that read it back took 6 us.
// One asm block: as statements the compiler took 6 ms for it, a tenth of a
// small circuit's compile.
#if NSAT_MODE_SAT
#define NSAT_VALUE "ld.volatile.global.u64 v, [%0+8];"       // count
#elif NSAT_MODE_QSAT
#define NSAT_VALUE "ld.volatile.global.u32 a, [%0+16];\n\tmov.b64 v, {a, 0};"      // tree
#else
#define NSAT_VALUE "ld.volatile.global.u32 a, [%0+24];\n\tmov.b64 v, {a, 0};"      // any
#endif
__device__ __forceinline__ void nsat_publish(LaunchOut* out, u64* host, u32 seq) {
    asm volatile(
        "{\n\t"
        ".reg .b64 m, v;\n\t"
        ".reg .b32 a, b, t, t0;\n\t"
        "ld.volatile.global.u64 m, [%0];\n\t"
        NSAT_VALUE "\n\t"
        "ld.volatile.global.u32 t0, [%0+32];\n\t"
        "mov.u32 t, %%globaltimer_lo;\n\t"
        "sub.u32 t, t, t0;\n\t"
        "st.volatile.global.u64 [%0], -1;\n\t"        // min_idx
        "st.volatile.global.u64 [%0+8], 0;\n\t"       // count
        "st.volatile.global.u64 [%0+16], 0;\n\t"      // tree, ticket
        "st.volatile.global.u32 [%0+24], 0;\n\t"      // any
        "mov.b64 {a, b}, m;\n\t"
        "mov.b64 m, {a, %2};\n\t"
        "st.volatile.global.u64 [%1], m;\n\t"
        "mov.b64 m, {b, %2};\n\t"
        "st.volatile.global.u64 [%1+8], m;\n\t"
        "mov.b64 {a, b}, v;\n\t"
        "mov.b64 m, {a, %2};\n\t"
        "st.volatile.global.u64 [%1+16], m;\n\t"
        "mov.b64 m, {b, %2};\n\t"
        "st.volatile.global.u64 [%1+24], m;\n\t"
        "mov.b64 m, {t, %2};\n\t"
        "st.volatile.global.u64 [%1+32], m;\n\t"
        "}" ::"l"(out), "l"(host), "r"(seq) : "memory");
}

// Ends a CTA, all threads together, after its last update of *out.
__device__ __forceinline__ void nsat_finish(LaunchOut* out, u64* host, u32 seq) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&out->ticket, 1u) == gridDim.x - 1u) {
            __threadfence();
            nsat_publish(out, host, seq);
        }
    }
}

#if NSAT_MODE_SAT
// --------------------------------------------------------------------------
// SAT: count every satisfying assignment and find the lowest one.
extern "C" __global__ void NSAT_BOUNDS
nsat_sat(u64 launch, LaunchOut* out, u64* host, u32 seq) {
    nsat_begin(out);
    const u32 lane = threadIdx.x & 31u;
    const u32 warp = threadIdx.x >> 5;
    const u32 cta = blockIdx.x;
    __shared__ u32 s_idx, s_cnt;
    if (threadIdx.x == 0) { s_idx = ~0u; s_cnt = 0u; }
    __syncthreads();
    u32 x[NSAT_NIN];
    nsat_inputs_fixed(x, lane, warp, cta, launch);
    u32 cnt = 0;
    u32 first_it = 0xffffffffu, first_bit = 0;
#pragma unroll 1
    for (u32 outer = 0; outer < (1u << NSAT_IT); outer += 1u << NSAT_INNER) {
        u32 ys[1 << NSAT_INNER];
        nsat_inputs_iter(x, outer);
        nsat_eval(x, ys);
#pragma unroll
        for (u32 inner = 0; inner < (1u << NSAT_INNER); inner++) {
            const u32 it = outer | inner;
            const u32 y = ys[inner];
            cnt += __popc(y);
            if (y != 0u && first_it == 0xffffffffu) { first_it = it; first_bit = __ffs(y) - 1; }
        }
    }
    // index within the CTA: 10 + IT + WB <= 25 bits, and at most 2^25 solutions
    // to count.  One pair of atomics per CTA: launches with few iterations per
    // warp would otherwise queue every warp on the same two addresses.
    u32 idx = ~0u;
    if (first_it != ~0u) idx = (((((warp << NSAT_IT) | first_it) << 5) | lane) << 5) | first_bit;
    idx = __reduce_min_sync(~0u, idx);
    cnt = __reduce_add_sync(~0u, cnt);
    if (lane == 0 && cnt != 0u) {
        atomicMin(&s_idx, idx);
        atomicAdd(&s_cnt, cnt);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_cnt != 0u) {
        atomicAdd(&out->count, (u64)s_cnt);
        atomicMin(&out->min_idx, ((u64)cta << (10 + NSAT_IT + NSAT_WB)) | s_idx);
    }
    nsat_finish(out, host, seq);
}
#endif

#if NSAT_MODE_QSAT
// --------------------------------------------------------------------------
// QSAT: AND/OR tree over the enumeration bits, innermost quantifier first.
// Nodes at level L cover 2^L consecutive items.  Units are the nodes at
// level M (one value of the first quantifier block each); a unit is
// decisive when its value differs from the first quantifier's identity
// (1 for Exists, 0 for All) and the lowest decisive unit is the witness.

template <int LVL, int CNT>
__device__ __forceinline__ u32 tree_up(u32 y) {
#pragma unroll
    for (int j = 0; j < CNT; j++) {
        if ((NSAT_ALLBITS >> (LVL + j)) & 1ull) y &= (y >> (1 << j));
        else y |= (y >> (1 << j));
    }
    return y;
}

// bits at multiples of 2^k inside a 32-bit node vector
__device__ __forceinline__ constexpr u32 unit_mask(int k) {
    return k == 0 ? 0xffffffffu : k == 1 ? 0x55555555u : k == 2 ? 0x11111111u
         : k == 3 ? 0x01010101u : k == 4 ? 0x00010001u : 0x1u;
}

// decisive unit positions among `nodes` node results whose units are 2^k nodes
__device__ __forceinline__ u32 decisive(u32 y, int k, int nodes) {
    const u32 valid = nodes >= 32 ? 0xffffffffu : ((1u << nodes) - 1u);
    return (NSAT_Q0ALL ? ~y : y) & unit_mask(k) & valid;
}

// number of consecutive levels from level 0 that share level 0's quantifier
__device__ constexpr int low_run(u64 allbits) {
    int k = 1;
    while (k < 64 && (((allbits >> k) ^ allbits) & 1ull) == 0ull) k++;
    return k;
}

// The tree above the chunks.  A chunk is the range of items one CTA evaluates
// at a time (levels below LC); 2^CB chunks make the launch.  The levels from
// LC up to the units (or the whole launch) are cut into blocks of one
// quantifier, at most 8 levels each, and every block node counts its children:
// a child with the deciding value (0 under All, 1 under Exists), or the last
// of its children, resolves the node, and the node's value goes on to the
// block above.  A chunk below a resolved node cannot change anything and is
// not evaluated, nor is one whose units lie above a decisive unit.  A node is
// 16 bits: 0x8000 once resolved, the count of its undecided children below.
// The generator cuts the blocks and writes the walks through them.
constexpr int NSAT_LC = 10 + NSAT_IT + NSAT_WB;
constexpr int NSAT_TOP = NSAT_M < NSAT_C ? NSAT_M : NSAT_C;
// Order of the chunks: 2^UB units side by side, the chunks of each in order.
// One deciding child ends a node's other children, so the chunks in flight
// are spread over units; within a unit depth first decides most per chunk.
// 30 inputs, 1500 gates, alternating blocks of up to six, three formulas: 171,
// 186 and 272 us with up to 2^7 units side by side, 242, 319 and 268 with 2^4,
// 643, 457 and 812 with one after another; 1270 us when every chunk is
// evaluated.
constexpr int NSAT_UNITS = NSAT_M >= NSAT_LC && NSAT_M < NSAT_C ? NSAT_C - NSAT_M : 0;   // unit bits of a chunk index
constexpr int NSAT_UB = NSAT_UNITS < 7 ? NSAT_UNITS : 7;
__device__ __forceinline__ u32 chunk_of(u32 t) {
    if constexpr (NSAT_UB == 0) {
        return t;
    } else {
        constexpr int IN = NSAT_CB - NSAT_UNITS;           // bits below the units
        const u32 unit = t & ((1u << NSAT_UB) - 1u);
        const u32 in = (t >> NSAT_UB) & ((1u << IN) - 1u);
        const u32 up = t >> (NSAT_UB + IN);
        return (((up << NSAT_UB) | unit) << IN) | in;
    }
}

// One thread: chunk c has value v.
__device__ __forceinline__ void chunk_value(u32 c, u32 v, u32* nodes, LaunchOut* out) {
    if (!nsat_nodes_resolve(c, v, nodes)) return;
    if constexpr (NSAT_M >= NSAT_C) out->tree = v;
    else if (v == (NSAT_Q0ALL ? 0u : 1u)) atomicMin(&out->min_idx, (u64)(c >> (NSAT_M - NSAT_LC)));
}

// Resident CTAs take chunks until none is left: chunk blockIdx.x first, then
// from the launch's counter (out->values), one at a time while they need
// evaluation, up to 16 at once while they turn out decided (nsat_claim).
// NSAT_ONE: the launch has a CTA for every chunk.
extern "C" __global__ void NSAT_BOUNDS
nsat_qsat(u64 launch, LaunchOut* out, u64* host, u32 seq, u32* nodes, u32 shared, const u32* __restrict__ data) {
    nsat_begin(out);
    constexpr int M = NSAT_M;
    // Folding.  When levels 0..9 (the word and the warp tile) and the lowest
    // FOLD iteration levels all carry level 0's quantifier and lie below the
    // units, their nodes are one AND (or OR) over 2^(10+FOLD) items, taken in
    // any order: a thread combines its words over 2^FOLD iterations with one
    // op per word, and a compare plus a warp vote gives the node at level
    // L0 = 10+FOLD.  Otherwise the word and tile trees run per iteration and
    // L0 = 10.  Stage 2 reduces the IT2 = IT-FOLD remaining iteration levels.
    constexpr int QLOW = low_run(NSAT_ALLBITS);
    constexpr bool FOLDED = M >= 10 && QLOW >= 10;
    constexpr int FOLD_CAP = QLOW < M ? QLOW : M;
    constexpr int FOLD = !FOLDED ? 0 : (FOLD_CAP < 10 + NSAT_IT ? FOLD_CAP : 10 + NSAT_IT) - 10;
    constexpr bool LOW_ALL = (NSAT_ALLBITS & 1ull) != 0ull;
    constexpr int L0 = 10 + FOLD;
    constexpr int IT2 = NSAT_IT - FOLD;
    constexpr int G1 = IT2 < 5 ? IT2 : 5;
    constexpr int G2 = IT2 - G1;
    const u32 lane = threadIdx.x & 31u;
    const u32 warp = threadIdx.x >> 5;
    __shared__ u32 s_last, s_res[32];
    u32 cta = chunk_of(blockIdx.x);             // not checked: nothing is decided yet
#if !NSAT_ONE
    __shared__ u32 s_claim[3];     // warp 0's claim: chunks [0] + the bits of [1]; the chunk to evaluate
    u32 ahead = 0u;        // warp 0, lane 0: the next claim, made while the last chunk of one is evaluated
    if (threadIdx.x == 0) {
        s_claim[0] = blockIdx.x;
        s_claim[1] = 0u;
        ahead = atomicAdd(&out->values, 1u);
    }
#endif
    for (;;) {
        // index within the chunk (at most 25 bits) of this warp's first item
        const u32 warp_base = warp << (10 + NSAT_IT);
        u32 x[NSAT_NIN];
#if !NSAT_DATA
        nsat_inputs_fixed(x, lane, warp, cta, launch);
#endif
        u32 cand = ~0u;        // lowest decisive unit seen by this thread (within the chunk)
        u32 acc1 = 0, acc2 = 0;
        u32 yacc = LOW_ALL ? 0xffffffffu : 0u;
#pragma unroll 1
        for (u32 outer = 0; outer < (1u << NSAT_IT); outer += 1u << NSAT_INNER) {
#if !NSAT_DATA
        u32 ys[1 << NSAT_INNER];
        nsat_inputs_iter(x, outer);
        nsat_eval(x, ys);
#endif
#pragma unroll
        for (u32 inner = 0; inner < (1u << NSAT_INNER); inner++) {
            const u32 it = outer | inner;
#if NSAT_DATA
            const u64 gw = ((u64)launch << (NSAT_C - 5)) + ((u64)cta << (NSAT_LC - 5)) + ((warp_base + (it << 10)) >> 5) + lane;
            u32 y = data[gw];
#else
            u32 y = ys[inner];
#endif
            u32 b, git;   // node value at level L0 (bit 0) and its index among the warp's L0 nodes
            if constexpr (FOLDED) {
                yacc = LOW_ALL ? (yacc & y) : (yacc | y);
                if (((it + 1u) & ((1u << FOLD) - 1u)) != 0u) continue;
                const bool v = LOW_ALL ? (yacc == 0xffffffffu) : (yacc != 0u);
                yacc = LOW_ALL ? 0xffffffffu : 0u;
                b = LOW_ALL ? (u32)__all_sync(0xffffffffu, v) : (u32)__any_sync(0xffffffffu, v);
                git = it >> FOLD;
            } else {
                const u32 tile_base = warp_base + (it << 10);   // first item of this warp tile
                // stage 0: the 32 lanes of the word (levels 0..4)
                if constexpr (M < 5) {
                    y = tree_up<0, M>(y);
                    const u32 d = decisive(y, M, 32);
                    if (d != 0u && cand == ~0u)
                        cand = ((tile_base + (lane << 5)) >> M) + ((u32)(__ffs(d) - 1) >> M);
                    continue;
                } else {
                    y = tree_up<0, 5>(y);
                }
                // stage 1: the 32 words of the warp tile (levels 5..9)
                b = __ballot_sync(0xffffffffu, y & 1u);
                if constexpr (M >= 5 && M < 10) {
                    b = tree_up<5, M - 5>(b);
                    const u32 d = decisive(b, M - 5, 32);
                    if (d != 0u && cand == ~0u)
                        cand = (tile_base >> M) + ((u32)(__ffs(d) - 1) >> (M - 5));
                    continue;
                } else {
                    b = tree_up<5, 5>(b);
                }
                git = it;
            }
            // stage 2: the warp's L0 nodes (levels L0..10+IT-1), 2^G1 at a time
            if constexpr (M >= L0 && IT2 > 0) {
                const u32 pos = git & ((1u << G1) - 1u);
                acc1 |= (b & 1u) << pos;
                if (pos == (1u << G1) - 1u) {
                    const u32 grp_base = warp_base + ((git - pos) << L0);
                    if constexpr (M < L0 + G1) {
                        const u32 y1 = tree_up<L0, M - L0>(acc1);
                        const u32 d = decisive(y1, M - L0, 1 << G1);
                        if (d != 0u && cand == ~0u)
                            cand = (grp_base >> M) + ((u32)(__ffs(d) - 1) >> (M - L0));
                    } else {
                        const u32 y1 = tree_up<L0, G1>(acc1);
                        acc2 |= (y1 & 1u) << (git >> G1);
                    }
                    acc1 = 0;
                }
            } else if constexpr (M >= L0) {
                acc2 = b & 1u;   // IT2 == 0: one L0 node is the warp's whole range
            }
        }
        }
        // stage 2b: groups of L0 nodes (levels L0+G1 .. 10+IT-1)
        u32 wres = 0;
        if constexpr (M >= L0 + G1 && IT2 > 0) {
            if constexpr (M < L0 + IT2) {
                const u32 y2 = tree_up<L0 + G1, M - L0 - G1>(acc2);
                const u32 d = decisive(y2, M - L0 - G1, 1 << G2);
                if (d != 0u && cand == ~0u)
                    cand = (warp_base >> M) + ((u32)(__ffs(d) - 1) >> (M - L0 - G1));
            } else {
                wres = tree_up<L0 + G1, G2>(acc2) & 1u;
            }
        } else if constexpr (M >= L0 && IT2 == 0) {
            wres = acc2 & 1u;
        }
        // per-warp lowest candidate, one atomic per warp
        if constexpr (M < 10 + NSAT_IT) {
            cand = __reduce_min_sync(0xffffffffu, cand);
            if (lane == 0 && cand != ~0u) atomicMin(&out->min_idx, ((u64)cta << (NSAT_LC - M)) + cand);
        }
        // stage 3: warps of the CTA (levels 10+IT .. 10+IT+WB-1); its value goes to
        // the tree above the chunks
        if constexpr (M >= 10 + NSAT_IT) {
            if (lane == 0) s_res[warp] = wres;
            __syncthreads();
            if (warp == 0) {
                const u32 mbits = __ballot_sync(0xffffffffu, lane < (1u << NSAT_WB) ? s_res[lane] : 0u);
                if constexpr (M < NSAT_LC) {
                    const u64 cta_base = (u64)cta << NSAT_LC;
                    const u32 y3 = tree_up<10 + NSAT_IT, M - 10 - NSAT_IT>(mbits);
                    const u32 d = decisive(y3, M - 10 - NSAT_IT, 1 << NSAT_WB);
                    if (lane == 0 && d != 0u)
                        atomicMin(&out->min_idx, (cta_base >> M) + (u64)((__ffs(d) - 1) >> (M - 10 - NSAT_IT)));
                } else {
                    const u32 cres = tree_up<10 + NSAT_IT, NSAT_WB>(mbits) & 1u;
                    if (lane == 0) chunk_value(cta, cres, nodes, out);
                }
            }
        }
        __syncthreads();       // s_claim and s_res are written again
#if NSAT_ONE
        break;
#else
        if (warp == 0) nsat_claim(lane, nodes, &out->min_idx, &out->values, s_claim, ahead);
        __syncthreads();
        cta = s_claim[2];
        if (cta == ~0u) break;
#endif
    }
    // the last CTA puts the nodes and the counter back to zero
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&out->ticket, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        for (u32 i = threadIdx.x; i < (NSAT_NODES + 1u) / 2u; i += NSAT_NT) nodes[i] = 0u;
        // the words release the host, and a launch of another stream may take
        // shared nodes over then: every thread's zeros come before them (which
        // takes 0.5-1 us; nodes of one stream need no more than its order)
        if (shared) {
            __threadfence();
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            out->values = 0u;
            nsat_publish(out, host, seq);
        }
    }
}
#endif

#if NSAT_MODE_TABLE
// --------------------------------------------------------------------------
// SATOSTOP next-state table: entry[s] = next(s) | STOP(s) << n.
// One thread evaluates 32 states bit-sliced, then transposes the 32x32 bit
// matrix (rows = outputs, columns = lanes) into per-state entries.

// Block-swap transposition of a 32x32 bit matrix: after the step for size j,
// rows k and k+j have exchanged their off-diagonal j x j blocks.  Sizes 16 and
// 8 are byte permutations.  As asm blocks of 16 rows: written as loops, it was
// two fifths of a small circuit's compile (46 of 114 ms).
#define NSAT_SWAP16(A, B) \
    "prmt.b32 t, %" #A ", %" #B ", 0x5410;\n\tprmt.b32 %" #B ", %" #A ", %" #B ", 0x7632;\n\tmov.b32 %" #A ", t;\n\t"
#define NSAT_SWAP8(A, B) \
    "prmt.b32 t, %" #A ", %" #B ", 0x6240;\n\tprmt.b32 %" #B ", %" #A ", %" #B ", 0x7351;\n\tmov.b32 %" #A ", t;\n\t"
// rows A, B <- A & M | (B << J) & ~M, (A >> J) & M | B & ~M
#define NSAT_SWAP(A, B, J, M) \
    "shl.b32 t, %" #B ", " #J ";\n\tshr.b32 s, %" #A ", " #J ";\n\t" \
    "lop3.b32 %" #A ", %" #A ", t, " #M ", 0xe4;\n\tlop3.b32 %" #B ", s, %" #B ", " #M ", 0xe4;\n\t"
#define NSAT_STEP(S, a, b, c, d, e, f, g, h, i, j, k, l, m, n, o, p) \
    S(a, b) S(c, d) S(e, f) S(g, h) S(i, j) S(k, l) S(m, n) S(o, p)
#define NSAT_SWAP4(A, B) NSAT_SWAP(A, B, 4, 0x0f0f0f0f)
#define NSAT_SWAP2(A, B) NSAT_SWAP(A, B, 2, 0x33333333)
#define NSAT_SWAP1(A, B) NSAT_SWAP(A, B, 1, 0x55555555)
#define NSAT_ROWS(A, k, B, l)                                                                                      \
    "+r"(A[k]), "+r"(A[k + 1]), "+r"(A[k + 2]), "+r"(A[k + 3]), "+r"(A[k + 4]), "+r"(A[k + 5]), "+r"(A[k + 6]),     \
        "+r"(A[k + 7]), "+r"(B[l]), "+r"(B[l + 1]), "+r"(B[l + 2]), "+r"(B[l + 3]), "+r"(B[l + 4]), "+r"(B[l + 5]), \
        "+r"(B[l + 6]), "+r"(B[l + 7])

__device__ __forceinline__ void transpose32(u32* a) {
#pragma unroll
    for (int k = 0; k < 16; k += 8)
        asm("{ .reg .b32 t;\n\t"
            NSAT_STEP(NSAT_SWAP16, 0, 8, 1, 9, 2, 10, 3, 11, 4, 12, 5, 13, 6, 14, 7, 15) "}" : NSAT_ROWS(a, k, a, k + 16));
#pragma unroll
    for (int k = 0; k < 32; k += 16)
        asm("{ .reg .b32 s, t;\n\t"
            NSAT_STEP(NSAT_SWAP8, 0, 8, 1, 9, 2, 10, 3, 11, 4, 12, 5, 13, 6, 14, 7, 15)
            NSAT_STEP(NSAT_SWAP4, 0, 4, 1, 5, 2, 6, 3, 7, 8, 12, 9, 13, 10, 14, 11, 15)
            NSAT_STEP(NSAT_SWAP2, 0, 2, 1, 3, 4, 6, 5, 7, 8, 10, 9, 11, 12, 14, 13, 15)
            NSAT_STEP(NSAT_SWAP1, 0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15) "}" : NSAT_ROWS(a, k, a, k + 8));
}

// Tables of 32-bit entries of 2^10 states and more are whole warps of words:
// a warp stages its entries in shared memory and writes them as one run.  A
// thread writing its own 128 bytes made every store instruction touch 32
// lines (2^28 entries: 715 us, 1.5 TB/s; staged 270 us).
constexpr bool NSAT_STAGED = NSAT_FMT == 0 && NSAT_NB >= 10;

extern "C" __global__ void NSAT_BOUNDS
nsat_table(u64 nwords, u64 w0, void* __restrict__ table, LaunchOut* out, u64* host, u32 seq) {
    nsat_begin(out);
    // entries of words w0 .. w0+nwords-1 (32 states each), stored from table[0]
    const u64 stride = (u64)gridDim.x * NSAT_NT;
    u32 anystop = 0;
#if NSAT_FMT == 0
    __shared__ u32 stage[NSAT_STAGED ? NSAT_NT / 32 : 1][NSAT_STAGED ? 32 * 33 : 1];
#endif
    for (u64 w = (u64)blockIdx.x * NSAT_NT + threadIdx.x; w < nwords; w += stride) {
        u32 x[NSAT_NIN];
        nsat_inputs_word(x, w0 + w);
        constexpr int ROWS = NSAT_FMT == 0 ? 32 : 64;
        u32 o[ROWS];
#pragma unroll
        for (int k = NSAT_NOUT; k < ROWS; k++) o[k] = 0u;
        nsat_eval_all(x, o);
        anystop |= o[NSAT_NOUT - 1];
        constexpr int lanes = NSAT_NB >= 5 ? 32 : (1 << NSAT_NB);
        transpose32(o);
#if NSAT_FMT == 0
        if constexpr (NSAT_STAGED) {
            const u32 lane = threadIdx.x & 31u;
            u32* st = stage[threadIdx.x >> 5];
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 32; k++) st[lane * 33 + k] = o[k];
            __syncwarp();
            u32* dst = reinterpret_cast<u32*>(table) + ((w - lane) << 5);
#pragma unroll 4
            for (int k = 0; k < 32; k++) dst[k * 32 + lane] = st[k * 33 + lane];
        } else {
            for (int l = 0; l < lanes; l++) reinterpret_cast<u32*>(table)[(w << 5) + l] = o[l];
        }
#else
        if (NSAT_NOUT > 32) transpose32(o + 32);
        u64* t64 = reinterpret_cast<u64*>(table) + (w << 5);
        if (lanes == 32) {
            ulonglong2* dst = reinterpret_cast<ulonglong2*>(t64);
#pragma unroll
            for (int q = 0; q < 16; q++) {
                ulonglong2 v;
                v.x = (u64)o[2 * q] | ((u64)o[32 + 2 * q] << 32);
                v.y = (u64)o[2 * q + 1] | ((u64)o[32 + 2 * q + 1] << 32);
                __stcs(dst + q, v);
            }
        } else {
            for (int l = 0; l < lanes; l++) t64[l] = (u64)o[l] | ((u64)o[32 + l] << 32);
        }
#endif
    }
    if (__any_sync(0xffffffffu, anystop != 0u) && (threadIdx.x & 31u) == 0) atomicOr(&out->any, 1u);
    nsat_finish(out, host, seq);
}
#endif
