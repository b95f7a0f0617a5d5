// codegen.cpp -- emit the per-circuit CUDA source compiled by NVRTC.
#include "codegen.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <sstream>
#include <unordered_map>

namespace nsat {

std::string KernelConfig::key() const {
    std::ostringstream s;
    s << "mode=" << (int)mode << " nin=" << nin << " nb=" << nb << " c=" << c << " it=" << it << " wb=" << wb << " cb=" << cb
      << " m=" << m << " q0all=" << q0all << " allbits=" << allbits << " data=" << data
      << " fmt=" << fmt << " nout=" << nout << " minb=" << minb << " sync=" << sync_every << " map=";
    for (int v : in_of_bit) s << v << ',';
    return s.str();
}

namespace {

const char* kPrelude = R"NSAT(
typedef unsigned int u32;
typedef unsigned long long u64;
)NSAT";

// LUTs of one asm block without barriers, and where the evaluators use blocks:
// from 400 LUTs (the compiler's sharing between iterations is worth more
// below: 24 inputs, 280 LUTs, run 139 instructions a word), for searches of up
// to 2 ms.  Blocks compile a 2000-3000-gate circuit 70-120 ms faster and run
// 0.1-0.9 % slower (33 inputs, 1216 LUTs: first solve 476 -> 350 ms, device
// time 17.74 -> 17.76 ms): longer searches keep the faster loop.
constexpr uint32_t kBlockLuts = 128;
constexpr size_t kBlocksFrom = 400;
bool use_blocks(const KernelConfig& kc, const LutNet& net) {
    if (kc.mode == Mode::TABLE) return true;
    if (net.luts.size() < kBlocksFrom) return false;
    return kc.mode == Mode::QSAT ||
           std::ldexp((double)net.luts.size(), (int)kc.nb - 5) < 2e-3 * kCompiledLutWordsPerS;
}

const uint32_t kLanePat[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};

void append_dec(std::string& o, uint32_t v) {
    char t[10];
    int d = 0;
    do { t[d++] = (char)('0' + v % 10); v /= 10; } while (v);
    while (d) o.push_back(t[--d]);
}

void append_tt(std::string& o, uint8_t tt) {
    static const char kHex[] = "0123456789abcdef";
    o += "0x";
    o.push_back(kHex[tt >> 4]);
    o.push_back(kHex[tt & 15]);
}

// One asm statement per LUT: the compiler hoists and shares single LUTs, which
// is worth half of a small circuit's work when it unrolls the iterations.
void emit_single_luts(std::string& b, const LutNet& net, uint32_t sync_every) {
    uint32_t k = 0;
    b.reserve(net.luts.size() * 112 + (sync_every ? net.luts.size() / sync_every * 20 : 0) + 16);
    for (const Lut& L : net.luts) {
        b += "    u32 w";
        append_dec(b, L.wire);
        b += "; asm(\"lop3.b32 %0, %1, %2, %3, ";
        append_tt(b, L.tt);
        b += ";\" : \"=r\"(w";
        append_dec(b, L.wire);
        b += ") : \"r\"(w";
        append_dec(b, L.in[0]);
        b += "), \"r\"(w";
        append_dec(b, L.in[1]);
        b += "), \"r\"(w";
        append_dec(b, L.in[2]);
        b += "));\n";
        if (sync_every && ++k % sync_every == 0) b += "    __syncthreads();\n";
    }
}

// One asm block per `seg` LUTs, whose operands are the wires that cross the
// block's ends.  The front end and the optimiser see one statement where there
// were `seg`: 1229 LUTs compile in 531 ms instead of 701, a
// 24-bit next-state table in 135 instead of 149.
void emit_lut_blocks(std::string& b, const LutNet& net, uint32_t seg, bool sync) {
    const size_t n = net.luts.size();
    std::unordered_map<uint32_t, size_t> last;       // wire -> last LUT that reads it (n: an output)
    for (size_t k = 0; k < n; k++)
        for (int i = 0; i < 3; i++) last[net.luts[k].in[i]] = k;
    for (const Output& o : net.outs) last[o.wire] = n;
    b.reserve(n * 48 + 256);
    std::unordered_map<uint32_t, std::string> name;
    for (size_t a = 0; a < n; a += seg) {
        const size_t e = std::min(n, a + seg);
        name.clear();
        std::string outs, ins, decl;
        uint32_t ops = 0, temps = 0;
        auto operand = [&](uint32_t w) {
            std::string t = "%";
            append_dec(t, ops++);
            name[w] = t;
        };
        for (size_t k = a; k < e; k++) {             // outputs first, as asm operands are numbered
            const uint32_t w = net.luts[k].wire;
            const auto l = last.find(w);
            if (l == last.end() || l->second < e) {
                std::string t = "t";
                append_dec(t, temps++);
                name[w] = t;
                continue;
            }
            operand(w);
            outs += (outs.empty() ? "\"=&r\"(w" : ", \"=&r\"(w");
            append_dec(outs, w);
            outs += ")";
            decl += decl.empty() ? "    u32 w" : ", w";
            append_dec(decl, w);
        }
        for (size_t k = a; k < e; k++)
            for (int i = 0; i < 3; i++) {
                const uint32_t w = net.luts[k].in[i];
                if (name.count(w)) continue;
                operand(w);
                ins += (ins.empty() ? "\"r\"(w" : ", \"r\"(w");
                append_dec(ins, w);
                ins += ")";
            }
        b += decl + ";\n    asm(\"{ .reg .b32 t<";
        append_dec(b, temps + 1);
        b += ">;\\n\"\n";
        for (size_t k = a; k < e; k++) {
            const Lut& L = net.luts[k];
            b += "\"lop3.b32 " + name[L.wire] + ", " + name[L.in[0]] + ", " + name[L.in[1]] + ", " + name[L.in[2]] + ", ";
            append_tt(b, L.tt);
            b += ";\\n\"\n";
        }
        b += "\"}\" : " + outs + " : " + ins + ");\n";
        if (sync && e - a == seg) b += "    __syncthreads();\n";
    }
}

// The evaluation of the LUTs, one lop3.b32 each with the truth table as its
// immediate.  sync_every > 0: a CTA barrier after every sync_every LUTs, so
// the CTA's warps walk the evaluation code together and share
// instruction-cache lines (the unrolled evaluation of a large circuit is larger
// than the instruction cache; c1 at 64: ALU pipe 89 % -> 0.99 of the lop3
// peak).  Only for kernels whose every thread runs the same number of
// evaluations.  The lines are appended directly: formatting them through
// printf took most of the generation time.
void emit_luts(std::ostringstream& s, const LutNet& net, bool blocks, uint32_t sync_every = 0) {
    for (uint32_t i : net.used_inputs) s << "    const u32 w" << i << " = x[" << i << "];\n";
    std::string b;
    if (blocks) emit_lut_blocks(b, net, sync_every ? sync_every : kBlockLuts, sync_every != 0);
    else emit_single_luts(b, net, sync_every);
    s.write(b.data(), (std::streamsize)b.size());
}

// Iterations evaluated together: 2^inner copies of the LUTs that depend on the
// iteration's lowest inner bits, beside one of the rest (shared).  In copy c
// those bits are the constants of c, which are folded here: the compiler does
// not fold every lop3 (36 inputs, 3018 gates, planted block: 83 or 163 ms by
// the circuit, 8.9-11.1 ms for six circuits folded here).  A copy that folds to
// a constant costs nothing, as half of the copies do for each bit that a
// conjunction tests.
struct Parts {
    uint32_t inner = 0;
    LutNet shared;                       // used_inputs: of the copies too
    std::vector<LutNet> copies;          // wires renamed; outs empty: constant
    std::vector<uint8_t> constant;       // the output, where a copy's is constant
    size_t luts() const {
        size_t n = shared.luts.size();
        for (const LutNet& c : copies) n += c.luts.size();
        return n;
    }
};

Parts fold(const KernelConfig& kc, const LutNet& net, uint32_t inner) {
    Parts p;
    p.inner = inner;
    uint32_t wires = kc.nin;
    for (const Lut& l : net.luts) wires = std::max(wires, l.wire + 1);
    for (const Output& o : net.outs) wires = std::max(wires, o.wire + 1);
    std::vector<uint8_t> gate(wires, 0), own(wires, 0);   // kc.nin counts a small circuit's padding too
    for (uint32_t k = 0; k < inner; k++)
        if (kc.in_of_bit[10 + k] >= 0) own[kc.in_of_bit[10 + k]] = 1;
    for (const Lut& l : net.luts) {
        gate[l.wire] = 1;
        own[l.wire] = own[l.in[0]] | own[l.in[1]] | own[l.in[2]];
    }
    std::vector<uint8_t> need(wires, 0);                  // wires that the copies read
    for (uint32_t c = 0; c < (1u << inner); c++) {
        const auto renamed = [&](uint32_t w) { return own[w] && gate[w] ? wires * (c + 1) + w : w; };
        std::vector<int8_t> value(wires, -1);             // constant value or -1
        for (uint32_t k = 0; k < inner; k++)
            if (kc.in_of_bit[10 + k] >= 0) value[kc.in_of_bit[10 + k]] = (int8_t)((c >> k) & 1u);
        std::vector<Lut> luts;
        for (const Lut& l : net.luts) {
            if (!own[l.wire]) continue;
            // fix the constant operands, and equal ones to each other
            uint32_t any = l.wire;
            for (const uint32_t w : l.in)
                if (value[w] < 0) any = w;
            uint8_t tt = 0;
            bool ones = true, zeros = true;
            for (uint32_t row = 0; row < 8; row++) {
                uint32_t at = 0;
                bool real = true;                         // the row gives equal wires equal values
                for (int i = 0; i < 3; i++) {
                    const uint32_t bit = (row >> (2 - i)) & 1u;
                    at = at << 1 | (value[l.in[i]] >= 0 ? (uint32_t)value[l.in[i]] : bit);
                    for (int h = 0; h < i; h++) {
                        const bool same = value[l.in[i]] < 0 && l.in[h] == l.in[i];
                        if (same && ((row >> (2 - h)) & 1u) != bit) real = false;
                    }
                }
                const uint32_t v = (l.tt >> at) & 1u;
                tt |= (uint8_t)(v << row);
                if (real) (v ? zeros : ones) = false;
            }
            if (zeros || ones) {
                value[l.wire] = ones ? 1 : 0;
                continue;
            }
            Lut m = l;
            m.tt = tt;
            for (uint32_t& w : m.in)
                if (value[w] >= 0) w = any;
            luts.push_back(m);
        }
        LutNet net_c;
        const Output out = net.outs[0];
        if (value[out.wire] >= 0) {
            p.constant.push_back((uint8_t)(value[out.wire] ^ (out.neg ? 1 : 0)));
        } else {
            p.constant.push_back(0);
            std::vector<uint8_t> live(wires, 0);
            live[out.wire] = 1;
            for (size_t k = luts.size(); k-- > 0;)
                if (live[luts[k].wire])
                    for (const uint32_t w : luts[k].in) live[w] = 1;
            for (uint32_t w = 0; w < wires; w++)
                if (live[w] && !(own[w] && gate[w])) need[w] = 1;
            for (Lut m : luts) {
                if (!live[m.wire]) continue;
                m.wire = renamed(m.wire);
                for (uint32_t& w : m.in) w = renamed(w);
                net_c.luts.push_back(m);
            }
            net_c.outs.push_back(Output{renamed(out.wire), out.neg});
        }
        p.copies.push_back(std::move(net_c));
    }
    for (uint32_t w = 0; w < wires; w++)
        if (need[w] && gate[w]) p.shared.outs.push_back(Output{w, false});
    std::vector<uint8_t> keep(net.luts.size(), 0);
    for (size_t k = net.luts.size(); k-- > 0;) {
        const Lut& l = net.luts[k];
        if (own[l.wire] || !need[l.wire]) continue;
        keep[k] = 1;
        for (const uint32_t w : l.in) need[w] = 1;
    }
    for (size_t k = 0; k < net.luts.size(); k++)
        if (keep[k]) p.shared.luts.push_back(net.luts[k]);
    for (uint32_t w = 0; w < wires; w++)
        if (need[w] && !gate[w]) p.shared.used_inputs.push_back(w);
    return p;
}

// inner is the largest (up to 4) whose code stays within a budget, which is
// about what the compiler's own unrolling took: 2400 LUTs or two copies for
// SAT, 640 (a quantifier tree's share of a copy counted as 40) or little more
// than one copy for QSAT, whose calls are shorter.  Device time in us and first
// call in ms, left to the compiler and so: SAT 81 LUTs, 32 inputs 395, 76 and
// 116, 70; 201 LUTs, 33 inputs 2993, 102 and 1384, 73; 652 LUTs, 30 inputs
// 1190, 198 and 1147, 108.  QSAT 14 LUTs, 30 inputs 61, 90 and 33, 100; 339
// LUTs, 26 inputs 41, 121 and 34, 122, both with the chunk tree's code as
// statements (emit_tree), which was 20-45 ms of these first calls.  With 400 for
// QSAT a 38-LUT adder takes 68 instead of 60 us and compiles no faster.
constexpr uint32_t kMostInner = 4;
Parts split(const KernelConfig& kc, const LutNet& net) {
    const bool sat = kc.mode == Mode::SAT;
    const size_t n = net.luts.size();
    const size_t budget = sat ? std::max<size_t>(2400, 2 * n + 16) : std::max<size_t>(640, n + n / 8 + 80);
    Parts best = fold(kc, net, 0);
    for (uint32_t k = 1; k <= std::min(kc.it, kMostInner); k++) {
        Parts p = fold(kc, net, k);
        if (p.luts() + ((sat ? 8u : 40u) << k) > budget) break;
        best = std::move(p);
    }
    return best;
}

// The tree above the chunks of a QSAT launch (device_template.cuh): a block's
// first node, the chunk bits below one of its nodes, the children that a node
// has, and their quantifier.
struct TreeBlock {
    uint32_t first, shift, children;
    bool all;
};

// The walks of a chunk up the blocks' nodes and the claims of chunks, as asm:
// nsat_nodes_resolve enters the value v of chunk c and returns whether it
// resolved the last block's node too; nsat_claim finds the next chunk that is
// not decided.  As statements they took up to a fifth of a formula's first call,
// which had become longer than with no tree at all (32-input adder with a key 88
// -> 108 ms, 80 so; 28 inputs, 80 gates, blocks of up to five 89 -> 98,
// 67 so).  A loop over a table in constant memory in place of the walks
// compiles as fast, but waits for each node's load (30 inputs, 1500 gates 183 ->
// 203 us).
void emit_tree(std::ostringstream& s, const KernelConfig& kc) {
    const uint32_t lc = 10 + kc.it + kc.wb, top = std::min(kc.m, kc.c);
    std::vector<TreeBlock> blocks;
    uint32_t nodes = 0;
    const auto all = [&](uint32_t l) { return ((kc.allbits >> l) & 1u) != 0; };
    for (uint32_t lo = lc, hi; lo < top; lo = hi) {
        for (hi = lo + 1; hi < top && hi - lo < 8 && all(hi) == all(lo); hi++) {}
        blocks.push_back(TreeBlock{nodes, hi - lc, 1u << (hi - lo), all(lo)});
        nodes += 1u << (kc.c - hi);
    }
    s << "constexpr u32 NSAT_NODES = " << nodes << "u;\n";
    const auto line = [&s](const std::string& l) { s << "\"" << l << "\\n\"\n"; };
    const auto num = [](uint64_t v) { return std::to_string(v); };

    s << "__device__ __forceinline__ bool nsat_nodes_resolve(u32 c, u32 v, u32* nodes) {\n"
      << "    u32 up = 0u;\n    asm volatile(\n";
    line("{ .reg .pred p; .reg .b32 i, h, m, o; .reg .b64 a;");
    for (size_t k = 0; k < blocks.size(); k++) {
        const TreeBlock& b = blocks[k];
        // node i: half h of word a
        line("shr.u32 i, %1, " + num(b.shift) + "; add.u32 i, i, " + num(b.first) +
             "; and.b32 h, i, 1; shl.b32 h, h, 4; shr.u32 i, i, 1; mul.wide.u32 a, i, 4; add.u64 a, a, %3;");
        // neither the deciding value nor the last child (or the node is resolved): done
        line("setp.ne.u32 p, %2, " + num(b.all ? 1 : 0) + "; @p bra R" + num(k) +
             "; mov.b32 m, 1; shl.b32 m, m, h; atom.global.add.u32 o, [a], m; shr.u32 o, o, h; and.b32 o, o, 0xffff;");
        line("setp.ne.u32 p, o, " + num(b.children - 1) + "; @p bra D;");
        line("R" + num(k) + ": mov.b32 m, 0x8000; shl.b32 m, m, h; atom.global.or.b32 o, [a], m; and.b32 o, o, m; "
             "setp.ne.u32 p, o, 0; @p bra D;");
    }
    line("mov.b32 %0, 1; D: }");
    s << ": \"+r\"(up) : \"r\"(c), \"r\"(v), \"l\"(nodes) : \"memory\");\n    return up != 0u;\n}\n";
    if (kc.cb <= kResidentBits) return;

    // One warp.  claim: first chunk index b, mask m of those not looked at yet,
    // the chunk found (~0: none left).  k: how many the next claim takes, 0 when
    // it has been made ahead.
    const uint32_t units = kc.m >= lc && kc.m < kc.c ? kc.c - kc.m : 0, side = std::min(units, 7u);
    const uint32_t in = kc.cb - units;
    s << "__device__ __forceinline__ void nsat_claim(u32 lane, const u32* nodes, const u64* lowest, u32* counter, "
      << "u32* claim, u32& ahead) {\n    asm volatile(\n";
    line("{ .reg .pred p, q; .reg .b32 t, i, m, k, b, c; .reg .b64 a, l, x; .reg .b16 v, w<" + num(blocks.size() + 1) + ">;");
    line("ld.shared.u32 b, [%5]; ld.shared.u32 m, [%5+4]; setp.ne.u32 p, m, 0; selp.b32 k, 1, 0, p;");
    // the next claim, by lane 0
    line("L: setp.ne.u32 p, m, 0; @p bra C;");
    line("setp.ne.u32 p, k, 0; setp.eq.and.u32 q, %1, 0, p; @q atom.global.add.u32 %0, [%4], k; max.u32 k, k, 1;");
    line("shfl.sync.idx.b32 b, %0, 0, 31, 0xffffffff; mov.u32 t, %%nctaid.x; add.u32 b, b, t;");
    line("mov.b32 m, 1; shl.b32 m, m, k; sub.u32 m, m, 1; shl.b32 k, k, 1; min.u32 k, k, 16;");
    // a lane each: p, chunk c is open
    line("C: add.u32 t, b, %1; shr.u32 i, m, %1; and.b32 i, i, 1; setp.ne.u32 p, i, 0; setp.lt.and.u32 p, t, " +
         num(1ull << kc.cb) + ", p;");
    if (side == 0) line("mov.b32 c, t;");
    else                                     // chunk_of
        line("and.b32 i, t, " + num((1u << side) - 1) + "; shr.u32 c, t, " + num(side + in) + "; shl.b32 c, c, " + num(side) +
             "; or.b32 c, c, i; shl.b32 c, c, " + num(in) + "; shr.u32 i, t, " + num(side) + "; and.b32 i, i, " +
             num((1u << in) - 1) + "; or.b32 c, c, i;");
    for (size_t k = 0; k < blocks.size(); k++)      // every load before the first use
        line("mov.b16 w" + num(k) + ", 0; shr.u32 i, c, " + num(blocks[k].shift) + "; add.u32 i, i, " + num(blocks[k].first) +
             "; mul.wide.u32 a, i, 2; add.u64 a, a, %2; @p ld.volatile.global.u16 w" + num(k) + ", [a];");
    // no unit below chunk c's (or its own, where a unit has several chunks) is decisive
    if (kc.m < kc.c) line("mov.b64 l, 0; @p ld.volatile.global.u64 l, [%3]; cvt.u64.u32 x, c;");
    line("mov.b16 v, 0;");
    for (size_t k = 0; k < blocks.size(); k++) line("or.b16 v, v, w" + num(k) + ";");
    line("and.b16 v, v, 0x8000; setp.eq.and.u16 p, v, 0, p;");
    if (kc.m < kc.c)
        line(kc.m >= lc ? "shr.u64 x, x, " + num(kc.m - lc) + "; setp.gt.and.u64 p, l, x, p;"
                        : "shl.b64 x, x, " + num(lc - kc.m) + "; setp.ge.and.u64 p, l, x, p;");
    line("vote.sync.ballot.b32 m, p, 0xffffffff; setp.eq.u32 p, m, 0; setp.lt.and.u32 q, b, " + num(1ull << kc.cb) +
         ", p; @q bra L;");
    // the first open one; the next claim ahead when it is the last of this one
    line("neg.s32 t, m; and.b32 t, t, m; bfind.u32 t, t; sub.u32 i, m, 1; and.b32 m, m, i;");
    line("shfl.sync.idx.b32 c, c, t, 31, 0xffffffff; selp.b32 c, -1, c, p;");
    line("setp.ne.u32 p, c, -1; setp.eq.and.u32 p, m, 0, p; setp.eq.and.u32 p, %1, 0, p; @p atom.global.add.u32 %0, [%4], 1;");
    line("setp.eq.u32 q, %1, 0; @q st.shared.u32 [%5], b; @q st.shared.u32 [%5+4], m; @q st.shared.u32 [%5+8], c; }");
    s << ": \"+r\"(ahead) : \"r\"(lane), \"l\"(nodes), \"l\"(lowest), \"l\"(counter), "
      << "\"r\"((u32)__cvta_generic_to_shared(claim)) : \"memory\");\n}\n";
}

}  // namespace

std::string generate_source(const KernelConfig& kc, const LutNet& net) {
    std::ostringstream s;
    s << "// generated: " << kc.key() << "\n";
    s << kPrelude;
    s << "#define NSAT_MODE_SAT " << (kc.mode == Mode::SAT ? 1 : 0) << "\n";
    s << "#define NSAT_MODE_QSAT " << (kc.mode == Mode::QSAT ? 1 : 0) << "\n";
    s << "#define NSAT_MODE_TABLE " << (kc.mode == Mode::TABLE ? 1 : 0) << "\n";
    s << "#define NSAT_DATA " << (kc.data ? 1 : 0) << "\n";
    s << "#define NSAT_FMT " << kc.fmt << "\n";
    s << "constexpr int NSAT_NIN = " << kc.nin << ";\n";
    s << "constexpr int NSAT_NOUT = " << kc.nout << ";\n";
    s << "constexpr int NSAT_NB = " << kc.nb << ";\n";
    s << "constexpr int NSAT_NT = " << kc.threads() << ";\n";
    if (kc.minb) s << "#define NSAT_BOUNDS __launch_bounds__(" << kc.threads() << ", " << kc.minb << ")\n";
    else s << "#define NSAT_BOUNDS __launch_bounds__(" << kc.threads() << ")\n";
    s << "constexpr int NSAT_IT = " << kc.it << ";\n";
    s << "constexpr int NSAT_WB = " << kc.wb << ";\n";
    s << "constexpr int NSAT_CB = " << kc.cb << ";\n";
    s << "constexpr int NSAT_C = " << kc.c << ";\n";
    s << "constexpr int NSAT_M = " << kc.m << ";\n";
    s << "constexpr int NSAT_Q0ALL = " << (kc.q0all ? 1 : 0) << ";\n";
    s << "constexpr u64 NSAT_ALLBITS = " << kc.allbits << "ull;\n";

    s << "#define NSAT_ONE " << (kc.cb <= kResidentBits ? 1 : 0) << "\n";
    const Parts parts = kc.mode == Mode::TABLE || kc.data ? Parts() : split(kc, net);
    s << "#define NSAT_INNER " << parts.inner << "\n";

    // enumeration: which circuit input each bit drives
    const uint32_t it_lo = 10, wb_lo = 10 + kc.it, cb_lo = wb_lo + kc.wb, c_lo = cb_lo + kc.cb;
    std::ostringstream fixed, iter, word;
    char buf[160];
    for (uint32_t p = 0; p < kc.nb; p++) {
        int in = kc.in_of_bit[p];
        if (in < 0) continue;
        if (p < 5) {
            snprintf(buf, sizeof(buf), "    x[%d] = 0x%08xu;\n", in, kLanePat[p]);
            fixed << buf;
            word << buf;
            continue;
        }
        snprintf(buf, sizeof(buf), "    x[%d] = 0u - (u32)((w >> %u) & 1ull);\n", in, p - 5);
        word << buf;
        if (p < it_lo) snprintf(buf, sizeof(buf), "    x[%d] = 0u - ((lane >> %u) & 1u);\n", in, p - 5);
        else if (p < wb_lo) {
            snprintf(buf, sizeof(buf), "    x[%d] = 0u - ((it >> %u) & 1u);\n", in, p - it_lo);
            iter << buf;
            continue;
        } else if (p < cb_lo) snprintf(buf, sizeof(buf), "    x[%d] = 0u - ((warp >> %u) & 1u);\n", in, p - wb_lo);
        else if (p < c_lo) snprintf(buf, sizeof(buf), "    x[%d] = 0u - ((cta >> %u) & 1u);\n", in, p - cb_lo);
        else if (p - c_lo < 64) snprintf(buf, sizeof(buf), "    x[%d] = 0u - (u32)((launch >> %u) & 1ull);\n", in, p - c_lo);
        else snprintf(buf, sizeof(buf), "    x[%d] = 0u;\n", in);
        fixed << buf;
    }
    s << "__device__ __forceinline__ void nsat_inputs_fixed(u32* x, u32 lane, u32 warp, u32 cta, u64 launch) {\n"
      << "    (void)lane; (void)warp; (void)cta; (void)launch;\n"
      << fixed.str() << "}\n";
    s << "__device__ __forceinline__ void nsat_inputs_iter(u32* x, u32 it) {\n    (void)it;\n"
      << iter.str() << "}\n";
    s << "__device__ __forceinline__ void nsat_inputs_word(u32* x, u64 w) {\n    (void)w;\n"
      << word.str() << "}\n";

    // circuit evaluation
    if (kc.mode == Mode::TABLE) {
        s << "__device__ __forceinline__ void nsat_eval_all(const u32* x, u32* o) {\n";
        emit_luts(s, net, use_blocks(kc, net));
        for (size_t j = 0; j < net.outs.size(); j++)
            s << "    o[" << j << "] = " << (net.outs[j].neg ? "~" : "") << "w" << net.outs[j].wire << ";\n";
        s << "}\n";
    } else {
        // the SAT and QSAT kernels run the same number of evaluations in every
        // thread of a CTA, so barriers inside the evaluation are safe
        const uint32_t sync = kc.threads() > 32 ? kc.sync_every : 0;
        const bool blocks = use_blocks(kc, net);
        s << "__device__ __forceinline__ void nsat_eval(const u32* x, u32* y) {\n";
        emit_luts(s, parts.shared, blocks, sync);
        for (size_t k = 0; k < parts.copies.size(); k++) {
            const LutNet& copy = parts.copies[k];
            emit_luts(s, copy, blocks, sync);
            s << "    y[" << k << "] = ";
            if (copy.outs.empty()) s << (parts.constant[k] ? "~0u" : "0u") << ";\n";
            else s << (copy.outs[0].neg ? "~" : "") << "w" << copy.outs[0].wire << ";\n";
        }
        s << "}\n";
    }
    if (kc.mode == Mode::QSAT) emit_tree(s, kc);
    s << kDeviceTemplate;
    return s.str();
}

}  // namespace nsat
