// Device entropy coder in the RleFseEncoder<int16_t> stream format (see entropy.cuh).
//
// Reference (JLiu-1/Falcons include/Falcons/encoder/RleFseEncoder.hpp):
//   preprocess_encode :850-895   method / delta decision from 256 x 32 sampled windows
//   encode (method 0) :897-982   runs of zeros + values as Elias-gamma class bytes + raw mantissas
//   fse_enc / fse_dec :150-187   class bytes FSE-coded in 64 Ki-symbol blocks
//   O1Lut             :354-391   context bucket of the previous code, zigzag symbol, 255 = escape
//   o1_normalize      :410-477   per-context normalization to 2^13
//   encode_o1tans     :582-751   S segments x K reverse-encoded interleaved chunks
//   encode_o1_ovf     :483-575   escape side stream (gamma + FSE, or raw int16)
//   decode            :984-1070, decode_o1tans :753-843
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <stdexcept>
#include <type_traits>
#include <vector>

#include "assemble.cuh"
#include "entropy.cuh"
#include "entropy_rules.cuh"
#include "fse.cuh"
#include "scan.cuh"

namespace fb2 {
namespace {

constexpr int FBLK = 1 << 16;
constexpr int O1_NCTX = 15;
constexpr int O1_PB = 13;
constexpr int O1_M = 1 << O1_PB;
constexpr int O1_NSYM = 256;
constexpr int kMaxK = 16;

__host__ __device__ __forceinline__ int o1_ctx(int code) {
    // magnitude buckets 1,2,3,4 | 5-7 | 8-11 | >= 12, doubled for the sign (RleFseEncoder.hpp:354-384)
    const int sgn = code < 0;
    const int a = sgn ? -code : code;
    const int m = min(a - 1, 3 + (a > 4) + (a > 7) + (a > 11));
    return a == 0 ? 0 : 1 + m * 2 + sgn;
}

__host__ __device__ __forceinline__ int o1_sym(int code) {
    const uint32_t zz = ((uint32_t)code << 1) ^ (uint32_t)(code >> 31);
    return zz < (uint32_t)(O1_NSYM - 1) ? (int)zz : O1_NSYM - 1;
}

__host__ __device__ __forceinline__ int unzz(uint32_t z) { return (int)((z >> 1) ^ (~(z & 1) + 1)); }

__host__ __device__ __forceinline__ uint32_t zigzag(int v) { return ((uint32_t)v << 1) ^ (uint32_t)(v >> 31); }

// ------------------------------------------------------------------ FSE class blocks
struct BlockJob {
    unsigned long long src;   // offset into the class array
    unsigned n;               // symbols
    unsigned flag;            // decode side: 0 raw, 1 FSE, 2 RLE
    unsigned long long in;    // decode side: offset of the payload (after flag / length)
    unsigned long long inlen; // decode side: payload length
    unsigned ck = 0xFFFFFFFFu; // decode side: first checkpoint of the block (none: all ones)
    unsigned pad = 0;
};

constexpr size_t kBlockSlot = FBLK + 64;

// FSE_compress on the device: header, tables and the 2-state reverse coding of one 64 Ki block
// (zfse/fse_compress.c FSE_compress_wksp).  The two state chains are interleaved and the symbol
// loads are issued ahead of the dependent table lookups.
// Decode checkpoint of an FSE block (two interleaved states): the decoder's bit position and both
// states just before it decodes symbol q * part (q >= 1).  Recorded by the encoder, stored in the
// stream's checkpoint frame, so that one block decodes as independent parts.
struct FseCkpt {
    uint32_t bitpos;
    uint16_t s0, s1;
};

// Decode checkpoint of a tANS chain: before the decoder decodes index lo + q * part (q >= 1), its
// bit position in the chain's stream, its state, the context (of the previous code) and the number
// of escapes the chain has consumed.  Recorded by the encoder into the stream's checkpoint frame.
struct O1Ckpt {
    uint32_t bitpos;
    uint32_t esc;
    uint16_t state;
    uint16_t ctx;
};

// Checkpoints of an n-symbol FSE block: one before every symbol q * part <= n - 3, q >= 1 (the
// last two symbols only initialise the encoder states).
__host__ __device__ __forceinline__ uint32_t fse_ckpt_count(uint32_t n, uint32_t part) {
    return n >= 3 ? (n - 3) / part : 0;
}

// FSE class block encoder (zfse/fse_compress.c FSE_compress), one group of 128 threads per 64
// Ki-symbol block (eight groups per CTA, below), the largest blocks first.  The group counts the
// block; its thread 0 normalizes and writes the table header; the group builds the coding tables
// in shared memory (the state table with warp match ranks, the symbol transforms per symbol, the
// step rows); two lanes of one warp then code the two state chains (symbols n-3 .. 0, each coded by
// the state of its index parity) side by side, recording every state with the bits that led to it;
// the group then packs in parallel: warps sum the bits of units of positions, a scan gives every
// unit its bit position, and the warps write the units (words shared with a neighbour merged with
// atomicOr); thread 0 appends the two final states and the end mark.  (Parts coded from guessed states
// do not meet the exact ones within a block of these skewed class streams.)  Writes the complete fse_enc record
// ([1][u32 len][data] | [0][raw] | [2][sym]) to the block's slot; the record flag goes into bits
// 56-63 of `sizes`.  `recs` is scratch of kFseRecWords words per block (the 16-bit step records of
// both chains).
constexpr unsigned kFseMaxLog = 11;               // the block coder's table log never exceeds 11
// Step rows: for every symbol, the next state and the emitted bits by state >> b, where b is the
// smaller of the symbol's two bit counts (the states from which it emits b + 1 start at a multiple
// of 2^(b + 1)).  A row has at most twice the symbol's cells, so all rows together fit 2 L entries.
// (A row of all L states a symbol saves the shift, but takes 40 KB for ten symbols, so that only four
// blocks fitted an SM: 758 blocks in two waves, 2.23 ms, now 1.05.)
constexpr unsigned kFseRows = 2u << kFseMaxLog;
// A block alone on its SM has room for a row of all L states a symbol instead, where its symbols are few enough: 32-bit
// cells, the next state times 4, which with the next symbol's row is the next cell's address, and its record.  A
// step then waits for one addition and one load: a full block's walk takes 520 us, with step rows 650 to 720.
constexpr unsigned kWideBytes = 24u << (kFseMaxLog + 2);
// Records per chain: every state (times 16, plus the bits emitted on the way to it), the last one too.
constexpr unsigned kFseChainRec = FBLK / 2 + 32;
constexpr unsigned kFseRecWords = kFseChainRec;  // both chains, 2 records per word
static_assert(kFseChainRec % 8 == 0, "records are moved as 16-byte vectors");
constexpr unsigned kFseBatch = 256;              // steps of a chain staged at a time, eight a lane and chain
constexpr unsigned kPackUnit = 512;              // emission positions a warp packs at a time, 16 a lane
constexpr unsigned kPackWords = (kPackUnit * kFseMaxLog + 31) / 32 + 1;
// A CTA codes G blocks side by side, one group of kFseGroupThreads threads each, with its own
// shared memory and its own named barrier.  G = 1, on an SM of its own (wide rows above), where the blocks and the
// chain encoder's CTAs together fit the SMs, or where few blocks outlast the chain encoder; G = kFseGroups
// otherwise: the CTA fills an SM (registers), so the blocks sit on an eighth as many SMs as one CTA per block would
// spread over, and the chain encoder launched beside them keeps the other SMs.
constexpr unsigned kFseGroups = 8, kFseGroupThreads = 128, kFseGroupWarps = kFseGroupThreads / 32;
constexpr unsigned kCountCopies = 8;  // histograms of the count, interleaved
struct FseGroupSmem {
    union {
        uint16_t row[kFseRows];
        uint32_t copies[256 * kCountCopies];         // while the block is counted
        uint32_t pack[kFseGroupWarps][kPackWords];   // after the walk: a warp's unit in words
    };
    union {
        uint4 ring[2][kFseBatch / 4 + 1];            // the chains' steps of a batch
        uint32_t unit[FBLK / kPackUnit];             // after the walk: bits before a unit
    };
    uint32_t count[256];
    uint32_t cumul[257];
    uint32_t scan[257];
    uint32_t step[256];  // of a symbol: its row's shared-memory address << 5 | b + 4
    fse::SymTT sym_tt[256];
    int16_t norm[256];
    uint16_t state_table[1 << kFseMaxLog];
    uint8_t sym[1 << kFseMaxLog];
    int mode;
    unsigned tl, hdr, fin[2], maxsv, high, bits, wide;
    uint32_t sh[32];
    unsigned long long tend;  // traced calls: when the walk ended
};
static_assert(sizeof(uint32_t) * 256 * kCountCopies <= sizeof(uint16_t) * kFseRows &&
              sizeof(uint32_t) * kFseGroupWarps * kPackWords <= sizeof(uint16_t) * kFseRows, "in the rows' space");

// A group's barrier.  bar.sync counts whole warps, so the warp is made convergent first (after
// code where some lanes ran on alone, such as the two chain lanes).
__device__ __forceinline__ void group_sync(unsigned bar) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kFseGroupThreads) : "memory");
}

// Phase times of a block (traced calls only): the global timer at the block's start and after its
// count, plan, tables, chain walk, pack and output, kFsePhases words per block.
constexpr int kFsePhases = 8;
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)::"memory");
    return t;
}
__device__ __forceinline__ void fse_phase(unsigned long long *phase, unsigned slot, int k) {
    if (phase) phase[(size_t)slot * kFsePhases + k] = global_ns();
}

// Exclusive scan over a group's threads (tid = index in the group), total of the group in `total`.
__device__ __forceinline__ uint32_t group_excl_scan(uint32_t v, uint32_t *sh, uint32_t &total, unsigned tid,
                                                    unsigned bar) {
    constexpr unsigned nw = kFseGroupThreads / 32;
    const unsigned lane = tid & 31u, wid = tid >> 5;
    const uint32_t incl = warp_incl_scan(v);
    if (lane == 31) sh[wid] = incl;
    group_sync(bar);
    if (wid == 0) {
        uint32_t x = lane < nw ? sh[lane] : 0u;
        x = warp_incl_scan(x);
        sh[lane] = x;
    }
    group_sync(bar);
    const uint32_t before = wid ? sh[wid - 1] : 0u;
    total = sh[nw - 1];
    group_sync(bar);
    return before + incl - v;
}

template <unsigned G>
__global__ void __launch_bounds__(G * kFseGroupThreads, kFseGroups / G)
    k_fse_encode_blocks(const uint8_t *__restrict__ cls, const BlockJob *__restrict__ jobs, unsigned njobs,
                        uint8_t *__restrict__ slots, unsigned long long *__restrict__ sizes,
                        uint8_t *__restrict__ scratch, uint32_t part, FseCkpt *__restrict__ cks,
                        uint32_t *recs, const uint32_t *__restrict__ order,
                        unsigned long long *__restrict__ phase) {
    extern __shared__ uint4 s_groups[];  // G groups' FseGroupSmem
    const unsigned grp = threadIdx.x / kFseGroupThreads, tid = threadIdx.x % kFseGroupThreads;
    const unsigned lane = tid & 31u, wid = tid >> 5;
    const unsigned slot = blockIdx.x * G + grp;
    if (slot >= njobs) return;  // the other groups synchronise on barriers of their own
    const unsigned bar = 1 + grp;  // named barrier of this group (0 is the CTA's)
    uint32_t *const wide_rows = reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(s_groups) + sizeof(FseGroupSmem));
    FseGroupSmem &w = reinterpret_cast<FseGroupSmem *>(s_groups)[grp];
    const unsigned b = order[slot];  // the largest blocks first
    if (tid == 0) fse_phase(phase, slot, 0);
    const BlockJob jb = jobs[b];
    const uint8_t *src = cls + jb.src;
    uint8_t *out = slots + (size_t)b * kBlockSlot;
    uint32_t *bw = reinterpret_cast<uint32_t *>(scratch + (size_t)b * kBlockSlot);
    uint16_t *rec = reinterpret_cast<uint16_t *>(recs + (size_t)b * kFseRecWords);
    FseCkpt *ck = cks ? cks + (size_t)b * (FBLK / part) : nullptr;
    const unsigned n = jb.n;
    // the block in aligned 16-byte words (the pool's allocations are 16-byte aligned with slack behind them)
    const unsigned lead = (unsigned)(jb.src & 15u);
    const uint4 *g4 = reinterpret_cast<const uint4 *>(src - lead);
    for (unsigned s = tid; s < 256 * kCountCopies; s += kFseGroupThreads) w.copies[s] = 0;
    group_sync(bar);
    // Count the symbols: runs of equal symbols within a word are added with one atomic, and neighbouring
    // lanes add to copies of their own, in banks of their own (a few symbols dominate the class streams).
    {
        const unsigned nw = (lead + n + 15) / 16;
        uint32_t *h = w.copies + (lane % kCountCopies);
        uint4 v = tid < nw ? g4[tid] : make_uint4(0, 0, 0, 0);
        for (unsigned wi = tid; wi < nw; wi += kFseGroupThreads) {
            const uint4 c = v;
            if (wi + kFseGroupThreads < nw) v = g4[wi + kFseGroupThreads];
            // the word's bytes [t0, t1) belong to the block
            const unsigned t0 = wi ? 0u : lead, t1 = min(16u, lead + n - wi * 16);
            unsigned cur = 0, run = 0;
#pragma unroll
            for (unsigned t = 0; t < 16; t++) {
                if (t < t0 || t >= t1) continue;
                const uint32_t q = t < 4 ? c.x : t < 8 ? c.y : t < 12 ? c.z : c.w;
                const unsigned sy = (q >> ((t & 3) * 8)) & 0xFFu;
                if (run && sy != cur) {
                    atomicAdd(h + cur * kCountCopies, run);
                    run = 0;
                }
                cur = sy;
                run++;
            }
            atomicAdd(h + cur * kCountCopies, run);
        }
    }
    group_sync(bar);
    for (unsigned s = tid; s < 256; s += kFseGroupThreads) {
        uint32_t v = 0;
#pragma unroll
        for (unsigned c = 0; c < kCountCopies; c++) v += w.copies[s * kCountCopies + c];
        w.count[s] = v;
    }
    group_sync(bar);
    if (tid == 0) fse_phase(phase, slot, 1);
    if (tid == 0) {
        int mode = 0;
        unsigned tl = 0, hdr = 0, maxSV = 255;
        {
            const int plan = fse::plan_block(w.count, n, kFseMaxLog, w.norm, &maxSV, &tl);
            if (plan == 1) {
                mode = 1;
            } else if (plan == 2) {
                if (kBlockSlot - 5 >= fse::ncount_bound(maxSV, tl) + 16) {
                    hdr = (unsigned)fse::write_ncount(out + 5, w.norm, maxSV, tl);
                    // the spread (zfse FSE_buildCTable): the low-probability (-1) symbols take the
                    // top cells; the cells of the others, in symbol order, go to the kept positions
                    // (j * step) & mask <= high in order of j (spread in parallel below; the
                    // sequential walk ends at position 0 exactly when the cells fill the kept
                    // positions)
                    uint32_t c = 0, high = (1u << tl) - 1;
                    for (unsigned s2 = 0; s2 <= maxSV; s2++) {
                        w.scan[s2] = c;
                        if (w.norm[s2] > 0) c += (uint32_t)w.norm[s2];
                        else if (w.norm[s2] == -1) w.sym[high--] = (uint8_t)s2;
                    }
                    w.scan[maxSV + 1] = c;
                    w.high = high;
                    if (hdr && c == high + 1) {
                        mode = 2;
                        w.cumul[0] = 0;
                        for (unsigned u = 1; u <= maxSV + 1; u++)
                            w.cumul[u] = w.cumul[u - 1] + (w.norm[u - 1] == -1 ? 1u : (uint32_t)w.norm[u - 1]);
                    }
                }
            }
        }
        unsigned present = 0;
        for (unsigned s2 = 0; s2 <= maxSV && mode == 2; s2++) present += w.norm[s2] != 0;
        w.wide = G == 1 && ((size_t)present << (tl + 2)) <= kWideBytes;
        w.mode = mode;
        w.tl = tl;
        w.hdr = hdr;
        w.maxsv = maxSV;
    }
    group_sync(bar);
    if (tid == 0) fse_phase(phase, slot, 2);
    if (w.mode == 2) {
        const unsigned tl = w.tl, L = 1u << tl, maxSV = w.maxsv;
        {
            // parallel spread: thread t ranks the kept positions of j in [t * per, (t + 1) * per)
            const uint32_t step = fse::table_step(L), mask = L - 1, high = w.high;
            const unsigned per = (L + kFseGroupThreads - 1) / kFseGroupThreads;
            const unsigned j0 = min(L, tid * per), j1 = min(L, j0 + per);
            uint32_t cnt = 0;
            for (unsigned j = j0; j < j1; j++) cnt += ((j * step) & mask) <= high;
            uint32_t tot;
            uint32_t kc = group_excl_scan(cnt, w.sh, tot, tid, bar);
            unsigned sy = 0;  // the symbol of cell kc: the last one whose first cell is <= kc
            for (unsigned lo = 0, hi = maxSV + 1; hi - lo > 1;) {
                const unsigned mid = (lo + hi) >> 1;
                if (w.scan[mid] <= kc) lo = mid;
                else hi = mid;
                sy = lo;
            }
            for (unsigned j = j0; j < j1; j++) {
                const uint32_t pos = (j * step) & mask;
                if (pos > high) continue;
                while (w.scan[sy + 1] <= kc) sy++;
                w.sym[pos] = (uint8_t)sy;
                kc++;
            }
            group_sync(bar);
        }
        // state table: the cells of every symbol in increasing order (match ranks within a warp)
        if (wid == 0) {
            for (unsigned u0 = 0; u0 < L; u0 += 32) {
                const unsigned u = u0 + lane;
                const unsigned sy = u < L ? w.sym[u] : 256u + lane;
                const unsigned peers = __match_any_sync(0xffffffffu, sy);
                const unsigned rank = __popc(peers & ((1u << lane) - 1u));
                if (u < L) w.state_table[w.cumul[sy] + rank] = (uint16_t)(L + u);
                __syncwarp();
                if (u < L && rank == (unsigned)__popc(peers) - 1u) w.cumul[sy] += rank + 1;
                __syncwarp();
            }
        }
        for (unsigned sy = tid; sy <= maxSV; sy += kFseGroupThreads) {
            const int nn = w.norm[sy];
            uint32_t total = 0, rows = 0;  // cells of the symbols before sy, and how many are present
            for (unsigned s2 = 0; s2 < sy; s2++) {
                total += w.norm[s2] == -1 ? 1u : (uint32_t)max(0, (int)w.norm[s2]);
                rows += w.norm[s2] != 0;
            }
            uint32_t low = tl;  // the smaller of the symbol's bit counts
            if (nn == 0) {
                w.sym_tt[sy].deltaNbBits = ((tl + 1) << 16) - L;
                w.sym_tt[sy].deltaFindState = 0;
            } else if (nn == -1 || nn == 1) {
                w.sym_tt[sy].deltaNbBits = (tl << 16) - L;
                w.sym_tt[sy].deltaFindState = (int32_t)total - 1;
            } else {
                const uint32_t maxBitsOut = tl - fse::highbit32((uint32_t)(nn - 1));
                const uint32_t minStatePlus = (uint32_t)nn << maxBitsOut;
                w.sym_tt[sy].deltaNbBits = (maxBitsOut << 16) - minStatePlus;
                w.sym_tt[sy].deltaFindState = (int32_t)total - nn;
                low = maxBitsOut - 1;
            }
            // the row starts at twice the cells before it (a row of L >> low entries has at most twice its cells)
            w.step[sy] = w.wide ? (uint32_t)__cvta_generic_to_shared(wide_rows) + (rows << (tl + 2))
                                : (((uint32_t)__cvta_generic_to_shared(w.row) + 4 * min(total, L - 1)) << 5) | (low + 4);
        }
        group_sync(bar);
        for (unsigned sy = 0, rows = 0; sy <= maxSV; sy++) {
            if (w.norm[sy] == 0) continue;
            if (w.wide) {
                const fse::SymTT t = w.sym_tt[sy];
                for (unsigned c = tid; c < L; c += kFseGroupThreads) {
                    const uint32_t nb = (L + c + t.deltaNbBits) >> 16;
                    const uint32_t x = w.state_table[(int32_t)((L + c) >> nb) + t.deltaFindState] - L;
                    wide_rows[(rows << tl) + c] = (x << 2) | (x << 4 | nb) << 16;
                }
                rows++;
                continue;
            }
            const unsigned low = (w.step[sy] & 31u) - 4;
            uint16_t *row = w.row + ((w.step[sy] >> 5) - (uint32_t)__cvta_generic_to_shared(w.row)) / 2;
            const fse::SymTT t = w.sym_tt[sy];
            for (unsigned c = tid; c < L >> low; c += kFseGroupThreads) {
                const uint32_t x = L + (c << low), nb = (x + t.deltaNbBits) >> 16;
                row[c] = (uint16_t)((w.state_table[(int32_t)(x >> nb) + t.deltaFindState] - L) << 4 | nb);
            }
        }
        group_sync(bar);
        if (tid == 0) fse_phase(phase, slot, 3);
        const unsigned ns = n - 2;  // emission position e codes symbol n - 3 - e, even positions by chain 0
        // The chains run on a warp that puts a CTA's eight two on each SM sub-partition (warp w of a CTA
        // issues from sub-partition w mod 4).
        if (wid == (grp & 3u)) {
            // Lane c < 2 codes chain c: the symbols n - 3 - c, n - 5 - c, .., starting from the state that
            // symbol n - 1 - c initialised.  A record is the state minus L, times 16, plus the bits that the
            // step to it emitted; a step shifts it down, adds the symbol's row and loads the next record.  What
            // a step needs of its symbol is laid out by the whole warp for kFseBatch steps at a time, its
            // symbols loaded a batch ahead, so that little but the chain itself is left to the two lanes: a
            // step waits for two additions and one load (22.5 ns; with the symbols unpacked by the chain's own
            // lane, 26).
            const unsigned m = lane < 2 ? (ns + 1 - lane) / 2 : 0;  // steps
            uint16_t *rk = rec + (lane & 1u) * kFseChainRec;
            uint32_t e = 0;
            if (lane < 2) {
                const fse::SymTT t = w.sym_tt[src[n - 1 - lane]];
                const uint32_t nb = (t.deltaNbBits + (1u << 15)) >> 16;
                const uint32_t u = (nb << 16) - t.deltaNbBits;
                e = (w.state_table[(int32_t)(u >> nb) + t.deltaFindState] - L) << 4;
            }
            // the two words that hold positions [e0, e0 + 16), the last of them first
            auto load = [&](unsigned e0, uint4 &x0, uint4 &x1) {
                x0 = x1 = make_uint4(0, 0, 0, 0);
                if (e0 >= ns) return;
                const unsigned w1 = (lead + n - 3 - e0) >> 4;
                x1 = __ldg(g4 + w1);
                if (w1) x0 = __ldg(g4 + w1 - 1);
            };
            const unsigned rot = ((lead + n - 3) & 15u) + 1, wrot = rot >> 2, brot = (rot & 3u) * 8;
            uint4 x0, x1;
            load(16 * lane, x0, x1);
            auto walk = [&](auto wide_tag) {
                constexpr bool WIDE = decltype(wide_tag)::value;
                uint32_t f = e >> 2;  // four times the state minus L
                for (unsigned j0 = 0; 2 * j0 < ns; j0 += kFseBatch) {
                    {
                        uint32_t x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w}, o[16];
                        if (wrot & 1u) {
#pragma unroll
                            for (int q = 0; q < 7; q++) x[q] = x[q + 1];
                        }
                        if (wrot & 2u) {
#pragma unroll
                            for (int q = 0; q < 6; q++) x[q] = x[q + 2];
                        }
                        if (wrot & 4u) {
#pragma unroll
                            for (int q = 0; q < 4; q++) x[q] = x[q + 4];
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) x[q] = __funnelshift_r(x[q], x[q + 1], brot);
#pragma unroll
                        for (int t = 0; t < 16; t++) o[t] = w.step[(x[(15 - t) >> 2] >> (8 * ((15 - t) & 3))) & 0xFFu];
#pragma unroll
                        for (int c = 0; c < 2; c++) {
                            w.ring[c][2 * lane] = make_uint4(o[c], o[c + 2], o[c + 4], o[c + 6]);
                            w.ring[c][2 * lane + 1] = make_uint4(o[c + 8], o[c + 10], o[c + 12], o[c + 14]);
                        }
                    }
                    load(2 * (j0 + kFseBatch) + 16 * lane, x0, x1);
                    __syncwarp();
                    if (lane < 2) {
                        auto step = [&f](uint32_t o, uint32_t e2) -> uint32_t {
                            uint16_t r;
                            if (WIDE) {
                                const uint32_t at = o + f;
                                uint16_t g;
                                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(g) : "r"(at));
                                asm volatile("ld.shared.u16 %0, [%1+2];" : "=h"(r) : "r"(at));
                                f = g;
                            } else {
                                const uint32_t at = (o >> 5) + 2 * __funnelshift_r(e2, 0u, o);
                                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(r) : "r"(at));
                            }
                            return r;
                        };
                        const uint4 *rg = w.ring[lane];
                        const unsigned steps = min(kFseBatch, m - min(m, j0)), ng = steps / 8;
                        uint4 a = rg[0], c = rg[1];
                        for (unsigned g = 0; g < ng; g++) {
                            const unsigned gn = (g + 1) % (kFseBatch / 8);
                            const uint4 an = rg[2 * gn], cn = rg[2 * gn + 1];
                            const uint32_t o[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
                            uint32_t r[8];
#pragma unroll
                            for (int t = 0; t < 8; t++) {
                                r[t] = e;
                                e = step(o[t], e);
                            }
                            *reinterpret_cast<uint4 *>(rk + j0 + 8 * g) =
                                make_uint4(r[0] | (r[1] << 16), r[2] | (r[3] << 16), r[4] | (r[5] << 16), r[6] | (r[7] << 16));
                            a = an;
                            c = cn;
                        }
                        const uint32_t *o = reinterpret_cast<const uint32_t *>(rg);
                        for (unsigned t = 8 * ng; t < steps; t++) {
                            rk[j0 + t] = (uint16_t)e;
                            e = step(o[t], e);
                        }
                    }
                    __syncwarp();  // the batch's steps are read
                }
            };
            if (G == 1 && w.wide) walk(std::true_type());
            else walk(std::false_type());
            if (lane < 2) {
                rk[m] = (uint16_t)e;
                w.fin[lane] = e >> 4;
            }
            if (lane == 0 && phase) w.tend = global_ns();
        } else {  // the bits' scratch starts at zero
            const unsigned long long most = (unsigned long long)ns * tl + 2 * tl + 1;
            constexpr unsigned kCap = (unsigned)(kBlockSlot / 4);
            const unsigned zw = (unsigned)((most + 31) / 32 + 1 < kCap ? (most + 31) / 32 + 1 : kCap);
            const unsigned t = tid - (wid > (grp & 3u) ? 32u : 0u);
            for (unsigned z = t; z < zw; z += kFseGroupThreads - 32) bw[z] = 0u;
        }
    }
    group_sync(bar);
    if (tid == 0 && phase) phase[(size_t)slot * kFsePhases + 4] = w.mode == 2 ? w.tend : global_ns();
    int mode = w.mode;
    size_t body = 0;
    if (mode == 2) {
        const unsigned tl = w.tl, ns = n - 2, nunits = (ns + kPackUnit - 1) / kPackUnit;
        constexpr unsigned kCap = (unsigned)(kBlockSlot / 4);
        // A lane takes 16 emission positions from 16 x on: eight records of each chain and the one after
        // them (a record's low bits are those that its step emitted, the count is in the next record).
        auto fetch = [&](unsigned x, uint4 &ra, uint4 &rb, uint32_t &na, uint32_t &nb) {
            ra = rb = make_uint4(0, 0, 0, 0);
            const bool in = 16 * x < ns;
            if (in) {
                ra = *reinterpret_cast<const uint4 *>(rec + 8 * x);
                rb = *reinterpret_cast<const uint4 *>(rec + kFseChainRec + 8 * x);
            }
            na = __shfl_down_sync(0xffffffffu, ra.x & 0xFFFFu, 1);
            nb = __shfl_down_sync(0xffffffffu, rb.x & 0xFFFFu, 1);
            if (in && (lane == 31 || 16 * x + 16 >= ns)) {
                na = rec[8 * x + 8];
                nb = rec[kFseChainRec + 8 * x + 8];
            }
        };
        auto rec_of = [](const uint4 &r, uint32_t after, unsigned j) -> uint32_t {
            const uint32_t q = j < 2 ? r.x : j < 4 ? r.y : j < 6 ? r.z : j < 8 ? r.w : after;
            return j & 1u ? q >> 16 : q & 0xFFFFu;
        };
        // the bits of a lane's positions
        auto bits_of = [&](unsigned x, const uint4 &ra, const uint4 &rb, uint32_t na, uint32_t nb) -> uint32_t {
            if (16 * x + 16 <= ns) {
                const uint32_t k = 0x000F000Fu;
                const uint32_t t = (ra.x & k) + (ra.y & k) + (ra.z & k) + (ra.w & k) + (rb.x & k) + (rb.y & k) + (rb.z & k) + (rb.w & k);
                return (t & 0xFFFFu) + (t >> 16) - (ra.x & 15u) - (rb.x & 15u) + (na & 15u) + (nb & 15u);
            }
            uint32_t t = 0;
#pragma unroll
            for (unsigned i = 0; i < 16; i++)
                if (16 * x + i < ns) t += (i & 1u ? rec_of(rb, nb, i / 2 + 1) : rec_of(ra, na, i / 2 + 1)) & 15u;
            return t;
        };
        for (unsigned u = wid; u < nunits; u += kFseGroupWarps) {
            uint4 ra, rb;
            uint32_t na, nb;
            fetch(32 * u + lane, ra, rb, na, nb);
            const uint32_t t = __reduce_add_sync(0xffffffffu, bits_of(32 * u + lane, ra, rb, na, nb));
            if (lane == 0) w.unit[u] = t;
        }
        group_sync(bar);
        if (wid == 0) {
            constexpr unsigned kPer = FBLK / kPackUnit / 32;
            uint32_t a[kPer], sum = 0;
#pragma unroll
            for (unsigned q = 0; q < kPer; q++) {
                a[q] = lane * kPer + q < nunits ? w.unit[lane * kPer + q] : 0u;
                sum += a[q];
            }
            const uint32_t incl = warp_incl_scan(sum);
            uint32_t run = incl - sum;
#pragma unroll
            for (unsigned q = 0; q < kPer; q++) {
                if (lane * kPer + q < nunits) w.unit[lane * kPer + q] = run;
                run += a[q];
            }
            if (lane == 31) w.bits = incl;
        }
        group_sync(bar);
        // The units' bits: merged into the warp's words, which leave as whole-word stores (a unit's two edge
        // words, shared with its neighbours, by atomicOr into the zeroed scratch).  Words past the block's slot
        // are dropped: such a block is stored raw.
        uint32_t *pw = w.pack[wid];
        for (unsigned u = wid; u < nunits; u += kFseGroupWarps) {
            const unsigned x = 32 * u + lane;
            uint4 ra, rb;
            uint32_t na, nb;
            fetch(x, ra, rb, na, nb);
            const uint32_t mine = bits_of(x, ra, rb, na, nb), incl = warp_incl_scan(mine);
            const uint32_t u0 = w.unit[u], b0 = u0 & 31u;
            const uint32_t nw = (b0 + __shfl_sync(0xffffffffu, incl, 31) + 31) >> 5;
            for (unsigned z = lane; z < nw; z += 32) pw[z] = 0;
            __syncwarp();
            uint32_t p = b0 + incl - mine, fill = p & 31u;
            uint32_t *o = pw + (p >> 5);
            unsigned long long acc = 0;
            // whether one of these positions codes a symbol with a checkpoint before it
            const bool marked = ck && 16 * x < ns && (part < 16 || ((n - 3 - 16 * x) & (part - 1)) < 16);
#pragma unroll
            for (unsigned i = 0; i < 16; i++) {
                if (16 * x + i >= ns) continue;
                const uint32_t v = (i & 1u ? rec_of(rb, nb, i / 2) : rec_of(ra, na, i / 2)) >> 4;
                const uint32_t k = (i & 1u ? rec_of(rb, nb, i / 2 + 1) : rec_of(ra, na, i / 2 + 1)) & 15u;
                acc |= (unsigned long long)(v & ((1u << k) - 1u)) << fill;
                fill += k;
                p += k;
                if (fill >= 32) {
                    atomicOr(o++, (uint32_t)acc);
                    acc >>= 32;
                    fill -= 32;
                }
                if (marked) {
                    const unsigned e = 16 * x + i, s = n - 3 - e;
                    // the decoder's states before symbol s: those after symbols s and s + 1, which are the
                    // states before the chains' next symbols
                    if (s > 0 && (s & (part - 1)) == 0)
                        ck[s / part - 1] = FseCkpt{u0 - b0 + p, (uint16_t)(rec[(e & 1u) * kFseChainRec + e / 2 + 1] >> 4),
                                                   (uint16_t)(rec[((e + 1) & 1u) * kFseChainRec + (e + 1) / 2] >> 4)};
                }
            }
            if ((uint32_t)acc) atomicOr(o, (uint32_t)acc);
            __syncwarp();
            for (unsigned z = lane; z < nw; z += 32) {
                const unsigned gw = (u0 >> 5) + z;
                if (gw >= kCap) continue;
                if (z == 0 || z == nw - 1) atomicOr(bw + gw, pw[z]);
                else bw[gw] = pw[z];
            }
            __syncwarp();
        }
        const uint32_t sym_bits = w.bits;  // bits of all symbols
        const uint32_t total = sym_bits + 2 * tl + 1;
        body = (total + 7) / 8;
        if (body + 8 > kBlockSlot - 5 - w.hdr || w.hdr + body >= n - 1) mode = 0;  // not worth coding: raw
        group_sync(bar);
        if (mode == 2 && tid == 0) {  // final states (odd, then even) and the end mark
            uint32_t p2 = sym_bits;
            auto put = [&](uint32_t v, uint32_t nb) {
                for (uint32_t b = 0; b < nb; b++, p2++)
                    if ((v >> b) & 1u) atomicOr(bw + (p2 >> 5), 1u << (p2 & 31u));
            };
            put(w.fin[n & 1u], tl);  // chain 0 codes the symbols of n - 1's parity
            put(w.fin[(n & 1u) ^ 1u], tl);
            put(1u, 1u);
        }
        group_sync(bar);
    }
    if (tid == 0) fse_phase(phase, slot, 5);
    if (mode == 0) {  // raw
        if (tid == 0) out[0] = 0;
        for (unsigned i = tid; i < n; i += kFseGroupThreads) out[1 + i] = src[i];
        if (tid == 0) sizes[b] = 1 + n;  // flag 0
    } else if (mode == 1) {  // a single repeated symbol
        if (tid == 0) {
            out[0] = 2;
            out[1] = src[0];
            sizes[b] = 2 | (2ULL << 56);
        }
    } else {
        const size_t r = w.hdr + body;
        uint8_t *d = out + 5 + w.hdr;
        const uint8_t *bb = reinterpret_cast<const uint8_t *>(bw);
        for (size_t i = tid; i < body; i += kFseGroupThreads) d[i] = bb[i];
        if (tid == 0) {
            out[0] = 1;
            const uint32_t rr = (uint32_t)r;
            out[1] = (uint8_t)rr;
            out[2] = (uint8_t)(rr >> 8);
            out[3] = (uint8_t)(rr >> 16);
            out[4] = (uint8_t)(rr >> 24);
            sizes[b] = (5 + r) | (1ULL << 56);
        }
    }
    if (phase) {
        group_sync(bar);
        if (tid == 0) fse_phase(phase, slot, 6);
    }
}

// Backward reader of a bit stream: hi and lo are the 64 bits below `pos`, aligned in registers from the 8-byte
// pieces q and q - 1 (q: the one that holds bit pos), with two more loaded behind them, so that neither a lane's
// own loads nor those that other lanes of its warp just asked for are waited on.  align() after at most 52
// bits taken.  Bits are counted from `base`, the stream's first byte rounded down to 8.
struct BackWindow {
    const uint2 *base;
    int32_t pos, q, qmin;
    uint2 a, b, c, d;
    uint32_t hi, lo;
    __device__ __forceinline__ uint2 piece(int32_t p) const { return p >= qmin ? __ldg(base + p) : make_uint2(0, 0); }
    // Starts below bit `bit` of the stream at sb; `front`: readable bytes in front of sb (pieces further in
    // front are not loaded: a damaged stream alone gets there).  Returns the stream's first bit.
    __device__ __forceinline__ int32_t init(const uint8_t *sb, unsigned long long front, int32_t bit) {
        const int32_t bit0 = (int32_t)(reinterpret_cast<uintptr_t>(sb) & 7) * 8;
        base = reinterpret_cast<const uint2 *>(reinterpret_cast<uintptr_t>(sb) & ~uintptr_t(7));
        qmin = -(int32_t)min((unsigned long long)(1 << 20), front >> 3);
        pos = bit0 + bit;
        q = pos >> 6;
        a = piece(q);
        b = piece(q - 1);
        c = piece(q - 2);
        d = piece(q - 3);
        align();
        return bit0;
    }
    __device__ __forceinline__ void align() {
        if (pos >> 6 != q) {  // at most one piece on
            q--;
            a = b;
            b = c;
            c = d;
            d = piece(q - 3);
        }
        const bool odd = pos & 32;
        const uint32_t x = odd ? a.y : a.x, y = odd ? a.x : b.y, z = odd ? b.y : b.x;
        hi = __funnelshift_r(y, x, pos);
        lo = __funnelshift_r(z, y, pos);
    }
    __device__ __forceinline__ void skip(uint32_t nb) {
        hi = __funnelshift_l(lo, hi, nb);
        lo <<= nb;
        pos -= (int32_t)nb;
    }
    __device__ __forceinline__ uint32_t take(uint32_t nb) {  // nb < 32
        const uint32_t v = __funnelshift_l(hi, 0u, nb);
        skip(nb);
        return v;
    }
};

// One CTA of kFseDecThreads per 64 Ki block: thread 0 reads the table header, the first warp
// builds the decode table in shared memory (zfse/fse_decompress.c FSE_buildDTable), then the block
// decodes either as one sequence (thread 0, two interleaved states,
// FSE_decompress_usingDTable_generic) or, when the stream carries checkpoints for it, as
// independent parts of `part` symbols, one per thread, each starting from its checkpoint and
// verified against the next one (a mismatch sets err[1] and the caller decodes again without
// checkpoints).
constexpr int kFseDecThreads = 64;  // parts of a block decode one per thread
constexpr unsigned kPartPad = 4;     // bytes between the parts' regions of the decoded block (>= 2:
                                     // the last part may hold two symbols past `part`)
// Dynamic shared memory: the decoded block (FBLK symbols plus kPartPad per part), which the table's spread
// uses first, then the decode table: 76 KB at parts of 1024 symbols, three blocks an SM.  (With room for the
// largest table two fitted: 310 against 217 us for 758 blocks.)  A table of a log above kFseDecLog, which no
// encoder here writes, takes the decoded block's place behind the spread, and its symbols go straight out.
constexpr unsigned kFseDecLog = 11;
static_assert((1 << fse::kMaxTableLog) * (1 + sizeof(fse::DEntry)) <= FBLK, "spread and largest table fit the block's place");
inline size_t fse_dec_smem(uint32_t part) { return FBLK + (FBLK / part) * kPartPad + (sizeof(fse::DEntry) << kFseDecLog); }
__global__ void __launch_bounds__(kFseDecThreads) k_fse_decode_blocks(const uint8_t *__restrict__ in,
                                                         const BlockJob *__restrict__ jobs,
                                                         uint8_t *__restrict__ cls, int *__restrict__ err,
                                                         uint32_t part, const FseCkpt *__restrict__ cks) {
    __shared__ int16_t s_norm[256];
    __shared__ uint32_t s_scan[257], s_next[256];
    __shared__ unsigned tl_sh, hdr_sh, maxsv_sh, high_sh;
    extern __shared__ uint4 s_out4[];
    uint8_t *s_out = reinterpret_cast<uint8_t *>(s_out4), *sym = s_out;
    const BlockJob jb = jobs[blockIdx.x];
    uint8_t *dst = cls + jb.src;
    const uint8_t *p = in + jb.in;
    if (jb.flag == 0) {
        for (unsigned i = threadIdx.x; i < jb.n; i += blockDim.x) dst[i] = p[i];
        return;
    }
    if (jb.flag == 2) {
        const uint8_t v = p[0];
        for (unsigned i = threadIdx.x; i < jb.n; i += blockDim.x) dst[i] = v;
        return;
    }
    const size_t size = (size_t)jb.inlen;
    // The decode table (zfse FSE_buildDTable), built by the warp: lane 0 reads the header and lays
    // the low-probability (-1) symbols on the top cells; the lanes spread the other cells (cell k
    // in symbol order goes to the k-th position (j * step) & mask <= high in order of j) and then
    // number every symbol's cells in cell order (warp match ranks, 32 cells at a time).
    if (threadIdx.x == 0) {
        unsigned maxSV = 255, tl = 0;
        const size_t hdr = fse::read_ncount(s_norm, &maxSV, &tl, p, size);
        bool ok = hdr != 0 && hdr < size && tl <= (unsigned)fse::kMaxTableLog;
        if (ok) {
            uint32_t c = 0, high = (1u << tl) - 1;
            for (unsigned s2 = 0; s2 <= maxSV; s2++) {
                s_scan[s2] = c;
                const int nn = s_norm[s2];
                if (nn > 0) c += (uint32_t)nn;
                else if (nn == -1) sym[high--] = (uint8_t)s2;
                s_next[s2] = nn == -1 ? 1u : (uint32_t)max(nn, 0);
            }
            s_scan[maxSV + 1] = c;
            ok = c == high + 1;  // the sequential spread ends at position 0 exactly then
            high_sh = high;
        }
        tl_sh = ok ? tl : 0xFFFFFFFFu;
        hdr_sh = (unsigned)hdr;
        maxsv_sh = maxSV;
        if (!ok) atomicExch(err, 1);
    }
    __syncthreads();
    const unsigned tl = tl_sh;
    if (tl == 0xFFFFFFFFu) return;
    const bool big = tl > kFseDecLog;
    fse::DEntry *const dt = reinterpret_cast<fse::DEntry *>(
        s_out + (big ? 1u << fse::kMaxTableLog : FBLK + (FBLK / part) * kPartPad));
    if (threadIdx.x < 32) {  // the table, by the first warp
        const unsigned lane = threadIdx.x, L = 1u << tl, maxSV = maxsv_sh;
        const uint32_t step = fse::table_step(L), mask = L - 1, high = high_sh;
        const unsigned per = (L + 31) / 32, j0 = min(L, lane * per), j1 = min(L, j0 + per);
        uint32_t cnt = 0;
        for (unsigned j = j0; j < j1; j++) cnt += ((j * step) & mask) <= high;
        uint32_t kc = cnt;  // exclusive warp scan
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, kc, o);
            if (lane >= (unsigned)o) kc += t;
        }
        kc -= cnt;
        unsigned sy = 0;  // the symbol of cell kc: the last one whose first cell is <= kc
        for (unsigned lo = 0, hi = maxSV + 1; hi - lo > 1;) {
            const unsigned mid = (lo + hi) >> 1;
            if (s_scan[mid] <= kc) lo = mid;
            else hi = mid;
            sy = lo;
        }
        for (unsigned j = j0; j < j1; j++) {
            const uint32_t pos = (j * step) & mask;
            if (pos > high) continue;
            while (s_scan[sy + 1] <= kc) sy++;
            sym[pos] = (uint8_t)sy;
            kc++;
        }
        __syncwarp();
        for (unsigned u0 = 0; u0 < L; u0 += 32) {
            const unsigned u = u0 + lane;
            const unsigned sv = u < L ? sym[u] : 256u + lane;
            const unsigned peers = __match_any_sync(0xffffffffu, sv);
            const unsigned rank = __popc(peers & ((1u << lane) - 1u));
            if (u < L) {
                const uint32_t ns = s_next[sv] + rank;
                const uint32_t nb = tl - fse::highbit32(ns);
                fse::DEntry e;
                e.symbol = (uint8_t)sv;
                e.nbBits = (uint8_t)nb;
                e.newState = (uint16_t)((ns << nb) - L);
                dt[u] = e;
            }
            __syncwarp();
            if (u < L && rank == (unsigned)__popc(peers) - 1u) s_next[sv] += rank + 1;
            __syncwarp();
        }
    }
    __syncthreads();
    const uint8_t *sp = p + hdr_sh;
    const uint32_t ssz = (uint32_t)(size - hdr_sh);
    const unsigned n = jb.n;
    const unsigned nparts = jb.ck == 0xFFFFFFFFu ? 1u : 1u + fse_ckpt_count(n, part);
    auto decode = [&](unsigned q, auto big_tag) {
        constexpr bool BIG = decltype(big_tag)::value;
        BackWindow br;
        uint32_t s0, s1;
        int32_t bit0;
        const unsigned start = q * (nparts > 1 ? part : 0u);
        const unsigned end = q + 1 < nparts ? start + part : n;
        const unsigned long long front = jb.in + hdr_sh;
        if (q == 0) {
            const uint8_t last = ssz ? sp[ssz - 1] : 0;
            if (last == 0) {
                atomicExch(err, 1);
                return;
            }
            bit0 = br.init(sp, front, (int32_t)(ssz - 1) * 8 + (int32_t)fse::highbit32(last));
            s0 = br.take(tl);
            s1 = br.take(tl);
            br.align();
        } else {
            const FseCkpt c = cks[jb.ck + q - 1];
            if (c.bitpos >= ssz * 8u || (c.s0 >> tl) || (c.s1 >> tl)) {
                atomicExch(err + 1, 1);
                return;
            }
            bit0 = br.init(sp, front, (int32_t)c.bitpos);
            s0 = c.s0;
            s1 = c.s1;
        }
        // Part q's symbols go to its own region of shared memory, kPartPad bytes more than a part
        // apart, four to a word: the parts' word stores then fall on different banks.
        uint8_t *so = BIG ? dst + start : s_out + (size_t)q * (nparts > 1 ? part + kPartPad : 0u);
        auto pair = [&]() -> uint32_t {  // two symbols; at most 2 * 13 bits
            const fse::DEntry e0 = dt[s0];
            const fse::DEntry e1 = dt[s1];
            s0 = e0.newState + br.take(e0.nbBits);
            s1 = e1.newState + br.take(e1.nbBits);
            return (uint32_t)e0.symbol | ((uint32_t)e1.symbol << 8);
        };
        unsigned i = start;
        for (; !BIG && i + 3 < end; i += 4) {
            const uint32_t lo = pair(), hi = pair();
            br.align();
            *reinterpret_cast<uint32_t *>(so + (i - start)) = lo | (hi << 16);
        }
        for (; i + 1 < end; i += 2) {
            const uint32_t v = pair();
            br.align();
            so[i - start] = (uint8_t)v;
            so[i - start + 1] = (uint8_t)(v >> 8);
        }
        if (i < end) so[i - start] = dt[s0].symbol;
        if (q + 1 < nparts) {
            const FseCkpt c = cks[jb.ck + q];
            if (c.s0 != s0 || c.s1 != s1 || br.pos != bit0 + (int32_t)c.bitpos) atomicExch(err + 1, 1);
        }
    };
    if (big) {
        for (unsigned q = threadIdx.x; q < nparts; q += blockDim.x) decode(q, std::true_type());
        return;
    }
    for (unsigned q = threadIdx.x; q < nparts; q += blockDim.x) decode(q, std::false_type());
    // the symbols leave in consecutive bytes across the CTA (each thread's part decoded into
    // shared memory, so that no warp store scatters over the parts)
    __syncthreads();
    if (nparts > 1) {
        // the last part runs to the block's end (up to two symbols past `part`, which its
        // region's padding holds)
        const unsigned lp = 31 - __clz(part);
        for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
            const unsigned r = min(i >> lp, nparts - 1);
            dst[i] = s_out[(size_t)r * (part + kPartPad) + (i - r * part)];
        }
    } else {
        for (unsigned i = threadIdx.x; i < n; i += blockDim.x) dst[i] = s_out[i];
    }
}

// Walks an fse_enc record sequence (host bytes) for n symbols starting at `off`; appends jobs.
size_t parse_blocks(const ByteView &h, size_t off, unsigned long long n, unsigned long long dst_base,
                    std::vector<BlockJob> &jobs) {
    const size_t len = h.len;
    unsigned long long done = 0;
    while (done < n) {
        const unsigned bn = (unsigned)std::min<unsigned long long>(n - done, FBLK);
        if (off >= len) throw std::invalid_argument("truncated FSE block stream");
        const uint8_t flag = h.at(off++);
        BlockJob j{dst_base + done, bn, flag, 0, 0};
        if (flag == 0) {
            if (off + bn > len) throw std::invalid_argument("truncated raw block");
            j.in = off;
            j.inlen = bn;
            off += bn;
        } else if (flag == 2) {
            if (off + 1 > len) throw std::invalid_argument("truncated RLE block");
            j.in = off;
            j.inlen = 1;
            off += 1;
        } else if (flag == 1) {
            if (off + 4 > len) throw std::invalid_argument("truncated FSE block header");
            const uint32_t rr = h.rd<uint32_t>(off);
            if (off + rr > len || bn < 3) throw std::invalid_argument("truncated FSE block");
            j.in = off;
            j.inlen = rr;
            off += rr;
        } else {
            throw std::invalid_argument("invalid FSE block flag");
        }
        jobs.push_back(j);
        done += bn;
    }
    return off;
}

// ------------------------------------------------------------------ Elias-gamma groups
// vals (u32, >= 1) of all groups concatenated; gstart has G+1 entries.
struct GammaOut {
    std::vector<std::vector<std::pair<const uint8_t *, size_t>>> cls_pieces;  // per group
    std::vector<std::vector<unsigned>> cls_n;                                  // symbols per block
    std::vector<std::vector<uint8_t>> cls_flag;                                // record flag per block
    std::vector<std::vector<const FseCkpt *>> cls_ck;                          // checkpoints per block
    std::vector<size_t> cls_bytes;                                             // per group
    std::vector<const uint8_t *> man_ptr;                                      // per group
    std::vector<size_t> man_bytes;                                             // per group
};

__global__ void k_gamma_cls(const uint32_t *__restrict__ v, long long n, uint8_t *__restrict__ cls) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        cls[i] = (uint8_t)(31 - __clz(v[i]));
}

// The values of group g, [gstart[g], gstart[g + 1]), are cut into units of kUnit from the group's start; unit u of
// the whole list belongs to the last group g with ustart[g] <= u.  A warp sums a unit's classes (its mantissa
// bits) and an exclusive scan of the unit sums gives every unit its first bit; a warp then packs or unpacks the
// unit's mantissas, kRun a lane at a time.
constexpr unsigned kUnit = 1024, kRun = 4;

__device__ __forceinline__ int unit_group(const unsigned long long *__restrict__ ustart, int G, unsigned long long u) {
    int lo = 0, hi = G - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ustart[mid] <= u) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(256) k_unit_bits(const uint8_t *__restrict__ cls,
                                                   const unsigned long long *__restrict__ gstart,
                                                   const unsigned long long *__restrict__ ustart, int G,
                                                   unsigned long long nunits, unsigned long long *__restrict__ usum) {
    const unsigned long long u = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned lane = threadIdx.x & 31u;
    if (u >= nunits) return;
    const int g = unit_group(ustart, G, u);
    const unsigned long long first = gstart[g] + (u - ustart[g]) * kUnit;
    const unsigned long long end = min(first + kUnit, gstart[g + 1]);
    uint32_t s = 0;
    for (unsigned long long i = first + lane; i < end; i += 32) s += cls[i];
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) usum[u] = s;
}

// The gamma value of an escape code, or a value itself.
__device__ __forceinline__ uint32_t gamma_value(int16_t code) { return zigzag((int)code) + 1u; }
__device__ __forceinline__ uint32_t gamma_value(uint32_t v) { return v; }

// Bits of every group (from the scan of the unit sums) and zeros in the words where a unit starts or a group
// ends, which neighbours share.
__global__ void k_gamma_heads(const unsigned long long *__restrict__ uoff, const unsigned long long *__restrict__ ustart,
                              int G, unsigned long long nunits, const unsigned long long *__restrict__ gword,
                              unsigned long long *__restrict__ gbits, uint32_t *__restrict__ words) {
    const unsigned long long u = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u < nunits) {
        const int g = unit_group(ustart, G, u);
        words[gword[g] + ((uoff[u] - uoff[ustart[g]]) >> 5)] = 0u;
    }
    if (u < (unsigned long long)G) {
        const unsigned long long b = uoff[ustart[u + 1]] - uoff[ustart[u]];
        gbits[u] = b;
        words[gword[u] + (b >> 5)] = 0u;
    }
}

// MSB-first packing of the mantissas (the k low bits of each value, k its class), a warp per unit: a warp scan
// of the lanes' bit counts gives each its place, the bits are merged in shared memory and whole big-endian words
// leave coalesced; a unit's first and last word by atomicOr.  Bound by issue: 49 M escapes take 131 us (a scan
// over all values, then an atomicOr of every mantissa into global memory, took 530).
constexpr int kUnitWarps = 8;
constexpr uint32_t kUnitWords = 32 * kRun * 31 / 32 + 2;
template <class V>
__global__ void __launch_bounds__(kUnitWarps * 32) k_gamma_pack_units(
    const V *__restrict__ vals, const uint8_t *__restrict__ cls, const unsigned long long *__restrict__ gstart,
    const unsigned long long *__restrict__ ustart, int G, unsigned long long nunits,
    const unsigned long long *__restrict__ uoff, const unsigned long long *__restrict__ gword,
    uint32_t *__restrict__ words) {
    __shared__ uint32_t s_buf[kUnitWarps][kUnitWords];
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const unsigned long long u = (unsigned long long)blockIdx.x * kUnitWarps + wid;
    if (u >= nunits) return;
    uint32_t *buf = s_buf[wid];
    for (uint32_t z = lane; z < kUnitWords; z += 32) buf[z] = 0u;
    const int g = unit_group(ustart, G, u);
    const unsigned long long first = gstart[g] + (u - ustart[g]) * kUnit, end = min(first + kUnit, gstart[g + 1]);
    const unsigned long long b0 = uoff[u] - uoff[ustart[g]];
    uint32_t *o = words + gword[g] + (b0 >> 5);
    uint32_t pos = (uint32_t)(b0 & 31);
    bool shared_first = true;
    __syncwarp();
    for (unsigned long long i0 = first; i0 < end; i0 += 32 * kRun) {
        const unsigned long long i = i0 + lane * kRun;
        uint32_t k[kRun], m[kRun], sum = 0;
#pragma unroll
        for (unsigned j = 0; j < kRun; j++) {
            k[j] = i + j < end ? cls[i + j] : 0u;
            m[j] = k[j] ? gamma_value(vals[i + j]) & ((1u << k[j]) - 1u) : 0u;
            sum += k[j];
        }
        const uint32_t incl = warp_incl_scan(sum);
        uint32_t p = pos + incl - sum;
        auto put = [&](unsigned long long v, uint32_t n) {  // the n <= 64 low bits of v
            const unsigned long long top = v << (64 - n);
            const uint32_t A = (uint32_t)(top >> 32), B = (uint32_t)top, w = p >> 5, sh = p & 31u, e = sh + n;
            atomicOr(buf + w, A >> sh);
            if (e > 32) atomicOr(buf + w + 1, __funnelshift_r(B, A, sh));
            if (e > 64) atomicOr(buf + w + 2, __funnelshift_r(0u, B, sh));
            p += n;
        };
        if (sum && sum <= 64) {
            unsigned long long v = 0;
#pragma unroll
            for (unsigned j = 0; j < kRun; j++) v = (v << k[j]) | m[j];
            put(v, sum);
        } else if (sum) {
#pragma unroll
            for (unsigned j = 0; j < kRun; j++)
                if (k[j]) put(m[j], k[j]);
        }
        const uint32_t tot = pos + __shfl_sync(0xffffffffu, incl, 31), full = tot >> 5;
        __syncwarp();
        for (uint32_t z = lane; z < full; z += 32) {
            const uint32_t w = __byte_perm(buf[z], 0, 0x0123);
            if (z == 0 && shared_first) atomicOr(o, w);
            else o[z] = w;
        }
        __syncwarp();
        const uint32_t rest = buf[full];
        __syncwarp();
        for (uint32_t z = lane; z <= full; z += 32) buf[z] = 0u;
        __syncwarp();
        if (lane == 0) buf[0] = rest;
        __syncwarp();
        shared_first = shared_first && full == 0;
        o += full;
        pos = tot & 31u;
    }
    if (lane == 0 && pos) atomicOr(o, __byte_perm(buf[0], 0, 0x0123));
}

// The FSE block coders' shared-memory limits, set once per device (a function attribute set while
// other threads launch the same kernel would only add driver work to every call).
void enable_fse_smem() {
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    FB2_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return;
    FB2_CUDA(cudaFuncSetAttribute(k_fse_encode_blocks<kFseGroups>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kFseGroups * sizeof(FseGroupSmem))));
    FB2_CUDA(cudaFuncSetAttribute(k_fse_encode_blocks<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(FseGroupSmem) + kWideBytes)));
    FB2_CUDA(cudaFuncSetAttribute(k_fse_decode_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fse_dec_smem(64)));
    done.fetch_or(bit, std::memory_order_acq_rel);
}

// The FSE class blocks of the gamma classes, launched by gamma_launch; gamma_pack packs the
// mantissas and gamma_finish collects both.  Between the two the caller may launch other work: the class
// blocks are long sequential chains, so they go to the GPU before the order-1 chain encoder.
struct GammaBlocks {
    long long T = 0;
    std::vector<unsigned long long> gstart;
    uint8_t *cls = nullptr;
    std::vector<BlockJob> jobs;
    std::vector<int> job_group;
    uint8_t *slots = nullptr;
    unsigned long long *sizes = nullptr;
    FseCkpt *cks = nullptr;
    size_t ck_per_block = 0;
    unsigned long long *phase = nullptr;  // per-block phase times, traced calls only
    // About how long the blocks take: 15 ns a symbol of the longest one, 1 ms for a full one, kFseGroups an SM in a wave.
    double ns() const {
        unsigned n = 0;
        for (const BlockJob &j : jobs) n = std::max(n, j.n);
        return 15.0 * n * (double)((jobs.size() + kFseGroups * sm_count() - 1) / (kFseGroups * sm_count()));
    }
};
// About how long the chain encoder takes for N codes, where most of its parts meet.
inline double chains_ns(long long N) { return 4e5 + 5e-3 * (double)N; }

// `beside`: CTAs of whole SMs that run next to the class blocks (the chain encoder's), for about `beside_ns`.
GammaBlocks gamma_launch(Pool &pool, uint8_t *cls, const std::vector<unsigned long long> &gstart, cudaStream_t st,
                         uint32_t ckpt_part, cudaEvent_t queued = nullptr, size_t beside = 0, double beside_ns = 0) {
    GammaBlocks gb;
    gb.gstart = gstart;
    const int G = (int)gstart.size() - 1;
    const long long T = (long long)gstart.back();
    gb.T = T;
    if (T == 0) {
        if (queued) FB2_CUDA(cudaEventRecord(queued, st));
        return gb;
    }
    gb.cls = cls;
    for (int g = 0; g < G; g++) {
        for (unsigned long long b = gstart[g]; b < gstart[g + 1]; b += FBLK) {
            gb.jobs.push_back(BlockJob{b, (unsigned)std::min<unsigned long long>(FBLK, gstart[g + 1] - b), 0, 0, 0});
            gb.job_group.push_back(g);
        }
    }
    const size_t nj = gb.jobs.size();
    if (std::getenv("FALCONS_TRACE"))
        std::fprintf(stderr, "[falcons trace] escapes: %lld values in %d groups, %zu class blocks\n", T, G, nj);
    gb.slots = pool.get<uint8_t>(nj * kBlockSlot);
    uint8_t *bits = pool.get<uint8_t>(nj * kBlockSlot);
    gb.sizes = pool.get<unsigned long long>(nj);
    gb.ck_per_block = ckpt_part ? FBLK / ckpt_part : 0;
    gb.cks = ckpt_part ? pool.get<FseCkpt>(nj * gb.ck_per_block) : nullptr;
    uint32_t *recs = pool.get<uint32_t>(nj * kFseRecWords);
    std::vector<uint32_t> order(nj);
    for (size_t j = 0; j < nj; j++) order[j] = (uint32_t)j;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return gb.jobs[a].n > gb.jobs[b].n; });
    Upload up;
    const size_t u_jobs = up.add(gb.jobs), u_order = up.add(order);
    up.send(pool, st);
    const BlockJob *d_jobs = up.get<BlockJob>(u_jobs);
    const uint32_t *d_order = up.get<uint32_t>(u_order);
    if (queued) FB2_CUDA(cudaEventRecord(queued, st));  // what the blocks wait for is on the stream
    const uint32_t part = ckpt_part ? ckpt_part : 4096u;
    if (std::getenv("FALCONS_TRACE")) {
        gb.phase = pool.get<unsigned long long>(nj * kFsePhases);
        FB2_CUDA(cudaMemsetAsync(gb.phase, 0, nj * kFsePhases * 8, st));
    }
    enable_fse_smem();
    // a block an SM where there are SMs for all, or where the few blocks outlast the other CTAs even if those come to two
    // waves without their SMs: 7 full blocks beside 6.5 M codes end at 1.02 ms eight a CTA and at 0.79 an SM each (the
    // chains at 0.29 and 0.31)
    const size_t sms = (size_t)sm_count();
    if (nj + beside > sms && !(4 * nj <= sms && 2 * beside_ns < gb.ns())) {
        constexpr unsigned G = kFseGroups;
        constexpr int smem = (int)(G * sizeof(FseGroupSmem));
        k_fse_encode_blocks<G><<<(unsigned)((nj + G - 1) / G), G * kFseGroupThreads, smem, st>>>(
            cls, d_jobs, (unsigned)nj, gb.slots, gb.sizes, bits, part, gb.cks, recs, d_order, gb.phase);
    } else {
        constexpr int smem = (int)(sizeof(FseGroupSmem) + kWideBytes);
        k_fse_encode_blocks<1><<<(unsigned)nj, kFseGroupThreads, smem, st>>>(
            cls, d_jobs, (unsigned)nj, gb.slots, gb.sizes, bits, part, gb.cks, recs, d_order, gb.phase);
    }
    FB2_CHECK_LAUNCH();
    return gb;
}

// The packed mantissas of the groups: words on the device, where each group's start in them.
struct GammaWords {
    uint32_t *buf = nullptr;
    std::vector<unsigned long long> gword;
    unsigned long long *d_gb = nullptr;  // bits per group
};

// Packs the mantissas (needs the classes and the values, not the class blocks).
template <class V>
GammaWords gamma_pack(Pool &pool, const uint8_t *cls, const std::vector<unsigned long long> &gstart, const V *d_vals,
                      cudaStream_t st) {
    GammaWords w;
    const int G = (int)gstart.size() - 1;
    if (gstart.back() == 0) return w;
    // every group's words: room for the longest mantissas (16 bits of an escape code's value, 31 of any)
    constexpr unsigned long long kMost = sizeof(V) == 2 ? 16 : 31;
    std::vector<unsigned long long> ust(G + 1, 0);
    w.gword.assign(G, 0);
    unsigned long long words = 0;
    for (int g = 0; g < G; g++) {
        const unsigned long long c = gstart[g + 1] - gstart[g];
        w.gword[g] = words;
        words += (c * kMost + 31) / 32 + 2;
        ust[g + 1] = ust[g] + (c + kUnit - 1) / kUnit;
    }
    const unsigned long long NU = ust[G];
    w.buf = pool.get<uint32_t>(words + 4);
    Upload up;
    const size_t u_gstart = up.add(gstart), u_ust = up.add(ust), u_gword = up.add(w.gword);
    up.send(pool, st);
    const unsigned long long *d_gstart = up.get<unsigned long long>(u_gstart), *d_ust = up.get<unsigned long long>(u_ust),
                             *d_gword = up.get<unsigned long long>(u_gword);
    unsigned long long *uoff = pool.get<unsigned long long>(NU + 1);
    w.d_gb = pool.get<unsigned long long>(G);
    k_unit_bits<<<grid_for((long long)NU * 32, 256), 256, 0, st>>>(cls, d_gstart, d_ust, G, NU, uoff);
    FB2_CHECK_LAUNCH();
    k_scan_small<unsigned long long><<<1, 1024, 0, st>>>(uoff, (long long)NU);
    FB2_CHECK_LAUNCH();
    k_gamma_heads<<<grid_for((long long)std::max<unsigned long long>(NU, G), 256), 256, 0, st>>>(uoff, d_ust, G, NU, d_gword,
                                                                                                w.d_gb, w.buf);
    FB2_CHECK_LAUNCH();
    k_gamma_pack_units<V><<<(unsigned)((NU + kUnitWarps - 1) / kUnitWarps), kUnitWarps * 32, 0, st>>>(
        d_vals, cls, d_gstart, d_ust, G, NU, uoff, d_gword, w.buf);
    FB2_CHECK_LAUNCH();
    return w;
}

// Collects the groups: the mantissas packed on stream ms, the class blocks coded on stream st.
GammaOut gamma_finish(const GammaBlocks &gb, const GammaWords &w, cudaStream_t st, cudaStream_t ms) {
    Trace tr("gamma");
    const int G = (int)gb.gstart.size() - 1;
    GammaOut out;
    out.cls_pieces.resize(G);
    out.cls_n.resize(G);
    out.cls_flag.resize(G);
    out.cls_ck.resize(G);
    out.cls_bytes.assign(G, 0);
    out.man_ptr.assign(G, nullptr);
    out.man_bytes.assign(G, 0);
    if (gb.T == 0) return out;
    const std::vector<unsigned long long> gbits = d2h(w.d_gb, (size_t)G, ms);
    tr.mark("group bits known");
    for (int g = 0; g < G; g++) {
        out.man_bytes[g] = (size_t)((gbits[g] + 7) / 8);
        out.man_ptr[g] = reinterpret_cast<const uint8_t *>(w.buf + w.gword[g]);
    }
    std::vector<unsigned long long> hs = d2h(gb.sizes, gb.jobs.size(), st);
    tr.mark("class blocks coded");
    if (gb.phase && tr.on) {
        const size_t nj = gb.jobs.size();
        const std::vector<unsigned long long> ph = d2h(gb.phase, nj * kFsePhases, st);
        unsigned long long t0 = ~0ULL, t1 = 0;
        double sum[6] = {0};
        for (size_t j = 0; j < nj; j++) {
            const unsigned long long *p = ph.data() + j * kFsePhases;
            t0 = std::min(t0, p[0]);
            t1 = std::max(t1, p[6]);
            for (int k = 0; k < 6; k++)
                if (p[k] && p[k + 1]) sum[k] += (double)(p[k + 1] - p[k]);
        }
        std::fprintf(stderr,
                     "[falcons trace] gamma class blocks: %zu, span %.3f ms; per block (us): count %.1f plan %.1f "
                     "tables %.1f chain walk %.1f pack %.1f output %.1f\n",
                     nj, (double)(t1 - t0) / 1e6, sum[0] / nj / 1e3, sum[1] / nj / 1e3, sum[2] / nj / 1e3,
                     sum[3] / nj / 1e3, sum[4] / nj / 1e3, sum[5] / nj / 1e3);
    }
    for (size_t j = 0; j < gb.jobs.size(); j++) {
        const int g = gb.job_group[j];
        const size_t sz = (size_t)(hs[j] & ((1ULL << 56) - 1));
        out.cls_pieces[g].push_back({gb.slots + j * kBlockSlot, sz});
        out.cls_n[g].push_back(gb.jobs[j].n);
        out.cls_flag[g].push_back((uint8_t)(hs[j] >> 56));
        out.cls_ck[g].push_back(gb.cks ? gb.cks + j * gb.ck_per_block : nullptr);
        out.cls_bytes[g] += sz;
    }
    return out;
}

GammaOut gamma_encode(Pool &pool, const uint32_t *d_vals, const std::vector<unsigned long long> &gstart,
                      cudaStream_t st, uint32_t ckpt_part) {
    const long long T = (long long)gstart.back();
    uint8_t *cls = pool.get<uint8_t>(T);
    if (T > 0) {
        k_gamma_cls<<<grid_for(T, 256), 256, 0, st>>>(d_vals, T, cls);
        FB2_CHECK_LAUNCH();
    }
    const GammaBlocks gb = gamma_launch(pool, cls, gstart, st, ckpt_part);
    return gamma_finish(gb, gamma_pack(pool, cls, gstart, d_vals, st), st, st);
}

// Adds the fse_enc records of group g, recording each record's header bytes for the index.
// Gathers the decode checkpoints of the streams in stream order and writes the FB2C frame.
struct CkptCollector {
    uint32_t o1_part = 0, fse_part = 0;
    const O1Ckpt *o1 = nullptr;
    unsigned long long n_o1 = 0;
    std::vector<std::pair<const FseCkpt *, uint32_t>> fse;
    unsigned long long n_fse = 0;
    void add_block(const FseCkpt *p, uint32_t count) {
        if (p && count) {
            fse.push_back({p, count});
            n_fse += count;
        }
    }
    void emit(Assembler &as) const {
        if (n_o1 + n_fse == 0 || !as.with_index) return;
        const unsigned long long content = kCkptHeader + n_o1 * sizeof(O1Ckpt) + n_fse * sizeof(FseCkpt);
        if (content >= 0xFFFFFFFFULL) return;
        uint8_t h[8 + kCkptHeader];
        static_assert(kCkptHeader == 32, "content header: tag, version, o1_part, fse_part, n_o1, n_fse");
        const uint32_t w[6] = {kSkippableMagic, (uint32_t)content, kCkptTag, kCkptVersion, o1_part, fse_part};
        memcpy(h, w, sizeof(w));
        memcpy(h + 24, &n_o1, 8);
        memcpy(h + 32, &n_fse, 8);
        as.tail_bytes(h, sizeof(h));
        as.tail_dev(o1, n_o1 * sizeof(O1Ckpt));
        for (auto &f : fse) as.tail_dev(f.first, (size_t)f.second * sizeof(FseCkpt));
    }
};
static_assert(sizeof(O1Ckpt) == 12 && sizeof(FseCkpt) == 8, "checkpoint record sizes are part of the frame format");

void add_class_pieces(Assembler &as, const GammaOut &go, int g, CkptCollector *cc = nullptr) {
    for (size_t b = 0; b < go.cls_pieces[g].size(); b++) {
        const auto &p = go.cls_pieces[g][b];
        if (cc && go.cls_flag[g][b] == 1) cc->add_block(go.cls_ck[g][b], fse_ckpt_count(go.cls_n[g][b], cc->fse_part));
        uint8_t h[5];
        size_t hl;
        const uint8_t flag = go.cls_flag[g][b];
        if (flag != 1) { h[0] = flag; hl = 1; }
        else {
            h[0] = 1;
            const uint32_t r = (uint32_t)(p.second - 5);
            memcpy(h + 1, &r, 4);
            hl = 5;
        }
        as.shadow(h, hl);
        as.dev(p.first, p.second);
    }
}

// Escape values (zigzag + 1, gamma-coded) of every unit, a warp per unit: v[i] = (1 << k) |
// mantissa, or, with `ovf`, the escape code unzz(v - 1) at its place gdst[g] + (i - gstart[g]).
// uoff is the exclusive scan of the unit bit sums; the warp takes its unit's values kRun a lane at a
// time, a warp scan of their classes giving each lane its mantissas' bit offset (a scan for every 32 values
// was most of the instructions: 250 us for 49 M values, this takes 116).  A class above 31 sets
// err 2, a mantissa past its group's region err 3.
__global__ void __launch_bounds__(256) k_gamma_unpack_units(
    const uint8_t *__restrict__ cls, const unsigned long long *__restrict__ gstart,
    const unsigned long long *__restrict__ ustart, int G, unsigned long long nunits,
    const unsigned long long *__restrict__ uoff, const unsigned long long *__restrict__ gman,
    const uint8_t *__restrict__ base, const unsigned long long *__restrict__ gman_len, uint32_t *__restrict__ v,
    int *__restrict__ err, const unsigned long long *__restrict__ gdst, int16_t *__restrict__ ovf) {
    const unsigned long long u = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned lane = threadIdx.x & 31u;
    if (u >= nunits) return;
    const int g = unit_group(ustart, G, u);
    const unsigned long long g0 = gstart[g];
    const unsigned long long first = g0 + (u - ustart[g]) * kUnit;
    const unsigned long long end = min(first + kUnit, gstart[g + 1]);
    const unsigned long long len = gman_len[g];
    const uint8_t *rb = base + gman[g];
    unsigned long long run = uoff[u] - uoff[ustart[g]];  // bit offset of the values below
    bool bad2 = false, bad3 = false;
    const uintptr_t ra = reinterpret_cast<uintptr_t>(rb);
    const uint32_t *rw = reinterpret_cast<const uint32_t *>(ra & ~uintptr_t(3));
    const unsigned lead = (unsigned)(ra & 3) * 8;
    for (unsigned long long i0 = first; i0 < end; i0 += 32 * kRun) {
        const unsigned long long i = i0 + lane * kRun;
        unsigned k[kRun];
        uint32_t sum = 0;
#pragma unroll
        for (unsigned j = 0; j < kRun; j++) {
            k[j] = i + j < end ? cls[i + j] : 0u;
            if (k[j] > 31) {
                bad2 = true;
                k[j] = 0;
            }
            sum += k[j];
        }
        const uint32_t incl = warp_incl_scan(sum);
        const unsigned long long bb = run + incl - sum;
        run += __shfl_sync(0xffffffffu, incl, 31);
        if (i >= end) continue;
        uint32_t val[kRun];
        if (((bb + sum + 7) >> 3) > len) {
            bad3 = true;
#pragma unroll
            for (unsigned j = 0; j < kRun; j++) val[j] = 1u << k[j];
        } else {
            // the lane's bits from the first word on, as big-endian words; 96 bits at a time cover the word's
            // offset and 64 bits (classes up to 16), more classes take a load a value
            unsigned long long at = lead + bb;
            auto word = [&](unsigned long long w, unsigned long long last) {  // words up to that of bit `last`
                return w <= last >> 5 ? __byte_perm(__ldg(rw + w), 0, 0x0123) : 0u;
            };
            if (sum <= 64) {
                const unsigned long long w = at >> 5, last = at + (sum ? sum - 1 : 0);
                const uint32_t x0 = sum ? word(w, last) : 0u, x1 = word(w + 1, last), x2 = word(w + 2, last);
                const unsigned o = (unsigned)(at & 31);
                uint32_t hi = __funnelshift_l(x1, x0, o), lo = __funnelshift_l(x2, x1, o);
#pragma unroll
                for (unsigned j = 0; j < kRun; j++) {
                    val[j] = __funnelshift_l(hi, 1u, k[j]);  // 1 << k with the mantissa below
                    hi = __funnelshift_l(lo, hi, k[j]);
                    lo <<= k[j];
                }
            } else {
#pragma unroll
                for (unsigned j = 0; j < kRun; j++) {
                    const unsigned long long w = at >> 5, last = at + (k[j] ? k[j] - 1 : 0);
                    const uint32_t x0 = k[j] ? word(w, last) : 0u, x1 = word(w + 1, last);
                    val[j] = __funnelshift_l(__funnelshift_l(x1, x0, (unsigned)(at & 31)), 1u, k[j]);
                    at += k[j];
                }
            }
        }
#pragma unroll
        for (unsigned j = 0; j < kRun; j++) {
            if (i + j >= end) continue;
            if (ovf) ovf[gdst[g] + (i + j - g0)] = (int16_t)unzz(val[j] - 1u);
            else v[i + j] = val[j];
        }
    }
    if (bad2) atomicExch(err, 2);
    if (bad3) atomicExch(err, 3);
}

// ------------------------------------------------------------------ delta
__global__ void k_delta(const int16_t *__restrict__ in, long long n, int16_t *__restrict__ out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = i ? (int16_t)(uint16_t)((uint16_t)in[i] - (uint16_t)in[i - 1]) : in[0];
}

// Inclusive prefix sum modulo 2^16 (un-delta), tile based.
__global__ void __launch_bounds__(kScanThreads) k_tile_sum16(const int16_t *__restrict__ in, long long n,
                                                            uint32_t *__restrict__ tile_sum) {
    const long long base = (long long)blockIdx.x * kScanTile;
    uint32_t s = 0;
    for (int j = 0; j < kScanItems; j++) {
        const long long i = base + (long long)j * kScanThreads + threadIdx.x;
        if (i < n) s += (uint16_t)in[i];
    }
    __shared__ uint32_t sh[32];
    uint32_t tot;
    block_excl_scan<uint32_t>(s, sh, tot);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot & 0xFFFF;
}

__global__ void __launch_bounds__(kScanThreads) k_tile_undelta(int16_t *__restrict__ io, long long n,
                                                              const uint32_t *__restrict__ tile_off) {
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        const long long i = base + j;
        v[j] = i < n ? (uint16_t)io[i] : 0u;
        s += v[j];
    }
    __shared__ uint32_t sh[32];
    uint32_t tot;
    uint32_t run = block_excl_scan<uint32_t>(s, sh, tot) + tile_off[blockIdx.x];
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        const long long i = base + j;
        run += v[j];
        if (i < n) io[i] = (int16_t)(uint16_t)run;
    }
}

void undelta(Pool &pool, int16_t *d, long long n, cudaStream_t st) {
    if (n <= 1) return;
    const long long tiles = (n + kScanTile - 1) / kScanTile;
    uint32_t *ts = pool.get<uint32_t>(tiles + 2);
    k_tile_sum16<<<(unsigned)tiles, kScanThreads, 0, st>>>(d, n, ts);
    FB2_CHECK_LAUNCH();
    k_scan_small<uint32_t><<<1, 1024, 0, st>>>(ts, tiles);
    FB2_CHECK_LAUNCH();
    k_tile_undelta<<<(unsigned)tiles, kScanThreads, 0, st>>>(d, n, ts);
    FB2_CHECK_LAUNCH();
}

// ------------------------------------------------------------------ method 0
__global__ void __launch_bounds__(kScanThreads) k_m0_tiles(const int16_t *__restrict__ q, long long n,
                                                          uint32_t *__restrict__ cnt, long long *__restrict__ last) {
    const long long base = (long long)blockIdx.x * kScanTile;
    uint32_t c = 0;
    long long l = -1;
    for (int j = 0; j < kScanItems; j++) {
        const long long i = base + (long long)j * kScanThreads + threadIdx.x;
        if (i < n && q[i] != 0) {
            c++;
            l = i > l ? i : l;
        }
    }
    __shared__ uint32_t sh[32];
    uint32_t tot;
    block_excl_scan<uint32_t>(c, sh, tot);
    __shared__ long long lm;
    if (threadIdx.x == 0) lm = -1;
    __syncthreads();
    if (l >= 0) atomicMax(&lm, l);
    __syncthreads();
    if (threadIdx.x == 0) {
        cnt[blockIdx.x] = tot;
        last[blockIdx.x] = lm;
    }
}

// Exclusive running max of tile "last nonzero" positions (one block, chunked); last[tiles] = overall max.
__global__ void __launch_bounds__(1024) k_prefix_last(long long *__restrict__ last, long long tiles) {
    __shared__ long long sh[1024];
    __shared__ long long carry;
    if (threadIdx.x == 0) carry = -1;
    __syncthreads();
    for (long long base = 0; base < tiles; base += blockDim.x) {
        const long long i = base + threadIdx.x;
        const long long v = i < tiles ? last[i] : -1;
        sh[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < (int)blockDim.x; o <<= 1) {
            const long long y = threadIdx.x >= (unsigned)o ? sh[threadIdx.x - o] : -1;
            __syncthreads();
            if (y > sh[threadIdx.x]) sh[threadIdx.x] = y;
            __syncthreads();
        }
        const long long before = threadIdx.x ? sh[threadIdx.x - 1] : -1;
        const long long c = carry;
        if (i < tiles) last[i] = before > c ? before : c;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = sh[threadIdx.x] > c ? sh[threadIdx.x] : c;
        __syncthreads();
    }
    if (threadIdx.x == 0) last[tiles] = carry;
}

__global__ void __launch_bounds__(kScanThreads) k_m0_extract(const int16_t *__restrict__ q, long long n,
                                                            const uint32_t *__restrict__ tile_off,
                                                            const long long *__restrict__ tile_prev,
                                                            uint32_t *__restrict__ runs, uint32_t *__restrict__ vals) {
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    int16_t v[kScanItems];
    uint32_t c = 0;
    long long l = -1;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        const long long i = base + j;
        v[j] = i < n ? q[i] : (int16_t)0;
        if (v[j] != 0) {
            c++;
            l = i;
        }
    }
    __shared__ uint32_t sh[32];
    uint32_t tot;
    uint32_t rank = block_excl_scan<uint32_t>(c, sh, tot) + tile_off[blockIdx.x];
    // previous nonzero before this thread's items: max over lower threads of their last, else tile carry
    __shared__ long long lastv[kScanThreads];
    lastv[threadIdx.x] = l;
    __syncthreads();
    // inclusive max-scan over threads (Hillis-Steele in shared memory)
    for (int o = 1; o < kScanThreads; o <<= 1) {
        long long y = threadIdx.x >= (unsigned)o ? lastv[threadIdx.x - o] : -1;
        __syncthreads();
        if (y > lastv[threadIdx.x]) lastv[threadIdx.x] = y;
        __syncthreads();
    }
    long long prev = threadIdx.x ? lastv[threadIdx.x - 1] : -1;
    if (prev < 0) prev = tile_prev[blockIdx.x];
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        if (v[j] != 0) {
            const long long i = base + j;
            runs[rank] = (uint32_t)(i - prev);  // L + 1
            vals[rank] = zigzag((int)v[j]) + 1u;
            prev = i;
            rank++;
        }
    }
}

// ------------------------------------------------------------------ method 1
struct SegInfo {
    unsigned long long lo, n, cs;   // segment start, length, chunk size
    int K;
    int pad;
};

// Per segment: the count of every (context, symbol) key of its chains (a chain's first code has
// context 0) and every chain's escape count; writes every code's key (context << 8 | symbol) for
// the chain encoder.  CTA (g, k + K u) takes the u-th slice of chain k of segment g (slice edges on
// multiples of 8 codes) and adds its counts to the segment's totals, which start at zero.  Codes are
// read 8 at a time as 16-byte vectors when q is 16-byte aligned (the code before a vector comes from
// the lane below); runs of equal keys within a vector are counted
// with one atomic, and the lanes of a warp spread their atomics over kHistCopies histograms.
// Bound by issue and the shared-memory pipe (a lookup and about one atomic a code): a table of the clamped
// code gives symbol and context in one lookup, where computing both took 60 instructions a code
// (134 M codes: 307 us, now 196).
constexpr int kHistCopies = 4;
constexpr int kLutSize = 257;  // codes clamped to -128 .. 128
constexpr size_t kHistSmem = (size_t)kHistCopies * O1_NCTX * O1_NSYM * 4 + (kLutSize + 7) / 8 * 16;
__global__ void __launch_bounds__(1024, 2) k_o1_hist(const int16_t *__restrict__ q, const SegInfo *__restrict__ segs,
                                                    uint32_t *__restrict__ hist, uint32_t *__restrict__ nvk,
                                                    uint16_t *__restrict__ keys, int vec) {
    extern __shared__ uint32_t hs[];  // kHistCopies histograms of O1_NCTX * O1_NSYM keys, then the table
    __shared__ uint32_t s_esc;
    constexpr int HN = O1_NCTX * O1_NSYM;
    uint16_t *const lut = reinterpret_cast<uint16_t *>(hs + kHistCopies * HN);  // 0x8000 escape | context << 8 | symbol
    const SegInfo sg = segs[blockIdx.x];
    const unsigned long long U = gridDim.y / sg.K, u = blockIdx.y / sg.K;
    const int k = (int)(blockIdx.y % sg.K);
    for (int i = threadIdx.x; i < kHistCopies * HN / 4; i += blockDim.x) reinterpret_cast<uint4 *>(hs)[i] = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < kLutSize; i += blockDim.x) {
        const int sy = o1_sym(i - 128);
        lut[i] = (uint16_t)((sy == O1_NSYM - 1 ? 0x8000 : 0) | (o1_ctx(i - 128) << 8) | sy);
    }
    if (threadIdx.x == 0) s_esc = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    uint32_t *h = hs + (lane % kHistCopies) * HN;
    auto entry = [&](int code) -> uint32_t { return lut[min(max(code, -128), 128) + 128]; };
    // the key of a code from its own entry and that of the code before it
    auto key_of = [](uint32_t before, uint32_t e) -> uint32_t { return (before & 0xF00u) | (e & 0xFFu); };
    const long long b = (long long)(sg.lo + (unsigned long long)k * sg.cs);
    const long long e = (long long)(sg.lo + min((unsigned long long)k * sg.cs + sg.cs, sg.n));
    if (e <= b) return;
    // this CTA's slice [sb, se) of the chain [b, e)
    const unsigned long long len = (unsigned long long)(e - b);
    auto edge = [&](unsigned long long v) -> long long {
        if (v == 0) return b;
        if (v >= U) return e;
        const long long x = (b + (long long)(len * v / U) + 7) & ~7LL;
        return x < e ? x : e;
    };
    const long long sb = edge(u), se = edge(u + 1);
    if (se <= sb) return;
    // codes [sb, hb) and [tb, se) one per thread, whole vectors [hb, tb) one per thread
    long long hb = se, tb = se;
    if (vec) {
        hb = min(se, (sb + 7) & ~7LL);
        tb = max(hb, se & ~7LL);
    }
    uint32_t ne = 0;
    const long long nh = hb - sb, nt = se - tb;
    for (long long j = threadIdx.x; j < nh + nt; j += blockDim.x) {
        const long long i = j < nh ? sb + j : tb + (j - nh);
        const uint32_t c = entry((int)q[i]), key = key_of(i == b ? 0u : entry((int)q[i - 1]), c);
        atomicAdd(&h[key], 1u);
        keys[i] = (uint16_t)key;
        ne += c >> 15;
    }
    const uint32_t nv = (uint32_t)((tb >> 3) - (hb >> 3));
    const uint4 *const q4 = reinterpret_cast<const uint4 *>(q) + (hb >> 3);
    uint4 *const k4 = reinterpret_cast<uint4 *>(keys) + (hb >> 3);
    const bool first = hb == b;  // the first vector starts the chain (context 0)
    for (uint32_t vb = threadIdx.x & ~31u; vb < nv; vb += blockDim.x) {  // warp-uniform
        const uint32_t vi = vb + lane;
        const bool act = vi < nv;
        const uint4 w = act ? __ldg(q4 + vi) : make_uint4(0, 0, 0, 0);
        const uint32_t below = __shfl_up_sync(0xffffffffu, w.w >> 16, 1);
        if (!act) continue;
        int prev = (int)(int16_t)below;  // the code before this vector
        if (lane == 0) prev = vi == 0 && first ? 0 : (int)reinterpret_cast<const int16_t *>(q4 + vi)[-1];
        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
        uint32_t ent[8], kk[8];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            // two codes clamped to -128 .. 128 and biased to 0 .. 256 (no borrow between the halves)
            const uint32_t t = (__vmins2(__vmaxs2(ww[m], 0xFF80FF80u), 0x00800080u) ^ 0x80008000u) - 0x7F807F80u;
            ent[2 * m] = lut[t & 0xFFFFu];
            ent[2 * m + 1] = lut[t >> 16];
        }
        uint32_t before = entry(prev), flags = 0;
#pragma unroll
        for (int m = 0; m < 8; m++) {
            kk[m] = key_of(before, ent[m]);
            before = ent[m];
            flags += ent[m] >> 15;
        }
        ne += flags;
        uint32_t rn = 1;
#pragma unroll
        for (int m = 1; m < 8; m++) {
            const bool same = kk[m] == kk[m - 1];
            if (!same) atomicAdd(&h[kk[m - 1]], rn);
            rn = same ? rn + 1 : 1;
        }
        atomicAdd(&h[kk[7]], rn);
        k4[vi] = make_uint4(kk[0] | (kk[1] << 16), kk[2] | (kk[3] << 16), kk[4] | (kk[5] << 16), kk[6] | (kk[7] << 16));
    }
    ne = __reduce_add_sync(0xffffffffu, ne);
    if (lane == 0 && ne) atomicAdd(&s_esc, ne);
    __syncthreads();
    uint32_t *gh = hist + (size_t)blockIdx.x * HN;
    for (int i = threadIdx.x; i < HN; i += blockDim.x) {
        uint32_t v = 0;
#pragma unroll
        for (int c = 0; c < kHistCopies; c++) v += hs[c * HN + i];
        if (v) atomicAdd(gh + i, v);
    }
    if (threadIdx.x == 0 && s_esc) atomicAdd(nvk + blockIdx.x * kMaxK + k, s_esc);
}

// Keeps every m-th decode checkpoint of every chain (the m-th, 2m-th, ... of chain c's
// src[soff[c] ..]), compacted to dst[doff[c] ..]: checkpoints m times as far apart.
__global__ void k_ck_thin(const O1Ckpt *__restrict__ src, const unsigned long long *__restrict__ soff,
                          const unsigned long long *__restrict__ doff, int nchains, uint32_t m,
                          O1Ckpt *__restrict__ dst) {
    const int c = blockIdx.y;
    if (c >= nchains) return;
    const unsigned long long n = doff[c + 1] - doff[c];
    for (unsigned long long j = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; j < n;
         j += (unsigned long long)gridDim.x * blockDim.x)
        dst[doff[c] + j] = src[soff[c] + (j + 1) * m - 1];
}

// The order-1 tables (RleFseEncoder.hpp:410-477 normalizes each context's counts to O1_M cells):
// one warp per (region, context) table, lanes holding 8 symbols each, with the rule of
// fse::normalize_count: every present symbol gets its nearest share of the cells (at least one)
// under a scale refined for the one-cell floor, then single cells move by marginal coded size
// (count / (n - 1/2) compared in integers) until the table is full.  An empty context gets all
// cells on symbol 0, a context with one symbol all cells on it.
// The moves are a serial chain (up to hundreds a table), so a move costs as little as it can: every
// symbol's marginal size is kept as an integer key and only the moved symbol's is computed again;
// the best key of the warp takes three warp reductions.  (Comparing the fractions themselves across
// the warp on every move took 107 us for the 30 tables of a 384^3 float64 field, this 44 us.)
__global__ void __launch_bounds__(256) k_o1_norm(const uint32_t *__restrict__ hist, int total_tables,
                                                 uint16_t *__restrict__ nf) {
    const int wt = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (wt >= total_tables) return;
    const uint32_t *cnt = hist + (size_t)wt * O1_NSYM;
    uint16_t *freq = nf + (size_t)wt * O1_NSYM;
    constexpr int PER = O1_NSYM / 32;
    uint32_t c[PER];
    int n[PER];
    unsigned long long total = 0;
    int present = 0;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        c[i] = cnt[lane + 32 * i];
        total += c[i];
        present += c[i] != 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    present = __reduce_add_sync(0xffffffffu, (unsigned)present);
    if (total == 0 || present == 1) {
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int sy = lane + 32 * i;
            freq[sy] = (uint16_t)(total == 0 ? (sy == 0 ? O1_M : 0) : (c[i] ? O1_M : 0));
        }
        return;
    }
    double mu = (double)O1_M / (double)total;
    int left = 0;
    for (int round = 0; round < 4; round++) {
        int ones = 0, sum = 0;
        unsigned long long ones_count = 0;
#pragma unroll
        for (int i = 0; i < PER; i++) {
            if (!c[i]) {
                n[i] = 0;
                continue;
            }
            const double share = floor((double)c[i] * mu + 0.5);
            int v = share < (double)O1_M ? (int)share : O1_M;
            if (v <= 1) {
                v = 1;
                ones++;
                ones_count += c[i];
            }
            n[i] = v;
            sum += v;
        }
        sum = (int)__reduce_add_sync(0xffffffffu, (unsigned)sum);
        ones = (int)__reduce_add_sync(0xffffffffu, (unsigned)ones);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ones_count += __shfl_xor_sync(0xffffffffu, ones_count, o);
        left = O1_M - sum;
        if (left == 0 || ones_count == total) break;
        mu = (double)(O1_M - ones) / (double)(total - ones_count);
    }
    if (left != 0) {
        // 2 c / (2 n + 1) for a cell more, 2 c / (2 n - 1) for a cell less, as floor(. 2^29): two
        // different fractions with denominators up to 16385 lie more than 2^-28.01 apart, so the keys
        // compare as the fractions do.  The largest key moves (complemented for a cell less; 0: none).
        const bool add = left > 0;
        auto key_of = [&](uint32_t cnt_i, int n_i) -> unsigned long long {
            if (!cnt_i || (!add && n_i < 2)) return 0;
            const unsigned long long k = ((unsigned long long)cnt_i << 30) / (unsigned)(add ? 2 * n_i + 1 : 2 * n_i - 1);
            return add ? k : ~k;
        };
        unsigned long long key[PER];
#pragma unroll
        for (int i = 0; i < PER; i++) key[i] = key_of(c[i], n[i]);
        for (; left != 0; left += add ? -1 : 1) {
            unsigned long long bk = key[0];
            int bi = 0;
#pragma unroll
            for (int i = 1; i < PER; i++)
                if (key[i] > bk) {
                    bk = key[i];
                    bi = i;
                }
            const uint32_t hi = (uint32_t)(bk >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
            const uint32_t lo = hi == mh ? (uint32_t)bk : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
            if ((mh | ml) == 0) break;  // nothing movable (cannot happen: fewer symbols than cells)
            const bool mine = hi == mh && lo == ml;
            const uint32_t bs = __reduce_min_sync(0xffffffffu, mine ? (uint32_t)(lane + 32 * bi) : ~0u);
            if (mine && bs == (uint32_t)(lane + 32 * bi)) {  // ties: the lower symbol
#pragma unroll
                for (int i = 0; i < PER; i++)
                    if (i == bi) {
                        n[i] += add ? 1 : -1;
                        key[i] = key_of(c[i], n[i]);
                    }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < PER; i++) freq[lane + 32 * i] = (uint16_t)n[i];
}

// ---- tANS tables for 15 contexts x 256 symbols, built by a whole CTA per table (zfse
// fse_compress.c FSE_buildCTable_wksp / fse_decompress.c FSE_buildDTable, restated in parallel).
// A table is 8192 cells and there are as few as 15 of them, so what bounds the build is one CTA's
// latency: 32 warps scan, spread and rank 256 cells each.  (One warp ranking all cells took 80 us
// for 15 encode tables and 101 us for the decode tables; this takes 9 and 17 us.)
constexpr int kTabThreads = 1024;
constexpr int kTabCells = O1_M / kTabThreads;  // visits, then cells, per thread
static_assert(kTabCells * 32 == O1_M / 32, "a warp ranks the 256 cells of its own span");
struct TabSmem {
    int16_t norm[O1_NSYM];
    uint32_t cum[O1_NSYM + 1];   // cells before every symbol (a -1 symbol holds one cell)
    uint32_t occ[O1_NSYM + 1];   // spread occurrences before every symbol (positive counts only)
    uint32_t scan[3][32];
    uint16_t cnt[32][O1_NSYM];   // cells of every symbol in every warp's span, then before it
    uint8_t sym[O1_M];
};

// The spread (fse::spread): symbol s takes the occurrences occ[s] .. occ[s+1]-1 of the visit order
// j -> (j * step) & mask that skips the cells above `high` (the -1 symbols' cells).  Every thread
// maps one run of j; a block scan of the kept visits gives each its occurrence number.  Returns
// false (for every thread) when the counts do not fill the table.
__device__ bool cta_spread(TabSmem &w) {
    constexpr uint32_t mask = O1_M - 1;
    const uint32_t step = fse::table_step(O1_M);
    uint32_t ones = 0, cells = 0;  // a -1 symbol's cell, the other symbols' cells
    if (threadIdx.x < O1_NSYM) {
        const int nn = w.norm[threadIdx.x];
        ones = nn == -1;
        cells = nn > 0 ? (uint32_t)nn : 0u;
    }
    uint32_t n_ones, n_cells;
    const uint32_t o = block_excl_scan<uint32_t>(ones, w.scan[0], n_ones);
    const uint32_t c = block_excl_scan<uint32_t>(cells, w.scan[1], n_cells);
    if (n_ones + n_cells != (uint32_t)O1_M) return false;
    if (threadIdx.x < O1_NSYM) {
        w.cum[threadIdx.x] = o + c;
        w.occ[threadIdx.x] = c;
        if (ones) w.sym[mask - o] = (uint8_t)threadIdx.x;  // the -1 symbols take the top cells in order
    }
    if (threadIdx.x == 0) {
        w.cum[O1_NSYM] = O1_M;
        w.occ[O1_NSYM] = n_cells;
    }
    const uint32_t high = mask - n_ones, j0 = threadIdx.x * kTabCells;
    uint32_t kept = 0;
#pragma unroll
    for (uint32_t j = 0; j < kTabCells; j++) kept += (((j0 + j) * step) & mask) <= high;
    uint32_t all;
    uint32_t k = block_excl_scan<uint32_t>(kept, w.scan[2], all);  // its barriers publish cum and occ
    int sy = 0;  // the symbol whose occurrences hold k: occ[sy] <= k < occ[sy + 1]
    for (int hi = O1_NSYM; hi - sy > 1;) {
        const int mid = (sy + hi) >> 1;
        if (w.occ[mid] <= k) sy = mid;
        else hi = mid;
    }
#pragma unroll
    for (uint32_t j = 0; j < kTabCells; j++) {
        const uint32_t pos = ((j0 + j) * step) & mask;
        if (pos > high) continue;
        while (w.occ[sy + 1] <= k) sy++;
        w.sym[pos] = (uint8_t)sy;
        k++;
    }
    __syncthreads();
    return true;
}

// For every cell u, f(u, s, rank) with rank = the cells of symbol s before u: match ranks within 32
// cells, counted up over the warp's span, then the counts of the spans before.
template <class F>
__device__ void cta_ranks(TabSmem &w, F &&f) {
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint16_t *cnt = w.cnt[wid];
    for (int s2 = lane; s2 < O1_NSYM; s2 += 32) cnt[s2] = 0;
    __syncwarp();
    uint32_t rank[kTabCells];
#pragma unroll
    for (int i = 0; i < kTabCells; i++) {
        const unsigned sy = w.sym[wid * (O1_M / 32) + i * 32 + lane];
        const unsigned peers = __match_any_sync(0xffffffffu, sy);
        const unsigned r = __popc(peers & ((1u << lane) - 1u));
        rank[i] = cnt[sy] + r;
        __syncwarp();
        if (r == (unsigned)__popc(peers) - 1u) cnt[sy] = (uint16_t)(rank[i] + 1);
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < O1_NSYM) {
        uint32_t run = 0;
#pragma unroll 8
        for (int v = 0; v < 32; v++) {
            const uint32_t c = w.cnt[v][threadIdx.x];
            w.cnt[v][threadIdx.x] = (uint16_t)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kTabCells; i++) {
        const unsigned u = wid * (O1_M / 32) + i * 32 + lane, sy = w.sym[u];
        f(u, sy, rank[i] + cnt[sy]);
    }
}

// A table set as the chain encoder holds it in shared memory: the 15 packed state tables, then two words per key.
constexpr unsigned kTabWords = O1_M * O1_PB / 32;  // packed words of a context's state table
constexpr size_t kEncSmem = ((size_t)O1_NCTX * kTabWords + (size_t)O1_NCTX * O1_NSYM * 2) * 4;
static_assert(kEncSmem % 16 == 0 && kEncSmem + 2048 <= 227 * 1024, "16-byte words; 2 KiB for the kernels' own arrays");
// The words of key context << 8 | symbol: deltaNbBits (state x emits (x + deltaNbBits) >> 16 bits) and 13
// times (deltaFindState + 8192 context), which added to 13 times the shifted state is the place of the next
// state's packed entry.
// The encoder's image of table blockIdx.x (k_o1_walk below): its state table packed, its symbol transforms.
__global__ void __launch_bounds__(kTabThreads) k_o1_ctable(const uint16_t *__restrict__ nf, uint32_t *__restrict__ image,
                                                         int *__restrict__ err) {
    __shared__ TabSmem w;
    __shared__ uint16_t st[O1_M + 4];  // cells by symbol, in increasing order
    const size_t t = blockIdx.x;
    for (int s2 = threadIdx.x; s2 < O1_NSYM; s2 += blockDim.x) w.norm[s2] = (int16_t)nf[t * O1_NSYM + s2];
    if (threadIdx.x < 4) st[O1_M + threadIdx.x] = 0;
    __syncthreads();
    if (!cta_spread(w)) {
        if (threadIdx.x == 0) atomicExch(err, 4);
        return;
    }
    cta_ranks(w, [&](uint32_t u, unsigned sy, uint32_t r) { st[w.cum[sy] + r] = (uint16_t)u; });
    __syncthreads();
    uint32_t *img = image + (t / O1_NCTX) * (kEncSmem / 4), c = (uint32_t)(t % O1_NCTX);
    for (unsigned wd = threadIdx.x; wd < kTabWords; wd += blockDim.x) {
        // bits [32 wd, 32 wd + 32) of the entries (entry j at bit 13 j): at most 4 of them
        const unsigned j0 = wd * 32 / O1_PB, sh = wd * 32 - j0 * O1_PB;
        unsigned long long v = 0;
#pragma unroll
        for (unsigned u = 0; u < 4; u++) v |= (unsigned long long)st[j0 + u] << (O1_PB * u);
        img[c * kTabWords + wd] = (uint32_t)(v >> sh);
    }
    for (int s2 = threadIdx.x; s2 < O1_NSYM; s2 += blockDim.x) {
        const int nn = w.norm[s2];
        const uint32_t total = w.cum[s2];
        fse::SymTT tt;
        if (nn == 0) {
            tt.deltaNbBits = ((O1_PB + 1) << 16) - O1_M;
            tt.deltaFindState = 0;
        } else if (nn == -1 || nn == 1) {
            tt.deltaNbBits = (O1_PB << 16) - O1_M;
            tt.deltaFindState = (int32_t)total - 1;
        } else {
            const uint32_t maxBitsOut = O1_PB - fse::highbit32((uint32_t)(nn - 1));
            const uint32_t minStatePlus = (uint32_t)nn << maxBitsOut;
            tt.deltaNbBits = (maxBitsOut << 16) - minStatePlus;
            tt.deltaFindState = (int32_t)total - nn;
        }
        reinterpret_cast<uint2 *>(img + O1_NCTX * kTabWords)[c * O1_NSYM + s2] =
            make_uint2(tt.deltaNbBits, (uint32_t)(tt.deltaFindState + (int32_t)(c << O1_PB)) * O1_PB);
    }
}

// Decode tables of table blockIdx.x:
//   cells  16 bits per cell: a symbol's cells are numbered in chunks of 128, the low 9 bits are the chunk (of
//          all the table's, in symbol order: at most 256 + 8192 / 128), the high 7 the number within it; with
//   info   one u32 per chunk: bits 0-3 the exponent of the lowest power of two above the symbol's count,
//          4-7 the context of the code, 8-15 the code (-128: escape), 16 escape, 18-31 the state number
//          (count + rank) of its first cell: 17 KiB a context, so that 11 to 13 of the 15 stay in shared memory
// From a cell's state number n = info's + number and exponent x the decoder has nbBits = 14 - x - (n >> x)
// and newState + 8192 = n << nbBits.  The last gridDim.x - ntab CTAs rank the contexts of a table set each.
struct DecRank {
    unsigned long long slot, ctx;  // 4 bits each: the slot of every context, the context of every slot
};
constexpr uint32_t kChunkBits = 7, kChunks = O1_NSYM + (O1_M >> kChunkBits);

// Slots by how often a decoder is in a context: the stationary distribution of the context chain that the
// counts imply (the next context is a function of the decoded code; escapes split between the two
// large-magnitude contexts 13 and 14).  Those two take slots 0 and 1, so that an escape's sign is the slot.
__device__ void rank_contexts(const uint16_t *__restrict__ nf, DecRank *__restrict__ out) {
    __shared__ double P[2][O1_NCTX * O1_NCTX];
    __shared__ double s_pi[O1_NCTX];
    __shared__ uint32_t s_n[O1_NCTX * O1_NCTX];  // half cells of a context whose code leads to another
    __shared__ int s_rank[13];
    const uint32_t t = threadIdx.x;
    if (t < O1_NCTX * O1_NCTX) s_n[t] = 0;
    __syncthreads();
    for (uint32_t k = t; k < O1_NCTX * O1_NSYM; k += blockDim.x) {
        const int nn = (int16_t)nf[k];
        if (nn == 0 || nn < -1) continue;
        const uint32_t c = k / O1_NSYM, sy = k % O1_NSYM, cells = nn < 0 ? 1u : (uint32_t)nn;
        if (sy == O1_NSYM - 1) {
            atomicAdd(&s_n[c * O1_NCTX + 13], cells);
            atomicAdd(&s_n[c * O1_NCTX + 14], cells);
        } else {
            atomicAdd(&s_n[c * O1_NCTX + o1_ctx(unzz(sy))], 2 * cells);
        }
    }
    __syncthreads();
    if (t < O1_NCTX * O1_NCTX) P[0][t] = (double)s_n[t] / (2 * O1_M);
    __syncthreads();
    int cur = 0;
    for (int it = 0; it < 7; it++, cur ^= 1) {  // the chain's 128th power by squaring
        if (t < O1_NCTX * O1_NCTX) {
            double v = 0;
            for (int k = 0; k < O1_NCTX; k++) v += P[cur][t / O1_NCTX * O1_NCTX + k] * P[cur][k * O1_NCTX + t % O1_NCTX];
            P[cur ^ 1][t] = v;
        }
        __syncthreads();
    }
    if (t < O1_NCTX) {
        double v = 0;
        for (int k = 0; k < O1_NCTX; k++) v += P[cur][k * O1_NCTX + t];
        s_pi[t] = v;
    }
    __syncthreads();
    if (t < 13) {
        int rank = 2;
#pragma unroll 1
        for (uint32_t d = 0; d < 13; d++) rank += s_pi[d] > s_pi[t] || (s_pi[d] == s_pi[t] && d < t);
        s_rank[t] = rank;
    }
    __syncthreads();
    if (t == 0) {
        DecRank r{0, 0};
        auto put = [&](int c, int slot) {
            r.slot |= (unsigned long long)slot << (4 * c);
            r.ctx |= (unsigned long long)c << (4 * slot);
        };
        put(13, 0);
        put(14, 1);
        for (int c = 0; c < 13; c++) put(c, s_rank[c]);
        *out = r;
    }
}

__global__ void __launch_bounds__(kTabThreads) k_o1_dtable(const uint16_t *__restrict__ nf, uint32_t ntab,
                                                         uint16_t *__restrict__ cells,
                                                         uint32_t *__restrict__ info, DecRank *__restrict__ rank,
                                                         int *__restrict__ err) {
    __shared__ TabSmem w;
    const size_t t = blockIdx.x;
    if (t >= ntab) {
        rank_contexts(nf + (t - ntab) * O1_NCTX * O1_NSYM, rank + (t - ntab));
        return;
    }
    uint32_t *inf = info + t * kChunks;
    uint16_t *ce = cells + t * O1_M;
    for (int s2 = threadIdx.x; s2 < O1_NSYM; s2 += blockDim.x) w.norm[s2] = (int16_t)nf[t * O1_NSYM + s2];
    // chunks that no symbol takes, and all of a table that cannot be: emits nothing, stays in its state
    constexpr uint32_t kStay = ((uint32_t)O1_M << 18) | 14u;
    for (uint32_t c = threadIdx.x; c < kChunks; c += blockDim.x) inf[c] = kStay;
    __syncthreads();
    if (!cta_spread(w)) {
        if (threadIdx.x == 0) atomicExch(err, 5);
        for (uint32_t u = threadIdx.x; u < O1_M; u += blockDim.x) ce[u] = 0;
        return;
    }
    const int my = threadIdx.x < O1_NSYM ? w.norm[threadIdx.x] : 0;
    const uint32_t mine = my == -1 ? 1u : ((uint32_t)max(my, 0) + (1u << kChunkBits) - 1) >> kChunkBits;
    uint32_t all;
    const uint32_t first = block_excl_scan<uint32_t>(mine, w.scan[0], all);
    if (threadIdx.x < O1_NSYM) {
        const uint32_t sy = threadIdx.x;
        const bool esc = sy == O1_NSYM - 1;
        const int code = esc ? -128 : unzz(sy);
        const uint32_t n = w.norm[sy] == -1 ? 1u : (uint32_t)max((int)w.norm[sy], 0);
        const uint32_t v = (n ? fse::highbit32(n) + 1 : 0u) | ((uint32_t)(esc ? 13 : o1_ctx(code)) << 4) |
                           ((uint32_t)(code & 0xFF) << 8) | (esc ? 1u << 16 : 0u);
        for (uint32_t j = 0; j < mine; j++) inf[first + j] = ((n + (j << kChunkBits)) << 18) | v;
        w.occ[sy] = first;  // done with by the spread
    }
    __syncthreads();
    cta_ranks(w, [&](uint32_t u, unsigned sy, uint32_t r) {
        ce[u] = (uint16_t)((w.occ[sy] + (r >> kChunkBits)) | ((r & ((1u << kChunkBits) - 1)) << 9));
    });
}

struct DecChain {
    unsigned long long in;      // stream byte offset
    unsigned long long inlen;   // stream length (0 = empty chunk)
    unsigned long long lo, n;   // output range
    unsigned long long ovf;     // first escape value of this chunk
    int table;                  // segment index (tables at table * 15)
    uint32_t nesc;              // escapes of this chunk
    uint32_t ck;                // first decode checkpoint of this chunk
    uint32_t pad;
};

// Items [first, first + count) of one table set (chains or parts) that a CTA takes.
struct ChainCta {
    int table;
    int first;
    int count;
};

// ---- parallel chain encoder
// Every chain is cut into parts of `part` codes, one part per thread.  A tANS encoder walks its
// chain backwards and only its state carries from one code to the next, so the parts are coded in
// steps, each a launch over all parts of all chains:
//   1. k_o1_walk: every part runs from a guessed entering state (the top part from the exact initial
//      state), writing the bits of every 8 codes as one record and keeping the state and the bit count
//      at every 64th index (`kept`, `kept_bits`) and its exit state;
//   2. k_o1_repair: every part runs again from the exit state of the part above, writing its records
//      and kept states over, until its state equals the one kept there (from there on the two runs, and
//      their records, are identical); a part that never meets has a new exit state;
//   3. k_o1_rounds, a CTA per chain: the parts whose entering state changed run again, in rounds;
//   4. where many parts did not meet, or rounds did not settle them: k_o1_maps, k_o1_compose and
//      k_o1_walk again (below);
//   5. k_o1_settle, a CTA per chain: scans the bit counts into every part's offset and writes the decode
//      checkpoints: state, bit position, context and escape count at every part start;
//   6. k_o1_place: joins the records' bits in the chain's slot.
// The stream is bit-identical to a sequential encoder's (the tANS states are fully determined).
//
// What bounds it: a walk is a serial chain of table lookups, so its time is the codes of a part times
// the latency of a step where few parts share an SM, and the shared-memory pipe (three lookups a code,
// each about 3.4 bank conflicts deep) where an SM is full of them.  So the parts of all chains are
// spread evenly over the SMs whatever chain they belong to (with all parts of a chain in one CTA, a
// field of one segment ran on 16 of the 148 SMs), over about kEncWarps warps of a CTA (fewer lanes a
// warp wait less for one another, more warps cost issue slots); the transforms of 8 codes are looked
// up ahead of their steps; and records of a fixed 16 bytes per 8 codes leave as whole coalesced
// vectors, where words stored as they filled hit a line a lane.  All launches together, before (one
// kernel, a CTA a chain) and now: 64^3 points 289 -> 118 us, 211 x 307 x 401 1144 -> 485 us, 1800 x 3600 at
// 1.4 bits a code 36.2 -> 1.1 ms, 512^3 at 8.5 bits 1021 -> 800 us, at 1.6 bits 62 -> 5.3 ms.
//
// All 15 context state tables stay in shared memory, as 13-bit entries (state - 8192) packed into
// words, so that no lookup leaves the SM and every context takes the same instructions (two 16-bit
// tables beside 13 packed ones cost every warp both paths); two words per key hold the symbol
// transform (one word fits too, but takes a dozen more instructions a code to unpack).  k_o1_ctable
// lays this image out once per table set; every CTA copies it in.
constexpr int kEncThreads = 1024;
constexpr uint32_t kEncWarps = 4, kMinEncPart = 512;
constexpr int kKeptShift = 6;  // kept states: every 64th index

// Parts [first, first + count) of one table set: warp w codes the parts first + w * lanes + l, l < lanes.
// Its records interleave (record r of lane l at rec + (w * records of a part + r) * lanes + l).
struct EncCta {
    int table;
    uint32_t first, count, lanes;
    uint32_t chain;          // chain of the first part
    unsigned long long rec;  // records of the CTAs before
};
struct EncChain {
    unsigned long long lo, hi;  // its codes
};
struct EncArgs {
    const uint16_t *keys;        // context of code i (0 at a chain's first code) << 8 | symbol, by k_o1_hist
    const EncChain *chains;
    const uint32_t *pstart;      // first part of every chain, then the number of parts
    uint32_t nchains, part, recs;  // codes per part, records per part
    uint32_t max_rounds;
    const uint32_t *image;       // table sets, kEncSmem bytes each
    const EncCta *ctas;
    // per part: exit state of the first walk and of the last one, entering state of the last one (map
    // path: the exact one, written ahead of its walk), bits, escapes, first record | lanes << 56, first bit
    // in the slots, records to place (bit 31: and the final state's)
    uint16_t *exit1, *exit2, *entry;
    uint32_t *bits, *esc, *nrec;
    unsigned long long *column, *at;
    uint16_t *kept, *kept_bits;
    uint4 *rec;
    int *err;                    // [0] error, [2] codes run again, [3] rounds, [5] parts that did not meet,
                                 // [6] chains that the rounds did not settle
};

// Records of one part: its groups of 8 codes (by index) and the final state's.
inline uint32_t part_records(uint32_t part) { return part / 8 + 2; }

// Whether rounds are left out, and whether the map path codes this call: where more than half of the parts did
// not meet their kept states, rounds pass a changed state down part by part, and where fewer did not, some chains
// may take more than max_rounds.  A round is a part's walk, 30 to 55 us, the map path 0.9 ms at 12.7 K parts (6.5 M
// codes) and 4 ms at 98 K (100 M), so the larger the call, the more rounds come before the maps.
inline uint32_t max_rounds(uint32_t nparts) { return 16 + nparts / 4096; }
__device__ __forceinline__ bool many_unmet(const EncArgs &A) {
    return (uint32_t)__ldcg(A.err + 5) > __ldg(A.pstart + A.nchains) / 2;
}
__device__ __forceinline__ bool map_path(const EncArgs &A) { return many_unmet(A) || __ldcg(A.err + 6) != 0; }

struct EncPartPos {
    uint32_t chain, p, nparts;
    long long a, first;  // the part's lowest code; the first (highest) one it codes
    bool is_top;         // the chain's last code initialises the state
};
// Part `id` (of a chain at or after `chain`).
__device__ __forceinline__ EncPartPos enc_part(const EncArgs &A, uint32_t id, uint32_t chain) {
    uint32_t hi = A.nchains;  // pstart[chain] <= id < pstart[hi]
    while (hi - chain > 1) {
        const uint32_t mid = (chain + hi) >> 1;
        if (__ldg(A.pstart + mid) <= id) chain = mid;
        else hi = mid;
    }
    EncPartPos r;
    const uint32_t p0 = __ldg(A.pstart + chain);
    const EncChain c = A.chains[chain];
    r.chain = chain;
    r.p = id - p0;
    r.nparts = __ldg(A.pstart + chain + 1) - p0;
    r.a = (long long)c.lo + (long long)r.p * A.part;
    r.is_top = r.p + 1 == r.nparts;
    r.first = r.is_top ? (long long)c.hi - 2 : r.a + A.part - 1;
    return r;
}

__device__ __forceinline__ void load_image(uint4 *smem, const uint32_t *image, int table) {
    const uint4 *src = reinterpret_cast<const uint4 *>(image + (size_t)table * (kEncSmem / 4));
#pragma unroll 4
    for (unsigned i = threadIdx.x; i < kEncSmem / 16; i += blockDim.x) smem[i] = __ldg(src + i);
}

// A record: bits 0-103 those of up to 8 codes (LSB first, as the stream), 120-127 their count.
__device__ __forceinline__ uint4 make_record(unsigned long long lo, unsigned long long hi, uint32_t n) {
    return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32) | (n << 24));
}

// The table set in the CTA's dynamic shared memory.
struct EncTables {
    static __device__ __forceinline__ const uint32_t *words() {
        extern __shared__ uint4 smem_raw[];
        return reinterpret_cast<const uint32_t *>(smem_raw);
    }
    // the transform of a key
    static __device__ __forceinline__ uint2 transform(uint32_t key) {
        return reinterpret_cast<const uint2 *>(words() + O1_NCTX * kTabWords)[key];
    }
    static __device__ __forceinline__ uint32_t entry(uint32_t bit) {
        const uint32_t *w = words() + (bit >> 5);
        return (__funnelshift_r(w[0], w[1], bit) & (O1_M - 1)) | O1_M;
    }
    // state x codes a key with transform e: the bits it emits, their number, the next state
    static __device__ __forceinline__ uint32_t next(uint32_t x, uint2 e, uint32_t &v, uint32_t &nb) {
        nb = (x + e.x) >> 16;
        const uint32_t r = x >> nb;
        v = x - (r << nb);
        return entry(r * O1_PB + e.y);
    }
    // FSE_initCState2: the state that codes symbol k with the fewest bits
    static __device__ __forceinline__ uint32_t init(uint32_t key) {
        const uint2 e = transform(key);
        const uint32_t nb = (e.x + (1u << 15)) >> 16;
        return entry((((nb << 16) - e.x) >> nb) * O1_PB + e.y);
    }
    // The 8 codes of a vector of keys, the last one first: their record's bits, their number.
    static __device__ __forceinline__ uint4 group(uint32_t &x, const uint4 &v, uint32_t &n) {
        const uint32_t k[8] = {v.w >> 16, v.w & 0xFFFFu, v.z >> 16, v.z & 0xFFFFu,
                               v.y >> 16, v.y & 0xFFFFu, v.x >> 16, v.x & 0xFFFFu};
        uint2 e[8];
#pragma unroll
        for (int j = 0; j < 8; j++) e[j] = transform(k[j]);
        unsigned long long q[2];
        uint32_t nq[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t w[2], nw[2];
#pragma unroll
            for (int g = 0; g < 2; g++) {
                uint32_t va, na, vb, nb;
                x = next(x, e[4 * h + 2 * g], va, na);
                x = next(x, e[4 * h + 2 * g + 1], vb, nb);
                w[g] = va | (vb << na);
                nw[g] = na + nb;
            }
            q[h] = (unsigned long long)w[0] | ((unsigned long long)w[1] << nw[0]);
            nq[h] = nw[0] + nw[1];
        }
        n = nq[0] + nq[1];
        return make_record(q[0] | (q[1] << nq[0]), nq[0] ? q[1] >> (64 - nq[0]) : 0ull, n);
    }
    // The same for the codes from i down to e of one vector's span.
    static __device__ __forceinline__ uint4 partial(uint32_t &x, const uint16_t *keys, long long i, long long e,
                                                    uint32_t &n) {
        unsigned long long lo = 0, hi = 0;
        n = 0;
        for (; i >= e; i--) {
            uint32_t v32, nb;
            x = next(x, transform(__ldg(keys + i)), v32, nb);
            const unsigned long long v = v32;
            if (n < 64) {
                lo |= v << n;
                if (n + nb > 64) hi |= v >> (64 - n);
            } else {
                hi |= v << (n - 64);
            }
            n += nb;
        }
        return make_record(lo, hi, n);
    }
};

// Codes keys[first] down to keys[a] by the vectors of 8 keys they lie in, fetched ahead: f(i, r, n, v)
// for every record r of n bits, i its lowest index and v its keys (only whole vectors: `whole`); stops and returns true where f does.
template <class F>
__device__ __forceinline__ bool walk_records(const uint16_t *__restrict__ keys, long long first,
                                             long long a, uint32_t &x, F &&f) {
    if (first < a) return false;
    long long g = first >> 3;
    const long long ga = a >> 3;
    const uint4 z = make_uint4(0, 0, 0, 0);
    uint32_t n;
    if ((first & 7) != 7 || g * 8 < a) {
        const long long e = max(g * 8, a);
        const uint4 r = EncTables::partial(x, keys, first, e, n);
        if (f(e, r, n, z, false)) return true;
        g--;
    }
    const long long gl = (a & 7) ? ga + 1 : ga;  // the lowest whole vector
    if (g >= gl) {
        // a ring of three vectors, each loaded into its place as soon as its keys are coded (a shift of
        // the ring would wait for the load it moves)
        const uint4 *kv = reinterpret_cast<const uint4 *>(keys);
        auto load = [&](long long j) { return j >= gl ? __ldg(kv + j) : z; };
        auto one = [&](uint4 &v) {
            const uint4 r = EncTables::group(x, v, n);
            if (f(g * 8, r, n, v, true)) return true;
            v = load(g - 3);
            g--;
            return false;
        };
        uint4 v0 = load(g), v1 = load(g - 1), v2 = load(g - 2);
        for (;;) {
            if (one(v0)) return true;
            if (g < gl) break;
            if (one(v1)) return true;
            if (g < gl) break;
            if (one(v2)) return true;
            if (g < gl) break;
        }
    }
    if (g >= ga) {
        const uint4 r = EncTables::partial(x, keys, g * 8 + 7, a, n);
        if (f(a, r, n, z, false)) return true;
    }
    return false;
}

// Runs the state through the codes without recording their bits.
__device__ __forceinline__ void walk_states(const uint16_t *keys, long long first, long long a,
                                            uint32_t &x) {
    walk_records(keys, first, a, x, [](long long, const uint4 &, uint32_t, const uint4 &, bool) { return false; });
}

// Escapes (symbol 255) among 8 keys.
__device__ __forceinline__ uint32_t escapes_of(const uint4 &v) {
    auto m = [](uint32_t w) { return ((w & 0x00FF00FFu) + 0x00010001u) & 0x01000100u; };  // bits 8 and 24
    return __popc(m(v.x) | (m(v.y) >> 1) | (m(v.z) >> 2) | (m(v.w) >> 3));
}

// The walk of every part: EXACT = false from a guessed entering state (the state that codes the next
// code with the fewest bits), true from the exact one (`entry`, the map path only).
template <bool EXACT>
__global__ void __launch_bounds__(kEncThreads) k_o1_walk(const EncArgs A) {
    extern __shared__ uint4 smem_raw[];
    if (EXACT && !map_path(A)) return;
    const EncCta w = A.ctas[blockIdx.x];
    load_image(smem_raw, A.image, w.table);
    __syncthreads();
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31u, item = wid * w.lanes + lane;
    if (lane >= w.lanes || item >= w.count) return;
    const uint32_t id = w.first + item;
    const EncPartPos P = enc_part(A, id, w.chain);
    const unsigned long long col = w.rec + (unsigned long long)wid * A.recs * w.lanes + lane;
    uint4 *out = A.rec + col;
    uint32_t x, esc = 0, bits = 0, span = 0;
    if (P.is_top) {
        const uint32_t k0 = __ldg(A.keys + P.first + 1);
        x = EncTables::init(k0);
        esc = (k0 & 0xFFu) == 0xFFu;
    } else {
        x = EXACT ? A.entry[id] : EncTables::init(__ldg(A.keys + P.first + 1));
    }
    walk_records(A.keys, P.first, P.a, x, [&](long long i, const uint4 &r, uint32_t n, const uint4 &v, bool whole) {
        *out = r;
        out += w.lanes;
        bits += n;
        span += n;
        if (whole) {
            esc += escapes_of(v);
        } else {
            long long j = i;  // the codes of the vector's span inside the part
            do esc += (__ldg(A.keys + j) & 0xFFu) == 0xFFu;
            while ((++j & 7) != 0 && j <= P.first);
        }
        if (((uint32_t)i & 63u) == 0) {
            A.kept[i >> kKeptShift] = (uint16_t)x;
            A.kept_bits[i >> kKeptShift] = (uint16_t)span;
            span = 0;
        }
        return false;
    });
    if (P.p == 0) {  // the final state, then the end mark
        A.rec[col + (unsigned long long)(A.recs - 1) * w.lanes] = make_record((x - O1_M) | (1u << O1_PB), 0, O1_PB + 1);
        bits += O1_PB + 1;
    }
    A.exit1[id] = (uint16_t)x;
    A.bits[id] = bits;
    A.esc[id] = esc;
    A.column[id] = col | ((unsigned long long)w.lanes << 56);
    if (EXACT || P.is_top) A.exit2[id] = (uint16_t)x;  // nothing to repair
}

// Runs a part again from entering state x until its state meets a kept one, writing records and kept
// states over.  Returns whether it met; `bits` is kept up to date.
__device__ __forceinline__ bool rerun_part(const EncArgs &A, const EncPartPos &P, uint32_t &x,
                                           unsigned long long column, uint32_t &bits, uint32_t &steps) {
    const uint32_t lanes = (uint32_t)(column >> 56);
    uint4 *const rec = A.rec + (column & ((1ULL << 56) - 1)), *out = rec;
    uint32_t fresh = 0, stale = 0, span = 0;
    // the state kept at the next 64th index below, loaded one kept index ahead
    long long ki = P.first & ~63LL;
    uint32_t kx = ki >= P.a ? A.kept[ki >> kKeptShift] : 0u, kb = ki >= P.a ? A.kept_bits[ki >> kKeptShift] : 0u;
    const bool met = walk_records(A.keys, P.first, P.a, x, [&](long long i, const uint4 &r, uint32_t n, const uint4 &, bool) {
        *out = r;
        out += lanes;
        fresh += n;
        span += n;
        if (i != ki) return false;
        stale += kb;
        A.kept_bits[i >> kKeptShift] = (uint16_t)span;
        span = 0;
        steps += 64;
        if (kx == x) return true;
        A.kept[i >> kKeptShift] = (uint16_t)x;
        ki -= 64;
        if (ki >= P.a) {
            kx = A.kept[ki >> kKeptShift];
            kb = A.kept_bits[ki >> kKeptShift];
        }
        return false;
    });
    if (met) {
        bits += fresh - stale;
    } else {
        bits = fresh;
        if (P.p == 0) {
            rec[(unsigned long long)(A.recs - 1) * lanes] = make_record((x - O1_M) | (1u << O1_PB), 0, O1_PB + 1);
            bits += O1_PB + 1;
        }
    }
    return met;
}

__global__ void __launch_bounds__(kEncThreads) k_o1_repair(const EncArgs A) {
    extern __shared__ uint4 smem_raw[];
    const EncCta w = A.ctas[blockIdx.x];
    load_image(smem_raw, A.image, w.table);
    __syncthreads();
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31u, item = wid * w.lanes + lane;
    uint32_t steps = 0, unmet = 0;
    if (lane < w.lanes && item < w.count) {
        const uint32_t id = w.first + item;
        const EncPartPos P = enc_part(A, id, w.chain);
        if (!P.is_top) {
            uint32_t x = A.exit1[id + 1], bits = A.bits[id];
            const bool met = rerun_part(A, P, x, A.column[id], bits, steps);
            const uint32_t ex1 = A.exit1[id];
            A.entry[id] = A.exit1[id + 1];
            A.exit2[id] = (uint16_t)(met ? ex1 : x);
            A.bits[id] = bits;
            unmet = !met && x != ex1;
        }
    }
    steps = __reduce_add_sync(0xffffffffu, steps);
    unmet = __reduce_add_sync(0xffffffffu, unmet);
    if (lane == 0 && steps) atomicAdd(A.err + 2, (int)steps);
    if (lane == 0 && unmet) atomicAdd(A.err + 5, (int)unmet);
}

// ---- the map path
// Where codes take a few bits each (smooth fields at loose bounds), a step changes the distance of two
// states by little more than a rounding, so runs from different states meet only after thousands to
// millions of codes, and the exact states would have to pass down a chain part by part (249 rounds,
// 36 ms, for 1800 x 3600 points at 1.4 bits a code).  Instead every run of parts (a super part) is
// coded from all 8192 entering states at once, as the map from its entering to its leaving state:
//   k_o1_maps     W warps a super part (four where the SMs hold few of them).  A step keeps the cyclic
//                 order of the states (within a symbol the next state grows with the state), so states
//                 that have become equal are neighbours: after 8, 16, 32 .. 512 codes and at every part end, neighbours that are equal
//                 are merged into one class (about 8192 / (s sqrt(n)) classes are left after n codes,
//                 with s the rounding of a step).  Every merge stores the map from the classes
//                 before it to those after, and the classes' states.
//   k_o1_compose  a CTA a chain: one thread follows the exact state from super part to super part
//                 (two lookups each), then a thread per super part follows its entering state through
//                 the merges to the entering state of every part.
// and k_o1_walk<true> then codes every part from its exact state.  All lanes of a super part code the
// same key, so a step is one conflicting shared-memory lookup a state.  A super part whose maps do
// not fit its scratch (long runs of nearly certain codes merge nothing) is walked through by the
// composing thread.
constexpr uint32_t kMaxSuper = 32;                    // parts per super part, at most
constexpr uint32_t kMapHdr = 4 + 2 * (7 + kMaxSuper);  // words of a super part's header
struct MapArgs {
    const uint32_t *sstart;  // first super part of every chain, then their number
    uint32_t spp;            // parts per super part
    uint32_t cap;            // 16-bit words of a super part's scratch
    uint16_t *scratch;
    uint32_t *hdr;           // [0] usable, [1] merges, [2] those before the first part end, [3] place of the
                             // composed map; then per merge the places of its map and its states
    const EncCta *ctas;      // super parts per CTA
};

// The barrier of a super part's W warps.
template <int W>
__device__ __forceinline__ void map_sync(unsigned bar) {
    __syncwarp();
    if (W > 1) asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(32 * W) : "memory");
}

// Runs states src[j] for j < n through the codes from i down to e, states tid, tid + T, .. by thread tid of
// T; dst[j] = the state after.  Warps without a state do nothing.
template <int T, int R>
__device__ __forceinline__ void map_run(const uint16_t *keys, long long i, long long e,
                                        const uint16_t *src, uint16_t *dst, uint32_t n, uint32_t tid) {
    if ((tid & ~31u) >= n) return;
    uint32_t X[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t j = tid + T * r;
        X[r] = j < n ? (uint32_t)__ldcg(src + j) : (uint32_t)O1_M;
    }
    auto step = [&](const uint2 &en) {
        uint32_t v, nb;
#pragma unroll
        for (int r = 0; r < R; r++) X[r] = EncTables::next(X[r], en, v, nb);
    };
    auto one = [&](long long j) { step(EncTables::transform(__ldg(keys + j))); };
    for (; i >= e && (i & 7) != 7; i--) one(i);
    if (i - 7 >= e) {
        const uint4 *kv = reinterpret_cast<const uint4 *>(keys);
        const uint4 z = make_uint4(0, 0, 0, 0);
        auto load = [&](long long j) { return j >= e ? __ldg(kv + (j >> 3)) : z; };
        auto eight = [&](uint4 &v) {  // a ring of three vectors, as in walk_records
            const uint32_t k[8] = {v.w >> 16, v.w & 0xFFFFu, v.z >> 16, v.z & 0xFFFFu,
                                   v.y >> 16, v.y & 0xFFFFu, v.x >> 16, v.x & 0xFFFFu};
            uint2 en[8];
#pragma unroll
            for (int j = 0; j < 8; j++) en[j] = EncTables::transform(k[j]);
            v = load(i - 24);
#pragma unroll
            for (int j = 0; j < 8; j++) step(en[j]);
            i -= 8;
        };
        uint4 v0 = load(i), v1 = load(i - 8), v2 = load(i - 16);
        for (;;) {
            eight(v0);
            if (i - 7 < e) break;
            eight(v1);
            if (i - 7 < e) break;
            eight(v2);
            if (i - 7 < e) break;
        }
    }
    for (; i >= e; i--) one(i);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t j = tid + T * r;
        if (j < n) __stcg(dst + j, (uint16_t)X[r]);
    }
}

template <int W>
__global__ void __launch_bounds__(kEncThreads) k_o1_maps(const EncArgs A, const MapArgs M) {
    extern __shared__ uint4 smem_raw[];
    constexpr uint32_t T = 32 * W;
    __shared__ uint32_t s_cnt[kEncThreads / 32];
    if (!map_path(A)) return;
    const EncCta w = M.ctas[blockIdx.x];
    load_image(smem_raw, A.image, w.table);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, tid = threadIdx.x % T, grp = threadIdx.x / T, wid = tid >> 5;
    const unsigned bar = 1 + grp;
    for (uint32_t it = grp; it < w.count; it += kEncThreads / T) {
        const uint32_t sid = w.first + it;
        uint32_t chain = w.chain, ch = A.nchains;
        while (ch - chain > 1) {
            const uint32_t mid = (chain + ch) >> 1;
            if (__ldg(M.sstart + mid) <= sid) chain = mid;
            else ch = mid;
        }
        const uint32_t nparts = __ldg(A.pstart + chain + 1) - __ldg(A.pstart + chain);
        const uint32_t p0 = (sid - __ldg(M.sstart + chain)) * M.spp, p1 = min(p0 + M.spp, nparts);
        const long long lo = (long long)A.chains[chain].lo, hi = (long long)A.chains[chain].hi;
        const bool is_top = p1 == nparts;
        uint16_t *ws = M.scratch + (size_t)sid * M.cap, *tmp = ws + M.cap - O1_M;
        uint32_t *hd = M.hdr + (size_t)sid * kMapHdr;
        const uint32_t room = M.cap - O1_M;
        // the chain's top super part has one entering state, the exact initial one
        uint32_t C = is_top ? 1u : (uint32_t)O1_M, at = 0, merges = 0, early = 0, C0 = 0;
        const uint16_t *cur = nullptr;
        if (is_top) {
            if (tid == 0) __stcg(ws, (uint16_t)EncTables::init(__ldg(A.keys + hi - 1)));
            cur = ws;
            at = 1;
            map_sync<W>(bar);
        }
        long long i = is_top ? hi - 2 : lo + (long long)p1 * A.part - 1;
        const long long start = i;
        uint32_t p = p1 - 1;  // the part being coded
        bool ok = true;
        for (;;) {
            const long long bottom = lo + (long long)p * A.part;
            long long e = bottom;
            if (C > 1 && p + 1 == p1) {  // early merges within the first part
                const long long done = start - i;
                const long long t = done < 8 ? 8 : done < 512 ? 2 * done : 0;
                if (t && start - t + 1 > bottom) e = start - t + 1;
            }
            for (uint32_t b = 0; b < C; b += 8 * T) {
                const uint32_t n = min(C - b, 8u * T);
                const uint16_t *src = cur ? cur + b : tmp + b;
                if (!cur) {  // all states
                    for (uint32_t j = tid; j < n; j += T) __stcg(tmp + b + j, (uint16_t)(O1_M + b + j));
                    map_sync<W>(bar);
                }
                if (n <= T) map_run<T, 1>(A.keys, i, e, src, tmp + b, n, tid);
                else if (n <= 2 * T) map_run<T, 2>(A.keys, i, e, src, tmp + b, n, tid);
                else if (n <= 4 * T) map_run<T, 4>(A.keys, i, e, src, tmp + b, n, tid);
                else map_run<T, 8>(A.keys, i, e, src, tmp + b, n, tid);
            }
            map_sync<W>(bar);
            // merge equal neighbours: every warp takes a run of whole 32s
            const uint32_t per = (C + T - 1) / T * 32, j0 = min(C, wid * per), j1 = min(C, j0 + per);
            auto kept = [&](uint32_t j) {  // lanes whose state differs from the one before it
                const uint32_t v = j + lane < j1 ? (uint32_t)__ldcg(tmp + j + lane) : 0u;
                uint32_t prev = __shfl_up_sync(0xffffffffu, v, 1);
                if (lane == 0) prev = j > 0 ? (uint32_t)__ldcg(tmp + j - 1) : 0u;  // 0 is no state
                return make_uint2(__ballot_sync(0xffffffffu, j + lane < j1 && v != prev), v);
            };
            uint32_t idx = 0, Cn = 0;
#pragma unroll 4
            for (uint32_t j = j0; j < j1; j += 32) Cn += __popc(kept(j).x);
            if (W > 1) {
                if (lane == 0) s_cnt[threadIdx.x >> 5] = Cn;
                map_sync<W>(bar);
                Cn = 0;
#pragma unroll
                for (uint32_t v = 0; v < W; v++) {
                    idx += v < wid ? s_cnt[grp * W + v] : 0u;
                    Cn += s_cnt[grp * W + v];
                }
            }
            const long long done = start - e + 1;
            if (at + C + Cn > room || (done >= 64 && Cn > 2048) || (done >= 1024 && Cn > 1024)) {
                ok = false;
                break;
            }
            uint16_t *map = ws + at, *list = map + C;
#pragma unroll 4
            for (uint32_t j = j0; j < j1; j += 32) {
                const uint2 k = kept(j);
                const uint32_t me = idx + __popc(k.x & ((2u << lane) - 1u)) - 1u;  // class of this lane's state
                if (j + lane < j1) {
                    __stcg(map + j + lane, (uint16_t)me);
                    if ((k.x >> lane) & 1u) __stcg(list + me, (uint16_t)k.y);
                }
                idx += __popc(k.x);
            }
            if (tid == 0) {
                hd[4 + 2 * merges] = at;
                hd[5 + 2 * merges] = at + C;
            }
            at += C + Cn;
            if (merges == 0) C0 = Cn;
            merges++;
            C = Cn;
            cur = list;
            map_sync<W>(bar);
            i = e - 1;
            if (e > bottom) {
                early++;
                continue;
            }
            if (p == p0) break;
            p--;
        }
        // the classes of the first merge, composed to the leaving state
        if (ok && at + C0 > room) ok = false;
        if (ok) {
            constexpr uint32_t kAhead = 8;  // chains of lookups in flight per thread
            for (uint32_t b = tid; b < C0; b += kAhead * T) {
                uint32_t idx[kAhead];
#pragma unroll
                for (uint32_t u = 0; u < kAhead; u++) idx[u] = min(b + u * T, C0 - 1);
                for (uint32_t m = 1; m < merges; m++) {
                    const uint16_t *map = ws + hd[4 + 2 * m];
#pragma unroll
                    for (uint32_t u = 0; u < kAhead; u++) idx[u] = __ldcg(map + idx[u]);
                }
                const uint16_t *last = ws + hd[5 + 2 * (merges - 1)];
#pragma unroll
                for (uint32_t u = 0; u < kAhead; u++)
                    if (b + u * T < C0) __stcg(ws + at + b + u * T, __ldcg(last + idx[u]));
            }
        }
        if (tid == 0) {
            hd[0] = ok;
            hd[1] = merges;
            hd[2] = early;
            hd[3] = at;
        }
        map_sync<W>(bar);
    }
}

constexpr int kComposeThreads = 256;
__global__ void __launch_bounds__(kComposeThreads) k_o1_compose(const EncArgs A, const MapArgs M,
                                                                const int *__restrict__ chain_table) {
    extern __shared__ uint4 smem_raw[];
    __shared__ uint16_t s_in[kEncThreads];  // entering state of every super part (at most one a part)
    if (!map_path(A)) return;
    const uint32_t chain = blockIdx.x, s0 = M.sstart[chain], ns = M.sstart[chain + 1] - s0;
    if (ns == 0) return;
    const uint32_t part0 = A.pstart[chain], nparts = A.pstart[chain + 1] - part0;
    bool bad = false;
    for (uint32_t s = threadIdx.x; s < ns; s += kComposeThreads) {
        // places of its first and its composed map (where the tables go, unless they are needed)
        const uint32_t *hd = M.hdr + (size_t)(s0 + s) * kMapHdr;
        reinterpret_cast<uint2 *>(smem_raw)[s] = make_uint2(hd[4], hd[3]);
        bad |= hd[0] == 0;
    }
    const bool walk = __syncthreads_or(bad);
    static_assert(kEncThreads * sizeof(uint2) <= kEncSmem, "the places fit the tables' space");
    if (walk) load_image(smem_raw, A.image, chain_table[chain]);
    __syncthreads();
    if (threadIdx.x == 0) {
        const long long lo = (long long)A.chains[chain].lo, hi = (long long)A.chains[chain].hi;
        uint32_t x = 0;
        for (uint32_t s = ns; s-- > 0;) {
            s_in[s] = (uint16_t)x;
            const uint16_t *ws = M.scratch + (size_t)(s0 + s) * M.cap;
            const bool is_top = s + 1 == ns;
            const uint32_t *hd = M.hdr + (size_t)(s0 + s) * kMapHdr;
            if (!walk || hd[0]) {
                const uint2 m = walk ? make_uint2(hd[4], hd[3]) : reinterpret_cast<const uint2 *>(smem_raw)[s];
                x = __ldcg(ws + m.y + __ldcg(ws + m.x + (is_top ? 0u : x - O1_M)));
                continue;
            }
            const uint32_t p0 = s * M.spp, p1 = min(p0 + M.spp, nparts);
            if (is_top) x = EncTables::init(__ldg(A.keys + hi - 1));
            for (uint32_t p = p1; p-- > p0;) {
                const long long a = lo + (long long)p * A.part;
                const bool tp = p + 1 == nparts;
                if (!tp) A.entry[part0 + p] = (uint16_t)x;
                walk_states(A.keys, tp ? hi - 2 : a + (long long)A.part - 1, a, x);
            }
        }
    }
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < ns; s += kComposeThreads) {
        const uint32_t *hd = M.hdr + (size_t)(s0 + s) * kMapHdr;
        if (!hd[0]) continue;
        const uint16_t *ws = M.scratch + (size_t)(s0 + s) * M.cap;
        const uint32_t p1 = min((s + 1) * M.spp, nparts), early = hd[2], merges = hd[1];
        uint32_t p = p1 - 1;
        A.entry[part0 + p] = s_in[s];
        uint32_t idx = s + 1 == ns ? 0u : (uint32_t)s_in[s] - O1_M;
        for (uint32_t m = 0; m + 1 < merges; m++) {
            idx = __ldcg(ws + hd[4 + 2 * m] + idx);
            if (m >= early) A.entry[part0 + --p] = __ldcg(ws + hd[5 + 2 * m] + idx);
        }
    }
}

// Whether a chain's rounds end after `round` for the maps' sake, by the parts it has left to run again: they fall by
// about the same factor from round to round, so those after rounds 4 and 8 tell how many more it takes; from
// there on, whether another chain's did.
__device__ __noinline__ bool rounds_too_many(const EncArgs &A, uint32_t round, bool need, uint32_t limit, int &left4) {
    if (round == 4) left4 = __syncthreads_count(need);
    if (round < 8) return false;
    if (round == 8) {
        const int left = __syncthreads_count(need);
        if (left > 1 && (left >= left4 || 8.f + 4.f * log2f((float)left) / log2f((float)left4 / (float)left) > (float)limit))
            return true;
    }
    return __syncthreads_or(threadIdx.x == 0 && __ldcg(A.err + 6) != 0);
}

// Rounds over the parts of this CTA's chain (one a thread, at most): a part runs again while the exit
// state of the part above is not the state it was last run from.  Returns whether all are settled after
// `limit` rounds; s_exit holds the exit states.  With FORECAST it may end after round 8: the parts left fall by about
// the same factor from round to round, so those after rounds 4 and 8 tell how many more it takes.
// (With 16 rounds for all: 100 M codes of which 48 % of the parts did not meet ran them and then the maps for 5
// chains of 176, 5.7 ms, where 29 rounds take 2.6; 384^3 float32 at REL 5e-3, where the parts left of three chains fall by
// 11 % a round, 4.5 ms, where 8 rounds tell and the maps follow, 3.7.)
template <bool FORECAST>
__device__ __forceinline__ bool repair_rounds(const EncArgs &A, uint32_t chain, int table, uint32_t limit,
                                              uint16_t *s_exit) {
    extern __shared__ uint4 smem_raw[];
    constexpr uint32_t kChanged = 0x8000u;  // bit 15 of an exit state: changed in the last round
    const uint32_t t = threadIdx.x, part0 = A.pstart[chain], nparts = A.pstart[chain + 1] - part0, id = part0 + t;
    const bool active = t < nparts;
    if (active) s_exit[t] = A.exit2[id];
    __syncthreads();
    bool need = t + 1 < nparts && s_exit[t + 1] != A.entry[id];
    if (!__syncthreads_or(need)) return true;
    load_image(smem_raw, A.image, table);
    __syncthreads();
    EncPartPos P{};
    uint32_t bits = 0, steps = 0;
    if (active) {
        P = enc_part(A, id, chain);
        bits = A.bits[id];
    }
    bool settled = false;
    int left4 = 0;
    for (uint32_t round = 1; round <= limit && !settled; round++) {
        uint32_t x = need ? s_exit[t + 1] & (kChanged - 1u) : 0u;
        __syncthreads();
        if (active) {
            uint32_t ex = s_exit[t] & (kChanged - 1u);
            if (need) {
                // a run that meets the kept states leaves as the run before it did
                A.entry[id] = (uint16_t)x;
                if (!rerun_part(A, P, x, A.column[id], bits, steps) && x != ex) ex = x | kChanged;
            }
            s_exit[t] = (uint16_t)ex;
        }
        if (t == 0) atomicMax(A.err + 3, (int)round);
        __syncthreads();
        need = t + 1 < nparts && (s_exit[t + 1] & kChanged);
        settled = !__syncthreads_or(need);
        if (FORECAST && !settled && round >= 4 && rounds_too_many(A, round, need, limit, left4)) break;
    }
    if (active) {
        s_exit[t] &= kChanged - 1u;
        A.exit2[id] = s_exit[t];
        A.bits[id] = bits;
    }
    if (steps) atomicAdd(A.err + 2, (int)steps);
    __syncthreads();
    return settled;
}

__global__ void __launch_bounds__(kEncThreads) k_o1_rounds(const EncArgs A, const int *__restrict__ chain_table) {
    __shared__ uint16_t s_exit[kEncThreads];
    if (many_unmet(A) || A.pstart[blockIdx.x + 1] == A.pstart[blockIdx.x]) return;
    if (!repair_rounds<true>(A, blockIdx.x, chain_table[blockIdx.x], A.max_rounds, s_exit) && threadIdx.x == 0)
        atomicAdd(A.err + 6, 1);
}

// A CTA per chain: every part's bit offset (the top part's bits come first), the decode checkpoints, and
// zeros in the words that k_o1_place merges.  (The rounds in front find nothing left to do.)
__global__ void __launch_bounds__(kEncThreads) k_o1_settle(const EncArgs A, const int *__restrict__ chain_table,
                                                          uint8_t *__restrict__ slots,
                                                          const unsigned long long *__restrict__ slot_off,
                                                          unsigned long long *__restrict__ blen,
                                                          O1Ckpt *__restrict__ cks,
                                                          const unsigned long long *__restrict__ ck_off,
                                                          uint32_t ck_every) {
    extern __shared__ uint4 smem_raw[];
    __shared__ uint16_t s_exit[kEncThreads];
    const uint32_t chain = blockIdx.x, t = threadIdx.x, part0 = A.pstart[chain];
    const uint32_t nparts = A.pstart[chain + 1] - part0;  // at most one a thread
    if (nparts == 0) {
        if (t == 0) blen[chain] = 0;
        return;
    }
    if (!repair_rounds<false>(A, chain, chain_table[chain], nparts + 2, s_exit) && t == 0) atomicExch(A.err, 5);
    const bool active = t < nparts;
    const uint32_t id = part0 + t;
    EncPartPos P{};
    uint32_t bits = 0, esc = 0;
    if (active) {
        P = enc_part(A, id, chain);
        bits = A.bits[id];
        esc = A.esc[id];
    }
    uint32_t *s_sum = reinterpret_cast<uint32_t *>(smem_raw);  // the tables are done with
    uint32_t total, esc_total;
    __syncthreads();
    const uint32_t below = block_excl_scan<uint32_t>(active ? bits : 0u, s_sum, total);
    const uint32_t esc_below = block_excl_scan<uint32_t>(active ? esc : 0u, s_sum + 32, esc_total);
    if (!active) return;
    const uint32_t off = total - below - bits;
    uint32_t *ow = reinterpret_cast<uint32_t *>(slots + slot_off[chain]);
    ow[off >> 5] = 0u;
    if (t == 0) {
        ow[total >> 5] = 0u;
        blen[chain] = ((unsigned long long)total + 7) / 8;
    }
    A.at[id] = slot_off[chain] * 8 + off;
    A.nrec[id] = (P.first < P.a ? 0u : (uint32_t)((P.first >> 3) - (P.a >> 3)) + 1u) | (t == 0 ? 0x80000000u : 0u);
    // decode checkpoint at every ck_every-th part start: the state the decoder holds before index a
    if (t > 0 && cks && t % ck_every == 0)
        cks[ck_off[chain] + t / ck_every - 1] =
            O1Ckpt{off + bits, esc_below, (uint16_t)(s_exit[t] - O1_M), (uint16_t)(__ldg(A.keys + P.a) >> 8)};
}

// Joins the parts' records in the slots, a warp per part and a record per lane: a warp scan of the bit
// counts gives every record its bit offset, the bits are merged in shared memory, and whole words leave
// coalesced; the part's first and last word, shared with its neighbours, by atomicOr (k_o1_settle zeroed
// them).  142 us for the 141 MB of a 512^3 field (2.9 TB/s with the records): bound by the issue of the
// merges.
constexpr int kPlaceWarps = 8;
constexpr uint32_t kPlaceWords = 32 * 104 / 32 + 2;  // 32 records, the word in front, one behind
__global__ void __launch_bounds__(kPlaceWarps * 32) k_o1_place(const EncArgs A, uint32_t *__restrict__ slots) {
    __shared__ uint32_t s_buf[kPlaceWarps][kPlaceWords];
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31u, id = blockIdx.x * kPlaceWarps + wid;
    if (id >= __ldg(A.pstart + A.nchains)) return;
    uint32_t *buf = s_buf[wid];
    const unsigned long long column = A.column[id], at = A.at[id];
    const uint32_t lanes = (uint32_t)(column >> 56), nr = A.nrec[id] & 0x7FFFFFFFu, nrec = nr + (A.nrec[id] >> 31);
    const uint4 *rec = A.rec + (column & ((1ULL << 56) - 1));
    uint32_t *o = slots + (at >> 5);
    uint32_t pos = (uint32_t)(at & 31u);  // bits in front of the next record in the words from o on
    bool shared_first = true;
    for (uint32_t z = lane; z < kPlaceWords; z += 32) buf[z] = 0u;
    auto load = [&](uint32_t r) -> uint4 {
        const uint32_t q = r < nr ? r : A.recs - 1;  // the final state's record comes last
        return r < nrec ? __ldcg(rec + (unsigned long long)q * lanes) : make_uint4(0, 0, 0, 0);
    };
    uint4 v = load(lane);
    __syncwarp();
    for (uint32_t r0 = 0; r0 < nrec; r0 += 32) {
        const uint4 nxt = load(r0 + 32 + lane);
        const uint32_t n = v.w >> 24, incl = warp_incl_scan(n), p = pos + incl - n;
        if (n) {
            const uint32_t w = p >> 5, sh = p & 31u, top = v.w & 0x00FFFFFFu, end = sh + n;
            atomicOr(buf + w, v.x << sh);
            if (end > 32) atomicOr(buf + w + 1, __funnelshift_l(v.x, v.y, sh));
            if (end > 64) atomicOr(buf + w + 2, __funnelshift_l(v.y, v.z, sh));
            if (end > 96) atomicOr(buf + w + 3, __funnelshift_l(v.z, top, sh));
            if (end > 128) atomicOr(buf + w + 4, __funnelshift_l(top, 0u, sh));
        }
        const uint32_t tot = pos + __shfl_sync(0xffffffffu, incl, 31), full = tot >> 5;
        __syncwarp();
        for (uint32_t z = lane; z < full; z += 32) {
            if (z == 0 && shared_first) atomicOr(o, buf[0]);
            else o[z] = buf[z];
        }
        __syncwarp();
        const uint32_t rest = buf[full];
        __syncwarp();
        for (uint32_t z = lane; z <= full; z += 32) buf[z] = 0u;
        __syncwarp();
        if (lane == 0) buf[0] = rest;
        __syncwarp();
        shared_first = shared_first && full == 0;
        o += full;
        pos = tot & 31u;
        v = nxt;
    }
    if (lane == 0 && pos) atomicOr(o, buf[0]);
}

// ---- chain decoder
// Decodes the parts of tANS chains, one part per thread: a part starts from the chain's checkpoint (bit
// position, state, context, escapes before it) or, part 0, from the stream's end; without checkpoints
// a chain is one part.  Each part that ends at a checkpoint checks that it arrived there; a mismatch sets err[1].
// Escapes are written as kEscape and filled in by k_o1_fill; only an escape's sign, which selects the next
// context, is read here.
//
// What bounds it: a part is a serial chain of lookups, so its time is the part's length times the
// step's latency where few parts share an SM, and issue slots and the shared-memory pipe where many do.  What
// a lane waits for, its whole warp waits for, so nothing on the chain may wait for memory beyond the SM:
//   * tables: 16 bits a cell and a word a chunk (k_o1_dtable) keep 13 of 15 contexts in shared memory and the
//     32 KiB of the two rarest mostly in L1 (with a word a cell 7 fit: 4 % of a 512^3 field's lookups then go to
//     L2, three warp steps of four among them; and where one table set codes levels of unlike statistics, a
//     part's busy contexts can be the rare ones of the whole: 1800 x 3600 points took 1.9 ms);
//   * stream bits: every lane keeps the 8-byte pieces around its position in registers, loaded two pieces
//     ahead; 64 bits are aligned for every 4 codes (at most 52 bits);
//   * signs: one bit an escape (k_sign_bits), a word ahead.
// Before (seven contexts of a word a cell, escapes and stream words read as they were needed) and now, with the
// fill: 64^3 points 216 -> 118 us, 1800 x 3600 2800 -> 900 us, 211 x 307 x 401 1110 -> 440 us, 384^3 float64 (87 %
// escapes) 3900 -> 975 us, 512^3 687 -> 595 us.
constexpr int kDecThreads = 1024;
constexpr uint32_t kDecWarps = 8;
constexpr int16_t kEscape = -128;  // no code: codes are within +-127
constexpr uint32_t kFillTile = 256;
constexpr uint32_t kCellSlots = 13;  // contexts whose cells are in shared memory; the chunks of all are
constexpr uint32_t kDecSmem = kCellSlots * O1_M * 2 + O1_NCTX * kChunks * 4;
static_assert(kDecSmem <= 227 * 1024, "the tables fit an SM's shared memory");
struct DecArgs {
    const uint8_t *in;
    const DecChain *chains;
    const uint32_t *pstart;  // first part of every chain, then the number of parts
    uint32_t nchains;
    const EncCta *ctas;
    const uint16_t *cells;
    const uint32_t *info;
    const DecRank *rank;
    const uint32_t *signs;     // sign bits of the escapes
    unsigned long long n_ovf;  // escapes
    const O1Ckpt *cks;
    unsigned long long part;   // codes per part
    int16_t *out;
    unsigned long long *tile;  // escapes before every kFillTile-th code
    int *err;
    int *over;                 // set by a chain with more escapes than `nesc`
};
__global__ void __launch_bounds__(kDecThreads) k_o1_decode_parts(const DecArgs A) {
    extern __shared__ uint4 smem_raw[];
    const EncCta w = A.ctas[blockIdx.x];
    const DecRank rk = A.rank[w.table];
    uint16_t *const cells = reinterpret_cast<uint16_t *>(smem_raw);
    uint32_t *const info = reinterpret_cast<uint32_t *>(cells + kCellSlots * O1_M);
    const size_t tab = (size_t)w.table * O1_NCTX;
    auto ctx_of = [&](uint32_t slot) { return (uint32_t)(rk.ctx >> (4 * slot)) & 15u; };
    auto slot_of = [&](uint32_t ctx) { return (uint32_t)(rk.slot >> (4 * ctx)) & 15u; };
    // the tables come in by all threads, however few decode
    for (uint32_t j = 0; j < kCellSlots; j++) {
        const uint4 *src = reinterpret_cast<const uint4 *>(A.cells + (tab + ctx_of(j)) * O1_M);
        for (uint32_t i = threadIdx.x; i < O1_M / 8; i += kDecThreads) smem_raw[j * (O1_M / 8) + i] = __ldg(src + i);
    }
    for (uint32_t i = threadIdx.x; i < O1_NCTX * kChunks; i += kDecThreads) {
        const uint32_t v = __ldg(A.info + (tab + ctx_of(i / kChunks)) * kChunks + i % kChunks);
        info[i] = (v & ~0xF0u) | (slot_of((v >> 4) & 15u) << 4);
    }
    __syncthreads();
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31u, it = wid * w.lanes + lane;
    if (lane >= w.lanes || it >= w.count) return;
    const uint32_t id = w.first + it;
    uint32_t c0 = w.chain, c1 = A.nchains;  // the chain of this part
    while (c1 - c0 > 1) {
        const uint32_t mid = (c0 + c1) >> 1;
        if (__ldg(A.pstart + mid) <= id) c0 = mid;
        else c1 = mid;
    }
    const DecChain ch = A.chains[c0];
    const uint32_t pt = id - __ldg(A.pstart + c0);
    const unsigned long long start = (unsigned long long)pt * A.part;
    if (ch.n == 0 || start >= ch.n || ch.inlen == 0 || ch.inlen >= (1ull << 28)) {
        atomicExch(A.err, 6);
        return;
    }
    const uint32_t n = (uint32_t)min(A.part, ch.n - start);
    const bool last = start + n >= ch.n;
    const uint8_t *const sb = A.in + ch.in;
    int32_t pos;                                                             // the stream's bits below it are unread
    uint32_t s = 0, slot, oi0 = 0;                                           // state (8192 ..), context's slot
    const uint32_t eend = last ? ch.nesc : A.cks[ch.ck + pt].esc;            // escapes up to the part's end
    if (pt == 0) {
        const uint8_t end = sb[ch.inlen - 1];
        if (end == 0) {
            atomicExch(A.err, 6);
            return;
        }
        pos = ((int32_t)ch.inlen - 1) * 8 + (int32_t)fse::highbit32(end);
        slot = slot_of(0);
    } else {
        const O1Ckpt k = A.cks[ch.ck + pt - 1];
        if (k.bitpos >= (uint32_t)ch.inlen * 8u || k.state >= O1_M || k.ctx >= O1_NCTX || k.esc > ch.nesc) {
            atomicExch(A.err + 1, 1);
            return;
        }
        pos = (int32_t)k.bitpos;
        s = O1_M + k.state;
        slot = slot_of(k.ctx);
        oi0 = k.esc;
    }
    BackWindow br;
    const int32_t bit0 = br.init(sb, ch.in, pos);
    if (pt == 0) {
        s = O1_M + br.take(O1_PB);
        br.align();
    }
    // ---- signs of the escapes from oi0 on: words k, k + 1 and k + 2 of the sign bits
    const unsigned long long e0 = ch.ovf + oi0;
    const uint32_t avail = (uint32_t)min((unsigned long long)(ch.nesc - oi0), A.n_ovf > e0 ? A.n_ovf - e0 : 0ull);
    const uint32_t *const sw = A.signs + (e0 >> 5);
    const uint32_t words = (uint32_t)((A.n_ovf + 31) / 32 - min((A.n_ovf + 31) / 32, e0 >> 5));
    auto sign_word = [&](uint32_t i) { return i < words ? __ldg(sw + i) : 0u; };
    uint32_t k = 0, w0 = sign_word(0), w1 = sign_word(1), w2 = sign_word(2), sgn;
    uint32_t oi = 0;
    const uint32_t e5 = (uint32_t)(e0 & 31);
    auto signs = [&]() {  // the next signs (at least 24) from bit 0 up
        const uint32_t b = e5 + oi;
        if ((b >> 5) != k) {
            k++;
            w0 = w1;
            w1 = w2;
            w2 = sign_word(k + 2);
        }
        sgn = __funnelshift_r(w0, w1, b);
    };
    signs();
    uint32_t seen = 0;  // bit 16: an escape where none was expected
    auto step = [&](auto esc_tag) -> uint32_t {  // one code: its chunk's word
        constexpr bool ESC = decltype(esc_tag)::value;
        uint32_t cell;
        if (slot < kCellSlots) cell = cells[(slot << O1_PB) + s - O1_M];
        else cell = __ldg(A.cells + (tab + ctx_of(slot)) * O1_M + s - O1_M);
        const uint32_t e = info[slot * kChunks + (cell & 511u)];
        const uint32_t ns = (e >> 18) + (cell >> 9), x = e & 15u, nb = 14u - x - (ns >> x);
        s = __funnelshift_l(br.hi, ns, nb);  // ns << nb with the next nb bits below
        br.skip(nb);
        slot = (e >> 4) & 15u;
        if (ESC) {
            const uint32_t esc = (e >> 16) & 1u;
            slot ^= esc & sgn;
            sgn >>= esc;
            oi += esc;
        } else {
            seen |= e;
        }
        return e;
    };
    int16_t *const o = A.out + ch.lo + start;
    const unsigned long long i0 = ch.lo + start;
    auto mark = [&](uint32_t j) {  // escapes before a tile's first code
        if (((i0 + j) & (kFillTile - 1)) == 0) A.tile[(i0 + j) / kFillTile] = e0 + oi;
    };
    auto single = [&](uint32_t j) {
        mark(j);
        o[j] = (int16_t)(int8_t)(step(std::true_type()) >> 8);
        br.align();
        signs();
    };
    // codes leave in aligned groups of eight (one 16-byte store) between a scalar head and tail
    uint32_t j = 0;
    for (; j < n && ((i0 + j) & 7); j++) single(j);
    auto eight = [&](auto esc_tag) {
        mark(j);
        if (decltype(esc_tag)::value) signs();
        uint32_t wv[4];
#pragma unroll
        for (int g = 0; g < 2; g++) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t x = step(esc_tag), y = step(esc_tag);
                // bytes 1 of both, sign-extended to 16 bits
                asm("prmt.b32 %0, %1, %2, 0xD591;" : "=r"(wv[2 * g + h]) : "r"(x), "r"(y));
            }
            br.align();
        }
        *reinterpret_cast<uint4 *>(o + j) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
        j += 8;
    };
    // where no lane of the warp is to meet an escape, a quarter of a step's instructions are left out
    if (__all_sync(__activemask(), oi0 + oi == eend)) {
        while (n - j >= 8) eight(std::false_type());
        if (seen & 0x10000u) atomicExch(A.cks ? A.err + 1 : A.over, 7);
    } else {
        while (n - j >= 8) eight(std::true_type());
    }
    signs();
    for (; j < n; j++) single(j);
    if (oi > avail) atomicExch(A.over, 7);
    if (!last) {
        const O1Ckpt k = A.cks[ch.ck + pt];
        if (k.state != s - O1_M || k.ctx != ctx_of(slot) || br.pos != bit0 + (int32_t)k.bitpos ||
            k.esc != oi0 + oi)
            atomicExch(A.err + 1, 1);
    } else if (br.pos < bit0 - 16) {
        atomicExch(A.err, 8);
    }
}

// Sign bits of the escape values: bit i of the bytes is value i's, a byte (a 16-byte vector) a thread.
__global__ void __launch_bounds__(256) k_sign_bits(const int16_t *__restrict__ v, unsigned long long n,
                                                   uint8_t *__restrict__ out) {
    const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (8 * i >= n) return;  // (the vector's values past the last are in the allocation's slack)
    const uint4 x = reinterpret_cast<const uint4 *>(v)[i];
    auto two = [](uint32_t w) { return ((w >> 15) & 1u) | ((w >> 30) & 2u); };
    out[i] = (uint8_t)(two(x.x) | (two(x.y) << 2) | (two(x.z) << 4) | (two(x.w) << 6));
}

// Fills in the escapes, a warp per kFillTiles tiles of 256 codes, 8 codes a lane: tile[t] is the number of
// escapes before a tile, so a warp scan gives every escape its value's place.  Bound by memory (the codes once
// in, and once out where a lane has an escape) and by issue: 143 us for 134 M codes, 14 % of them escapes.
constexpr uint32_t kFillTiles = 4;
__global__ void __launch_bounds__(256) k_o1_fill(int16_t *__restrict__ codes, long long n,
                                                 const unsigned long long *__restrict__ tile,
                                                 const int16_t *__restrict__ ovf, unsigned long long n_ovf,
                                                 const int2 *__restrict__ err) {
    const uint32_t lane = threadIdx.x & 31u;
    const long long t0 = ((long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5)) * kFillTiles;
    uint4 v[kFillTiles];
    unsigned long long at[kFillTiles];
#pragma unroll
    for (uint32_t k = 0; k < kFillTiles; k++) {
        const long long i0 = (t0 + k) * kFillTile + lane * 8;
        v[k] = i0 + 8 <= n ? *reinterpret_cast<const uint4 *>(codes + i0) : make_uint4(0, 0, 0, 0);
        at[k] = (t0 + k) * (long long)kFillTile < n ? tile[t0 + k] : 0;
    }
    // a part that gave up has written neither its codes nor its tiles, and the call fails or decodes again
    const int2 failed = *err;
    if (failed.x | failed.y) return;
#pragma unroll
    for (uint32_t k = 0; k < kFillTiles; k++) {
        const long long i0 = (t0 + k) * kFillTile + lane * 8;
        uint32_t wv[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
        if (i0 < n && i0 + 8 > n) {  // the last codes
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (i0 + u < n) wv[u >> 1] |= (uint32_t)(uint16_t)codes[i0 + u] << (16 * (u & 1));
        }
        uint32_t m[8], cnt = 0;  // which codes are escapes
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t x = wv[u] ^ 0xFF80FF80u;
            m[2 * u] = (x & 0xFFFFu) == 0;
            m[2 * u + 1] = x < 0x10000u;
            cnt += m[2 * u] + m[2 * u + 1];
        }
        const uint32_t incl = warp_incl_scan(cnt);
        if (cnt == 0) continue;
        const unsigned long long e = at[k] + incl - cnt;
        const int16_t *src = ovf + e;
        const bool have = e + cnt <= n_ovf;  // else a damaged stream: its values are not read
        uint32_t val[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            // a predicated load (a branch around each would cost as much again)
            val[u] = 0;
            asm("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p ld.global.nc.u16 %0, [%1];\n}"
                : "+r"(val[u])
                : "l"(src), "r"(have ? m[u] : 0u));
            src += m[u];
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t lo = m[2 * u] ? val[2 * u] : wv[u], hi = m[2 * u + 1] ? val[2 * u + 1] << 16 : wv[u];
            wv[u] = (lo & 0xFFFFu) | (hi & 0xFFFF0000u);
        }
        if (i0 + 8 <= n) {
            *reinterpret_cast<uint4 *>(codes + i0) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
        } else {
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (i0 + u < n) codes[i0 + u] = (int16_t)(wv[u >> 1] >> (16 * (u & 1)));
        }
    }
}

// Groups consecutive items (chains or parts) of one table into CTAs.  One CTA fills an SM (its
// tables take the shared memory), so the CTAs should be at most one per SM: every run of one table
// gets CTAs in proportion to its size (greedily, always to the run whose CTAs are largest), and
// a run's items are split evenly among its CTAs.  More items than SMs x max_per take several waves.
struct ItemRun {
    size_t first, len;
    int table;
};

// Runs of consecutive items with one table.
std::vector<ItemRun> table_runs(const std::vector<int> &chain_table) {
    std::vector<ItemRun> runs;
    const size_t n = chain_table.size();
    for (size_t i = 0; i < n;) {
        size_t j = i;
        while (j < n && chain_table[j] == chain_table[i]) j++;
        runs.push_back({i, j - i, chain_table[i]});
        i = j;
    }
    return runs;
}

std::vector<ChainCta> run_ctas(const std::vector<ItemRun> &runs, size_t n, size_t max_per) {
    std::vector<ChainCta> out;
    const size_t sms = (size_t)sm_count();
    std::vector<size_t> ctas(runs.size(), 1);
    if (runs.size() <= sms && n <= sms * max_per) {
        auto size_of = [&](size_t r) { return (runs[r].len + ctas[r] - 1) / ctas[r]; };
        for (size_t used = runs.size(); used < sms; used++) {
            size_t best = 0;
            for (size_t r = 1; r < runs.size(); r++)
                if (size_of(r) > size_of(best)) best = r;
            if (size_of(best) <= 1) break;
            ctas[best]++;
        }
    }
    for (size_t r = 0; r < runs.size(); r++) {
        size_t c = std::max<size_t>(ctas[r], (runs[r].len + max_per - 1) / max_per);
        c = std::min(c, runs[r].len);
        const int t = runs[r].table;
        for (size_t k = 0; k < c; k++) {
            const size_t a = runs[r].first + runs[r].len * k / c;
            const size_t b = runs[r].first + runs[r].len * (k + 1) / c;
            if (b > a) out.push_back(ChainCta{t, (int)a, (int)(b - a)});
        }
    }
    return out;
}

// The CTAs over the items of every chain: item start[c] is the first of chain c's, start.back() their number.
std::vector<EncCta> item_ctas(const std::vector<int> &chain_table, const std::vector<uint32_t> &start, size_t max_per) {
    std::vector<ItemRun> runs = table_runs(chain_table);
    for (auto &r : runs) r = ItemRun{start[r.first], start[r.first + r.len] - start[r.first], r.table};
    runs.erase(std::remove_if(runs.begin(), runs.end(), [](const ItemRun &r) { return r.len == 0; }), runs.end());
    std::vector<EncCta> out;
    if (runs.empty()) return out;
    for (const ChainCta &c : run_ctas(runs, start.back(), max_per)) {
        EncCta e{c.table, (uint32_t)c.first, (uint32_t)c.count, 1, 0, 0};
        e.chain = (uint32_t)(std::upper_bound(start.begin(), start.end(), e.first) - start.begin()) - 1;
        out.push_back(e);
    }
    return out;
}

void enable_big_smem() {
    // once per device (a set of flags, one bit per device ordinal below 64)
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    FB2_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return;
    FB2_CUDA(cudaFuncSetAttribute(k_o1_decode_parts, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDecSmem));
    for (const void *k : {(const void *)k_o1_walk<false>, (const void *)k_o1_walk<true>, (const void *)k_o1_repair,
                          (const void *)k_o1_maps<1>,
                          (const void *)k_o1_maps<4>, (const void *)k_o1_compose, (const void *)k_o1_rounds, (const void *)k_o1_settle})
        FB2_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEncSmem));
    FB2_CUDA(cudaFuncSetAttribute(k_o1_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHistSmem));
    done.fetch_or(bit, std::memory_order_acq_rel);
}

// The parts of every chain and the CTAs that code them.
struct ChainParts {
    std::vector<EncChain> chains;   // kMaxK a segment
    std::vector<int> table;         // table set of every chain
    std::vector<uint32_t> pstart, sstart;  // first part and first super part of every chain
    uint32_t spp = 1;               // parts per super part
    std::vector<EncCta> ctas, map_ctas;
    unsigned long long records = 0;
    size_t u_chains, u_table, u_pstart, u_sstart, u_ctas, u_map_ctas;  // the lists in an upload
    void add(Upload &up) {
        u_chains = up.add(chains);
        u_table = up.add(table);
        u_pstart = up.add(pstart);
        u_sstart = up.add(sstart);
        u_ctas = up.add(ctas);
        u_map_ctas = up.add(map_ctas);
    }
};
ChainParts chain_parts(const std::vector<SegInfo> &segs, const std::vector<int> &seg_region, int K, uint32_t part) {
    ChainParts cp;
    const size_t n = segs.size() * kMaxK;
    cp.pstart.assign(n + 1, 0);
    cp.sstart.assign(n + 1, 0);
    for (size_t c = 0; c < n; c++) {
        const SegInfo &sg = segs[c / kMaxK];
        const unsigned long long k = c % kMaxK, lo = sg.lo + k * sg.cs;
        const unsigned long long hi = k < (unsigned long long)K ? std::min(lo + sg.cs, sg.lo + sg.n) : lo;
        cp.chains.push_back({lo, std::max(lo, hi)});
        cp.table.push_back(seg_region[c / kMaxK]);
        cp.pstart[c + 1] = cp.pstart[c] + (hi > lo ? (uint32_t)((hi - lo + part - 1) / part) : 0);
    }
    // super parts: about eight an SM (the states of a super part's first codes cost as much as its next
    // 8 Ki codes), more where that would make them long
    while (cp.spp < kMaxSuper && cp.pstart[n] / cp.spp > (uint32_t)(sm_count() * 8)) cp.spp *= 2;
    for (size_t c = 0; c < n; c++)
        cp.sstart[c + 1] = cp.sstart[c] + (cp.pstart[c + 1] - cp.pstart[c] + cp.spp - 1) / cp.spp;
    cp.ctas = item_ctas(cp.table, cp.pstart, kEncThreads);
    cp.map_ctas = item_ctas(cp.table, cp.sstart, kEncThreads);
    for (EncCta &e : cp.ctas) {
        e.lanes = std::min(32u, (e.count + kEncWarps - 1) / kEncWarps);
        e.rec = cp.records;
        cp.records += (unsigned long long)((e.count + e.lanes - 1) / e.lanes) * e.lanes * part_records(part);
    }
    return cp;
}

void encode_chains(Pool &pool, const ChainParts &cp, const Upload &up, const uint16_t *keys, size_t N, const uint32_t *image, uint32_t part,
                   uint8_t *slots, const unsigned long long *d_soff, unsigned long long *blen, O1Ckpt *cks,
                   const unsigned long long *d_ck_off, uint32_t ck_every, int *d_err, cudaStream_t st) {
    const uint32_t nchains = (uint32_t)cp.chains.size(), nparts = cp.pstart.back(), nsuper = cp.sstart.back();
    const int *d_table = up.get<int>(cp.u_table);
    EncArgs A{};
    A.keys = keys;
    A.chains = up.get<EncChain>(cp.u_chains);
    A.pstart = up.get<uint32_t>(cp.u_pstart);
    A.nchains = nchains;
    A.part = part;
    A.recs = part_records(part);
    A.max_rounds = max_rounds(nparts);
    A.image = image;
    A.ctas = up.get<EncCta>(cp.u_ctas);
    uint16_t *p16 = pool.get<uint16_t>((size_t)nparts * 3);
    A.exit1 = p16;
    A.exit2 = p16 + nparts;
    A.entry = p16 + 2 * (size_t)nparts;
    uint32_t *p32 = pool.get<uint32_t>((size_t)nparts * 3);
    A.bits = p32;
    A.esc = p32 + nparts;
    A.nrec = p32 + 2 * (size_t)nparts;
    A.column = pool.get<unsigned long long>((size_t)nparts * 2);
    A.at = A.column + nparts;
    A.kept = pool.get<uint16_t>(2 * ((N >> kKeptShift) + 2));
    A.kept_bits = A.kept + (N >> kKeptShift) + 2;
    A.err = d_err;
    // The maps' scratch takes the records' place: the map path writes them anew after its maps are used.
    MapArgs M{};
    M.sstart = up.get<uint32_t>(cp.u_sstart);
    M.spp = cp.spp;
    M.cap = (uint32_t)(O1_M + 28 * 1024 + 320 * cp.spp);
    uint8_t *area = pool.get<uint8_t>(std::max((size_t)cp.records * sizeof(uint4), (size_t)nsuper * M.cap * 2));
    A.rec = reinterpret_cast<uint4 *>(area);
    M.scratch = reinterpret_cast<uint16_t *>(area);
    M.hdr = pool.get<uint32_t>((size_t)nsuper * kMapHdr);
    M.ctas = up.get<EncCta>(cp.u_map_ctas);
    enable_big_smem();
    const unsigned nc = (unsigned)cp.ctas.size();
    k_o1_walk<false><<<nc, kEncThreads, kEncSmem, st>>>(A);
    FB2_CHECK_LAUNCH();
    k_o1_repair<<<nc, kEncThreads, kEncSmem, st>>>(A);
    FB2_CHECK_LAUNCH();
    k_o1_rounds<<<nchains, kEncThreads, kEncSmem, st>>>(A, d_table);
    FB2_CHECK_LAUNCH();
    // a warp a super part where they fill the SMs' warps, four (the first codes' many states go faster)
    // where not: 6.5 M codes take 850 us with four and 1265 with one, 134 M 11.7 and 3.9 ms
    if (nsuper > (uint32_t)sm_count() * kEncThreads / 128)
        k_o1_maps<1><<<(unsigned)cp.map_ctas.size(), kEncThreads, kEncSmem, st>>>(A, M);
    else
        k_o1_maps<4><<<(unsigned)cp.map_ctas.size(), kEncThreads, kEncSmem, st>>>(A, M);
    FB2_CHECK_LAUNCH();
    k_o1_compose<<<nchains, kComposeThreads, kEncSmem, st>>>(A, M, d_table);
    FB2_CHECK_LAUNCH();
    k_o1_walk<true><<<nc, kEncThreads, kEncSmem, st>>>(A);
    FB2_CHECK_LAUNCH();
    k_o1_settle<<<nchains, kEncThreads, kEncSmem, st>>>(A, d_table, slots, d_soff, blen, cks, d_ck_off, ck_every);
    FB2_CHECK_LAUNCH();
    k_o1_place<<<(nparts + kPlaceWarps - 1) / kPlaceWarps, kPlaceWarps * 32, 0, st>>>(
        A, reinterpret_cast<uint32_t *>(slots));
    FB2_CHECK_LAUNCH();
}

// Sum of the per-segment histograms of each table region (segments [rs[r], rs[r+1])).
__global__ void k_region_hist(const uint32_t *__restrict__ seg_hist, const int *__restrict__ rs,
                              uint32_t *__restrict__ reg_hist) {
    const int r = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= O1_NCTX * O1_NSYM) return;
    uint32_t s = 0;
    for (int g = rs[r]; g < rs[r + 1]; g++) s += seg_hist[(size_t)g * O1_NCTX * O1_NSYM + i];
    reg_hist[(size_t)r * O1_NCTX * O1_NSYM + i] = s;
}

// Sixteen codes of a thread in eight words (16-byte vectors when the code array is 16-byte aligned: tile starts
// are multiples of 16 codes), zeros past the end, and which of them are escapes (bit j: code j).  An escape is
// what clamping to -127 .. 127 changes, two codes at a time.
__device__ __forceinline__ uint32_t escape_mask(const int16_t *__restrict__ q, long long n, long long base,
                                                uint32_t (&w)[8]) {
    static_assert(kScanItems == 16, "two 16-byte vectors per thread");
    if (base + kScanItems <= n && (reinterpret_cast<uintptr_t>(q) & 15) == 0) {
        const uint4 *p4 = reinterpret_cast<const uint4 *>(q + base);
        const uint4 a = __ldg(p4), b = __ldg(p4 + 1);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
        w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const long long i = base + 2 * k;
            w[k] = (i < n ? (uint32_t)(uint16_t)q[i] : 0u) | (i + 1 < n ? (uint32_t)(uint16_t)q[i + 1] << 16 : 0u);
        }
    }
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t d = __vmins2(__vmaxs2(w[k], 0xFF81FF81u), 0x007F007Fu) ^ w[k];
        if (d & 0xFFFFu) m |= 1u << (2 * k);
        if (d >> 16) m |= 2u << (2 * k);
    }
    return m;
}

__global__ void __launch_bounds__(kScanThreads) k_esc_tiles(const int16_t *__restrict__ q, long long n,
                                                           uint32_t *__restrict__ cnt) {
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    uint32_t w[8];
    const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(escape_mask(q, n, base, w)));
    __shared__ uint32_t total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    if ((threadIdx.x & 31u) == 0 && c) atomicAdd(&total, c);
    __syncthreads();
    if (threadIdx.x == 0) cnt[blockIdx.x] = total;
}

// Escapes before each of npos code positions: the tile offset of the position's tile (exclusive
// scan of the tile counts) plus the escapes of the tile before the position, one warp per position.
__global__ void __launch_bounds__(256) k_esc_before(const int16_t *__restrict__ q,
                                                    const uint32_t *__restrict__ tile_off,
                                                    const unsigned long long *__restrict__ pos, int npos,
                                                    unsigned long long *__restrict__ out) {
    const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = (int)(threadIdx.x & 31u);
    if (w >= npos) return;
    const unsigned long long p = pos[w], t = p / kScanTile;
    uint32_t c = 0;
    uint32_t v[8];
    for (unsigned long long i = t * kScanTile + kScanItems * lane; i < p; i += 32 * kScanItems)
        c += (uint32_t)__popc(escape_mask(q, (long long)p, (long long)i, v));
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) out[w] = (unsigned long long)tile_off[t] + c;
}

// The escapes in index order, and their classes.  Bound by issue: testing the codes as symbols, twice, took 33
// instructions a code (134 M codes: 183 us; k_esc_tiles 62), the masks take 97 (56).
__global__ void __launch_bounds__(kScanThreads) k_esc_extract(const int16_t *__restrict__ q, long long n,
                                                             const uint32_t *__restrict__ tile_off,
                                                             uint8_t *__restrict__ cls, int16_t *__restrict__ raw) {
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    uint32_t w[8];
    const uint32_t m = escape_mask(q, n, base, w);
    __shared__ uint32_t sh[32];
    // the tile's escapes are staged in shared memory in order, then leave as contiguous runs
    __shared__ int16_t sv[kScanTile];
    uint32_t tot;
    int16_t *at = sv + block_excl_scan<uint32_t>((uint32_t)__popc(m), sh, tot);
    if (m) {
#pragma unroll
        for (int j = 0; j < kScanItems; j++)
            if ((m >> j) & 1u) *at++ = (int16_t)(j & 1 ? w[j >> 1] >> 16 : w[j >> 1] & 0xFFFFu);
    }
    __syncthreads();
    const uint32_t t0 = tile_off[blockIdx.x];
    for (uint32_t k = threadIdx.x; k < tot; k += blockDim.x) {
        const int16_t e = sv[k];
        cls[t0 + k] = (uint8_t)(31 - __clz(gamma_value(e)));
        raw[t0 + k] = e;
    }
}

__global__ void k_m0_scatter(const uint32_t *__restrict__ runs, const uint32_t *__restrict__ vals,
                             const unsigned long long *__restrict__ start, long long nv, long long n,
                             int16_t *__restrict__ out) {
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < nv; j += (long long)gridDim.x * blockDim.x) {
        const unsigned long long pos = start[j] + runs[j] - 1;
        if ((long long)pos < n) out[pos] = (int16_t)unzz(vals[j] - 1u);
    }
}

__global__ void k_sample_windows(const int16_t *__restrict__ q, const unsigned long long *__restrict__ off, int nw,
                                 int wl, int16_t *__restrict__ outp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nw * wl) outp[i] = q[off[i / wl] + (i % wl)];
}

// Decodes gamma groups whose class streams are fse_enc records in host-visible bytes `h`
// (also present on the device at `d`).  vals must hold the group totals.
void gamma_decode(Pool &pool, const uint8_t *d, const ByteView &h,
                  const std::vector<size_t> &cls_off, const std::vector<size_t> &man_off,
                  const std::vector<size_t> &man_len, const std::vector<unsigned long long> &gstart,
                  uint32_t *d_vals, int *d_err, cudaStream_t st, const FseCkpt *d_fck = nullptr,
                  uint32_t fpart = 0, unsigned long long n_fck = 0, const std::vector<unsigned long long> &gdst = {},
                  int16_t *d_ovf = nullptr) {
    const int G = (int)gstart.size() - 1;
    const long long T = (long long)gstart.back();
    if (T == 0) return;
    std::vector<BlockJob> jobs;
    for (int g = 0; g < G; g++) parse_blocks(h, cls_off[g], gstart[g + 1] - gstart[g], gstart[g], jobs);
    if (d_fck && fpart) {
        // the checkpoints belong to the FSE-coded blocks in stream order
        unsigned long long used = 0;
        for (auto &j : jobs)
            if (j.flag == 1) {
                const uint32_t c = fse_ckpt_count(j.n, fpart);
                j.ck = c ? (uint32_t)used : 0xFFFFFFFFu;
                used += c;
            }
        if (used != n_fck)
            for (auto &j : jobs) j.ck = 0xFFFFFFFFu;
    }
    std::vector<unsigned long long> gman(G), glen(G), ust(G + 1, 0);
    for (int g = 0; g < G; g++) {
        gman[g] = man_off[g];
        glen[g] = man_len[g];
        ust[g + 1] = ust[g] + (gstart[g + 1] - gstart[g] + kUnit - 1) / kUnit;
    }
    const unsigned long long NU = ust[G];
    Upload up;
    const size_t u_jobs = up.add(jobs), u_gstart = up.add(gstart), u_gman = up.add(gman), u_glen = up.add(glen),
                 u_ust = up.add(ust), u_gdst = up.add(gdst);
    up.send(pool, st);
    const BlockJob *dj = up.get<BlockJob>(u_jobs);
    const unsigned long long *d_gstart = up.get<unsigned long long>(u_gstart), *d_gman = up.get<unsigned long long>(u_gman),
                             *d_glen = up.get<unsigned long long>(u_glen), *d_ust = up.get<unsigned long long>(u_ust),
                             *d_gdst = gdst.empty() ? nullptr : up.get<unsigned long long>(u_gdst);
    uint8_t *cls = pool.get<uint8_t>(T);
    enable_fse_smem();
    const uint32_t dpart = fpart ? fpart : FBLK;
    k_fse_decode_blocks<<<(unsigned)jobs.size(), kFseDecThreads, fse_dec_smem(dpart), st>>>(d, dj, cls, d_err, dpart, d_fck);
    FB2_CHECK_LAUNCH();
    unsigned long long *usum = pool.get<unsigned long long>(NU + 1);
    unsigned long long *uoff = pool.get<unsigned long long>(NU + 1);
    void *sc = pool.get<uint8_t>(scan_scratch_bytes((long long)NU, 8));
    k_unit_bits<<<grid_for((long long)NU * 32, 256), 256, 0, st>>>(cls, d_gstart, d_ust, G, NU, usum);
    FB2_CHECK_LAUNCH();
    exclusive_scan<unsigned long long, unsigned long long>(usum, (long long)NU, uoff, sc, st);
    k_gamma_unpack_units<<<grid_for((long long)NU * 32, 256), 256, 0, st>>>(cls, d_gstart, d_ust, G, NU, uoff, d_gman,
                                                                           d, d_glen, d_vals, d_err, d_gdst, d_ovf);
    FB2_CHECK_LAUNCH();
}



}  // namespace

// ================================================================== public
EntropyChoice choose_entropy(Context &ctx, const int16_t *d_codes, size_t n, cudaStream_t st) {
    (void)ctx;
    // RleFseEncoder::preprocess_encode: 256 windows x 32 codes
    size_t NW = 256, WL = 32;
    if (n < NW * WL) {
        WL = n / NW;
        if (!WL) WL = 1;
    }
    size_t step = (n > NW * WL) ? (n - WL) / NW : WL;
    if (!step) step = 1;
    std::vector<unsigned long long> offs;
    for (size_t w = 0; w < NW; w++) {
        const size_t off = w * step;
        if (off + WL > n) break;
        offs.push_back(off);
    }
    EntropyChoice ch{0, false};
    size_t z = 0, zd = 0, cnt = 0, cntd = 0;
    if (!offs.empty()) {
        Pool pool(st);
        unsigned long long *d_off = h2d(pool, offs, st);
        int16_t *d_s = pool.get<int16_t>(offs.size() * WL);
        const int tot = (int)(offs.size() * WL);
        k_sample_windows<<<(tot + 255) / 256, 256, 0, st>>>(d_codes, d_off, (int)offs.size(), (int)WL, d_s);
        FB2_CHECK_LAUNCH();
        std::vector<int16_t> s = d2h(d_s, (size_t)tot, st);
        for (size_t w = 0; w < offs.size(); w++) {
            int16_t prev = s[w * WL];
            for (size_t t = 0; t < WL; t++) {
                const int16_t x = s[w * WL + t];
                if (x == 0) z++;
                if (t > 0 && x == prev) zd++;
                prev = x;
            }
            cnt += WL;
            cntd += WL - 1;
        }
    }
    const double p0 = cnt ? 1.0 * z / cnt : 1.0;
    const double dzeros = (cnt && cntd) ? (1.0 * zd / cntd - p0) : 0.0;
    ch.delta = dzeros > 0.005;
    ch.method = (p0 >= 0.80) ? 0 : 1;
    if (n < (size_t)20 * O1_NCTX * O1_NSYM) ch.method = 0;
    return ch;
}

void entropy_encode_into(Pool &pool, Assembler &as, const int16_t *d_codes_in, size_t n, const EntropyChoice &ch,
                         cudaStream_t st, const EntropyTuning &tune) {
    Trace tr("encode");
    const long long N = (long long)n;
    const int16_t *q = d_codes_in;
    if (ch.delta && N > 0) {
        int16_t *dq = pool.get<int16_t>(N);
        k_delta<<<grid_for(N, 256), 256, 0, st>>>(d_codes_in, N, dq);
        FB2_CHECK_LAUNCH();
        q = dq;
    }
    const uint8_t mb = (uint8_t)(ch.method | (ch.delta ? 0x80 : 0));
    CkptCollector cc;
    {
        const uint32_t part = tune.ckpt_part;
        const bool pow2 = part >= 64 && part <= (uint32_t)FBLK && (part & (part - 1)) == 0;
        cc.o1_part = cc.fse_part = pow2 ? part : 0;
    }
    as.val<uint8_t>(mb);
    as.val<uint16_t>(0);  // lo_
    as.val<uint16_t>(0);  // mode_
    if (ch.method == 0) {
        const long long tiles = std::max<long long>(1, (N + kScanTile - 1) / kScanTile);
        uint32_t *tcnt = pool.get<uint32_t>(tiles + 2);
        long long *tlast = pool.get<long long>(tiles + 2);
        FB2_CUDA(cudaMemsetAsync(tcnt, 0, (tiles + 2) * 4, st));
        if (N > 0) {
            k_m0_tiles<<<(unsigned)tiles, kScanThreads, 0, st>>>(q, N, tcnt, tlast);
            FB2_CHECK_LAUNCH();
        } else {
            FB2_CUDA(cudaMemsetAsync(tlast, 0xff, 8, st));
        }
        k_scan_small<uint32_t><<<1, 1024, 0, st>>>(tcnt, tiles);
        FB2_CHECK_LAUNCH();
        k_prefix_last<<<1, 1024, 0, st>>>(tlast, tiles);
        FB2_CHECK_LAUNCH();
        const uint32_t nv32 = d2h(tcnt + tiles, 1, st)[0];
        const long long lastnz = d2h(tlast + tiles, 1, st)[0];
        const unsigned long long nv = nv32;
        const bool trailing = N > 0 && lastnz < N - 1;
        const unsigned long long nr = nv + (trailing ? 1 : 0);
        uint32_t *buf = pool.get<uint32_t>(nr + nv + 2);  // runs [0, nr), values [nr, nr + nv)
        if (N > 0 && nv > 0) {
            k_m0_extract<<<(unsigned)tiles, kScanThreads, 0, st>>>(q, N, tcnt, tlast, buf, buf + nr);
            FB2_CHECK_LAUNCH();
        }
        if (trailing) {
            const uint32_t tr = (uint32_t)(N - 1 - lastnz + 1);  // L + 1
            FB2_CUDA(cudaMemcpyAsync(buf + nv, &tr, 4, cudaMemcpyHostToDevice, st));
            FB2_CUDA(cudaStreamSynchronize(st));
        }
        GammaOut go = gamma_encode(pool, buf, {0ULL, nr, nr + nv}, st, cc.fse_part);
        as.val<uint64_t>(nr);
        as.val<uint64_t>(nv);
        as.val<uint64_t>(go.cls_bytes[0]);
        as.val<uint64_t>(go.cls_bytes[1]);
        as.val<uint64_t>(go.man_bytes[0]);
        as.val<uint64_t>(go.man_bytes[1]);
        add_class_pieces(as, go, 0, &cc);
        add_class_pieces(as, go, 1, &cc);
        as.dev(go.man_ptr[0], go.man_bytes[0]);
        as.dev(go.man_ptr[1], go.man_bytes[1]);
    } else {
        // ---- segmentation: K chains per segment, S segments (decoder reads S and K from the stream)
        const int K = std::max(1, std::min(kMaxK, tune.o1_streams));
        // S segments as the reference sizes them, N / 8 Mi within [1, 16] (RleFseEncoder.hpp:582-587):
        // every segment carries its own 7.5 KiB table set, so few segments keep the payload as small
        // as the reference's; parallelism comes from the chains and their parts instead.
        long long S = tune.o1_segment > 0 ? std::max<long long>(1, (N + tune.o1_segment - 1) / tune.o1_segment)
                                          : std::min<long long>(16, std::max<long long>(1, N / (8LL << 20)));
        if (S > N) S = std::max<long long>(1, N);
        // every segment must be non-empty: an empty one ends after its N and K words
        while (S > 1 && (S - 1) * ((N + S - 1) / S) >= N) S--;
        const long long seg = (N + S - 1) / S;
        std::vector<SegInfo> segs(S);
        for (long long g = 0; g < S; g++) {
            const long long lo = g * seg;
            const long long hi = std::min<long long>(lo + seg, N);
            const long long ng = std::max<long long>(0, hi - lo);
            segs[g] = SegInfo{(unsigned long long)lo, (unsigned long long)ng,
                              (unsigned long long)((ng + K - 1) / K), K, 0};
        }
        // encoder part size, a power of two up to the decode checkpoint spacing: a chain's parts fit one
        // CTA's threads, and a part is shorter than the spacing where the parts would not give every SM
        // four full warps (a walk's time is then the length of a part: 64^3 codes 67 us in parts of 1024,
        // 38 in parts of 512), but not so short that a run seldom meets the kept states within it (parts of
        // 256: a walk of 25 us, but the rounds after it took 44 instead of 29, and a mean step the same)
        unsigned long long max_cs = 1;
        for (const auto &sg : segs) max_cs = std::max<unsigned long long>(max_cs, sg.cs);
        auto parts_of = [&](uint32_t part) { return (max_cs + part - 1) / part; };
        uint32_t enc_part = std::min<uint32_t>(cc.o1_part ? cc.o1_part : 1024u, 1024u);
        while (parts_of(enc_part) > (unsigned long long)kEncThreads) enc_part *= 2;
        if (cc.o1_part && cc.o1_part < enc_part) cc.o1_part = enc_part;
        while (enc_part > kMinEncPart && parts_of(enc_part / 2) <= (unsigned long long)kEncThreads &&
               N / enc_part < (long long)sm_count() * 128)
            enc_part /= 2;
        const uint32_t ck_every = cc.o1_part ? cc.o1_part / enc_part : 1u;
        // decode checkpoints of every chain: one before each index lo + q * part, q >= 1
        const long long nchains_all = S * kMaxK;
        std::vector<unsigned long long> ck_off(nchains_all + 1, 0);
        for (long long g = 0; g < S; g++)
            for (int k = 0; k < kMaxK; k++) {
                unsigned long long cnt = 0;
                if (k < K && cc.o1_part) {
                    const unsigned long long clo = segs[g].lo + (unsigned long long)k * segs[g].cs;
                    const unsigned long long chi = std::min(clo + segs[g].cs, segs[g].lo + segs[g].n);
                    if (chi > clo) cnt = (chi - clo - 1) / cc.o1_part;
                }
                ck_off[g * kMaxK + k + 1] = ck_off[g * kMaxK + k] + cnt;
            }
        cc.n_o1 = ck_off.back();
        O1Ckpt *o1ck = cc.n_o1 ? pool.get<O1Ckpt>(cc.n_o1) : nullptr;
        cc.o1 = o1ck;
        // table regions: segments whose statistics come from the same part of the code stream
        // share one table set (tune.regions holds the code positions where statistics change)
        std::vector<int> seg_region(S, 0), rs{0};
        if (tune.per_segment_tables) {
            for (long long g = 0; g < S; g++) seg_region[g] = (int)g;
            for (long long g = 1; g <= S; g++) rs.push_back((int)g);
        } else {
            int prev_rr = -1;
            for (long long g = 0; g < S; g++) {
                int rr = 0;
                for (long long b : tune.regions)
                    if (b > 0 && (unsigned long long)b <= segs[g].lo) rr++;
                if (g > 0 && rr != prev_rr) rs.push_back((int)g);
                seg_region[g] = (int)rs.size() - 1;
                prev_rr = rr;
            }
            rs.push_back((int)S);
        }
        const int R = (int)rs.size() - 1;
        // chain output slots
        std::vector<unsigned long long> soff(nchains_all + 1, 0);
        for (long long g = 0; g < S; g++)
            for (int k = 0; k < kMaxK; k++) {
                const unsigned long long c = (k < K) ? segs[g].cs * 2 + 64 : 0;
                soff[g * kMaxK + k + 1] = soff[g * kMaxK + k] + ((c + 15) & ~15ULL);
            }
        // the segments' starts and the end, before which the escapes are counted
        std::vector<unsigned long long> pos(S + 1, (unsigned long long)N);
        for (long long g = 0; g < S; g++) pos[g] = segs[g].lo;
        // what the kernels need to know of segments, chains and slots goes to the device in one copy
        Upload up;
        const size_t u_segs = up.add(segs), u_ck_off = up.add(ck_off), u_rs = up.add(rs),
                     u_soff = up.add(soff), u_pos = up.add(pos);
        ChainParts cp = chain_parts(segs, seg_region, K, enc_part);
        cp.add(up);
        up.send(pool, st);
        const SegInfo *d_segs = up.get<SegInfo>(u_segs);
        const unsigned long long *d_ck_off = o1ck ? up.get<unsigned long long>(u_ck_off) : nullptr;
        // the key counts, the chains' escape counts and the error words, cleared together; the last two and the
        // chains' lengths, read together at the end
        const size_t n_hist = (size_t)S * O1_NCTX * O1_NSYM, n_nvk = (size_t)nchains_all;
        uint32_t *hist = pool.get<uint32_t>(n_hist + n_nvk + 8 + 2 * n_nvk);
        uint32_t *nvk = hist + n_hist;
        int *d_err = reinterpret_cast<int *>(nvk + n_nvk);
        unsigned long long *blen = reinterpret_cast<unsigned long long *>(d_err + 8);
        uint16_t *keys = pool.get<uint16_t>((size_t)N + 8);
        FB2_CUDA(cudaMemsetAsync(hist, 0, (n_hist + n_nvk + 8) * 4, st));
        // The escape side stream (escape values in index order, their gamma classes, the FSE class
        // blocks) needs only the codes, so it forks before the histogram pass and runs next to it,
        // the table builds and the chain encoder.
        const long long tiles = std::max<long long>(1, (N + kScanTile - 1) / kScanTile);
        uint32_t *tcnt = pool.get<uint32_t>(tiles + 2);
        FB2_CUDA(cudaMemsetAsync(tcnt, 0, (tiles + 2) * 4, st));
        const bool fork = tune.side != nullptr && tune.fork_ev != nullptr && tune.join_ev != nullptr;
        cudaStream_t es = fork ? tune.side : st;
        if (fork) {
            FB2_CUDA(cudaEventRecord(tune.fork_ev, st));
            FB2_CUDA(cudaStreamWaitEvent(es, tune.fork_ev, 0));
        }
        struct Join {  // the calling stream waits for the second one before anything is freed
            bool on;
            cudaStream_t st, es;
            cudaEvent_t ev;
            void operator()() {
                if (on) {
                    cudaEventRecord(ev, es);
                    cudaStreamWaitEvent(st, ev, 0);
                    on = false;
                }
            }
            ~Join() { (*this)(); }
        } join{fork, st, es, tune.join_ev};
        Pool spool(es);  // scratch of the escape side stream, handed to `pool` once joined
        struct Hold {  // should a call fail: scratch of `es` that `st` reads is not given back before it is read
            bool on;
            cudaStream_t st, es;
            cudaEvent_t ev;
            ~Hold() {
                if (on) {
                    cudaEventRecord(ev, st);
                    cudaStreamWaitEvent(es, ev, 0);
                }
            }
        } hold{false, st, es, tune.fork_ev};
        if (N > 0) {
            k_esc_tiles<<<(unsigned)tiles, kScanThreads, 0, es>>>(q, N, tcnt);
            FB2_CHECK_LAUNCH();
        }
        k_scan_small<uint32_t><<<1, 1024, 0, es>>>(tcnt, tiles);
        FB2_CHECK_LAUNCH();
        // escapes before every segment start (the groups of the escape stream)
        unsigned long long *d_gstart = spool.get<unsigned long long>(S + 1);
        k_esc_before<<<(unsigned)((S + 1 + 7) / 8), 256, 0, es>>>(q, tcnt, up.get<unsigned long long>(u_pos), (int)(S + 1),
                                                                 d_gstart);
        FB2_CHECK_LAUNCH();
        tr.gpu("escape counts done", es);
        enable_big_smem();
        tr.gpu("histogram start", st);
        {
            // slices of a chain: at least 16 Ki codes (clearing and adding up its histogram costs a CTA as much
            // as 8 Ki codes), 4 Ki where the chains would leave SMs idle, and at most as many as fill whole waves
            // of two CTAs an SM, five at most.  (A CTA for every slice of all 16 chains had each chain's 1024 or
            // so codes a trip of their own: 1800 x 3600 points 41 us, now 18; 64^3 38, now 7.)
            const long long chains = S * K, wave = 2ll * sm_count();
            long long U = std::max<long long>(1, (long long)max_cs / 16384);
            while (chains * U < sm_count() && (long long)max_cs / U > 4096) U *= 2;
            if (chains * U > wave) U = std::max<long long>(1, std::min<long long>(5, chains * U / wave) * wave / chains);
            k_o1_hist<<<dim3((unsigned)S, (unsigned)(K * U)), 1024, kHistSmem, st>>>(
                q, d_segs, hist, nvk, keys, (reinterpret_cast<uintptr_t>(q) & 15) == 0);
        }
        FB2_CHECK_LAUNCH();
        tr.gpu("histogram done", st);
        uint32_t *rhist = hist;
        if (!tune.per_segment_tables) {
            rhist = pool.get<uint32_t>((size_t)R * O1_NCTX * O1_NSYM);
            const int *d_rs = up.get<int>(u_rs);
            k_region_hist<<<dim3((O1_NCTX * O1_NSYM + 255) / 256, R), 256, 0, st>>>(hist, d_rs, rhist);
            FB2_CHECK_LAUNCH();
        }
        const int ntab = R * O1_NCTX;
        uint16_t *nf = pool.get<uint16_t>((size_t)ntab * O1_NSYM);
        k_o1_norm<<<(ntab + 7) / 8, 256, 0, st>>>(rhist, ntab, nf);
        FB2_CHECK_LAUNCH();
        // the chain encoder's shared-memory image of every table set
        uint32_t *image = pool.get<uint32_t>((size_t)R * (kEncSmem / 4));
        k_o1_ctable<<<ntab, kTabThreads, 0, st>>>(nf, image, d_err);
        FB2_CHECK_LAUNCH();
        // escapes in index order, on the second stream (the host waits here for their count; the
        // histogram pass and the table builds, launched above, run meanwhile)
        const std::vector<unsigned long long> gstart = d2h(d_gstart, (size_t)S + 1, es);
        const unsigned long long E = gstart[S];
        uint8_t *ecls = spool.get<uint8_t>(E + 1);
        int16_t *eraw = spool.get<int16_t>(E + 1);
        if (E > 0) {
            k_esc_extract<<<(unsigned)tiles, kScanThreads, 0, es>>>(q, N, tcnt, ecls, eraw);
            FB2_CHECK_LAUNCH();
        }
        tr.gpu("escapes extracted", es);
        // the class blocks (long sequential chains) reach the GPU before the chain encoder, so that
        // they take a few SMs of their own instead of waiting for the chain encoder's last wave
        const bool queue_first = fork && tune.queued_ev != nullptr;
        const GammaBlocks gblocks = gamma_launch(spool, ecls, gstart, es, cc.fse_part,
                                                 queue_first ? tune.queued_ev : nullptr, cp.ctas.size(), chains_ns(N));
        tr.gpu("class blocks done", es);
        if (queue_first) FB2_CUDA(cudaStreamWaitEvent(st, tune.queued_ev, 0));
        tr.mark("class blocks launched");
        const unsigned long long *d_soff = up.get<unsigned long long>(u_soff);
        uint8_t *slots = pool.get<uint8_t>(soff.back() + 16);
        tr.mark("tables launched");
        tr.gpu("chain encoder start", st);
        encode_chains(pool, cp, up, keys, (size_t)N, image, enc_part, slots, d_soff, blen, o1ck, d_ck_off, ck_every, d_err, st);
        tr.gpu("chain encoder done", st);
        tr.mark("chains launched");
        // The mantissas go behind the one that is to end first, the chain encoder or the class blocks (whether the
        // chains take the map path, 0.9 ms at 6.5 M codes, is known on the device alone).  384^3 f64, 758 blocks
        // beside 56 M codes: behind the blocks 2.63 ms a call, behind the chains 2.50; 512^3 f32, where both take
        // as long, the same; 211 x 307 x 401 f32, 3 short blocks: 2.56 ms a round trip behind the blocks, 2.67
        // behind the chains.
        const bool behind_chains = queue_first && chains_ns(N) < gblocks.ns();
        cudaStream_t ms = behind_chains ? st : es;
        hold.on = behind_chains;
        const GammaWords gwords = gamma_pack(behind_chains ? pool : spool, ecls, gstart, eraw, ms);
        tr.gpu("escape mantissas packed", ms);
        GammaOut go = gamma_finish(gblocks, gwords, es, ms);
        // the chains' escape counts (stream header) from the histogram pass; their sums per segment
        // are the escape groups counted above
        const std::vector<uint32_t> ends = d2h(nvk, n_nvk + 8 + 2 * n_nvk, st);
        const uint32_t *h_nvk = ends.data();
        for (long long g = 0; g < S; g++) {
            unsigned long long e = 0;
            for (int k = 0; k < K; k++) e += h_nvk[g * kMaxK + k];
            if (e != gstart[g + 1] - gstart[g]) throw std::runtime_error("escape counts of the two passes differ");
        }
        tr.mark("escapes coded");
        int h_err[8];
        std::memcpy(h_err, h_nvk + n_nvk, sizeof(h_err));
        std::vector<unsigned long long> h_blen(n_nvk);
        std::memcpy(h_blen.data(), h_nvk + n_nvk + 8, n_nvk * 8);
        tr.gpu_dump();
        if (h_err[0]) throw std::runtime_error("tANS encoding failed (table construction or chain repair)");
        // Decode checkpoints cost 12 bytes each: keep them within 1.5 % of the chains' bytes by
        // keeping every m-th one (m a power of two; the decoder's parts become m times longer, so
        // streams whose codes take a few bits each, where the checkpoints weigh most, decode with
        // fewer, longer parts).
        if (cc.n_o1) {
            unsigned long long chain_bytes = 0;
            for (auto b : h_blen) chain_bytes += b;
            uint32_t m = 1;
            while (m < (1u << 16) && 12ull * (cc.n_o1 / m) * 1000 > 15 * chain_bytes) m *= 2;
            if (m > 1) {
                std::vector<unsigned long long> noff(nchains_all + 1, 0);
                const unsigned long long part2 = (unsigned long long)cc.o1_part * m;
                for (long long g = 0; g < S; g++)
                    for (int k = 0; k < kMaxK; k++) {
                        unsigned long long cnt = 0;
                        if (k < K) {
                            const unsigned long long clo = segs[g].lo + (unsigned long long)k * segs[g].cs;
                            const unsigned long long chi = std::min(clo + segs[g].cs, segs[g].lo + segs[g].n);
                            if (chi > clo) cnt = (chi - clo - 1) / part2;
                        }
                        noff[g * kMaxK + k + 1] = noff[g * kMaxK + k] + cnt;
                    }
                O1Ckpt *thin = noff.back() ? pool.get<O1Ckpt>(noff.back()) : nullptr;
                if (thin) {
                    unsigned long long *d_noff = h2d(pool, noff, st);
                    k_ck_thin<<<dim3(4, (unsigned)nchains_all), 256, 0, st>>>(o1ck, d_ck_off, d_noff,
                                                                            (int)nchains_all, m, thin);
                    FB2_CHECK_LAUNCH();
                }
                cc.o1 = thin;
                cc.n_o1 = noff.back();
                cc.o1_part = (uint32_t)part2;
            }
        }
        if (tr.on)
            std::fprintf(stderr, "[falcons trace] encode chain repair: %d codes re-run, %d rounds, %d of %u parts not met, %d chains unsettled; "
                         "%lld segments, %d chains each\n", h_err[2], h_err[3], h_err[5], cp.pstart.back(), h_err[6], S, K);
        tr.mark("chains done");
        join();
        pool.take(spool);
        hold.on = false;
        for (auto b : h_blen)
            if (b == ~0ULL) throw std::runtime_error("tANS chain overflow");
        as.val<uint64_t>((uint64_t)S);
        as.host.reserve(as.host.size() + (size_t)S * (16 + 16 * K + 32));
        as.pieces.reserve(as.pieces.size() + (size_t)S * (K + 8) + 64);
        for (long long g = 0; g < S; g++) {
            // the segment's header words (N, K, chain lengths, escape counts) in one piece
            uint64_t hw[2 + 2 * kMaxK];
            hw[0] = segs[g].n;
            hw[1] = (uint64_t)K;
            for (int k = 0; k < K; k++) hw[2 + k] = h_blen[g * kMaxK + k];
            for (int k = 0; k < K; k++) hw[2 + K + k] = h_nvk[g * kMaxK + k];
            as.bytes(hw, (size_t)(2 + 2 * K) * 8);
            as.dev(nf + (size_t)seg_region[g] * O1_NCTX * O1_NSYM, O1_NCTX * O1_NSYM * 2);
            for (int k = 0; k < K; k++) as.dev(slots + soff[g * kMaxK + k], h_blen[g * kMaxK + k]);
            const unsigned long long ne = gstart[g + 1] - gstart[g];
            if (ne == 0) {
                as.val<uint8_t>(0);
            } else {
                const size_t raw = ne * 2;
                const size_t cm = go.cls_bytes[g] + go.man_bytes[g] + 16;
                if (cm >= raw) {
                    as.val<uint8_t>(0);
                    as.dev(eraw + gstart[g], raw);
                } else {
                    as.val<uint8_t>(1);
                    as.val<uint64_t>(go.cls_bytes[g]);
                    as.val<uint64_t>(go.man_bytes[g]);
                    add_class_pieces(as, go, (int)g, &cc);
                    as.dev(go.man_ptr[g], go.man_bytes[g]);
                }
            }
        }
    }
    cc.emit(as);
}

size_t entropy_encode(Context &ctx, const int16_t *d_codes, size_t n, const EntropyChoice &ch, uint8_t *d_out,
                      size_t cap, cudaStream_t st, const EntropyTuning &tune) {
    (void)ctx;
    Pool pool(st);
    Assembler as;
    entropy_encode_into(pool, as, d_codes, n, ch, st, tune);
    if (as.pos > cap) throw std::length_error("The buffer for compressed data is not large enough.");
    as.run(pool, d_out, st);
    return (size_t)as.pos;
}

bool parse_ckpt_header(const uint8_t *h, const uint8_t *d_content, size_t avail, DecodeCheckpoints &out) {
    if (avail < kCkptHeader) return false;
    uint32_t w[4];
    uint64_t n1, n2;
    memcpy(w, h, 16);
    memcpy(&n1, h + 16, 8);
    memcpy(&n2, h + 24, 8);
    if (w[0] != kCkptTag || w[1] != kCkptVersion) return false;
    if (n1 > avail / sizeof(O1Ckpt) || n2 > avail / sizeof(FseCkpt)) return false;
    if (kCkptHeader + n1 * sizeof(O1Ckpt) + n2 * sizeof(FseCkpt) != avail) return false;
    out.d_o1 = d_content + kCkptHeader;
    out.n_o1 = n1;
    out.o1_part = w[2];
    out.d_fse = out.d_o1 + n1 * sizeof(O1Ckpt);
    out.n_fse = n2;
    out.fse_part = w[3];
    return true;
}

// `counts`: a chain's escape count in the header bounds its escapes; else it only says where its values start.
static size_t decode_payload(Context &ctx, const uint8_t *d_in, const ByteView &h, size_t n, int16_t *d_codes,
                             cudaStream_t st, const DecodeCheckpoints *ck, bool counts) {
    Trace tr("decode");
    Pool pool(st);
    tr.gpu("decode begin", st);
    // checkpoint arrays, copied to aligned scratch (their place in the stream has any alignment)
    auto pow2 = [](uint32_t v) { return v >= 64 && v <= (uint32_t)FBLK && (v & (v - 1)) == 0; };
    const O1Ckpt *o1ck = nullptr;
    const FseCkpt *fck = nullptr;
    uint32_t o1_part = 0, f_part = 0;
    unsigned long long n_o1ck = 0, n_fck = 0;
    if (ck && ck->n_o1 && ck->d_o1 && pow2(ck->o1_part) && ck->n_o1 < (1ULL << 32)) {
        O1Ckpt *d = pool.get<O1Ckpt>(ck->n_o1);
        launch_gather(pool, {Piece{ck->d_o1, 0, ck->n_o1 * sizeof(O1Ckpt)}}, reinterpret_cast<uint8_t *>(d), st);
        o1ck = d;
        o1_part = ck->o1_part;
        n_o1ck = ck->n_o1;
    }
    if (ck && ck->n_fse && ck->d_fse && pow2(ck->fse_part) && ck->n_fse < (1ULL << 32)) {
        FseCkpt *d = pool.get<FseCkpt>(ck->n_fse);
        launch_gather(pool, {Piece{ck->d_fse, 0, ck->n_fse * sizeof(FseCkpt)}}, reinterpret_cast<uint8_t *>(d), st);
        fck = d;
        f_part = ck->fse_part;
        n_fck = ck->n_fse;
    }
    const size_t len = h.len;
    size_t off = 0;
    const uint8_t mb = h.rd<uint8_t>(off);
    h.rd<uint16_t>(off);
    h.rd<uint16_t>(off);
    const bool delta = (mb & 0x80) != 0;
    const int method = mb & 0x7F;
    const long long N = (long long)n;
    int *d_err = pool.get<int>(4);
    FB2_CUDA(cudaMemsetAsync(d_err, 0, 16, st));
    if (method == 0) {
        const unsigned long long nr = h.rd<uint64_t>(off), nv = h.rd<uint64_t>(off);
        const unsigned long long s_rcl = h.rd<uint64_t>(off), s_vcl = h.rd<uint64_t>(off);
        const unsigned long long rbp = h.rd<uint64_t>(off), vbp = h.rd<uint64_t>(off);
        const size_t o_rcl = off, o_vcl = o_rcl + s_rcl, o_rman = o_vcl + s_vcl, o_vman = o_rman + rbp;
        const size_t end = o_vman + vbp;
        if (end > len || nv > (unsigned long long)N || nr > (unsigned long long)N + 1)
            throw std::invalid_argument("Invalid or truncated Falcons entropy payload");
        uint32_t *buf = pool.get<uint32_t>(nr + nv + 2);
        gamma_decode(pool, d_in, h, {o_rcl, o_vcl}, {o_rman, o_vman}, {(size_t)rbp, (size_t)vbp},
                     {0ULL, nr, nr + nv}, buf, d_err, st, fck, f_part, n_fck);
        FB2_CUDA(cudaMemsetAsync(d_codes, 0, (size_t)N * 2, st));
        if (nv > 0) {
            unsigned long long *start = pool.get<unsigned long long>(nr + 1);
            void *sc = pool.get<uint8_t>(scan_scratch_bytes((long long)nr, 8));
            exclusive_scan<uint32_t, unsigned long long>(buf, (long long)nr, start, sc, st);
            k_m0_scatter<<<grid_for((long long)nv, 256), 256, 0, st>>>(buf, buf + nr, start, (long long)nv, N,
                                                                      d_codes);
            FB2_CHECK_LAUNCH();
        }
        off = end;
    } else if (method == 1) {
        unsigned long long S = h.rd<uint64_t>(off);
        if (S == 0) S = 1;
        if (S > (unsigned long long)std::max<long long>(N, 1)) throw std::invalid_argument("invalid segment count");
        const unsigned long long seg = ((unsigned long long)N + S - 1) / S;
        // the decoder and the fill store codes as 16-byte vectors: for an output off 16 bytes they work on scratch
        const bool aligned = (reinterpret_cast<uintptr_t>(d_codes) & 15) == 0;
        int16_t *const out = aligned ? d_codes : pool.get<int16_t>((size_t)N);
        std::vector<DecChain> chains;
        std::vector<size_t> nf_off(S);
        std::vector<size_t> cls_off, man_off, man_len;
        std::vector<unsigned long long> gstart{0};
        std::vector<int> gseg;
        struct RawOvf {
            size_t off;
            unsigned long long n, dst;
        };
        std::vector<RawOvf> raws;
        unsigned long long ovf_total = 0;
        for (unsigned long long g = 0; g < S; g++) {
            const unsigned long long lo = g * seg;
            unsigned long long hi = lo + seg;
            if (hi > (unsigned long long)N) hi = N;
            const unsigned long long ng = hi > lo ? hi - lo : 0;
            h.rd<uint64_t>(off);  // stored N (the decoder uses the computed length)
            const unsigned long long K = h.rd<uint64_t>(off);
            if (ng == 0) continue;
            if (K < 1 || K > (unsigned long long)kMaxK) throw std::invalid_argument("invalid tANS stream count");
            const unsigned long long cs = (ng + K - 1) / K;
            unsigned long long bl[kMaxK], nk[kMaxK];
            for (unsigned long long k = 0; k < K; k++) bl[k] = h.rd<uint64_t>(off);
            for (unsigned long long k = 0; k < K; k++) nk[k] = h.rd<uint64_t>(off);
            nf_off[g] = off;
            off += O1_NCTX * O1_NSYM * 2;
            unsigned long long sp = off, tot_ov = 0;
            for (unsigned long long k = 0; k < K; k++) {
                const unsigned long long clo = lo + k * cs;
                unsigned long long chi = clo + cs;
                if (chi > hi) chi = hi;
                DecChain c{sp, bl[k], clo, chi > clo ? chi - clo : 0, ovf_total + tot_ov, (int)g,
                           (uint32_t)std::min<unsigned long long>(nk[k], 0xFFFFFFFFULL), 0, 0};
                chains.push_back(c);
                sp += bl[k];
                tot_ov += nk[k];
            }
            off = sp;
            if (off > len) throw std::invalid_argument("Invalid or truncated Falcons entropy payload");
            // escape block (decode_o1_ovf)
            const uint8_t mode = h.rd<uint8_t>(off);
            if (tot_ov > 0) {
                if (mode == 0) {
                    if (off + tot_ov * 2 > len) throw std::invalid_argument("truncated escape block");
                    raws.push_back(RawOvf{off, tot_ov, ovf_total});
                    off += tot_ov * 2;
                } else {
                    const unsigned long long s_vcl = h.rd<uint64_t>(off);
                    const unsigned long long vbp = h.rd<uint64_t>(off);
                    cls_off.push_back(off);
                    man_off.push_back(off + s_vcl);
                    man_len.push_back(vbp);
                    gstart.push_back(gstart.back() + tot_ov);
                    gseg.push_back((int)g);
                    // decoded values land at the group's position in a separate array, moved below
                    raws.push_back(RawOvf{~size_t(0), tot_ov, ovf_total});
                    off += s_vcl + vbp;
                    if (off > len) throw std::invalid_argument("truncated escape block");
                }
            }
            ovf_total += tot_ov;
        }
        for (unsigned long long g = 0; g < S; g++)
            if (nf_off[g] + O1_NCTX * O1_NSYM * 2 > len) throw std::invalid_argument("truncated tANS tables");
        tr.mark("segments parsed");
        // escape values, decoded on the side stream while this stream builds the decode tables
        // (raw blocks are copied; gamma groups are unpacked straight into their place)
        int16_t *ovf = pool.get<int16_t>(ovf_total + 1);
        uint32_t *signs = pool.get<uint32_t>(ovf_total / 32 + 1);
        SideFork fork(ctx, st);
        Pool spool(fork.side);
        {
            std::vector<Piece> pcs;
            std::vector<unsigned long long> conv_dst;
            for (auto &r : raws) {
                if (r.off != ~size_t(0)) pcs.push_back(Piece{d_in + r.off, r.dst * 2, r.n * 2});
                else conv_dst.push_back(r.dst);
            }
            if (!conv_dst.empty()) {
                gamma_decode(spool, d_in, h, cls_off, man_off, man_len, gstart, nullptr, d_err, fork.side, fck, f_part,
                             n_fck, conv_dst, ovf);
            }
            launch_gather(spool, pcs, reinterpret_cast<uint8_t *>(ovf), fork.side);
            if (ovf_total > 0) {
                k_sign_bits<<<(unsigned)((ovf_total + 2047) / 2048), 256, 0, fork.side>>>(ovf, ovf_total,
                                                                                         reinterpret_cast<uint8_t *>(signs));
                FB2_CHECK_LAUNCH();
            }
        }
        tr.gpu("escapes decoded", fork.side);
        tr.mark("escapes launched");
        // decode tables of every segment (segments that share counts build the same tables: no one waits
        // for a comparison)
        const uint32_t ntab = (uint32_t)S * O1_NCTX;
        uint16_t *nf = pool.get<uint16_t>((size_t)ntab * O1_NSYM);
        {
            std::vector<Piece> pcs;
            for (unsigned long long g = 0; g < S; g++) {
                const size_t at = nf_off[g] ? nf_off[g] : nf_off[0];  // an empty segment has no counts of its own
                pcs.push_back(Piece{d_in + at, g * O1_NCTX * O1_NSYM * 2, O1_NCTX * O1_NSYM * 2});
            }
            launch_gather(pool, pcs, reinterpret_cast<uint8_t *>(nf), st);
        }
        DecArgs A{};
        uint16_t *cells = pool.get<uint16_t>((size_t)ntab * O1_M);
        uint32_t *info = pool.get<uint32_t>((size_t)ntab * kChunks);
        DecRank *rank = pool.get<DecRank>(S);
        k_o1_dtable<<<ntab + (unsigned)S, kTabThreads, 0, st>>>(nf, ntab, cells, info, rank, d_err);
        FB2_CHECK_LAUNCH();
        tr.gpu("decode tables built", st);
        // checkpoint base of every chain; the checkpoints are used only if their count matches
        bool parts_ok = false;
        if (o1ck) {
            unsigned long long tot = 0;
            for (auto &c : chains) {
                c.ck = (uint32_t)tot;
                if (c.n) tot += (c.n - 1) / o1_part;
            }
            parts_ok = tot == n_o1ck;
        }
        if (!counts)
            for (auto &c : chains)
                c.nesc = (uint32_t)std::min<unsigned long long>(ovf_total - std::min(ovf_total, c.ovf), 0xFFFFFFFFull);
        // without checkpoints a chain is one part
        const unsigned long long part = parts_ok ? o1_part : kWholeChain;
        std::vector<uint32_t> pstart(chains.size() + 1, 0);
        std::vector<int> chain_table(chains.size());
        for (size_t i = 0; i < chains.size(); i++) {
            const unsigned long long np = chain_part_count(chains[i].n, parts_ok ? o1_part : 0);
            if (np == ~0ull) throw std::invalid_argument("tANS chain without checkpoints too long");
            pstart[i + 1] = pstart[i] + (uint32_t)np;
            chain_table[i] = chains[i].table;
        }
        std::vector<EncCta> ctas = item_ctas(chain_table, pstart, kDecThreads);
        for (auto &c : ctas) c.lanes = std::min(32u, (c.count + kDecWarps - 1) / kDecWarps);
        A.in = d_in;
        Upload up;
        const size_t u_chains = up.add(chains), u_pstart = up.add(pstart), u_ctas = up.add(ctas);
        up.send(pool, st);
        A.chains = up.get<DecChain>(u_chains);
        A.pstart = up.get<uint32_t>(u_pstart);
        A.nchains = (uint32_t)chains.size();
        A.ctas = up.get<EncCta>(u_ctas);
        A.cells = cells;
        A.info = info;
        A.rank = rank;
        A.signs = signs;
        A.n_ovf = ovf_total;
        A.cks = parts_ok ? o1ck : nullptr;
        A.part = part;
        A.out = out;
        A.tile = pool.get<unsigned long long>((size_t)N / kFillTile + 1);
        A.err = d_err;
        // without checkpoints, more escapes than the header counts have the payload decoded again without the counts
        A.over = counts && !parts_ok ? d_err + 1 : d_err;
        enable_big_smem();
        fork.join();  // the chains consume the escapes' signs
        tr.mark("parts listed");
        if (!ctas.empty()) {
            k_o1_decode_parts<<<(unsigned)ctas.size(), kDecThreads, kDecSmem, st>>>(A);
            FB2_CHECK_LAUNCH();
        }
        tr.gpu("chains decoded", st);
        if (ovf_total > 0) {
            const long long per = 8ll * kFillTiles * kFillTile;  // codes a CTA
            k_o1_fill<<<(unsigned)((N + per - 1) / per), 256, 0, st>>>(out, N, A.tile, ovf, ovf_total, reinterpret_cast<const int2 *>(d_err));
            FB2_CHECK_LAUNCH();
        }
        if (!aligned) FB2_CUDA(cudaMemcpyAsync(d_codes, out, (size_t)N * 2, cudaMemcpyDeviceToDevice, st));
    } else {
        throw std::invalid_argument("unsupported entropy method");
    }
    tr.mark("chains launched");
    tr.gpu("escapes filled in", st);
    if (delta) undelta(pool, d_codes, N, st);
    std::vector<int> he = d2h(d_err, 2, st);
    tr.gpu_dump();
    tr.mark("chains done");
    if (he[1] && ck) {
        // a checkpoint did not match the stream: decode again, sequentially
        if (tr.on) std::fprintf(stderr, "[falcons trace] decode checkpoint mismatch: decoding sequentially\n");
        return decode_payload(ctx, d_in, h, n, d_codes, st, nullptr, true);
    }
    if (he[1]) return decode_payload(ctx, d_in, h, n, d_codes, st, nullptr, false);
    if (he[0]) throw std::invalid_argument("Invalid or corrupted Falcons entropy payload");
    return off;
}

size_t entropy_decode(Context &ctx, const uint8_t *d_in, const ByteView &h, size_t n, int16_t *d_codes,
                      cudaStream_t st, const DecodeCheckpoints *ck) {
    return decode_payload(ctx, d_in, h, n, d_codes, st, ck, true);
}


}  // namespace fb2
