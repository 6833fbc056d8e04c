// BPE merge engine: exact Hugging Face merge order in a handful of data-parallel rounds.
//
// Hugging Face pops queue entries in (rank, position) order and skips an entry whose tokens were
// consumed.  A round here takes every pair whose rank is below B = min over the present ranks r of
// F[r], where F[r] is the lowest rank of any pair containing the token rank r creates: nothing
// created during the round can rank below B, so the round's outcome is the greedy matching of the
// candidate pairs in priority order.  On a path that choice has a closed form: follow the strictly
// improving priorities to the left and to the right of a candidate down to the local optimum; the
// candidate is taken iff both walks have even length.  The two parities are prefix-XORs along runs
// of set bits in two bit masks (32 positions per mask word): carry-propagating bit tricks inside a
// word, a carry handed from word to word.  Equal ranks on neighbouring pairs (runs of one token)
// fall out of the same rule because priority is (rank, position): every other pair from the left.
// Rounds repeat until no pair has a rank: 5-7 rounds for DNA words of any length.
//
// A table whose merge operands may be created by later ranks has no usable F; for it the host
// selects single_step: one merge per round, the leftmost pair of the lowest rank.
//
// Two kernels share that rule.
//
// bpe_lanes_kernel<W> (words up to 1,024 * W positions, W warps per word): every lane owns a
//   contiguous chunk of the word, at most 32 positions = one mask word, held as a column of a
//   slot-major token array in shared memory (slot j of lane g at j * (T + 2) + g, so that both
//   "all lanes read slot j" and "one lane walks its slots" are free of bank conflicts).  A lane
//   walks its chunk in a fully unrolled loop: tokens come from shared memory at compile-time
//   offsets, the looked-up entries stay in registers, the masks are built bit by bit in registers,
//   and nothing but the chunk borders, the carries and the compaction offsets crosses lanes.  After
//   the selection every surviving token is written to its new global position in the other buffer,
//   re-dealt so that all lanes again own equally many positions.
//
// Longer words are cut into overlapping windows that run bpe_lanes_kernel and are joined exactly (see BpeWindows).
//
// bpe_long_kernel (what the windows cannot join, and tables without batched rounds; one block of 32 warps per
//   word): the same round over arrays in global memory (tokens in place in the output area, ranks and masks in caller scratch),
//   position-parallel: lane i of a warp handles position 32 g + i and masks come from ballots.
//
// Merged tokens (uint16, Hugging Face ids) and per-row counts go to the caller's scratch; the emit
// kernels produce the final ids / mask layout.
//
// Same result as the rule the reference kernel states (src/dnatok_bpe_kernel/dnatok_bpe.cu:3-5,
// 172-176); that kernel walks the ranks one by one with per-rank bucket lists in global memory
// and one 256-thread block per sequence (:237-740).
#pragma once
#include "common.cuh"

namespace dnatok {

constexpr uint32_t BPE_NONE = 0xFFFFu;          // no rank
constexpr uint32_t BPE_FULL = 0xFFFFFFFFu;

// Length classes: class c < BPE_LONG_CLASS holds words of up to 1,024 << c positions and runs
// bpe_lanes_kernel<1 << c>; the last class holds everything longer and runs bpe_long_kernel.
constexpr int BPE_LANE_SLOTS = 32;              // positions one lane can own
constexpr int BPE_LONG_CLASS = 6;
constexpr int BPE_N_CLASSES = BPE_LONG_CLASS + 1;
constexpr int BPE_LONG_WARPS = 32;
constexpr int64_t BPE_MAX_POSITIONS = (int64_t)1 << 30;     // longest word of the long class
constexpr int BPE_WIN = 1024;                   // a window of a long word: what one warp holds ...
constexpr int BPE_WIN_OVERLAP = 128;            // ... and the positions it shares with the window after it
constexpr int BPE_WIN_STEP = BPE_WIN - BPE_WIN_OVERLAP;

__host__ __device__ constexpr int bpe_class_capacity(int c) { return (32 * BPE_LANE_SLOTS) << c; }
// warps per block for teams of W warps
__host__ __device__ constexpr int bpe_block_warps(int W) { return W < 8 ? 8 : W; }
// shared memory of one team: two token buffers, and for teams of several warps the exchange arrays
__host__ __device__ constexpr int bpe_team_bytes(int W) {
    return 2 * BPE_LANE_SLOTS * (32 * W + 2) * 2 + (W > 1 ? 32 * W * 8 : 0);
}
// caller scratch of one word of the long class: ranks (2 bytes per position) and three mask words per 32 positions
__host__ __device__ constexpr int64_t bpe_long_bytes(int64_t n) { return ((2 * n + 15) / 16 + 3 * ((n + 127) / 128)) * 16; }

struct BpeDeviceTable {
    const uint32_t* disp;        // [n_tokens] row displacement of the left token
    const uint2* slots;          // x = (rank << 16) | created, y = (left << 16) | F; all ones when empty
    const uint16_t* merge_out;   // [n_merges] token created by a rank
    const uint2* hot;            // [32 * 32] pairs of ids < 32: x as in slots, y = (F << 16) | rank; all ones when no merge
    const uint16_t* byte_tok;    // [256]
    int32_t single_step;
    uint32_t hot_ranks;          // every rank below this creates an id < 32
    uint32_t bytes_hot;          // 1: every initial symbol is an id < 32
    uint32_t filler;             // one past the largest token id: a token whose pairs never merge (disp and slots have room for it)
    const uint4* first;          // the first round in letters (BpeHostTable::first), NULL when there is none
    uint32_t first_hot;          // it creates small ids only
    // the table packed for shared memory (NULL when it does not exist): 16-bit displacements, 32-bit slots
    // (left << 16) | rank, one word (F << 16) | created id per rank
    const uint4* compact;
    uint32_t compact_bytes, compact_slot, compact_info, compact_last;
};

// Shared-memory addresses of the three parts of the packed table.
struct BpeSmemTable { uint32_t disp, slot, info, last; };

// One table entry: x = (rank << 16) | created id, y = (left id << 16) | F.  Ranks compare like the x
// words themselves (equal ranks create equal ids), so x is what the kernels keep per pair.  What
// the kernels work with is the pair (x, key), key = (F << 16) | rank: the minimum of the keys over a
// word gives the bound B (upper half) and tells whether any pair merges.  The table in shared
// memory holds (x, key) directly; an entry from global memory is checked against its left id first.
__device__ __forceinline__ uint2 bpe_cold_entry(const BpeDeviceTable& t, uint32_t a, uint32_t b) {
    uint2 s = __ldg(t.slots + __ldg(t.disp + a) + b);
    s.y = (s.y >> 16) == a ? __byte_perm(s.x, s.y, 0x5432) : BPE_FULL;
    if (s.y == BPE_FULL) s.x = BPE_FULL;
    return s;
}

constexpr int BPE_HOT_STRIDE = 36;              // row stride of the shared-memory table: the 16 pairs of four consecutive ids fall into 16 different banks
constexpr int BPE_HOT_WORDS = 33 * BPE_HOT_STRIDE;   // row and column 32 stay empty: 32 is the filler token behind the end of a word
constexpr uint32_t BPE_FILLER = 32;

// odd(i) = c(i) & ~odd(i-1), odd(-1) = 0: parity of the length of the run of set bits ending at
// each bit.
__device__ __forceinline__ uint32_t run_parity(uint32_t c) {
    const uint32_t se = c & ~(c << 1) & 0x55555555u;   // runs that start on an even bit
    const uint32_t fe = c & ~(c + se);                 // all bits of those runs
    const uint32_t fo = c & ~fe;
    return (fe & 0x55555555u) | (fo & 0xAAAAAAAAu);
}
// The run that starts at bit 0: with odd(-1) = 1 exactly its parities flip.
__device__ __forceinline__ uint32_t first_run(uint32_t c) { return c & ~(c + 1u); }

// Carry functions {0,1} -> {0,1} as two bits: bit 0 = f(0), bit 1 = f(1).
__device__ __forceinline__ uint32_t carry_apply(uint32_t f, bool x) { return (f >> (x ? 1 : 0)) & 1u; }
// first a, then b
__device__ __forceinline__ uint32_t carry_then(uint32_t a, uint32_t b) {
    return carry_apply(b, a & 1u) | (carry_apply(b, (a >> 1) & 1u) << 1);
}

// Run parities of one mask word per lane, the runs continuing from lane to lane: upwards
// (DOWN = false: bit `top` of lane l-1 precedes bit 0 of lane l) or downwards (DOWN = true: bit
// `top` of lane l+1 precedes bit 0 of lane l).  Every word holds top + 1 bits; `full` is the word
// with all of them set.  A word passes its incoming parity on only when all its bits are set;
// unless some lane has such a word the neighbour's own top bit is the carry and one shuffle
// replaces the scan over carry functions.
//
// chain_prepare does everything that does not depend on the parity entering the block of 32 lanes
// and returns the block's carry function (what leaves the block as a function of what enters);
// chain_finish takes the entering parity and gives the lane's parities.
struct ChainPrep {
    uint32_t odd0, fr;   // parities with nothing entering the word; the run they flip on when something does
    uint32_t f;          // fast: parity leaving the word; else: carry function from the block's entry to this word's exit
    bool fast;
};

// L: lanes of a segment; the lanes of a warp form 32 / L segments whose words are separate (L < 32: `lane` is the lane
// within its segment, and nothing enters a segment).
template <bool DOWN, int L = 32>
__device__ __forceinline__ ChainPrep chain_prepare(uint32_t c, int top, uint32_t full, int lane, uint32_t& block_fn) {
    ChainPrep p;
    p.odd0 = run_parity(c);
    p.fr = first_run(c);
    const uint32_t out0 = (p.odd0 >> top) & 1u;
    p.fast = __ballot_sync(BPE_FULL, c == full) == 0u;
    if (p.fast) {
        p.f = out0;
        if (L == 32) block_fn = __shfl_sync(BPE_FULL, out0, DOWN ? 0 : 31) * 3u;      // a constant function
    } else {
        uint32_t f = out0 | ((((p.odd0 ^ p.fr) >> top) & 1u) << 1);
#pragma unroll
        for (int d = 1; d < L; d <<= 1) {
            const uint32_t other = DOWN ? __shfl_down_sync(BPE_FULL, f, d, L) : __shfl_up_sync(BPE_FULL, f, d, L);
            if (DOWN ? lane + d < L : lane >= d) f = carry_then(other, f);     // the lanes before this one apply first
        }
        p.f = f;
        if (L == 32) block_fn = __shfl_sync(BPE_FULL, f, DOWN ? 0 : 31);
    }
    return p;
}

template <bool DOWN, int L = 32>
__device__ __forceinline__ uint32_t chain_finish(const ChainPrep& p, bool carry, int lane) {
    const uint32_t before = DOWN ? __shfl_down_sync(BPE_FULL, p.f, 1, L) : __shfl_up_sync(BPE_FULL, p.f, 1, L);
    const bool cin = (DOWN ? lane == L - 1 : lane == 0) ? carry : (p.fast ? before != 0u : carry_apply(before, carry) != 0u);
    return cin ? p.odd0 ^ p.fr : p.odd0;
}

// Both steps for blocks visited one after the other: `carry` enters the block and leaves it updated.
template <bool DOWN, int L = 32>
__device__ __forceinline__ uint32_t chain_parity(uint32_t c, int top, uint32_t full, bool& carry, int lane) {
    uint32_t fn = 0;
    const ChainPrep p = chain_prepare<DOWN, L>(c, top, full, lane, fn);
    const uint32_t odd = chain_finish<DOWN, L>(p, carry, lane);
    if (L == 32) carry = carry_apply(fn, carry) != 0u;
    return odd;
}

// Where the merge kernels leave a row's final token count (the count after truncation plus the special
// tokens), so that no separate pass over the rows is needed: lengths may be NULL.
struct BpeLengths {
    int32_t* lengths;
    int64_t cap_content;     // most content tokens a row may keep
    int32_t n_special;
    int32_t clip_is_error;   // rows cut by the output width (not by requested truncation) get DNATOK_ROW_CLIPPED
    // When ids is set the merge kernels also write every finished row in its final padded layout ([CLS] tokens
    // [SEP] padding, or the padding first), so no output pass follows; otherwise the tokens go to the scratch buffer.
    void* ids;
    void* mask;              // may be NULL
    int64_t out_stride;
    int32_t cls_id, sep_id, pad_id, pad_left;
    int32_t id_bits, mask_bits;
    // 1: the caller did not zero the status words: the kernel that sees a row first (the binning pass, or the merge
    // kernel when rows are not binned) writes the row's word instead of OR-ing into it
    int32_t store_status;
};
// A row's status bits into its word.
__device__ __forceinline__ void bpe_put_status(int32_t* status, int64_t row, int32_t bits, bool store) {
    if (!status) return;
    if (store) status[row] = bits;
    else if (bits) atomicOr(status + row, bits);
}
__device__ __forceinline__ int32_t bpe_put_length(const BpeLengths& L, int64_t row, int64_t n) {
    const int64_t kept = n < L.cap_content ? n : L.cap_content;
    if (L.lengths) L.lengths[row] = (int32_t)kept + L.n_special;
    return (L.clip_is_error && n > kept) ? 4 : 0;            // DNATOK_ROW_CLIPPED
}

// One finished row of n tokens into the caller's padded layout, the columns dealt to the T threads that worked on
// the row (g: this thread's index among them); tok(i) returns token i.
// i_lo, i_hi: only the columns of tokens [i_lo, i_hi); what precedes the first token and what follows the last
// one belong to the pieces that hold those.
template <typename TokFn>
__device__ __forceinline__ void bpe_write_row(const BpeLengths& L, int64_t row, int n, int g, int T, TokFn tok, int i_lo = 0,
                                              int i_hi = INT32_MAX) {
    const int stride = (int)L.out_stride;
    const int kept = n < L.cap_content ? n : (int)L.cap_content;
    const bool has_cls = L.cls_id >= 0, has_sep = L.sep_id >= 0;
    const int total = kept + (has_cls ? 1 : 0) + (has_sep ? 1 : 0);
    const int c0 = (L.pad_left ? stride - total : 0) + (has_cls ? 1 : 0);     // column of the first content token
    const int64_t base = row * L.out_stride;
    const int col_lo = i_lo > 0 ? c0 + i_lo : 0, col_hi = i_hi < n && c0 + i_hi < stride ? c0 + i_hi : stride;
    for (int col = col_lo + g; col < col_hi; col += T) {
        const int i = col - c0;
        int32_t v = L.pad_id;
        bool on = true;
        if (i >= 0 && i < kept) v = (int32_t)tok(i);
        else if (i == -1 && has_cls) v = L.cls_id;
        else if (i == kept && has_sep) v = L.sep_id;
        else on = false;
        if (L.id_bits == 64) reinterpret_cast<int64_t*>(L.ids)[base + col] = v;
        else reinterpret_cast<int32_t*>(L.ids)[base + col] = v;
        if (L.mask) {
            if (L.mask_bits == 64) reinterpret_cast<int64_t*>(L.mask)[base + col] = on;
            else if (L.mask_bits == 32) reinterpret_cast<int32_t*>(L.mask)[base + col] = on;
            else reinterpret_cast<uint8_t*>(L.mask)[base + col] = on;
        }
    }
}


// Bin rows by length: class_count[c] rows land in class_list[c * n_rows ...].  One atomic per
// warp and class (rows of a batch mostly share a class).  Classes outside class_mask are not
// launched by the host; a row that belongs to one is flagged instead of being dropped silently.
// short_bins: rows of the first class that fit a half, a quarter or an eighth of a warp are listed apart, k-th bin
// (1 << k rows per warp) with its counter at class_count[BPE_SHORT_COUNT + k] and its list backwards from the end of
// class k's, which it cannot meet: a row is in one list only.
constexpr int BPE_SHORT_BINS = 3;
constexpr int BPE_SHORT_COUNT = BPE_N_CLASSES + 1;            // after the counters of the windows; bins count from 1
__global__ void bpe_classify_kernel(const int64_t* __restrict__ offsets, int64_t n_rows,
                                    int32_t* __restrict__ class_count, int32_t* __restrict__ class_list,
                                    int32_t* __restrict__ counts, int32_t* __restrict__ status,
                                    uint32_t class_mask, BpeLengths len_out, bool short_bins) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int c = -1;
    if (i < n_rows) {
        const int64_t n = offsets[i + 1] - offsets[i];
        int32_t bits = 0;
        counts[i] = 0;
        if (n > 0) {
            c = 0;
            while (c < BPE_LONG_CLASS && (int64_t)bpe_class_capacity(c) < n) ++c;
            if (n > BPE_MAX_POSITIONS) { bits = 1; c = -1; }
            else if (!((class_mask >> c) & 1u)) { bits = 8; c = -1; }   // outside the caller's length hint
            else if (short_bins)
                for (int k = BPE_SHORT_BINS; k >= 1 && c == 0; --k)
                    if (n <= (bpe_class_capacity(0) >> k)) c = BPE_SHORT_COUNT + k;
        }
        if (c < 0) {                                              // no kernel will visit this row
            bpe_put_length(len_out, i, 0);
            if (len_out.ids) bpe_write_row(len_out, i, 0, 0, 1, [](int) { return 0u; });
        }
        bpe_put_status(status, i, bits, len_out.store_status != 0);
    }
    const int n_lists = short_bins ? BPE_SHORT_COUNT + BPE_SHORT_BINS + 1 : BPE_N_CLASSES;
    for (int k = 0; k < n_lists; ++k) {
        const uint32_t m = __ballot_sync(0xffffffffu, c == k);
        if (m == 0) continue;
        const int leader = __ffs(m) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(class_count + k, __popc(m));
        base = __shfl_sync(0xffffffffu, base, leader);
        const int at = base + __popc(m & ((1u << lane) - 1u));
        if (c == k) class_list[k < BPE_N_CLASSES ? (int64_t)k * n_rows + at : (int64_t)(k - BPE_SHORT_COUNT + 1) * n_rows - 1 - at] = (int32_t)i;
    }
}

// Barrier over the W warps of one team (team index `team` within a block of BW warps).
// BAR0 is the hardware barrier of team 0; code that runs teams of several widths in one block gives every
// width its own range of barriers.
template <int W, int BW, int BAR0 = 1>
__device__ __forceinline__ void team_sync(int team) {
    if (W == 1) __syncwarp();
    else if (W == BW) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(team + BAR0), "r"(W * 32) : "memory");
}

// Shared-memory accesses by 32-bit address in the shared window: the lanes kernel keeps its buffer
// addresses in registers and reaches every slot with a compile-time offset.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts_u16(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint2 lds_u64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}

// A pair's lookup in steps, each of which asks for what the next one needs: the pass over a lane's slots runs them one slot
// apart, so that no step waits for a load that was issued just before it.
//   ST: displacement, slot, rank entry, all from the packed table in shared memory;
//   otherwise displacement and entry, from global memory.
// Between the steps: d = displacement; s = slot word or entry; i = rank entry.
struct BpeLook { uint32_t a, b, d; uint2 s; uint32_t i; };
template <bool ST>
__device__ __forceinline__ void bpe_look_disp(BpeLook& k, const BpeSmemTable& st, const BpeDeviceTable& t, uint32_t a, uint32_t b) {
    k.a = a;
    k.b = b;
    k.d = ST ? lds_u16(st.disp + 2u * a) : __ldg(t.disp + a);
}
template <bool ST>
__device__ __forceinline__ void bpe_look_slot(BpeLook& k, const BpeSmemTable& st, const BpeDeviceTable& t) {
    if (ST) k.s.x = lds_u32(st.slot + 4u * min(k.d + k.b, st.last));
    else k.s = __ldg(t.slots + (k.d + k.b));
}
__device__ __forceinline__ void bpe_look_info(BpeLook& k, const BpeSmemTable& st) {
    k.i = lds_u32(st.info + 4u * ((k.s.x >> 16) == k.a ? k.s.x & 0xFFFFu : 0u));
}
// The finished entry (x, key).
template <bool ST>
__device__ __forceinline__ uint2 bpe_look_entry(const BpeLook& k) {
    uint2 e;
    if (ST) {
        const bool hit = (k.s.x >> 16) == k.a;
        e.x = hit ? (k.s.x << 16) | (k.i & 0xFFFFu) : BPE_FULL;
        e.y = hit ? (k.i & 0xFFFF0000u) | (k.s.x & 0xFFFFu) : BPE_FULL;
    } else {
        e.y = (k.s.y >> 16) == k.a ? __byte_perm(k.s.x, k.s.y, 0x5432) : BPE_FULL;
        e.x = e.y == BPE_FULL ? BPE_FULL : k.s.x;
    }
    return e;
}

// floor(x / d) for 1 <= d <= 32, x < 2^16: __umulhi(2 x + 1, ceil(2^31 / d)).
__device__ __forceinline__ uint32_t bpe_inv(uint32_t d) { return (0x80000000u + d - 1u) / d; }

// The per-slot bodies of the lanes kernel run from the lane's last slot down to slot 0 through a
// switch on the slot count with fall-through cases: one indirect jump instead of a guard per slot,
// every slot index a compile-time constant (shared-memory offsets, register names, mask bits), and
// no value handed from slot to slot except the accumulators.
#define BPE_SLOTS_DOWN(X) \
    X(31) X(30) X(29) X(28) X(27) X(26) X(25) X(24) X(23) X(22) X(21) X(20) X(19) X(18) X(17) X(16) \
    X(15) X(14) X(13) X(12) X(11) X(10) X(9) X(8) X(7) X(6) X(5) X(4) X(3) X(2) X(1) X(0)

#ifndef BPE_LANES_MIN_BLOCKS
#define BPE_LANES_MIN_BLOCKS 4
#endif
__host__ __device__ constexpr int bpe_min_blocks(int W) { return W <= 8 ? BPE_LANES_MIN_BLOCKS : W == 16 ? 2 : 1; }

// Which candidates of a round are taken when one warp holds the word (or 32 / L words, L lanes each): sel, the
// positions that survive, this lane's place among the survivors and their number.  link_r / link_l: the right / left
// neighbour is a candidate that goes first; valid: the lane's positions that hold a token.
template <int L>
__device__ __forceinline__ void bpe_select_warp(uint32_t cand, uint32_t link_r, uint32_t link_l, uint32_t valid, int top, int sh,
                                                uint32_t full, int g, int part, bool single_step, uint32_t& sel, uint32_t& kept, int& q0,
                                                int& n_new) {
    bool carry = false;
    const uint32_t odd_r = __brev(chain_parity<true, L>(__brev(link_r) >> sh, top, full, carry, g) << sh);
    carry = false;
    const uint32_t odd_l = chain_parity<false, L>(link_l, top, full, carry, g);
    sel = cand & ~odd_l & ~odd_r;
    if (single_step) {                                       // only the leftmost pair of the lowest rank
        uint32_t any = __ballot_sync(BPE_FULL, sel != 0u);
        if (L < 32) any = (any >> (part * L)) & (BPE_FULL >> (32 - L));
        sel = g == __ffs(any) - 1 ? (sel & (0u - sel)) : 0u;
    }
    uint32_t prev = __shfl_up_sync(BPE_FULL, sel >> top, 1, L);
    if (g == 0) prev = 0u;
    kept = valid & ~((sel << 1) | prev);
    const int x = __popc(kept);
    int incl = x;
#pragma unroll
    for (int d = 1; d < L; d <<= 1) {
        const int y = __shfl_up_sync(BPE_FULL, incl, d, L);
        if (g >= d) incl += y;
    }
    q0 = incl - x;
    n_new = __shfl_sync(BPE_FULL, incl, L - 1, L);
}

constexpr int BPE_FIRST_BYTES = 4096 + 32;

// Block-wide tables of the lanes code, in static shared memory of the kernel that runs it.
struct BpeLanesShared {
    uint2* hot;          // [BPE_HOT_WORDS] direct table for pairs of small ids, row stride BPE_HOT_STRIDE
    uint16_t* btok;      // [256] initial symbol of every byte
    uint8_t* first;      // [4096 + 32] the first round in letters
    uint32_t* inv;       // [BPE_LANE_SLOTS + 1] bpe_inv(d)
    uint32_t* red;       // [BW] per-warp partial minima
    uint32_t* fn;        // [BW] per-warp carry functions of the two walks
    uint32_t* blk;       // [BW] per-warp survivor count and border bits
    int32_t* word;       // [BW] claimed word index, at the team's first warp
};
#define BPE_LANES_SHARED(BW_, sh)                                      \
    __shared__ uint2 sh##_hot[BPE_HOT_WORDS];                          \
    __shared__ uint16_t sh##_btok[256];                                \
    __shared__ uint4 sh##_first[BPE_FIRST_BYTES / 16];                 \
    __shared__ uint32_t sh##_inv[BPE_LANE_SLOTS + 1];                  \
    __shared__ uint32_t sh##_red[BW_], sh##_fn[BW_], sh##_blk[BW_];    \
    __shared__ int32_t sh##_word[BW_];                                 \
    const BpeLanesShared sh{sh##_hot, sh##_btok, reinterpret_cast<uint8_t*>(sh##_first), sh##_inv, sh##_red, sh##_fn, sh##_blk, sh##_word}

// FIRST: the kernel runs words of one warp, which is where the first round in letters is.
template <int BW, bool FIRST>
__device__ __forceinline__ void bpe_lanes_setup(const BpeLanesShared& sh, const BpeDeviceTable& t) {
    for (int i = threadIdx.x; i < BPE_HOT_WORDS; i += BW * 32) sh.hot[i] = make_uint2(BPE_FULL, BPE_FULL);
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * 32; i += BW * 32) sh.hot[(i >> 5) * BPE_HOT_STRIDE + (i & 31)] = __ldg(t.hot + i);
    for (int i = threadIdx.x; i < 256; i += BW * 32) sh.btok[i] = __ldg(t.byte_tok + i);
    if (FIRST && t.first)
        for (int i = threadIdx.x; i < BPE_FIRST_BYTES / 16; i += BW * 32) reinterpret_cast<uint4*>(sh.first)[i] = __ldg(t.first + i);
    if (threadIdx.x >= 1 && threadIdx.x <= BPE_LANE_SLOTS) sh.inv[threadIdx.x] = bpe_inv(threadIdx.x);
    __syncthreads();
}

// The words of one list through teams of W warps, in a block of BW warps whose teams each own TEAM_BYTES of
// the dynamic shared memory.  list == NULL: no binning was done because the caller vouches that every row
// fits; the n_words rows are taken as they come, and a row longer than direct_limit is flagged and left empty.
// WIN: the words are the windows of long rows (bpe_window_plan_kernel): offsets holds a (start, end) pair per
// window, window i's tokens go to out_tok + i * BPE_WIN and its count to counts[i] (-1: it did not converge).
// SPAN (one team that is the whole block): one word, `span_bytes` bytes from `span_begin`; tokens to out_tok, count to *counts.
// G (one warp per team only): words a warp works on at once, 32 / G lanes each.  A round's work outside the slots (scans,
// votes, walk parities) costs a warp the same whatever the word's length, so short words share it.
template <int W, int BW, int BAR0, int TEAM_BYTES, bool ST = false, bool WIN = false, int G = 1, bool SPAN = false>
__device__ __forceinline__ void bpe_lanes_body(const BpeLanesShared& sh, const BpeSmemTable& stab, uint16_t* const sm,
                 const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets,
                 const int32_t* __restrict__ list, const int n_words,
                 int32_t* __restrict__ work_counter, const BpeDeviceTable& t,
                 uint16_t* __restrict__ out_tok, int32_t* __restrict__ counts,
                 int32_t* __restrict__ status, const BpeLengths& len_out, int32_t direct_limit, int64_t span_begin = 0,
                 int32_t span_bytes = 0) {
    constexpr int P = BPE_LANE_SLOTS;
    static_assert(!SPAN || (W == BW && WIN), "a span is a window that the whole block works on");
    static_assert(G == 1 || (W == 1 && !WIN), "only single warps share words");
    constexpr int T = 32 * W / G;                // lanes of a word
    constexpr int L = 32 / G;                    // ... and of them in one warp
    constexpr int STRIDE = 32 * W + 2;           // elements between the slots of one lane
    constexpr int BUF = P * STRIDE;              // one token buffer
    static_assert(TEAM_BYTES >= (int)bpe_team_bytes(W), "team area too small");
    uint16_t* const s_btok = sh.btok;
    uint32_t* const s_inv = sh.inv;
    uint32_t* const s_red = sh.red;
    uint32_t* const s_fn = sh.fn;
    uint32_t* const s_blk = sh.blk;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int team = warp / W, tw = warp % W;    // team, warp within team
    int32_t* const s_word = sh.word + team * W;
    const int g = G > 1 ? lane % L : tw * 32 + lane;   // lane within the word's lanes
    const int part = lane / L;                   // which of the warp's words (G > 1)
    // All token traffic goes through shared-memory byte addresses held in registers.
    constexpr uint32_t S2 = 2 * STRIDE;          // bytes between the slots of one lane
    const uint32_t team_base = (uint32_t)team * (TEAM_BYTES / 2);
    const uint32_t hot_base = smem_u32(sh.hot);
    uint32_t cur = smem_u32(sm + team_base + (G > 1 ? lane : g)); // this lane's column in the buffer of live tokens
    uint32_t nxt = cur + 2 * BUF;                // ... and in the buffer the round writes
    uint32_t* const xf = reinterpret_cast<uint32_t*>(sm + team_base + 2 * BUF);   // [T] entry of every lane's first pair (W > 1)
    uint32_t* const xl = xf + T;                                                  // [T] entry of every lane's last pair  (W > 1)

    // work_counter == NULL: the batch is a single wave (no more words than teams in the grid), and team k of block b
    // takes word b + k * blocks, with no counter to claim from (and none to zero before the launch)
    bool first = true;
    for (;;) {
        int wi;
        if (!work_counter) {
            wi = !first ? n_words : SPAN ? 0 : (int)blockIdx.x + (int)gridDim.x * (team * G + (G > 1 ? part : 0));
            first = false;
        } else if (G > 1) {
            wi = 0;
            if (lane == 0) wi = atomicAdd(work_counter, G);
            wi = __shfl_sync(BPE_FULL, wi, 0) + part;
        } else if (W == 1) {
            wi = 0;
            if (lane == 0) wi = atomicAdd(work_counter, 1);
            wi = __shfl_sync(BPE_FULL, wi, 0);
        } else {
            if (g == 0) s_word[0] = atomicAdd(work_counter, 1);
            team_sync<W, BW, BAR0>(team);
            wi = s_word[0];
        }
        if (G > 1 ? !__any_sync(BPE_FULL, wi < n_words) : wi >= n_words) {
            team_sync<W, BW, BAR0>(team);                    // the claim slot is reused by whatever this team runs next
            break;
        }
        const bool here = G == 1 || wi < n_words;            // the last words may not fill a warp
        const int row = !here ? 0 : !list ? wi : G > 1 ? list[-wi] : list[wi];    // short rows are listed backwards (bpe_classify_kernel)
        const int64_t oi = WIN ? 2 * (int64_t)wi : (int64_t)row;
        const int64_t off = SPAN ? span_begin : offsets[oi];
        const int64_t n64 = SPAN ? (int64_t)span_bytes : here ? offsets[oi + 1] - off : 0;
        int n = (int)n64;                                    // 1 <= n <= T * P by classification (windows: by construction)
        // direct rows are not vetted: an empty row, one whose offsets decrease (empty as well), or one the hint misstated
        if (G > 1 && !list && (n64 < 0 || n64 > direct_limit)) n = 0;          // finished with the others of its warp
        if (G == 1 && !WIN && !list && (n64 < 1 || n64 > direct_limit)) {
            if (g == 0) {
                counts[row] = 0;
                bpe_put_length(len_out, row, 0);
                bpe_put_status(status, row, n64 > 0 ? 8 : 0, len_out.store_status != 0);
            }
            if (len_out.ids) bpe_write_row(len_out, row, 0, g, T, [](int) { return 0u; });
            team_sync<W, BW, BAR0>(team);                          // everybody has read the claimed index
            continue;
        }
        uint32_t Pp = (uint32_t)(n + T - 1) / T;             // positions per lane: lane g owns [g Pp, (g + 1) Pp)
        if (G > 1) Pp = max(__reduce_max_sync(BPE_FULL, Pp), 1u);   // the same for all words of the warp
        uint32_t inv = s_inv[Pp];

        // While every token of the word is a small id (all_hot) the pairs come from the shared-memory
        // table and the filler behind the end of the word is that table's empty row 32; afterwards they
        // come from the table in global memory and the filler is the id one past the vocabulary.
        bool all_hot = t.bytes_hot != 0u;
        uint32_t filler = all_hot ? BPE_FILLER : t.filler;
        if (G == 1 && g == 0) sts_u16(cur + 2 * T, filler);  // what the last lane sees as "the next lane's first token"
        // Every lane fetches its own chunk of the word as aligned 32-bit words (all requested before the
        // first is used), maps the bytes to tokens and fills its column.
        {
            const uint32_t c0 = (uint32_t)g * Pp;            // first position of this lane
            const uintptr_t a0 = reinterpret_cast<uintptr_t>(bytes + off + c0);
            const uint32_t mis = (uint32_t)(a0 & 3u);
            const uint32_t* src = reinterpret_cast<const uint32_t*>(a0 - mis);
            const int first = (int)c0 - (int)mis;            // position of byte 0 of src[0]
            uint32_t w[P / 4 + 1];
#pragma unroll
            for (int k = 0; k <= P / 4; ++k)                 // a word is read when it holds a byte of the word
                w[k] = (4 * k < (int)(Pp + mis) && first + 4 * k < n && first + 4 * k + 3 >= 0 && (G == 1 || n > 0)) ? __ldg(src + k) : 0u;
#pragma unroll
            for (int k = 0; k < P / 4; ++k) w[k] = __funnelshift_r(w[k], w[k + 1], 8 * mis);    // bytes 4k .. 4k + 3 of the chunk
            if (W == 1 && t.first && Pp >= 4u) {
                // ---- the first round, on the letters.  Candidates and order bits come four positions at a time from a
                // table indexed by six letters' codes; the letters never become tokens in the buffer, the round's result
                // does.  Against a round that looks up a token and a pair per position: 16,384 rows of 1,024 bytes,
                // vocabulary 4,096, 158 -> 146 us.
                const int top = (int)Pp - 1, sh_ = 32 - (int)Pp;
                const uint32_t full = BPE_FULL >> sh_;
                const int len = min(max(n - (int)c0, 0), (int)Pp);
                const uint32_t valid = len >= 32 ? BPE_FULL : ((1u << len) - 1u);
                uint32_t cw[3] = {0u, 0u, 0u}, alien = 0;    // 2-bit codes, position 0 lowest; bytes that are no letter
#pragma unroll
                for (int k = 0; k < P / 4; ++k) {
                    if (4 * k < (int)Pp) {
                        const uint32_t c = (w[k] >> 1) & 0x03030303u;
                        const uint32_t lo = c & 0x01010101u, hi = (c >> 1) & 0x01010101u, both = lo & hi;
                        const uint32_t d = w[k] ^ (0x41414141u + 2u * lo + 0x13u * hi - 0x0Fu * both);   // A C T G
                        cw[k / 4] |= ((c * 0x00041041u >> 18) & 0xFFu) << (8 * (k % 4));
                        const uint32_t m = (((d & 0x7f7f7f7fu) + 0x7f7f7f7fu) | d) & 0x80808080u;
                        alien |= (((m >> 7) * 0x01020408u) >> 24) << (4 * k);
                    }
                }
                const uint32_t ok = valid & ~alien;
                // the next lane's first letters behind this lane's last one
                uint32_t nx = __shfl_down_sync(BPE_FULL, (cw[0] & 0x3Fu) | ((ok << 6) & 0xC0u), 1, L);
                if (g == L - 1) nx = 0u;
                {
                    uint64_t lo = (uint64_t)cw[0] | ((uint64_t)cw[1] << 32);
                    const uint32_t at = 2u * Pp;
                    if (at < 64u) lo = (lo & ((1ull << at) - 1ull)) | ((uint64_t)(nx & 0x3Fu) << at);
                    cw[0] = (uint32_t)lo;
                    cw[1] = (uint32_t)(lo >> 32);
                    cw[2] = at > 58u ? (nx & 0x3Fu) >> (64u - at) : 0u;
                }
                const uint32_t pairs = ok & ((ok >> 1) | (((nx >> 6) & 1u) << top));                  // both letters of the pair are there
                const uint32_t pairs_up = (pairs >> 1) | (((nx >> 6) & (nx >> 7) & 1u) << top);       // ... and of the pair after it
                uint32_t cand = 0, gt = 0;
                const uint32_t tab = smem_u32(sh.first);
#pragma unroll
                for (int k = 0; k < P / 4; ++k) {
                    if (4 * k < (int)Pp) {
                        const uint32_t six = k % 4 == 3 ? __funnelshift_r(cw[k / 4], cw[k / 4 + 1], 24) : cw[k / 4] >> (8 * (k % 4));
                        const uint32_t v = lds_u8(tab + (six & 0xFFFu));
                        cand |= (v & 15u) << (4 * k);
                        gt |= (v >> 4) << (4 * k);
                    }
                }
                cand &= pairs;
                gt = (gt | ~pairs) & pairs_up;               // a pair that is not there ranks behind every other
                uint32_t gt_before = __shfl_up_sync(BPE_FULL, gt >> top, 1, L);
                if (g == 0) gt_before = 1u;
                const uint32_t leq = ~((gt << 1) | (gt_before & 1u));
                uint32_t sel, kept;
                int q0, n_new;
                bpe_select_warp<L>(cand, cand & gt, cand & leq, valid, top, sh_, full, g, part, false, sel, kept, q0, n_new);
                all_hot = all_hot && t.first_hot != 0u;
                filler = all_hot ? BPE_FILLER : t.filler;
                uint32_t Pn = (uint32_t)(n_new + T - 1) / T;
                if (G > 1) Pn = max(__reduce_max_sync(BPE_FULL, Pn), 1u);
                const uint32_t inv_n = s_inv[Pn];
                const uint32_t back = 2 * (Pn * STRIDE - 1);
                const uint32_t dst = cur - 2 * g;            // the buffer is free: this is the first thing written to it
                const uint32_t single = smem_u32(s_btok), made = tab + 4096u;
                uint32_t q = (uint32_t)q0 + (uint32_t)__popc(kept);
                switch (Pp) {
#define BPE_F(J)                                                                              \
                case J + 1: {                                                                 \
                    const bool keep_ = (kept & (1u << J)) != 0u;                              \
                    if (keep_) --q;                                                           \
                    const uint32_t l_ = __umulhi(2u * q + 1u, inv_n);                         \
                    const uint32_t two_ = (J) % 16 == 15 ? __funnelshift_r(cw[(J) / 16], cw[(J) / 16 + 1], 30) : cw[(J) / 16] >> (2 * ((J) % 16)); \
                    const uint32_t tk_ = lds_u16((sel & (1u << J)) ? made + 2u * (two_ & 15u) : single + 2u * ((w[(J) / 4] >> (8 * ((J) % 4))) & 0xFFu)); \
                    if (keep_) sts_u16(dst + q * S2 - l_ * back, tk_);                        \
                }
                BPE_SLOTS_DOWN(BPE_F)
#undef BPE_F
                default: break;
                }
                for (uint32_t pt = (uint32_t)n_new + (uint32_t)g; pt < Pn * T; pt += T) {    // filler, as after every round
                    const uint32_t l_ = __umulhi(2u * pt + 1u, inv_n);
                    sts_u16(dst + pt * S2 - l_ * back, filler);
                    if (G == 1) break;
                }
                if (G == 1 && g == 0) sts_u16(dst + 2 * T, filler);
                n = n_new; Pp = Pn; inv = inv_n;
            } else {
#pragma unroll
                for (int k = 0; k < P / 4; ++k) {
                    if (4 * k < (int)Pp) {
#pragma unroll
                        for (int bb = 0; bb < 4; ++bb) {
                            const uint32_t tk = s_btok[(w[k] >> (8 * bb)) & 0xFFu];
                            sts_u16(cur + (4 * k + bb) * S2, (int)c0 + 4 * k + bb < n ? tk : filler);
                        }
                    }
                }
            }
        }
        team_sync<W, BW, BAR0>(team);

        int round = 0;
        const int max_rounds = (G > 1 ? __reduce_max_sync(BPE_FULL, n) : n) + 2;
        for (; round < max_rounds; ++round) {
            const int top = (int)Pp - 1, sh = 32 - (int)Pp;
            const int p0 = g * (int)Pp;
            uint32_t t_up = lds_u16(cur + 2);                // the next lane's first token; then handed from slot to slot: the token one slot up
            if (G > 1 && g == L - 1) t_up = filler;

            // ---- A: entries of the lane's pairs, the word's bound, "right neighbour ranks better" bits.
            // While every token of the word is a small id all pairs come from the shared-memory table and
            // the slots are straight-line code; afterwards each lane takes the table its pair needs.
            // The slots run from the last one down; a lookup's steps are spread over the slots after it (BpeLook), the token
            // of a slot is read one slot ahead, and the entries in flight when a lane starts are empty ones.  A slot that
            // waits for its own lookup: vocabulary 32,000, 16,384 rows of 1,024 bytes 192 -> 183 us, 8,192 rows of 2,048
            // 216 -> 190 us; vocabulary 4,096, 2,000 rows of 1,024 bytes 28 -> 26 us, large batches unchanged.
            uint32_t val[P + 4];                             // x word of every pair's entry: (rank << 16) | created id
            uint32_t gt = 0;                                 // bit j: the pair right of slot j's ranks better
            uint32_t emin = BPE_FULL;
            uint32_t a_next = lds_u16(cur + (Pp - 1u) * S2);
#define BPE_TAKE(J, E)                                                                        \
                    val[J] = (E).x;                                                           \
                    emin = min(emin, (E).y);                                                  \
                    if ((J) < P && val[J] > val[(J) + 1]) gt |= 1u << ((J) & 31);
#define BPE_TOKENS(J)                                                                         \
                        const uint32_t a = a_next, b = t_up;                                  \
                        t_up = a;                                                             \
                        if (J) a_next = lds_u16(cur + ((J) ? (J) - 1 : 0) * S2);
            if (all_hot) {
                uint2 e = make_uint2(BPE_FULL, BPE_FULL);
                switch (Pp) {
#define BPE_A(J)                                                                              \
                    case J + 1: {                                                             \
                        BPE_TOKENS(J)                                                         \
                        BPE_TAKE(J + 1, e)                                                    \
                        e = lds_u64(hot_base + (a * BPE_HOT_STRIDE + b) * 8u);   /* the filler's pairs are empty */ \
                    }
                    BPE_SLOTS_DOWN(BPE_A)
#undef BPE_A
                    default: break;
                }
                BPE_TAKE(0, e)
            } else if (ST) {
                BpeLook k1, k2, k3;                          // waiting for its slot, for its rank entry, finished
                k1.a = k2.a = k3.a = 0; k1.b = 0; k1.d = stab.last; k2.s.x = k3.s.x = BPE_FULL; k3.i = 0;
                switch (Pp) {
#define BPE_STEP(J)                                                                           \
                        { const uint2 e = bpe_look_entry<true>(k3); BPE_TAKE(J + 3, e) }      \
                        k3 = k2; bpe_look_info(k3, stab);                                     \
                        k2 = k1; bpe_look_slot<true>(k2, stab, t);
#define BPE_A(J)                                                                              \
                    case J + 1: {                                                             \
                        BPE_TOKENS(J)                                                         \
                        BPE_STEP(J)                                                           \
                        bpe_look_disp<true>(k1, stab, t, a, b);                               \
                    }
                    BPE_SLOTS_DOWN(BPE_A)
#undef BPE_A
                    default: break;
                }
                BPE_STEP(-1)
#undef BPE_STEP
                { const uint2 e = bpe_look_entry<true>(k3); BPE_TAKE(1, e) }
                k3 = k2; bpe_look_info(k3, stab);
                { const uint2 e = bpe_look_entry<true>(k3); BPE_TAKE(0, e) }
            } else {
                BpeLook k1, k2;                              // waiting for its entry, finished
                k1.a = k1.b = filler; k1.d = 0u; k2.a = filler; k2.s = make_uint2(BPE_FULL, BPE_FULL);
                switch (Pp) {
#define BPE_A(J)                                                                              \
                    case J + 1: {                                                             \
                        BPE_TOKENS(J)                                                         \
                        { const uint2 e = bpe_look_entry<false>(k2); BPE_TAKE(J + 2, e) }     \
                        k2 = k1; bpe_look_slot<false>(k2, stab, t);                           \
                        bpe_look_disp<false>(k1, stab, t, a, b);                              \
                    }
                    BPE_SLOTS_DOWN(BPE_A)
#undef BPE_A
                    default: break;
                }
                { const uint2 e = bpe_look_entry<false>(k2); BPE_TAKE(1, e) }
                k2 = k1; bpe_look_slot<false>(k2, stab, t);
                { const uint2 e = bpe_look_entry<false>(k2); BPE_TAKE(0, e) }
            }
#undef BPE_TAKE
#undef BPE_TOKENS
            uint32_t v_top = val[0];                         // the entry of the last slot, whichever register holds it
            switch (top) {
#define BPE_T(J) case J: v_top = val[J]; break;
                BPE_SLOTS_DOWN(BPE_T)
#undef BPE_T
                default: break;
            }
            gt &= (1u << top) - 1u;                          // the last slot was compared with nothing; set below
            const uint32_t v_first = val[0];
            if (G == 1) emin = __reduce_min_sync(BPE_FULL, emin);
            else {
#pragma unroll
                for (int d = 1; d < L; d <<= 1) emin = min(emin, __shfl_xor_sync(BPE_FULL, emin, d));
            }
            uint32_t v_nf, v_pl;                             // the next lane's first entry, the previous lane's last entry
            if (W == 1) {
                v_nf = __shfl_down_sync(BPE_FULL, v_first, 1, L);
                v_pl = __shfl_up_sync(BPE_FULL, v_top, 1, L);
                if (g == L - 1) v_nf = BPE_FULL;
                if (g == 0) v_pl = BPE_FULL;
            } else {
                xf[g] = v_first;
                xl[g] = v_top;
                if (lane == 0) s_red[warp] = emin;
                team_sync<W, BW, BAR0>(team);
#pragma unroll
                for (int k = 0; k < W; ++k) emin = min(emin, s_red[team * W + k]);
                v_nf = g + 1 < T ? xf[g + 1] : BPE_FULL;
                v_pl = g > 0 ? xl[g - 1] : BPE_FULL;
            }
            // no pair can merge: done (uniform over the team; words that share a warp wait for the last one, unchanged)
            if (G > 1 ? __all_sync(BPE_FULL, emin == BPE_FULL) : emin == BPE_FULL) break;
            const uint32_t Bs = emin & 0xFFFF0000u;          // rank < B  <=>  entry < B << 16

            // ---- B: candidate and link masks of the lane's positions
            if (v_top > v_nf) gt |= 1u << top;
            uint32_t cand = 0, vmax = 0;                     // vmax: the highest-ranking candidate's entry
            switch (Pp) {
#define BPE_B(J) case J + 1: if (val[J] < Bs) { cand |= 1u << J; vmax = max(vmax, val[J]); }
                BPE_SLOTS_DOWN(BPE_B)
#undef BPE_B
                default: break;
            }
            // the round creates small ids only if all its candidates rank below t.hot_ranks
            const bool big = (vmax >> 16) >= t.hot_ranks && cand != 0u;
            const uint32_t full = BPE_FULL >> sh;
            const uint32_t leq = (~(gt << 1) & ~1u) | (v_pl <= v_first ? 1u : 0u);   // bit j: rank(j-1) <= rank(j)
            const uint32_t link_r = cand & gt;               // the right neighbour is a candidate that goes first
            const uint32_t link_l = cand & leq;              // the left neighbour is a candidate that goes first
            const int len = min(max(n - p0, 0), (int)Pp);
            const uint32_t valid = len >= 32 ? BPE_FULL : ((1u << len) - 1u);

            // ---- selection on the masks
            uint32_t sel, kept;
            int q0, n_new;
            if (W == 1) {
                all_hot = all_hot && !__any_sync(BPE_FULL, big);
                bpe_select_warp<L>(cand, link_r, link_l, valid, top, sh, full, g, part, t.single_step != 0, sel, kept, q0, n_new);
            } else {
                // every warp works on its own 32 lanes; what crosses warps are the blocks' carry functions
                // (first barrier) and their survivor counts with the border bits (second barrier)
                uint32_t fn_r, fn_l;
                const ChainPrep pr = chain_prepare<true>(__brev(link_r) >> sh, top, full, lane, fn_r);
                const ChainPrep pl = chain_prepare<false>(link_l, top, full, lane, fn_l);
                const uint32_t any_cand = t.single_step ? __ballot_sync(BPE_FULL, cand != 0u) : 0u;
                const bool any_big = __any_sync(BPE_FULL, big);
                if (lane == 0) s_fn[warp] = fn_r | (fn_l << 2) | (any_cand ? 16u : 0u) | (any_big ? 32u : 0u);
                team_sync<W, BW, BAR0>(team);
                bool carry_r = false, carry_l = false, earlier = false;
#pragma unroll
                for (int k = 0; k < W; ++k) all_hot = all_hot && !(s_fn[team * W + k] & 32u);
                for (int k = W - 1; k > tw; --k) carry_r = carry_apply(s_fn[team * W + k] & 3u, carry_r) != 0u;
                for (int k = 0; k < tw; ++k) {
                    const uint32_t f = s_fn[team * W + k];
                    carry_l = carry_apply((f >> 2) & 3u, carry_l) != 0u;
                    earlier = earlier || (f & 16u);
                }
                const uint32_t odd_r = __brev(chain_finish<true>(pr, carry_r, lane) << sh);
                const uint32_t odd_l = chain_finish<false>(pl, carry_l, lane);
                sel = cand & ~odd_l & ~odd_r;
                if (t.single_step)                           // only the leftmost pair of the lowest rank
                    sel = (!earlier && lane == __ffs(any_cand) - 1) ? (cand & (0u - cand)) : 0u;
                uint32_t prev = __shfl_up_sync(BPE_FULL, sel >> top, 1);
                if (lane == 0) prev = 0u;                    // corrected below from the block before
                kept = valid & ~((sel << 1) | prev);
                const int x = __popc(kept);
                int incl = x;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(BPE_FULL, incl, d);
                    if (lane >= d) incl += y;
                }
                const uint32_t first_valid = __shfl_sync(BPE_FULL, valid & 1u, 0);
                if (lane == 31) s_blk[warp] = (uint32_t)incl | ((sel >> top) << 16) | (first_valid << 17);
                team_sync<W, BW, BAR0>(team);
                // lane k looks at block k: its count drops by one when the block before it merged across the border
                const uint32_t w = lane < W ? s_blk[team * W + lane] : 0u;
                uint32_t lost = __shfl_up_sync(BPE_FULL, (w >> 16) & 1u, 1);
                if (lane == 0) lost = 0u;
                lost &= (w >> 17) & 1u;
                const int tot = (int)(w & 0xFFFFu) - (int)lost;
                int bincl = tot;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(BPE_FULL, bincl, d);
                    if (lane >= d) bincl += y;
                }
                const int base = __shfl_sync(BPE_FULL, bincl - tot, tw);
                n_new = __shfl_sync(BPE_FULL, bincl, 31);
                const bool mine_lost = __shfl_sync(BPE_FULL, lost, tw) != 0u;
                if (mine_lost && lane == 0) kept &= ~1u;
                q0 = base + incl - x - ((mine_lost && lane > 0) ? 1 : 0);
            }

            // ---- C: merge, and deal the survivors out again in the other buffer, last slot first.
            // Position q goes to lane l = q / Pn, slot q - l Pn: byte 2 (q STRIDE - l (Pn STRIDE - 1)) of the buffer.
            uint32_t Pn = (uint32_t)(n_new + T - 1) / T;
            if (G > 1) Pn = __reduce_max_sync(BPE_FULL, Pn);
            const uint32_t inv_n = s_inv[Pn];
            const uint32_t back = 2 * (Pn * STRIDE - 1);
            const uint32_t dst = nxt - 2 * g;                // start of the buffer the round writes
            uint32_t q = (uint32_t)q0 + (uint32_t)__popc(kept);
            uint32_t tk_next = lds_u16(cur + (Pp - 1u) * S2);
            switch (Pp) {
#define BPE_C(J)                                                                              \
                case J + 1: {                                                                 \
                    const uint32_t tk_ = tk_next;                                             \
                    if (J) tk_next = lds_u16(cur + ((J) ? (J) - 1 : 0) * S2);                 \
                    const bool keep_ = (kept & (1u << J)) != 0u;                              \
                    if (keep_) --q;                                                           \
                    const uint32_t l_ = __umulhi(2u * q + 1u, inv_n);                         \
                    if (keep_) sts_u16(dst + q * S2 - l_ * back, (sel & (1u << J)) ? val[J] : tk_); \
                }
                BPE_SLOTS_DOWN(BPE_C)
#undef BPE_C
                default: break;
            }
            {                                                // filler behind the new end, up to the lanes' common slot count
                filler = all_hot ? BPE_FILLER : t.filler;
                for (uint32_t pt = (uint32_t)n_new + (uint32_t)g; pt < Pn * T; pt += T) {    // one trip unless words share the warp
                    const uint32_t l_ = __umulhi(2u * pt + 1u, inv_n);
                    sts_u16(dst + pt * S2 - l_ * back, filler);
                    if (G == 1) break;
                }
                if (G == 1 && g == 0) sts_u16(dst + 2 * T, filler);    // the column behind the last lane
            }
            team_sync<W, BW, BAR0>(team);
            const uint32_t sw = cur; cur = nxt; nxt = sw;
            n = n_new; Pp = Pn; inv = inv_n;
        }

        if (!WIN && len_out.ids) {
            const uint32_t col0 = cur - 2 * g;               // the team's buffer
            if (here) bpe_write_row(len_out, row, n, g, T, [&](int q) {
                const uint32_t l = __umulhi(2u * (uint32_t)q + 1u, inv);
                return lds_u16(col0 + 2 * (((uint32_t)q - l * Pp) * STRIDE + l));
            });
        } else {
            uint16_t* const out = out_tok + (WIN ? (int64_t)wi * BPE_WIN : off);
            for (int q = g; q < n; q += T) {
                const uint32_t l = __umulhi(2u * (uint32_t)q + 1u, inv);
                out[q] = (uint16_t)lds_u16(cur - 2 * g + 2 * (((uint32_t)q - l * Pp) * STRIDE + l));
            }
        }
        if (WIN) {
            if (g == 0) counts[wi] = round >= max_rounds ? -1 : n;
        } else if (g == 0 && here) {
            counts[row] = n;
            int32_t bits = bpe_put_length(len_out, row, n) | (round >= max_rounds ? 2 : 0);
            if (G > 1 && !list && n64 > direct_limit) bits = 8;                               // longer than the hint: left empty
            bpe_put_status(status, row, bits, len_out.store_status != 0 && !list);   // binned rows were written by the binning pass
        }
        team_sync<W, BW, BAR0>(team);
    }
}

// W: warps per word.  WIN: the words are windows of long rows, their number is *list_count.
template <int W, bool WIN = false, int G = 1>
__global__ void __launch_bounds__(bpe_block_warps(W) * 32, bpe_min_blocks(W))
bpe_lanes_kernel(const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets,
                 const int32_t* __restrict__ list, const int32_t* __restrict__ list_count,
                 int32_t* __restrict__ work_counter, BpeDeviceTable t,
                 uint16_t* __restrict__ out_tok, int32_t* __restrict__ counts,
                 int32_t* __restrict__ status, BpeLengths len_out, int32_t n_direct, int32_t direct_limit) {
    constexpr int BW = bpe_block_warps(W);
    extern __shared__ uint4 bpe_dyn[];
    BPE_LANES_SHARED(BW, sh);
    bpe_lanes_setup<BW, W == 1>(sh, t);
    bpe_lanes_body<W, BW, 1, (int)bpe_team_bytes(W), false, WIN, G>(sh, BpeSmemTable{}, reinterpret_cast<uint16_t*>(bpe_dyn), bytes, offsets,
                                                                 list, WIN || list ? *list_count : n_direct, work_counter, t, out_tok,
                                                                 counts, status, len_out, direct_limit);
}

// The same for a vocabulary whose packed table fits into shared memory beside the teams' buffers: one block of
// 32 warps per SM, the table copied in once per block, every lookup of the general mode answered from it.
constexpr int BPE_ST_WARPS = 32;
__host__ __device__ constexpr size_t bpe_st_team_area(int W) { return (size_t)(BPE_ST_WARPS / W) * bpe_team_bytes(W); }
template <int W, bool WIN = false, int G = 1>
__global__ void __launch_bounds__(BPE_ST_WARPS * 32, 1)
bpe_lanes_st_kernel(const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets,
                    const int32_t* __restrict__ list, const int32_t* __restrict__ list_count,
                    int32_t* __restrict__ work_counter, BpeDeviceTable t,
                    uint16_t* __restrict__ out_tok, int32_t* __restrict__ counts,
                    int32_t* __restrict__ status, BpeLengths len_out, int32_t n_direct, int32_t direct_limit) {
    // Launched with programmatic stream serialisation when the launch before it in the stream may be a kernel: this
    // grid's blocks can be placed while that one drains, and wait here until it is complete and visible.
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    extern __shared__ uint4 bpe_dyn[];
    BPE_LANES_SHARED(BPE_ST_WARPS, sh);
    uint4* const tab = bpe_dyn + bpe_st_team_area(W) / 16;
    for (uint32_t i = threadIdx.x; i < t.compact_bytes / 16; i += BPE_ST_WARPS * 32) tab[i] = __ldg(t.compact + i);
    bpe_lanes_setup<BPE_ST_WARPS, W == 1>(sh, t);                     // ends with a block-wide barrier
    const uint32_t base = smem_u32(tab);
    const BpeSmemTable stab{base, base + t.compact_slot, base + t.compact_info, t.compact_last};
    {
        // A small batch is spread over all blocks: only as many teams of a block take part as the words per
        // block ask for (words are claimed from one counter, and the blocks that start first would otherwise
        // take them all while other SMs stay idle).
        const int n_words = WIN || list ? *list_count : n_direct;
        const int active = (n_words + (int)gridDim.x * G - 1) / ((int)gridDim.x * G);
        if ((int)(threadIdx.x >> 5) / W >= active) return;
    }
    // sixteen teams of two warps need sixteen hardware barriers: barrier 0 is theirs as well once the set-up is over
    bpe_lanes_body<W, BPE_ST_WARPS, (W == 2 ? 0 : 1), (int)bpe_team_bytes(W), true, WIN, G>(sh, stab, reinterpret_cast<uint16_t*>(bpe_dyn),
                                                                     bytes, offsets, list, WIN || list ? *list_count : n_direct,
                                                                     work_counter, t, out_tok, counts, status, len_out, direct_limit);
}

// Rows of the first length class only, binned by how many of them fit a warp, in one launch: every warp works through
// the bins from the longest rows down, so the batch has one tail.  Vocabularies of a few thousand tokens bring their
// packed table into shared memory (ST), as above.
template <bool ST>
__global__ void __launch_bounds__(ST ? BPE_ST_WARPS * 32 : 256, ST ? 1 : BPE_LANES_MIN_BLOCKS)
bpe_short_kernel(const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets, const int32_t* __restrict__ class_list,
                 int64_t n_rows, const int32_t* __restrict__ class_count, int32_t* __restrict__ work, BpeDeviceTable t,
                 uint16_t* __restrict__ out_tok, int32_t* __restrict__ counts, int32_t* __restrict__ status, BpeLengths len_out) {
    constexpr int BW = ST ? BPE_ST_WARPS : 8;
    extern __shared__ uint4 bpe_dyn[];
    BPE_LANES_SHARED(BW, sh);
    BpeSmemTable stab{};
    if (ST) {
        uint4* const tab = bpe_dyn + bpe_st_team_area(1) / 16;
        for (uint32_t i = threadIdx.x; i < t.compact_bytes / 16; i += BW * 32) tab[i] = __ldg(t.compact + i);
        const uint32_t base = smem_u32(tab);
        stab = BpeSmemTable{base, base + t.compact_slot, base + t.compact_info, t.compact_last};
    }
    bpe_lanes_setup<BW, true>(sh, t);
    uint16_t* const sm = reinterpret_cast<uint16_t*>(bpe_dyn);
#define BPE_BIN(K, LIST)                                                                                                      \
    bpe_lanes_body<1, BW, 1, (int)bpe_team_bytes(1), ST, false, (1 << K)>(sh, stab, sm, bytes, offsets, LIST,                  \
        class_count[K ? BPE_SHORT_COUNT + K : 0], work + (K ? BPE_SHORT_COUNT + K : 0), t, out_tok, counts, status, len_out, 0);
    BPE_BIN(0, class_list)
    BPE_BIN(1, class_list + 2 * n_rows - 1)
    BPE_BIN(2, class_list + 3 * n_rows - 1)
    BPE_BIN(3, class_list + 4 * n_rows - 1)
#undef BPE_BIN
}

// Rows of several length classes in one launch: a block of BPE_MIXED_WARPS warps works through the classes
// from the widest team to the narrowest, splitting into more and more teams on the way, so a batch of mixed
// lengths has one tail instead of one per class.  levels.classes[k] holds the classes (bit c: class c) that
// run with teams of 1 << k warps; a team's area at every width lies inside the area of the team it was part
// of one width up, and every width has its own hardware barriers, so teams move on without waiting for their
// block.
constexpr int BPE_MIXED_WARPS = 16;
constexpr int BPE_MIXED_LEVELS = 5;
__host__ __device__ constexpr size_t bpe_mixed_warp_bytes() {      // shared memory per warp so that every width fits
    size_t m = 0;
    for (int w = 1; w <= BPE_MIXED_WARPS; w *= 2) {
        const size_t per = (bpe_team_bytes(w) + (size_t)w - 1) / (size_t)w;
        if (per > m) m = per;
    }
    return (m + 15) / 16 * 16;
}
__host__ __device__ constexpr size_t bpe_mixed_bytes() { return bpe_mixed_warp_bytes() * BPE_MIXED_WARPS; }
struct BpeMixedLevels { uint32_t classes[BPE_MIXED_LEVELS]; };

template <int W, int BAR0>
__device__ __forceinline__ void bpe_mixed_level(const BpeLanesShared& sh, uint16_t* sm, uint32_t classes,
                 const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets,
                 const int32_t* __restrict__ class_list, int64_t n_rows, const int32_t* __restrict__ class_count,
                 int32_t* __restrict__ work, const BpeDeviceTable& t, uint16_t* __restrict__ out_tok,
                 int32_t* __restrict__ counts, int32_t* __restrict__ status, const BpeLengths& len_out) {
    for (; classes; classes &= classes - 1u) {
        const int c = __ffs(classes) - 1;
        bpe_lanes_body<W, BPE_MIXED_WARPS, BAR0, (int)(bpe_mixed_warp_bytes() * W)>(
            sh, BpeSmemTable{}, sm, bytes, offsets, class_list + (int64_t)c * n_rows, class_count[c], work + c, t, out_tok, counts, status,
            len_out, 0);
    }
}

__global__ void __launch_bounds__(BPE_MIXED_WARPS * 32, 2)
bpe_mixed_kernel(const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets,
                 const int32_t* __restrict__ class_list, int64_t n_rows, const int32_t* __restrict__ class_count,
                 int32_t* __restrict__ work, BpeDeviceTable t, uint16_t* __restrict__ out_tok,
                 int32_t* __restrict__ counts, int32_t* __restrict__ status, BpeLengths len_out, BpeMixedLevels levels) {
    extern __shared__ uint4 bpe_dyn[];
    BPE_LANES_SHARED(BPE_MIXED_WARPS, sh);
    bpe_lanes_setup<BPE_MIXED_WARPS, true>(sh, t);
    uint16_t* const sm = reinterpret_cast<uint16_t*>(bpe_dyn);
#define BPE_LEVEL(K, BAR0) \
    bpe_mixed_level<(1 << K), BAR0>(sh, sm, levels.classes[K], bytes, offsets, class_list, n_rows, class_count, work, t, \
                                    out_tok, counts, status, len_out);
    BPE_LEVEL(4, 0) BPE_LEVEL(3, 1) BPE_LEVEL(2, 3) BPE_LEVEL(1, 7) BPE_LEVEL(0, 0)
#undef BPE_LEVEL
}
#undef BPE_SLOTS_DOWN

// Words beyond the lanes kernel's capacity, in windows.  A long word is cut into windows of BPE_WIN positions, each
// sharing BPE_WIN_OVERLAP positions with the next; the windows are merged like any other short words, one warp or
// small team each, and joined afterwards at a token that both windows hold at the same place in their overlap.
//
// The join is exact.  Take the merges of a word in their order and look at two neighbouring tokens of its result: no
// merge ever crossed the places where they begin, meet and end, so the merges inside them ran exactly as they run on
// these two tokens' text alone, which therefore encodes to the same two tokens.  Conversely, if every two neighbours
// of a sequence of tokens encode to themselves, the sequence is the result for the whole text: before the first merge
// that crossed one of its borders the merges on either side ran as they run on that pair alone, which would have
// crossed as well.  (The argument needs no more than the rule itself: lowest rank first, leftmost first.)  Cutting two
// windows' results at a common token leaves only neighbours that one of the two windows holds.  A border without a
// common token (a repeat longer than the overlap) is mended by merging more text at once (bpe_mend_word); a word for which
// that fails goes to bpe_long_kernel.
//
// One block per word, position-parallel in global memory, left all but a few SMs idle on such batches: 33 words of
// 40,000 to 400,000 bytes (vocabulary 4,096) took 2,507 us; in windows they take 90 us (merge 67, numbering 8,
// joins 7, scan 3, copy 5), of which an eighth is work done twice in the overlaps.  With a homopolymer of 600 bp across one
// border of every word the call takes 205 us instead of 156, with ten in every word 531 us; 2,640 to 2,740 us when such
// words were left to bpe_long_kernel.
struct BpeWindows {
    int64_t* span;        // [2 * windows] first byte and end of every window in the batch
    int32_t* row_of;      // [windows] index of its word in the list of long words
    int32_t* count;       // [windows] merged tokens
    int32_t* keep;        // [windows] tokens up to the join with the next window (-1: there is none)
    int32_t* skip;        // [windows] tokens that the window before holds already
    int32_t* base;        // [windows] tokens of its word before it
    int32_t* first;       // [words + 1] first window of every word
    int32_t* total;       // [words] tokens of the word (-1: left to bpe_long_kernel)
    uint16_t* tok;        // [windows * BPE_WIN] merged tokens
};

__device__ __forceinline__ int bpe_window_count(int64_t n) { return (int)((n - BPE_WIN_OVERLAP + BPE_WIN_STEP - 1) / BPE_WIN_STEP); }

// One block: numbers the windows of all long words and writes their spans.
__global__ void __launch_bounds__(1024)
bpe_window_plan_kernel(const int64_t* __restrict__ offsets, const int32_t* __restrict__ list, const int32_t* __restrict__ list_count,
                       BpeWindows w, int32_t* __restrict__ n_windows) {
    __shared__ int32_t s_warp[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_words = *list_count;
    int carry = 0;
    for (int i0 = 0; i0 < n_words; i0 += 1024) {
        const int i = i0 + tid;
        int nw = 0;
        if (i < n_words) { const int r = list[i]; nw = bpe_window_count(offsets[r + 1] - offsets[r]); }
        int x = nw;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(BPE_FULL, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int k = 0; k < 32; ++k) { if (k < warp) before += s_warp[k]; all += s_warp[k]; }
        if (i < n_words) w.first[i] = carry + before + x - nw;
        carry += all;
        __syncthreads();
    }
    if (tid == 0) { w.first[n_words] = carry; *n_windows = carry; }
    __syncthreads();
    for (int i = warp; i < n_words; i += 32) {
        const int r = list[i], f = w.first[i], nw = w.first[i + 1] - f;
        const int64_t off = offsets[r], end = offsets[r + 1];
        for (int k = lane; k < nw; k += 32) {
            const int64_t a = off + (int64_t)k * BPE_WIN_STEP;
            w.span[2 * (int64_t)(f + k)] = a;
            w.span[2 * (int64_t)(f + k) + 1] = a + BPE_WIN < end ? a + BPE_WIN : end;
            w.row_of[f + k] = i;
        }
    }
}

// One warp per window: where it joins the next window of its word.  tok_len[id]: bytes of a token.
constexpr int BPE_JOIN_WARPS = 8;
__global__ void __launch_bounds__(BPE_JOIN_WARPS * 32)
bpe_window_join_kernel(BpeWindows w, const int32_t* __restrict__ n_windows, const uint16_t* __restrict__ tok_len) {
    constexpr int OV = BPE_WIN_OVERLAP, PER = OV / 32;
    __shared__ uint16_t s_id[BPE_JOIN_WARPS][2][OV];          // token that starts at a position of the overlap (0xFFFF: none) ...
    __shared__ int16_t s_at[BPE_JOIN_WARPS][2][OV];           // ... and its index in its window
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = *n_windows;
    for (int i = blockIdx.x * BPE_JOIN_WARPS + warp; i < n; i += gridDim.x * BPE_JOIN_WARPS) {
        const int ca = w.count[i];
        const bool first = i == 0 || w.row_of[i - 1] != w.row_of[i];
        const bool last = i + 1 == n || w.row_of[i + 1] != w.row_of[i];
        if (first && lane == 0) w.skip[i] = 0;
        if (last) { if (lane == 0) w.keep[i] = ca; continue; }
        const int cb = w.count[i + 1];
        const uint16_t* const ta = w.tok + (int64_t)i * BPE_WIN;
        const uint16_t* const tb = ta + BPE_WIN;
#pragma unroll
        for (int k = 0; k < PER; ++k) s_id[warp][0][lane + 32 * k] = s_id[warp][1][lane + 32 * k] = 0xFFFFu;
        __syncwarp();
        uint32_t id[2][PER];
        int len[2][PER], sum[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int r = PER * lane + k;                     // this window's tokens from its end, the next one's from its start
            id[0][k] = r < ca ? (uint32_t)ta[ca - 1 - r] : 0xFFFFu;
            id[1][k] = r < cb ? (uint32_t)tb[r] : 0xFFFFu;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                len[s][k] = id[s][k] != 0xFFFFu ? (int)__ldg(tok_len + id[s][k]) : OV;
                sum[s] += len[s][k];
            }
        }
        int at[2] = {sum[0], sum[1]};
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int y = __shfl_up_sync(BPE_FULL, at[s], d);
                if (lane >= d) at[s] += y;
            }
        at[0] -= sum[0];
        at[1] -= sum[1];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int r = PER * lane + k;
            at[0] += len[0][k];                               // bytes from this token's start to the window's end
            if (at[0] <= OV && id[0][k] != 0xFFFFu) { s_id[warp][0][OV - at[0]] = (uint16_t)id[0][k]; s_at[warp][0][OV - at[0]] = (int16_t)(ca - 1 - r); }
            if (at[1] < OV && id[1][k] != 0xFFFFu) { s_id[warp][1][at[1]] = (uint16_t)id[1][k]; s_at[warp][1][at[1]] = (int16_t)r; }
            at[1] += len[1][k];
        }
        __syncwarp();
        int keep = -1, skip = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int p = lane + 32 * k;
            const uint32_t a = s_id[warp][0][p];
            const uint32_t hit = __ballot_sync(BPE_FULL, a != 0xFFFFu && a == s_id[warp][1][p]);
            if (hit && keep < 0) {
                const int q = 32 * k + __ffs(hit) - 1;
                keep = s_at[warp][0][q] + 1;
                skip = s_at[warp][1][q] + 1;
            }
        }
        if (lane == 0) { w.keep[i] = ca < 0 || cb < 0 ? -1 : keep; w.skip[i + 1] = skip; }
        __syncwarp();
    }
}

// The tokens [skip, keep) of a piece that took the places of windows [f, j), dealt to the windows' own places.
__device__ __forceinline__ void bpe_deal_piece(const BpeWindows& w, int f, int j, int skip, int keep) {
    for (int k = f + (int)threadIdx.x; k < j; k += blockDim.x) {
        const int lo = max(skip - (k - f) * BPE_WIN, 0), hi = min(keep - (k - f) * BPE_WIN, BPE_WIN);
        w.skip[k] = hi > lo ? lo : 0;
        w.keep[k] = hi > lo ? hi : 0;
    }
}

// The borders without a common token of the word in windows [f0, f1), by a block of 32 warps; false: the word is left.
//
// A repeat that covers the overlap gives no common token when the windows take it up at different places.  The window
// before such a border is merged again together with the windows after it, as one piece that is joined as windows are: with
// the piece or window before it in its first overlap, and with the first window whose overlap with the piece holds a common
// token.  Three windows are tried, then twelve, then 36, the widest team's 32,768 positions; a repeat beyond that leaves the word
// to bpe_long_kernel.  A piece takes the windows' own places: it starts where its first window does, and the tokens that
// begin before the overlap with window j ends are no more than 896 (j - f) + 128, which 1,024 (j - f) places hold.
constexpr int BPE_MEND_WINDOWS = 36;
static_assert(BPE_WIN + (BPE_MEND_WINDOWS - 1) * BPE_WIN_STEP <= bpe_class_capacity(BPE_LONG_CLASS - 1), "a piece is one word of the widest team");
__device__ __forceinline__ bool bpe_mend_word(const BpeLanesShared& sh, uint16_t* const sm, const uint8_t* __restrict__ bytes, const BpeWindows& w,
                                           const int f0, const int f1, const BpeDeviceTable& t, const uint16_t* __restrict__ tok_len,
                                           uint16_t* const stage) {
    constexpr int OV = BPE_WIN_OVERLAP, PER = OV / 32, T = BPE_LONG_WARPS * 32;
    __shared__ uint16_t s_left[2][OV];                        // overlap before the piece: token that starts there, its index
    __shared__ int32_t s_n, s_found, s_warp[BPE_LONG_WARPS];
    uint16_t* const zone_id = sm;                             // [windows of the piece][OV]: the piece's tokens in the overlaps,
    uint16_t* const zone_at = sm + BPE_MEND_WINDOWS * OV;     // in the merge's buffers once it is done
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int cur = f0, left_f = 0, left_skip = 0, left_end = -1;   // the piece before: first window, tokens skipped, window it joins
    for (;;) {
        __syncthreads();
        if (tid == 0) s_found = INT32_MAX;
        __syncthreads();
        for (int k = cur + tid; k < f1; k += T)
            if (w.keep[k] < 0) { atomicMin(&s_found, k); break; }
        __syncthreads();
        const int f = s_found;                                // the next border without a common token
        if (f == INT32_MAX) return true;
        if (f == f1 - 1) return false;                        // a window that did not converge
        const int64_t a = w.span[2 * (int64_t)f];
        uint16_t* const tok = stage + a;
        int n, last, hit;
        for (int m = 3;; m = min(4 * m, BPE_MEND_WINDOWS)) {
            last = min(f + m, f1) - 1;
            bpe_lanes_body<BPE_LONG_WARPS, BPE_LONG_WARPS, 1, bpe_team_bytes(BPE_LONG_WARPS), false, true, 1, true>(
                sh, BpeSmemTable{}, sm, bytes, nullptr, nullptr, 1, nullptr, t, tok, &s_n, nullptr, BpeLengths{}, 0, a,
                (int32_t)(w.span[2 * (int64_t)last + 1] - a));
            __syncthreads();
            n = s_n;
            if (n < 0) return false;
            const int zones = last - f + 1;
            for (int i = tid; i < zones * OV; i += T) zone_id[i] = 0xFFFFu;
            if (tid == 0) s_found = INT32_MAX;
            // where the piece's tokens start: every thread takes a run of them
            const int per = (n + T - 1) / T, q0 = min(tid * per, n), q1 = min(q0 + per, n);
            int sum = 0;
            for (int q = q0; q < q1; ++q) sum += (int)__ldg(tok_len + tok[q]);
            int at = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(BPE_FULL, at, d);
                if (lane >= d) at += y;
            }
            if (lane == 31) s_warp[warp] = at;
            __syncthreads();
            at -= sum;
            for (int k = 0; k < warp; ++k) at += s_warp[k];
            for (int q = q0; q < q1; ++q) {
                const uint32_t id = tok[q];
                const int z = at / BPE_WIN_STEP, p = at - z * BPE_WIN_STEP;
                if (p < OV && z < zones) { zone_id[z * OV + p] = (uint16_t)id; zone_at[z * OV + p] = (uint16_t)q; }
                at += (int)__ldg(tok_len + id);
            }
            __syncthreads();
            // the first window that holds one of them at the same place: (window, place, index in the window)
            for (int z = 1 + warp; z < zones; z += BPE_LONG_WARPS) {
                const int cb = w.count[f + z];
                const uint16_t* const tb = w.tok + (int64_t)(f + z) * BPE_WIN;
                uint32_t id[PER];
                int start[PER], own = 0;
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    const int r = PER * lane + k;
                    id[k] = r < cb ? (uint32_t)tb[r] : 0xFFFFu;
                    start[k] = own;
                    own += id[k] != 0xFFFFu ? (int)__ldg(tok_len + id[k]) : OV;
                }
                int before = own;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(BPE_FULL, before, d);
                    if (lane >= d) before += y;
                }
                before -= own;
                uint32_t best = BPE_FULL;
#pragma unroll
                for (int k = PER - 1; k >= 0; --k) {
                    const int p = before + start[k];
                    if (id[k] != 0xFFFFu && p < OV && zone_id[z * OV + p] == id[k]) best = (uint32_t)((z * OV + p) * OV + PER * lane + k);
                }
                best = __reduce_min_sync(BPE_FULL, best);
                if (lane == 0 && best != BPE_FULL) atomicMin(&s_found, (int)best);
            }
            __syncthreads();
            hit = s_found;
            if (hit != INT32_MAX || last == f1 - 1) break;
            if (m == BPE_MEND_WINDOWS) return false;
            __syncthreads();
        }
        // the join before the piece
        int skip = 0;
        if (f > f0) {
            if (left_end != f && warp == 0) {                 // a window, from its end
                const int ca = w.count[f - 1];
                const uint16_t* const ta = w.tok + (int64_t)(f - 1) * BPE_WIN;
                uint32_t id[PER];
                int end[PER], own = 0;
#pragma unroll
                for (int k = 0; k < PER; ++k) s_left[0][lane + 32 * k] = 0xFFFFu;
                __syncwarp();
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    const int r = PER * lane + k;
                    id[k] = r < ca ? (uint32_t)ta[ca - 1 - r] : 0xFFFFu;
                    own += id[k] != 0xFFFFu ? (int)__ldg(tok_len + id[k]) : OV;
                    end[k] = own;                             // bytes from this token's start to the end of the lane's first one
                }
                int before = own;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(BPE_FULL, before, d);
                    if (lane >= d) before += y;
                }
                before -= own;
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    const int p = OV - (before + end[k]);
                    if (id[k] != 0xFFFFu && p >= 0) { s_left[0][p] = (uint16_t)id[k]; s_left[1][p] = (uint16_t)(ca - 1 - (PER * lane + k)); }
                }
            }
            __syncthreads();
            if (tid == 0) s_found = INT32_MAX;
            __syncthreads();
            if (tid < OV && s_left[0][tid] != 0xFFFFu && s_left[0][tid] == zone_id[tid]) atomicMin(&s_found, tid);
            __syncthreads();
            const int p = s_found;
            if (p == INT32_MAX) return false;
            skip = (int)zone_at[p] + 1;
            if (left_end == f) bpe_deal_piece(w, left_f, f, left_skip, (int)s_left[1][p] + 1);
            else if (tid == 0) w.keep[f - 1] = (int)s_left[1][p] + 1;
        }
        const int zp = hit / OV, z = zp / OV;                 // the join after it, or the end of the word
        const int j = hit == INT32_MAX ? f1 : f + z;
        uint16_t* const dst = w.tok + (int64_t)f * BPE_WIN;
        for (int q = tid; q < min(n, (j - f) * BPE_WIN); q += T) dst[q] = tok[q];
        bpe_deal_piece(w, f, j, skip, hit == INT32_MAX ? n : (int)zone_at[zp] + 1);
        if (hit == INT32_MAX) return true;
        if (tid == 0) w.skip[j] = hit % OV + 1;
        __syncthreads();                                      // s_left has been read
        if (tid < OV) { s_left[0][tid] = zone_id[z * OV + tid]; s_left[1][tid] = zone_at[z * OV + tid]; }
        left_f = f; left_skip = skip; left_end = j; cur = j;
    }
}

// One block per long word: its token count and the place of every window's tokens, or its entry in the list of words
// that are left to bpe_long_kernel.  Borders without a common token are mended first.
__global__ void __launch_bounds__(BPE_LONG_WARPS * 32, 1)
bpe_window_scan_kernel(const uint8_t* __restrict__ bytes, const int32_t* __restrict__ list, const int32_t* __restrict__ list_count,
                       BpeWindows w, BpeDeviceTable t, const uint16_t* __restrict__ tok_len, uint16_t* __restrict__ out_tok,
                       int32_t* __restrict__ counts, int32_t* __restrict__ status, BpeLengths len_out,
                       int32_t* __restrict__ left_list, int32_t* __restrict__ left_count) {
    extern __shared__ uint4 bpe_dyn[];
    BPE_LANES_SHARED(BPE_LONG_WARPS, sh);
    __shared__ int32_t s_warp[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_words = *list_count;
    bool ready = false;                                       // the merge's tables are in shared memory
    for (int i = blockIdx.x; i < n_words; i += gridDim.x) {
        const int f = w.first[i], nw = w.first[i + 1] - f;
        int carry, bad;
        for (bool mended = false;; mended = true) {
            carry = bad = 0;
            for (int k0 = 0; k0 < nw; k0 += 1024) {
                const int k = k0 + tid;
                int v = 0;
                if (k < nw) {
                    const int keep = w.keep[f + k];
                    if (keep < 0) bad = 1;
                    v = keep - w.skip[f + k];
                }
                int x = v;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(BPE_FULL, x, d);
                    if (lane >= d) x += y;
                }
                if (lane == 31) s_warp[warp] = x;
                bad = __syncthreads_or(bad);
                int before = 0, all = 0;
#pragma unroll
                for (int q = 0; q < 32; ++q) { if (q < warp) before += s_warp[q]; all += s_warp[q]; }
                if (k < nw) w.base[f + k] = carry + before + x - v;
                carry += all;
                __syncthreads();
            }
            if (!bad || mended) break;
            if (!ready) bpe_lanes_setup<BPE_LONG_WARPS, false>(sh, t);
            ready = true;
            if (!bpe_mend_word(sh, reinterpret_cast<uint16_t*>(bpe_dyn), bytes, w, f, f + nw, t, tok_len, out_tok)) break;
            __syncthreads();
        }
        if (tid == 0) {
            const int row = list[i];
            w.total[i] = bad ? -1 : carry;
            if (bad) left_list[atomicAdd(left_count, 1)] = row;
            else {
                counts[row] = carry;
                bpe_put_status(status, row, bpe_put_length(len_out, row, carry), false);
            }
        }
    }
}

// One warp per window: its tokens to their place in the row.
__global__ void __launch_bounds__(BPE_JOIN_WARPS * 32)
bpe_window_write_kernel(const int64_t* __restrict__ offsets, const int32_t* __restrict__ list, BpeWindows w,
                        const int32_t* __restrict__ n_windows, uint16_t* __restrict__ out_tok, BpeLengths len_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = *n_windows;
    for (int i = blockIdx.x * BPE_JOIN_WARPS + warp; i < n; i += gridDim.x * BPE_JOIN_WARPS) {
        const int word = w.row_of[i], total = w.total[word];
        if (total < 0) continue;
        const int row = list[word], skip = w.skip[i], m = w.keep[i] - skip, base = w.base[i];
        if (m == 0) continue;                                 // its tokens are in the pieces around it
        const uint16_t* const src = w.tok + (int64_t)i * BPE_WIN + skip;
        if (len_out.ids) {
            bpe_write_row(len_out, row, total, lane, 32, [&](int q) { return (uint32_t)src[q - base]; }, base, base + m);
        } else {
            uint16_t* const dst = out_tok + offsets[row] + base;
            for (int q = lane; q < m; q += 32) dst[q] = src[q];
        }
    }
}

// Words beyond the lanes kernel's capacity: one block per word, state in global memory.  The
// tokens live in place in the output area (uint16 at the input offsets); ranks and the three mask
// arrays sit in a per-word piece of `long_area`, claimed from `long_cursor` by the block.
__global__ void __launch_bounds__(BPE_LONG_WARPS * 32)
bpe_long_kernel(const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets,
                const int32_t* __restrict__ list, const int32_t* __restrict__ list_count,
                int32_t* __restrict__ work_counter, BpeDeviceTable t, uint16_t* __restrict__ out_tok,
                int32_t* __restrict__ counts, int32_t* __restrict__ status,
                uint8_t* __restrict__ long_area, unsigned long long* __restrict__ long_cursor, BpeLengths len_out) {
    constexpr int W = BPE_LONG_WARPS;
    __shared__ uint32_t s_red[W][2];
    __shared__ uint2 s_hot[32 * 32];
    __shared__ long long s_word[2];                           // claimed word index / new length, scratch offset
    for (int i = threadIdx.x; i < 32 * 32; i += W * 32) s_hot[i] = __ldg(t.hot + i);
    __syncthreads();
    const int lane = threadIdx.x & 31, tw = threadIdx.x >> 5;
    const int tt = threadIdx.x;
    const uint32_t lt = (1u << lane) - 1u;
    const int n_words = *list_count;

    for (;;) {
        if (tt == 0) {
            const int w = atomicAdd(work_counter, 1);
            s_word[0] = w;
            if (w < n_words) {
                const int r = list[w];
                s_word[1] = (long long)atomicAdd(long_cursor, (unsigned long long)bpe_long_bytes(offsets[r + 1] - offsets[r]));
            }
        }
        __syncthreads();
        const int wi = (int)s_word[0];
        if (wi >= n_words) break;
        const int row = list[wi];
        const int64_t off = offsets[row];
        int n = (int)(offsets[row + 1] - off);
        const int G0 = (n + 31) >> 5;
        uint16_t* tok = out_tok + off;                                    // [n] live tokens, compact
        uint8_t* piece = long_area + s_word[1];
        uint16_t* rk = reinterpret_cast<uint16_t*>(piece);                // [n] rank of the pair (i, i+1)
        uint32_t* m_leq = reinterpret_cast<uint32_t*>(piece + ((2 * (int64_t)n + 15) / 16) * 16);   // bit i: rank(i-1) <= rank(i); later: survivors
        uint32_t* m_cs = m_leq + ((G0 + 3) / 4) * 4;                      // candidates, then selected pairs
        uint32_t* g_aux = m_cs + ((G0 + 3) / 4) * 4;                      // right-walk parity, then output base
        __syncthreads();                                                  // s_word is free again

        for (int i = tt; i < n; i += W * 32) tok[i] = __ldg(t.byte_tok + __ldg(bytes + off + i));
        __syncthreads();

        int round = 0;
        const int max_rounds = n + 2;
        for (; round < max_rounds; ++round) {
            const int groups = (n + 31) >> 5;
            // ---- 1: ranks of all pairs, bound B, lowest rank
            uint32_t bmin = BPE_NONE, gmin = BPE_NONE;
            for (int g = tw; g < groups; g += W) {
                const int i = g * 32 + lane;
                uint32_t r = BPE_NONE, fut = BPE_NONE;
                if (i + 1 < n) {
                    const uint32_t a = tok[i], b = tok[i + 1];
                    const uint2 e = (a | b) < 32u ? s_hot[a * 32u + b] : bpe_cold_entry(t, a, b);
                    r = e.x >> 16; fut = e.y >> 16;
                }
                if (i < n) rk[i] = (uint16_t)r;
                gmin = min(gmin, r);
                if (r != BPE_NONE) bmin = min(bmin, fut);
            }
            gmin = __reduce_min_sync(BPE_FULL, gmin);
            bmin = __reduce_min_sync(BPE_FULL, bmin);
            if (lane == 0) { s_red[tw][0] = gmin; s_red[tw][1] = bmin; }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < W; ++k) { gmin = min(gmin, s_red[k][0]); bmin = min(bmin, s_red[k][1]); }
            if (gmin == BPE_NONE) break;                       // no pair can merge: done (uniform over the block)
            const uint32_t B = t.single_step ? gmin + 1 : bmin;

            // ---- 2: candidate masks and "not worse than my left neighbour" masks
            for (int g = tw; g < groups; g += W) {
                const int i = g * 32 + lane;
                const uint32_t r = i < n ? (uint32_t)rk[i] : BPE_NONE;
                uint32_t rp = __shfl_up_sync(BPE_FULL, r, 1);
                if (lane == 0) rp = i > 0 ? (uint32_t)rk[i - 1] : BPE_NONE;
                const uint32_t cand = __ballot_sync(BPE_FULL, r < B);
                const uint32_t leq = __ballot_sync(BPE_FULL, rp <= r);
                if (lane == 0) { m_cs[g] = cand; m_leq[g] = leq; }
            }
            __syncthreads();

            // ---- 3: on the masks, one lane per 32 positions (first warp)
            if (tw == 0) {
                const int blocks = (groups + 31) >> 5;
                bool carry = false;                            // right walks, last block first
                for (int b = blocks - 1; b >= 0; --b) {
                    const int g = b * 32 + lane;
                    const bool live = g < groups;
                    const uint32_t cand = live ? m_cs[g] : 0u;
                    const uint32_t leq = live ? m_leq[g] : BPE_FULL;
                    const uint32_t leq_next = g + 1 < groups ? m_leq[g + 1] : BPE_FULL;
                    // bit i: the right neighbour ranks strictly better: not (rank(i) <= rank(i+1))
                    const uint32_t link = cand & ~((leq >> 1) | (leq_next << 31));
                    const uint32_t odd = __brev(chain_parity<true>(__brev(link), 31, BPE_FULL, carry, lane));
                    if (live) g_aux[g] = odd;
                }
                __syncwarp();
                carry = false;                                 // left walks, selection, survivors, output bases
                uint32_t sel_carry = 0;                        // was the position before the block selected
                int base = 0;
                bool took = false;
                for (int b = 0; b < blocks; ++b) {
                    const int g = b * 32 + lane;
                    const bool live = g < groups;
                    const uint32_t cand = live ? m_cs[g] : 0u;
                    const uint32_t leq = live ? m_leq[g] : 0u;
                    const uint32_t oddl = chain_parity<false>(cand & leq, 31, BPE_FULL, carry, lane);
                    uint32_t sel = live ? (cand & ~oddl & ~g_aux[g]) : 0u;
                    if (t.single_step) {                       // only the leftmost pair of the lowest rank
                        const uint32_t any = __ballot_sync(BPE_FULL, sel != 0);
                        const int first = __ffs(any) - 1;
                        sel = (!took && lane == first) ? (sel & (0u - sel)) : 0u;
                        took = took || any != 0;
                    }
                    uint32_t prev = __shfl_up_sync(BPE_FULL, sel, 1) >> 31;
                    if (lane == 0) prev = sel_carry;
                    sel_carry = __shfl_sync(BPE_FULL, sel, 31) >> 31;
                    const int cnt_pos = n - g * 32;            // positions of this group
                    const uint32_t valid = !live ? 0u : (cnt_pos >= 32 ? BPE_FULL : ((1u << cnt_pos) - 1u));
                    const uint32_t kept = valid & ~((sel << 1) | prev);
                    int x = __popc(kept), incl = x;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const int y = __shfl_up_sync(BPE_FULL, incl, d);
                        if (lane >= d) incl += y;
                    }
                    if (live) { m_cs[g] = sel; m_leq[g] = kept; g_aux[g] = (uint32_t)(base + incl - x); }
                    base += __shfl_sync(BPE_FULL, incl, 31);
                }
                if (lane == 0) s_word[0] = base;
            }
            __syncthreads();

            // ---- 4: merge and compact in place, W groups at a time
            const int n_new = (int)s_word[0];
            for (int g0 = 0; g0 < groups; g0 += W) {
                const int g = g0 + tw;
                const int i = g * 32 + lane;
                uint32_t v = 0, kept = 0;
                int base = 0;
                if (g < groups) {
                    const uint32_t sel = m_cs[g];
                    kept = m_leq[g];                           // survivors of this group, from step 3
                    base = (int)g_aux[g];
                    if (i < n) v = tok[i];
                    if ((sel >> lane) & 1u) v = __ldg(t.merge_out + rk[i]);
                }
                __syncthreads();                               // every warp has read its tokens of this tile
                if ((kept >> lane) & 1u) tok[base + __popc(kept & lt)] = (uint16_t)v;
            }
            __syncthreads();
            n = n_new;
        }

        if (len_out.ids) bpe_write_row(len_out, row, n, tt, W * 32, [&](int q) { return (uint32_t)tok[q]; });
        if (tt == 0) {
            counts[row] = n;
            const int32_t bits = bpe_put_length(len_out, row, n) | (round >= max_rounds ? 2 : 0);
            bpe_put_status(status, row, bits, false);
        }
        __syncthreads();
    }
}

}  // namespace dnatok
