// One token per source element: the single-base / byte path (uint8 source through a 256-entry
// shared-memory LUT) and the output stage of the BPE path (uint16 merged tokens, identity).
// Special tokens, truncation, padding and the attention mask are produced in the same pass.
#pragma once
#include <type_traits>
#include "common.cuh"

namespace dnatok {

constexpr int EMIT_THREADS = 256;

template <typename SrcT, bool USE_LUT>
__device__ __forceinline__ int32_t emit_load(const SrcT* __restrict__ p, const int32_t* s_lut) {
    if (USE_LUT) return s_lut[(uint8_t)__ldg(p)];
    return (int32_t)__ldg(p);
}

constexpr int EMIT_WARPS = EMIT_THREADS / 32;
constexpr int EMIT_SPAN = 512;           // output columns one warp produces per trip ...
constexpr int EMIT_SPAN_WIDE = 1024;     // ... and for 32-bit ids on long rows, where a trip of 512 stores too little

// Padded output [n_rows, out_stride].  counts == nullptr: a row's content is its byte span.
//
// A warp takes SPAN consecutive columns of one row.  The source elements under those columns are
// fetched as aligned 16-byte chunks (one or two per lane) into a per-warp shared-memory window,
// whatever the row's byte alignment and the one-column shift a leading special token causes; each
// lane then reads the N = 16/sizeof(IdT) elements of its output vector back as aligned words plus a
// funnel shift, maps them (LUT or identity) and issues one 16-byte store, so both the global loads
// and the global stores of a warp are contiguous.  Vectors that touch a special token, the
// truncation point or the padding take a per-column route.
template <typename SrcT, typename IdT, bool USE_LUT, int SPAN>
__global__ void __launch_bounds__(EMIT_THREADS)
emit_padded_kernel(const SrcT* __restrict__ src, const uint8_t* __restrict__ src_begin,
                   const uint8_t* __restrict__ src_end, const int64_t* __restrict__ offsets,
                   const int32_t* __restrict__ counts, int64_t n_rows,
                   const int32_t* __restrict__ lut, RowFormat f, IdT* __restrict__ ids,
                   void* __restrict__ mask, int32_t* __restrict__ lengths_out,
                   int32_t* __restrict__ status, int64_t spans_per_row, int64_t n_spans) {
    constexpr int N = Vec16<IdT>::N;
    constexpr int SZ = (int)sizeof(SrcT);
    constexpr int CHUNKS = SPAN * SZ / 16 + 1;               // 16-byte chunks covering a span at any alignment
    constexpr int VB = N * SZ;                                // source bytes under one output vector: 2, 4 or 8
    // Launched with programmatic stream serialisation: the next launch of the stream may be set up while this grid
    // drains, and this grid starts its work only once everything before it in the stream is complete and visible.
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ int32_t s_lut[256];
    __shared__ uint4 s_win[EMIT_WARPS][CHUNKS + 1];
    if (USE_LUT) {
        for (int i = threadIdx.x; i < 256; i += EMIT_THREADS) s_lut[i] = lut[i];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t* win = reinterpret_cast<const uint32_t*>(s_win[warp]);
    const bool has_cls = f.cls_id >= 0, has_sep = f.sep_id >= 0;
    const int64_t stride = f.out_stride;
    const bool small = n_spans <= 0x7fffffff;

    constexpr int R = (CHUNKS + 31) / 32;                     // window chunks per lane

    struct Span {
        int64_t row, cs, n, T, shift, t_lo;
        const uint8_t* wbase;
        int ncol, a, need;                                    // need: window chunks that hold content of this span
        bool any_content;
    };
    auto describe = [&](int64_t span) {
        Span p;
        if (small) {
            const uint32_t r32 = (uint32_t)span / (uint32_t)spans_per_row;
            p.row = r32;
            p.cs = (int64_t)((uint32_t)span - r32 * (uint32_t)spans_per_row) * SPAN;
        } else {
            p.row = span / spans_per_row;
            p.cs = (span - p.row * spans_per_row) * SPAN;
        }
        const int64_t off = offsets[p.row];
        const int64_t n_in = counts ? (int64_t)counts[p.row] : offsets[p.row + 1] - off;
        p.n = n_in < f.cap_content ? n_in : f.cap_content;
        p.T = p.n + (has_cls ? 1 : 0) + (has_sep ? 1 : 0);
        p.shift = f.pad_left ? stride - p.T : 0;
        if (p.cs == 0 && lane == 0) {
            if (lengths_out) lengths_out[p.row] = (int32_t)p.T;
            if (status) {
                const int32_t bits = (f.clip_is_error && n_in > p.n) ? 4 : 0;
                if (f.store_status) status[p.row] = bits;       // the caller left the words unset: written, not OR-ed
                else if (bits) atomicOr(status + p.row, bits);
            }
        }
        p.ncol = (int)(stride - p.cs < SPAN ? stride - p.cs : SPAN);
        p.t_lo = p.cs - (p.shift + (has_cls ? 1 : 0));        // content index under the span's first column
        const uint8_t* wptr = reinterpret_cast<const uint8_t*>(src + off) + p.t_lo * SZ;
        p.a = (int)(reinterpret_cast<uintptr_t>(wptr) & 15);
        p.wbase = wptr - p.a;
        p.any_content = p.t_lo + p.ncol > 0 && p.t_lo < p.n;  // else the span is specials and padding only
        {
            // content columns of the span end at min(t_lo + ncol, n); chunks past them are not fetched
            const int64_t t_hi = p.t_lo + p.ncol < p.n ? p.t_lo + p.ncol : p.n;
            p.need = p.any_content ? (int)((p.a + (t_hi - p.t_lo) * SZ + 15) >> 4) + 1 : 0;
        }
        return p;
    };
    // the span's source window as aligned 16-byte chunks, into registers
    auto fetch = [&](const Span& p, uint4* regs) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int k = lane + 32 * q;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (k < p.need && k < CHUNKS) {
                const uint8_t* g = p.wbase + 16 * k;
                if (g >= src_begin && g + 16 <= src_end) v = __ldg(reinterpret_cast<const uint4*>(g));
                else {
                    uint8_t tmp[16];
#pragma unroll
                    for (int b = 0; b < 16; ++b) tmp[b] = (g + b >= src_begin && g + b < src_end) ? __ldg(g + b) : (uint8_t)0;
                    v = *reinterpret_cast<uint4*>(tmp);
                }
            }
            regs[q] = v;
        }
    };

    const int64_t span_step = (int64_t)gridDim.x * EMIT_WARPS;
    int64_t span = (int64_t)blockIdx.x * EMIT_WARPS + warp;
    if (span >= n_spans) return;
    Span cur = describe(span);
    uint4 pre[R];
    fetch(cur, pre);
    for (;;) {
        // the window of this span goes to shared memory; the next span's window is requested right away
        __syncwarp();
#pragma unroll
        for (int q = 0; q < R; ++q) if (lane + 32 * q < CHUNKS) s_win[warp][lane + 32 * q] = pre[q];
        __syncwarp();
        const int64_t next = span + span_step;
        const bool more = next < n_spans;
        Span nxt = cur;
        if (more) { nxt = describe(next); fetch(nxt, pre); }

        const int64_t row = cur.row, cs = cur.cs, n = cur.n, T = cur.T, shift = cur.shift, t_lo = cur.t_lo;
        const int ncol = cur.ncol, a = cur.a;
        const bool any_content = cur.any_content;
        IdT* orow = ids + row * stride + cs;
        const bool aligned = (reinterpret_cast<uintptr_t>(orow) & 15) == 0;

        // content occupies columns [c_lo, c_hi) of the span: vectors inside need no per-column checks
        int c_lo = 0, c_hi = 0;
        {
            const int64_t lo64 = t_lo < 0 ? -t_lo : 0, hi64 = n - t_lo;
            c_lo = (int)(lo64 < ncol ? lo64 : ncol);
            c_hi = (int)(hi64 < 0 ? 0 : (hi64 < ncol ? hi64 : ncol));
        }
        // ---- ids
        for (int v = lane; v * N < ncol; v += 32) {
            const int c0 = v * N;                              // column within the span
            const int boff = a + c0 * SZ;                      // byte offset of the vector's source in the window
            const uint32_t sh = (uint32_t)(boff & 3) * 8u;
            const uint32_t* wp = win + (boff >> 2);
            uint32_t lo = 0, hi = 0;
            if (any_content) {
                const uint32_t w0 = wp[0], w1 = wp[1];
                lo = __funnelshift_r(w0, w1, sh);
                if (VB > 4) hi = __funnelshift_r(w1, wp[2], sh);
            }
            IdT vals[N];
            const int64_t t0 = t_lo + c0;
            const bool interior = c0 >= c_lo && c0 + N <= c_hi;
#pragma unroll
            for (int e = 0; e < N; ++e) {
                uint32_t word = (e * SZ < 4) ? lo : hi;
                uint32_t x = SZ == 1 ? (word >> (8 * (e & 3))) & 0xFFu : (word >> (16 * (e & 1))) & 0xFFFFu;
                int32_t val = USE_LUT ? s_lut[x & 0xFFu] : (int32_t)x;
                if (!interior) {
                    const int64_t t = t0 + e;                  // content index of this column
                    const int64_t col = cs + c0 + e - shift;   // token index within the row
                    if (t < 0 || t >= n) {
                        val = f.pad_id;
                        if (has_cls && col == 0) val = f.cls_id;
                        else if (has_sep && col == T - 1 && col >= 0) val = f.sep_id;
                    }
                }
                vals[e] = (IdT)val;
            }
            if (aligned && c0 + N <= ncol) store_vec<IdT>(orow + c0, vals);
            else {
#pragma unroll
                for (int e = 0; e < N; ++e) if (c0 + e < ncol) orow[c0 + e] = vals[e];
            }
        }

        // ---- mask: ones on [shift, shift + T)
        if (f.mask_bits) {
            const int64_t lo = shift - cs, hi = shift + T - cs;
            if (f.mask_bits == 64) warp_mask_row<int64_t>((int64_t*)mask + row * stride + cs, ncol, lo, hi, lane);
            else if (f.mask_bits == 32) warp_mask_row<int32_t>((int32_t*)mask + row * stride + cs, ncol, lo, hi, lane);
            else warp_mask_row<uint8_t>((uint8_t*)mask + row * stride + cs, ncol, lo, hi, lane);
        }
        if (!more) break;
        span = next;
        cur = nxt;
    }
}

// The same layout for short rows, flat: a thread takes one 16-byte vector of the ids (then of the mask) wherever it lies,
// finds its row by a division and goes on to the next row where the vector crosses into it.  A span per row leaves most of a
// warp's trip empty when a row has a few dozen columns; a thread's division and its row's bounds cost more than a span once
// rows are long.  Spans against flat, 16 million characters: 22 columns, 64-bit ids and mask 438 / 121 us, 102 columns
// 114 / 100, 152 columns 86 / 97; 32-bit ids and an 8-bit mask 22 columns 563 / 79 us, 302 columns 60 / 56, 402 columns
// 51 / 55; the merged tokens of 65,536 reads of 50 to 300 bp 59 / 16 us.
template <typename SrcT, typename IdT, bool USE_LUT>
__global__ void __launch_bounds__(EMIT_THREADS)
emit_short_kernel(const SrcT* __restrict__ src, int64_t n_src, const int64_t* __restrict__ offsets, const int32_t* __restrict__ counts,
                  int64_t n_rows, const int32_t* __restrict__ lut, RowFormat f, IdT* __restrict__ ids, void* __restrict__ mask,
                  int32_t* __restrict__ lengths_out, int32_t* __restrict__ status) {
    constexpr int N = Vec16<IdT>::N;
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ int32_t s_lut[256];
    if (USE_LUT) {
        for (int i = threadIdx.x; i < 256; i += EMIT_THREADS) s_lut[i] = lut[i];
        __syncthreads();
    }
    const uint32_t stride = (uint32_t)f.out_stride;
    const uint32_t cls = f.cls_id >= 0 ? 1u : 0u, n_special = cls + (f.sep_id >= 0 ? 1u : 0u);
    const uint32_t cap = (uint32_t)(f.cap_content < (int64_t)stride ? f.cap_content : (int64_t)stride);
    // Below 2^30 (launch_emit): the counters below run up to one step of the grid beyond it, at most 19.4 million elements
    // (148 SMs x 32 blocks x 256 threads x 16 mask bytes), and stay within 32 bits.
    const uint32_t total = (uint32_t)n_rows * stride;
    const uint32_t step = gridDim.x * EMIT_THREADS, first = blockIdx.x * EMIT_THREADS + threadIdx.x;
    auto elements = [&](uint32_t row, uint32_t* n_in) -> uint32_t {   // content tokens of a row that are kept
        const int64_t n = counts ? (int64_t)counts[row] : offsets[row + 1] - offsets[row];
        *n_in = (uint32_t)(n < 0 ? 0 : n < 0x7fffffff ? n : 0x7fffffff);          // offsets that decrease make an empty row
        return *n_in < cap ? *n_in : cap;
    };
    // The elements of a row that lie in the source buffer; the others are read as 0, as the span kernel does.
    auto readable = [&](int64_t off, uint32_t n) -> uint32_t {
        const int64_t room = off < 0 ? 0 : n_src - off;
        return room < (int64_t)n ? (uint32_t)(room < 0 ? 0 : room) : n;
    };
    const bool ids_aligned = (reinterpret_cast<uintptr_t>(ids) & 15) == 0;
    for (uint32_t g = first * N; g < total; g += step * N) {
        uint32_t row = g / stride, col = g - row * stride, n_in;
        uint32_t n = elements(row, &n_in);
        uint32_t start = (f.pad_left ? stride - n - n_special : 0u) + cls;      // column of the first content token
        int64_t off = offsets[row];
        uint32_t have = readable(off, n);
        const SrcT* p = src + off;
        IdT vals[N];
#pragma unroll
        for (int e = 0; e < N; ++e) {
            int32_t v = f.pad_id;
            if (g + e < total) {
                if (col == stride) {
                    col = 0; ++row;
                    n = elements(row, &n_in);
                    start = (f.pad_left ? stride - n - n_special : 0u) + cls;
                    off = offsets[row];
                    have = readable(off, n);
                    p = src + off;
                }
                const uint32_t t = col - start;                   // wraps below the content
                if (t < have) v = emit_load<SrcT, USE_LUT>(p + t, s_lut);
                else if (t < n) v = USE_LUT ? s_lut[0] : 0;
                else if (cls && t == 0xFFFFFFFFu) v = f.cls_id;
                else if (n_special > cls && t == n) v = f.sep_id;
                if (col == 0) {
                    if (lengths_out) lengths_out[row] = (int32_t)(n + n_special);
                    if (status) {
                        const int32_t bits = (f.clip_is_error && n_in > n) ? 4 : 0;
                        if (f.store_status) status[row] = bits;
                        else if (bits) atomicOr(status + row, bits);
                    }
                }
                ++col;
            }
            vals[e] = (IdT)v;
        }
        if (ids_aligned && g + N <= total) store_vec<IdT>(ids + g, vals);
        else {
#pragma unroll
            for (int e = 0; e < N; ++e) if (g + e < total) ids[g + e] = vals[e];
        }
    }
    auto write_mask = [&](auto* m) {
        using M = typename std::remove_reference<decltype(*m)>::type;
        constexpr int NM = Vec16<M>::N;
        const bool m_aligned = (reinterpret_cast<uintptr_t>(m) & 15) == 0;
        for (uint32_t g = first * NM; g < total; g += step * NM) {
            uint32_t row = g / stride, col = g - row * stride, n_in;
            uint32_t T = elements(row, &n_in) + n_special, lo = f.pad_left ? stride - T : 0u;
            M vals[NM];
#pragma unroll
            for (int e = 0; e < NM; ++e) {
                if (col == stride && g + e < total) {
                    col = 0; ++row;
                    T = elements(row, &n_in) + n_special;
                    lo = f.pad_left ? stride - T : 0u;
                }
                vals[e] = (M)(col - lo < T ? 1 : 0);
                ++col;
            }
            if (m_aligned && g + NM <= total) store_vec<M>(m + g, vals);
            else {
#pragma unroll
                for (int e = 0; e < NM; ++e) if (g + e < total) m[g + e] = vals[e];
            }
        }
    };
    if (f.mask_bits == 64) write_mask(reinterpret_cast<int64_t*>(mask));
    else if (f.mask_bits == 32) write_mask(reinterpret_cast<int32_t*>(mask));
    else if (f.mask_bits == 8) write_mask(reinterpret_cast<uint8_t*>(mask));
}

// Ragged output: ids is one flat array, row i occupies [out_offsets[i], out_offsets[i+1]).
//
// A warp takes RAGGED_SPAN consecutive elements, finds the row under the first one with a 32-way search, and goes
// through the rows' pieces of the span.  Each piece is fetched and written as emit_padded_kernel does it: aligned 16-byte
// chunks of the source into the warp's window, 16-byte stores of ids read back at the piece's own shift.  The bounds of
// 32 rows at a time sit in the lanes' registers.  The grid covers an upper bound of the total; spans past the real total
// do nothing.  Bound by the stores: 38.5 million characters in 16,384 rows, 64-bit ids, 72 us = 4.8 TB/s (109 us with a
// thread per vector that looked up each element's row and loaded its source byte by byte).
constexpr int RAGGED_SPAN = 1024;
template <typename SrcT, typename IdT, bool USE_LUT>
__global__ void __launch_bounds__(EMIT_THREADS)
emit_ragged_kernel(const SrcT* __restrict__ src, const uint8_t* __restrict__ src_begin, const uint8_t* __restrict__ src_end,
                   const int64_t* __restrict__ offsets, const int64_t* __restrict__ out_offsets, int64_t n_rows,
                   const int32_t* __restrict__ lut, RowFormat f, IdT* __restrict__ ids, void* __restrict__ mask) {
    constexpr int N = Vec16<IdT>::N;
    constexpr int SZ = (int)sizeof(SrcT);
    constexpr int CHUNKS = RAGGED_SPAN * SZ / 16 + 2;         // 16-byte chunks covering a piece at any alignment
    constexpr int VB = N * SZ;                                 // source bytes under one output vector: 2, 4 or 8
    __shared__ int32_t s_lut[256];
    __shared__ uint4 s_win[EMIT_WARPS][CHUNKS + 1];
    if (USE_LUT) {
        for (int i = threadIdx.x; i < 256; i += EMIT_THREADS) s_lut[i] = lut[i];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* const win = reinterpret_cast<uint8_t*>(s_win[warp]);
    const uint32_t* const win32 = reinterpret_cast<const uint32_t*>(win);
    const int cls = f.cls_id >= 0 ? 1 : 0, sep = f.sep_id >= 0 ? 1 : 0;
    const int64_t total = out_offsets[n_rows];
    const bool aligned = (reinterpret_cast<uintptr_t>(ids) & 15) == 0;
    for (int64_t g0 = ((int64_t)blockIdx.x * EMIT_WARPS + warp) * RAGGED_SPAN; g0 < total; g0 += (int64_t)gridDim.x * EMIT_WARPS * RAGGED_SPAN) {
        const int m = (int)(total - g0 < RAGGED_SPAN ? total - g0 : RAGGED_SPAN);
        // the last row that starts at or before g0
        int64_t lo = 0, size = n_rows;
        while (size > 1) {
            const int64_t step = (size + 31) >> 5, at = lo + lane * step;
            const uint32_t before = __ballot_sync(0xffffffffu, lane * step < size && out_offsets[at] <= g0);
            const int k = 31 - __clz(before);                  // bit 0 is always set
            lo += k * step;
            size = size - k * step < step ? size - k * step : step;
        }
        int64_t row0 = lo;                                     // lane l holds the bounds of row row0 + l
        int64_t r_start = 0, r_end = 0, r_src = 0;
        auto load_rows = [&]() {
            const int64_t r = row0 + lane;
            r_end = r_start = total;
            if (r < n_rows) { r_start = out_offsets[r]; r_end = out_offsets[r + 1]; r_src = offsets[r]; }
        };
        load_rows();
        for (int g = 0; g < m;) {                              // element within the span
            const uint32_t past = __ballot_sync(0xffffffffu, r_end > g0 + g);
            if (past == 0u) { row0 += 32; load_rows(); continue; }
            const int k = __ffs(past) - 1;                     // the row under element g (rows before it are empty or done)
            const int64_t row_start = __shfl_sync(0xffffffffu, r_start, k), row_end = __shfl_sync(0xffffffffu, r_end, k);
            const int64_t row_src = __shfl_sync(0xffffffffu, r_src, k);
            const int g_end = (int)(row_end - g0 < m ? row_end - g0 : m);
            const int ncol = g_end - g;
            const int64_t t_lo = g0 + g - row_start - cls;     // content index under the piece's first element, -1 for [CLS]
            const int64_t n = row_end - row_start - cls - sep; // content tokens of the row
            const int c_lo = t_lo < 0 ? 1 : 0;
            const int c_hi = (int)(n - t_lo < ncol ? n - t_lo : ncol);      // content lies under [c_lo, c_hi) of the piece
            const uint8_t* const wptr = reinterpret_cast<const uint8_t*>(src + row_src) + t_lo * SZ;
            const int a = (int)(reinterpret_cast<uintptr_t>(wptr) & 15);
            const uint8_t* const wbase = wptr - a;
            const int need = c_hi > c_lo ? (a + c_hi * SZ + 15) >> 4 : 0;
            __syncwarp();                                      // the piece before this one has been read
            for (int q = lane; q < need; q += 32) {
                const uint8_t* p = wbase + 16 * q;
                uint4 v;
                if (p >= src_begin && p + 16 <= src_end) v = __ldg(reinterpret_cast<const uint4*>(p));
                else {
                    uint8_t tmp[16];
#pragma unroll
                    for (int b = 0; b < 16; ++b) tmp[b] = (p + b >= src_begin && p + b < src_end) ? __ldg(p + b) : (uint8_t)0;
                    v = *reinterpret_cast<uint4*>(tmp);
                }
                s_win[warp][q] = v;
            }
            __syncwarp();
            // vectors at multiples of N elements of the whole output; the ones at the piece's ends are written element by element
            const int v_off = (int)((g0 + g) & (N - 1));       // elements of the first vector that lie before the piece
            IdT* const dst = ids + g0 + g;
            for (int c0 = N * lane - v_off; c0 < ncol; c0 += 32 * N) {
                if (aligned && c0 >= c_lo && c0 + N <= c_hi) {
                    const int at = a + c0 * SZ;
                    const uint32_t sh = (uint32_t)(at & 3) * 8u;
                    const uint32_t* wp = win32 + (at >> 2);
                    const uint32_t w0 = wp[0], w1 = wp[1];
                    const uint32_t lo32 = __funnelshift_r(w0, w1, sh);
                    uint32_t hi32 = 0;
                    if (VB > 4) hi32 = __funnelshift_r(w1, wp[2], sh);
                    IdT vals[N];
#pragma unroll
                    for (int e = 0; e < N; ++e) {
                        const uint32_t word = (e * SZ < 4) ? lo32 : hi32;
                        const uint32_t x = SZ == 1 ? (word >> (8 * (e & 3))) & 0xFFu : (word >> (16 * (e & 1))) & 0xFFFFu;
                        vals[e] = (IdT)(USE_LUT ? s_lut[x & 0xFFu] : (int32_t)x);
                    }
                    store_vec<IdT>(dst + c0, vals);
                } else {
#pragma unroll
                    for (int e = 0; e < N; ++e) {
                        const int c = c0 + e;
                        if (c < 0 || c >= ncol) continue;
                        int32_t v = c < c_lo ? f.cls_id : f.sep_id;
                        if (c >= c_lo && c < c_hi) {
                            const uint32_t x = SZ == 1 ? (uint32_t)win[a + c] : (uint32_t)*reinterpret_cast<const uint16_t*>(win + a + 2 * c);
                            v = USE_LUT ? s_lut[x & 0xFFu] : (int32_t)x;
                        }
                        dst[c] = (IdT)v;
                    }
                }
            }
            g = g_end;
        }
        if (mask && f.mask_bits) {
            if (f.mask_bits == 64) warp_write_run<int64_t>((int64_t*)mask + g0, m, lane, [](int64_t) { return (int64_t)1; });
            else if (f.mask_bits == 32) warp_write_run<int32_t>((int32_t*)mask + g0, m, lane, [](int64_t) { return (int32_t)1; });
            else warp_write_run<uint8_t>((uint8_t*)mask + g0, m, lane, [](int64_t) { return (uint8_t)1; });
        }
    }
}

// Tokenizers whose id of a row's first character differs from the id the same character gets later
// (the reference keeps a second "start" table for them and patches column 0,
// src/dna_tokenizer.py:1779-1820 with :527-631): after the rows are written, one thread per row puts
// the start id under the row's first content column.
template <typename IdT>
__global__ void start_fix_kernel(const uint8_t* __restrict__ bytes, const int64_t* __restrict__ offsets, int64_t n_rows,
                                 const int32_t* __restrict__ start_lut, RowFormat f, IdT* __restrict__ ids,
                                 const int64_t* __restrict__ out_offsets) {
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n_rows) return;
    const int64_t off = offsets[row], n_in = offsets[row + 1] - off;
    const int64_t n = n_in < f.cap_content ? n_in : f.cap_content;
    if (n <= 0) return;
    const int has_cls = f.cls_id >= 0 ? 1 : 0, has_sep = f.sep_id >= 0 ? 1 : 0;
    const IdT v = (IdT)__ldg(start_lut + __ldg(bytes + off));
    if (f.out_stride == 0) { ids[out_offsets[row] + has_cls] = v; return; }
    const int64_t T = n + has_cls + has_sep;
    const int64_t shift = f.pad_left ? f.out_stride - T : 0;
    ids[row * f.out_stride + shift + has_cls] = v;
}

// Row lengths of the one-token-per-character path (no data is read): min(n, cap) + specials.
__global__ void span_lengths_kernel(const int64_t* __restrict__ offsets, int64_t n_rows, RowFormat f, int32_t* __restrict__ lengths,
                                    int32_t* __restrict__ status) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows) return;
    const int64_t n_in = offsets[i + 1] - offsets[i];
    const int64_t n = n_in < f.cap_content ? n_in : f.cap_content;
    lengths[i] = (int32_t)(n + (f.cls_id >= 0 ? 1 : 0) + (f.sep_id >= 0 ? 1 : 0));
    if (status && f.clip_is_error && n_in > n) atomicOr(status + i, 4);
}

// What a caller wants to know of a batch's per-row words before it goes on: the largest length, all status bits, and one
// word copied along (the end of the output offsets).  Every block leaves its share in the call's own words in pinned host
// memory, and the host puts the few of them together: nothing is shared between calls, zeroed or allocated on the device.
// One launch and one wait where a reduction and a copy per value took two to four.
constexpr int SUMMARY_THREADS = 256;
constexpr int SUMMARY_PER_BLOCK = 4096;
constexpr int SUMMARY_BLOCKS = 128;      // most blocks of a launch; above 524,288 rows a block takes more than its 4,096
struct RowSummary {
    RowSummary* next;                    // host: list of the words that no call is using
    int64_t word;
    int32_t longest[SUMMARY_BLOCKS], bits[SUMMARY_BLOCKS];
};
__global__ void __launch_bounds__(SUMMARY_THREADS)
row_summary_kernel(const int32_t* __restrict__ lengths, const int32_t* __restrict__ status, int64_t n_rows, const int64_t* __restrict__ word,
                   RowSummary* __restrict__ out) {
    __shared__ int32_t s_longest[SUMMARY_THREADS / 32], s_bits[SUMMARY_THREADS / 32];
    const int tid = threadIdx.x;
    int32_t longest = 0, bits = 0;
    for (int64_t i = (int64_t)blockIdx.x * SUMMARY_THREADS + tid; i < n_rows; i += (int64_t)gridDim.x * SUMMARY_THREADS) {
        if (lengths) longest = max(longest, lengths[i]);
        if (status) bits |= status[i];
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    bits = (int32_t)__reduce_or_sync(0xffffffffu, (unsigned)bits);
    if ((tid & 31) == 0) { s_longest[tid >> 5] = longest; s_bits[tid >> 5] = bits; }
    __syncthreads();
    if (tid) return;
    for (int k = 1; k < SUMMARY_THREADS / 32; ++k) { longest = max(longest, s_longest[k]); bits |= s_bits[k]; }
    out->longest[blockIdx.x] = longest;
    out->bits[blockIdx.x] = bits;
    if (blockIdx.x == 0) out->word = word ? *word : 0;
}

// Exclusive scan of int32 lengths into int64 offsets, one block, 4,096 rows per trip: every thread takes four
// consecutive lengths (one 16-byte load), so a batch of a few thousand rows is one load, one block-wide scan and
// one round of stores instead of a chain of them.
__global__ void __launch_bounds__(1024)
scan_lengths_kernel(const int32_t* __restrict__ lengths, int64_t n_rows, int64_t* __restrict__ out_offsets) {
    __shared__ int64_t s_warp[32];
    __shared__ int64_t s_carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) { s_carry = 0; out_offsets[0] = 0; }
    __syncthreads();
    const bool vec_ok = (reinterpret_cast<uintptr_t>(lengths) & 15) == 0;
    for (int64_t base = 0; base < n_rows; base += 4096) {
        const int64_t i = base + 4 * (int64_t)tid;
        int32_t l[4] = {0, 0, 0, 0};
        if (vec_ok && i + 4 <= n_rows) {
            const int4 q = *reinterpret_cast<const int4*>(lengths + i);
            l[0] = q.x; l[1] = q.y; l[2] = q.z; l[3] = q.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) if (i + e < n_rows) l[e] = lengths[i + e];
        }
        const int64_t v = (int64_t)l[0] + l[1] + l[2] + l[3];
        int64_t x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int64_t w = s_warp[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, w, d);
                if (lane >= d) w += y;
            }
            s_warp[lane] = w;
        }
        __syncthreads();
        const int64_t incl = x + (warp ? s_warp[warp - 1] : 0) + s_carry;     // through this thread's four rows
        int64_t run = incl - v;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            run += l[e];
            if (i + e < n_rows) out_offsets[i + e + 1] = run;
        }
        __syncthreads();
        if (tid == 1023) s_carry = incl;
        __syncthreads();
    }
}

}  // namespace dnatok
