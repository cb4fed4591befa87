// How a step's tokens are spread over its sequences, read on the device from the cumulative lengths cu_q [n_seqs + 1] (a row whose
// length is not positive is no sequence: a recorded step has room for more than there are), for recurrences that take sequences of
// at least so many tokens by chunks and shorter ones token by token.  All device functions are a warp's together: every lane gets the
// result.
#pragma once

#include "common.cuh"

#include <limits.h>

// Which sequences a launch is about: those of from <= tokens < below.  `beside` > 0: the limit between short and long (`from` of the
// long, `below` of the short) is looked up: where the step has `few` or fewer sequences shorter than it, all are long, else those of
// `beside` tokens are.
// `direct`: all of them, the rows of the launch are the step's (a lookup costs every block a trip to memory).  `recorded`: the launch is
// replayed for other lengths.  Its rows are fewer than the sequences there may be, a block goes on from row to row, and it works only
// where there are lo to hi such sequences (lo 0: however many).
// `ordered`: the rows of such a launch are the sequences in this order, four bits each (at most sixteen), the longest first: what blocks there are
// beyond the multiprocessors then begin behind short sequences' blocks, and the longest chain does not begin last.
struct PbSequences {
    int n_seqs, from, below, few, beside, direct, recorded, lo, hi, ordered;
    unsigned long long order;
};

// The limit between short and long that holds for the step's lengths.
__device__ __forceinline__ int pb_length_limit(const int32_t* cu_q, int n_seqs, int length, int few, int beside, int lane) {
    int shorter = 0;
#pragma unroll 8
    for (int r = lane; r < n_seqs; r += 32) {
        const int n = cu_q[r + 1] - cu_q[r];
        shorter += n > 0 && n < length;
    }
    return __reduce_add_sync(0xffffffffu, shorter) <= few ? 1 : beside;
}

// Index of the `index`-th sequence of from <= tokens < below, or -1; with `all`, count: how many of them there are.  A lane has AT_ONCE
// rows under way at a time: with eight a recorded step's 256 rows are one trip to memory.
template <int AT_ONCE>
__device__ __forceinline__ int pb_nth_sequence(const int32_t* cu_q, int n_seqs, int from, int below, int index, int lane, bool all, int& count) {
    int found = -1;
    count = 0;
    for (int r0 = 0; r0 < n_seqs; r0 += 32 * AT_ONCE) {
        int n[AT_ONCE];
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            const int r = r0 + 32 * i + lane;
            n[i] = r < n_seqs ? cu_q[r + 1] - cu_q[r] : 0;
        }
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            const bool is = n[i] > 0 && n[i] >= from && n[i] < below;
            const unsigned who = __ballot_sync(0xffffffffu, is);
            const unsigned hit = __ballot_sync(0xffffffffu, is && count + __popc(who & ((1u << lane) - 1u)) == index);
            if (hit) found = r0 + 32 * i + __ffs(hit) - 1;
            count += __popc(who);
        }
        if (found >= 0 && !all) break;
    }
    return found;
}

// Calls work(sequence, limit) for the sequences that are this block's; all threads together.  RECORDED (an instance of its own: the loop
// over them costs registers): one after the other, else the one.
template <bool RECORDED, typename F>
__device__ __forceinline__ void pb_for_sequences(const int32_t* cu_q, const PbSequences& s, F work) {
    const int lane = threadIdx.x & 31;
    int count;
    if constexpr (!RECORDED) {
        const int seq = s.direct ? (s.ordered ? (int)(s.order >> (4 * blockIdx.y)) & 15 : (int)blockIdx.y) : pb_nth_sequence<4>(cu_q, s.n_seqs, s.from, s.below, blockIdx.y, lane, false, count);
        if (seq >= 0 && cu_q[seq + 1] > cu_q[seq]) work(seq, s.from);
    } else {
        int from = s.from, below = s.below;
        if (s.beside > 0) {
            if (below == INT_MAX) from = pb_length_limit(cu_q, s.n_seqs, from, s.few, s.beside, lane);
            else below = pb_length_limit(cu_q, s.n_seqs, below, s.few, s.beside, lane);
        }
        for (int index = blockIdx.y;; index += gridDim.y) {
            const int seq = pb_nth_sequence<8>(cu_q, s.n_seqs, from, below, index, lane, s.lo > 0, count);
            if (seq < 0 || (s.lo > 0 && (count < s.lo || count > s.hi))) return;
            work(seq, from);
            __syncthreads();                                // the next one's work uses the same shared memory
        }
    }
}

// Chunks of L tokens that a sequence of n has, counted from `least` tokens on.
template <int L>
__device__ __forceinline__ int pb_chunks_of(int n, int least) { return n > 0 && n >= least ? (n + L - 1) / L : 0; }

// Chunks of the sequences before `seq`.
template <int L>
__device__ __forceinline__ int pb_chunks_before(const int32_t* cu_q, int seq, int least, int lane) {
    int n = 0;
    for (int r = lane; r < seq; r += 32) n += pb_chunks_of<L>(cu_q[r + 1] - cu_q[r], least);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    return n;
}

// First token of the chunk that number `slot` of all is, and how many tokens it has (0: there is none).  A lane has four rows.
template <int L>
__device__ __forceinline__ int pb_find_chunk(const int32_t* cu_q, int n_seqs, int least, int slot, int lane, int& first) {
    int base = 0;
    for (int r0 = 0; r0 < n_seqs; r0 += 128) {
        int at[5], n = 0;
#pragma unroll
        for (int i = 0; i < 5; ++i) at[i] = cu_q[min(r0 + 4 * lane + i, n_seqs)];       // a row past the last: no tokens
#pragma unroll
        for (int i = 0; i < 4; ++i) n += pb_chunks_of<L>(at[i + 1] - at[i], least);
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, base + upto > slot);
        if (hit) {
            int left = slot - base - (upto - n), tokens = 0;       // in the lane that has the chunk: its number among the lane's
            bool found = false;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = pb_chunks_of<L>(at[i + 1] - at[i], least);
                if (!found && left < c) {
                    found = true;
                    first = at[i] + left * L;
                    tokens = min(L, at[i + 1] - first);
                }
                if (!found) left -= c;
            }
            const int owner = __ffs(hit) - 1;
            first = __shfl_sync(0xffffffffu, first, owner);
            return __shfl_sync(0xffffffffu, tokens, owner);
        }
        base += __shfl_sync(0xffffffffu, upto, 31);
    }
    return 0;
}

// Rows of a recorded launch of `each` blocks a row: twice `blocks` a multiprocessor, no more than the sequences there may be.  (256 rows
// of a step with room for 256 requests, nearly all of them empty, took 30 to 90 us; with few rows a block's sequences wait for one
// another: 60 single tokens of the gated delta rule, 32 heads, 264 us at two blocks, 244 at six.)
static inline int pb_recorded_rows(int most, long long each, int blocks) {
    const long long rows = (2ll * blocks * pb_multiprocessors() + each - 1) / each;
    return (int)(rows < most ? rows : most);
}

// Columns of a head's state that a block of a walk over chunks takes: 64, 32 or 16 (at most `widest`, a divisor of `cols`), the most
// that still gives four fifths of the multiprocessors a block when so many sequences walk: wide slices share what does not depend on
// the columns, narrow ones are a shorter chain each.  Here: the least number of sequences for which that is `width` or more.
static inline int pb_width_from(int width, int heads, int cols, int widest) {
    const int sms = pb_multiprocessors(), fill = sms - sms / 5;
    int from = INT_MAX;
    for (int w = width; w <= widest; w <<= 1) {
        if (cols % w) continue;
        const long long states = (long long)heads * (cols / w), n = (fill + states - 1) / states;
        if (n < from) from = (int)n;
    }
    return from;
}
// Calls launch(width, rows, sequences) for every width that some number of sequences up to n_long picks.  `counted`: there are n_long
// of them, and one launch; else the launches are recorded, and the number of sequences says on the device which of them works.
template <typename F>
static inline int pb_for_widths(int heads, int cols, int narrowest, int widest, PbSequences s, int n_long, int counted, F launch) {
    for (int w = narrowest; w <= widest; w <<= 1) {
        const int lo = w == narrowest ? 1 : pb_width_from(w, heads, cols, widest);
        const int next = w == widest ? INT_MAX : pb_width_from(2 * w, heads, cols, widest);
        const int hi = next <= n_long ? next - 1 : n_long;
        if (lo > hi || (counted && hi != n_long)) continue;
        s.direct = counted && s.from <= 1 && n_long == s.n_seqs; s.recorded = !counted; s.lo = lo; s.hi = hi;
        if (int e = launch(w, counted ? hi : pb_recorded_rows(hi, (long long)heads * (cols / w), 1), s)) return e;
    }
    return 0;
}
