// The short causal convolution of four taps over a run of neighbouring rows, for kernels in which a thread takes four
// neighbouring channels: acc = bias + sum_j w_j raw[row - 3 + j], then silu, in float32.  Inputs ahead of the step's rows come from
// the ring [slots, 4, channels] (position p at p mod 4) and are zero before the sequence's start.
//
// Bound by issue, not by memory (2,048 rows of 4,096 channels: 62 % of the issue slots, 13 % of the bandwidth, 132 instructions
// a row and warp), more so where every row looked up its slot and position and asked every tap whether it exists.  A run that lies inside one sequence, three tokens or more behind the step's first (all but one run in a long prompt's
// hundreds), asks once, turns each input into float32 once, and takes two channels an instruction.
// us on B200, before / now: 4,096 rows of 10,240 channels into planes and float32 98 / 80, 2,048 of 3,072 with unit norms 22 / 18, 2,048 of 4,096 in
// bfloat16 18 / 13.5.
#pragma once

#include "common.cuh"

namespace conv_run {

constexpr int kTaps = 4;

struct Source {
    const __nv_bfloat16* rows;     // the run's first row, at the thread's first channel
    long long row_stride;
    const __nv_bfloat16* ring;     // [slots][kTaps][channels], at the thread's first channel
    int channels;
    const int* row_slot;
    const int* row_pos;
    const int* seq_lens;           // tokens a slot held before the step
};

__device__ __forceinline__ unsigned long long floats_of(uint32_t two) { return pack2(__uint_as_float(two << 16), __uint_as_float(two & 0xffff0000u)); }

// Steps of few entries, for which the time of a launch counts: every row finds its place alone, all rows' places and the sequences' lengths
// ahead of the first result.  (A first look that decides between two ways waits once more, and more instructions are fetched; us with / without, 16 to 512 rows
// of 1,024 channels 5.2 / 4.4, 100 rows of 10,240 5.7 / 5.5, 2,048 of 1,024 6.6 / 7.1, 512 of 4,096 6.3 / 7.0.)
constexpr long long kFewEntries = 1200000;
inline bool few_entries(int n_rows, int channels) { return (long long)n_rows * channels <= kFewEntries; }

// put(r, y): the four results of row r, for r in [0, n_here).  w[i][j]: tap j of channel i.  `first`: the run's first row's number.
template <int ROWS, bool FEW, typename Put>
__device__ __forceinline__ void run(const Source& s, int first, int n_here, const float (&w)[4][kTaps], const float (&bias)[4], Put&& put) {
    uint2 raw[ROWS + kTaps - 1];       // raw[j]: the row j - 3 rows after `first`
#pragma unroll
    for (int j = 0; j < ROWS + kTaps - 1; ++j) {
        const int back = kTaps - 1 - j;
        raw[j] = back <= first && -back < n_here ? *reinterpret_cast<const uint2*>(s.rows - (long long)back * s.row_stride) : make_uint2(0, 0);
    }
    int slot[ROWS], pos[ROWS], local[ROWS];       // (FEW) local: a row's index among its sequence's rows of this step
    bool inside = false;
    if constexpr (FEW) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            slot[r] = s.row_slot[first + min(r, n_here - 1)];
            pos[r] = s.row_pos[first + min(r, n_here - 1)];
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) local[r] = pos[r] - s.seq_lens[slot[r]];
    } else {
        const int slot0 = s.row_slot[first], pos0 = s.row_pos[first], last = first + n_here - 1;
        const int slot1 = s.row_slot[last], pos1 = s.row_pos[last];
        inside = n_here == ROWS && slot0 == slot1 && pos1 - pos0 == ROWS - 1 && pos0 - s.seq_lens[slot0] >= kTaps - 1;
    }
    if (inside) {
        unsigned long long w01[kTaps], w23[kTaps], x01[kTaps], x23[kTaps];
        const unsigned long long b01 = pack2(bias[0], bias[1]), b23 = pack2(bias[2], bias[3]);
#pragma unroll
        for (int j = 0; j < kTaps; ++j) {
            w01[j] = pack2(w[0][j], w[1][j]);
            w23[j] = pack2(w[2][j], w[3][j]);
            x01[j] = floats_of(raw[j].x);
            x23[j] = floats_of(raw[j].y);
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            x01[(r + kTaps - 1) % kTaps] = floats_of(raw[r + kTaps - 1].x);
            x23[(r + kTaps - 1) % kTaps] = floats_of(raw[r + kTaps - 1].y);
            unsigned long long a01 = b01, a23 = b23;
#pragma unroll
            for (int j = 0; j < kTaps; ++j) {
                a01 = fma2(w01[j], x01[(r + j) % kTaps], a01);
                a23 = fma2(w23[j], x23[(r + j) % kTaps], a23);
            }
            float y[4];
            unpack2(a01, y[0], y[1]);
            unpack2(a23, y[2], y[3]);
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] = silu_of<__nv_bfloat16>(y[i]);
            put(r, y);
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (r >= n_here) break;
        if constexpr (!FEW) {
            slot[r] = s.row_slot[first + r];
            pos[r] = s.row_pos[first + r];
            local[r] = pos[r] - s.seq_lens[slot[r]];
        }
        uint2 in[kTaps];
#pragma unroll
        for (int j = 0; j < kTaps; ++j) in[j] = raw[r + j];
        if (local[r] < kTaps - 1) {
#pragma unroll
            for (int back = 1; back < kTaps; ++back) {
                if (back <= local[r]) continue;
                in[kTaps - 1 - back] = back > pos[r] ? make_uint2(0, 0)           // before the sequence's start
                    : *reinterpret_cast<const uint2*>(s.ring + ((size_t)slot[r] * kTaps + (pos[r] - back) % kTaps) * s.channels);
            }
        }
        float y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float acc = bias[i];
#pragma unroll
            for (int j = 0; j < kTaps; ++j) {
                if (kTaps - 1 - j > pos[r]) continue;
                const uint32_t two = i < 2 ? in[j].x : in[j].y;
                acc = fmaf(w[i][j], __uint_as_float(i & 1 ? two & 0xffff0000u : two << 16), acc);
            }
            y[i] = silu_of<__nv_bfloat16>(acc);
        }
        put(r, y);
    }
}

}  // namespace conv_run
