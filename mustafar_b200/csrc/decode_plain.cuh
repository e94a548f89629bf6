// The decode kernels' products one position at a time, for the ranges whose result holds a NaN.
//
// A fragment register holds two positions of one tile and the B operand takes one of them away with a zero (BForms in
// decode_common.cuh), so an infinity or a NaN at one position also makes the sum of its partner NaN: another token's
// score, another output channel.  The kernels therefore look at what they hand out, and a CTA that finds a NaN walks its
// range again here and overwrites its results: a value then reaches its own row only.  Finite data pays for one compare
// per result (64 sequences x 32768 tokens: 1312 us before, 1299 us with the parameters in constant memory instead of copied);
// with a NaN in one of 512 kv heads the same call takes 1315 us, with one in every head 11.1 ms.  One thread per row (token
// of a block, or output channel), values straight from global memory, fp32 sums, no waits.
#pragma once

#include "decode_common.cuh"

namespace mfar {

// One 64-token block of one tensor of a kv head: the fp16 cache.  value() is false where a position is absent; a block whose
// range the staging refuses counts as empty.
struct PlainBlock {
    const unsigned long long* bm;
    const int* acc;
    const __half* vals;
    int start;
    unsigned halves;

    __device__ __forceinline__ PlainBlock(const Sparse& sp, int h, int64_t block, int cap) {
        const int64_t tile0 = block * kTilesPerBlock;
        const int64_t head0 = sp.nz_off ? 8ll * sp.nz_off[h] : h * sp.nz_hs;
        bm = sp.bmp + h * sp.bmp_hs + tile0;
        acc = sp.acc + h * sp.acc_hs + tile0;
        start = acc[0];
        const int end = acc[kTilesPerBlock];
        const bool bad = block_range_bad(start, end, static_cast<unsigned>(cap) * 2u, head0, sp.nz_extent);
        vals = sp.nz + head0 + 2ll * start;
        halves = bad ? 0u : 2u * static_cast<unsigned>(end - start);
    }
    __device__ __forceinline__ bool value(int tile, int pos, float& v) const {
        const unsigned long long b = bm[tile];
        const unsigned at = 2u * static_cast<unsigned>(acc[tile] - start) + static_cast<unsigned>(pos ? __popcll(b >> (64 - pos)) : 0);
        if (!((b >> (63 - pos)) & 1u) || at >= halves) return false;
        v = __half2float(vals[at]);
        return true;
    }
};

// ... and of the quantised one: fp16((code - zero) * scale), subtraction and product in fp32
template <int BITS, bool GROUP32>
struct PlainQuantBlock {
    const unsigned long long* bm;
    const int* off;
    const __half* scales;
    const __half* zeros;
    const unsigned* packed;
    long long packed_words;

    __device__ __forceinline__ PlainQuantBlock(const QSparse& sp, int h, int64_t block) {
        const int64_t tile0 = h * sp.meta_hs + block * kTilesPerBlock;
        constexpr int ngrp = GROUP32 ? 2 : 1;
        bm = sp.bmp + h * sp.bmp_hs + block * kTilesPerBlock;
        off = sp.tile_off + tile0;
        scales = sp.scales + tile0 * ngrp;
        zeros = sp.zeros + tile0 * ngrp;
        packed = sp.packed;
        packed_words = sp.packed_words;
    }
    __device__ __forceinline__ bool value(int tile, int pos, float& v) const {
        constexpr int per_word = 32 / BITS;
        const unsigned long long b = bm[tile];
        const int first = off[tile];
        const int words = (__popcll(b) + per_word - 1) / per_word;
        if (!((b >> (63 - pos)) & 1u) || first < 0 || static_cast<long long>(first) + words > packed_words) return false;
        const int rank = pos ? __popcll(b >> (64 - pos)) : 0;
        const unsigned code = (packed[first + rank / per_word] >> (rank % per_word * BITS)) & ((1u << BITS) - 1u);
        const int par = GROUP32 ? 2 * tile + (rank >= 32) : tile;
        v = __half2float(__float2half_rn((static_cast<float>(code) - __half2float(zeros[par])) * __half2float(scales[par])));
        return true;
    }
};

// Fused attention: the record of (kv head h, split) over blocks blk0 .. blk0 + nb - 1 of the compressed cache or, from split
// nsplit on, of the dense window.  Absent positions are zeros that take part in the sums.  red: 2 * G * 64 floats, ps:
// [G][ps_stride] halves, alpha: G floats, all in shared memory.  Called by the whole CTA (128 threads).
template <int G, int QBITS, bool GROUP32>
__device__ __noinline__ void plain_attention(const DecodeParams& p, int h, int split, int blk0, int nb, int W, float* red,
                                             unsigned short* ps, int ps_stride, float* alpha) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool is_window = split >= p.nsplit;
    const int token = tid & 63, half = tid >> 6;   // K: this thread's row and half of the channels; V: tid is the channel
    constexpr int kHeadsPerWarp = (G + 3) / 4;
    float s[G], o[G], m_run[kHeadsPerWarp], l_run[kHeadsPerWarp];
#pragma unroll
    for (int g = 0; g < G; ++g) o[g] = 0.f;
#pragma unroll
    for (int j = 0; j < kHeadsPerWarp; ++j) { m_run[j] = -INFINITY; l_run[j] = 0.f; }
    const __half* q = p.q + static_cast<int64_t>(h) * G * p.q_stride;
    const int64_t q_stride = p.q_stride;

    auto block_of = [&](bool key, int64_t block) {
        if constexpr (QBITS != 0)
            return PlainQuantBlock<QBITS, GROUP32>(key ? p.kq : p.vq, h, block);
        else
            return PlainBlock(key ? p.k : p.v, h, block, p.cap);
    };
    // scores of this thread's token over its half of the channels; value(c): K at that token
    auto scores = [&](auto value) {
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] = 0.f;
#pragma unroll 4
        for (int c = half * 64; c < half * 64 + 64; c += 2) {
            const float v0 = value(c), v1 = value(c + 1);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float2 x = __half22float2(*reinterpret_cast<const __half2*>(q + g * q_stride + c));
                s[g] = fmaf(v1, x.y, fmaf(v0, x.x, s[g]));
            }
        }
    };
    // this thread's channel over the block's tokens; value(t): V at that channel
    auto outputs = [&](auto value) {
#pragma unroll
        for (int g = 0; g < G; ++g) o[g] *= alpha[g];
#pragma unroll 4
        for (int t = 0; t < 64; t += 2) {
            const float v0 = value(t), v1 = value(t + 1);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float2 x = __half22float2(*reinterpret_cast<const __half2*>(ps + g * ps_stride + t));
                o[g] = fmaf(v1, x.y, fmaf(v0, x.x, o[g]));
            }
        }
    };

    for (int i = 0; i < nb; ++i) {
        const int tok0 = (blk0 + i) * 64;
        if (is_window) {
            const __half* w = p.kwin + h * p.win_hs + static_cast<int64_t>(tok0 + token) * p.win_ts;
            const bool there = tok0 + token < W;
            scores([&](int c) { return there ? __half2float(w[c]) : 0.f; });
        } else {
            const auto block = block_of(true, blk0 + i);
            scores([&](int c) { float v = 0.f; block.value(c, token, v); return v; });
        }
        __syncthreads();   // (everybody is done with the arrays of the block before)
#pragma unroll
        for (int g = 0; g < G; ++g) red[(half * G + g) * 64 + token] = s[g];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kHeadsPerWarp; ++j) {
            const int g = warp + 4 * j;
            if (g < G) {
                float x[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int t = lane + 32 * e;
                    x[e] = (red[g * 64 + t] + red[(G + g) * 64 + t]) * p.scale_log2;
                    if (is_window && tok0 + t >= W) x[e] = -INFINITY;
                }
                const float m_new = fmaxf(m_run[j], warp_max_f32(fmaxf(x[0], x[1])));
                const float a = fast_exp2(m_run[j] - m_new);
                float sum = 0.f;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const __half pr = __float2half_rn(fast_exp2(x[e] - m_new));   // rounded where the fragment form rounds
                    sum += __half2float(pr);
                    ps[g * ps_stride + lane + 32 * e] = __half_as_ushort(pr);
                }
                l_run[j] = l_run[j] * a + sum;
                m_run[j] = m_new;
                if (lane == 0) alpha[g] = a;
            }
        }
        __syncthreads();
        if (is_window) {
            const __half* w = p.vwin + h * p.win_hs + static_cast<int64_t>(tok0) * p.win_ts + tid;
            const int64_t ts = p.win_ts;
            outputs([&](int t) { return tok0 + t < W ? __half2float(w[t * ts]) : 0.f; });
        } else {
            const auto block = block_of(false, blk0 + i);
            outputs([&](int t) { float v = 0.f; block.value(half * 64 + t, token, v); return v; });
        }
    }
    float* rec = p.ws + (static_cast<int64_t>(h) * p.nrec + split) * G * kPartialStride;
#pragma unroll
    for (int g = 0; g < G; ++g) rec[g * kPartialStride + tid] = o[g];
#pragma unroll
    for (int j = 0; j < kHeadsPerWarp; ++j) {
        const int g = warp + 4 * j;
        if (g < G) {
            const float l = warp_sum_f32(l_run[j]);
            if (lane == 0) {
                rec[g * kPartialStride + kPartM] = m_run[j];
                rec[g * kPartialStride + kPartL] = l;
            }
        }
    }
}

// Single products of the fp16 cache, blocks blk0 .. blk0 + nb - 1 of kv head h.  Only the positions that are there are
// multiplied: a query channel or probability that is not finite reaches the rows that keep a value for it.
template <int G>
__device__ __noinline__ void plain_key_scores(const DecodeParams& p, int h, int blk0, int nb, float* red) {
    const int token = threadIdx.x & 63, half = threadIdx.x >> 6;
    const __half* q = p.q + static_cast<int64_t>(h) * G * p.q_stride;
    const int64_t q_stride = p.q_stride;
    for (int i = 0; i < nb; ++i) {
        const PlainBlock block(p.k, h, blk0 + i, p.cap);
        float s[G];
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] = 0.f;
#pragma unroll 4
        for (int c = half * 64; c < half * 64 + 64; ++c) {
            float v;
            if (block.value(c, token, v)) {
#pragma unroll
                for (int g = 0; g < G; ++g) s[g] = fmaf(v, __half2float(q[g * q_stride + c]), s[g]);
            }
        }
        __syncthreads();   // (the other half of the block before has been read)
        if (half) {
#pragma unroll
            for (int g = 0; g < G; ++g) red[g * 64 + token] = s[g];
        }
        __syncthreads();
        if (!half) {
            __half* dst = p.s_out + static_cast<int64_t>(h) * G * p.s_stride + static_cast<int64_t>(blk0 + i) * 64 + token;
#pragma unroll
            for (int g = 0; g < G; ++g) dst[g * p.s_stride] = __float2half_rn(s[g] + red[g * 64 + token]);
        }
    }
}

template <int G>
__device__ __noinline__ void plain_value_record(const DecodeParams& p, int h, int split, int blk0, int nb) {
    const int pos = threadIdx.x & 63, half = threadIdx.x >> 6;   // channel 64 * half + pos
    float o[G];
    const int64_t p_stride = p.p_stride;
#pragma unroll
    for (int g = 0; g < G; ++g) o[g] = 0.f;
    for (int i = 0; i < nb; ++i) {
        const PlainBlock block(p.v, h, blk0 + i, p.cap);
        const __half* prob = p.p_in + static_cast<int64_t>(h) * G * p_stride + static_cast<int64_t>(blk0 + i) * 64;
#pragma unroll 4
        for (int t = 0; t < 64; ++t) {
            float v;
            if (block.value(half * 64 + t, pos, v)) {
#pragma unroll
                for (int g = 0; g < G; ++g) o[g] = fmaf(v, __half2float(prob[g * p_stride + t]), o[g]);
            }
        }
    }
    float* rec = p.ws + (static_cast<int64_t>(h) * p.nrec + split) * G * kPartialStride + threadIdx.x;
#pragma unroll
    for (int g = 0; g < G; ++g) rec[g * kPartialStride] = o[g];
}

}  // namespace mfar
