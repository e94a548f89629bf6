// Building blocks shared by the fp16 and the quantised decode kernels:
// mbarrier / bulk-copy wrappers (1-D cp.async.bulk, no multicast), the expansion of bitmap tiles
// into tensor-core fragments, the split-KV partial record and the launch parameters.
#pragma once

#include "common.cuh"

namespace mfar {

// ---------------------------------------------------------------- mbarrier + TMA 1-D bulk copy
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false when the limit ran out (caller records MFAR_DEV_TIMEOUT and leaves).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_timer_ns();
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (global_timer_ns() - t0 > kWaitLimitNs) return false;
    }
}
// global -> this CTA's shared memory; src/dst 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst_smem)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// ---------------------------------------------------------------- small math helpers
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float warp_max_f32(float v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, d));
    return v;
}
__device__ __forceinline__ float warp_sum_f32(float v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
    return v;
}

// A lane owns byte `kb` of a tile's 64-bit bitmap (bit 63-i = element i), i.e. positions 8*kb .. 8*kb+7: sel / mh / ml
// are the lane constants that extract that byte and mask the bits in front of it (hi, lo = the bitmap's words).  The rank
// of the lane's first position is the popcount of the bits before its byte.
__device__ __forceinline__ void lane_byte_constants(int kb, unsigned& sel, unsigned& mh, unsigned& ml) {
    sel = 7u - kb;
    mh = kb == 0 ? 0u : (kb >= 4 ? 0xffffffffu : (0xffffffffu << (32 - 8 * kb)));
    ml = kb <= 4 ? 0u : (0xffffffffu << (64 - 8 * kb));
}

__device__ __forceinline__ unsigned ldg_nc_u32(const void* p) {
    unsigned v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// ---------------------------------------------------------------- tensor-core fragments of decoded tiles
__device__ __forceinline__ void mma16816(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                         unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A fragments: register k of a tile's byte holds two of its 8 positions, pair_pos(k, 0) in the low half and
// pair_pos(k, 1) in the high half, zero where the bit is clear.  Which two is free (the B operand tells them apart):
// fp16 values and 4-bit codes pair k with k + 4, 2-bit codes 2k with 2k + 1.
template <int QBITS>
__host__ __device__ constexpr int pair_pos(int k, int par) { return QBITS == 2 ? 2 * k + par : k + 4 * par; }

// One tile of packed halves: every set bit of byte `sel` takes the next half (a predicated load); the two half bytes
// have a read pointer each.
__device__ __forceinline__ void expand_tile(unsigned lo, unsigned hi, const unsigned short* vals, unsigned sel, unsigned mh,
                                            unsigned ml, unsigned (&r)[4]) {
    const unsigned byte = __byte_perm(lo, hi, sel);
    const unsigned short* p0 = vals + (__popc(hi & mh) + __popc(lo & ml));
    const unsigned short* p1 = p0 + __popc(byte & 0xf0u);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        unsigned v = 0;
        if (byte & (0x80u >> k)) { v = *p0; ++p0; }
        if (byte & (0x08u >> k)) { const unsigned h = *p1; ++p1; v = __byte_perm(v, h, 0x5410); }
        r[k] = v;
    }
}

// Where a tile's coefficient (query channel, probability) goes in the B operand: a register of A holds two positions of
// ONE tile, so it enters B as (c, 0) for the first position and as (0, c) for the second.  Up to 4 query heads fill the 8
// columns with both forms (column = head + 4 * form); 8 heads take one mma per form.  The zero does not take an infinity or a
// NaN away: results with a NaN are computed again without pairs (decode_plain.cuh).
template <int G>
struct BForms {
    static constexpr int FORMS = G == 8 ? 2 : 1;
    int head;              // query head whose coefficients this lane loads
    unsigned sel0, sel1;   // place the low / high half of a register of two adjacent tiles' coefficients
    int ahead, aform;      // head of accumulator column 2*cp (and + 1), and its form (G <= 4)
    __device__ __forceinline__ BForms(int tb, int cp) {
        head = G == 8 ? tb : (tb & 3);
        const bool second = G != 8 && tb >= 4;
        sel0 = second ? 0x1044u : 0x4410u;
        sel1 = second ? 0x3244u : 0x4432u;
        ahead = G == 8 ? 2 * cp : 2 * (cp & 1);
        aform = G == 8 ? 0 : cp >> 1;
    }
    // position inside the lane's byte of register k of an accumulator of form f
    template <int QBITS>
    __device__ __forceinline__ int pos(int k, int f) const {
        return FORMS == 2 ? pair_pos<QBITS>(k, f) : (aform ? pair_pos<QBITS>(k, 1) : pair_pos<QBITS>(k, 0));
    }
};

// d[f][j] += the eight tiles of a step (r1: tile 2*cp, r2: tile 2*cp + 1 of the lane's column) times their coefficients cc
template <int G>
__device__ __forceinline__ void mma_step(float (&d)[BForms<G>::FORMS][2][4], const unsigned (&r1)[4], const unsigned (&r2)[4],
                                         const BForms<G>& bf, unsigned cc) {
    const unsigned b0 = __byte_perm(cc, 0u, bf.sel0), b1 = __byte_perm(cc, 0u, bf.sel1);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        mma16816(d[0][j], r1[2 * j], r1[2 * j + 1], r2[2 * j], r2[2 * j + 1], b0, b1);
        if (BForms<G>::FORMS == 2)
            mma16816(d[BForms<G>::FORMS - 1][j], r1[2 * j], r1[2 * j + 1], r2[2 * j], r2[2 * j + 1], b0 << 16, b1 << 16);
    }
}

template <int G>
__device__ __forceinline__ void load_coef(const float* p, float (&c)[G]) {
    if constexpr (G == 1) {
        c[0] = p[0];
    } else if constexpr (G == 2) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        c[0] = t.x; c[1] = t.y;
    } else {
#pragma unroll
        for (int g = 0; g < G; g += 4) {
            const float4 t = *reinterpret_cast<const float4*>(p + g);
            c[g] = t.x; c[g + 1] = t.y; c[g + 2] = t.z; c[g + 3] = t.w;
        }
    }
}

// Split-KV partial of one (kv head, split, q head of the group): 128 un-normalised
// output channels, then the running max (log2 domain) and the running sum.
constexpr int kPartialStride = kD + 4;  // floats; keeps records 16-byte aligned
constexpr int kPartM = kD;
constexpr int kPartL = kD + 1;

enum { MODE_KEY = 1, MODE_VALUE = 2 };
constexpr int kSlackHalves = 64;  // a decode never reads further than this past a stage's values
constexpr int kMaxBlocksPerSplit = 256;
// splits per kv head, whatever a caller asks for; the fp16 cache takes more where kMaxBlocksPerSplit needs them
constexpr int kMaxSplits = 480;

struct Sparse {
    const unsigned long long* bmp;
    const int* acc;
    const __half* nz;
    const int* nz_off;
    int64_t bmp_hs, acc_hs, nz_hs;
    int64_t nz_extent;   // halves addressable from nz (0 = unknown: the extent check is skipped)
};

// one tensor of the quantised cache (mfar_compress_quant)
struct QSparse {
    const unsigned long long* bmp;
    const int* tile_off;
    const __half* scales;
    const __half* zeros;
    const unsigned* packed;
    int64_t bmp_hs, meta_hs;
    long long packed_words;
};

template <int BITS_>
struct QBuf {   // one staged tensor of one 64-token block of the quantised cache
    static constexpr int BITS = BITS_;
    static constexpr int WPT = 64 * BITS_ / 32;  // words per tile slot
    uint2 bm[128];
    unsigned sz[128 * 2];                        // (scale | zero << 16) per group
    unsigned words[128 * WPT + 4];
};

struct DecodeParams {
    Sparse k, v;
    QSparse kq, vq;        // fused attention over the quantised cache (k, v unused then)
    const __half* q;       // [Bq][q_stride]
    int64_t q_stride;
    const __half* kwin;    // dense window [Bh][W][128]
    const __half* vwin;
    int64_t win_hs, win_ts;
    int W;
    const int* W_dev;      // optional: window length in device memory (then W is its upper bound)
    const int* L_dev;      // optional: compressed tokens in device memory (then nblk is their upper bound, in blocks)
    int nblk, nsplit, bps; // compressed blocks, splits over them, blocks per split
    int cap;               // halves of packed values a stage can hold per tensor
    float scale_log2;      // softmax scale * log2(e)
    float* ws;             // split partials
    int nrec;              // partial records per kv head in ws
    __half* s_out;         // MODE_KEY  : [Bq][s_stride]
    int64_t s_stride;
    int rows;              // MODE_KEY  : result rows per query head; row 0 is the product, the rest is zero-filled
    int64_t row_stride;
    const __half* p_in;    // MODE_VALUE: [Bq][p_stride]
    int64_t p_stride;
    unsigned* dev_status;
    int nwin, wbps;        // CTAs (and records) per kv head for the dense window behind the nsplit ones, 64-token blocks each
    // fused attention only: the CTA that finishes a kv head last merges its records into out
    unsigned* counters;    // one per kv head, zero between launches; NULL = no merge (a combine launch follows)
    __half* out;
    int64_t out_stride;
};

// The first kCounterBytes of every decode workspace hold one arrival counter per kv head (fused attention); the
// split records of every entry point start behind them, whatever the head count, so that calls of different shapes
// can share a workspace without touching each other's counters.
constexpr size_t kCounterBytes = 64 * 1024;
constexpr int kMaxCountedHeads = static_cast<int>(kCounterBytes / 4);
inline size_t counters_bytes(int) { return kCounterBytes; }
// the fused kernel's merge keeps a weight per query head and record in its reduction buffer, 4 * kD floats per query head;
// with more records (or more kv heads than counters) they are merged by a second launch
constexpr int kMaxMergedRecords = 4 * kD;
inline unsigned* merge_counters(void* workspace, int n_kv_heads, int nrec) {
    return n_kv_heads <= kMaxCountedHeads && nrec <= kMaxMergedRecords ? static_cast<unsigned*>(workspace) : nullptr;
}

// Checks one 64-token block's packed range before it is copied: block start `blk` and end `nxt` in uint32 units
// (entries of accum), stage capacity `capb` in bytes, start of the head inside nz and the extent of nz in halves.
// A bulk copy needs a 16-byte aligned source and a size that is a multiple of 16 bytes.
__device__ __forceinline__ bool block_range_bad(int blk, int nxt, unsigned capb, int64_t head_start_halves,
                                                int64_t nz_extent) {
    const long long d = (static_cast<long long>(nxt) - blk) * 4;
    bool bad = d < 0 || d > capb || blk < 0 || (blk & 3) || (d & 15);
    if (nz_extent > 0) bad |= head_start_halves + 2ll * nxt > nz_extent;
    return bad;
}

// fused decode attention (decode_attn.cu): grid (grid_x, n_kv_heads); G in {1, 2, 4, 8}
int launch_decode_attn(const DecodeParams& p, int G, int n_kv_heads, int grid_x, cudaStream_t s);
// the same over the quantised cache p.kq / p.vq: bits in {2, 4}, group32 = a second scale / zero-point from nonzero 32 on
int launch_decode_attn_quant(const DecodeParams& p, int G, int bits, bool group32, int n_kv_heads, int grid_x,
                             cudaStream_t s);
// merge of the split-KV records (normalise = 1) or plain sum (normalise = 0), one CTA per q head
// (rows > 1: rows 1.. of every head, row_stride apart, are zero-filled)
int launch_combine(const float* ws, int nrec, int G, int normalise, void* out, int64_t out_stride, int n_q_heads,
                   cudaStream_t s, int rows = 1, int64_t row_stride = 0);

// Zero-fills rows 1 .. rows - 1 (row 0 too with `first` = 0) of one 64-token block's scores for G query heads, 16 bytes a
// store: a separate fill of the padded result would move it through memory a second time.
template <int G>
__device__ __forceinline__ void zero_score_rows(__half* block, int64_t head_stride, int rows, int64_t row_stride, int first) {
    const int per_head = (rows - first) * 8;
    for (int i = threadIdx.x; i < G * per_head; i += blockDim.x) {
        const int g = i / per_head, r = first + (i % per_head) / 8;
        *reinterpret_cast<uint4*>(block + g * head_stride + r * row_stride + 8 * (i & 7)) = make_uint4(0u, 0u, 0u, 0u);
    }
}

// The dense window of a kv head is dealt out over p.nwin CTAs of p.wbps 64-token blocks.  A window block reads its K and
// then its V rows straight from global memory, two exposed trips per block, so a CTA with all blocks outlasts a short split
// (8 kv heads x 1024 tokens, window 384: 20.8 us with one CTA, 10.1 us with six).  A window CTA takes half of a split's
// blocks, so that it does not outlast one.  More CTAs also cost: where they push a grid of k <= 5 CTAs per SM beyond k, a
// few SMs with one CTA too many are what the call waits for (8 x 10240, window 128: 18.8 us with one window CTA, 25.4 us with
// two).  They are then only as many as fit, provided that none gets more than 4/3 of a split's blocks.
// Measured over 8 .. 256 kv heads, 512 .. 32768 tokens, windows of 65 .. 384, fp16 with 4 and 8 query heads and 2-bit codes
// (1530 calls): 6.0 % less time on average than one CTA for the window, more than 3 % slower than that in 25 calls (12 % at
// worst).  The first form, one block per CTA while the grid stayed under 4 CTAs per SM and no look at k: 4.5 % less time,
// more than 3 % slower in 106 calls (42 % at worst).
// records: what the workspace has room for (at least nsplit + 1).
constexpr int kMaxWindowSplits = 16;
inline int window_records(int window) {
    const int nwb = (window + 63) / 64;
    return nwb < 1 ? 1 : (nwb < kMaxWindowSplits ? nwb : kMaxWindowSplits);
}
inline void split_window(DecodeParams& p, int n_kv_heads, int n_sm, long long records) {
    const int nwb = (p.W + 63) / 64;
    p.nwin = p.wbps = 0;
    if (nwb > 0) {
        const long long fit = static_cast<long long>(n_sm > 0 ? n_sm : 1);
        auto per_sm = [&](int nwin) { return (static_cast<long long>(n_kv_heads) * (p.nsplit + nwin) + fit - 1) / fit; };
        auto ctas = [&](int blocks) { return (nwb + blocks - 1) / blocks; };
        int wb = p.bps / 2 < 1 ? 1 : p.bps / 2;
        const long long k = per_sm(1);
        if (k <= 5 && per_sm(ctas(wb)) > k) {
            const long long room = k * fit / n_kv_heads - p.nsplit;   // >= 1: one window CTA fits
            const int blocks = ctas(static_cast<int>(room < nwb ? room : nwb));
            if (3 * blocks <= 4 * p.bps) wb = blocks;
        }
        long long most = records - p.nsplit;
        if (most > kMaxWindowSplits) most = kMaxWindowSplits;
        const int least = static_cast<int>((nwb + most - 1) / most);
        if (wb < least) wb = least;
        if (wb > nwb) wb = nwb;
        p.wbps = wb;
        p.nwin = ctas(wb);
    }
    p.nrec = p.nsplit + p.nwin;
}

// Split count of the 64-token-block decode kernels.  The grid is n_kv_heads * ns CTAs of bps = ceil(nblk / ns) blocks.
// The cost of a candidate follows a model fitted to a sweep of ns over batch 1..64 and 4k..32k tokens with the kernel that
// had 4 CTAs per SM and one window CTA (all times in units of one block on an otherwise idle SM, ~2 us):
//   * a CTA costs w = bps + 1.1 (prologue, partial record);
//   * x = CTAs / SMs is the load per SM; an SM's throughput with o = min(x, 4) resident CTAs is
//     rate(o) = 1 / 2 / 2.76 / 2.13 at o = 1 / 2 / 3 / 4, linear in between (the dip at 4 is the fit's
//     way of saying that a grid which fits in one not-quite-full wave beats one that needs two);
//   * the last, partly filled wave costs another 0.8 w once the SMs hold more than one CTA;
//   * merging the records adds 0.035 per record.
// The kernels have changed since (5 CTAs per SM for most, window CTAs, cheaper codes).  Measured with them over 150 shapes
// (8 .. 512 kv heads x 1024 .. 32768 tokens, window 128, 1, 4 and 8 query heads, fp16 and 2-bit): the pick costs 2.3 % more
// than the best swept ns on average, more than 2 % in 38 of them, at worst 12 % for fp16 (256 kv heads x 1024 tokens, 1 query
// head: 2 splits, 4 are better) and 22 % for 2-bit codes (8 x 1024: 16 splits of the model, of which the quantised call uses
// half).  A refit to 5 CTAs per SM gave 2.4 % instead of 4.3 % over 136 shapes but made 7 x 10176 tokens with 8 query heads
// 106 -> 114 us and 8 x 4096 of 4-bit codes 70 -> 79 us: one model does not fit all variants.
inline int model_split_count(int n_kv_heads, int nblk, int min_ns, int max_ns, int n_sm) {
    if (max_ns > nblk) max_ns = nblk;
    if (min_ns < 1) min_ns = 1;
    if (n_sm < 1) n_sm = 1;
    int ns = min_ns;
    double best = -1.0;
    for (int cand = min_ns; cand <= max_ns; ++cand) {
        const int bps = (nblk + cand - 1) / cand;
        const int real = (nblk + bps - 1) / bps;
        const double x = static_cast<double>(n_kv_heads) * real / n_sm;
        const double w = bps + 1.1;
        double cost = w;
        if (x > 1.0) {
            const double o = x < 4.0 ? x : 4.0;
            const double rate = o < 2.0 ? o : (o < 3.0 ? 2.0 + 0.76 * (o - 2.0) : 2.76 - 0.63 * (o - 3.0));
            cost = x * w / rate + 0.8 * w * (x - 1.0 < 1.0 ? x - 1.0 : 1.0);
        }
        cost += 0.035 * real;
        if (best < 0 || cost < best) {
            best = cost;
            ns = real;
        }
    }
    return ns;
}

}  // namespace mfar
