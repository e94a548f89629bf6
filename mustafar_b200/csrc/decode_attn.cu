// Fused decode attention over the bitmap + packed-fp16 cache:
//   q.K^T over the compressed tokens, online softmax, P.V, split-KV partial records, and the merge of the
//   records by the CTA that finishes a kv head last (one launch per call); further CTAs per kv head handle
//   the dense recent-token window.
//
// A CTA (4 warps) walks a range of 64-token blocks of ONE kv head and serves all G query heads that share it, so
// the compressed bytes are read once.  Per block the two bitmap arrays (1 KiB each) and the two packed-value
// ranges travel into a 2-stage shared-memory ring by 1-D bulk copies (cp.async.bulk + mbarrier, no multicast),
// issued by one thread one block ahead.
//
// Decode: a lane owns one BYTE (8 positions) of the bitmaps of TWO tiles.  The rank of the byte's first position is
// the popcount of the bitmap bits before it; every set bit then takes the next packed half from shared memory
// (a predicated 16-bit load), absent positions stay zero, and two positions of a tile share a 32-bit register.  Those
// registers ARE fragments of mma.sync.m16n8k16 (fp16 in, fp32 accumulate):
//   K phase   S[token][head]   = sum_c K[token][c] q[c][head]     rows = tokens,   k = channels (= K tiles)
//   V phase   O[channel][head] = sum_t V[t][channel] p[t][head]   rows = channels, k = tokens   (= V tiles)
// The two positions of a register are told apart by the B operand (BForms in decode_common.cuh): up to 4 query heads
// fill the 8 columns twice, 8 heads take two instructions.  Against registers that pair two TILES this halves the
// accumulators of up to 4 heads (128 -> 96 registers, 5 CTAs per SM instead of 4) and the score stores: 64 sequences x
// 32768 tokens, 4 heads per kv head, 1361 -> 1327 us; 7 x 10176 tokens, 8 heads, 110 -> 106 us.  Over 360
// shapes each (8 .. 512 kv heads x 256 .. 32768 tokens, window dealt out) 2, 4 and 8 heads take 10, 10 and 6 % less time than
// that form, one head 7 % less, but 3 .. 8 % more at 16 .. 56 kv heads x 4096 tokens and up (4 CTAs per SM with 128 registers
// there: 4 % more over all shapes).  What the kernel waits for now is the shared-memory traffic of the
// predicated loads: 71 % of the data pipe, 62 % of the issue slots, neither saturated.
//
// The same kernel serves the quantised cache (QBITS = 2 or 4): there a tile's code words, bitmap, scale and zero-point
// are staged by the threads themselves (4-byte cp.async, one tile of each tensor per thread, one block ahead); a lane
// takes the codes of its byte out of a 32-bit window that starts at its rank, moves them to their positions with two
// masked shifts (masks from a 2 KiB table indexed by the bitmap byte) and turns them into fp16((code - zero) * scale) two
// at a time: 2-bit codes by a byte permute out of the tile's four values, which the staging thread computes in fp32 - the
// reference's arithmetic (kernel_quant/csrc/SpMM_Kernel_Quant.cuh:235-240) -, 4-bit codes by an exact fp16 subtraction
// and one rounded product, which gives the same bits (zero-points outside +-1024 go through fp32).  Against one
// predicated step per position: 32 x 16384 tokens of 2-bit codes 583 -> 450 us, 8 x 4096 of 4-bit codes with a scale per
// 32 nonzeros, half of the values kept, 82.7 -> 69.6 us.  The integer pipe, issue and the shared-memory pipe are each used
// to about 60 %.
#include "decode_plain.cuh"

namespace mfar {

constexpr int kAWarps = 4;
constexpr int kAThreads = kAWarps * 32;
constexpr int kAStages = 2;
constexpr int kPsStride = 72;      // halves per probability row: 36 words, so the 8 head rows fall in different banks
constexpr int kPlaneStride = 72;   // floats per (warp, head) score plane

__host__ __device__ inline size_t attn_stage_bytes(int cap) {
    return 2 * (1024 + (static_cast<size_t>(cap) + kSlackHalves) * 2);
}

struct SpreadTable { uint2 e[256]; };

struct AttnLayout {
    size_t stages, bars, ps, red, alpha, koff, voff, kblk, vblk, spread, total;
    size_t s_kbm, s_vbm, s_kval, s_vval;
    // qbuf_bytes > 0: quantised cache, a stage is two QBuf (K then V) instead of bitmaps + packed halves
    __host__ __device__ AttnLayout(int cap, int G, size_t qbuf_bytes = 0) {
        s_kbm = 0;
        s_vbm = 1024;
        s_kval = 2048;
        s_vval = 2048 + (static_cast<size_t>(cap) + kSlackHalves) * 2;
        size_t o = 0;
        stages = o; o += kAStages * (qbuf_bytes ? 2 * qbuf_bytes : attn_stage_bytes(cap));
        bars = o;   o += 64;
        ps = o;     o += 8 * kPsStride * 2;
        red = o;    o += static_cast<size_t>(kAWarps) * G * kD * 4;   // score planes, later the output reduction
        alpha = o;  o += 64;
        koff = voff = kblk = vblk = spread = o;
        if (qbuf_bytes) {
            o += sizeof(SpreadTable);
        } else {
            o += 2 * 128 * 4;
            voff = o;   o += 2 * 128 * 4;
            kblk = o;   o += (kMaxBlocksPerSplit + 4) * 4;
            vblk = o;   o += (kMaxBlocksPerSplit + 4) * 4;
        }
        total = o;
    }
};

// byte permute with the full selector (bit 3 of a nibble replicates the byte's sign)
__device__ __forceinline__ unsigned prmt(unsigned a, unsigned b, unsigned s) {
    unsigned d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
    return d;
}

__device__ __forceinline__ void cp_async4(void* dst_smem, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// ---- quantised tiles
// A lane's codes are consecutive in the tile's code words from bit rank * BITS on.  They are spread to their positions
// inside a register, four positions (half a bitmap byte) at a time: an element moves up by the number of absent positions
// in front of it, first by two (mask `two`, set where such an element arrives), then by one (mask `one`).  Table entry of a
// bitmap byte (bit 7 = first position), read from shared memory:
//   2-bit codes: x = two | one << 16 (2 bits per position), y = 4 in the nibble of every absent position
//   4-bit codes: x = two, y = one (4 bits per position)
template <int BITS>
constexpr SpreadTable make_spread_table() {
    SpreadTable t{};
    for (unsigned byte = 0; byte < 256; ++byte) {
        unsigned two = 0, one = 0, absent = 0;
        for (int half = 0; half < 2; ++half) {
            int rank = 0;
            for (int i = 0; i < 4; ++i) {
                const int pos = 4 * half + i;
                if ((byte >> (7 - pos)) & 1u) {
                    const int d = i - rank;
                    if (d & 2) two |= ((1u << BITS) - 1u) << (BITS * (4 * half + rank + 2));
                    if (d & 1) one |= ((1u << BITS) - 1u) << (BITS * pos);
                    ++rank;
                } else {
                    absent |= 4u << (4 * pos);
                }
            }
        }
        t.e[byte].x = BITS == 2 ? (two | one << 16) : two;
        t.e[byte].y = BITS == 2 ? absent : one;
    }
    return t;
}
static __device__ const SpreadTable g_spread2 = make_spread_table<2>();
static __device__ const SpreadTable g_spread4 = make_spread_table<4>();

// One staged tensor of one 64-token block.  par, one entry per 64 or 32 nonzeros of a tile:
//   2-bit: the four dequantised fp16 values as bytes, x = low bytes, y = high bytes
//   4-bit: x = scale, y = -(1024 + zero-point), each twice as fp16; a zero-point for which fp16 would not give code - zero
//          exactly (no integer, or beyond +-1024) has y = kWideZero and x = (scale | zero << 16)
constexpr unsigned kWideZero = 0xffffffffu;   // a pair of NaNs, which no zero-point in range gives
template <int BITS_, bool GROUP32>
struct AttnQBuf {
    static constexpr int BITS = BITS_;
    static constexpr int WPT = 64 * BITS_ / 32;  // code words per tile slot
    static constexpr int NG = GROUP32 ? 2 : 1;
    uint2 bm[128];
    uint2 par[128 * NG];
    unsigned words[128 * WPT + 4];
};

// (code - zero) * scale in fp32, rounded to fp16 once, for the four 2-bit codes
__device__ __forceinline__ uint2 dequant_bytes(float scale, float zero) {
    unsigned v[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const __half2 h = __floats2half2_rn((static_cast<float>(2 * j) - zero) * scale, (static_cast<float>(2 * j + 1) - zero) * scale);
        v[j] = *reinterpret_cast<const unsigned*>(&h);
    }
    return make_uint2(__byte_perm(v[0], v[1], 0x6420), __byte_perm(v[0], v[1], 0x7531));
}

__device__ __forceinline__ uint2 dequant_pair(float scale, float zero, unsigned raw) {
    if (!(fabsf(zero) <= 1024.f) || zero != rintf(zero)) return make_uint2(raw, kWideZero);
    const __half2 s = __float2half2_rn(scale), c = __float2half2_rn(-(1024.f + zero));
    return make_uint2(*reinterpret_cast<const unsigned*>(&s), *reinterpret_cast<const unsigned*>(&c));
}

// 0xffff per half: bit 7 of byte 0 / bit 7 of byte `second`, replicated (prmt's selectors 8.. copy a byte's sign)
template <int SECOND>
__device__ __forceinline__ unsigned half_mask(unsigned x) { return prmt(x, 0u, SECOND == 1 ? 0x9988u : 0xaa88u); }

// 2-bit codes at their positions (4 bits per position, code in the low two) -> pairs (2k, 2k + 1).
// One value table: 4..7 = absent = the zero operand of the byte permute.
__device__ __forceinline__ void codes_to_halves2(unsigned codes, uint2 par, unsigned (&r)[4]) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const unsigned c = j ? codes >> 16 : codes;
        const unsigned l = __byte_perm(par.x, 0u, c), h = __byte_perm(par.y, 0u, c);
        r[2 * j] = __byte_perm(l, h, 0x5140);
        r[2 * j + 1] = __byte_perm(l, h, 0x7362);
    }
}
// Two value tables: 4..7 = the second one; absent positions (bit 2 of a nibble of `absent`) are masked.
__device__ __forceinline__ void codes_to_halves2(unsigned codes, unsigned absent, uint2 par0, uint2 par1, unsigned (&r)[4]) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const unsigned c = j ? codes >> 16 : codes;
        const unsigned l = __byte_perm(par0.x, par1.x, c), h = __byte_perm(par0.y, par1.y, c);
        // nibbles of byte j*2 are positions 4j, 4j + 1: bring their bit 2 to bit 7 of two bytes
        const unsigned a = __byte_perm(absent << 5, absent << 1, j ? 0x7362 : 0x5140);
        r[2 * j] = __byte_perm(l, h, 0x5140) & ~half_mask<1>(a);
        r[2 * j + 1] = __byte_perm(l, h, 0x7362) & ~half_mask<1>(a >> 16);
    }
}

// 4-bit codes at their positions -> pairs (k, k + 4); `present` has one bit per position, first position in bit 7;
// `later` (two groups) is 0xf at the positions that use the second parameters.
template <bool GROUP32>
__device__ __forceinline__ void codes_to_halves4(unsigned codes, unsigned present, unsigned later, uint2 par0, uint2 par1, unsigned (&r)[4]) {
    const unsigned both = present | (present << 12);   // byte 0: positions 0.., byte 1: positions 4.., first in the top bit
    if (par0.y == kWideZero || (GROUP32 && par1.y == kWideZero)) {   // rare: the same in fp32
        float s[2], z[2];
#pragma unroll
        for (int g = 0; g < (GROUP32 ? 2 : 1); ++g) {
            const uint2 par = g ? par1 : par0;
            const unsigned short sh = static_cast<unsigned short>(par.x & 0xffffu);
            s[g] = __half2float(__ushort_as_half(sh));
            z[g] = par.y == kWideZero ? __half2float(__ushort_as_half(static_cast<unsigned short>(par.x >> 16)))
                                      : -1024.f - __half2float(__ushort_as_half(static_cast<unsigned short>(par.y & 0xffffu)));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int sh = 4 * (k + 4 * e);
                const bool g = GROUP32 && ((later >> sh) & 1u);
                v[e] = (static_cast<float>((codes >> sh) & 15u) - (g ? z[GROUP32 ? 1 : 0] : z[0])) * (g ? s[GROUP32 ? 1 : 0] : s[0]);
            }
            const __half2 h2 = __floats2half2_rn(v[0], v[1]);
            r[k] = *reinterpret_cast<const unsigned*>(&h2) & half_mask<1>(both << k);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        unsigned s = par0.x, c = par0.y;
        if (GROUP32) {
            const unsigned m = half_mask<2>(k == 0 ? later << 4 : later >> (4 * (k > 0 ? k - 1 : 0)));
            s = (s & ~m) | (par1.x & m);
            c = (c & ~m) | (par1.y & m);
        }
        // 1024 + code, minus (1024 + zero): exact, so the one rounding is the product's, as in fp32
        const unsigned q = ((codes >> (4 * k)) & 0x000f000fu) | 0x64006400u;
        const __half2 d = __hadd2(*reinterpret_cast<const __half2*>(&q), *reinterpret_cast<const __half2*>(&c));
        const __half2 v = __hmul2(d, *reinterpret_cast<const __half2*>(&s));
        r[k] = *reinterpret_cast<const unsigned*>(&v) & half_mask<1>(both << k);
    }
}

// Codes in packed order (from bit 0) to their positions, both halves of a byte at once: `first` = the nonzeros of its first
// half.  2-bit codes of one tile in 16 bits; 4-bit codes in 32.
template <int BITS>
__device__ __forceinline__ unsigned split_halves(unsigned w, int first) {
    return __byte_perm(w, w >> (BITS * first), BITS == 2 ? 0x0040 : 0x5410);
}
template <int BITS>
__device__ __forceinline__ unsigned spread_codes(unsigned x, unsigned two, unsigned one) {
    x = (x & ~two) | ((x << (2 * BITS)) & two);
    return (x & ~one) | ((x << BITS) & one);
}
// 2 -> 4 bits per position: half 0 / 1 of x
__device__ __forceinline__ unsigned widen_codes(unsigned x, int half) {
    unsigned y = __byte_perm(x, 0u, half ? 0x4342 : 0x4140);
    y = (y | (y << 4)) & 0x0f0f0f0fu;
    return (y | (y << 2)) & 0x33333333u;
}

// Byte `sel` of tiles c and c + 1 of a staged block.
template <int BITS, bool GROUP32>
__device__ __forceinline__ void expand_tiles_q(const AttnQBuf<BITS, GROUP32>& b, const uint2* spread, int c, unsigned sel,
                                               unsigned mh, unsigned ml, unsigned (&r1)[4], unsigned (&r2)[4]) {
    constexpr int WPT = AttnQBuf<BITS, GROUP32>::WPT;
    const uint4 bm = *reinterpret_cast<const uint4*>(&b.bm[c]);
    unsigned byte[2], win[2], flags[2];
    uint2 e[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const unsigned lo = t ? bm.z : bm.x, hi = t ? bm.w : bm.y;
        byte[t] = __byte_perm(lo, hi, sel) & 0xffu;   // the table's index: sel fills the upper bytes with another one
        e[t] = spread[byte[t]];
        const unsigned rank = __popc(hi & mh) + __popc(lo & ml);
        const int first = __popc(byte[t] & 0xf0u);
        const unsigned o = rank * BITS;
        const unsigned* w = b.words + (c + t) * WPT + (o >> 5);
        win[t] = split_halves<BITS>(__funnelshift_r(w[0], w[1], o), first);   // shift taken modulo 32
        if (GROUP32) {   // all ones for the nonzeros from number 32 of the tile on
            const int before = max(0, 32 - static_cast<int>(rank));
            flags[t] = split_halves<BITS>(__funnelshift_lc(0u, 0xffffffffu, BITS * before), first);
        }
    }
    if (BITS == 2) {   // both tiles in one register
        const unsigned two = __byte_perm(e[0].x, e[1].x, 0x5410), one = __byte_perm(e[0].x, e[1].x, 0x7632);
        const unsigned x = spread_codes<2>(__byte_perm(win[0], win[1], 0x5410), two, one);
        if (GROUP32) {
            const unsigned f = spread_codes<2>(__byte_perm(flags[0], flags[1], 0x5410), two, one);
#pragma unroll
            for (int t = 0; t < 2; ++t)
                codes_to_halves2(widen_codes(x, t) | ((widen_codes(f, t) << 1) & 0x44444444u), e[t].y, b.par[(c + t) * 2],
                                 b.par[(c + t) * 2 + 1], t ? r2 : r1);
        } else {
#pragma unroll
            for (int t = 0; t < 2; ++t) codes_to_halves2(widen_codes(x, t) | e[t].y, b.par[c + t], t ? r2 : r1);
        }
    } else {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const unsigned x = spread_codes<4>(win[t], e[t].x, e[t].y);
            if (GROUP32)
                codes_to_halves4<true>(x, byte[t], spread_codes<4>(flags[t], e[t].x, e[t].y), b.par[(c + t) * 2], b.par[(c + t) * 2 + 1],
                                       t ? r2 : r1);
            else
                codes_to_halves4<false>(x, byte[t], 0u, b.par[c + t], b.par[c + t], t ? r2 : r1);
        }
    }
}

__device__ __forceinline__ float4 ldcg_f32x4(const float* p) {
    float4 v;
    asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float ldcg_f32(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// record of (kv head h, split, query head g) inside the workspace
__device__ __forceinline__ float* record_ptr(const DecodeParams& p, int G, int h, int split, int g) {
    return p.ws + ((static_cast<int64_t>(h) * p.nrec + split) * G + g) * kPartialStride;
}

// 5 CTAs per SM (96 registers); the quantised cache with 8 heads needs two accumulator sets and would spill at 96
template <int G, int QBITS, bool GROUP32>
__global__ void __launch_bounds__(kAThreads, (QBITS != 0 && G == 8) ? 4 : 5) decode_attn_kernel(const __grid_constant__ DecodeParams p) {
    constexpr bool QUANT = QBITS != 0;
    using QB = AttnQBuf<QUANT ? QBITS : 2, GROUP32>;
    extern __shared__ __align__(128) unsigned char smem[];
    const AttnLayout lay(p.cap, G, QUANT ? sizeof(QB) : 0);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + lay.bars);
    unsigned short* ps = reinterpret_cast<unsigned short*>(smem + lay.ps);    // [8][kPsStride] probabilities, fp16
    float* red = reinterpret_cast<float*>(smem + lay.red);                     // [warp][G][kPlaneStride] scores
    float* alpha_s = reinterpret_cast<float*>(smem + lay.alpha);               // [8]
    unsigned* koff = reinterpret_cast<unsigned*>(smem + lay.koff);             // [2][128] halves, relative to the block
    unsigned* voff = reinterpret_cast<unsigned*>(smem + lay.voff);
    int* kblk = reinterpret_cast<int*>(smem + lay.kblk);                       // block starts (uint32 units) of this split
    int* vblk = reinterpret_cast<int*>(smem + lay.vblk);
    const uint2* spread = reinterpret_cast<const uint2*>(smem + lay.spread);
    __shared__ int s_last;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tb = lane >> 2, cp = lane & 3;   // fragment row (= bitmap byte) and k pair of this lane
    const int h = blockIdx.y;
    const int split = blockIdx.x;
    const bool is_window = split >= p.nsplit;
    unsigned sel, mh, ml;
    lane_byte_constants(tb, sel, mh, ml);

    // the compressed length may live in device memory (a captured launch keeps working while blocks are appended):
    // p.nblk is then its upper bound, the grid was sized for that bound, and the blocks actually there are dealt
    // out again over the same number of splits (splits past the end write an empty record)
    int nblk = p.nblk, bps = p.bps;
    if (p.L_dev) {
        nblk = max(0, min(*p.L_dev / 64, p.nblk));
        bps = p.nsplit > 0 ? (nblk + p.nsplit - 1) / p.nsplit : 0;
    }
    const int blk0 = is_window ? (split - p.nsplit) * p.wbps : split * bps;
    const int W = (is_window && p.W_dev) ? max(0, min(*p.W_dev, p.W)) : p.W;
    int nb = is_window ? min(p.wbps, (W + 63) / 64 - blk0) : min(bps, nblk - blk0);
    if (nb < 0) nb = 0;

    // ---- prologue
    const BForms<G> bf(tb, cp);
    constexpr int FORMS = BForms<G>::FORMS;
    // query: channels warp*32 + 8*g + 2*cp, +1 of head bf.head (window: head tb, the B operand of its dense layout)
    unsigned qp[4] = {0u, 0u, 0u, 0u};
    {
        const int qh = is_window ? tb : bf.head;
        if (qh < G) {
            const __half* qrow = p.q + (static_cast<int64_t>(h) * G + qh) * p.q_stride + warp * 32 + 2 * cp;
#pragma unroll
            for (int g = 0; g < 4; ++g) qp[g] = ldg_nc_u32(qrow + 8 * g);
        }
    }
    if (QUANT && !is_window) {
        const uint2* src = QBITS == 2 ? g_spread2.e : g_spread4.e;
        for (int i = tid; i < 256; i += kAThreads) const_cast<uint2*>(spread)[i] = src[i];
    }
    for (int i = tid; i < 8 * kPsStride / 2; i += kAThreads) reinterpret_cast<unsigned*>(ps)[i] = 0u;
    const int* kacc = QUANT ? nullptr : p.k.acc + h * p.k.acc_hs;
    const int* vacc = QUANT ? nullptr : p.v.acc + h * p.v.acc_hs;
    if (!QUANT && !is_window) {
        for (int i = tid; i <= nb; i += kAThreads) {
            kblk[i] = kacc[static_cast<int64_t>(blk0 + i) * kTilesPerBlock];
            vblk[i] = vacc[static_cast<int64_t>(blk0 + i) * kTilesPerBlock];
        }
    }
    if (tid == 0) {
        for (int s = 0; s < kAStages; ++s) mbar_init(&bars[s], 1);
        mbar_fence_init();
    }
    __syncthreads();

    const int64_t k_head0 = QUANT ? 0 : (p.k.nz_off ? 8ll * p.k.nz_off[h] : h * p.k.nz_hs);
    const int64_t v_head0 = QUANT ? 0 : (p.v.nz_off ? 8ll * p.v.nz_off[h] : h * p.v.nz_hs);
    const __half* knz = p.k.nz + k_head0;
    const __half* vnz = p.v.nz + v_head0;
    const size_t stg = attn_stage_bytes(p.cap);
    const unsigned capb = static_cast<unsigned>(p.cap) * 2u;

    // producer: bring block i of this split into stage i % kAStages (thread 0 only)
    auto issue = [&](int i) {
        unsigned char* st = smem + lay.stages + static_cast<size_t>(i % kAStages) * stg;
        unsigned long long* bar = &bars[i % kAStages];
        const int64_t tile0 = static_cast<int64_t>(blk0 + i) * kTilesPerBlock;
        unsigned kbytes = static_cast<unsigned>(kblk[i + 1] - kblk[i]) * 4u;
        unsigned vbytes = static_cast<unsigned>(vblk[i + 1] - vblk[i]) * 4u;
        const bool bad = block_range_bad(kblk[i], kblk[i + 1], capb, k_head0, p.k.nz_extent) ||
                         block_range_bad(vblk[i], vblk[i + 1], capb, v_head0, p.v.nz_extent);
        if (bad) {   // the bitmaps are still copied, the values are not
            if (p.dev_status) atomicOr(p.dev_status, MFAR_DEV_BADMETA);
            kbytes = vbytes = 0;
        }
        mbar_expect_tx(bar, 2048 + kbytes + vbytes);
        bulk_g2s(st + lay.s_kbm, p.k.bmp + h * p.k.bmp_hs + tile0, 1024, bar);
        if (kbytes) bulk_g2s(st + lay.s_kval, knz + 2ll * kblk[i], kbytes, bar);
        bulk_g2s(st + lay.s_vbm, p.v.bmp + h * p.v.bmp_hs + tile0, 1024, bar);
        if (vbytes) bulk_g2s(st + lay.s_vval, vnz + 2ll * vblk[i], vbytes, bar);
    };

    // per-tile offsets of the next block travel through registers (one K and one V tile per thread)
    int nxt_k = 0, nxt_v = 0;
    auto fetch_offsets = [&](int i) {
        const int64_t t = static_cast<int64_t>(blk0 + i) * kTilesPerBlock + tid;
        nxt_k = kacc[t];
        nxt_v = vacc[t];
    };
    auto store_offsets = [&](int i) {
        const unsigned lim = static_cast<unsigned>(p.cap);
        koff[(i & 1) * 128 + tid] = min(static_cast<unsigned>(2 * (nxt_k - kblk[i])), lim);
        voff[(i & 1) * 128 + tid] = min(static_cast<unsigned>(2 * (nxt_v - vblk[i])), lim);
    };

    // quantised cache: thread t owns K tile t and V tile t of a block; their metadata travels through registers
    // one block ahead, the code words go straight to the tile's slot of the stage
    struct Meta { uint2 bm; int off; unsigned sz[2]; };
    Meta mk{}, mv{};
    auto q_load_meta = [&](const QSparse& sp, int i, Meta& m) {
        const int64_t t = static_cast<int64_t>(blk0 + i) * kTilesPerBlock + tid;
        const unsigned long long bmw = sp.bmp[h * sp.bmp_hs + t];
        m.bm = make_uint2(static_cast<unsigned>(bmw), static_cast<unsigned>(bmw >> 32));
        const int64_t mi = h * sp.meta_hs + t;
        m.off = sp.tile_off[mi];
        const int ngrp = GROUP32 ? 2 : 1;
        m.sz[1] = 0u;
#pragma unroll
        for (int g = 0; g < ngrp; ++g)
            m.sz[g] = static_cast<unsigned>(__half_as_ushort(sp.scales[mi * ngrp + g])) |
                      (static_cast<unsigned>(__half_as_ushort(sp.zeros[mi * ngrp + g])) << 16);
    };
    auto q_stage = [&](const QSparse& sp, const Meta& m, QB& b) {
        constexpr int CAPW = 32 / (QUANT ? QBITS : 2);
        b.bm[tid] = m.bm;
#pragma unroll
        for (int g = 0; g < QB::NG; ++g) {
            const float scale = __half2float(__ushort_as_half(static_cast<unsigned short>(m.sz[g] & 0xffffu)));
            const float zero = __half2float(__ushort_as_half(static_cast<unsigned short>(m.sz[g] >> 16)));
            b.par[tid * QB::NG + g] = QB::BITS == 2 ? dequant_bytes(scale, zero)
                                                    : dequant_pair(scale, zero, m.sz[g]);
        }
        const int n = (__popc(m.bm.x) + __popc(m.bm.y) + CAPW - 1) / CAPW;
        if (m.off < 0 || static_cast<long long>(m.off) + n > sp.packed_words) {
            if (n > 0 && p.dev_status) atomicOr(p.dev_status, MFAR_DEV_BADMETA);
            b.bm[tid] = make_uint2(0u, 0u);     // the tile contributes nothing
            return;
        }
        const unsigned* src = sp.packed + m.off;
        for (int j = 0; j < n; ++j) cp_async4(&b.words[tid * QB::WPT + j], src + j);
    };
    auto qbuf = [&](int i, int which) -> QB& {
        return *reinterpret_cast<QB*>(smem + lay.stages + (static_cast<size_t>(i % kAStages) * 2 + which) * sizeof(QB));
    };

    if (!is_window && nb > 0) {
        if (QUANT) {
            q_load_meta(p.kq, 0, mk);
            q_load_meta(p.vq, 0, mv);
            q_stage(p.kq, mk, qbuf(0, 0));
            q_stage(p.vq, mv, qbuf(0, 1));
            cp_async_commit();
            if (nb > 1) { q_load_meta(p.kq, 1, mk); q_load_meta(p.vq, 1, mv); }
        } else {
            if (tid == 0)
                for (int i = 0; i < min(nb, kAStages - 1); ++i) issue(i);
            fetch_offsets(0);
            store_offsets(0);
        }
    }
    __syncthreads();

    // running state.  dv[hf][f][j]: columns = heads bf.ahead, + 1 of form f (G <= 4: bf.aform); rows = the positions of
    // pair 2*j (d0, d1) and 2*j + 1 (d2, d3) in byte tb, i.e. channels 64*hf + 8*tb + pair_pos
    float dv[2][FORMS][2][4];
#pragma unroll
    for (int f = 0; f < FORMS; ++f)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) dv[a][f][i][e] = 0.f;
    // softmax state of head g lives in warp g % 4: m uniform, l a per-lane partial sum
    constexpr int kHeadsPerWarp = (G + kAWarps - 1) / kAWarps;
    float m_run[kHeadsPerWarp], l_run[kHeadsPerWarp];
#pragma unroll
    for (int j = 0; j < kHeadsPerWarp; ++j) { m_run[j] = -INFINITY; l_run[j] = 0.f; }

    bool timed_out = false;
    for (int i = 0; i < nb; ++i) {
        const unsigned char* st = smem + lay.stages + static_cast<size_t>(i % kAStages) * stg;
        const uint2* kbm = reinterpret_cast<const uint2*>(st + lay.s_kbm);
        const uint2* vbm = reinterpret_cast<const uint2*>(st + lay.s_vbm);
        const unsigned short* kval = reinterpret_cast<const unsigned short*>(st + lay.s_kval);
        const unsigned short* vval = reinterpret_cast<const unsigned short*>(st + lay.s_vval);
        const unsigned* ko = koff + (i & 1) * 128;
        const unsigned* vo = voff + (i & 1) * 128;

        if (!is_window) {
            if (QUANT) {
                cp_async_wait_all();
            } else {
                if (i + 1 < nb) fetch_offsets(i + 1);
                if (!mbar_wait(&bars[i % kAStages], (i / kAStages) & 1)) timed_out = true;
            }
        }
        if (__syncthreads_or(timed_out)) { timed_out = true; break; }   // also publishes the stage hand-off below
        // every warp is done with block i-1, so its stage can take block i + kAStages - 1
        if (!is_window) {
            if (QUANT) {
                if (i + 1 < nb) {
                    q_stage(p.kq, mk, qbuf(i + 1, 0));
                    q_stage(p.vq, mv, qbuf(i + 1, 1));
                    cp_async_commit();
                    if (i + 2 < nb) { q_load_meta(p.kq, i + 2, mk); q_load_meta(p.vq, i + 2, mv); }
                }
            } else if (tid == 0 && i + kAStages - 1 < nb) {
                issue(i + kAStages - 1);
            }
        }

        // ------------------------------------------------------------ K phase: this warp's 32 channels x 64 tokens
        // score planes [warp][head][slot], slot = 8*j + tb for token 8*tb + j (the 32 lanes of a store hit 32 banks)
        float* pl = red + static_cast<size_t>(warp) * G * kPlaneStride;
        if (!is_window) {
            float dk[FORMS][2][4];
#pragma unroll
            for (int f = 0; f < FORMS; ++f)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) dk[f][j][e] = 0.f;
#pragma unroll
            for (int kg = 0; kg < 4; ++kg) {
                unsigned r1[4], r2[4];
                const int c = warp * 32 + kg * 8 + 2 * cp;
                if (QUANT) {
                    expand_tiles_q<QB::BITS, GROUP32>(qbuf(i, 0), spread, c, sel, mh, ml, r1, r2);
                } else {
                    const uint4 bm = *reinterpret_cast<const uint4*>(kbm + c);
                    const uint2 of = *reinterpret_cast<const uint2*>(ko + c);
                    expand_tile(bm.x, bm.y, kval + of.x, sel, mh, ml, r1);
                    expand_tile(bm.z, bm.w, kval + of.y, sel, mh, ml, r2);
                }
                mma_step<G>(dk, r1, r2, bf, qp[kg]);
            }
#pragma unroll
            for (int f = 0; f < FORMS; ++f)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        // token 8*tb + t
                        const int t = bf.template pos<QBITS>(2 * j + (e >> 1), f);
                        if (bf.ahead + (e & 1) < G) pl[(bf.ahead + (e & 1)) * kPlaneStride + 8 * t + tb] = dk[f][j][e];
                    }
        } else {
            // dense window: the A fragment is two adjacent channels of one token, a 32-bit load; rows = tokens 8*tb + j
            // (d0, d1) and + 4 (d2, d3), columns = heads 2*cp, 2*cp + 1
            float dk[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) dk[j][e] = 0.f;
            const __half* kw = p.kwin + h * p.win_hs;
#pragma unroll
            for (int kg = 0; kg < 2; ++kg) {
                const int c = warp * 32 + kg * 16 + 2 * cp;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int t0 = (blk0 + i) * 64 + 8 * tb + j, t1 = t0 + 4;
                    unsigned a0 = 0, a1 = 0, a2 = 0, a3 = 0;
                    if (t0 < W) { a0 = ldg_nc_u32(kw + t0 * p.win_ts + c); a2 = ldg_nc_u32(kw + t0 * p.win_ts + c + 8); }
                    if (t1 < W) { a1 = ldg_nc_u32(kw + t1 * p.win_ts + c); a3 = ldg_nc_u32(kw + t1 * p.win_ts + c + 8); }
                    mma16816(dk[j], a0, a1, a2, a3, qp[2 * kg], qp[2 * kg + 1]);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (2 * cp + (e & 1) < G) pl[(2 * cp + (e & 1)) * kPlaneStride + (j + 4 * (e >> 1)) * 8 + tb] = dk[j][e];
        }
        __syncthreads();

        // ------------------------------------------------------------ scores -> probabilities (warp g % 4 owns head g)
#pragma unroll
        for (int j = 0; j < kHeadsPerWarp; ++j) {
            const int g = warp + j * kAWarps;
            if (g < G) {
                float s0 = 0.f, s1 = 0.f;
#pragma unroll
                for (int w = 0; w < kAWarps; ++w) {
                    const float2 t = *reinterpret_cast<const float2*>(red + (static_cast<size_t>(w) * G + g) * kPlaneStride + 2 * lane);
                    s0 += t.x;
                    s1 += t.y;
                }
                // slots 2*lane, 2*lane + 1 hold tokens 16*(lane % 4) + lane / 4 and + 8
                const int tok0 = 16 * (lane & 3) + (lane >> 2), tok1 = tok0 + 8;
                s0 *= p.scale_log2;
                s1 *= p.scale_log2;
                if (is_window) {
                    if ((blk0 + i) * 64 + tok0 >= W) s0 = -INFINITY;
                    if ((blk0 + i) * 64 + tok1 >= W) s1 = -INFINITY;
                }
                const float m_new = fmaxf(m_run[j], warp_max_f32(fmaxf(s0, s1)));
                const float a = fast_exp2(m_run[j] - m_new);   // exp2(-inf) = 0 on the first block
                // the probability that enters P.V is rounded to fp16 (as the reference model does before its
                // value op); the running sum uses the same rounded value
                const __half h0 = __float2half_rn(fast_exp2(s0 - m_new)), h1 = __float2half_rn(fast_exp2(s1 - m_new));
                l_run[j] = l_run[j] * a + (__half2float(h0) + __half2float(h1));
                m_run[j] = m_new;
                ps[g * kPsStride + tok0] = __half_as_ushort(h0);
                ps[g * kPsStride + tok1] = __half_as_ushort(h1);
                if (lane == 0) alpha_s[g] = a;
            }
        }
        if (!QUANT && !is_window && i + 1 < nb) store_offsets(i + 1);
        __syncthreads();

        // ------------------------------------------------------------ V phase: this warp's 16 tokens x 128 channels
        {
            float a0 = 1.f, a1 = 1.f;
            if (bf.ahead < G) a0 = alpha_s[bf.ahead];
            if (bf.ahead + 1 < G) a1 = alpha_s[bf.ahead + 1];
            if (__any_sync(kFull, a0 != 1.f || a1 != 1.f)) {
#pragma unroll
                for (int f = 0; f < FORMS; ++f)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            dv[hf][f][j][0] *= a0; dv[hf][f][j][1] *= a1;
                            dv[hf][f][j][2] *= a0; dv[hf][f][j][3] *= a1;
                        }
            }
        }
        // a tile is 64 channels of one token; the window's values have the same shape, read as 32-bit pairs of channels
#pragma unroll
        for (int vg = 0; vg < 2; ++vg) {
            const int t = warp * 16 + vg * 8 + 2 * cp;
            const unsigned pp = *reinterpret_cast<const unsigned*>(ps + bf.head * kPsStride + t);   // tokens t, t + 1
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                unsigned r1[4], r2[4];
                if (!is_window) {
                    if (QUANT) {
                        expand_tiles_q<QB::BITS, GROUP32>(qbuf(i, 1), spread, hf * 64 + t, sel, mh, ml, r1, r2);
                    } else {
                        const uint4 bm = *reinterpret_cast<const uint4*>(vbm + hf * 64 + t);
                        const uint2 of = *reinterpret_cast<const uint2*>(vo + hf * 64 + t);
                        expand_tile(bm.x, bm.y, vval + of.x, sel, mh, ml, r1);
                        expand_tile(bm.z, bm.w, vval + of.y, sel, mh, ml, r2);
                    }
                } else {
                    const __half* vw = p.vwin + h * p.win_hs + hf * 64 + 8 * tb;
                    auto row = [&](int tok, unsigned (&r)[4]) {
                        uint4 x = make_uint4(0u, 0u, 0u, 0u);
                        if (tok < W) x = ldg_nc_u4(vw + tok * p.win_ts);
                        if (pair_pos<QBITS>(0, 1) == 1) {
                            r[0] = x.x; r[1] = x.y; r[2] = x.z; r[3] = x.w;
                        } else {
                            r[0] = __byte_perm(x.x, x.z, 0x5410); r[1] = __byte_perm(x.x, x.z, 0x7632);
                            r[2] = __byte_perm(x.y, x.w, 0x5410); r[3] = __byte_perm(x.y, x.w, 0x7632);
                        }
                    };
                    row((blk0 + i) * 64 + t, r1);
                    row((blk0 + i) * 64 + t + 1, r2);
                }
                mma_step<G>(dv[hf], r1, r2, bf, pp);
            }
        }
    }

    if (timed_out && tid == 0 && p.dev_status) atomicOr(p.dev_status, MFAR_DEV_TIMEOUT);

    // ---- epilogue: sum the four warps' partial outputs and write the record (an empty one after a timeout, so
    // that the merge below still sees every record arrive)
    __syncthreads();
#pragma unroll
    for (int f = 0; f < FORMS; ++f)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c = bf.template pos<QBITS>(2 * j + (e >> 1), f);
                    const int g = bf.ahead + (e & 1);
                    if (g < G) red[(static_cast<size_t>(warp) * G + g) * kD + hf * 64 + 8 * tb + c] = dv[hf][f][j][e];
                }
    __syncthreads();
    bool has_nan = false;
    for (int idx = tid; idx < G * kD; idx += kAThreads) {
        const int g = idx / kD, c = idx % kD;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kAWarps; ++w) s += red[(static_cast<size_t>(w) * G + g) * kD + c];
        record_ptr(p, G, h, split, g)[c] = timed_out ? 0.f : s;
        has_nan |= s != s;
    }
#pragma unroll
    for (int j = 0; j < kHeadsPerWarp; ++j) {
        const int g = warp + j * kAWarps;
        if (g < G) {
            const float l = warp_sum_f32(l_run[j]);
            if (lane == 0) {
                float* rec = record_ptr(p, G, h, split, g);
                rec[kPartM] = timed_out ? -INFINITY : m_run[j];
                rec[kPartL] = timed_out ? 0.f : l;
            }
        }
    }

    // ---- merge: the CTA that arrives last at this kv head's counter combines all records
    //      out = sum_s O_s 2^(m_s - M) / sum_s l_s 2^(m_s - M)
    __threadfence();
    // an infinity or NaN has reached its partner's row, too (a NaN probability reaches every channel): once more without pairs
    if (__syncthreads_or(has_nan && !timed_out)) {
        plain_attention<G, QBITS, GROUP32>(p, h, split, blk0, nb, W, red, ps, kPsStride, alpha_s);
        __threadfence();
        __syncthreads();
    }
    if (p.counters == nullptr) return;
    if (tid == 0) {
        const unsigned arrived = atomicAdd(p.counters + h, 1u) + 1u;
        s_last = arrived == gridDim.x;
        if (s_last) p.counters[h] = 0u;   // ready for the next launch
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // warp w merges heads w, w + 4: its lanes fetch the records' (m, l) in parallel, the weights go through shared
    // memory (the reduction buffer is free again), then every lane sums four channels over the records
    const int nrec = p.nrec;
    float* wgt = red;   // [G][nrec], nrec <= kMaxMergedRecords
    for (int g = warp; g < G; g += kAWarps) {
        const float* base = record_ptr(p, G, h, 0, g);
        const int64_t step = static_cast<int64_t>(G) * kPartialStride;
        float M = -INFINITY;
        for (int s = lane; s < nrec; s += 32) M = fmaxf(M, ldcg_f32(base + s * step + kPartM));
        M = warp_max_f32(M);
        float l = 0.f;
        for (int s = lane; s < nrec; s += 32) {
            const float ms = ldcg_f32(base + s * step + kPartM);
            const float w = (ms == -INFINITY) ? 0.f : fast_exp2(ms - M);
            l += w * ldcg_f32(base + s * step + kPartL);
            wgt[g * nrec + s] = w;
        }
        l = warp_sum_f32(l);
        __syncwarp();
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* col = base + 4 * lane;
        int s = 0;
        for (; s + 4 <= nrec; s += 4) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = ldcg_f32x4(col + (s + u) * step);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float w = wgt[g * nrec + s + u];
                o.x += w * v[u].x; o.y += w * v[u].y; o.z += w * v[u].z; o.w += w * v[u].w;
            }
        }
        for (; s < nrec; ++s) {
            const float4 v = ldcg_f32x4(col + s * step);
            const float w = wgt[g * nrec + s];
            o.x += w * v.x; o.y += w * v.y; o.z += w * v.z; o.w += w * v.w;
        }
        const float inv = l > 0.f ? 1.f / l : 0.f;
        __half* dst = p.out + (static_cast<int64_t>(h) * G + g) * p.out_stride + 4 * lane;
        dst[0] = __float2half_rn(o.x * inv);
        dst[1] = __float2half_rn(o.y * inv);
        dst[2] = __float2half_rn(o.z * inv);
        dst[3] = __float2half_rn(o.w * inv);
    }
}

template <int G, int QBITS, bool GROUP32>
static int launch_attn(const DecodeParams& p, int n_kv_heads, int grid_x, cudaStream_t s) {
    const AttnLayout lay(p.cap, G, QBITS ? sizeof(AttnQBuf<QBITS ? QBITS : 2, GROUP32>) : 0);
    static size_t configured[64] = {0};   // largest dynamic shared memory size opted into so far, per device
    int dev = 0;
    if (!cuda_ok(cudaGetDevice(&dev)) || dev < 0 || dev >= 64) return MFAR_ERR_LAUNCH;
    if (lay.total > configured[dev]) {
        if (!cuda_ok(cudaFuncSetAttribute(decode_attn_kernel<G, QBITS, GROUP32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(lay.total))))
            return MFAR_ERR_LAUNCH;
        configured[dev] = lay.total;
    }
    decode_attn_kernel<G, QBITS, GROUP32><<<dim3(grid_x, n_kv_heads), kAThreads, lay.total, s>>>(p);
    return launch_status();
}

template <int QBITS, bool GROUP32>
static int dispatch_attn(const DecodeParams& p, int G, int n_kv_heads, int grid_x, cudaStream_t s) {
    switch (G) {
        case 1: return launch_attn<1, QBITS, GROUP32>(p, n_kv_heads, grid_x, s);
        case 2: return launch_attn<2, QBITS, GROUP32>(p, n_kv_heads, grid_x, s);
        case 4: return launch_attn<4, QBITS, GROUP32>(p, n_kv_heads, grid_x, s);
        case 8: return launch_attn<8, QBITS, GROUP32>(p, n_kv_heads, grid_x, s);
        default: return MFAR_ERR_ARG;
    }
}

int launch_decode_attn(const DecodeParams& p, int G, int n_kv_heads, int grid_x, cudaStream_t s) {
    return dispatch_attn<0, false>(p, G, n_kv_heads, grid_x, s);
}

int launch_decode_attn_quant(const DecodeParams& p, int G, int bits, bool group32, int n_kv_heads, int grid_x,
                             cudaStream_t s) {
    if (bits == 2) return group32 ? dispatch_attn<2, true>(p, G, n_kv_heads, grid_x, s) : dispatch_attn<2, false>(p, G, n_kv_heads, grid_x, s);
    if (bits == 4) return group32 ? dispatch_attn<4, true>(p, G, n_kv_heads, grid_x, s) : dispatch_attn<4, false>(p, G, n_kv_heads, grid_x, s);
    return MFAR_ERR_ARG;
}

}  // namespace mfar
