// batch_kernels.cu -- the compress passes of the batched engine.
//
// Each pass is one templated stage kernel over the (item, tile) pairs of a launch; a table gives the
// item of every tile.  Passes that rank elements across tiles
// (RLE heads, GFC offsets) claim tiles from a counter and chain them with the decoupled
// look-back of scan.cuh, per item.  Every pass reads its input length from the stream table and
// writes its outputs' lengths there; tile 0 (or the tile that ends the input) writes metadata.
// Byte layouts are the per-encoding ones of encodings.cu (and of the reference).
//
// The stage kernels read their inputs through the read-only path (every input was written by an
// earlier launch).  batch_persist_c.cu compiles this file a second time, with GTSC_PERSISTENT_TU and
// coherent loads, for the persistent kernel, in which later passes read what earlier passes of the
// same launch wrote.
#include "batch_dev.cuh"

#include <algorithm>
#include <type_traits>

namespace gtsc {

namespace {

// ------------------------------------------------------------------------------- min / max
// VPT values of a view starting at base (zeros past the view): one vector run when a run is whole
// 16-byte chunks, else element loads
template <int ES, int VPT>
__device__ __forceinline__ void load_view_any(const BItem &it, const ViewCtx &vc, const uint8_t *src, uint64_t base,
                                              uint64_t (&v)[VPT])
{
    if constexpr ((VPT * ES) % 16 == 0) {
        load_view<ES, VPT>(it, vc, src, base, v);
    } else {
#pragma unroll
        for (int j = 0; j < VPT; j++) v[j] = base + j < vc.n ? view_elem<ES>(it, vc, src, base + j) : 0;
    }
}

// A tile of it.p[0] values (the tuned min/max tile; a multiple of kBThreads * VPT): rounds of VPT
// consecutive values a thread, two rounds loaded before either is reduced.
template <int ES, int VPT>
__device__ void p_minmax_v(const BItem &it, uint32_t tile, StreamDesc *S)
{
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    const uint64_t T = it.p[0];
    const uint64_t t0 = (uint64_t)tile * T;
    if (t0 >= n) return;
    const uint64_t end = n < t0 + T ? n : t0 + T;
    const Order o = (Order)it.order;
    constexpr uint64_t R = (uint64_t)kBThreads * VPT;  // values of one round of the block
    uint64_t kmin = ~0ull, kmax = 0;
    if constexpr (ES <= 4) {
        // 32-bit keys of the same order (sign bit flipped for integers, order_key's map for floats),
        // turned into the accumulator's 64-bit keys once per thread
        const bool f32 = o == ORD_F32;
        constexpr uint32_t SH = 32 - 8 * ES;
        uint32_t k32min = ~0u, k32max = 0;
        bool seen = false;
        auto key32 = [&](uint32_t u) {
            if (f32) return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
            return (uint32_t)((int32_t)(u << SH) >> SH) ^ 0x80000000u;
        };
        for (uint64_t b0 = t0 + (uint64_t)threadIdx.x * VPT; b0 < end; b0 += 2 * R) {
            const uint64_t b1 = b0 + R;
            uint32_t u[2][VPT];
            {
                uint64_t v[VPT];
                load_view_any<ES, VPT>(it, vc, in.ptr, b0, v);
#pragma unroll
                for (int j = 0; j < VPT; j++) u[0][j] = (uint32_t)v[j];
                if (b1 < end) load_view_any<ES, VPT>(it, vc, in.ptr, b1, v);
#pragma unroll
                for (int j = 0; j < VPT; j++) u[1][j] = (uint32_t)v[j];
            }
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint64_t base = r ? b1 : b0;
                const uint32_t cnt = base >= end ? 0u : end - base < (uint64_t)VPT ? (uint32_t)(end - base) : VPT;
#pragma unroll
                for (int j = 0; j < VPT; j++) {
                    const bool ok = (uint32_t)j < cnt && !(f32 && (u[r][j] & 0x7fffffffu) > 0x7f800000u);
                    const uint32_t k = key32(u[r][j]);
                    k32min = ok && k < k32min ? k : k32min;
                    k32max = ok && k > k32max ? k : k32max;
                    seen |= ok;
                }
            }
        }
        if (seen) {
            const uint32_t umin = f32 ? ((k32min & 0x80000000u) ? (k32min ^ 0x80000000u) : ~k32min)
                                      : (k32min ^ 0x80000000u);
            const uint32_t umax = f32 ? ((k32max & 0x80000000u) ? (k32max ^ 0x80000000u) : ~k32max)
                                      : (k32max ^ 0x80000000u);
            kmin = order_key(umin, 4, o);  // umin / umax are sign-extended to 32 bits
            kmax = order_key(umax, 4, o);
        }
    } else {
        for (uint64_t base = t0 + (uint64_t)threadIdx.x * VPT; base < end; base += R) {
            uint64_t v[VPT];
            load_view_any<ES, VPT>(it, vc, in.ptr, base, v);
#pragma unroll
            for (int j = 0; j < VPT; j++) {
                if (base + j >= end || is_nan_bits(v[j], o)) continue;
                const uint64_t k = order_key(v[j], ES, o);
                kmin = k < kmin ? k : kmin;
                kmax = k > kmax ? k : kmax;
            }
        }
    }
    block_minmax(kmin, kmax);
    if (threadIdx.x == 0) {
        MinMaxAcc *acc = (MinMaxAcc *)it.scratch;
        if (kmin != ~0ull) atomicMax(&acc->nkmin, (unsigned long long)~kmin);
        if (kmax != 0) atomicMax(&acc->kmax, (unsigned long long)kmax);
    }
}

// the min/max pass with the tuned values per thread (it.p[1]: 1, 2, 4, 8 or 16)
template <int ES>
__device__ void p_minmax(const BItem &it, uint32_t tile, StreamDesc *S)
{
    switch (it.p[1]) {
    case 1: p_minmax_v<ES, 1>(it, tile, S); break;
    case 2: p_minmax_v<ES, 2>(it, tile, S); break;
    case 4: p_minmax_v<ES, 4>(it, tile, S); break;
    case 8: p_minmax_v<ES, 8>(it, tile, S); break;
    default: p_minmax_v<ES, 16>(it, tile, S); break;
    }
}

// ------------------------------------------------------------------------------- delta
template <int ES>
__device__ void p_delta_enc(const BItem &it, uint32_t tile, StreamDesc *S)
{
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    if (tile == 0 && threadIdx.x == 0) {
        StreamDesc &m = S[it.out[0]];
        if (n) {
            st_elem<ES>(m.ptr, 0, view_elem<ES>(it, vc, in.ptr, 0));
            m.len = ES;
            S[it.out[1]].len = (n - 1) * ES;
        } else {
            m.len = 0;
            S[it.out[1]].len = 0;
        }
    }
    const uint64_t m = n ? n - 1 : 0;
    const uint64_t base = (uint64_t)tile * kBTile + (uint64_t)threadIdx.x * kBVPT;
    if (base >= m) return;
    uint64_t v[kBVPT];
    load_view<ES, kBVPT>(it, vc, in.ptr, base, v);
    const uint64_t next = base + kBVPT < n ? view_elem<ES>(it, vc, in.ptr, base + kBVPT) : 0;
    uint64_t d[kBVPT];
#pragma unroll
    for (int j = 0; j + 1 < (int)kBVPT; j++) d[j] = wrap_es(v[j + 1] - v[j], ES);
    d[kBVPT - 1] = wrap_es(next - v[kBVPT - 1], ES);
    store_run<ES, kBVPT>(S[it.out[1]].ptr, base, m, d);
}

// ------------------------------------------------------------------------------- scale
template <int ES>
__device__ void p_scale_sub(const BItem &it, uint32_t tile, StreamDesc *S)
{
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    uint64_t mnb = 0, mxb = 0;
    acc_minmax((const MinMaxAcc *)it.scratch, ES, ORD_INT, mnb, mxb);
    const uint64_t mn = scale_min(mnb, mxb, ES);
    if (tile == 0 && threadIdx.x == 0) {
        if (n) {
            st_elem<ES>(S[it.out[0]].ptr, 0, mn);
            S[it.out[0]].len = ES;
        } else {
            S[it.out[0]].len = 0;
        }
        S[it.out[1]].len = n * ES;
    }
    const uint64_t base = (uint64_t)tile * kBTile + (uint64_t)threadIdx.x * kBVPT;
    if (base >= n) return;
    uint64_t v[kBVPT];
    load_view<ES, kBVPT>(it, vc, in.ptr, base, v);
#pragma unroll
    for (int j = 0; j < (int)kBVPT; j++) v[j] = wrap_es(v[j] - mn, ES);
    store_run<ES, kBVPT>(S[it.out[1]].ptr, base, n, v);
}

// ------------------------------------------------------------------------------- AFL pack
__device__ __forceinline__ void sm_or(uint32_t a, uint32_t v) { asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }

__device__ __forceinline__ uint32_t afl_slot(uint32_t i) { return i + (i >> 4); }
// Packs the rows of a unit (16 bytes of values a lane and row) into the warp's words of shared memory,
// which are zero: a lane's values become up to 5 words from bit i * b on, or-ed in (a word is shared by
// the lanes whose bits it holds).  SMALL: they fit one word.
template <int ES, bool SMALL>
__device__ __forceinline__ void pack_rows(const ViewCtx &vc, const uint8_t *src, uint64_t u0, uint32_t cnt, uint32_t b,
                                          uint32_t words)
{
    using V = word_t<ES>;
    constexpr uint32_t N = 16 / ES, ROW = 32 * N, R = ES == 4 ? 4 : 1;
    const V mask = b >= 8 * sizeof(V) ? ~(V)0 : ((V)1 << b) - 1;
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll 1
    for (uint32_t r0 = 0; r0 * ROW < cnt; r0 += R) {
        V v[R][N];
#pragma unroll
        for (uint32_t r = 0; r < R; r++) {
            const uint32_t i = (r0 + r) * ROW + lane * N;
            if (i < cnt) load_vec<ES>(vc, src, u0 + i, v[r]);  // zeros past the view
        }
#pragma unroll
        for (uint32_t r = 0; r < R; r++) {
            const uint32_t i = (r0 + r) * ROW + lane * N, bit = i * b;
            if (i >= cnt) continue;
            uint32_t at = words + 4 * (bit >> 5);
            if constexpr (SMALL) {
                uint32_t x = 0;
#pragma unroll
                for (int k = (int)N - 1; k >= 0; k--) x = x << b | (uint32_t)(v[r][k] & mask);
                const uint32_t s = bit & 31;
                sm_or(at, x << s);
                const uint32_t hi = __funnelshift_l(x, 0u, s);
                if (hi) sm_or(at + 4, hi);
            } else {
                uint64_t acc = 0;
                uint32_t fill = bit & 31;
                auto put = [&](uint32_t x, uint32_t w) {  // w <= 32 bits
                    acc |= (uint64_t)x << fill;
                    fill += w;
                    if (fill >= 32) {
                        sm_or(at, (uint32_t)acc);
                        at += 4;
                        acc >>= 32;
                        fill -= 32;
                    }
                };
#pragma unroll
                for (int k = 0; k < (int)N; k++) {
                    const V x = v[r][k] & mask;
                    put(x, b);
                }
                if (fill) sm_or(at, (uint32_t)acc);
            }
        }
    }
}

// AFL packing (n * s read, n * b / 8 written).  Values of up to 4 bytes read plainly: a warp packs a unit
// whose packed words no other unit shares, in its own part of shared memory, and stores them whole; no
// barrier lies between units.  Views (a delta's neighbours, a scale's constant) and 8-byte values: a
// thread packs 16 consecutive values between two barriers.  That form's 16-byte loads lie 64 bytes
// apart, which binds it by L1 where nothing else does, but it shares the neighbours of a view in
// registers.  2^26 int32: 31 bits, plain 0.219 -> 0.113 ms (4.7 TB/s); a scaled delta in 5 bits 0.139 ->
// 0.107, by the setup done once for a block's tiles of an item (as units 0.164); the 256 mixed columns
// 0.69 -> 0.56.  64 registers, four blocks an SM: with 48 and five the units took 0.167.
template <int ES>
__device__ void p_afl_pack(const BItem &it, uint32_t tile, uint32_t step, uint32_t end, StreamDesc *S, unsigned char *sm)
{
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    uint64_t mnb = 0, mxb = 0;
    int b;
    if (it.vflags & 1) {
        // the view ends with a scale by c = scale_min(min, max) of the scale's input: c = 0 leaves
        // [min, max]; c = min maps onto [0, max - min], unless max - min passes the type's largest
        // value (scale_min keeps c = min for the most negative min): then values wrap negative
        // and the width is the full word, as BITLEN gives for any negative minimum
        // the last scale of the view (static indices: no local-memory copy of the context)
        uint64_t c = 0;
        const uint8_t *scr = nullptr;
#pragma unroll
        for (int k = 0; k < kMaxViewOps; k++)
            if (it.vop[k] == V_SCALE) {
                c = vc.c[k];
                scr = it.vscr[k];
            }
        acc_minmax((const MinMaxAcc *)scr, ES, ORD_INT, mnb, mxb);
        if (c == 0) {
            b = bitlen_signed(sext(mnb, ES), sext(mxb, ES), ES);
        } else {
            const uint64_t span = (uint64_t)sext(mxb, ES) - (uint64_t)sext(mnb, ES);
            const uint64_t tmax = (ES == 8 ? ~0ull : ((1ull << (8 * ES)) - 1)) >> 1;
            b = span > tmax ? 8 * ES : bitlen_signed(0, (int64_t)span, ES);
        }
    } else {
        acc_minmax((const MinMaxAcc *)it.scratch, ES, ORD_INT, mnb, mxb);
        b = bitlen_signed(sext(mnb, ES), sext(mxb, ES), ES);
    }
    const uint64_t W = 8ull * ES;
    const uint64_t out_bytes = n ? (b * n + W - 1) / W * ES : 0;
    if (tile == 0 && threadIdx.x == 0) {
        StreamDesc &m = S[it.out[0]];
        if (n) {
            m.ptr[0] = (uint8_t)b;
            m.ptr[1] = (uint8_t)(int8_t)(out_bytes * 8 - n * (uint64_t)b);
            m.ptr[2] = 0;
            m.ptr[3] = 0;
            m.len = 4;
        } else {
            m.len = 0;
        }
        S[it.out[1]].len = out_bytes;
    }
    if constexpr (ES <= 4) {
    if (vc.plain) {
    constexpr uint32_t UNIT = kBPackUnit;
    const uint32_t lane = threadIdx.x & 31, pieces = UNIT / 128 * (uint32_t)b;  // of 16 bytes, of a unit's output
    uint8_t *const out0 = S[it.out[1]].ptr;
    uint4 *wq = (uint4 *)(sm + (threadIdx.x >> 5) * (UNIT * ES));
    const uint32_t words = (uint32_t)__cvta_generic_to_shared(wq);
#pragma unroll 1
    for (; tile < end; tile += step) {
        const uint64_t u0 = (uint64_t)tile * kBTile + (threadIdx.x >> 5) * UNIT;
        if (u0 >= n) break;
        const uint32_t cnt = (uint32_t)(n - u0 < UNIT ? n - u0 : UNIT);
        __syncwarp();  // the warp's words of the tile before are stored
        for (uint32_t i = lane; i < pieces; i += 32) wq[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        if (16 / ES * b <= 32) pack_rows<ES, true>(vc, in.ptr, u0, cnt, (uint32_t)b, words);
        else pack_rows<ES, false>(vc, in.ptr, u0, cnt, (uint32_t)b, words);
        __syncwarp();
        const uint64_t o0 = u0 / 8 * (uint64_t)b;  // the unit's first byte of the output
        uint8_t *out = out0 + o0;
        const uint64_t left = out_bytes - o0;
        for (uint32_t i = lane; i < pieces; i += 32) {
            if (16ull * i + 16 <= left) {
                ((uint4 *)out)[i] = wq[i];
            } else {
                for (uint32_t k = 16 * i; k < 16 * i + 16 && k < left; k++) out[k] = ((const uint8_t *)wq)[k];
            }
        }
    }
    return;
    }
    }
    uint8_t *const out = S[it.out[1]].ptr;
    unsigned long long *sv = (unsigned long long *)sm;
#pragma unroll 1
    for (; tile < end; tile += step) {
    const uint64_t t0 = (uint64_t)tile * kBTile;
    if (t0 >= n) return;
    __syncthreads();  // the tile before is stored
    if constexpr (ES <= 4) {
        // b <= 32.  Thread t packs its 16 values (tile bits [16 b t, 16 b (t + 1))) into a register
        // and stores whole words to the tile's words in shared memory; the word it shares with the
        // thread before it (a start inside a word) and the one it shares with the thread after it
        // (an end inside a word) are or-ed in.  Word w sits at w + w / 32, so that threads storing
        // b / 2 words apart spread over the banks.  A tile's output starts on a word: 4096 b / 32.
        uint32_t *ow = (uint32_t *)sv;
        auto slot = [](uint32_t w) { return w + (w >> 5); };
        const uint32_t vmask32 = b >= 32 ? ~0u : ((1u << b) - 1);
        uint64_t v[kBVPT];
        const uint64_t base = t0 + (uint64_t)threadIdx.x * kBVPT;
        load_view<ES, kBVPT>(it, vc, in.ptr, base, v);
        const uint32_t bit0 = threadIdx.x * kBVPT * (uint32_t)b;
        if (bit0 & 31) ow[slot(bit0 >> 5)] = 0;
        __syncthreads();
        uint32_t wi = bit0 >> 5, fill = bit0 & 31;
        bool shared_first = fill != 0;
        uint64_t acc = 0;
#pragma unroll
        for (int j = 0; j < (int)kBVPT; j++) {
            const uint32_t u = base + j < n ? ((uint32_t)v[j] & vmask32) : 0u;
            acc |= (uint64_t)u << fill;
            fill += (uint32_t)b;
            if (fill >= 32) {
                if (shared_first) atomicOr(&ow[slot(wi)], (uint32_t)acc);
                else ow[slot(wi)] = (uint32_t)acc;
                shared_first = false;
                ++wi;
                acc >>= 32;
                fill -= 32;
            }
        }
        if (fill) atomicOr(&ow[slot(wi)], (uint32_t)acc);
        __syncthreads();
        const uint64_t total_words = (out_bytes + 3) / 4;
        const uint64_t w0 = t0 * (uint64_t)b / 32;
        uint64_t w_end = w0 + 128u * (uint32_t)b;
        if (w_end > total_words) w_end = total_words;
        for (uint64_t w = w0 + threadIdx.x; w < w_end; w += kBThreads) {
            const uint32_t word = ow[slot((uint32_t)(w - w0))];
            if (4 * w + 4 <= out_bytes) {
                reinterpret_cast<uint32_t *>(out)[w] = word;
            } else {
                for (int k = 0; k < 4; k++)
                    if (4 * w + k < out_bytes) out[4 * w + k] = (uint8_t)(word >> (8 * k));
            }
        }
        continue;
    }
    const uint64_t vmask = b >= 64 ? ~0ull : ((1ull << b) - 1);
    const uint64_t cnt = n - t0 < kBTile ? n - t0 : kBTile;
    // the tile's values in shared memory, skewed by one slot per 16 values (afl_slot) so that a
    // thread's run of 16 and the word gather below both spread over the banks
    if (vc.plain && cnt == kBTile && ((uintptr_t)in.ptr & 15) == 0) {
        const uint8_t *src = in.ptr + t0 * ES;
        constexpr int PER = 16 / ES;
        for (int c = threadIdx.x; c < (int)kBTile / PER; c += kBThreads) {
            const uint4 v = ld_chunk(src + 16 * c);
#pragma unroll
            for (int j = 0; j < PER; j++) sv[afl_slot(c * PER + j)] = chunk_elem<ES>(v, j) & vmask;
        }
    } else {
        uint64_t v[kBVPT];
        const uint64_t base = t0 + (uint64_t)threadIdx.x * kBVPT;
        load_view<ES, kBVPT>(it, vc, in.ptr, base, v);
#pragma unroll
        for (int j = 0; j < (int)kBVPT; j++) {
            const uint32_t i = threadIdx.x * kBVPT + j;
            sv[afl_slot(i)] = base + j < n ? (v[j] & vmask) : 0ull;
        }
    }
    if (threadIdx.x < 4) sv[afl_slot(kBTile + threadIdx.x)] = 0;
    __syncthreads();
    const uint64_t total_words = (out_bytes + 3) / 4;
    const uint64_t w0 = t0 * (uint64_t)b / 32;
    uint64_t w_end = (t0 + kBTile) * (uint64_t)b / 32;
    if (w_end > total_words) w_end = total_words;
    for (uint64_t w = w0 + threadIdx.x; w < w_end; w += kBThreads) {
        const uint32_t p = (uint32_t)(w - w0) * 32u;
        uint32_t a = p / (uint32_t)b;
        const uint32_t s = p - a * (uint32_t)b;
        uint64_t acc = sv[afl_slot(a)] >> s;
        int filled = b - (int)s;
        ++a;
        while (filled < 32) {
            acc |= sv[afl_slot(a)] << filled;
            filled += b;
            ++a;
        }
        const uint32_t word = (uint32_t)acc;
        if (4 * w + 4 <= out_bytes) {
            reinterpret_cast<uint32_t *>(out)[w] = word;
        } else {
            for (int k = 0; k < 4; k++)
                if (4 * w + k < out_bytes) out[4 * w + k] = (uint8_t)(word >> (8 * k));
        }
    }
    }
}

// calls f with an element size as a constant (an integral_constant)
template <class F>
__device__ __forceinline__ void with_size(int es, F f)
{
    switch (es) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    default: f(std::integral_constant<int, 8>()); break;
    }
}

// ------------------------------------------------------------------------------- histogram
__device__ __forceinline__ uint64_t bhash(uint64_t k)
{
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}

struct HTab {
    BHistHdr *hdr;
    unsigned long long *keys;
    unsigned int *counts;
    unsigned int *used;
    unsigned long long *nan;   // 4 per histogram tile
    unsigned long long *part;  // top-k partials: 4 x (key, bits, count) per histogram tile
    uint64_t cap;
};
__device__ __forceinline__ HTab htab(const BItem &it)
{
    // p[0] = table capacity, p[1] = histogram tiles, p[2] = table offset in the node scratch
    HTab t;
    t.cap = it.p[0];
    uint8_t *b = it.scratch + it.p[2];
    t.hdr = (BHistHdr *)b;
    t.keys = (unsigned long long *)(b + 16);
    t.counts = (unsigned int *)(b + 16 + 8 * t.cap);
    t.used = (unsigned int *)(b + 16 + 12 * t.cap);
    t.nan = (unsigned long long *)(b + 16 + 16 * t.cap);
    t.part = t.nan + 4 * it.p[1];
    return t;
}

__device__ void g_insert(const HTab &t, unsigned long long key, unsigned int c, uint32_t *status)
{
    constexpr unsigned long long EMPTY = ~0ull;
    if (key == EMPTY) {
        atomicAdd(&t.hdr->special, c);
        return;
    }
    const uint64_t mask = t.cap - 1;
    uint64_t h = bhash(key) & mask;
    for (uint64_t probe = 0; probe < t.cap && probe < 8192; probe++) {
        const unsigned long long prev = atomicCAS(t.keys + h, EMPTY, key);
        if (prev == EMPTY) {
            // the lanes that took a slot together reserve their places in the list with one addition
            const unsigned took = __activemask(), lane = threadIdx.x & 31;
            const int leader = __ffs(took) - 1;
            unsigned int u = 0;
            if ((int)lane == leader) u = atomicAdd(&t.hdr->used, (unsigned)__popc(took));
            u = __shfl_sync(took, u, leader) + __popc(took & ((1u << lane) - 1));
            t.used[u] = (unsigned int)h;
            atomicAdd(t.counts + h, c);
            return;
        }
        if (prev == key) {
            atomicAdd(t.counts + h, c);
            return;
        }
        h = (h + 1) & mask;
    }
    atomicExch(&t.hdr->overflow, 1u);
    set_status(status, GTSC_ERR_CAPACITY);
}

// Adds P (key, count) pairs of a thread to the node's global table (a zero count adds nothing).
// Each key's first slot is read with a plain load, all P loads in flight together: after a
// column's first tiles most keys are already there, and their counts are then added with
// reductions that nothing waits for.  A key not at its first slot takes the full insert.  (Keys
// never move once set, so a slot read holding the key is the key's slot.)
template <int P>
__device__ __forceinline__ void g_insert_many(const HTab &t, const unsigned long long (&key)[P],
                                              const uint32_t (&cnt)[P], uint32_t *status)
{
    constexpr unsigned long long EMPTY = ~0ull;
    const uint64_t mask = t.cap - 1;
    uint64_t h[P];
    unsigned long long cur[P];
#pragma unroll
    for (int j = 0; j < P; j++) {
        h[j] = bhash(key[j]) & mask;
        cur[j] = cnt[j] && key[j] != EMPTY ? *(volatile const unsigned long long *)(t.keys + h[j]) : EMPTY;
    }
#pragma unroll
    for (int j = 0; j < P; j++) {
        if (!cnt[j]) continue;
        if (key[j] != EMPTY && cur[j] == key[j]) atomicAdd(t.counts + h[j], cnt[j]);
        else g_insert(t, key[j], cnt[j], status);
    }
}

// The shared table of a histogram block: buckets of two (key, count) slots.  Values of up to 4 bytes
// have 32-bit keys (8 bytes a slot), 8-byte values 64-bit ones (12).  An empty slot holds a mark, any
// value that does not hash to its bucket, so that a lookup needs no test for empty slots: MARK, and
// MARK2 in MARK's own bucket.  The two marks themselves are never put in the table.  Behind it lie
// the warps' queues of values to insert.
constexpr uint32_t kHistQueue = 64;  // values of a warp's queue

// Accesses of the tables by shared-memory address: through generic pointers each addition was compiled
// with a test of the address space around it (full histogram of 2^26 Zipf ids 0.309 -> 0.287 ms).
__device__ __forceinline__ void sm_add(uint32_t a, uint32_t c) { asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(c) : "memory"); }
__device__ __forceinline__ void sm_pair(uint32_t a, uint32_t &x, uint32_t &y)
{
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ void sm_pair(uint32_t a, uint64_t &x, uint64_t &y)
{
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ uint32_t sm_cas(uint32_t a, uint32_t old, uint32_t v)
{
    asm volatile("atom.shared.cas.b32 %0, [%1], %2, %3;" : "=r"(v) : "r"(a), "r"(old), "r"(v) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t sm_cas(uint32_t a, uint64_t old, uint64_t v)
{
    asm volatile("atom.shared.cas.b64 %0, [%1], %2, %3;" : "=l"(v) : "r"(a), "l"(old), "l"(v) : "memory");
    return v;
}
__device__ __forceinline__ void sm_put(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sm_put(uint32_t a, uint64_t v) { asm volatile("st.shared.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ void sm_get(uint32_t a, uint32_t &v) { asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory"); }
__device__ __forceinline__ void sm_get(uint32_t a, uint64_t &v) { asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory"); }

template <int ES>
struct HistTable {
    using K = word_t<ES>;
    static constexpr K MARK = (K)0x8f1b5c37a4d96e21ull, MARK2 = (K)0xe3779a4d51c2b867ull;
    static constexpr uint32_t KB = sizeof(K);
    uint32_t keys, counts, queue;  // shared-memory addresses; the queue of this warp
    uint32_t buckets;
    __device__ __forceinline__ HistTable(const unsigned char *smem, uint32_t bytes)
    {
        const uint32_t table = bytes - (blockDim.x / 32) * kHistQueue * 8;
        buckets = table / (2 * (KB + 4)) & ~1u;  // whole 16-byte pieces of either array
        keys = (uint32_t)__cvta_generic_to_shared(smem);
        counts = keys + 2 * buckets * KB;
        queue = keys + table + (threadIdx.x / 32) * kHistQueue * 8;
    }
    __device__ __forceinline__ uint32_t bucket(K v) const
    {
        uint32_t m = (uint32_t)v;
        if (ES == 8) m ^= (uint32_t)((uint64_t)v >> 32);
        return __umulhi(m * 0x9E3779B1u, buckets);  // multiplicative hash scaled to the buckets
    }
    __device__ __forceinline__ K mark(uint32_t b) const { return b == bucket(MARK) ? MARK2 : MARK; }
    // v's count if its bucket holds it, else 0
    __device__ __forceinline__ uint32_t find(K v) const
    {
        const uint32_t b = bucket(v);
        K k0, k1;
        sm_pair(keys + 2 * KB * b, k0, k1);
        const uint32_t c = counts + 8 * b;
        return k0 == v ? c : k1 == v ? c + 4 : 0u;
    }
};

struct HistShared {
    unsigned long long nan[4];  // the smallest NaN sort keys so far
    uint32_t used;              // slots taken
};
static __shared__ HistShared s_hist;

// c occurrences of a value that its bucket does not hold yet.  A full table takes no more keys: what
// its bucket does not hold goes to the node's global table.
template <int ES>
__device__ __noinline__ void hist_insert(unsigned char *smem, uint32_t bytes, const BItem &it, word_t<ES> v, uint32_t c,
                                         uint32_t *status)
{
    using T = HistTable<ES>;
    const T h(smem, bytes);
    if (v != T::MARK && v != T::MARK2) {
        uint32_t b = h.bucket(v);
        const int probes = *(volatile uint32_t *)&s_hist.used < h.buckets + h.buckets / 2 ? 4 : 1;
        for (int p = 0; p < probes; p++) {
            const typename T::K mark = h.mark(b);
            typename T::K k[2];
            sm_pair(h.keys + 2 * T::KB * b, k[0], k[1]);
#pragma unroll
            for (int w = 0; w < 2; w++) {
                if (k[w] == mark) {
                    k[w] = sm_cas(h.keys + T::KB * (2 * b + w), mark, v);
                    if (k[w] == mark) {
                        atomicAdd(&s_hist.used, 1u);
                        k[w] = v;
                    }
                }
                if (k[w] == v) {
                    sm_add(h.counts + 4 * (2 * b + w), c);
                    return;
                }
            }
            b = b + 1 == h.buckets ? 0 : b + 1;
        }
    }
    g_insert(htab(it), (unsigned long long)v, c, status);
}

// keeps the four smallest NaN sort keys: what a slot gives up moves on to the next
__device__ __noinline__ void hist_nan(unsigned long long k)
{
    if (k >= *(volatile unsigned long long *)&s_hist.nan[3]) return;
    for (int j = 0; j < 4; j++) {
        const unsigned long long old = atomicMin(&s_hist.nan[j], k);
        k = old > k ? old : k;
    }
}

// an empty table (all threads; barriers on both sides are the caller's)
template <int ES>
__device__ __forceinline__ void hist_clear(unsigned char *smem, uint32_t bytes)
{
    using T = HistTable<ES>;
    const T h(smem, bytes);
    constexpr uint32_t PER = 16 / T::KB;  // keys of a 16-byte piece
    const uint32_t special = h.bucket(T::MARK), keys = 2 * h.buckets / PER, all = keys + 2 * h.buckets / 4;
    uint4 *q = (uint4 *)smem;
    constexpr uint64_t M = ES == 8 ? (uint64_t)T::MARK : (uint64_t)T::MARK << 32 | (uint64_t)T::MARK;
    for (uint32_t i = threadIdx.x; i < all; i += blockDim.x)
        q[i] = i < keys ? make_uint4((uint32_t)M, (uint32_t)(M >> 32), (uint32_t)M, (uint32_t)(M >> 32)) : make_uint4(0, 0, 0, 0);
    // MARK's own bucket: by the thread that cleared it
    if (threadIdx.x == special * 2 / PER % blockDim.x) {
        sm_put(h.keys + 2 * T::KB * special, T::MARK2);
        sm_put(h.keys + 2 * T::KB * special + T::KB, T::MARK2);
    }
    if (threadIdx.x < 4) s_hist.nan[threadIdx.x] = ~0ull;
    if (threadIdx.x == 4) s_hist.used = 0;
}

// the table's counts to the node's global table, the NaN keys to `tile`'s list
template <int ES>
__device__ __forceinline__ void hist_flush(unsigned char *smem, uint32_t bytes, const BItem &it, uint32_t tile,
                                           uint32_t *status)
{
    using T = HistTable<ES>;
    const T h(smem, bytes);
    const HTab t = htab(it);
    const uint32_t slots = 2 * h.buckets;
    for (uint32_t i0 = threadIdx.x; i0 < slots; i0 += 4 * blockDim.x) {
        unsigned long long k[4];
        uint32_t c[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t i = i0 + j * blockDim.x;
            typename T::K x = 0;
            c[j] = 0;  // as an empty slot's
            if (i < slots) {
                sm_get(h.keys + T::KB * i, x);
                sm_get(h.counts + 4 * i, c[j]);
            }
            k[j] = x;
        }
        g_insert_many<4>(t, k, c, status);
    }
    if (threadIdx.x < 4) t.nan[4ull * tile + threadIdx.x] = s_hist.nan[threadIdx.x];
}

// Counts the values of a tile in the block's table.  Issue-bound before (86 warp instructions per 32
// values: one value at a time, each a probe loop in which the warp waits for its slowest lane); now a
// thread takes 16 bytes of values a round, two rounds in flight, looks all of them up at once (one shared
// load a value gives its bucket's two keys) and adds to the counts of those found.  The others go to
// the warp's queue and are inserted 32 at a time, so that a row with one new value does not run the
// insert for one lane.  A thread whose values are all equal adds them at once, a warp of one value
// adds once.
template <int ES>
__device__ __forceinline__ void hist_tile(unsigned char *smem, uint32_t bytes, const BItem &it, uint32_t tile,
                                          StreamDesc *S, uint32_t *status)
{
    using T = HistTable<ES>;
    using K = typename T::K;
    constexpr int N = 16 / ES;
    const T h(smem, bytes);
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n, HT = it.p[3], t0 = (uint64_t)tile * HT;
    const Order o = (Order)it.order;
    if (t0 >= n) return;
    const uint64_t end = n < t0 + HT ? n : t0 + HT;
    auto insert = [&](K v, uint32_t c) {
        if (is_nan_bits(v, o)) for (uint32_t q = 0; q < c && q < 4; q++) hist_nan(order_key(v, ES, o));
        else hist_insert<ES>(smem, bytes, it, v, c, status);
    };
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t step = (uint64_t)blockDim.x * N;
    uint32_t queued = 0;  // values in the warp's queue (fewer than 32 between rows)
    for (uint64_t w0 = t0 + (uint64_t)(threadIdx.x - lane) * N; w0 < end; w0 += 2 * step) {
        K u[2][N];
        const uint64_t b0 = w0 + lane * N, b1 = b0 + step;
        if (b0 < end) load_vec<ES>(vc, in.ptr, b0, u[0]);
        if (b1 < end) load_vec<ES>(vc, in.ptr, b1, u[1]);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint64_t base = r ? b1 : b0;
            const int cnt = base >= end ? 0 : end - base < (uint64_t)N ? (int)(end - base) : N;  // this lane's values
            K(&v)[N] = u[r];
            bool same = cnt == N;
#pragma unroll
            for (int q = 1; q < N; q++) same = same && v[q] == v[0];
            if (__all_sync(0xffffffffu, same)) {
                int one;
                __match_all_sync(0xffffffffu, v[0], &one);
                if (!one) {
                    const uint32_t c = h.find(v[0]);
                    if (c) sm_add(c, N);
                    else insert(v[0], N);
                } else if (lane == 0) {
                    insert(v[0], 32 * N);
                }
                __syncwarp();
                continue;
            }
            uint32_t count[N];
#pragma unroll
            for (int q = 0; q < N; q++) count[q] = h.find(v[q]);
#pragma unroll
            for (int q = 0; q < N; q++) {
                const bool new_one = q < cnt && !count[q];
                if (q < cnt && count[q]) sm_add(count[q], 1u);
                const uint32_t m = __ballot_sync(0xffffffffu, new_one);
                if (m) {
                    if (new_one) sm_put(h.queue + T::KB * (queued + __popc(m & ((1u << lane) - 1))), v[q]);
                    queued += __popc(m);
                    __syncwarp();
                    if (queued >= 32) {
                        K x, rest;
                        sm_get(h.queue + T::KB * lane, x);
                        sm_get(h.queue + T::KB * (32 + lane), rest);
                        insert(x, 1u);
                        __syncwarp();
                        queued -= 32;
                        if (lane < queued) sm_put(h.queue + T::KB * lane, rest);
                        __syncwarp();
                    }
                }
            }
        }
    }
    if (lane < queued) {
        K x;
        sm_get(h.queue + T::KB * lane, x);
        insert(x, 1u);
    }
    __syncwarp();
}

// one tile on its own (the persistent schedule)
template <int ES>
__device__ __forceinline__ void p_hist(const BItem &it, uint32_t tile, StreamDesc *S, uint32_t *status, unsigned char *smem)
{
    hist_clear<ES>(smem, kBHistBytesPersist);
    __syncthreads();
    hist_tile<ES>(smem, kBHistBytesPersist, it, tile, S, status);
    __syncthreads();
    hist_flush<ES>(smem, kBHistBytesPersist, it, tile, status);
}

// elements of a compress pass's view
__device__ __forceinline__ uint64_t view_len(const BItem &it, const StreamDesc *S)
{
    int nd = 0;
    for (int k = 0; k < kMaxViewOps; k++) nd += it.vop[k] == V_DELTA;
    const uint64_t n_src = S[it.in[0]].len / it.es;
    return n_src > (uint64_t)nd ? n_src - nd : 0;
}

// The k most frequent values of an item.  A candidate is a count and a sort key (unique among the
// table's values, so the bits follow from it); more occurrences first, then the smaller key.
struct Cand {
    unsigned long long key;
    uint32_t count;  // 0 = none
};
__device__ __forceinline__ bool cbetter(const Cand &a, const Cand &b)
{
    return a.count > b.count || (a.count == b.count && a.count != 0 && a.key < b.key);
}
__device__ __forceinline__ void cpush(Cand (&l)[4], Cand c)
{
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const bool up = cbetter(c, l[i]);
        const Cand x = l[i];
        l[i] = up ? c : x;
        c = up ? x : c;
    }
}
// the four best of a warp's lists: candidate j in every lane's r[j]
__device__ __forceinline__ void warp_top4(Cand (&l)[4], Cand (&r)[4])
{
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t best = __reduce_max_sync(0xffffffffu, l[0].count);
        bool in = l[0].count == best && best;
        const uint32_t hi = __reduce_min_sync(0xffffffffu, in ? (uint32_t)(l[0].key >> 32) : ~0u);
        in = in && (uint32_t)(l[0].key >> 32) == hi;
        const uint32_t lo = __reduce_min_sync(0xffffffffu, in ? (uint32_t)l[0].key : ~0u);
        in = in && (uint32_t)l[0].key == lo;
        r[j] = Cand{(unsigned long long)hi << 32 | lo, best};
        // equal candidates (NaNs) are taken one at a time
        const unsigned who = __ballot_sync(0xffffffffu, in);
        if (in && (threadIdx.x & 31) == (uint32_t)__ffs(who) - 1) {
            l[0] = l[1];
            l[1] = l[2];
            l[2] = l[3];
            l[3] = Cand{0, 0};
        }
    }
}
// ... of a block's lists, in the first warp's lanes
__device__ __forceinline__ void block_top4(Cand (&l)[4], Cand (&r)[4])
{
    __shared__ Cand s_c[kBThreads / 32 * 4];
    warp_top4(l, r);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (lane == (uint32_t)j) s_c[4 * warp + j] = r[j];
    __syncthreads();
    if (warp == 0) {
        static_assert(kBThreads / 32 * 4 == 32, "one candidate a lane");
        Cand m[4] = {s_c[lane], {0, 0}, {0, 0}, {0, 0}};
        warp_top4(m, r);
    }
}

// The item's blocks that have work -- one per 512 table slots taken and NaN keys listed -- each take a
// slice of the used-slot list (and of the NaN lists), reduce it to a top-4, clear their slots for the
// next step and write the top-4 to the partial list; the last one to finish (threadfence + counter)
// merges the partials, writes the result and resets the header.  A table of which a fifth is taken (one
// larger than L2: a 32nd) is walked in order instead: 12 bytes a slot each way in whole lines, where the
// list takes four scattered accesses a value.  2^26 different int32 (a quarter taken): 23.3 -> 0.7 ms.
template <int ES>
__device__ __forceinline__ void put_top(const BItem &it, StreamDesc *S, const Cand (&r)[4]);

constexpr uint64_t kWalkCap = 1 << 22;  // slots (12 bytes each) of a table that L2 holds

// block `tile` of `blocks`
template <int ES>
__device__ __forceinline__ void topk_blocks(const BItem &it, uint32_t tile, uint32_t blocks, StreamDesc *S)
{
    constexpr unsigned long long EMPTY = ~0ull;
    __shared__ bool s_last;
    const HTab t = htab(it);
    const Order o = (Order)it.order;
    const uint64_t used = *(volatile unsigned int *)&t.hdr->used, n = view_len(it, S), nan_n = 4 * ((n + it.p[3] - 1) / it.p[3]);
    const uint64_t want = (used + nan_n + 511) / 512;
    if (blocks > it.tiles) blocks = it.tiles;  // the partial list holds one entry a histogram tile
    const uint32_t T = want > blocks ? blocks : want ? (uint32_t)want : 1u;
    if (tile >= T) return;
    const uint64_t slice = (used + T - 1) / T, nslice = (nan_n + T - 1) / T;
    const uint64_t lo = (uint64_t)tile * slice, hi = lo + slice < used ? lo + slice : used;
    const uint64_t nlo = (uint64_t)tile * nslice, nhi = nlo + nslice < nan_n ? nlo + nslice : nan_n;
    Cand l[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}}, r[4];
    if (used * (t.cap > kWalkCap ? 32 : 5) > t.cap) {
        const uint64_t pairs = t.cap / 2, step = (uint64_t)T * kBThreads;
        ulonglong2 *keys = (ulonglong2 *)t.keys;
        uint2 *counts = (uint2 *)t.counts;
        for (uint64_t i = (uint64_t)tile * kBThreads + threadIdx.x; i < pairs; i += 2 * step) {
            ulonglong2 k[2];
            uint2 c[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const bool in = i + q * step < pairs;
                k[q] = in ? keys[i + q * step] : make_ulonglong2(EMPTY, EMPTY);
                c[q] = in ? counts[i + q * step] : make_uint2(0, 0);
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (k[q].x == EMPTY && k[q].y == EMPTY) continue;
                keys[i + q * step] = make_ulonglong2(EMPTY, EMPTY);
                counts[i + q * step] = make_uint2(0, 0);
                if (k[q].x != EMPTY) cpush(l, Cand{order_key(k[q].x, ES, o), c[q].x});
                if (k[q].y != EMPTY) cpush(l, Cand{order_key(k[q].y, ES, o), c[q].y});
            }
        }
    } else
    for (uint64_t i = lo + threadIdx.x; i < hi; i += 4 * kBThreads) {
        unsigned int h[4], c[4];
        unsigned long long k[4];
#pragma unroll
        for (int q = 0; q < 4; q++) h[q] = i + q * kBThreads < hi ? t.used[i + q * kBThreads] : 0u;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (i + q * kBThreads < hi) {
                k[q] = t.keys[h[q]];
                c[q] = t.counts[h[q]];
                t.keys[h[q]] = EMPTY;
                t.counts[h[q]] = 0;
            }
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (i + q * kBThreads < hi) cpush(l, Cand{order_key(k[q], ES, o), c[q]});
    }
    if (tile == 0 && threadIdx.x == 0 && t.hdr->special) cpush(l, Cand{order_key(EMPTY, ES, o), t.hdr->special});
    for (uint64_t i = nlo + threadIdx.x; i < nhi; i += kBThreads) {
        const unsigned long long k = t.nan[i];
        if (k != EMPTY) cpush(l, Cand{k, 1u});
    }
    block_top4(l, r);
    if (T > 1) {
        unsigned long long *part = t.part + (uint64_t)tile * 12;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (threadIdx.x == (uint32_t)j) {
                part[3 * j] = r[j].key;
                part[3 * j + 1] = r[j].count;
            }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(&t.hdr->pad, 1u) == T - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        Cand m[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
        for (uint64_t i = threadIdx.x; i < 4ull * T; i += kBThreads) {
            const volatile unsigned long long *q = t.part + 3 * i;
            cpush(m, Cand{q[0], (uint32_t)q[1]});
        }
        block_top4(m, r);
    }
    if (threadIdx.x == 0) {
        put_top<ES>(it, S, r);
        t.hdr->used = 0;
        t.hdr->special = 0;
        t.hdr->overflow = 0;
        t.hdr->pad = 0;
    }
}

// ------------------------------------------------------------------------------- candidates
constexpr uint32_t kSampleSmem = 3072 * 12 + 4 * 512 + 4 * 64 + 16;
// The most frequent values of a node, in most columns without a full histogram: a sample names up to
// 400 candidates; one pass counts each candidate exactly and every other value in one of 4096 hash
// buckets; a bucket's count bounds the count of each value in it, so when the least of the k best
// candidates occurs more often than the largest bucket, those k are the most frequent ones, ties
// included.  (A NaN never equals another: each occurs once, and the four smallest are candidates too.)
// Where that proves nothing (values of nearly equal frequency), the item is flagged and the full
// histogram below runs.  The counting pass has no inserts: one lookup and one addition a value.  It is
// bound by issue and by the additions of equal values to one counter (14 % of the ids are one value).
// 2^26 Zipf(1.1) ids: histogram and top-k 0.550 -> 0.165 ms, of which the counting pass 0.125 (2.1 TB/s;
// 0.154 without the next rounds' loads in flight); the full histogram alone 0.287.  A tick table of 24
// such columns of 2^20 values: 0.41 -> 0.29 ms.
constexpr uint32_t kCandBuckets = kBCandSlots / 2;
struct CandArea {
    uint32_t *flag, *counts, *coarse;
    unsigned long long *nan;  // the complements of the four smallest NaN sort keys, 0 = none
    uint8_t *keys;
    __device__ __forceinline__ CandArea(const BItem &it)
    {
        uint8_t *b = it.scratch + it.cand;
        flag = (uint32_t *)b;
        nan = (unsigned long long *)(b + 16);
        counts = (uint32_t *)(b + 48);
        coarse = counts + kBCandSlots;
        keys = b + kBCandZero;
    }
};
// the hash of a value: its top 9 bits are its candidate bucket, its top 12 its coarse bucket
template <int ES>
__device__ __forceinline__ uint32_t cand_hash(word_t<ES> v)
{
    uint32_t m = (uint32_t)v;
    if (ES == 8) m = (m ^ (uint32_t)((uint64_t)v >> 32)) + (uint32_t)((uint64_t)v >> 45);
    return m * 0x9E3779B1u;
}
static_assert(kCandBuckets == 1u << 9 && kBCandCoarse == 1u << 12, "cand_hash's bits");

// One block an item: 2048 values spread over the column into a table in shared memory, all of them if there
// are at most 400 different ones, else the most frequent, up to 128, into the candidate table, the most
// frequent first, as a bucket holds two.  With 128 in any case, columns of 256 equally frequent values never
// proved anything (2^22 doubles of 256 values and 1 % others, dictionary: 258 us, now 110; before there were
// candidates 204); with 400 in any case Zipf ids took longer.  Where the sample shows that the counting will
// prove nothing it flags the item, and the full histogram starts without it (2^24 int16 of 1000 values:
// 261 -> 217 us, before there were candidates 245).
template <int ES>
__device__ __forceinline__ void p_hist_sample(const BItem &it, StreamDesc *S, unsigned char *smem)
{
    using K = word_t<ES>;
    using T = HistTable<ES>;
    constexpr uint32_t SAMPLE = 2048, SLOTS = 3072, ALL = 400, MOST = 128, HEAVY = 8;
    static_assert(SAMPLE == 1u << 11 && SLOTS * 12 + 4 * kCandBuckets + 4 * 64 + 16 <= kSampleSmem, "the sample's shared memory");
    const CandArea area(it);
    K *keys = (K *)smem;
    uint32_t *counts = (uint32_t *)(smem + SLOTS * 8), *fill = counts + SLOTS, *of_count = fill + kCandBuckets;
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    const Order o = (Order)it.order;
    for (uint32_t i = threadIdx.x; i < SLOTS; i += kBThreads) {
        keys[i] = T::MARK;
        counts[i] = 0;
    }
    for (uint32_t i = threadIdx.x; i < kCandBuckets + 64; i += kBThreads) fill[i] = 0;  // and of_count
    __syncthreads();
    constexpr int PER = SAMPLE / kBThreads;
    K v[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const uint64_t i = threadIdx.x + j * kBThreads;
        const uint64_t pos = n <= SAMPLE ? i : i * n >> 11;
        v[j] = pos < n ? (K)view_elem<ES>(it, vc, in.ptr, pos) : T::MARK;
    }
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const K x = v[j];
        if (x == T::MARK || x == T::MARK2 || is_nan_bits(x, o)) continue;
        uint32_t s = __umulhi(cand_hash<ES>(x), SLOTS);
        for (;;) {  // more slots than values: ends
            K cur = ((volatile K *)keys)[s];
            if (cur == T::MARK) {
                if constexpr (ES == 8) cur = atomicCAS((unsigned long long *)keys + s, (unsigned long long)T::MARK, (unsigned long long)x);
                else cur = atomicCAS(keys + s, T::MARK, x);
                if (cur == T::MARK) cur = x;
            }
            if (cur == x) {
                atomicAdd(counts + s, 1u);
                break;
            }
            s = s + 1 == SLOTS ? 0 : s + 1;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < SLOTS; i += kBThreads)
        if (counts[i]) atomicAdd(of_count + (counts[i] < 63 ? counts[i] : 63), 1u);
    __syncthreads();
    // every warp by itself: how many values occur lane, 32 + lane times or more
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = of_count[lane], hi = of_count[32 + lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_down_sync(0xffffffffu, lo, d), y = __shfl_down_sync(0xffffffffu, hi, d);
        if (lane + d < 32) {
            lo += x;
            hi += y;
        }
    }
    lo += __shfl_sync(0xffffffffu, hi, 0);
    // the largest count that more than `most` values reach, 0 if none does
    auto reached = [&](uint32_t most) -> uint32_t {
        const uint32_t h = __ballot_sync(0xffffffffu, hi > most), l = __ballot_sync(0xffffffffu, lane && lo > most);
        return h ? 63 - __clz(h) : l ? 31 - __clz(l) : 0;
    };
    const uint32_t distinct = __shfl_sync(0xffffffffu, lo, 1);
    const uint32_t t = distinct <= ALL ? 1 : reached(MOST) + 1;                 // the smallest count taken
    const uint32_t passes = distinct <= ALL && distinct > MOST ? 3 : 2;         // (few values leave no bucket short)
    K *image = (K *)area.keys;
#pragma unroll 1
    for (uint32_t pass = 0; pass < passes; pass++) {
        for (uint32_t i = threadIdx.x; i < SLOTS; i += kBThreads) {
            const uint32_t c = counts[i];
            if (c < t || c == 0 || pass != (c >= HEAVY ? 0 : c > 1 ? 1 : passes - 1)) continue;
            const uint32_t b = cand_hash<ES>(keys[i]) >> 23, w = atomicAdd(fill + b, 1u);
            if (w < 2) image[2 * b + w] = keys[i];
        }
        __syncthreads();
    }
    // The counting pass is for nothing when the k-th best is no better than chance among values of one
    // frequency: of such, m1 of which occur once and m2 twice, about m1 l^(c-1) / c! occur c times,
    // l = 2 m2 / m1 (over 400 of them: l below 6).  A k-th best of two is chance only if many others
    // occur twice.
    const uint32_t kth = reached((uint32_t)it.mode - 1), two = __shfl_sync(0xffffffffu, lo, 2), three = __shfl_sync(0xffffffffu, lo, 3);
    if (threadIdx.x == kBThreads - 1 && t > 1 && kth < 63) {
        const float m1 = (float)(distinct - two), l = m1 > 0 ? fminf(2 * (float)(two - three) / m1, 6.f) : 0.f;
        const float enough = (float)it.mode * (kth == 2 ? 4.f : 0.25f);
        float chance = m1;
        for (uint32_t j = 2; j <= kth && (chance >= enough || (float)j <= l); j++) chance *= __fdividef(l, (float)j);
        if (chance >= enough) *area.flag = 1;
    }
    const uint32_t special = cand_hash<ES>(T::MARK) >> 23;
    for (uint32_t b = threadIdx.x; b < kCandBuckets; b += kBThreads)
        for (uint32_t w = fill[b]; w < 2; w++) image[2 * b + w] = b == special ? T::MARK2 : T::MARK;
}

// shared memory of the counting pass: keys, counts, coarse counts, a word a lane that takes the
// additions of NaNs (nobody reads it), the smallest NaNs
constexpr uint32_t kCandNan = 8 * kBCandSlots + 4 * (kBCandSlots + kBCandCoarse) + 4 * 32, kCandSmem = kCandNan + 32;

// keeps the four largest of the nk given to it: what a place gives up moves on to the next
__device__ __noinline__ void cand_nan(unsigned long long *nan, unsigned long long nk)
{
    if (nk <= *(volatile unsigned long long *)(nan + 3)) return;
    for (int j = 0; j < 4; j++) {
        const unsigned long long old = atomicMax(nan + j, nk);
        nk = old < nk ? old : nk;
    }
}

template <int ES>
__device__ __forceinline__ void cand_load(const BItem &it, unsigned char *smem)
{
    const CandArea area(it);
    constexpr uint32_t KW = kBCandSlots * sizeof(word_t<ES>) / 16, CW = (kCandSmem - 8 * kBCandSlots) / 16;
    for (uint32_t i = threadIdx.x; i < KW; i += blockDim.x) ((uint4 *)smem)[i] = ldg((const uint4 *)area.keys + i);
    for (uint32_t i = threadIdx.x; i < CW; i += blockDim.x) ((uint4 *)(smem + 8 * kBCandSlots))[i] = make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void cand_flush(const BItem &it, const unsigned char *smem)
{
    const CandArea area(it);
    const uint32_t *c = (const uint32_t *)(smem + 8 * kBCandSlots);
    for (uint32_t i = threadIdx.x; i < kBCandSlots + kBCandCoarse; i += blockDim.x)
        if (c[i]) atomicAdd(area.counts + i, c[i]);  // coarse follows counts
    const unsigned long long *nan = (const unsigned long long *)(smem + kCandNan);
    if (threadIdx.x < 4 && nan[threadIdx.x]) cand_nan(area.nan, nan[threadIdx.x]);
}

// clears the code words of values [t0, end) (out1 after its 16 + 4*es header)
__device__ __forceinline__ void clear_codes(const BItem &it, uint64_t t0, uint64_t end, StreamDesc *S)
{
    uint32_t *words = (uint32_t *)(S[it.out[1]].ptr + 16 + 4 * it.es);
    for (uint64_t w = t0 / 16 + threadIdx.x; w < (end + 15) / 16; w += blockDim.x) words[w] = 0u;
}

// A tile of the counting pass (n * s read).  A dictionary's 2-bit code words are cleared by the way.
template <int ES, bool FP>
__device__ __forceinline__ void cand_tile_of(const BItem &it, uint32_t tile, StreamDesc *S, unsigned char *smem)
{
    using K = word_t<ES>;
    constexpr int N = 16 / ES;
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n, HT = it.p[3], t0 = (uint64_t)tile * HT;
    if (t0 >= n) return;
    const uint64_t end = n < t0 + HT ? n : t0 + HT;
    if (it.mode == 4) clear_codes(it, t0, end, S);
    const uint32_t keys = (uint32_t)__cvta_generic_to_shared(smem), counts = keys + 8 * kBCandSlots;
    const uint32_t lane = threadIdx.x & 31;
    constexpr Order FO = ES == 8 ? ORD_F64 : ORD_F32;
    auto place = [&](K v) -> uint32_t {  // the address of v's counter
        const uint32_t h = cand_hash<ES>(v), b = h >> 23;
        K k0, k1;
        sm_pair(keys + 2 * sizeof(K) * b, k0, k1);
        const uint32_t c = counts + 8 * b;
        const uint32_t a = k0 == v ? c : k1 == v ? c + 4 : counts + 4 * kBCandSlots + 4 * (h >> 20);
        return FP && is_nan_bits(v, FO) ? counts + 4 * (kBCandSlots + kBCandCoarse) + 4 * lane : a;
    };
    auto nans = [&](K v, uint32_t c) {  // c occurrences of v, if it is a NaN
        if (FP && is_nan_bits(v, FO))
            for (uint32_t q = 0; q < c && q < 4; q++)
                cand_nan((unsigned long long *)(smem + kCandNan), ~(unsigned long long)order_key(v, ES, FO));
    };
    const uint64_t step = (uint64_t)blockDim.x * N;
    // two rounds' loads are in flight while two are counted (fewer for narrow types: registers)
    constexpr int R = ES == 1 ? 1 : 2;
    K u[R][N], next[R][N];
    uint64_t w0 = t0 + (uint64_t)(threadIdx.x - lane) * N;
#pragma unroll
    for (int r = 0; r < R; r++)
        if (w0 + lane * N + r * step < end) load_vec<ES>(vc, in.ptr, w0 + lane * N + r * step, next[r]);
    for (; w0 < end; w0 += R * step) {
        const uint64_t b0 = w0 + lane * N;
#pragma unroll
        for (int r = 0; r < R; r++) {
#pragma unroll
            for (int q = 0; q < N; q++) u[r][q] = next[r][q];
            const uint64_t b = b0 + (R + r) * step;
            if (b < end) load_vec<ES>(vc, in.ptr, b, next[r]);
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint64_t base = b0 + r * step;
            const int cnt = base >= end ? 0 : end - base < (uint64_t)N ? (int)(end - base) : N;  // this lane's values
            K(&v)[N] = u[r];
            bool same = cnt == N;
#pragma unroll
            for (int q = 1; q < N; q++) same = same && v[q] == v[0];
            if (__all_sync(0xffffffffu, same)) {  // runs: one addition a thread, or a warp
                int one;
                __match_all_sync(0xffffffffu, v[0], &one);
                if (!one || lane == 0) {
                    sm_add(place(v[0]), one ? 32 * N : N);
                    nans(v[0], one ? 32 * N : N);
                }
                continue;
            }
            uint32_t at[N];
#pragma unroll
            for (int q = 0; q < N; q++) at[q] = place(v[q]);
#pragma unroll
            for (int q = 0; q < N; q++)
                if (q < cnt) sm_add(at[q], 1u);
            if (FP) {
#pragma unroll
                for (int q = 0; q < N; q++)
                    if (q < cnt) nans(v[q], 1u);
            }
        }
    }
}

template <int ES>
__device__ __forceinline__ void cand_tile(const BItem &it, uint32_t tile, StreamDesc *S, unsigned char *smem)
{
    if (ES >= 4 && it.order != ORD_INT) cand_tile_of<ES, (ES >= 4)>(it, tile, S, smem);
    else cand_tile_of<ES, false>(it, tile, S, smem);
}

// one tile on its own (the persistent schedule)
template <int ES>
__device__ __forceinline__ void p_hist_count(const BItem &it, uint32_t tile, StreamDesc *S, unsigned char *smem)
{
    const uint64_t n = view_len(it, S), t0 = (uint64_t)tile * it.p[3];
    if (t0 >= n) return;
    if (*CandArea(it).flag) {
        if (it.mode == 4) clear_codes(it, t0, n < t0 + it.p[3] ? n : t0 + it.p[3], S);
        return;
    }
    cand_load<ES>(it, smem);
    __syncthreads();
    cand_tile<ES>(it, tile, S, smem);
    __syncthreads();
    cand_flush(it, smem);
}

// the k most frequent values to where the split reads them: dict after out1's 16-byte header, const at
// the start of its metadata (which may lie anywhere: bytes)
template <int ES>
__device__ __forceinline__ void put_top(const BItem &it, StreamDesc *S, const Cand (&r)[4])
{
    const Order o = (Order)it.order;
    const int k = it.mode;
    uint8_t *dst = k == 1 ? S[it.out[0]].ptr : S[it.out[1]].ptr + 16;
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (j < k) {
            const uint64_t v = r[j].count ? order_unkey(r[j].key, ES, o) : 0ull;
            for (int b = 0; b < ES; b++) dst[j * ES + b] = (uint8_t)(v >> (8 * b));
        }
}

// one block an item: the k best candidates, or the flag
template <int ES>
__device__ __forceinline__ void p_cand_top(const BItem &it, StreamDesc *S)
{
    __shared__ uint32_t s_max;
    const CandArea area(it);
    const Order o = (Order)it.order;
    const bool flagged = *area.flag != 0;  // already, by the sample
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    constexpr int PER = (int)(kBCandSlots / kBThreads), COARSE = (int)(kBCandCoarse / kBThreads / 4);
    uint32_t c[PER], most = 0;
    word_t<ES> k[PER];
    uint4 g[COARSE];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const uint32_t i = threadIdx.x + j * kBThreads;
        c[j] = ldg(area.counts + i);
        k[j] = ldg((const word_t<ES> *)area.keys + i);
    }
#pragma unroll
    for (int j = 0; j < COARSE; j++) g[j] = ldg((const uint4 *)area.coarse + threadIdx.x + j * kBThreads);
    if (flagged) return;
    Cand l[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}}, r[4];
#pragma unroll
    for (int j = 0; j < COARSE; j++) most = max(max(most, max(g[j].x, g[j].y)), max(g[j].z, g[j].w));
#pragma unroll
    for (int j = 0; j < PER; j++)
        if (c[j]) cpush(l, Cand{order_key(k[j], ES, o), c[j]});
    if (threadIdx.x < 4 && area.nan[threadIdx.x]) cpush(l, Cand{~area.nan[threadIdx.x], 1u});
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_max, most);
    block_top4(l, r);  // its barriers publish s_max
    if (threadIdx.x == 0) {
        const uint32_t least = it.mode == 1 ? r[0].count : r[3].count;
        if (s_max == 0 || s_max < least) put_top<ES>(it, S, r);
        else *area.flag = 1;
    }
}

#ifndef GTSC_PERSISTENT_TU
// The counting pass's stage launch: as many blocks as are resident, striding over the tiles; a block
// keeps its counters while its tiles are of one item.
__global__ void __launch_bounds__(kBThreads, 4)
k_bcount(const BItem *items, const uint32_t *item_of, StreamDesc *S, uint32_t total_tiles)
{
    __shared__ __align__(16) unsigned char smem[kCandSmem];
    constexpr uint32_t NONE = 0xffffffffu;
    __shared__ bool s_flagged;  // the item's sample says that the counts would prove nothing
    uint32_t t = blockIdx.x, cur = NONE;
    while (t < total_tiles) {
        const uint32_t k = item_of[t];
        if (k != cur) {
            __syncthreads();  // the counters are complete, nobody reads the previous descriptor any more
            if (cur != NONE && !s_flagged) cand_flush(shared_item_ref(), smem);
            __syncthreads();
            shared_item(items, k);
            const uint32_t flag = threadIdx.x == 0 ? *CandArea(shared_item_ref()).flag : 0;  // loads beside the others
            with_size(shared_item_ref().es, [&](auto es) { cand_load<decltype(es)::value>(shared_item_ref(), smem); });
            if (threadIdx.x == 0) s_flagged = flag != 0;
            __syncthreads();
            cur = k;
        }
        const BItem &it = shared_item_ref();
        const uint32_t tile = t - (uint32_t)it.tile_base;
        const uint64_t n = view_len(it, S), t0 = (uint64_t)tile * it.p[3];
        if (t0 >= n) {
            const uint64_t next = it.tile_base + it.tiles;  // the next item's first tile
            if (next >= total_tiles) break;
            t = (uint32_t)(next + (blockIdx.x + gridDim.x - next % gridDim.x) % gridDim.x);
            continue;
        }
        if (!s_flagged) with_size(it.es, [&](auto es) { cand_tile<decltype(es)::value>(shared_item_ref(), tile, S, smem); });
        else if (it.mode == 4) clear_codes(it, t0, n < t0 + it.p[3] ? n : t0 + it.p[3], S);
        t += gridDim.x;
    }
    __syncthreads();
    if (cur != NONE && !s_flagged) cand_flush(shared_item_ref(), smem);
}

// The items of a launch whose flag is set, in order, f(index) for each; the block's threads look at 256
// or more of them at a time.
template <class F>
__device__ __forceinline__ void flagged_items(const BItem *items, int n_items, F f)
{
    __shared__ uint32_t s_mask[32];
    for (int i0 = 0; i0 < n_items; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x;
        const bool on = i < n_items && *CandArea(items[i]).flag != 0;
        const uint32_t m = __ballot_sync(0xffffffffu, on);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) s_mask[threadIdx.x >> 5] = m;
        if (!__syncthreads_or(on)) continue;
        for (uint32_t w = 0; w < blockDim.x / 32; w++)
            for (uint32_t rest = s_mask[w]; rest; rest &= rest - 1) f(i0 + 32 * w + __ffs(rest) - 1);
        __syncthreads();
    }
}

// The full histogram's stage launch, over the flagged items: as many blocks as are resident, striding
// over an item's tiles.  A block keeps its table while it is at most half full.
__global__ void __launch_bounds__(kBHistThreads, 2)
k_bhist(const BItem *items, int n_items, StreamDesc *S, uint32_t *status)
{
    extern __shared__ __align__(16) unsigned char table[];
    flagged_items(items, n_items, [&](int k) {
        __syncthreads();
        const BItem &it = shared_item(items, k);
        with_size(it.es, [&](auto es) {
            constexpr int E = decltype(es)::value;
            const uint64_t n = view_len(it, S), tiles = (n + it.p[3] - 1) / it.p[3];
            bool dirty = false;  // the table holds counts, up to tile `last`
            uint32_t last = 0;
            for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
                if (dirty) {  // the tile before went into this table too: its NaN keys are listed with this one's
                    if (threadIdx.x < 4) htab(it).nan[4ull * last + threadIdx.x] = ~0ull;
                } else {
                    hist_clear<E>(table, kBHistBytes);
                    __syncthreads();
                }
                hist_tile<E>(table, kBHistBytes, it, (uint32_t)t, S, status);
                last = (uint32_t)t;
                dirty = true;
                // one decision for the block: the threads' reads lie before the barrier
                const uint32_t used = *(volatile uint32_t *)&s_hist.used;
                if (__syncthreads_or(used > (E == 8 ? kBHistBytes / 24 : kBHistBytes / 16))) {
                    hist_flush<E>(table, kBHistBytes, it, last, status);
                    dirty = false;
                    __syncthreads();
                }
            }
            if (dirty) hist_flush<E>(table, kBHistBytes, it, last, status);
        });
    });
}

__global__ void __launch_bounds__(kBThreads, 4) k_btopk(const BItem *items, int n_items, StreamDesc *S)
{
    flagged_items(items, n_items, [&](int k) {
        __syncthreads();
        const BItem &it = shared_item(items, k);
        with_size(it.es, [&](auto es) { topk_blocks<decltype(es)::value>(it, blockIdx.x, gridDim.x, S); });
    });
}
#endif

// ------------------------------------------------------------------------------- split
// the outside variant of patch, beside SplitMode
constexpr int kSplitOutside = 100;
// code bytes of a warp in a dictionary's split: a unit's, from any place in a code word
constexpr uint32_t kSplitCodes = kBSplitUnit + 16;

// a split's element as a signed value, for the min / max of its classes
template <int ES>
using sword_t = std::conditional_t<ES == 8, int64_t, int32_t>;

template <int ES>
__device__ __forceinline__ void warp_min_max(sword_t<ES> &mn, sword_t<ES> &mx)
{
    if constexpr (ES == 8) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int64_t a = __shfl_xor_sync(0xffffffffu, mn, o), b = __shfl_xor_sync(0xffffffffu, mx, o);
            mn = a < mn ? a : mn;
            mx = b > mx ? b : mx;
        }
    } else {
        mn = __reduce_min_sync(0xffffffffu, mn);
        mx = __reduce_max_sync(0xffffffffu, mx);
    }
}

// a < b in the element's own arithmetic (lt_native), in registers of its width
template <int ES, bool FP>
__device__ __forceinline__ bool lt_word(word_t<ES> a, word_t<ES> b)
{
    if constexpr (FP && ES == 8) return __longlong_as_double((long long)a) < __longlong_as_double((long long)b);
    else if constexpr (FP) return __uint_as_float(a) < __uint_as_float(b);
    else return (std::make_signed_t<elem_t<ES>>)a < (std::make_signed_t<elem_t<ES>>)b;
}

// 16 bytes holding one 2-bit code each (or anything, where no code is) -> a code word (byte k's low
// bits at 2 k)
__device__ __forceinline__ uint32_t pack_codes(const uint4 &q)
{
    // the product's top byte gathers the four codes of a word: no two of its terms share a bit
    auto four = [](uint32_t w) { return ((w & 0x03030303u) * 0x01041040u) >> 24; };
    return four(q.x) | four(q.y) << 8 | four(q.z) << 16 | four(q.w) << 24;
}

// What a split compares its values with.
template <int ES>
struct SplitArgs {
    word_t<ES> match[4];  // const / dict: the values looked for; a NaN never matches: another one in its place
    bool all_nan;         // none is left
    word_t<ES> thr, low;  // patch: the threshold (outside: the high bound) and the low bound
};

// the classes of R rows: x is a match
template <int ES, int MODE, bool FP>
__device__ __forceinline__ bool split_yes(word_t<ES> x, const SplitArgs<ES> &a)
{
    if constexpr (MODE == SPLIT_NOT_CONST) return x != a.match[0] || a.all_nan;
    else if constexpr (MODE == SPLIT_DICT)
        return (x == a.match[0] || x == a.match[1] || x == a.match[2] || x == a.match[3]) && !a.all_nan;
    else if constexpr (MODE == kSplitOutside)  // OutsideOperator (stencil_operators.hpp:14-25)
        return !(lt_word<ES, FP>(a.thr, x) || lt_word<ES, FP>(x, a.low));
    else return lt_word<ES, FP>(x, a.thr);
}

// R rows of a unit: their ballots go to lane j (row j) of `mine`; FOLD: the signed min / max of the
// matches and of the rest go to mm
template <int ES, int MODE, bool FP, bool FOLD, bool FULL, int R>
__device__ __forceinline__ void split_ballots(const ViewCtx &vc, const uint8_t *src, uint64_t base, uint32_t cnt,
                                              uint32_t j0, const SplitArgs<ES> &a, uint32_t &mine, sword_t<ES> (&mm)[4])
{
    using SV = sword_t<ES>;
    constexpr SV LO = ES == 8 ? (SV)INT64_MIN : (SV)INT32_MIN, HI = ~LO;
    const uint32_t lane = threadIdx.x & 31;
    const int left = (int)cnt - (int)lane;
    word_t<ES> v[R];
    load_rows<ES, R, FULL>(vc, src, base, cnt, v);
#pragma unroll
    for (int j = 0; j < R; j++) {
        const bool in = FULL || 32 * j < left, y = in && split_yes<ES, MODE, FP>(v[j], a);
        const uint32_t b = __ballot_sync(0xffffffffu, y);
        mine = lane == j0 + j ? b : mine;
        if (FOLD) {
            const SV x = (SV)(std::make_signed_t<elem_t<ES>>)v[j];
            const bool no = in && !y;
            mm[0] = min(mm[0], y ? x : HI);
            mm[1] = max(mm[1], y ? x : LO);
            mm[2] = min(mm[2], no ? x : HI);
            mm[3] = max(mm[3], no ? x : LO);
        }
    }
}

// A split takes two passes over its input: this one finds the classes (n * s read, n / 8 written) and
// the other moves the values, so that no block ever waits for another's count.  One warp a unit of
// 1024 values, in rows of 32: a row's ballot is its stencil word.  Also the min / max of the classes
// that an AFL child packs (integer order, as its own min/max pass would compute it).
template <int ES, int MODE, bool FP>
__device__ __forceinline__ void split_count(const BItem &it, uint32_t tile, uint32_t step, uint32_t end, StreamDesc *S)
{
    using V = word_t<ES>;
    using SV = sword_t<ES>;
    constexpr int R = 8;
    constexpr bool CONST = MODE == SPLIT_NOT_CONST, DICT = MODE == SPLIT_DICT;
    constexpr uint32_t WARPS = kBThreads / 32;
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    const Order o = (Order)it.order;
    uint8_t *meta = S[it.out[0]].ptr;
    if (tile == 0 && threadIdx.x == 0) {
        meta[CONST ? ES : 0] = (uint8_t)(n % 8);
        if (n == 0) {
            S[it.out[0]].len = 0;
            S[it.out[1]].len = 0;
            if (!CONST) S[it.out[2]].len = 0;
        }
    }
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SplitArgs<ES> a{};
    if constexpr (CONST || DICT) {
        const uint8_t *tp = CONST ? meta : S[it.out[1]].ptr + 16;
        V good = 0;
        a.all_nan = true;
#pragma unroll
        for (int k = CONST ? 0 : 3; k >= 0; k--) {
            const V x = CONST ? (V)ld_unaligned<ES>(tp) : (V)ld_elem<ES>(tp, k);
            a.match[k] = x;
            if (!is_nan_bits(x, o)) {
                good = x;
                a.all_nan = false;
            }
        }
#pragma unroll
        for (int k = CONST ? 0 : 3; k >= 0; k--)
            if (is_nan_bits(a.match[k], o)) a.match[k] = good;
    } else {
        uint64_t mnb = 0, mxb = 0, thr, low = 0;
        if (!acc_minmax((const MinMaxAcc *)it.scratch, ES, o, mnb, mxb) && n) mnb = mxb = view_elem<ES>(it, vc, in.ptr, 0);
        if (MODE == kSplitOutside) d_outside_patch_bounds(mnb, mxb, it.dt, ES, low, thr);  // thr: the high bound
        else thr = d_patch_threshold(mnb, mxb, it.dt, ES);
        a.thr = (V)thr;
        a.low = (V)low;
    }
    const bool fold_y = it.p[2] != 0, fold_n = it.p[3] != 0;
    constexpr SV LO = ES == 8 ? (SV)INT64_MIN : (SV)INT32_MIN, HI = ~LO;
    __shared__ uint32_t s_tot[WARPS];
    __shared__ unsigned long long s_fold[WARPS][4];
#pragma unroll 1
    for (; tile < end; tile += step) {
    const uint64_t w0 = (uint64_t)tile * kBSplitTile + warp * kBSplitUnit;  // the warp's first value
    const uint32_t cnt = w0 >= n ? 0u : (uint32_t)(n - w0 < kBSplitUnit ? n - w0 : kBSplitUnit);
    SV mm[4] = {HI, LO, HI, LO};
    uint32_t mine = 0;
    if (fold_y || fold_n) {
#pragma unroll 1
        for (uint32_t j = 0; 32 * j < cnt; j += R) {
            if (32 * (j + R) <= cnt) split_ballots<ES, MODE, FP, true, true, R>(vc, in.ptr, w0 + 32 * j, 32 * R, j, a, mine, mm);
            else split_ballots<ES, MODE, FP, true, false, R>(vc, in.ptr, w0 + 32 * j, cnt - 32 * j, j, a, mine, mm);
        }
    } else {
#pragma unroll 1
        for (uint32_t j = 0; 32 * j < cnt; j += R) {
            if (32 * (j + R) <= cnt) split_ballots<ES, MODE, FP, false, true, R>(vc, in.ptr, w0 + 32 * j, 32 * R, j, a, mine, mm);
            else split_ballots<ES, MODE, FP, false, false, R>(vc, in.ptr, w0 + 32 * j, cnt - 32 * j, j, a, mine, mm);
        }
    }
    const uint32_t total = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(mine));
    if (32 * lane < cnt) {
        uint32_t word = mine;
        const uint32_t left = cnt - 32 * lane;  // Stencil::pack's index clamp: the last element fills the last byte
        if (left < 32 && ((word >> (left - 1)) & 1u)) word |= ~0u << left;
        ((uint32_t *)(meta + (CONST ? ES + 1 : 1)))[w0 / 32 + lane] = word;  // 4-byte aligned (layout)
    }
    if (lane == 0) s_tot[warp] = total;
    if (fold_y || fold_n) {
        warp_min_max<ES>(mm[0], mm[1]);
        warp_min_max<ES>(mm[2], mm[3]);
        if (lane == 0) {  // as the accumulators hold them; 0 = nothing seen
            const uint64_t sign = 1ull << 63;
            const bool ys = fold_y && total, ns = fold_n && cnt > total;
            s_fold[warp][0] = ys ? ~((uint64_t)(int64_t)mm[0] ^ sign) : 0ull;
            s_fold[warp][1] = ys ? (uint64_t)(int64_t)mm[1] ^ sign : 0ull;
            s_fold[warp][2] = ns ? ~((uint64_t)(int64_t)mm[2] ^ sign) : 0ull;
            s_fold[warp][3] = ns ? (uint64_t)(int64_t)mm[3] ^ sign : 0ull;
        }
    }
    __syncthreads();
    if (warp == 0) {
        static_assert(WARPS == 8, "a tile's unit counts are 8 halfwords");
        const uint32_t c = lane < WARPS ? s_tot[lane] : 0u;
        unsigned long long *groups = (unsigned long long *)(it.scratch + it.p[0]);
        uint16_t *counts = (uint16_t *)((uint8_t *)groups + bsplit_group_bytes(it.tiles));
        if (lane < WARPS) counts[(uint64_t)tile * WARPS + lane] = (uint16_t)c;
        const uint32_t sum = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && sum) atomicAdd(groups + tile / kBSplitGroup, (unsigned long long)sum);
    } else if (warp == 1 && lane < 4 && (lane < 2 ? fold_y : fold_n)) {
        unsigned long long x = 0;
        for (int w = 0; w < (int)WARPS; w++) x = s_fold[w][lane] > x ? s_fold[w][lane] : x;
        MinMaxAcc *acc = (MinMaxAcc *)it.p[lane < 2 ? 2 : 3];
        unsigned long long *dst = lane & 1 ? &acc->kmax : &acc->nkmin;
        if (x > *(volatile unsigned long long *)dst) atomicMax(dst, x);  // most tiles do not move it
    }
    __syncthreads();  // the next tile's counts
    }
}

__device__ __forceinline__ void p_split_count(const BItem &it, uint32_t tile, uint32_t step, uint32_t end, StreamDesc *S)
{
    with_size(it.es, [&](auto es) {
        constexpr int E = decltype(es)::value;
        if (it.mode == SPLIT_DICT) split_count<E, SPLIT_DICT, false>(it, tile, step, end, S);
        else if (it.mode == SPLIT_NOT_CONST) split_count<E, SPLIT_NOT_CONST, false>(it, tile, step, end, S);
        else if (E >= 4 && it.order != ORD_INT) {
            if (it.p[1]) split_count<E, kSplitOutside, (E >= 4)>(it, tile, step, end, S);
            else split_count<E, SPLIT_LOWER, (E >= 4)>(it, tile, step, end, S);
        } else {
            if (it.p[1]) split_count<E, kSplitOutside, false>(it, tile, step, end, S);
            else split_count<E, SPLIT_LOWER, false>(it, tile, step, end, S);
        }
    });
}

// R rows of a unit to their runs: yes / no point at the unit's first match / other value (no: at this
// lane's), code at its first code byte
template <int ES, int MODE, bool FULL, int R>
__device__ __forceinline__ void split_rows(const ViewCtx &vc, const uint8_t *src, uint64_t base, uint32_t cnt, uint32_t j0,
                                           uint32_t word, uint32_t pre, const word_t<ES> (&top)[4], elem_t<ES> *yes,
                                           elem_t<ES> *no, unsigned char *code)
{
    const uint32_t lane = threadIdx.x & 31, bit = 1u << lane;
    const int left = (int)cnt - (int)lane;
    word_t<ES> v[R];
    load_rows<ES, R, FULL>(vc, src, base, cnt, v);
#pragma unroll
    for (int j = 0; j < R; j++) {
        const uint32_t m = __shfl_sync(0xffffffffu, word, j0 + j);
        const uint32_t r = __shfl_sync(0xffffffffu, pre, j0 + j) + __popc(m & (bit - 1));
        if (m & bit) {
            if constexpr (MODE == SPLIT_DICT) {
                const uint32_t e1 = v[j] == top[1], e2 = v[j] == top[2], e3 = v[j] == top[3];
                code[r] = (uint8_t)(e1 | (e2 << 1) | (e3 * 3u));
            } else {
                yes[r] = (elem_t<ES>)v[j];
            }
        } else if (MODE != SPLIT_NOT_CONST && (FULL || 32 * j < left)) {
            no[32 * (int)(j0 + j) - (int)r] = (elem_t<ES>)v[j];
        }
    }
}

// The second pass: every unit's values to the match and the other stream (n * s read again -- from L2
// for all but the largest columns -- and written).  The matches before a unit are the sums of the groups
// before its tile's, of the tiles before it in the group and of the units before it in the tile (a number
// for every 2^19 values before it: a term in the square of the length, which does not show yet from 2^26
// to 2^30 int32, both passes 0.169 -> 2.56 ms, where the look-back took 0.38 -> 5.92); a
// value's rank in its unit comes from the stencil words.  Rows are stored straight to the two runs;
// only a dictionary's 2-bit codes pass through shared memory, to be packed 16 a word.
// 2^26 int32, both passes: patch 0.430 -> 0.182 ms, Zipf(1.1) dictionary 0.506 -> 0.233 ms (0.206 and
// 0.247 with the setup done for every tile).  One pass with
// the rows held in registers behind a look-back took 0.26 and 0.29 ms (its warps wait at the barrier of
// the look-back); the same with two tiles in flight a block 0.27 and 0.33 ms (too few warps).
template <int ES, int MODE, bool OWN>
__device__ __forceinline__ void split_move(const BItem &it, uint32_t tile, uint32_t step, uint32_t end, StreamDesc *S,
                                           unsigned char *sm)
{
    using V = word_t<ES>;
    constexpr int R = 8;
    constexpr bool CONST = MODE == SPLIT_NOT_CONST, DICT = MODE == SPLIT_DICT;
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint8_t *meta = S[it.out[0]].ptr;
    uint8_t *const out1 = S[it.out[1]].ptr, *const out2 = CONST ? nullptr : S[it.out[2]].ptr;
    V top[4] = {0, 0, 0, 0};
    if constexpr (DICT)
        for (int k = 1; k < 4; k++) top[k] = (V)ld_elem<ES>(out1 + 16, k);
#pragma unroll 1
    for (; tile < end; tile += step) {
    const uint64_t w0 = (uint64_t)tile * kBSplitTile + warp * kBSplitUnit;  // the warp's first value
    if (w0 >= n) break;
    const uint32_t cnt = (uint32_t)(n - w0 < kBSplitUnit ? n - w0 : kBSplitUnit);
    uint32_t word = 32 * lane < cnt ? ld_sum<OWN>((const uint32_t *)(meta + (CONST ? ES + 1 : 1)) + w0 / 32 + lane) : 0u;
    if (cnt < 32 * lane + 32 && cnt > 32 * lane) word &= (1u << (cnt - 32 * lane)) - 1;
    // the matches before the unit
    const unsigned long long *groups = (const unsigned long long *)(it.scratch + it.p[0]);
    const uint4 *counts = (const uint4 *)((const uint8_t *)groups + bsplit_group_bytes(it.tiles));
    unsigned long long part = 0;
    const uint32_t g = tile / kBSplitGroup;
    for (uint32_t k = lane; k < g; k += 32) part += ld_sum<OWN>(groups + k);
    auto halves = [](uint32_t w) { return (w & 0xffffu) + (w >> 16); };
    for (uint32_t k = g * kBSplitGroup + lane; k < tile; k += 32) {
        const uint4 q = ld_sum<OWN>(counts + k);
        part += halves(q.x) + halves(q.y) + halves(q.z) + halves(q.w);
    }
    if (lane < warp) part += ld_sum<OWN>((const uint16_t *)(counts + tile) + lane);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
    const uint64_t yes0 = part, no0 = w0 - yes0;
    uint32_t pre = __popc(word);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, pre, d);
        if (lane >= d) pre += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
    pre -= __popc(word);
    elem_t<ES> *yes = DICT ? nullptr : (elem_t<ES> *)out1 + yes0;
    elem_t<ES> *no = CONST ? nullptr : (elem_t<ES> *)out2 + no0 + lane;
    unsigned char *codes = sm + warp * kSplitCodes;
    const uint32_t c0 = (uint32_t)(yes0 & 15);  // the unit's first code inside its code word
#pragma unroll 1
    for (uint32_t j = 0; 32 * j < cnt; j += R) {
        // a const node moves its mismatches only: rows without one are not read again
        if (CONST && !__any_sync(0xffffffffu, lane >= j && lane < j + R && word)) continue;
        if (32 * (j + R) <= cnt) split_rows<ES, MODE, true, R>(vc, in.ptr, w0 + 32 * j, 32 * R, j, word, pre, top, yes, no, codes + c0);
        else split_rows<ES, MODE, false, R>(vc, in.ptr, w0 + 32 * j, cnt - 32 * j, j, word, pre, top, yes, no, codes + c0);
    }
    if constexpr (DICT) {
        // the unit's codes, 16 a word; the first and the last word may be shared with the neighbour
        // units and are or-ed in (the words start zeroed)
        __syncwarp();
        uint32_t *words = (uint32_t *)(out1 + 16 + 4 * ES) + (yes0 >> 4);
        const uint32_t codes_end = total ? c0 + total : 0;
        for (uint32_t k = lane; 16 * k < codes_end; k += 32) {
            uint32_t x = pack_codes(((const uint4 *)codes)[k]);
            const uint32_t lo = 16 * k < c0 ? c0 - 16 * k : 0, hi = codes_end - 16 * k < 16 ? codes_end - 16 * k : 16;
            if (lo == 0 && hi == 16) {
                words[k] = x;
            } else {  // bytes outside [lo, hi) are of an earlier unit
                x &= (hi == 16 ? ~0u : (1u << (2 * hi)) - 1) & (~0u << (2 * lo));
                if (x) atomicOr(words + k, x);
            }
        }
        __syncwarp();  // the next tile's codes
    }
    if (lane == 0 && w0 + kBSplitUnit >= n) {  // the unit of the last value: lengths and headers
        const uint64_t m = yes0 + total;
        if constexpr (CONST) {
            S[it.out[0]].len = ES + 1 + (n + 7) / 8;
            S[it.out[1]].len = m * ES;
        } else if constexpr (DICT) {
            uint64_t *sz = (uint64_t *)S[it.out[1]].ptr;
            sz[0] = 4;
            sz[1] = m;
            S[it.out[0]].len = 1 + (n + 7) / 8;
            S[it.out[1]].len = m ? 16 + 4 * ES + 4 * ((m + 15) / 16) : 0;
            S[it.out[2]].len = (n - m) * ES;
        } else {
            S[it.out[0]].len = 1 + (n + 7) / 8;
            S[it.out[1]].len = m * ES;
            S[it.out[2]].len = (n - m) * ES;
        }
    }
    }
}

template <int ES, bool OWN = false>
__device__ __forceinline__ void p_split(const BItem &it, uint32_t tile, uint32_t step, uint32_t end, StreamDesc *S,
                                        unsigned char *sm)
{
    if (it.mode == SPLIT_DICT) split_move<ES, SPLIT_DICT, OWN>(it, tile, step, end, S, sm);
    else if (it.mode == SPLIT_NOT_CONST) split_move<ES, SPLIT_NOT_CONST, OWN>(it, tile, step, end, S, sm);
    else split_move<ES, SPLIT_LOWER, OWN>(it, tile, step, end, S, sm);
}

// tiles of a short column's split
__device__ __forceinline__ uint32_t short_split_tiles(const BItem &it, const StreamDesc *S)
{
    const uint64_t t = (view_len(it, S) + kBSplitTile - 1) / kBSplitTile;
    return t < 1 ? 1u : t < kBShortTiles ? (uint32_t)t : kBShortTiles;
}

#ifndef GTSC_PERSISTENT_TU
// Both passes over short columns, a cluster a column and a block a tile.  One column, patch of 5000 / 20001
// int32, whole compress step: 31 / 33 -> 29 / 31 us.
__global__ void __cluster_dims__(kBShortTiles, 1, 1) __launch_bounds__(kBThreads, 4)
k_bsplit_short(const BItem *items, StreamDesc *S)
{
    __shared__ __align__(16) unsigned char smem[kSplitCodes * (kBThreads / 32)];
    const BItem &it = shared_item(items, blockIdx.x / kBShortTiles);
    const uint32_t tile = blockIdx.x % kBShortTiles;
    const bool mine = tile < short_split_tiles(it, S);
    if (mine) p_split_count(it, tile, 1, tile + 1, S);
    cluster_sync();
    if (mine) with_size(it.es, [&](auto es) { p_split<decltype(es)::value, true>(it, tile, 1, tile + 1, S, smem); });
}
#endif

// ------------------------------------------------------------------------------- RLE
template <int ES>
__device__ void p_rle_heads(const BItem &it, uint32_t tile, StreamDesc *S, uint8_t *xs)
{
    __shared__ unsigned long long ws[32];
    __shared__ unsigned long long s_prefix;
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    const uint64_t n = vc.n;
    const Order o = (Order)it.order;
    Lookback lb = lookback_at(it.scratch + it.p[0], it.tiles);
    uint32_t *starts = (uint32_t *)(it.scratch + it.p[1]);
    if (n == 0) {
        if (tile == 0 && threadIdx.x == 0) {
            *(int32_t *)S[it.out[0]].ptr = 0;
            S[it.out[0]].len = 4;
            S[it.out[1]].len = 0;
            S[it.out[2]].len = 0;
        }
        return;
    }
    if ((uint64_t)tile * kBTile >= n) return;  // past the input: no successor needs this tile
    const uint64_t base = (uint64_t)tile * kBTile + (uint64_t)threadIdx.x * kBVPT;
    uint64_t v[kBVPT];
    load_view_x<ES, kBVPT>(it, vc, in.ptr, base, v, xs);
    const uint64_t prev = base > 0 && base - 1 < n ? view_elem<ES>(it, vc, in.ptr, base - 1) : 0;
    uint32_t heads = 0;
#pragma unroll
    for (int j = 0; j < (int)kBVPT; j++) {
        const uint64_t i = base + j;
        if (i < n && (i == 0 || !bsame(v[j], j ? v[j - 1] : prev, o))) heads |= 1u << j;
    }
    unsigned long long total;
    const unsigned long long excl = block_exclusive_scan<kBThreads>((unsigned long long)__popc(heads), ws, total);
    if (threadIdx.x < 32) {
        const unsigned long long e = lookback_exclusive(lb, tile, total);
        if (threadIdx.x == 0) s_prefix = e;
    }
    __syncthreads();
    uint64_t r = s_prefix + excl;
    uint8_t *values = S[it.out[2]].ptr;
#pragma unroll
    for (int j = 0; j < (int)kBVPT; j++)
        if ((heads >> j) & 1u) {
            st_elem<ES>(values, r, v[j]);
            starts[r] = (uint32_t)(base + j);
            ++r;
        }
    if (base < n && base + kBVPT >= n) {
        *(int32_t *)S[it.out[0]].ptr = (int32_t)r;
        S[it.out[0]].len = 4;
        S[it.out[1]].len = 4 * r;
        S[it.out[2]].len = ES * r;
    }
}

__device__ void p_rle_lengths(const BItem &it, uint32_t tile, StreamDesc *S)
{
    int nd = 0;
    for (int k = 0; k < kMaxViewOps; k++) nd += it.vop[k] == V_DELTA;
    const uint64_t n_src = S[it.in[0]].len / it.es;
    const uint64_t n = n_src > (uint64_t)nd ? n_src - nd : 0;
    const uint64_t runs = S[it.out[1]].len / 4;
    const uint32_t *starts = (const uint32_t *)(it.scratch + it.p[1]);
    int32_t *lengths = (int32_t *)S[it.out[1]].ptr;
    const uint64_t r0 = (uint64_t)tile * kBTile;
    for (uint64_t r = r0 + threadIdx.x; r < runs && r < r0 + kBTile; r += kBThreads) {
        const uint64_t next = r + 1 < runs ? starts[r + 1] : n;
        lengths[r] = (int32_t)(next - starts[r]);
    }
}

// ------------------------------------------------------------------------------- floatToInt
__device__ __forceinline__ const double *pow10_table()
{
    __shared__ double t[10];
    if (threadIdx.x < 10) {
        double v = 1.0;
        for (unsigned i = 0; i < threadIdx.x; i++) v *= 10.0;
        t[threadIdx.x] = v;
    }
    __syncthreads();
    return t;
}

template <int ES>
__device__ __forceinline__ double as_double(uint64_t u, Order o)
{
    if (o == ORD_F32) return (double)__uint_as_float((uint32_t)u);
    if (o == ORD_F64) return __longlong_as_double((long long)u);
    if (ES == 8) return __ll2double_rn((long long)u);
    return (double)sext(u, ES);
}

template <int ES>
__device__ __forceinline__ float as_float_T(uint64_t u, Order o)
{
    if (o == ORD_F32) return __uint_as_float((uint32_t)u);
    if (o == ORD_F64) return __double2float_rn(__longlong_as_double((long long)u));
    if (ES == 8) return __ll2float_rn((long long)u);
    return __int2float_rn((int)sext(u, ES));
}

template <int ES>
__device__ __forceinline__ uint64_t f2i_dec_one(int k, int p, Order o, const double *p10)
{
    if (o == ORD_F32) return __float_as_uint(__double2float_rn(__ddiv_rn((double)__int2float_rn(k), p10[p])));
    if (o == ORD_F64) return (uint64_t)__double_as_longlong(__ddiv_rn((double)k, p10[p]));
    if (ES == 8) return (uint64_t)__double2ll_rz(__ddiv_rn((double)k, p10[p]));
    const long long t = sext((uint64_t)(long long)k, ES);
    return (uint64_t)(long long)__double2int_rz(__ddiv_rn((double)t, p10[p]));
}

// node scratch of floatToInt: StatsAcc at 0, lossy flag at 64
template <int ES>
__device__ void p_f2i_stats(const BItem &it, uint32_t tile, StreamDesc *S)
{
    const StreamDesc in = S[it.in[0]];
    const uint64_t n = in.len / ES;
    const uint64_t t0 = (uint64_t)tile * kBTile;
    if (t0 >= n) return;
    const Order o = (Order)it.order;
    uint64_t kmin = ~0ull, kmax = 0;
    int steps = 0;
    const uint64_t end = n < t0 + kBTile ? n : t0 + kBTile;
    for (uint64_t i = t0 + threadIdx.x; i < end; i += kBThreads) {
        const uint64_t u = ld_elem<ES>(in.ptr, i);
        if (!is_nan_bits(u, o)) {
            const uint64_t k = order_key(u, ES, o);
            kmin = k < kmin ? k : kmin;
            kmax = k > kmax ? k : kmax;
        }
        const int s = d_precision_steps(as_float_T<ES>(u, o));
        steps = s > steps ? s : steps;
    }
    for (int off = 16; off > 0; off >>= 1) {
        const int x = __shfl_xor_sync(0xffffffffu, steps, off);
        steps = x > steps ? x : steps;
    }
    __shared__ int s_steps[kBThreads / 32];
    if ((threadIdx.x & 31) == 0) s_steps[threadIdx.x >> 5] = steps;
    block_minmax(kmin, kmax);
    if (threadIdx.x == 0) {
        for (int w = 1; w < kBThreads / 32; w++) steps = s_steps[w] > steps ? s_steps[w] : steps;
        StatsAcc *acc = (StatsAcc *)it.scratch;
        if (kmin != ~0ull) atomicMax(&acc->mm.nkmin, (unsigned long long)~kmin);
        if (kmax != 0) atomicMax(&acc->mm.kmax, (unsigned long long)kmax);
        atomicMax(&acc->prec_steps, (unsigned int)steps);
    }
}

// FloatEncoding::Encode's decision (float_encoding.cu:29-43) from the stats pass
template <int ES>
__device__ __forceinline__ int f2i_decide(const BItem &it, const uint8_t *col, uint64_t n, bool &transform)
{
    const StatsAcc *acc = (const StatsAcc *)it.scratch;
    const Order o = (Order)it.order;
    const unsigned steps = acc->prec_steps > 10 ? 10 : acc->prec_steps;
    int p = d_precision_of((int)steps);
    transform = false;
    if (p < 10 && n) {
        uint64_t mnb = 0, mxb = 0;
        if (!acc_minmax(&acc->mm, ES, o, mnb, mxb)) mnb = mxb = ld_elem<ES>(col, 0);
        long long sc = 1;
        for (int i = 0; i < p; i++) sc *= 10;
        bool ok;
        if (o == ORD_F32) {
            const float a = __fmul_rn(__uint_as_float((uint32_t)mnb), (float)sc);
            const float b = __fmul_rn(__uint_as_float((uint32_t)mxb), (float)sc);
            ok = a > -2147483648.0f && b < 2147483648.0f;
        } else if (o == ORD_F64) {
            const double a = __dmul_rn(__longlong_as_double((long long)mnb), (double)sc);
            const double b = __dmul_rn(__longlong_as_double((long long)mxb), (double)sc);
            ok = a > -2147483648.0 && b < 2147483647.0;
        } else {
            ok = sext(mnb, ES) * sc > (long long)INT32_MIN && sext(mxb, ES) * sc < (long long)INT32_MAX;
        }
        if (ok) transform = true;
        else p = 10;
    }
    return p;
}

// the raw branch (p = 10): the bytes of the tile's elements that fall in the stream's whole 32-bit
// words (`words`), block-striped; whole words when the input is 4-byte aligned (the output, a node
// stream, always is), else bytes
template <int ES>
__device__ __forceinline__ void f2i_copy_words(uint8_t *out, const uint8_t *in, uint32_t tile, uint64_t words)
{
    constexpr uint64_t B = (uint64_t)kBTile * ES;  // bytes of one tile
    const uint64_t b0 = (uint64_t)tile * B, b1 = b0 + B < 4 * words ? b0 + B : 4 * words;
    if (((uintptr_t)in & 3) == 0) {
        for (uint64_t w = b0 / 4 + threadIdx.x; w < b1 / 4; w += kBThreads)
            ((uint32_t *)out)[w] = ldg((const uint32_t *)in + w);
    } else {
        for (uint64_t b = b0 + threadIdx.x; b < b1; b += kBThreads) out[b] = ldg(in + b);
    }
}

template <int ES>
__device__ void p_f2i_enc(const BItem &it, uint32_t tile, StreamDesc *S)
{
    const double *p10 = pow10_table();
    const StreamDesc in = S[it.in[0]];
    const uint64_t n = in.len / ES;
    bool transform;
    const int p = f2i_decide<ES>(it, in.ptr, n, transform);
    if (tile == 0 && threadIdx.x == 0) {
        if (n) {
            *(int32_t *)S[it.out[0]].ptr = p;
            S[it.out[0]].len = 4;
            S[it.out[1]].len = transform ? 4 * n : (n * ES) / 4 * 4;
        } else {
            S[it.out[0]].len = 0;
            S[it.out[1]].len = 0;
        }
    }
    // block-striped: the k-th access of a warp covers 32 consecutive elements (or words)
    const uint64_t t0 = (uint64_t)tile * kBTile;
    if (t0 >= n) return;
    uint8_t *out = S[it.out[1]].ptr;
    if (transform) {
        const Order o = (Order)it.order;
        const uint64_t wm = ES == 8 ? ~0ull : ((1ull << (8 * ES)) - 1);
        bool bad = false;
        for (int j = 0; j < (int)kBVPT; j++) {
            const uint64_t i = t0 + (uint64_t)j * kBThreads + threadIdx.x;
            if (i >= n) break;
            const uint64_t u = ld_elem<ES>(in.ptr, i);
            const int k = (int)(long long)__double2ll_rn(__dmul_rn(as_double<ES>(u, o), p10[p]));
            ((int32_t *)out)[i] = k;
            if (((f2i_dec_one<ES>(k, p, o, p10) ^ u) & wm) != 0) bad = true;
        }
        if (bad) atomicExch((unsigned int *)(it.scratch + 64), 1u);
    } else {
        f2i_copy_words<ES>(out, in.ptr, tile, (n * ES) / 4);
    }
}

// the lossless check failed: the raw p = 10 branch
template <int ES>
__device__ void p_f2i_raw(const BItem &it, uint32_t tile, StreamDesc *S)
{
    if (*(volatile unsigned int *)(it.scratch + 64) == 0) return;
    const StreamDesc in = S[it.in[0]];
    const uint64_t n = in.len / ES;
    const uint64_t bytes = (n * ES) / 4 * 4;
    if (tile == 0 && threadIdx.x == 0) {
        *(int32_t *)S[it.out[0]].ptr = 10;
        S[it.out[1]].len = bytes;
    }
    f2i_copy_words<ES>(S[it.out[1]].ptr, in.ptr, tile, bytes / 4);
}

// ------------------------------------------------------------------------------- GFC
// node scratch of GFC: p[0] look-back, p[1] chunk sizes (int32), p[2] inclusive ends (u64), p[3] layout

// A double chunk is built in a 1 KB ring of the warp's shared memory and stored in 512-byte blocks,
// 16 bytes a lane (its payload bytes, up to 8 a lane, would otherwise be that many partial global
// stores); a float chunk, at most 4 bytes a lane, is stored directly.  Positions count bytes from
// the 16-byte aligned address at or below the chunk's start; only the bytes in [lo, hi) are stored.
constexpr uint32_t kGfcStage = 1024;

__device__ __forceinline__ void gfc_flush(uint8_t *al, const uint8_t *ring, uint32_t b, uint32_t lo, uint32_t hi,
                                          int lane)
{
    const uint32_t p = b + 16 * (uint32_t)lane;
    if (p >= lo && p + 16 <= hi) {
        *(uint4 *)(al + p) = *(const uint4 *)(ring + (p & (kGfcStage - 1)));
    } else {
        for (uint32_t k = 0; k < 16; k++)
            if (p + k >= lo && p + k < hi) al[p + k] = ring[(p + k) & (kGfcStage - 1)];
    }
}

template <bool DBL>
__device__ void p_gfc_compress(const BItem &it, uint32_t tile, StreamDesc *S, uint8_t *sm)
{
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<DBL ? 8 : 4>(it, in);
    const uint64_t n = vc.n;
    const DGfc g = d_gfc_geom(DBL, n, 0, 0);
    if (tile == 0 && threadIdx.x == 0) {
        if (n) {
            int32_t *m = (int32_t *)S[it.out[0]].ptr;
            m[0] = g.blocks;
            m[1] = g.wpb;
            m[2] = (int32_t)n;
            S[it.out[0]].len = 12;
            S[it.out[1]].len = 4 * (uint64_t)g.warps;
        } else {
            S[it.out[0]].len = 0;
            S[it.out[1]].len = 0;
            S[it.out[2]].len = 0;
        }
    }
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)tile * kBGfcChunks + (threadIdx.x >> 5);
    if (w >= g.warps) return;
    uint8_t *layout = it.scratch + it.p[3];
    int32_t *sizes = (int32_t *)(it.scratch + it.p[1]);
    int32_t *ends = (int32_t *)S[it.out[1]].ptr;
    const uint64_t cb = d_gfc_begin(g, w), ce = d_gfc_cut(g, w);
    const uint64_t start = d_gfc_start(g, w);
    uint64_t last = 0;
    uint8_t *ring = sm + (threadIdx.x >> 5) * kGfcStage;
    const uint32_t mis = (uint32_t)((uintptr_t)(layout + start) & 15);
    uint8_t *al = layout + start - mis;
    uint32_t fr = mis, flushed = 0;  // positions: the next subchunk's header, the bytes stored
    // values of the next 4 subchunks are in flight while one is encoded
    uint64_t xb[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint64_t i = cb + 32 * q + lane;
        xb[q] = cb + 32 * q < ce && i < n ? view_elem<DBL ? 8 : 4>(it, vc, in.ptr, i) : 0;
    }
    for (uint64_t s0 = cb; s0 < ce; s0 += 128)
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint64_t s = s0 + 32 * q;
        if (s >= ce) break;
        const uint64_t x = xb[q];
        {
            const uint64_t i = s + 128 + lane;
            xb[q] = s + 128 < ce && i < n ? view_elem<DBL ? 8 : 4>(it, vc, in.ptr, i) : 0;
        }
        uint64_t diff;
        uint32_t sign, mb, code;
        if (DBL) {
            diff = x - last;
            sign = (uint32_t)((diff >> 60) & 8);
            if (sign) diff = 0ull - diff;
            const uint32_t lz = (uint32_t)__clzll((long long)diff) >> 3;
            mb = lz == 6 ? 3 : 8 - lz;
            code = mb >= 3 ? mb - 1 : mb;
        } else {
            uint32_t d = (uint32_t)x - (uint32_t)last;
            sign = (d >> 28) & 8;
            if (sign) d = 0u - d;
            mb = 4 - ((uint32_t)__clz((int)d) >> 3);
            code = mb;
            diff = d;
        }
        const uint32_t nib = sign | code;
        uint32_t incl = mb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t prev_nib = __shfl_up_sync(0xffffffffu, nib, 1);
        const uint32_t pl = fr + 16 + (incl - mb);
        if constexpr (DBL) {
            if (lane & 1) ring[(fr + (lane >> 1)) & (kGfcStage - 1)] = (uint8_t)(prev_nib | (nib << 4));
            for (uint32_t b = 0; b < mb; b++) ring[(pl + b) & (kGfcStage - 1)] = (uint8_t)(diff >> (8 * b));
        } else {
            if (lane & 1) al[fr + (lane >> 1)] = (uint8_t)(prev_nib | (nib << 4));
            for (uint32_t b = 0; b < mb; b++) al[pl + b] = (uint8_t)(diff >> (8 * b));
        }
        fr += 16 + total;  // at most 272 bytes a subchunk: the ring holds [flushed, fr) below 784 bytes
        if (s == cb) last = __shfl_sync(0xffffffffu, x, 31);
        if constexpr (DBL) {
            __syncwarp();
            if (fr - flushed >= 512) {
                gfc_flush(al, ring, flushed, mis, 0xffffffffu, lane);
                flushed += 512;
                __syncwarp();
            }
        }
    }
    if (DBL && flushed < fr) gfc_flush(al, ring, flushed, mis, fr, lane);
    if (lane == 31) {
        ends[w] = (int32_t)(start + fr - mis);
        sizes[w] = (int32_t)(fr - mis);
    }
}

// one warp copies n bytes between any addresses: head bytes up to a 4-byte aligned destination,
// then whole words funnel-shifted out of aligned source words, then the tail.  Eight words a lane
// are loaded before any is stored, so the loads are in flight together.
__device__ __forceinline__ void warp_copy(uint8_t *dst, const uint8_t *src, uint64_t n, int lane)
{
    const uint64_t head = (4 - ((uintptr_t)dst & 3)) & 3;
    const uint64_t h = head < n ? head : n;
    if ((uint64_t)lane < h) dst[lane] = src[lane];
    if (n <= h) return;
    uint32_t *d = (uint32_t *)(dst + h);
    const uint8_t *sp = src + h;
    const uint64_t words = (n - h) / 4;
    const uint32_t sh = 8 * (uint32_t)((uintptr_t)sp & 3);
    const uint32_t *sw = (const uint32_t *)((uintptr_t)sp & ~(uintptr_t)3);
    constexpr int U = 8;
    uint64_t k = lane;
    if (sh == 0) {
        for (; k + (U - 1) * 32 < words; k += U * 32) {
            uint32_t r[U];
#pragma unroll
            for (int u = 0; u < U; u++) r[u] = ldg(sw + k + u * 32);
#pragma unroll
            for (int u = 0; u < U; u++) d[k + u * 32] = r[u];
        }
        for (; k < words; k += 32) d[k] = ldg(sw + k);
    } else {
        for (; k + (U - 1) * 32 < words; k += U * 32) {
            uint32_t r[U], q[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                r[u] = ldg(sw + k + u * 32);
                q[u] = ldg(sw + k + u * 32 + 1);
            }
#pragma unroll
            for (int u = 0; u < U; u++) d[k + u * 32] = __funnelshift_r(r[u], q[u], sh);
        }
        for (; k < words; k += 32) d[k] = __funnelshift_r(ldg(sw + k), ldg(sw + k + 1), sh);
    }
    const uint64_t tail = (n - h) - 4 * words;
    if ((uint64_t)lane < tail) ((uint8_t *)d)[4 * words + lane] = sp[4 * words + lane];
}

template <bool DBL>
__device__ void p_gfc_compact(const BItem &it, uint32_t tile, StreamDesc *S)
{
    int nd = 0;
    for (int k = 0; k < kMaxViewOps; k++) nd += it.vop[k] == V_DELTA;
    const uint64_t n_src = S[it.in[0]].len / (DBL ? 8 : 4);
    const uint64_t n = n_src > (uint64_t)nd ? n_src - nd : 0;
    const DGfc g = d_gfc_geom(DBL, n, 0, 0);
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)tile * kBGfcChunks + (threadIdx.x >> 5);
    if (w >= g.warps) return;
    const int32_t *sizes = (const int32_t *)(it.scratch + it.p[1]);
    const unsigned long long *incl = (const unsigned long long *)(it.scratch + it.p[2]);
    const uint8_t *layout = it.scratch + it.p[3];
    const uint64_t size = (uint64_t)(uint32_t)sizes[w];
    const uint64_t dst0 = incl[w] - size;
    const uint8_t *src = layout + d_gfc_start(g, w);
    uint8_t *out = S[it.out[2]].ptr;
    warp_copy(out + dst0, src, size, lane);
    if (w == g.warps - 1 && lane == 0) S[it.out[2]].len = incl[w];
}

// ------------------------------------------------------------------------------- view nodes
// Metadata of a delta / scale node whose output is only read through its child's view: delta's
// first value, scale's minimum (scale_min of its min / max).  One thread per item.
template <int ES>
__device__ void p_vmeta(const BItem &it, StreamDesc *S)
{
    if (threadIdx.x != 0) return;
    const StreamDesc in = S[it.in[0]];
    const ViewCtx vc = view_ctx<ES>(it, in);
    StreamDesc &m = S[it.out[0]];
    if (vc.n == 0) {
        m.len = 0;
        return;
    }
    uint64_t v;
    if (it.mode == GTSC_DELTA) {
        v = view_elem<ES>(it, vc, in.ptr, 0);
    } else {
        uint64_t mnb = 0, mxb = 0;
        acc_minmax((const MinMaxAcc *)it.scratch, ES, ORD_INT, mnb, mxb);
        v = scale_min(mnb, mxb, ES);
    }
    st_elem<ES>(m.ptr, 0, v);
    m.len = ES;
}

// ------------------------------------------------------------------------------- dispatch
constexpr size_t stage_smem(int op)
{
    return op == B_AFL_PACK ? 8 * (kBTile + kBTile / 16 + 8)
         : op == B_HIST     ? kCandSmem
         : op == B_HIST_SAMPLE ? kSampleSmem
         : op == B_HIST_FULL ? kBHistBytesPersist
         : op == B_SPLIT    ? kSplitCodes * (kBThreads / 32)  // a dictionary's codes, a byte each
         : op == B_RLE_HEADS ? kXchgBlockBytes
         : op == B_GFC_COMPRESS ? kGfcStage * (kBThreads / 32)
                            : 16;
}

// Tiles of an item that do work in a pass (the grid is sized for worst-case capacities; the real
// stream lengths are only known on the device).  Tile 0 of a pass that writes metadata always
// runs.  Passes not listed run every reserved tile.
template <int OP>
__device__ __forceinline__ uint32_t stage_extent(const BItem &it, const StreamDesc *S)
{
    auto cdiv = [](uint64_t a, uint64_t b) { return (a + b - 1) / b; };
    auto view_n = [&]() {
        int nd = 0;
        for (int k = 0; k < kMaxViewOps; k++) nd += it.vop[k] == V_DELTA;
        const uint64_t n_src = S[it.in[0]].len / it.es;
        return n_src > (uint64_t)nd ? n_src - nd : 0;
    };
    uint64_t e = it.tiles;
    if constexpr (OP == B_MINMAX) e = cdiv(view_n(), it.p[0]);  // the tuned min/max tile
    else if constexpr (OP == B_DELTA_ENC) {
        const uint64_t n = view_n();
        e = cdiv(n ? n - 1 : 0, kBTile);
        if (e == 0) e = 1;
    } else if constexpr (OP == B_SCALE_SUB || OP == B_AFL_PACK || OP == B_F2I_ENC || OP == B_F2I_RAW) {
        e = cdiv(view_n(), kBTile);
        if (e == 0) e = 1;
    } else if constexpr (OP == B_SPLIT_COUNT || OP == B_SPLIT) {
        e = cdiv(view_n(), kBSplitTile);
        if (e == 0) e = 1;
    } else if constexpr (OP == B_F2I_STATS) e = cdiv(view_n(), kBTile);
    else if constexpr (OP == B_RLE_LENGTHS) e = cdiv(S[it.out[1]].len / 4, kBTile);
    else if constexpr (OP == B_GFC_COMPRESS || OP == B_GFC_COMPACT) {
        const DGfc g = d_gfc_geom(it.es == 8, view_n(), 0, 0);
        e = cdiv((uint64_t)g.warps, kBGfcChunks);
        if (OP == B_GFC_COMPRESS && e == 0) e = 1;
    }
    return (uint32_t)(e < it.tiles ? e : it.tiles);
}

// `step`, `end`: passes that loop over an item's tiles themselves (stage_item_loop) run tile, tile + step,
// ... below end; the others run `tile`
template <int OP>
__device__ __forceinline__ void run_stage(const BItem &it, uint32_t tile, uint32_t step, uint32_t end, StreamDesc *S,
                                          uint32_t *status, unsigned char *smem);

// passes that set up (stream pointers, view, widths, classes: a chain of dependent loads) once for all of
// a block's tiles of an item
constexpr bool stage_item_loop(int op) { return op == B_AFL_PACK || op == B_SPLIT_COUNT || op == B_SPLIT; }

// passes whose tiles all do the same streaming work run persistent grids (see stage_grid)
constexpr bool stage_persistent(int op)
{
    return op == B_MINMAX || op == B_DELTA_ENC || op == B_SCALE_SUB || op == B_AFL_PACK || op == B_F2I_STATS ||
           op == B_F2I_ENC || op == B_F2I_RAW || op == B_RLE_LENGTHS || op == B_SPLIT_COUNT || op == B_SPLIT;
}

// One launch of a pass over every item.  Look-back passes take one tile per block in claim order;
// the others are persistent: an occupancy-sized grid strides over the tiles, skipping from a tile
// past its item's real extent straight to its first tile of the next item.
// resident blocks per SM the compiler keeps registers for (measured per pass on the mixed workload)
constexpr int stage_min_blocks(int op)
{
    return op == B_AFL_PACK || op == B_GFC_COMPRESS || op == B_TOPK ? 4 : 5;
}

template <int OP>
__global__ void __launch_bounds__(kBThreads, stage_min_blocks(OP))
k_bstage(const BItem *items, const uint32_t *item_of, StreamDesc *S, uint32_t *counter, uint32_t *status,
         uint32_t total_tiles)
{
    constexpr bool DYN = OP == B_RLE_HEADS || OP == B_GFC_SCAN;
    __shared__ __align__(16) unsigned char smem[stage_smem(OP)];
    if constexpr (!stage_persistent(OP)) {
        uint32_t tile;
        const BItem &it = locate<DYN>(items, item_of, counter, tile);
        if (tile >= it.tiles) return;
        run_stage<OP>(it, tile, 1, tile + 1, S, status, smem);
    } else {
        uint32_t t = blockIdx.x;
        uint32_t cur = 0xffffffffu;  // the item in the shared descriptor
        while (t < total_tiles) {
            const uint32_t k = item_of[t];
            if (k != cur) {
                __syncthreads();  // nobody reads the previous descriptor any more
                shared_item(items, k);
                cur = k;
            }
            const BItem &it = shared_item_ref();
            const uint32_t tile = t - (uint32_t)it.tile_base;
            const uint32_t extent = stage_extent<OP>(it, S);
            if (tile >= extent) {
                const uint64_t next = it.tile_base + it.tiles;  // the next item's first tile
                if (next >= total_tiles) break;
                t = (uint32_t)(next + (blockIdx.x + gridDim.x - next % gridDim.x) % gridDim.x);
                continue;
            }
            run_stage<OP>(it, tile, gridDim.x, extent, S, status, smem);
            if constexpr (stage_item_loop(OP)) t += (extent - 1 - tile) / gridDim.x * gridDim.x;
            __syncthreads();  // the next tile reuses the shared memory
            t += gridDim.x;
        }
    }
}

template <int OP>
__device__ __forceinline__ void run_stage(const BItem &it, uint32_t tile, uint32_t step, uint32_t end, StreamDesc *S,
                                          uint32_t *status, unsigned char *smem)
{
#define GTSC_ES_SWITCH(CALL)                       \
    switch (it.es) {                               \
    case 1: { constexpr int E = 1; CALL; } break;  \
    case 2: { constexpr int E = 2; CALL; } break;  \
    case 4: { constexpr int E = 4; CALL; } break;  \
    default: { constexpr int E = 8; CALL; } break; \
    }
    if constexpr (OP == B_MINMAX) { GTSC_ES_SWITCH(p_minmax<E>(it, tile, S)) }
    else if constexpr (OP == B_DELTA_ENC) { GTSC_ES_SWITCH(p_delta_enc<E>(it, tile, S)) }
    else if constexpr (OP == B_SCALE_SUB) { GTSC_ES_SWITCH(p_scale_sub<E>(it, tile, S)) }
    else if constexpr (OP == B_AFL_PACK) { GTSC_ES_SWITCH(p_afl_pack<E>(it, tile, step, end, S, smem)) }
    else if constexpr (OP == B_HIST_SAMPLE) { GTSC_ES_SWITCH(p_hist_sample<E>(it, S, smem)) }
    else if constexpr (OP == B_HIST) { GTSC_ES_SWITCH(p_hist_count<E>(it, tile, S, smem)) }
    else if constexpr (OP == B_TOPK) { GTSC_ES_SWITCH(p_cand_top<E>(it, S)) }
    else if constexpr (OP == B_HIST_FULL) {
        if (*CandArea(it).flag) { GTSC_ES_SWITCH(p_hist<E>(it, tile, S, status, smem)) }
    } else if constexpr (OP == B_TOPK_FULL) {
        if (*CandArea(it).flag) { GTSC_ES_SWITCH(topk_blocks<E>(it, tile, it.tiles, S)) }
    }
    else if constexpr (OP == B_VMETA) { GTSC_ES_SWITCH(p_vmeta<E>(it, S)) }
    else if constexpr (OP == B_SPLIT_COUNT) { p_split_count(it, tile, step, end, S); }
    else if constexpr (OP == B_SPLIT) { GTSC_ES_SWITCH(p_split<E>(it, tile, step, end, S, smem)) }
    else if constexpr (OP == B_RLE_HEADS) { GTSC_ES_SWITCH(p_rle_heads<E>(it, tile, S, smem)) }
    else if constexpr (OP == B_RLE_LENGTHS) { p_rle_lengths(it, tile, S); }
    else if constexpr (OP == B_F2I_STATS) { GTSC_ES_SWITCH(p_f2i_stats<E>(it, tile, S)) }
    else if constexpr (OP == B_F2I_ENC) { GTSC_ES_SWITCH(p_f2i_enc<E>(it, tile, S)) }
    else if constexpr (OP == B_F2I_RAW) { GTSC_ES_SWITCH(p_f2i_raw<E>(it, tile, S)) }
    else if constexpr (OP == B_GFC_COMPRESS) {
        if (it.es == 8) p_gfc_compress<true>(it, tile, S, smem);
        else p_gfc_compress<false>(it, tile, S, smem);
    } else if constexpr (OP == B_GFC_SCAN) {
        p_gfc_scan(it, tile, S, it.es == 8, it.mode != 0);
    } else if constexpr (OP == B_GFC_COMPACT) {
        if (it.es == 8) p_gfc_compact<true>(it, tile, S);
        else p_gfc_compact<false>(it, tile, S);
    }
#undef GTSC_ES_SWITCH
}

#ifdef GTSC_PERSISTENT_TU
// ------------------------------------------------------------------------------- persistent step
constexpr size_t persist_smem_c()
{
    size_t m = 16;
    for (int op = 0; op < B_NUM_OPS; op++) m = stage_smem(op) > m ? stage_smem(op) : m;
    return m;
}

// tiles of an item that do work: the streaming passes skip tiles past the real length, as their
// stage launches do; every other pass runs all its tiles
__device__ __forceinline__ uint32_t persist_extent_c(int op, const BItem &it, const StreamDesc *S)
{
    switch (op) {
    case B_MINMAX: return stage_extent<B_MINMAX>(it, S);
    case B_DELTA_ENC: return stage_extent<B_DELTA_ENC>(it, S);
    case B_SCALE_SUB: return stage_extent<B_SCALE_SUB>(it, S);
    case B_AFL_PACK: return stage_extent<B_AFL_PACK>(it, S);
    case B_F2I_STATS: return stage_extent<B_F2I_STATS>(it, S);
    case B_F2I_ENC: return stage_extent<B_F2I_ENC>(it, S);
    case B_F2I_RAW: return stage_extent<B_F2I_RAW>(it, S);
    case B_RLE_LENGTHS: return stage_extent<B_RLE_LENGTHS>(it, S);
    case B_SPLIT_COUNT: return stage_extent<B_SPLIT_COUNT>(it, S);
    case B_SPLIT: return stage_extent<B_SPLIT>(it, S);
    default: return it.tiles;
    }
}

// The whole compress step in one launch: every pass kind behind one switch, tiles pulled from the
// queue of batch.hpp (PUnit).
__global__ void __launch_bounds__(kBThreads, 4) k_bpersist_c(PersistArgs a)
{
    __shared__ __align__(16) unsigned char smem[persist_smem_c()];
    persist_loop(
        a, [](int op, const BItem &it, const StreamDesc *S) { return persist_extent_c(op, it, S); },
        [&](int op, const BItem &it, uint32_t tile) {
        switch (op) {
#define GTSC_RUN(OPC) case OPC: run_stage<OPC>(it, tile, 1, tile + 1, a.S, a.status, smem); break;
            GTSC_RUN(B_MINMAX)
            GTSC_RUN(B_DELTA_ENC)
            GTSC_RUN(B_SCALE_SUB)
            GTSC_RUN(B_AFL_PACK)
            GTSC_RUN(B_HIST_SAMPLE)
            GTSC_RUN(B_HIST)
            GTSC_RUN(B_TOPK)
            GTSC_RUN(B_HIST_FULL)
            GTSC_RUN(B_TOPK_FULL)
        case B_SPLIT_COUNT: case B_SPLIT: case B_SPLIT_SHORT: {  // short: the column's tiles by this block
            const uint32_t end = op == B_SPLIT_SHORT ? short_split_tiles(it, a.S) : tile + 1;
            if (op != B_SPLIT) run_stage<B_SPLIT_COUNT>(it, tile, 1, end, a.S, a.status, smem);
            if (op == B_SPLIT_SHORT) __syncthreads();
            if (op != B_SPLIT_COUNT) run_stage<B_SPLIT>(it, tile, 1, end, a.S, a.status, smem);
            break;
        }
            GTSC_RUN(B_RLE_HEADS)
            GTSC_RUN(B_RLE_LENGTHS)
            GTSC_RUN(B_F2I_STATS)
            GTSC_RUN(B_F2I_ENC)
            GTSC_RUN(B_F2I_RAW)
            GTSC_RUN(B_GFC_COMPRESS)
            GTSC_RUN(B_GFC_SCAN)
            GTSC_RUN(B_GFC_COMPACT)
            GTSC_RUN(B_VMETA)
#undef GTSC_RUN
        default: set_status(a.status, GTSC_ERR_ARG); break;
        }
    });
}

#endif  // GTSC_PERSISTENT_TU

}  // namespace

#ifdef GTSC_PERSISTENT_TU
void launch_batch_persistent_c(const PersistArgs &a, cudaStream_t s)
{
    if (a.total == 0) return;
    int per_sm = 0;
    GTSC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bpersist_c, kBThreads, 0));
    const uint64_t grid = std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * (uint64_t)sm_count(),
                                             (uint64_t)a.total);
    k_bpersist_c<<<(unsigned)grid, kBThreads, 0, s>>>(a);
    GTSC_CUDA(cudaGetLastError());
}
#else

void launch_batch_decode_stage(int op, const BItem *d_items, const uint32_t *d_item_of, int n_items,
                               uint64_t total_tiles, StreamDesc *d_streams, uint32_t *d_counter, uint32_t *d_status,
                               cudaStream_t s);

// Grid of a stage launch: as many blocks as can be resident at once for the streaming passes (the
// kernel strides over the tiles), else one block per tile (look-back passes claim each tile once).
template <class K>
unsigned stage_grid(K kernel, int op, uint64_t total_tiles)
{
    // persistent where every tile does the same streaming work; one block per tile where tiles differ
    // a lot (GFC chunks, histograms, top-k) and independent blocks balance better
    if (!stage_persistent(op)) return (unsigned)total_tiles;
    int per_sm = 0;
    GTSC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBThreads, 0));
    const uint64_t resident = (uint64_t)std::max(per_sm, 1) * (uint64_t)sm_count();
    return (unsigned)std::min<uint64_t>(total_tiles, resident);
}

void launch_batch_stage(int op, const BItem *d_items, const uint32_t *d_item_of, int n_items, uint64_t total_tiles,
                        StreamDesc *d_streams, uint32_t *d_counter, uint32_t *d_status, cudaStream_t s)
{
    if (n_items == 0 || total_tiles == 0) return;
    if (total_tiles > 0x7fffffffull) fail(GTSC_ERR_CAPACITY, "batch: too many tiles in one stage");
    switch (op) {
#define GTSC_STAGE(OPC)                                                                                              \
    case OPC: {                                                                                                      \
        const unsigned g = stage_grid(k_bstage<OPC>, OPC, total_tiles);                                              \
        k_bstage<OPC><<<g, kBThreads, 0, s>>>(d_items, d_item_of, d_streams, d_counter, d_status, (uint32_t)total_tiles); \
        break;                                                                                                       \
    }
        GTSC_STAGE(B_MINMAX)
        GTSC_STAGE(B_DELTA_ENC)
        GTSC_STAGE(B_SCALE_SUB)
        GTSC_STAGE(B_AFL_PACK)
        GTSC_STAGE(B_HIST_SAMPLE)
    case B_HIST: {
        int per_sm = 0;
        GTSC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bcount, kBThreads, 0));
        const uint64_t resident = (uint64_t)std::max(per_sm, 1) * (uint64_t)sm_count();
        k_bcount<<<(unsigned)std::min<uint64_t>(total_tiles, resident), kBThreads, 0, s>>>(d_items, d_item_of, d_streams,
                                                                                        (uint32_t)total_tiles);
        break;
    }
    case B_HIST_FULL: {
        GTSC_CUDA(cudaFuncSetAttribute(k_bhist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBHistBytes));
        int per_sm = 0;
        GTSC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bhist, (int)kBHistThreads, kBHistBytes));
        const uint64_t resident = (uint64_t)std::max(per_sm, 1) * (uint64_t)sm_count();
        k_bhist<<<(unsigned)std::min<uint64_t>(total_tiles, resident), kBHistThreads, kBHistBytes, s>>>(
            d_items, n_items, d_streams, d_status);
        break;
    }
    case B_TOPK_FULL:
        k_btopk<<<(unsigned)std::min<uint64_t>(total_tiles, 4 * (uint64_t)sm_count()), kBThreads, 0, s>>>(d_items, n_items,
                                                                                                        d_streams);
        break;
        GTSC_STAGE(B_TOPK)
        GTSC_STAGE(B_SPLIT_COUNT)
        GTSC_STAGE(B_SPLIT)
    case B_SPLIT_SHORT:
        k_bsplit_short<<<(unsigned)n_items * kBShortTiles, kBThreads, 0, s>>>(d_items, d_streams);
        break;
        GTSC_STAGE(B_RLE_HEADS)
        GTSC_STAGE(B_RLE_LENGTHS)
        GTSC_STAGE(B_F2I_STATS)
        GTSC_STAGE(B_F2I_ENC)
        GTSC_STAGE(B_F2I_RAW)
        GTSC_STAGE(B_GFC_COMPRESS)
        GTSC_STAGE(B_GFC_SCAN)
        GTSC_STAGE(B_GFC_COMPACT)
        GTSC_STAGE(B_VMETA)
#undef GTSC_STAGE
    default:
        launch_batch_decode_stage(op, d_items, d_item_of, n_items, total_tiles, d_streams, d_counter, d_status, s);
        return;
    }
    GTSC_CUDA(cudaGetLastError());
}

#endif  // GTSC_PERSISTENT_TU

}  // namespace gtsc
