// zfp_device.cuh -- fixed-rate ZFP float32 3-D block codec, device side.
//
// Decoding follows shaders/zfp_decompress.comp:195-384 value for value: a
// 1-bit "block is nonzero" flag, an 8-bit biased common exponent, the embedded
// bit-plane code over 32 planes with group tests (decode_ints, :265-294),
// negabinary to two's complement (:260-263), the ZFP_PERM3D reorder (:101-185),
// the separable inverse lift along z, y, x (:296-354) and the scale by
// 2^(emax-30) (:378-382).  Bit offsets are 64-bit (the reference multiplies
// block_index*max_bits in 32 bits, :199, which wraps past 2^32 bits).
//
// The GB300 decoder stages each block's words in shared memory, parses them
// one group test per loop step through a 64-bit window with both outcomes
// computed by selects (lanes stay converged), and turns the bit planes into
// coefficients with three delta-swap stages over 8-plane chunks (see "Staged
// decoder").
#pragma once

#include <stdint.h>

#include "zfp_perm.inc"

namespace bcmc {

constexpr uint32_t kZfpMaxBitsLimit = 64u * 32u;  // rate <= 32 bits/value

// inverse_lift (zfp_decompress.comp:296-332).  WGSL integer arithmetic wraps,
// and streams that are not encoder output (or corrupt ones) do overflow here,
// so adds, subtracts and left shifts run in uint32 (C++ signed overflow would
// be undefined and the compiler may assume it away); only >> is on int32
// (arithmetic shift, as on the reference's int).
__device__ __forceinline__ void zfp_inv_lift(int32_t& x, int32_t& y, int32_t& z, int32_t& w)
{
    uint32_t ux = (uint32_t)x, uy = (uint32_t)y, uz = (uint32_t)z, uw = (uint32_t)w;
    uy += (uint32_t)((int32_t)uw >> 1);
    uw -= (uint32_t)((int32_t)uy >> 1);
    uy += uw;
    uw <<= 1;
    uw -= uy;
    uz += ux;
    ux <<= 1;
    ux -= uz;
    uy += uz;
    uz <<= 1;
    uz -= uy;
    uw += ux;
    ux <<= 1;
    ux -= uw;
    x = (int32_t)ux;
    y = (int32_t)uy;
    z = (int32_t)uz;
    w = (int32_t)uw;
}

__device__ __forceinline__ void zfp_inverse_transform(int32_t* v)
{
#pragma unroll
    for (int i = 0; i < 16; ++i) zfp_inv_lift(v[i], v[i + 16], v[i + 32], v[i + 48]);  // z
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const int b = 16 * z + x;
            zfp_inv_lift(v[b], v[b + 4], v[b + 8], v[b + 12]);  // y
        }
#pragma unroll
    for (int i = 0; i < 16; ++i) zfp_inv_lift(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);  // x
}

// 2^(emax-30) exactly (ldexp(1.f, emax-30), zfp_decompress.comp:378)
__device__ __forceinline__ float zfp_inv_weight(int32_t emax)
{
    const int32_t e = emax - 30;
    if (e >= -126 && e <= 127) return __int_as_float((e + 127) << 23);
    return ldexpf(1.0f, e);
}

// ---------------------------------------------------------------------------
// Staged decoder: the block's compressed words are first copied into shared
// memory (coalesced loads by the CTA for runs of consecutive blocks, or one
// block per thread), then parsed there.
//
// Parse (zfp_parse_planes): one loop step per group-test read.  A step loads
// the 64-bit window after the test (three words, two funnel shifts) and
// computes both outcomes with selects: a 1 (the run of zeros after it is the
// window's trailing zeros, clamped by the bit budget and by coefficient 63,
// decode_ints' two limits) or a 0, which ends the plane and takes the next
// plane's raw bits from the same window.  Only the plane store and the loop
// exit branch, so a warp's lanes stay converged although their blocks take
// different numbers of steps.  A block's leading empty planes (single 0 group
// tests while nothing is significant) are skipped at once.  On the 512^3
// spectral field at rate 2 (about 19 steps per block) this took the full
// decode from 0.390 ms (8-bit group-test table steps, a bit-by-bit tail near
// the limits, branches per outcome) to 0.257 ms; the branching form of the
// same step measured 0.333 ms.  With trailing zeros and masks by one instruction
// each, whole-plane stores, the multiply-add deposit and one window a step it
// takes 0.226 ms (220 -> 203 M warp instructions).
//
// Deposit (zfp_planes_deposit): the plane masks go to a per-thread row of
// shared memory; each 8-plane chunk is read back as 8 rows of 64 bits and all
// eight 8x8 byte columns are transposed at once by three delta-swap stages,
// after which byte g of row k is coefficient 8g + k's digits in those planes.
// ---------------------------------------------------------------------------

// PTX shifts clamp the count: a shift by 32 or more gives 0 (the host
// branch states the same for host builds of this header)
__device__ __forceinline__ uint32_t zfp_shl(uint32_t x, uint32_t s)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(s));
    return r;
#else
    return s >= 32u ? 0u : x << s;
#endif
}
__device__ __forceinline__ uint32_t zfp_shr(uint32_t x, uint32_t s)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("shr.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(s));
    return r;
#else
    return s >= 32u ? 0u : x >> s;
#endif
}

// the low word of hi:lo shifted right by s, up to 32
__device__ __forceinline__ uint32_t zfp_window(uint32_t lo, uint32_t hi, uint32_t s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_rc(lo, hi, s);
#else
    return s >= 32u ? hi : __funnelshift_r(lo, hi, s);
#endif
}
// the low m bits, all from 32 on
__device__ __forceinline__ uint32_t zfp_low(uint32_t m)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(r) : "r"(m));
    return r;
#else
    return m >= 32u ? 0xffffffffu : (1u << m) - 1u;
#endif
}
// the zeros below the lowest 1, all ones (a large number) for 0
__device__ __forceinline__ uint32_t zfp_ctz(uint32_t x)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("bfind.shiftamt.u32 %0, %1;" : "=r"(r) : "r"(__brev(x)));
    return r;
#else
    return x ? (uint32_t)__builtin_ctz(x) : 0xffffffffu;
#endif
}

__device__ __forceinline__ uint32_t zfp_clz(uint32_t x)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__clz((int)x);
#else
    return x ? (uint32_t)__builtin_clz(x) : 32u;
#endif
}

// decode_ints' bit planes (zfp_decompress.comp:265-294) as masks.  `w`: the
// block's words (LSB first), readable for three words past the block; `pos`:
// the first bit after the header.  Plane r (bit 31 - r of the coefficients)
// goes to pl[2(r - r0)] (coefficients 0..31) and pl[2(r - r0) + 1] (32..63),
// where *r0 is the number of leading empty planes, which are not stored.
// Returns the number of planes decoded, r0 included.
//
// A 64-bit window after the group test suffices: a run in it is cut at 63
// coefficients first, raw bits after a group test number at most 63 (n < 64
// there), and 64 raw bits are read only where no group test is (n = 64).
__device__ __forceinline__ uint32_t zfp_parse_planes(const uint32_t* w, uint32_t pos, uint32_t budget, uint32_t* pl,
                                                     uint32_t* r0p)
{
    uint32_t bits = budget, n = 0, xlo = 0, xhi = 0;
    const uint32_t a0 = __funnelshift_r(w[pos >> 5], w[(pos >> 5) + 1], pos & 31u);
    const uint32_t r0 = min(a0 ? (uint32_t)__ffs(a0) - 1u : 32u, bits);
    pos += r0;
    bits -= r0;
    *r0p = r0;
    uint32_t r = r0;
    if (r == 32u || bits == 0u) return r;
    pl -= 2u * r0;
    for (;;) {
        const uint32_t i = pos >> 5, sh = pos & 31u;
        const uint32_t w0 = w[i], w1 = w[i + 1], w2 = w[i + 2];
        const bool gtr = n < 64u && bits != 0u;  // a group test is read
        const bool one = gtr && (w0 >> sh & 1u);
        // the 64 bits after it (or from here, if none is)
        const uint32_t o = gtr ? 1u : 0u, c0 = zfp_window(w0, w1, sh + o), c1 = zfp_window(w1, w2, sh + o);
        // a 1: t zeros before the next one (all ones: none within the window)
        const uint32_t t = min(zfp_ctz(c0), zfp_ctz(c1) | 32u);
        // a 0 (or no read): the plane ends; the next plane's raw bits follow
        const uint32_t be = bits - o, m = min(n, be);
        const uint32_t lim = min(63u - n, be);
        const uint32_t z = min(t, lim), hit = t < lim ? 1u : 0u;
        const uint32_t nt = n + z;  // the coefficient that becomes significant
        if (!one) {
            reinterpret_cast<uint2*>(pl)[r] = make_uint2(xlo, xhi);
            ++r;
            if (r == 32u || be == 0u) break;
        }
        const uint32_t rlo = c0 & zfp_low(m), rhi = c1 & zfp_shr(0xffffffffu, 64u - m);
        const uint32_t tlo = xlo | zfp_shl(1u, nt), thi = xhi | zfp_shl(1u, nt - 32u);
        xlo = one ? tlo : rlo;
        xhi = one ? thi : rhi;
        const uint32_t adv = one ? 1u + z + hit : o + m;
        pos += adv;
        bits -= adv;
        n = one ? nt + 1u : n;
    }
    return r;
}

// delta swap: the bits of a at (mask << s) exchange with the bits of b at mask
__device__ __forceinline__ void zfp_dswap(uint32_t& a, uint32_t& b, uint32_t s, uint32_t mask)
{
    const uint32_t t = ((a >> s) ^ b) & mask;
    b ^= t;
    a ^= t << s;
}

// The 8x8 bit matrices of the eight byte columns of 8 rows (L: columns 0-3, H:
// 4-7), transposed at once by three delta-swap stages.
__device__ __forceinline__ void zfp_transpose(uint32_t* L, uint32_t* H)
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        zfp_dswap(L[j], L[j + 4], 4, 0x0F0F0F0Fu);
        zfp_dswap(H[j], H[j + 4], 4, 0x0F0F0F0Fu);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if ((j & 2) == 0) {
            zfp_dswap(L[j], L[j + 2], 2, 0x33333333u);
            zfp_dswap(H[j], H[j + 2], 2, 0x33333333u);
        }
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        zfp_dswap(L[j], L[j + 1], 1, 0x55555555u);
        zfp_dswap(H[j], H[j + 1], 1, 0x55555555u);
    }
}

// Rows of stored planes 8c .. 8c + 7 (row j = stored plane 8c + 7 - j, zero
// past `np`), transposed: byte g of row k is then coefficient 8g + k's bits
// of those planes, the first at bit 7.
__device__ __forceinline__ void zfp_chunk(const uint32_t* pl, uint32_t c, uint32_t np, uint32_t* L, uint32_t* H)
{
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint4 v = reinterpret_cast<const uint4*>(pl + 16u * c)[q];
        const uint32_t p0 = 8u * c + 2u * (uint32_t)q;
        L[7 - 2 * q] = p0 < np ? v.x : 0u;
        H[7 - 2 * q] = p0 < np ? v.y : 0u;
        L[6 - 2 * q] = p0 + 1u < np ? v.z : 0u;
        H[6 - 2 * q] = p0 + 1u < np ? v.w : 0u;
    }
    zfp_transpose(L, H);
}

// Coefficients (stream order) from the stored planes r0 .. planes - 1.  A plane
// is a negabinary digit: a coefficient is the sum of +-2^p over its digits' bit
// positions p, plus for even p, minus for odd (mod 2^32, as (u ^ 0xaaaaaaaa) -
// 0xaaaaaaaa is).  A chunk's byte of digits, the lowest at position k, is so
// ((byte ^ 0xaa) - 0xaa) * (-2)^k: the exclusive-or is done to four bytes at
// once, the subtractions of all chunks are one constant, and a coefficient takes
// a byte permute and a multiply-add a chunk -- of which the second is in the pipe
// that has time left -- where a permute, a shift, an or, and the two steps from
// negabinary at the end took 2.3 of the other's.
__device__ __forceinline__ void zfp_planes_deposit(const uint32_t* pl, uint32_t planes, uint32_t r0, uint32_t* v)
{
    const uint32_t np = planes - r0;
    // (-2)^k of chunk c, k = 24 - r0 - 8 c; 1 where k is negative: that chunk has fewer than 8 planes
    const auto scale_of = [&](uint32_t c) {
        const int32_t k = 24 - (int32_t)(r0 + 8u * c);
        const uint32_t s = k > 0 ? 1u << k : 1u;
        return k > 0 && (k & 1) ? 0u - s : s;
    };
    const auto chunk = [&](uint32_t c, uint32_t* L, uint32_t* H) {
        zfp_chunk(pl, c, np, L, H);
        const int32_t k = 24 - (int32_t)(r0 + 8u * c);
        if (k < 0) {  // its planes to the low end
            const uint32_t s = (uint32_t)-k, keep = zfp_shr(0xffu, s) * 0x01010101u;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                L[j] = zfp_shr(L[j], s) & keep;
                H[j] = zfp_shr(H[j], s) & keep;
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            L[j] ^= 0xaaaaaaaau;
            H[j] ^= 0xaaaaaaaau;
        }
    };
    uint32_t scales = scale_of(0u);
    for (uint32_t c = 1; c * 8u < np; ++c) scales += scale_of(c);
    const uint32_t base = 0u - 0xaau * scales;
    {
        uint32_t L[8], H[8];
        chunk(0u, L, H);
        const uint32_t scale = scale_of(0u);
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                v[8 * g + k] = __byte_perm(L[k], 0u, 0x4440u | (uint32_t)g) * scale + base;
                v[8 * (g + 4) + k] = __byte_perm(H[k], 0u, 0x4440u | (uint32_t)g) * scale + base;
            }
    }
    for (uint32_t c = 1; c * 8u < np; ++c) {
        uint32_t L[8], H[8];
        chunk(c, L, H);
        const uint32_t scale = scale_of(c);
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                v[8 * g + k] += __byte_perm(L[k], 0u, 0x4440u | (uint32_t)g) * scale;
                v[8 * (g + 4) + k] += __byte_perm(H[k], 0u, 0x4440u | (uint32_t)g) * scale;
            }
    }
}

// One block from its words `w` (2 * rate 32-bit words, 64 * rate bits; staged
// in shared memory, or in place in global memory), readable for three words
// past the block.  `pl` is the thread's plane scratch: 64 words, 16-byte
// aligned (a row of shared memory, or a thread-local array).
__device__ __forceinline__ void zfp_decode_staged(const uint32_t* w, uint32_t max_bits, uint32_t* pl, float* out)
{
    const uint32_t h = w[0];
    if (!(h & 1u)) {
#pragma unroll
        for (int i = 0; i < 64; ++i) out[i] = 0.0f;
        return;
    }
    const int32_t emax = (int32_t)((h >> 1) & 255u) - 127;
    uint32_t r0;
    const uint32_t planes = zfp_parse_planes(w, 9u, max_bits - 9u, pl, &r0);
    uint32_t u[64];
    zfp_planes_deposit(pl, planes, r0, u);
    int32_t v[64];
    BCMC_ZFP_GATHER(v, (int32_t)u)
    zfp_inverse_transform(v);
    const float wt = zfp_inv_weight(emax);
#pragma unroll
    for (int i = 0; i < 64; ++i) out[i] = __fmul_rn(wt, __int2float_rn(v[i]));
}

// Shared memory of a staged decode CTA of `threads` threads at `rate`: the
// staged words (2 * rate per block, 4 words of padding) and 68 words of plane
// scratch per thread (64 used; 68 keeps the threads' 16-byte rows on
// different banks).  A thread's row also holds its decoded block for the
// warp's coalesced store (zfp_store_warp).
constexpr uint32_t kZfpPlaneWords = 68;
__host__ __device__ __forceinline__ uint32_t zfp_stage_words(uint32_t threads, uint32_t rate)
{
    return threads * 2u * rate + 4u;
}
__host__ __device__ __forceinline__ size_t zfp_stage_smem(uint32_t threads, uint32_t rate)
{
    return ((size_t)zfp_stage_words(threads, rate) + (size_t)threads * kZfpPlaneWords) * 4u;
}
__device__ __forceinline__ uint32_t* zfp_stage_planes(uint32_t* s_words, uint32_t threads, uint32_t rate)
{
    return s_words + zfp_stage_words(threads, rate) + threadIdx.x * kZfpPlaneWords;
}

// The warp's decoded blocks to out[k * 64 ..] for the warp's k-th block,
// k < count, with coalesced 16-byte stores: each thread writes its block into
// its own row (`row`, from zfp_stage_planes), then the warp stores two blocks
// per instruction.  Every lane of the warp calls it (a lane without a block
// passes nothing to write: `v` is not read when has_block is false).
__device__ __forceinline__ void zfp_store_warp(uint32_t* row, const float* v, bool has_block, float* out,
                                               uint32_t count)
{
    if (has_block) {
        float4* r4 = reinterpret_cast<float4*>(row);
#pragma unroll
        for (int i = 0; i < 16; ++i) r4[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
    __syncwarp();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t* row0 = row - lane * kZfpPlaneWords;
#pragma unroll
    for (uint32_t k = 0; k < 16; ++k) {
        const uint32_t blk = 2u * k + (lane >> 4);
        if (blk < count)
            reinterpret_cast<float4*>(out + (uint64_t)blk * 64u)[lane & 15u] =
                *reinterpret_cast<const float4*>(row0 + blk * kZfpPlaneWords + 4u * (lane & 15u));
    }
    __syncwarp();
}

// Copies the words of blocks b0 .. b0+nb-1 (consecutive) to s_words with
// coalesced 8-byte loads, and zeroes the 4 padding words.  All the CTA's
// threads call it; the caller synchronises before reading.
__device__ __forceinline__ void zfp_stage_run(const uint64_t* __restrict__ words, uint64_t b0, uint32_t nb,
                                              uint32_t rate, uint32_t* s_words)
{
    const uint64_t* src = words + b0 * rate;
    uint2* dst = reinterpret_cast<uint2*>(s_words);
    const uint32_t n = nb * rate;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint64_t x = __ldg(src + i);
        dst[i] = make_uint2((uint32_t)x, (uint32_t)(x >> 32));
    }
    if (threadIdx.x < 4) s_words[2u * n + threadIdx.x] = 0u;
}

// Copies the words of block b to this thread's slot of s_words (2 * rate
// words at threadIdx.x * 2 * rate).  The 4 padding words after the last slot
// are zeroed by thread 0; the caller synchronises before any thread reads.
__device__ __forceinline__ void zfp_stage_block(const uint64_t* __restrict__ words, uint64_t b, uint32_t rate,
                                                uint32_t* s_words)
{
    const uint64_t* src = words + b * rate;
    uint2* dst = reinterpret_cast<uint2*>(s_words + threadIdx.x * 2u * rate);
    for (uint32_t i = 0; i < rate; ++i) {
        const uint64_t x = __ldg(src + i);
        dst[i] = make_uint2((uint32_t)x, (uint32_t)(x >> 32));
    }
}

// ---------------------------------------------------------------------------
// Encoder (the reference only decodes): block-floating-point cast, forward
// lift along x, y, z, negabinary reorder and embedded bit-plane coding with
// group tests, per the published fixed-rate ZFP method (Lindstrom 2014).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void zfp_fwd_lift(int32_t& x, int32_t& y, int32_t& z, int32_t& w)
{
    x += w; x >>= 1; w -= x;
    z += y; z >>= 1; y -= z;
    x += z; x >>= 1; z -= x;
    w += y; w >>= 1; y -= w;
    w += y >> 1; y -= w >> 1;
}

// The block's coefficients in stream order, negabinary, from its 64 values; *ep
// is the biased common exponent.  False for a block coded as zero.
__device__ __forceinline__ bool zfp_forward(const float* f, uint32_t* u, uint32_t* ep)
{
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 64; ++i) amax = fmaxf(amax, fabsf(f[i]));
    int emax = -127;
    if (amax > 0.0f) frexpf(amax, &emax);
    *ep = (uint32_t)(emax + 127);
    if (*ep == 0u) return false;
    const int sh = 30 - emax;
    int32_t v[64];
    if (sh <= 127) {  // 2^sh is a float: the product rounds as ldexpf does
        const float w = __int_as_float((sh + 127) << 23);
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = (int32_t)__fmul_rn(f[i], w);
    } else {
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = (int32_t)ldexpf(f[i], sh);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) zfp_fwd_lift(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);  // x
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const int b = 16 * z + x;
            zfp_fwd_lift(v[b], v[b + 4], v[b + 8], v[b + 12]);  // y
        }
#pragma unroll
    for (int i = 0; i < 16; ++i) zfp_fwd_lift(v[i], v[i + 16], v[i + 32], v[i + 48]);  // z
    uint32_t un[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) un[i] = ((uint32_t)v[i] + 0xaaaaaaaau) ^ 0xaaaaaaaau;
    BCMC_ZFP_SCATTER(u, un)
    return true;
}

// Planes 8c .. 8c + 7 of the coefficients (plane 0: bit 31) as masks, coefficient
// i at bit i: plane p of the chunk goes to pl[2p] (0..31) and pl[2p + 1].  The
// rows of bytes are transposed by the decoder's three delta-swap stages.
__device__ __forceinline__ void zfp_planes(const uint32_t* u, uint32_t c, uint32_t* pl)
{
    uint32_t L[8], H[8];
    const uint32_t sel = (3u - c) | ((7u - c) << 4);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        L[k] = __byte_perm(__byte_perm(u[k], u[8 + k], sel), __byte_perm(u[16 + k], u[24 + k], sel), 0x5410u);
        H[k] = __byte_perm(__byte_perm(u[32 + k], u[40 + k], sel), __byte_perm(u[48 + k], u[56 + k], sel), 0x5410u);
    }
    zfp_transpose(L, H);
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        pl[2 * p] = L[7 - p];
        pl[2 * p + 1] = H[7 - p];
    }
}

// Bits appended to a row of 32-bit words: the word being filled is kept in a
// register, and an append (up to 64 bits, the ones above its length zero) stores
// the three words it can reach without reading any.
struct RowWriter {
    uint32_t* row;
    uint32_t pos, cur;

    __device__ __forceinline__ void put(uint32_t lo, uint32_t hi, uint32_t len)
    {
        const uint32_t i = pos >> 5, sh = pos & 31u;
        const uint32_t t0 = cur | (lo << sh), t1 = __funnelshift_l(lo, hi, sh), t2 = __funnelshift_l(hi, 0u, sh);
        row[i] = t0;
        row[i + 1] = t1;
        row[i + 2] = t2;
        pos += len;
        const uint32_t d = (pos >> 5) - i;
        cur = d == 0u ? t0 : (d == 1u ? t1 : t2);
    }
};

// Words of a block's row: the block's bits, and three more that an append at its
// end touches (RowWriter::put).
__host__ __device__ __forceinline__ constexpr uint32_t zfp_encode_row_words(uint32_t rate) { return 2u * rate + 3u; }

// One block into its row of zeroed words (zfp_encode_row_words).  `pl`: 32 words
// of scratch.
//
// encode_ints of the published method, in the decoder's steps: a step is either
// a group test that finds a coefficient (a 1, the zeros before it, and its 1
// unless the bits or the 63 coefficients before it run out first) or the end of
// the plane with the next plane's raw bits, both computed by selects, so that a
// warp's lanes stay together although their blocks take different numbers of
// steps; they wait for each other at every sixteenth plane (eighth: 57 us at
// 256^3 and rate 4, sixteenth: 49 us).  A bit at a time into a 64-bit buffer,
// with the planes picked bit by bit out of 64 coefficients, took 378 us.
__device__ __forceinline__ void zfp_encode_row(const float* f, uint32_t max_bits, uint32_t* row, uint32_t* pl)
{
    uint32_t u[64], e;
    if (!zfp_forward(f, u, &e)) return;  // a single 0 bit
    uint32_t any = 0;
#pragma unroll
    for (int i = 0; i < 64; ++i) any |= u[i];
    RowWriter out{row, 9u, 1u | ((e & 255u) << 1)};
    row[0] = out.cur;
    uint32_t bits = max_bits - 9u;
    // the leading empty planes, a 0 each
    const uint32_t r0 = zfp_clz(any);
    if (r0 >= bits || r0 == 32u) return;
    bits -= r0;
    out.pos += r0;
    if (out.pos >= 32u) out.cur = 0u;
#pragma unroll
    for (int i = 0; i < 64; ++i) u[i] <<= r0;
    uint32_t n = 0;
    for (uint32_t c = 0; 8u * c < 32u - r0; c += 2) {
        zfp_planes(u, c, pl);
        zfp_planes(u, c + 1, pl + 16);
        const uint32_t np = min(32u - r0 - 8u * c, 16u);  // planes of the chunk
        // the first plane's raw bits
        uint32_t p = 0, o = 0;
        uint32_t xlo, xhi;
        {
            const uint32_t lo = pl[0], hi = pl[1], m = min(n, bits);
            out.put(lo & (zfp_shl(1u, m) - 1u), hi & zfp_shr(0xffffffffu, 64u - m), m);
            bits -= m;
            xlo = m >= 32u ? zfp_shr(hi, m - 32u) : __funnelshift_r(lo, hi, m);
            xhi = zfp_shr(hi, m);
        }
        for (;;) {
            const bool test = n < 64u && bits != 0u;  // a group test is written
            const bool one = test && (xlo | xhi) != 0u;
            o = test ? 1u : 0u;
            // a 1: t zeros before the next significant coefficient
            const uint32_t t = xlo ? (uint32_t)__ffs(xlo) - 1u : (uint32_t)__ffs(xhi) + 31u;
            const uint32_t lim = min(63u - n, bits - 1u);
            const uint32_t z = min(t, lim), hit = t < lim ? 1u : 0u;
            // a 0 (or no test): the plane ends, the next one's raw bits follow
            const uint32_t be = bits - o, m = min(n, be);
            if (!one && (++p == np || be == 0u)) break;
            const uint32_t plo = pl[2 * (p & 15u)], phi = pl[2 * (p & 15u) + 1];
            const uint32_t rlo = plo & (zfp_shl(1u, m) - 1u), rhi = phi & zfp_shr(0xffffffffu, 64u - m);
            const uint32_t vlo = one ? 1u | (hit ? zfp_shl(1u, z + 1u) : 0u) : rlo << o;
            const uint32_t vhi = one ? (hit ? zfp_shl(1u, z - 31u) : 0u) : __funnelshift_l(rlo, rhi, o);
            const uint32_t len = one ? 1u + z + hit : o + m;
            out.put(vlo, vhi, len);
            bits -= len;
            n = one ? n + z + 1u : n;
            const uint32_t slo = one ? xlo : plo, shi = one ? xhi : phi, s = one ? z + 1u : m;
            xlo = s >= 32u ? zfp_shr(shi, s - 32u) : __funnelshift_r(slo, shi, s);
            xhi = zfp_shr(shi, s);
        }
        out.put(0u, 0u, o);  // the 0 that ended the chunk's last plane
        bits -= o;
        if (bits == 0u) return;
    }
}

// The same to its place in a stream of 64-bit words, a block at a time (k_encode
// stores a warp's rows together; this is the form that host builds test).
struct BitWriter {
    unsigned long long* words;
    uint64_t first;  // the block's first word

    __device__ __forceinline__ void init(unsigned long long* w, uint64_t bit_offset)
    {
        words = w;
        first = bit_offset >> 6;
    }
    __device__ __forceinline__ void finish() {}
};
__device__ __forceinline__ void zfp_encode_block(const float* f, uint32_t max_bits, BitWriter& bw)
{
    uint32_t row[zfp_encode_row_words(kZfpMaxBitsLimit / 64u)] = {}, pl[32];
    zfp_encode_row(f, max_bits, row, pl);
    for (uint32_t i = 0; i < max_bits / 64u; ++i)
        bw.words[bw.first + i] = (unsigned long long)row[2 * i] | ((unsigned long long)row[2 * i + 1] << 32);
}

}  // namespace bcmc
