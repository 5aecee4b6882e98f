// Products of packed rows (Q4_K, Q8_0, Q6_K) with a few columns of activations on tcgen05, in 32-bit grade: the body that the batched Q8_0 GEMV, the Q6_K
// GEMV of many rows (both gemv_tc.cu) and the sorted MoE layer (Q4_K, moe_slots.cu) share.
//
// The weights are A and come from tensor memory, where the warps that unpack them put them:
//   * Q4_K: a weight is d * (sc * q) - dmin * m.  sc * q is an integer of at most 945, exact in f16, so one AND-OR and one f16x2 multiply-add turn
//     two nibbles into the operand (1024 + q) * sc - 1024 * sc without rounding (a high nibble stays in place as 16 q).  d and dmin
//     meet the 256-weight sums in f32.  Q8_0, Q6_K: the integers themselves; the scales meet the sums of 32 in f32.
//   * Q4_K, Q6_K: an activation is x = 2^e * (hi + lo) with f16 hi and lo and one power of two per 256 elements of a column: 22 bits, error at most
//     2^-22 of the value or 2^-35 of the largest of the 256 (which is brought near the top of f16's range, because the halves that meet high
//     nibbles are stored as x / 16 and end at its smallest step).
//   * Q8_0, Q6_K of K < 2048: x = 2^e * (hi + 2^-14 * (lo + rest)), hi an integer of at most 2^11: the sum of 32 products with a weight's integer stays below 2^24 and
//     is exact, however the tensor cores round their sums; lo and rest are the other bits, as f16, and share their sums, which are 2^-11 of
//     the others.  All 24 bits of a value down to 2^-11 of the largest of the 256 are kept, and 23 down to 2^-25.  Two halves alone (22 bits and sums
//     that the tensor cores cut off) were 4 % further from 64 bits than f32 products at K = 256, and up to 40 % with a few large channels.
//   * Q4_K: sum_j m_j * (sum of x over block j) is one more product of K = 16 per 256: A = 32 m twice, B = both halves of the block sums / 32.
// Q4_K: an Inf or a NaN among a column's 256 activations makes its scale, and with it the column, NaN.  Sums per block: it is a half like others.
//
// A CTA walks steps of 128 rows x 256 K.  Teams of four warps take the steps, or the halves of steps, in turn: a thread owns a row (tensor-memory
// lane), unpacks its weights from the raw superblocks (TMA ring) and stores them to tensor memory.  The sums' warps read a step's sums
// back, apply d, dmin and 2^e and add; one more warp issues the products and one the copies.  With SUBS = 2 two tiles of 128 rows share the
// activations' copies (gate and up of the same outputs, or 256 rows).
// Every wait is bounded; a wait that gives up sets the CTA's abort flag and all roles leave.
//
// Bound: the unpacking warps and the hand-overs between roles, 850 to 1000 clocks per step of 8 columns (2.8 warp instructions per
// weight and 32 rows; a step's bytes arrive in 800), the products from about 40 columns on.  Why the roles are split like this, measured on one Q4_K matrix of
// 152064 x 3584 with 8 columns (a product that gemv_imma.cu serves, faster over a whole step): the unpacking warps also reading the sums, two CTAs of 8
// warps per SM, 114 us; sums in warps of their own but one issuing warp, which pays a wait of about 150 clocks per barrier, 102; an issuing warp per
// place of the sums 83; no integer divisions in the sums' warps 75; one piece per step 73.
#pragma once

#include "gemv_common.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace runit {
namespace tcr {

// What a step looks like:
//   Q4K_8   up to 8 columns, both halves side by side as the 16 columns of one product; hi of the last 64 K behind all of lo, in the columns of lo
//   Q4K_48  up to 48 columns in multiples of 16, the halves in turn into the same sums
//   Q8_0_8  up to 8 columns, hi and lo side by side; a sum for each of the eight blocks, because their scales are f16 values that
//           no integer factor expresses
//   Q6K_8   one column; block b of it has columns b (hi) and 8 + b (lo) of one product to itself, with zeros in the others' rows: one load of sixteen
//           sums and not eight
//   Q6K_8R  the same with the rest in columns 16 + b (24 to 31 are not used: their rows are whatever lies behind the image's)
// Image of 256 activations of N columns (128-byte swizzled rows of 64 elements, in the order of split_column):
//   Q4K_8   4 panels of 16 rows (8 hi, 8 lo), then a panel whose row n holds the block sums of column n
//   Q4K_48  4 panels of N rows of hi, 4 of lo, one of block sums
//   else    4 panels of 16 or 24 rows: 8 hi, 8 lo, 8 rest (Q8_0: the rest in a product of its own with the columns of lo; the columns of hi meet rows of
//           zeros there, which lie ahead of the images)
enum Kind { Q4K_8, Q4K_48, Q8_0_8, Q6K_8, Q6K_8R };

template <Kind K> struct Cfg {
    static constexpr bool kQ6 = K == Q6K_8 || K == Q6K_8R, kBlocks = K == Q8_0_8 || kQ6, kRest = K == Q8_0_8 || K == Q6K_8R;      // sums per block; three parts of an activation
    static constexpr uint32_t kCols = K == Q4K_48 ? 48 : 8;
    // kParts: a step is unpacked in one piece, or in halves (an empty tensor memory holds two steps, not three)
    static constexpr uint32_t kParts = K == Q4K_48 || kQ6 ? 2 : 1, kTeams = K == Q4K_8 ? 3 : kQ6 ? 4 : 2, kSumWarps = K == Q4K_48 ? 12 : K == Q8_0_8 ? 8 : 4;
    static constexpr uint32_t kSum0 = 4 * kTeams, kMma = kSum0 + kSumWarps, kMmaWarps = K == Q4K_8 ? 3 : 2, kCopyW = kMma + kMmaWarps, kCopyB = kCopyW + 1, kThreads = 32 * (kCopyB + 1);      // warps by role
    static constexpr uint32_t kUnit = K == Q8_0_8 ? 272 : kQ6 ? 240 : 144, kWBytes = 128 * kUnit;      // bytes of 256 weights; raw superblocks of a step
    // rings: raw steps, activations' images, unpacked pieces (kSteps steps) in tensor memory, sums; columns' scales and rows' scales (see the bounds below)
    static constexpr uint32_t kW = K == Q4K_8 ? 6 : 4, kB = K == Q4K_48 ? 2 : 4, kSteps = K == Q4K_8 ? 3 : 2, kA = kSteps * kParts, kD = kSteps;
    static constexpr uint32_t kXs = K == Q4K_48 ? 8 : 16, kRows = 8, kMins = kSteps;
    static constexpr uint32_t kBRow = K == Q4K_8 ? 1280 : K == Q4K_48 ? 1152 : kRest ? 1536 : 1024;       // bytes of an image per column
    static constexpr uint32_t kBStage = kCols * kBRow, kOffB = K == Q4K_8 || K == Q8_0_8 ? 1024 : 0;     // eight rows of zeros, then the images
    static constexpr uint32_t kPanel = (kRest ? 24 : 16) * 128;                                           // of an image with sums per block
    static constexpr uint32_t kMinCol = 128 * kSteps, kDCol = kMinCol + (kBlocks ? 0 : 32);
    static constexpr uint32_t kDCols = K == Q4K_48 ? 96 : K == Q8_0_8 ? 128 : K == Q6K_8 ? 16 : 32, kMOff = kDCols / 2;          // sums of a step: products, then minimums; or of its blocks
    static constexpr uint32_t kRowScale = kBlocks ? 16 : 4;                                // bytes of a row's scales: eight d; d and dmin
    static constexpr uint32_t kOffW = kOffB + kB * kBStage, kOffXs = kOffW + kW * kWBytes, kOffRows = kOffXs + kXs * kCols * 4, kOffBar = kOffRows + kRows * 128 * kRowScale;
    static constexpr uint32_t kBars = 2 * (kA + kW + kB + kD) + kMmaWarps;
    static constexpr uint32_t kOffAt = kOffBar + kBars * 8 + 16;                 // Q6_K: where a raw step's rows start (row_start)
    static constexpr uint32_t kSmem = kOffAt + 4 * kW + 1024;
    static constexpr int kAcc = K == Q4K_8 ? 8 : K == Q4K_48 ? 16 : kQ6 ? 1 : 4;           // sums of a thread and tile
    static_assert(kBStage % 1024 == 0 && kWBytes % 128 == 0 && kOffRows % 16 == 0 && kOffBar % 8 == 0 && kSmem <= 227 * 1024, "shared memory");
    static_assert((kBlocks || kMinCol + 8 * kMins <= kDCol) && kMinCol <= kDCol && kDCol + kD * kDCols <= 512, "tensor memory");
    // A piece is unpacked once that of the step kSteps before has been multiplied, the minimums of that step with it.  Its sums had a place then, so
    // the sums up to step s - kSteps - kD have been read (one group of warps reads them in order), and with them the rows' scales that step s
    // replaces.  The copies of a step's columns' scales wait for the raw steps kW before to have been unpacked.
    // A team and an issuing warp have their own places in the rings that they wait on: a parity tells two phases of a place apart and not three.
    static_assert(kA % kTeams == 0 && kW * kParts % kTeams == 0 && kMmaWarps == kSteps && kD == kMmaWarps, "places of a team, of an issuing warp");
    static_assert(!kQ6 || (kTeams <= kA && kTeams <= kW * kParts), "a team's first piece waits for weights alone");
    static_assert(kRows > kSteps + kD && kMins == kSteps && kXs * (K == Q4K_48 ? 2 : 1) > kW + kSteps + kD, "rings of scales");
};

// The products with hi, and those with lo and the rest.
__device__ __forceinline__ float with_low(float hi, float lo) { return fmaf(lo, 6.103515625e-5f, hi); }      // 2^-14
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// 1024 + the field, as f16x2: one LOP3
__device__ __forceinline__ uint32_t field(uint32_t w, uint32_t mask) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(mask), "r"(0x64006400u));
    return r;
}
// two nibbles in place (mask 0x000F000F or 0x00F000F0) -> f16x2 of sc * nibble (16 * sc * nibble): exact
__device__ __forceinline__ uint32_t scaled_pair(uint32_t w, uint32_t mask, __half2 sc, __half2 bias) {
    return as_u32(__hfma2(as_half2(field(w, mask)), sc, bias));
}
// byte j of p as f16x2 (sc, sc); and -1024 times it
__device__ __forceinline__ __half2 scale_pair(uint32_t p, uint32_t j) {
    return __hsub2(as_half2(__byte_perm(p, 0x64646464u, 0x4040u + 0x0101u * j)), as_half2(0x64006400u));
}

// Where activations lie in a row of a 128-byte swizzled panel of 64 K.  Q4_K: a weight word's eight elements are consecutive in K, low nibbles
// 0, 2, 1, 3, high nibbles 0, 2, 1, 3; 8 bytes per word w and half.  Q8_0: in order; 16 bytes per 8 elements.
__device__ __forceinline__ uint32_t chunk_offset(uint32_t row, uint32_t chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// Eight consecutive activations by a lane: element 8 * lane and on of a column's 256.
__device__ __forceinline__ void load8(const float* x, bool live, float (&v)[8]) {
    if (!live) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = 0.f;
    } else if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const float4 a = *reinterpret_cast<const float4*>(x), b = *reinterpret_cast<const float4*>(x + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = x[i];
    }
}
// One column's 256 activations by a warp (load8) into the panels of an image: panels of hi from `hi` on, of lo from `lo`, `panel` bytes apart, and for
// Q4_K the block sums' panel `sums`, in the rows given (else the rest eight rows behind lo).  Returns the column's scale.
template <Kind K>
__device__ __forceinline__ float split_column(const float (&v)[8], uint32_t lane, uint8_t* hi, uint32_t hi_row, uint8_t* lo, uint32_t lo_row, uint32_t panel,
                                              uint8_t* sums, uint32_t sum_row) {
    float amax = 0.f;
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const bool finite = fabsf(v[i]) <= 3.4028235e38f;
        if (finite || !Cfg<K>::kBlocks) amax = fmaxf(amax, fabsf(v[i]));
        if (!Cfg<K>::kBlocks) bad |= !finite;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    bad = __any_sync(0xffffffffu, bad);
    // 2^e such that the largest |x| / 2^e lies in [2^14, 2^15): so does a 32nd of a block's sum (with a rest: [2^10, 2^11)).  e is held above
    // -116 so that both powers are normal numbers.
    int e = (int)((__float_as_uint(amax) >> 23) & 255u) - 127 - (Cfg<K>::kRest ? 10 : 14);
    e = e < -116 ? -116 : e;
    const float inv = __uint_as_float((uint32_t)(127 - e) << 23);
    const uint32_t block = lane >> 2, half = block & 1;
    __half h[8], l[8], rest[8];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        // with sums per block an Inf or a NaN goes through the products like any value
        const bool finite = !Cfg<K>::kBlocks || fabsf(v[i]) <= 3.4028235e38f;
        const float w = bad ? 0.f : finite ? v[i] * inv : v[i];
        const float ws = !Cfg<K>::kBlocks && half ? w * 0.0625f : w;       // meets 16 q
        h[i] = __float2half_rn(Cfg<K>::kRest ? rintf(ws) : ws);
        float r = finite ? ws - __half2float(h[i]) : 0.f;
        if (Cfg<K>::kRest) r *= 16384.f;
        l[i] = __float2half_rn(r);
        rest[i] = __float2half_rn(r - __half2float(l[i]));
        sum += w;
    }
    hi += (block >> 1) * panel;
    lo += (block >> 1) * panel;
    if constexpr (Cfg<K>::kBlocks) {
        const uint32_t c = 4 * half + (lane & 3);
        *reinterpret_cast<uint4*>(hi + chunk_offset(hi_row, c)) = *reinterpret_cast<const uint4*>(h);
        *reinterpret_cast<uint4*>(lo + chunk_offset(lo_row, c)) = *reinterpret_cast<const uint4*>(l);
        if (Cfg<K>::kRest) *reinterpret_cast<uint4*>(lo + chunk_offset(lo_row + 8, c)) = *reinterpret_cast<const uint4*>(rest);
    } else {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t w = 2 * (lane & 3) + i;
            const __half2 ph[2] = {__halves2half2(h[4 * i], h[4 * i + 2]), __halves2half2(h[4 * i + 1], h[4 * i + 3])};
            const __half2 pl[2] = {__halves2half2(l[4 * i], l[4 * i + 2]), __halves2half2(l[4 * i + 1], l[4 * i + 3])};
            *reinterpret_cast<uint2*>(hi + chunk_offset(hi_row, w) + 8 * half) = *reinterpret_cast<const uint2*>(ph);
            *reinterpret_cast<uint2*>(lo + chunk_offset(lo_row, w) + 8 * half) = *reinterpret_cast<const uint2*>(pl);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if ((lane & 3) == 0) {
            sum *= 0.03125f;
            const uint32_t si = (block >> 1) + 4 * half;              // the order of the unpacked minimums
            const __half sh = __float2half_rn(sum), sl = __float2half_rn(sum - __half2float(sh));
            *reinterpret_cast<__half*>(sums + chunk_offset(sum_row, 0) + 2 * si) = sh;
            *reinterpret_cast<__half*>(sums + chunk_offset(sum_row, 1) + 2 * si) = sl;
        }
    }
    return bad ? __uint_as_float(0x7FC00000u) : __uint_as_float((uint32_t)(e + 127) << 23);
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// Half H (128 weights) of a row, as f16 pairs in the order of split_column, into 64 columns of tensor memory at `at`, 16 at a time.
template <int H> __device__ __forceinline__ void unpack_q4k(const uint8_t* raw, const Q4KScales& sc, uint32_t at) {
#pragma unroll
    for (int jj = 0; jj < 2; jj++) {
        const int j = 2 * H + jj;
        const uint4 q0 = *reinterpret_cast<const uint4*>(raw + 16 + 32 * j), q1 = *reinterpret_cast<const uint4*>(raw + 32 + 32 * j);
        const uint32_t q[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        const __half2 sl = scale_pair(sc.sl, j), sh = scale_pair(sc.sh, j);
        const __half2 bl = __hmul2(sl, as_half2(0xE400E400u)), bh = __hmul2(sh, as_half2(0xE400E400u));       // -1024 * scale
#pragma unroll
        for (int c = 0; c < 2; c++) {
            uint32_t o[16];
#pragma unroll
            for (int w = 0; w < 4; w++) {
                const uint32_t x = q[4 * c + w], y = x >> 8;
                o[4 * w + 0] = scaled_pair(x, 0x000F000Fu, sl, bl);
                o[4 * w + 1] = scaled_pair(y, 0x000F000Fu, sl, bl);
                o[4 * w + 2] = scaled_pair(x, 0x00F000F0u, sh, bh);
                o[4 * w + 3] = scaled_pair(y, 0x00F000F0u, sh, bh);
            }
            tmem_st16(at + 32 * jj + 16 * c, o);
        }
    }
}
// Q8_0: 34 words a half, from word 2 H of 36 at byte 128 H; a byte becomes 1024 + 128 + q without arithmetic.
template <int H> __device__ __forceinline__ uint2 unpack_q8_0(const uint8_t* raw, uint32_t at) {
    uint32_t sc[2];
#pragma unroll
    for (int p = 0; p < 2; p++) {                  // pairs of blocks: 17 words from word (17 p + 2 H) % 4 of 20
        constexpr int kFirst[2] = {2 * H, 17 + 2 * H};
        uint32_t w[20];
#pragma unroll
        for (int i = 0; i < 5; i++) *reinterpret_cast<uint4*>(w + 4 * i) = *reinterpret_cast<const uint4*>(raw + 128 * H + kFirst[p] / 4 * 16 + 16 * i);
        const int w0 = kFirst[p] % 4;
#pragma unroll
        for (int b = 0; b < 2; b++) {
            uint32_t o[16];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t x = (b ? w[w0 + 9 + i] : __funnelshift_r(w[w0 + i], w[w0 + i + 1], 16)) ^ 0x80808080u;
                o[2 * i + 0] = as_u32(__hsub2(as_half2(__byte_perm(x, 0x64646464u, 0x4140u)), as_half2(0x64806480u)));
                o[2 * i + 1] = as_u32(__hsub2(as_half2(__byte_perm(x, 0x64646464u, 0x4342u)), as_half2(0x64806480u)));
            }
            tmem_st16(at + 32 * p + 16 * b, o);
        }
        sc[p] = __byte_perm(w[w0], w[w0 + 8], 0x7610);
    }
    return make_uint2(sc[0], sc[1]);
}

// Q6_K: rows start on even bytes, and a copy on a multiple of 16.  Rows eight apart start alike, so a step comes as eight boxes, box r with rows
// r, r + 8, ..., each from the last multiple of 16 before its unit.  at: (2 unit | bytes of a row << 8), both mod 16: a row's first byte in its box.
__device__ __forceinline__ uint32_t row_start(uint32_t at, uint32_t r) { return (at + r * (at >> 8)) & 14; }
// The tile's row of a lane of tensor memory: a warp reads eight rows of each of four boxes (240-byte pitch: eight banks apart by 4; where the boxes
// start differently, K / 256 = 2 mod 4, all 32 banks).
__device__ __forceinline__ uint32_t q6k_row(uint32_t t) { return 8 * ((t & 7) + 8 * (t >> 6)) + ((t >> 3) & 7); }

// Q6_K, half h of a row that starts `shift` bits (0 or 16) behind its first word: 16 words of low nibbles for every two of four blocks, 8 of high
// bits; a byte becomes 1024 + 32 + q without arithmetic.  Returns the four blocks' scales.
__device__ __forceinline__ uint32_t unpack_q6k(const uint8_t* raw, uint32_t h, uint32_t shift, uint32_t at) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(raw);
    auto word = [&](uint32_t i) { return __funnelshift_r(w[i], w[i + 1], shift); };
#pragma unroll
    for (int g = 0; g < 2; g++) {                  // words 4 g .. of the blocks: 16 of their 32 elements
        uint32_t a0[4], a1[4], hb[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            a0[i] = word(16 * h + 4 * g + i);
            a1[i] = word(16 * h + 8 + 4 * g + i);
            hb[i] = word(32 + 8 * h + 4 * g + i);
        }
#pragma unroll
        for (int b = 0; b < 4; b++) {
            uint32_t o[8];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t a = b & 1 ? a1[i] : a0[i], top = b == 0 ? hb[i] << 4 : b == 1 ? hb[i] << 2 : b == 2 ? hb[i] : hb[i] >> 2;
                const uint32_t q = ((b & 2 ? a >> 4 : a) & 0x0F0F0F0Fu) | (top & 0x30303030u);
                o[2 * i + 0] = as_u32(__hsub2(as_half2(__byte_perm(q, 0x64646464u, 0x4140u)), as_half2(0x64206420u)));
                o[2 * i + 1] = as_u32(__hsub2(as_half2(__byte_perm(q, 0x64646464u, 0x4342u)), as_half2(0x64206420u)));
            }
            tmem_st8(at + 16 * b + 8 * g, o);
        }
    }
    // the first of a block's two scales serves all of it: bytes 0, 2, 4, 6 of the half's eight
    return __byte_perm(word(48 + 2 * h), word(49 + 2 * h), 0x6420u);
}

// A stretch of units of K over SUBS row tiles, with one image of activations per unit.
struct Run {
    const CUtensorMap* map[2];
    int32_t row[2];
    uint32_t u0, u1;
    const uint8_t* b;            // image of unit u0; the next ones follow
    const float* xs;             // scales of unit u0, likewise
    uint32_t n;                  // columns of the image (Q4K_48: a multiple of 16), 8 otherwise
};

// One CTA's rings and roles.  The kernel issues the copies itself (warps kCopyW and kCopyB); work() is everything else.
// P: kSubs (row tiles that share an image, 1 or 2); uint32_t begin(), end(), steps(): runs and steps of this CTA;  Run run(uint32_t i);
//    bool few() (sums per block: at most four columns, a thread takes two of them and not four);
//    void finish(uint32_t i, float (&acc)[kSubs][kAcc], uint32_t warp, uint32_t lane): the sums of a run, thread by thread (warp: of the sums' warps);
//    zeroes them.
template <Kind K, int SUBS> struct Block {
    using C = Cfg<K>;
    static constexpr uint32_t COLS = C::kCols;
    uint32_t base, warp, lane, a_full, a_empty, w_full, w_empty, b_full, b_empty, d_full, d_empty, drain, tmem;
    uint8_t* base_p;
    volatile int* abort_flag;
    bool ok;

    __device__ __forceinline__ Block(uint8_t* smem_raw) {
        const uint32_t tid = threadIdx.x;
        base = (smem_u32(smem_raw) + 1023u) & ~1023u;
        base_p = smem_raw + (base - smem_u32(smem_raw));
        warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
        lane = tid & 31;
        a_full = base + C::kOffBar;
        a_empty = a_full + 8 * C::kA;
        w_full = a_empty + 8 * C::kA;
        w_empty = w_full + 8 * C::kW;
        b_full = w_empty + 8 * C::kW;
        b_empty = b_full + 8 * C::kB;
        d_full = b_empty + 8 * C::kB;
        d_empty = d_full + 8 * C::kD;
        drain = d_empty + 8 * C::kD;
        abort_flag = reinterpret_cast<volatile int*>(base_p + C::kOffBar + C::kBars * 8 + 4);
        ok = true;
        if (tid == 0) {
            for (uint32_t i = 0; i < C::kA; i++) {
                mbar_init(a_full + 8 * i, 4);
                mbar_init(a_empty + 8 * i, 1);
            }
            for (uint32_t i = 0; i < C::kW; i++) {
                mbar_init(w_full + 8 * i, 1);
                mbar_init(w_empty + 8 * i, 4 * C::kParts);
            }
            for (uint32_t i = 0; i < C::kB; i++) {
                mbar_init(b_full + 8 * i, 1);
                mbar_init(b_empty + 8 * i, SUBS);
            }
            for (uint32_t i = 0; i < C::kD; i++) {
                mbar_init(d_full + 8 * i, 1);
                mbar_init(d_empty + 8 * i, C::kSumWarps);
            }
            for (uint32_t i = 0; i < C::kMmaWarps; i++) mbar_init(drain + 8 * i, 1);
            *abort_flag = 0;
            fence_mbar_init();
        }
        if (tid < C::kOffB / 16) {
            reinterpret_cast<uint4*>(base_p)[tid] = make_uint4(0, 0, 0, 0);
            fence_proxy_async();
        }
        if (warp == C::kMma) {
            tmem_alloc(base + C::kOffBar + C::kBars * 8, 512);
            tmem_relinquish();
        }
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
        // not before the allocation is known to be done: a CTA of the next grid must not take the columns first
        grid_launch_dependents();
        tmem = *reinterpret_cast<volatile uint32_t*>(base_p + C::kOffBar + C::kBars * 8);
    }
    // the whole warp waits, and goes on or gives up together
    __device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        return ok = __all_sync(0xffffffffu, mbar_wait_timed(bar, parity, abort_flag));
    }
    // places and barriers of a raw step, of an image; free: waits until what was there is no longer needed
    __device__ __forceinline__ uint32_t raw(uint32_t s) const { return base + C::kOffW + s % C::kW * C::kWBytes; }
    __device__ __forceinline__ uint32_t raw_bar(uint32_t s) const { return w_full + 8 * (s % C::kW); }
    __device__ __forceinline__ bool raw_free(uint32_t s) { return s < C::kW || wait(w_empty + 8 * (s % C::kW), (s / C::kW - 1) & 1); }
    __device__ __forceinline__ uint32_t scales(uint32_t c) const { return base + C::kOffXs + c % C::kXs * COLS * 4; }
    __device__ __forceinline__ uint32_t image(uint32_t c) const { return base + C::kOffB + c % C::kB * C::kBStage; }
    __device__ __forceinline__ uint32_t image_bar(uint32_t c) const { return b_full + 8 * (c % C::kB); }
    __device__ __forceinline__ bool image_free(uint32_t c) { return c < C::kB || wait(b_empty + 8 * (c % C::kB), (c / C::kB - 1) & 1); }

    // A step's sums have a place of their own, so the issuing warps take the steps in turn (one warp alone, with a wait for every barrier,
    // takes 1440 clocks a step).
    template <class P> __device__ __forceinline__ void products(P& p) {
        const uint32_t w = warp - C::kMma;
        grid_dependency_wait();                    // bounded waits begin behind it: the grid before may take as long as it likes
        auto step = [&](uint32_t s, uint32_t c, uint32_t n) {
            const uint32_t panel = n * 128, idesc = umma_idesc_f16(128, n, 0), bs = c % C::kB, ds = s % C::kD, d = tmem + C::kDCol + ds * C::kDCols;
            const uint32_t img_at = C::kOffB + bs * C::kBStage;
            const uint64_t img = umma_desc_sw128(base + img_at);
            // eight rows of zeros, and that far behind them eight rows of the image: Q8_0 the rest (of panel 0), Q4_K hi of the last panel
            const uint64_t apart = umma_desc_sw128(base, img_at + (K == Q4K_8 ? 3 * 2048 : 2048));
            if (!wait(b_full + 8 * bs, (c / C::kB) & 1)) return;
            if (s >= C::kD && !wait(d_empty + 8 * ds, (s / C::kD - 1) & 1)) return;
#pragma unroll
            for (uint32_t h = 0; h < C::kParts; h++) {
                constexpr uint32_t kK = 16 / C::kParts;        // products of a piece
                const uint32_t e = C::kParts * s + h, as = e % C::kA, at = tmem + 8 * kK * as;
                if (!wait(a_full + 8 * as, (e / C::kA) & 1)) return;
                tc_fence_after_sync();
                if (elect_one()) {
#pragma unroll
                    for (uint32_t j = 0; j < kK; j++) {
                        const uint32_t k = h * kK + j, p0 = (k >> 2) * (C::kBlocks ? C::kPanel : panel), sum = K == Q8_0_8 ? d + 16 * (k >> 1) : d;
                        const uint64_t in = (k & 3) * 2, b = img + (p0 >> 4) + in;
                        if (K == Q4K_8 && k >= 12) umma_f16_ts(d, at + 8 * j, apart + (64ull << 32) + in, idesc, 1);
                        else umma_f16_ts(sum, at + 8 * j, K == Q4K_48 ? b + (4 * panel >> 4) : b, idesc, K == Q8_0_8 ? k & 1 : k);
                        if (K == Q8_0_8) umma_f16_ts(sum, at + 8 * j, apart + ((uint64_t)(p0 >> 4) << 32) + in, idesc, 1);
                    }
                    // hi behind lo: the tensor cores cut a sum off at each product, and as long as there is only lo in it, at 2^-11 of the others
#pragma unroll
                    for (uint32_t j = 0; j < kK; j++) {
                        const uint32_t k = h * kK + j;
                        if (K == Q4K_48) umma_f16_ts(d, at + 8 * j, img + ((k >> 2) * panel >> 4) + (k & 3) * 2, idesc, 1);
                        if (K == Q4K_8 && k >= 12) umma_f16_ts(d, at + 8 * j, apart + (k & 3) * 2, idesc, 1);
                    }
                    if (!C::kBlocks && h == 0)
                        umma_f16_ts(d + C::kMOff, tmem + C::kMinCol + 8 * (s % C::kMins), img + ((K == Q4K_8 ? 4 : 8) * panel >> 4), idesc, 0);
                    umma_commit(a_empty + 8 * as);
                    if (h + 1 == C::kParts) {
                        umma_commit(d_full + 8 * ds);
                        umma_commit(b_empty + 8 * bs);
                    }
                }
                __syncwarp();
            }
        };
        if constexpr (K == Q4K_48) {
            const uint32_t i0 = p.begin(), i1 = p.end();
            for (uint32_t i = i0, s0 = 0; i < i1 && ok; i++) {
                const Run r = p.run(i);
                const uint32_t s1 = s0 + (r.u1 - r.u0) * SUBS;
                for (uint32_t s = s0 + (w + C::kMmaWarps - s0 % C::kMmaWarps) % C::kMmaWarps; s < s1 && ok; s += C::kMmaWarps) step(s, s / SUBS, r.n);
                s0 = s1;
            }
        } else {
            const uint32_t steps = p.steps();
            for (uint32_t s = w; s < steps && ok; s += C::kMmaWarps) step(s, s / SUBS, K == Q6K_8R ? 32 : 16);
        }
        // whoever gives up, and when: no product is in flight when the tensor memory goes back
        if (elect_one()) umma_commit(drain + 8 * w);
        __syncwarp();
        mbar_wait(drain + 8 * w, 0);
    }
    // A team takes every kTeams-th piece, whichever rows and columns it is of.
    __device__ __forceinline__ void unpack(uint32_t steps) {
        const uint32_t row = (warp & 3) * 32 + lane, lanes = ((warp & 3) * 32) << 16, pieces = steps * C::kParts;
        // Q6_K: a team's first piece needs nothing but weights, which come ahead of the dependency wait; a raw step of the others waits for its
        // columns' scales as well.  Every bounded wait for something else begins behind it.
        if (!C::kQ6) grid_dependency_wait();
        for (uint32_t e = warp >> 2; e < pieces; e += C::kTeams) {
            const uint32_t s = e / C::kParts, h = e % C::kParts, ws = s % C::kW;
            if (C::kQ6 && e >= C::kTeams && e < 2 * C::kTeams) grid_dependency_wait();
            if (!wait(w_full + 8 * ws, (s / C::kW) & 1)) break;
            const uint8_t* raw = base_p + C::kOffW + ws * C::kWBytes + (C::kQ6 ? 0 : row * C::kUnit);
            uint8_t* const scales = base_p + C::kOffRows + ((s % C::kRows) * 128 + row) * C::kRowScale;
            const uint32_t as = e % C::kA, at = tmem + lanes + 128 / C::kParts * as;
            uint4 head = make_uint4(0, 0, 0, 0);
            if (!C::kBlocks) head = *reinterpret_cast<const uint4*>(raw);
            const Q4KScales sc = q4k_unpack_scales(head.y, head.z, head.w);
            if (e >= C::kA && !wait(a_empty + 8 * as, (e / C::kA - 1) & 1)) break;
            tc_fence_after_sync();
            if constexpr (C::kQ6) {
                const uint32_t r = q6k_row(row) & 7, start = row_start(*reinterpret_cast<volatile uint32_t*>(base_p + C::kOffAt + 4 * ws), r), shift = 8 * (start & 2);
                raw += (16 * r + (q6k_row(row) >> 3)) * C::kUnit + (start & ~3u);
                *reinterpret_cast<uint32_t*>(scales + 4 * h) = unpack_q6k(raw, h, shift, at);
                if (h == 0) *reinterpret_cast<uint32_t*>(scales + 8) = __funnelshift_r(reinterpret_cast<const uint32_t*>(raw)[52], 0u, shift);
            } else if constexpr (C::kBlocks) {
                const uint2 lo = unpack_q8_0<0>(raw, at), hi = unpack_q8_0<1>(raw, at + 64);
                *reinterpret_cast<uint4*>(scales) = make_uint4(lo.x, lo.y, hi.x, hi.y);
            } else {
                if (h == 0) {
                    uint32_t m[8];
#pragma unroll
                    for (int w = 0; w < 4; w++) {       // 32 * minimum, exact
                        const uint32_t b2 = __byte_perm(w < 2 ? sc.ml : sc.mh, 0x64646464u, (w & 1) ? 0x4342u : 0x4140u);
                        m[w] = m[4 + w] = as_u32(__hfma2(as_half2(b2), as_half2(0x50005000u), as_half2(0xF800F800u)));
                    }
                    tmem_st8(tmem + lanes + C::kMinCol + 8 * (s % C::kMins), m);
                    *reinterpret_cast<uint32_t*>(scales) = head.x;
                    unpack_q4k<0>(raw, sc, at);
                    if (C::kParts == 1) unpack_q4k<1>(raw, sc, at + 64);
                } else unpack_q4k<1>(raw, sc, at);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(w_empty + 8 * ws);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full + 8 * as);
        }
    }
    template <class P> __device__ __forceinline__ void sums(P& p) {
        const uint32_t sw = warp - C::kSum0, part = sw >> 2, row = (sw & 3) * 32 + lane, lanes = ((sw & 3) * 32) << 16, i0 = p.begin(), i1 = p.end();
        float acc[SUBS][C::kAcc];
#pragma unroll
        for (int i = 0; i < SUBS * C::kAcc; i++) (&acc[0][0])[i] = 0.f;
        uint32_t s = 0, c = 0;
        grid_dependency_wait();                    // before finish() stores
        for (uint32_t i = i0; i < i1 && ok; i++) {
            const Run r = p.run(i);
            for (uint32_t u = r.u0; u < r.u1 && ok; u++, c++) {
                const float* xs = reinterpret_cast<const float*>(base_p + C::kOffXs) + (c % C::kXs) * COLS;
#pragma unroll
                for (uint32_t sub = 0; sub < SUBS; sub++, s++) {
                    const uint32_t ds = s % C::kD, dt = tmem + lanes + C::kDCol + ds * C::kDCols;
                    const uint8_t* scales = base_p + C::kOffRows + ((s % C::kRows) * 128 + row) * C::kRowScale;
                    float* to = acc[sub];
                    if (!wait(d_full + 8 * ds, (s / C::kD) & 1)) break;
                    tc_fence_after_sync();
                    if constexpr (C::kQ6) {
                        const uint4 d4 = *reinterpret_cast<const uint4*>(scales);
                        const float d = half_bits_to_float(d4.z);
                        uint32_t v[16];
                        float rest[8], t = 0.f;
                        tmem_ld16(dt, v);
                        if (C::kRest) tmem_ld8(dt + 16, rest);
                        tmem_ld_wait();
#pragma unroll
                        for (int b = 0; b < 8; b++) {
                            const float hi = __uint_as_float(v[b]), lo = __uint_as_float(v[8 + b]);
                            t = fmaf(d * (float)(int8_t)((b < 4 ? d4.x : d4.y) >> (8 * (b & 3))), C::kRest ? with_low(hi, lo + rest[b]) : hi + lo, t);
                        }
                        to[0] = fmaf(xs[0], t, to[0]);
                    } else if constexpr (C::kBlocks) {
                        const uint4 d4 = *reinterpret_cast<const uint4*>(scales);
                        const uint32_t dw[4] = {d4.x, d4.y, d4.z, d4.w};
                        // four users, or two: four blocks at a time
                        const uint32_t users = p.few() ? 2 : 4, col = users * part;
                        float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            float hi[4][4], lo[4][4];
#pragma unroll
                            for (int b = 0; b < 4; b++) {
                                tmem_ld4(dt + 16 * (4 * h + b) + col, hi[b]);
                                tmem_ld4(dt + 16 * (4 * h + b) + 8 + col, lo[b]);
                            }
                            tmem_ld_wait();
#pragma unroll
                            for (int b = 0; b < 4; b++) {
                                const uint32_t w = dw[2 * h + (b >> 1)];
                                const float db = half_bits_to_float(b & 1 ? w >> 16 : w);
#pragma unroll
                                for (uint32_t j = 0; j < 4; j++)
                                    if (j < users) t[j] = fmaf(db, with_low(hi[b][j], lo[b][j]), t[j]);
                            }
                        }
#pragma unroll
                        for (uint32_t j = 0; j < 4; j++)
                            if (j < users) to[j] = fmaf(xs[col + j], t[j], to[j]);
                    } else {
                        const uint32_t dd = *reinterpret_cast<const uint32_t*>(scales);
                        const float d = half_bits_to_float(dd & 0xFFFFu), dm = -half_bits_to_float(dd >> 16);
                        if constexpr (K == Q4K_8) {
                            float v0[8], v1[8], mm[8];
                            tmem_ld8(dt, v0);
                            tmem_ld8(dt + 8, v1);
                            tmem_ld8(dt + C::kMOff, mm);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 8; j++) to[j] = fmaf(xs[j], fmaf(d, v0[j] + v1[j], dm * mm[j]), to[j]);
                        } else {
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                const uint32_t col = 8 * (3 * q + part);
                                if (col < r.n) {
                                    float v[8], mm[8];
                                    tmem_ld8(dt + col, v);
                                    tmem_ld8(dt + C::kMOff + col, mm);
                                    tmem_ld_wait();
#pragma unroll
                                    for (int j = 0; j < 8; j++) to[8 * q + j] = fmaf(xs[col + j], fmaf(d, v[j], dm * mm[j]), to[8 * q + j]);
                                }
                            }
                        }
                    }
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty + 8 * ds);
                }
            }
            if (ok) p.finish(i, acc, sw, lane);
        }
    }
    template <class P> __device__ __forceinline__ void work(P& p) {
        if (warp >= C::kMma) products(p);
        else if (warp >= C::kSum0) sums(p);
        else unpack(p.steps());
    }
    __device__ __forceinline__ void leave(int32_t* status) {
        if (!ok) *abort_flag = 1;
        __syncwarp();
        tc_fence_before_sync();
        __syncthreads();
        if (warp == C::kMma) {
            tc_fence_after_sync();
            tmem_dealloc(tmem, 512);
        }
        if (threadIdx.x == 0 && *abort_flag && status) atomicExch(status, 1);
    }
};

}  // namespace tcr
}  // namespace runit
