// Fused-dequant GEMVs for the formats the reference only dequantises on the CPU at load time: Q5_0, Q5_K and Q6_K
// (crates/engine/src/forward.rs:900-949, 979-1012; files quantised as "Q4_K_M" mix them in: Q6_K for ffn_down and the
// output matrix, Q5_0 / Q5_K in some attention matrices, docs/STATUS_REPORT.md:19-27).  The reference expands such
// tensors to f32 or f16 and runs its f16 GEMV on them; here they stay packed in HBM (0.69 / 0.69 / 0.82 bytes per weight
// instead of 2) and are decoded in registers, so a decode step streams 2.4 - 2.9 times fewer bytes for them.
//
// Kernel: one warp per row, lane l decodes 8 of the 256 weights of a unit (a Q5_K / Q6_K superblock, or 8 Q5_0 blocks)
// exactly as the reference's loops index them; the packed bytes of 4 units at a time arrive through a per-warp ring of
// three cp.async stages that runs across the warp's rows (rows are only 2- or 4-byte aligned in these formats, so the
// copies are 4-byte ones from the aligned word below); f32 accumulation, shuffle reduction, optional f32 residual.
// HBM-bound in principle; at ~7 instructions per weight it is issue-bound at roughly half the HBM rate on B200.
#include "gemv_common.cuh"
#include "gemv_int8.cuh"
#include "runit_internal.h"
#include "tma.cuh"

namespace runit {
namespace kq {

constexpr int kWarps = 8;       // per CTA
constexpr int kChunk = 4;       // units per stage
constexpr int kStages = 3;

template <int FMT> struct KTraits;
template <> struct KTraits<RUNIT_FMT_Q5_0> { static constexpr int UB = 176; };   // 8 blocks of 22 bytes
template <> struct KTraits<RUNIT_FMT_Q5K>  { static constexpr int UB = 176; };
template <> struct KTraits<RUNIT_FMT_Q6K>  { static constexpr int UB = 210; };

// Partial dot product of this lane's 8 weights of one unit with x (xu = the unit's 256 activations in global memory).
template <int FMT>
__device__ __forceinline__ float unit_dot(const uint8_t* u, const float* __restrict__ xu, int lane, int nblk) {
    float acc = 0.f;
    if (FMT == RUNIT_FMT_Q6K) {
        // forward.rs:920-949: {ql[128]; qh[64]; i8 scales[16]; f16 d}
        const float d = half_bits_to_float((uint32_t)u[208] | ((uint32_t)u[209] << 8));
        const int8_t* sc = reinterpret_cast<const int8_t*>(u + 192);
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int a = u[64 * half + lane], c = u[64 * half + lane + 32], h = u[128 + 32 * half + lane];
            const int q1 = ((a & 15) | ((h & 3) << 4)) - 32, q2 = ((c & 15) | (((h >> 2) & 3) << 4)) - 32;
            const int q3 = ((a >> 4) | (((h >> 4) & 3) << 4)) - 32, q4 = ((c >> 4) | (((h >> 6) & 3) << 4)) - 32;
            const float* xh = xu + 128 * half + lane;
            float s = (float)sc[8 * half + 0] * ((float)q1 * xh[0]);
            s = fmaf((float)sc[8 * half + 2], (float)q2 * xh[32], s);
            s = fmaf((float)sc[8 * half + 4], (float)q3 * xh[64], s);
            s = fmaf((float)sc[8 * half + 6], (float)q4 * xh[96], s);
            acc = fmaf(d, s, acc);
        }
    } else if (FMT == RUNIT_FMT_Q5K) {
        // forward.rs:979-1012: {f16 d; f16 dmin; scales[12]; qh[32]; qs[128]}; fifth bit of element e = bit e%8 of qh[e/8]
        const uint32_t h0 = *reinterpret_cast<const uint16_t*>(u) | ((uint32_t)*reinterpret_cast<const uint16_t*>(u + 2) << 16);
        const float d = half_bits_to_float(h0), dmin = half_bits_to_float(h0 >> 16);
        const uint8_t* s = u + 4;
        const uint8_t* qh = u + 16;
        const uint8_t* qs = u + 48;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            // get_scale_min_k4 (forward.rs:359-369) for indices j and j + 4
            const float sc_lo = (float)(s[j] & 63), m_lo = (float)(s[j + 4] & 63);
            const float sc_hi = (float)((s[j + 8] & 15) | ((s[j] >> 6) << 4)), m_hi = (float)((s[j + 8] >> 4) | ((s[j + 4] >> 6) << 4));
            const int v = qs[32 * j + lane];
            const int e_lo = 64 * j + lane, e_hi = e_lo + 32;
            const int q_lo = (v & 15) | (((qh[e_lo >> 3] >> (e_lo & 7)) & 1) << 4);
            const int q_hi = (v >> 4) | (((qh[e_hi >> 3] >> (e_hi & 7)) & 1) << 4);
            const float x_lo = xu[e_lo], x_hi = xu[e_hi];
            acc = fmaf(d * sc_lo * (float)q_lo - dmin * m_lo, x_lo, acc);
            acc = fmaf(d * sc_hi * (float)q_hi - dmin * m_hi, x_hi, acc);
        }
    } else {
        // forward.rs:900-919: blocks {f16 d; qh[4]; qs[16]}; lane l: block l / 4, bytes 4 (l % 4) .. + 3
        const int b = lane >> 2, j0 = (lane & 3) * 4;
        if (b < nblk) {
            const uint8_t* blk = u + 22 * b;
            const float d = half_bits_to_float((uint32_t)blk[0] | ((uint32_t)blk[1] << 8));
            const uint32_t qh = (uint32_t)blk[2] | ((uint32_t)blk[3] << 8) | ((uint32_t)blk[4] << 16) | ((uint32_t)blk[5] << 24);
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int j = j0 + i, v = blk[6 + j];
                const int x0 = (v & 15) | (((qh >> j) & 1) << 4), x1 = (v >> 4) | (((qh >> (j + 16)) & 1) << 4);
                s = fmaf((float)(x0 - 16), xu[32 * b + j], s);
                s = fmaf((float)(x1 - 16), xu[32 * b + j + 16], s);
            }
            acc = d * s;
        }
    }
    return acc;
}

struct Args {
    const uint8_t* w;
    const float* x;
    float* y;
    const float* res;
    uint32_t m, k, n_units, row_bytes, nb;   // nb: 32-blocks per row (Q5_0: the last unit may hold fewer than 8)
};

template <int FMT>
__global__ void __launch_bounds__(kWarps * 32) gemv_kquant_kernel(const Args a) {
    constexpr int UB = KTraits<FMT>::UB;
    constexpr int SB = (kChunk * UB + 4 + 15) / 16 * 16;   // stage bytes: the chunk plus the alignment shift
    __shared__ __align__(16) uint8_t ring[kWarps][kStages][SB];
    grid_dependency_wait();
    grid_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gw = blockIdx.x * kWarps + warp, n_warps = gridDim.x * kWarps;
    if (gw >= a.m) return;
    const uint32_t n_chunks = (a.n_units + kChunk - 1) / kChunk;
    const uint32_t my_rows = (a.m - gw + n_warps - 1) / n_warps;
    const uint32_t n_steps = my_rows * n_chunks;   // (row, chunk) pairs of this warp, in order

    // chunk t of this warp: row gw + (t / n_chunks) * n_warps, units [c * kChunk, ...)
    auto issue = [&](uint32_t t) {
        if (t < n_steps) {
            const uint32_t row = gw + (t / n_chunks) * n_warps, c = t % n_chunks;
            const uint32_t units = min((uint32_t)kChunk, a.n_units - c * kChunk);
            const size_t start = (size_t)row * a.row_bytes + (size_t)c * kChunk * UB;
            const size_t bytes = FMT == RUNIT_FMT_Q5_0 ? min((size_t)units * UB, (size_t)a.row_bytes - (size_t)c * kChunk * UB) : (size_t)units * UB;
            const uint32_t shift = (uint32_t)((reinterpret_cast<uintptr_t>(a.w) + start) & 3u);
            const uint8_t* src = a.w + start - shift;
            const uint32_t words = (uint32_t)((shift + bytes + 3) / 4);
            const uint32_t dst = smem_u32(&ring[warp][t % kStages][0]);
            for (uint32_t wd = lane; wd < words; wd += 32) cp_async4(dst + 4 * wd, src + 4 * (size_t)wd);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < kStages - 1; s++) issue(s);
    float acc = 0.f;
    for (uint32_t t = 0; t < n_steps; t++) {
        issue(t + kStages - 1);
        cp_async_wait<kStages - 1>();
        __syncwarp();
        const uint32_t row = gw + (t / n_chunks) * n_warps, c = t % n_chunks;
        const uint32_t units = min((uint32_t)kChunk, a.n_units - c * kChunk);
        const size_t start = (size_t)row * a.row_bytes + (size_t)c * kChunk * UB;
        const uint32_t shift = (uint32_t)((reinterpret_cast<uintptr_t>(a.w) + start) & 3u);
        const uint8_t* base = &ring[warp][t % kStages][shift];
        for (uint32_t i = 0; i < units; i++) {
            const uint32_t u = c * kChunk + i;
            const int nblk = FMT == RUNIT_FMT_Q5_0 ? min(8, (int)(a.nb - u * 8u)) : 8;
            acc += unit_dot<FMT>(base + i * UB, a.x + (size_t)u * 256, lane, nblk);
        }
        __syncwarp();   // the stage may be refilled by the next issue
        if (c + 1 == n_chunks) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) a.y[row] = a.res ? a.res[row] + acc : acc;
            acc = 0.f;
        }
    }
    cp_async_wait<0>();
}

// ───────────────────────── Q6_K and Q5_K, tile kernel ─────────────────────────
// Every warp owns a tile of 32 rows and walks all 256-weight units of K (4 tiles per CTA), or a share of them (split).  Per unit it
// copies the rows' packed bytes into its own two-stage ring together with the 256 activations, which it turns into three signed
// 8-bit limbs per element with one power-of-two scale per 32 (prep_int_block: 23 bits, exact to f32 rounding).  The 5- and 6-bit
// fields, unsigned bytes once their upper bits are merged in, are the A operand of mma.sync.m16n8k32, one MMA per 16 rows x 32 weights:
//   * the eight columns carry limbs 0 and 1 of FOUR blocks at once: column n holds limb n & 1 of block n >> 1 of a group of four and
//     zeros in the MMAs of the group's other blocks, so four MMAs add into one register tile;
//   * limb 2 of all eight blocks goes the same way into a second tile, column n = block (n >> 1) + 4 (n & 1), so that lane
//     (g, t) ends up with every limb's exact sums of blocks t and t + 4 of its rows g and g + 8.
// 16 MMAs for 16 rows x 256 weights; integers, combination and error against 64 bits are those of dp4a on the same limbs.
// Bound: instruction issue (unpacking, the activations' limbs where they are not prepared) at 11 warps per SM, which the stages'
// shared memory allows.  Measured, lane = row with dp4a before: Q6_K 152064 x 3584 164 -> 133 us (125 in a stream over three matrices,
// 3.6 TB/s), 3584 x 18944 25.6 -> 22.4, 32000 x 2048 26.1 -> 23.5; Q5_K 152064 x 3584 106 -> 100, 3584 x 3584 8.4 -> 7.8.
namespace kt {

template <int FMT> struct Tile {
    static constexpr int kUnit = FMT == RUNIT_FMT_Q6K ? 210 : 176;
    // Q6_K rows start on even bytes only: the unit arrives as the 16-byte pieces that hold it (14 of them) and is read from its
    // offset; 240 and 176 are odd multiples of 16, which spreads the eight rows of a fragment over the banks
    static constexpr int kPitch = FMT == RUNIT_FMT_Q6K ? 240 : 176;
    static constexpr int kXOff = 32 * kPitch, kStage = kXOff + 1024, kSmem = 4 * 2 * kStage;
};
constexpr int kS = 2;

struct Args {
    const uint8_t* w;
    const float* x;
    float* y;
    const float* res;
    uint32_t m, nb, row_bytes;
    // split > 0 (matrices with few rows): a CTA owns ONE tile and one of `split` shares of K; its 4 warps take every
    // 4 * split-th superblock each, the CTA files one partial sum per row in part[share][row], and the CTA that takes the
    // last of the tile's tickets adds the shares in order (deterministic) and stores the rows.
    uint32_t split;
    float* part;
    uint32_t* tickets;       // one word per tile, zero at rest
    const uint8_t* xq;       // PRE: the prepared activations, kXq bytes per unit
    uint32_t wait_first;     // the predecessor may be a kernel that writes the weights
};
constexpr int kXq = IntX<8>::BYTES;                  // 832: a multiple of 16

// The activations' limbs, scales and sums, once per call: one warp per unit.
__global__ void __launch_bounds__(32) kquant_prepare_kernel(const float* __restrict__ x, uint8_t* __restrict__ xq) {
    __shared__ __align__(16) uint8_t out[kXq];
    grid_launch_dependents();                        // the GEMV may request its first weights
    grid_dependency_wait();
    const int lane = threadIdx.x;
    const float4* xr = reinterpret_cast<const float4*>(x + (size_t)blockIdx.x * 256) + 2 * lane;
    const float4 a = xr[0], b = xr[1];
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    prep_int_block<8, 8, 0>(out, v, lane);
    __syncwarp();
    uint4* dst = reinterpret_cast<uint4*>(xq + (size_t)blockIdx.x * kXq);
    dst[lane] = reinterpret_cast<const uint4*>(out)[lane];
    if (lane < kXq / 16 - 32) dst[32 + lane] = reinterpret_cast<const uint4*>(out)[32 + lane];
}

__device__ __forceinline__ uint32_t ld32(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

// Unpacked words of 16 rows x one block for this lane: a[0], a[1] = first word of rows g and g + 8, a[2], a[3] = second word.
// Words 2t and 2t + 1 of the block's eight.
template <int FMT> struct Rows;

template <> struct Rows<RUNIT_FMT_Q6K> {             // forward.rs:920-949
    const uint8_t* p[2];                             // the rows' units; even addresses
    uint32_t q[2][4][2];                             // [row][group of 32 of the half][word]
    __device__ __forceinline__ void init(const uint8_t* r0, const uint8_t* r1) { p[0] = r0; p[1] = r1; }
    __device__ __forceinline__ void load(int b, int t) {
        if (b & 3) return;
        const int h = b >> 2;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint8_t* al = p[r] - (reinterpret_cast<uintptr_t>(p[r]) & 2u);
            const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(p[r]) & 2u) * 8u;
            auto pair = [&](int off, uint32_t& w0, uint32_t& w1) {
                const uint32_t x0 = ld32(al + off), x1 = ld32(al + off + 4), x2 = ld32(al + off + 8);
                w0 = __funnelshift_r(x0, x1, sh);
                w1 = __funnelshift_r(x1, x2, sh);
            };
            uint32_t a[2], c[2], u[2];
            pair(64 * h + 8 * t, a[0], a[1]);
            pair(64 * h + 32 + 8 * t, c[0], c[1]);
            pair(128 + 32 * h + 8 * t, u[0], u[1]);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                q[r][0][i] = (a[i] & 0x0F0F0F0Fu) | ((u[i] << 4) & 0x30303030u);
                q[r][1][i] = (c[i] & 0x0F0F0F0Fu) | ((u[i] << 2) & 0x30303030u);
                q[r][2][i] = ((a[i] >> 4) & 0x0F0F0F0Fu) | (u[i] & 0x30303030u);
                q[r][3][i] = ((c[i] >> 4) & 0x0F0F0F0Fu) | ((u[i] >> 2) & 0x30303030u);
            }
        }
    }
    __device__ __forceinline__ uint32_t word(int b, int r, int i) const { return q[r][b & 3][i]; }
    // d * scale * (sum q v - 32 sum v) * s of block b = t + 4 * gr; the reference takes scales[2 b]
    __device__ __forceinline__ float value(int gr, int r, int t, float dot, float sx, float sv) const {
        const int b = t + 4 * gr;
        const float d = __half2float(*reinterpret_cast<const __half*>(p[r] + 208));
        const float sc = (float)reinterpret_cast<const int8_t*>(p[r])[192 + 2 * b];
        return d * ((sc * sx) * (dot - 32.f * sv));
    }
};

template <> struct Rows<RUNIT_FMT_Q5K> {             // forward.rs:979-1012
    const uint8_t* p[2];                             // 16-byte aligned
    uint32_t q[2][2][2];                             // [row][low, high nibbles of the chunk][word]
    __device__ __forceinline__ void init(const uint8_t* r0, const uint8_t* r1) { p[0] = r0; p[1] = r1; }
    __device__ __forceinline__ void load(int b, int t) {
        if (b & 1) return;
        const int j = b >> 1;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint2 w = *reinterpret_cast<const uint2*>(p[r] + 48 + 32 * j + 8 * t);
            // this lane's eight elements of a block have their fifth bits in one byte
            const uint32_t fl = p[r][16 + 8 * j + t], fh = p[r][16 + 8 * j + 4 + t];
            q[r][0][0] = (w.x & 0x0F0F0F0Fu) | (((fl & 15u) * 0x02040810u) & 0x10101010u);
            q[r][0][1] = (w.y & 0x0F0F0F0Fu) | (((fl >> 4) * 0x02040810u) & 0x10101010u);
            q[r][1][0] = ((w.x >> 4) & 0x0F0F0F0Fu) | (((fh & 15u) * 0x02040810u) & 0x10101010u);
            q[r][1][1] = ((w.y >> 4) & 0x0F0F0F0Fu) | (((fh >> 4) * 0x02040810u) & 0x10101010u);
        }
    }
    __device__ __forceinline__ uint32_t word(int b, int r, int i) const { return q[r][b & 1][i]; }
    __device__ __forceinline__ float value(int gr, int r, int t, float dot, float sx, float sv) const {
        const uint4 hd = *reinterpret_cast<const uint4*>(p[r]);                                // d, dmin, packed scales and mins
        const float d = half_bits_to_float(hd.x), dmin = half_bits_to_float(hd.x >> 16);
        const Q4KScales s = q4k_unpack_scales(hd.y, hd.z, hd.w);
        const uint32_t sel = 0x4440u + (uint32_t)((t >> 1) + 2 * gr);                          // block b: index b / 2, + 4 if odd
        const float sc = (float)__byte_perm((t & 1) ? s.sh : s.sl, 0u, sel), mn = (float)__byte_perm((t & 1) ? s.mh : s.ml, 0u, sel);
        return sx * (d * sc * dot - dmin * mn * sv);
    }
};

// PRE: the activations were prepared by a launch of their own (their limbs are a sixth of the instructions per unit otherwise).
template <int FMT, bool PRE>
__global__ void __launch_bounds__(128) gemv_kquant_tile_kernel(const Args a) {
    using T = Tile<FMT>;
    extern __shared__ __align__(16) uint8_t kt_smem[];
    __shared__ float red[4][32];
    __shared__ uint32_t s_last;
    grid_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    uint8_t* ring = kt_smem + warp * (kS * T::kStage);
    // split == 0: every warp owns a tile of 32 rows and walks all of K; else the CTA owns tile blockIdx.x
    const uint32_t row0 = a.split ? blockIdx.x * 32 : (blockIdx.x * 4 + warp) * 32;
    if (row0 >= a.m) return;
    const uint32_t rows_here = min(32u, a.m - row0);
    const uint32_t u0 = a.split ? blockIdx.y * 4 + warp : 0u, ustep = a.split ? 4u * a.split : 1u;
    const int n_it = u0 < a.nb ? (int)((a.nb - u0 + ustep - 1) / ustep) : 0;
    const size_t first = (size_t)row0 * a.row_bytes, total = (size_t)a.m * a.row_bytes;

    auto issue_w = [&](int it) {
        if (it >= n_it) return;
        const uint32_t u = u0 + ustep * (uint32_t)it;
        const uint32_t st = smem_u32(ring + (it % kS) * T::kStage);
        if (FMT == RUNIT_FMT_Q6K) {
            // four lanes per row, 16-byte pieces 4 i + t from the one that holds the unit's first byte (the matrix itself is
            // 16-byte aligned); nothing is read past the matrix
            const bool inner = row0 + 32 < a.m;      // a row follows: whole pieces
#pragma unroll
            for (int rg = 0; rg < 4; rg++) {
                const uint32_t r = 8 * rg + g;
                const size_t from = (first + (size_t)r * a.row_bytes + (size_t)u * 210) & ~(size_t)15;
                const uint8_t* src = a.w + from + 16 * t;
                const uint32_t dst = st + r * T::kPitch + 16 * t;
                if (inner) {
#pragma unroll
                    for (int i = 0; i < 3; i++) cp_async16(dst + 64 * i, src + 64 * i);
                    if (t < 2) cp_async16(dst + 192, src + 192);
                } else if (r < rows_here) {
                    const uint32_t left = (uint32_t)min((size_t)256, total - from);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const uint32_t at = 64 * i + 16 * t;
                        if (at < left && at < 224)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + 64 * i), "l"(src + 64 * i), "r"(min(16u, left - at)) : "memory");
                    }
                }
            }
        } else {
            const uint8_t* base = a.w + first + (size_t)u * 176;
#pragma unroll
            for (int i = 0; i < 11; i++) {
                const uint32_t c = (uint32_t)lane + 32u * i, r = c / 11u, col = c - 11u * r;      // 352 chunks of 16 bytes
                if (r < rows_here) cp_async16(st + r * T::kPitch + 16 * col, base + (size_t)r * a.row_bytes + 16 * col);
            }
        }
    };
    auto issue_x = [&](int it) {
        if (it < n_it) {
            const uint32_t u = u0 + ustep * (uint32_t)it, st = smem_u32(ring + (it % kS) * T::kStage) + T::kXOff;
            const uint8_t* xu = PRE ? a.xq + (size_t)u * kXq : reinterpret_cast<const uint8_t*>(a.x + (size_t)u * 256);
            cp_async16(st + 16 * lane, xu + 16 * lane);
            if (!PRE || lane < kXq / 16 - 32) cp_async16(st + 16 * (32 + lane), xu + 16 * (32 + lane));
        }
        cp_async_commit();
    };
    // the weights do not depend on the kernel before, unless it is the caller's own; its output may be x or the residual
    if (a.wait_first) grid_dependency_wait();
#pragma unroll
    for (int s = 0; s < kS; s++) issue_w(s);
    grid_dependency_wait();
#pragma unroll
    for (int s = 0; s < kS; s++) issue_x(s);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};             // rows g, g + 8, g + 16, g + 24, this lane's blocks
    for (int it = 0; it < n_it; it++) {
        cp_async_wait<kS - 1>();
        __syncwarp();
        uint8_t* stg = ring + (it % kS) * T::kStage;
        if (!PRE) {   // activations of the unit -> limbs, scales, block sums (in place)
            float v[8];
            const float4* xr = reinterpret_cast<const float4*>(stg + T::kXOff) + 2 * lane;
            const float4 t0 = xr[0], t1 = xr[1];
            v[0] = t0.x; v[1] = t0.y; v[2] = t0.z; v[3] = t0.w; v[4] = t1.x; v[5] = t1.y; v[6] = t1.z; v[7] = t1.w;
            __syncwarp();
            prep_int_block<8, 8, 0>(stg + T::kXOff, v, lane);
            __syncwarp();
        }
        const uint8_t* xq = stg + T::kXOff;
        // this lane's column: limb g & 1 of blocks g >> 1 and (g >> 1) + 4; limb 2 of block (g >> 1) + 4 (g & 1)
        uint32_t bx[2][2], bz[2];
        {
            const uint8_t *c0 = xq + (g >> 1) * 96 + (g & 1) * 32, *c1 = c0 + 4 * 96, *cz = xq + ((g >> 1) + 4 * (g & 1)) * 96 + 64;
            const int o0 = 8 * t, o1 = 8 * t + 4;
            bx[0][0] = ld32(c0 + o0); bx[0][1] = ld32(c0 + o1);
            bx[1][0] = ld32(c1 + o0); bx[1][1] = ld32(c1 + o1);
            bz[0] = ld32(cz + o0); bz[1] = ld32(cz + o1);
        }
        uint32_t shift[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            shift[i] = FMT == RUNIT_FMT_Q6K ? (uint32_t)(first + (size_t)(8 * i + g) * a.row_bytes + (size_t)(u0 + ustep * (uint32_t)it) * 210) & 15u : 0u;
        const float* sx = reinterpret_cast<const float*>(xq + IntX<8>::SCALE);
        const int* sv = reinterpret_cast<const int*>(xq + IntX<8>::VSUM);
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
            Rows<FMT> rows;
            rows.init(stg + (16 * mt + g) * T::kPitch + shift[2 * mt], stg + (16 * mt + 8 + g) * T::kPitch + shift[2 * mt + 1]);
            int c[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}}, z[4] = {0, 0, 0, 0};
#pragma unroll
            for (int b = 0; b < 8; b++) {
                rows.load(b, t);
                const bool mine = (g >> 1) == (b & 3), third = mine && (g & 1) == (b >> 2);
                const uint32_t a0 = rows.word(b, 0, 0), a1 = rows.word(b, 1, 0), a2 = rows.word(b, 0, 1), a3 = rows.word(b, 1, 1);
                mma_u8s8_acc(c[b >> 2], a0, a1, a2, a3, mine ? bx[b >> 2][0] : 0u, mine ? bx[b >> 2][1] : 0u);
                mma_u8s8_acc(z, a0, a1, a2, a3, third ? bz[0] : 0u, third ? bz[1] : 0u);
            }
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int gr = 0; gr < 2; gr++) {
                    // sum q * v over the block, exact in every limb
                    const float dot = fmaf((float)z[2 * r + gr], 65536.f, (float)(c[gr][2 * r + 1] * 256 + c[gr][2 * r]));   // |.| < 63 * 32 * 128 * 257 < 2^27
                    acc[2 * mt + r] += rows.value(gr, r, t, dot, sx[t + 4 * gr], (float)sv[t + 4 * gr]);
                }
        }
        __syncwarp();
        issue_w(it + kS);
        issue_x(it + kS);
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < 4; i++) {
        acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 1);
        acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 2);
        if (t == 0) red[warp][8 * i + g] = acc[i];
    }
    if (a.split == 0) {
        __syncwarp();
        if ((uint32_t)lane < rows_here) {
            const uint32_t row = row0 + lane;
            const float v = red[warp][lane];
            a.y[row] = a.res ? a.res[row] + v : v;
        }
        return;
    }
    __syncthreads();
    if (warp == 0) {
        const float v = ((red[0][lane] + red[1][lane]) + red[2][lane]) + red[3][lane];
        if ((uint32_t)lane < rows_here) __stcg(&a.part[(size_t)blockIdx.y * a.m + row0 + lane], v);
        __threadfence();
        __syncwarp();
        if (lane == 0) s_last = atomicAdd(&a.tickets[blockIdx.x], 1u) == a.split - 1;
    }
    __syncthreads();
    if (s_last && warp == 0) {
        __threadfence();
        if ((uint32_t)lane < rows_here) {
            const uint32_t row = row0 + lane;
            float v = a.res ? a.res[row] : 0.f;
            for (uint32_t sp = 0; sp < a.split; sp++) v += __ldcg(&a.part[(size_t)sp * a.m + row]);
            a.y[row] = v;
        }
        if (lane == 0) a.tickets[blockIdx.x] = 0;
    }
}

}  // namespace kt

// ───────────────────────── Q5_0, tile kernel ─────────────────────────
// Lane = row, three dp4a per four weights.  (On the MMAs of the kernel above, whose fragments re-read a block's fifth bits in four
// lanes, 18944 x 3584 took 21.9 us against 18.6.)  K a multiple of 256: a unit is eight 22-byte blocks (176 bytes, 256 weights),
// rows are then multiples of 176 bytes and the copy is the Q5_K one (16-byte cp.async, pitch 176).  Inside the unit the blocks alternate between
// word-aligned and two bytes off, which a compile-time funnel shift takes care of.  A word of qs gives four low-nibble weights (elements 4 g ..) and four
// high-nibble weights (elements 16 + 4 g ..); their fifth bits are nibbles g and 4 + g of qh (forward.rs:900-918); the
// "- 16" is taken through the block's sum of activations.
namespace q50t {

constexpr int kPitch = 176;
constexpr int kXOff = 32 * kPitch;
constexpr int kStage = kXOff + 1024;
constexpr int kS = 2;

__global__ void __launch_bounds__(128) gemv_q5_0_tile_kernel(const kt::Args a) {
    extern __shared__ __align__(16) uint8_t q50_smem[];
    __shared__ float red[4][32];
    __shared__ uint32_t s_last;
    grid_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* ring = q50_smem + warp * (kS * kStage);
    const uint32_t row0 = a.split ? blockIdx.x * 32 : (blockIdx.x * 4 + warp) * 32;
    if (row0 >= a.m) return;
    const uint32_t rows_here = min(32u, a.m - row0);
    const uint32_t u0 = a.split ? blockIdx.y * 4 + warp : 0u, ustep = a.split ? 4u * a.split : 1u;
    const int n_it = u0 < a.nb ? (int)((a.nb - u0 + ustep - 1) / ustep) : 0;

    auto issue = [&](int it) {
        if (it < n_it) {
            const uint32_t u = u0 + ustep * (uint32_t)it;
            const uint32_t st = smem_u32(ring + (it % kS) * kStage);
            const uint8_t* base = a.w + (size_t)row0 * a.row_bytes + (size_t)u * 176;
#pragma unroll
            for (int i = 0; i < 11; i++) {
                const uint32_t c = (uint32_t)lane + 32u * i, r = c / 11u, col = c - 11u * r;
                if (r < rows_here) cp_async16(st + r * kPitch + 16 * col, base + (size_t)r * a.row_bytes + 16 * col);
            }
            const float* xu = a.x + (size_t)u * 256;
            cp_async16(st + kXOff + 16 * lane, xu + 4 * lane);
            cp_async16(st + kXOff + 16 * (32 + lane), xu + 4 * (32 + lane));
        }
        cp_async_commit();
    };
    grid_dependency_wait();
#pragma unroll
    for (int s = 0; s < kS; s++) issue(s);
    float acc = 0.f;
    for (int it = 0; it < n_it; it++) {
        cp_async_wait<kS - 1>();
        __syncwarp();
        uint8_t* stg = ring + (it % kS) * kStage;
        {
            float v[8];
            const float4* xr = reinterpret_cast<const float4*>(stg + kXOff) + 2 * lane;
            const float4 t0 = xr[0], t1 = xr[1];
            v[0] = t0.x; v[1] = t0.y; v[2] = t0.z; v[3] = t0.w; v[4] = t1.x; v[5] = t1.y; v[6] = t1.z; v[7] = t1.w;
            __syncwarp();
            prep_int_block<8, 8, 0>(stg + kXOff, v, lane);
            __syncwarp();
        }
        if ((uint32_t)lane < rows_here) {
            const uint4* ru = reinterpret_cast<const uint4*>(stg + lane * kPitch);
            uint32_t al[45];                         // the unit's 44 words (al[44] only feeds discarded bytes)
#pragma unroll
            for (int j = 0; j < 11; j++) {
                const uint4 t = ru[j];
                al[4 * j] = t.x; al[4 * j + 1] = t.y; al[4 * j + 2] = t.z; al[4 * j + 3] = t.w;
            }
            al[44] = 0;
            // 32 bits at the (even, compile-time) byte offset e of the unit
            auto F = [&](int e) -> uint32_t { return (e & 3) ? __funnelshift_r(al[e >> 2], al[(e >> 2) + 1], 16) : al[e >> 2]; };
            const uint8_t* xq = stg + kXOff;
            const float* sx = reinterpret_cast<const float*>(xq + IntX<8>::SCALE);
            const int* sv = reinterpret_cast<const int*>(xq + IntX<8>::VSUM);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const float d = half_bits_to_float(F(22 * b) & 0xFFFFu);
                const uint32_t qh = F(22 * b + 2);
                const uint4* xl = reinterpret_cast<const uint4*>(xq + b * 96);
                int s0 = 0, s1 = 0, s2 = 0;
                uint32_t w[4];
#pragma unroll
                for (int g = 0; g < 4; g++) w[g] = F(22 * b + 6 + 4 * g);
#pragma unroll
                for (int hf = 0; hf < 2; hf++) {
                    const uint4 l0 = xl[hf], l1 = xl[2 + hf], l2 = xl[4 + hf];
                    const uint32_t x0[4] = {l0.x, l0.y, l0.z, l0.w}, x1[4] = {l1.x, l1.y, l1.z, l1.w}, x2[4] = {l2.x, l2.y, l2.z, l2.w};
#pragma unroll
                    for (int g = 0; g < 4; g++) {
                        const uint32_t nib = (qh >> (16 * hf + 4 * g)) & 15u;
                        const uint32_t q = ((hf ? (w[g] >> 4) : w[g]) & 0x0F0F0F0Fu) | (((nib * 0x00204081u) & 0x01010101u) << 4);
                        s0 = dp4a_us(q, x0[g], s0);
                        s1 = dp4a_us(q, x1[g], s1);
                        s2 = dp4a_us(q, x2[g], s2);
                    }
                }
                const float dot = fmaf((float)s2, 65536.f, fmaf((float)s1, 256.f, (float)s0)) - 16.f * (float)sv[b];
                acc = fmaf(d * sx[b], dot, acc);
            }
        }
        __syncwarp();
        issue(it + kS);
    }
    cp_async_wait<0>();
    if (a.split == 0) {
        if ((uint32_t)lane < rows_here) {
            const uint32_t row = row0 + lane;
            a.y[row] = a.res ? a.res[row] + acc : acc;
        }
        return;
    }
    red[warp][lane] = acc;
    __syncthreads();
    if (warp == 0) {
        const float v = ((red[0][lane] + red[1][lane]) + red[2][lane]) + red[3][lane];
        if ((uint32_t)lane < rows_here) __stcg(&a.part[(size_t)blockIdx.y * a.m + row0 + lane], v);
        __threadfence();
        __syncwarp();
        if (lane == 0) s_last = atomicAdd(&a.tickets[blockIdx.x], 1u) == a.split - 1;
    }
    __syncthreads();
    if (s_last && warp == 0) {
        __threadfence();
        if ((uint32_t)lane < rows_here) {
            const uint32_t row = row0 + lane;
            float v = a.res ? a.res[row] : 0.f;
            for (uint32_t sp = 0; sp < a.split; sp++) v += __ldcg(&a.part[(size_t)sp * a.m + row]);
            a.y[row] = v;
        }
        if (lane == 0) a.tickets[blockIdx.x] = 0;
    }
}

}  // namespace q50t

template <int FMT>
static int32_t launch(runit_ctx* ctx, const char* name, const void* w, const void* x, void* y, const void* res, uint32_t m, uint32_t k) {
    if (!ctx) return RUNIT_ERR_BAD_ARG;
    RUNIT_REQUIRE(ctx, w && x && y, "%s: null pointer", name);
    RUNIT_REQUIRE(ctx, m > 0 && m <= (1u << 28), "%s: m=%u out of range", name, m);
    const uint32_t be = FMT == RUNIT_FMT_Q5_0 ? 32u : 256u;
    RUNIT_REQUIRE(ctx, k > 0 && k % be == 0 && k <= (1u << 24), "%s: k=%u is not a positive multiple of %u", name, k, be);
    RUNIT_REQUIRE(ctx, runit_aligned(w, 16) && runit_aligned(x, 16) && runit_aligned(y, 4) && (!res || runit_aligned(res, 4)),
                  "%s: weights and input 16-byte aligned, output 4-byte aligned", name);
    // Q6_K on the tensor cores, from 64 tiles of 128 rows on (us, the kernels below / tensor cores: 8192 rows of K = 256 5.7 / 4.8, 2048 9.5 / 8.6, 3584 13.6 / 10.4,
    // 14336 34 / 30; 12000 x 1024 10.9 / 7.9, 18944 x 3584 24 / 14, 40000 x 3584 50 / 28, 152064 x 3584 127 / 87, 128256 x 4096 120 / 95; 4096 rows of
    // K = 512 5.7 / 6.9, 3584 8.7 / 8.1, 14336 20.4 / 20.2; 2560 x 14336 13.4 / 15.2)
    if (FMT == RUNIT_FMT_Q6K && m >= 8192 && ctx->tune.kquant_variant == 0 && ctx->tune.kquant_prepare == 0 && ctx->tune.kquant_split == 0 &&
        gemv_q6k_tc_applies(ctx, w, m, k))
        return gemv_q6k_tc(ctx, name, w, (const float*)x, (float*)y, (const float*)res, m, k);
    // the tile kernel needs a tile of 32 rows per warp: with fewer than two warps' worth of tiles per scheduler the first
    // kernel (one warp per row) keeps more of the machine busy
    if ((FMT != RUNIT_FMT_Q5_0 || k % 256 == 0) && ctx->tune.kquant_variant != 1) {
        kt::Args t;
        const uint32_t tiles = (m + 31) / 32, sms = (uint32_t)ctx->sm_count, nbk = k / 256;
        // few tiles: shares of K go to different CTAs (2..16 shares, about one superblock per warp at least, fewer than 8 CTAs
        // per SM; measured on 3584 x 3584: 4 shares 15 -> 9 us, and on 18944 x 3584 two shares gain nothing)
        uint32_t split = 0;
        if (tiles < 8 * sms && ctx->d_kq && tiles <= 2048 && nbk >= 8) {
            split = 1;
            while (split < 16 && tiles * split * 2 < 8 * sms && 4 * split * 2 <= nbk + 2) split *= 2;
            if (ctx->tune.kquant_split > 0) split = (uint32_t)min(16, ctx->tune.kquant_split);
            if ((size_t)split * m * 4 > (1u << 20)) split = 0;
        }
        if (tiles < 8 * sms && split == 0 && ctx->tune.kquant_variant != 2) goto first_kernel;
        t.split = split;
        t.part = reinterpret_cast<float*>((uint8_t*)ctx->d_kq + 8192);
        t.tickets = reinterpret_cast<uint32_t*>(ctx->d_kq);
        t.w = (const uint8_t*)w;
        t.x = (const float*)x;
        t.y = (float*)y;
        t.res = (const float*)res;
        t.m = m;
        t.nb = k / 256;
        t.row_bytes = (k / 256) * (FMT == RUNIT_FMT_Q6K ? 210u : 176u);
        // The preparing launch costs 2 us, and rows of few units gain nothing from it (us without / with it).  K = 1024, Q6_K 300 MB 94 / 105;
        // 2048, Q6_K 110 MB 47 / 44, 300 MB 91 / 97; 2560, Q6_K 260 MB 80 / 88, Q5_K 350 MB 100 / 103; 3072, 160 to 450 MB, -3 to +8 % in turn;
        // 3584, Q6_K 160 MB 59 / 59, 220 MB 80 / 74, 450 MB 127 / 125, Q5_K 130 MB 46 / 48, 350 MB 100 / 95; 4096 to 12288, 160 MB and
        // more: 1 to 10 % faster with it.
        const bool pays = k >= 3584 && (uint64_t)m * t.row_bytes >= 150000000ull;
        const bool pre = FMT != RUNIT_FMT_Q5_0 && split == 0 && ctx->d_xq && (size_t)t.nb * kt::kXq <= ctx->xq_bytes &&
                         (ctx->tune.kquant_prepare == 0 ? pays : ctx->tune.kquant_prepare == 1);
        t.xq = (const uint8_t*)ctx->d_xq;
        t.wait_first = ctx->foreign_kernels ? 1u : 0u;
        int smem;
        void (*kern)(const kt::Args);
        if constexpr (FMT == RUNIT_FMT_Q5_0) {
            smem = 4 * q50t::kS * q50t::kStage;
            kern = q50t::gemv_q5_0_tile_kernel;
        } else {
            smem = kt::Tile<FMT>::kSmem;
            kern = pre ? kt::gemv_kquant_tile_kernel<FMT, true> : kt::gemv_kquant_tile_kernel<FMT, false>;
        }
        static bool configured[2][64] = {{false}};
        if (ctx->device >= 0 && ctx->device < 64 && !configured[pre][ctx->device]) {
            RUNIT_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            configured[pre][ctx->device] = true;
        }
        if (pre) {
            runit_launch_chain(ctx, kt::kquant_prepare_kernel, dim3(t.nb), dim3(32), t.x, (uint8_t*)ctx->d_xq);
            const int32_t st = runit_after_launch(ctx, "gemv_kquant_prepare_x");
            if (st != RUNIT_OK) return st;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = split ? dim3(tiles, split) : dim3((m + 127) / 128);
        cfg.blockDim = dim3(128);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = ctx->tune.pdl ? 1 : 0;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cudaError_t e = cudaLaunchKernelEx(&cfg, kern, t);
        if (e != cudaSuccess) return runit_fail(ctx, RUNIT_ERR_LAUNCH, "launch of %s failed: %s", name, cudaGetErrorString(e));
        return runit_after_launch(ctx, name);
    }
first_kernel:
    Args a;
    a.w = (const uint8_t*)w;
    a.x = (const float*)x;
    a.y = (float*)y;
    a.res = (const float*)res;
    a.m = m;
    a.k = k;
    a.nb = k / 32;
    a.n_units = (k + 255) / 256;
    a.row_bytes = FMT == RUNIT_FMT_Q5_0 ? (k / 32) * 22 : (k / 256) * (uint32_t)KTraits<FMT>::UB;
    uint32_t grid = (m + kWarps - 1) / kWarps;
    const uint32_t cap = (uint32_t)ctx->sm_count * 8u;   // 64 warps per SM
    if (grid > cap) grid = cap;
    runit_launch_chain(ctx, gemv_kquant_kernel<FMT>, dim3(grid), dim3(kWarps * 32), a);
    return runit_after_launch(ctx, name);
}

}  // namespace kq
}  // namespace runit

using namespace runit;

extern "C" {

int32_t runit_gemv_q5_0_f32in_f32out(runit_ctx_t* ctx, const void* w, const void* x, void* y, uint32_t m, uint32_t k) {
    return kq::launch<RUNIT_FMT_Q5_0>(ctx, "gemv_q5_0_f32in_f32out", w, x, y, nullptr, m, k);
}
int32_t runit_gemv_q5_0_add_f32_f32in(runit_ctx_t* ctx, const void* w, const void* x, void* y, const void* r, uint32_t m, uint32_t k) {
    if (ctx) RUNIT_REQUIRE(ctx, r, "gemv_q5_0_add_f32_f32in: null residual");
    return kq::launch<RUNIT_FMT_Q5_0>(ctx, "gemv_q5_0_add_f32_f32in", w, x, y, r, m, k);
}
int32_t runit_gemv_q5k_f32in_f32out(runit_ctx_t* ctx, const void* w, const void* x, void* y, uint32_t m, uint32_t k) {
    return kq::launch<RUNIT_FMT_Q5K>(ctx, "gemv_q5k_f32in_f32out", w, x, y, nullptr, m, k);
}
int32_t runit_gemv_q5k_add_f32_f32in(runit_ctx_t* ctx, const void* w, const void* x, void* y, const void* r, uint32_t m, uint32_t k) {
    if (ctx) RUNIT_REQUIRE(ctx, r, "gemv_q5k_add_f32_f32in: null residual");
    return kq::launch<RUNIT_FMT_Q5K>(ctx, "gemv_q5k_add_f32_f32in", w, x, y, r, m, k);
}
int32_t runit_gemv_q6k_f32in_f32out(runit_ctx_t* ctx, const void* w, const void* x, void* y, uint32_t m, uint32_t k) {
    return kq::launch<RUNIT_FMT_Q6K>(ctx, "gemv_q6k_f32in_f32out", w, x, y, nullptr, m, k);
}
int32_t runit_gemv_q6k_add_f32_f32in(runit_ctx_t* ctx, const void* w, const void* x, void* y, const void* r, uint32_t m, uint32_t k) {
    if (ctx) RUNIT_REQUIRE(ctx, r, "gemv_q6k_add_f32_f32in: null residual");
    return kq::launch<RUNIT_FMT_Q6K>(ctx, "gemv_q6k_add_f32_f32in", w, x, y, r, m, k);
}

}  // extern "C"
