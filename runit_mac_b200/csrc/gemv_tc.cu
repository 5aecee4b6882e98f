// Batched (2..8 activation rows) Q8_0 GEMV on tcgen05 (tc_rows.cuh): the weights stream once and are unpacked into tensor memory, the first two of the
// activations' three parts are the 16 columns of one product, the third goes through one of its own.
//
// A pre-pass splits the activations once per call.  Work is cut into items of (128 rows, share of K); the shares of a row depend on K alone
// and are added in order, so an output's bits depend neither on the other matrices of a launch nor on how the items fall on the CTAs.  Each
// CTA takes a stretch of consecutive items: the tiles that it has whole it stores itself, those that it shares with its neighbours are filed share by share and
// added by the warp that files last.
//
// The same kernel takes one activation row of Q6_K (gemv_kquant.cu has the line).  Its rows start on even bytes, which no tiled load takes: rows
// eight apart start alike modulo 16, so a step comes as eight boxes of 16 rows, each from the last multiple of 16 before its unit.  152064 x 3584:
// 127 -> 87 us (5.1 TB/s).  There the warp that would copy images splits the one activation row itself, a unit per step, into images
// whose other values stay zeros: a pre-pass cost 1.5 to 3.5 us a call (152064 x 3584 90 us, 18944 x 512 6.0 against 4.5).  Bound now by the
// unpacking warps' instructions and the copies together (with the pre-pass, without the arithmetic 79, with an eighth of the copies 78).  Copying words with cp.async instead, 322; six teams 112, unpacking ahead of the wait for the place 96.
// Error against 64 bits 0.9e-7 to 1.1e-7 from K = 2048 on (the kernels before 2.7e-7), and with three parts below that 6.0e-8 to 7.0e-8 (8.3e-8 to 9.2e-8).
//
// Bound: the unpacking warps, about 1000 clocks per 128 x 256 weights and SM (2.1 TB/s), and some 4 us between dependent calls (the pre-pass and
// its hand-over).  The packed f32 kernel, which still serves small ones of 2 to 4 rows (gemv_tc_pays), multiplies every weight 8 times on the CUDA cores.
// Decoding steps, us, f32 -> now: width 3584, two layers and a head of 30000 rows, 2 / 4 / 8 sequences 293 / 420 / 906 -> 183 / 183 / 188; width 2048, four layers,
// 271 / 363 / 689 -> 219 / 225 / 233; width 1024, eight layers, 211 / 273 / 511 -> 197 / 230 / 262.  Error against 64 bits 5.9e-8 at K = 256, 7.7e-8 at 2048, 1.0e-7
// at 18944 (f32 products 7.8e-8, 9.6e-8, 1.4e-7; the two halves of 22 bits that were here before, 4 to 8 % faster, 8.1e-8, 9.5e-8, 1.2e-7, and more
// than f32 products where a few activations dominate).  The 4-bit formats stay with gemv_imma.cu: the same kernel for them took 362 us where that one
// takes 350 (Q4_K, 7B, four layers and head, 8 sequences), 332 against 353 (Q4_0, 4 sequences) and 198 against 187 (width 2048).
#include <cuda_fp16.h>

#include "runit_internal.h"
#include "tc_rows.cuh"

namespace runit {
namespace tcg {

constexpr tcr::Kind kKind = tcr::Q8_0_8;
using C = tcr::Cfg<kKind>;

// One CTA per 256 activations, one warp per activation row (rows behind the batch are zeros).
__global__ void __launch_bounds__(256) split_kernel(const float* __restrict__ x, uint8_t* __restrict__ images, float* __restrict__ scales, uint32_t k, uint32_t batch) {
    __shared__ __align__(16) uint8_t out[C::kBStage];
    const uint32_t u = blockIdx.x, n = threadIdx.x >> 5, lane = threadIdx.x & 31;
    grid_launch_dependents();      // the product may start requesting its weights; it waits for this grid before it reads anything else
    grid_dependency_wait();
    float v[8];
    tcr::load8(x + (size_t)n * k + (size_t)u * 256 + 8 * lane, n < batch, v);
    const float scale = tcr::split_column<kKind>(v, lane, out, n, out, 8 + n, C::kPanel, nullptr, 0);
    if (lane == 0) scales[u * 8 + n] = scale;
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(images + (size_t)u * C::kBStage);
    for (uint32_t i = threadIdx.x; i < C::kBStage / 16; i += 256) dst[i] = reinterpret_cast<const uint4*>(out)[i];
}

// Up to three matrices that share the activations (q | k | v, gate | up) ride one launch: segment i owns the row tiles from tile0[i] on.
struct Args {
    const float* x;              // Q6_K
    const uint8_t* images;       // else
    const float* scales;
    float* y[3];
    const float* res[3];
    uint32_t m[3], tile0[3];
    uint32_t nseg, units, shares, items, batch;
    uint32_t inverse;            // 2^32 / shares, rounded up (0: one share): the quotient's high word, exact below 2^32 / shares
    float* part;                 // [tile's place][share][sum of a thread][thread]
    uint32_t* tickets;           // [tile's place][warp], zero at rest
    int32_t* status;
};
struct Maps {
    CUtensorMap m[3];
};

template <tcr::Kind K> struct Policy {
    using C = tcr::Cfg<K>;
    static constexpr int kAcc = C::kAcc;
    const Args& a;
    const Maps& maps;
    const uint32_t i0, i1;       // items of this CTA
    float total[kAcc];

    __device__ __forceinline__ Policy(const Args& args, const Maps& m)
        : a(args), maps(m), i0((uint32_t)((uint64_t)blockIdx.x * args.items / gridDim.x)), i1((uint32_t)((uint64_t)(blockIdx.x + 1) * args.items / gridDim.x)) {}

    __device__ __forceinline__ bool few() const { return a.batch <= 4; }

    __device__ __forceinline__ uint32_t begin() const { return i0; }
    __device__ __forceinline__ uint32_t end() const { return i1; }
    // 32-bit divisions cost the sums' warps more than a step's sums
    __device__ __forceinline__ uint32_t by_shares(uint32_t v) const { return a.inverse ? __umulhi(v, a.inverse) : v; }
    __device__ __forceinline__ uint32_t unit(uint32_t i) const {
        const uint32_t tile = by_shares(i);
        return tile * a.units + by_shares((i - tile * a.shares) * a.units);
    }
    __device__ __forceinline__ uint32_t steps() const { return unit(i1) - unit(i0); }
    __device__ __forceinline__ int segment(uint32_t tile) const { return a.nseg > 2 && tile >= a.tile0[2] ? 2 : a.nseg > 1 && tile >= a.tile0[1] ? 1 : 0; }
    __device__ __forceinline__ tcr::Run run(uint32_t i) const {
        const uint32_t tile = by_shares(i), share = i - tile * a.shares;
        const int s = segment(tile);
        tcr::Run r;
        r.map[0] = &maps.m[s];
        r.row[0] = (int32_t)((tile - a.tile0[s]) * 128);
        r.u0 = by_shares(share * a.units);
        r.u1 = by_shares((share + 1) * a.units);
        r.b = a.images + (size_t)r.u0 * C::kBStage;
        r.xs = a.scales + r.u0 * 8;
        r.n = 8;
        return r;
    }
    __device__ __forceinline__ void store(uint32_t tile, uint32_t warp, uint32_t lane) const {
        const int s = segment(tile);
        const uint32_t t = (warp & 3) * 32 + lane, row = (tile - a.tile0[s]) * 128 + (C::kQ6 ? tcr::q6k_row(t) : t), m = a.m[s];
        if (row >= m) return;
#pragma unroll
        for (uint32_t j = 0; j < kAcc; j++) {
            const uint32_t users = kAcc == 1 ? 1 : few() ? 2 : 4, c = users * (warp >> 2) + j;
            if (j >= users) break;
            if (c < a.batch) {
                const size_t o = (size_t)c * m + row;
                a.y[s][o] = a.res[s] ? total[j] + a.res[s][o] : total[j];
            }
        }
    }
    __device__ __forceinline__ void finish(uint32_t i, float (&acc)[1][kAcc], uint32_t warp, uint32_t lane) {
        const uint32_t tile = by_shares(i), share = i - tile * a.shares, t0 = tile * a.shares;
        if (t0 >= i0 && t0 + a.shares <= i1) {
#pragma unroll
            for (int j = 0; j < kAcc; j++) total[j] = share ? total[j] + acc[0][j] : acc[0][j];
            if (share + 1 == a.shares) store(tile, warp, lane);
        } else {
            // the place of a tile that several CTAs share: the first CTA that starts inside it
            const uint32_t place = (uint32_t)(((uint64_t)(t0 + 1) * gridDim.x + a.items - 1) / a.items);
            constexpr uint32_t kT = 32 * C::kSumWarps;
            static_assert(kAcc * kT * 4 <= kPartBytes, "a share's place");
            float* p = a.part + (size_t)place * kMaxShares * (kPartBytes / 4) + warp * 32 + lane;
#pragma unroll
            for (int j = 0; j < kAcc; j++) __stcg(p + (share * kAcc + j) * kT, acc[0][j]);
            if (share + 1 == a.shares || i + 1 == i1) {
                const uint32_t mine = i - (t0 > i0 ? t0 : i0) + 1;
                uint32_t before = 0;
                __threadfence();
                __syncwarp();
                if (lane == 0) before = atomicAdd(&a.tickets[place * 8 + warp], mine);
                before = __shfl_sync(0xffffffffu, before, 0);
                if (before + mine == a.shares) {
                    __threadfence();
#pragma unroll
                    for (int j = 0; j < kAcc; j++) total[j] = __ldcg(p + j * kT);
                    for (uint32_t q = 1; q < a.shares; q++)
#pragma unroll
                        for (int j = 0; j < kAcc; j++) total[j] += __ldcg(p + (q * kAcc + j) * kT);
                    store(tile, warp, lane);
                    if (lane == 0) a.tickets[place * 8 + warp] = 0;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kAcc; j++) acc[0][j] = 0.f;
    }
};

template <tcr::Kind K>
__global__ void __launch_bounds__(tcr::Cfg<K>::kThreads, 1) gemv_tc_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Args a) {
    using C = tcr::Cfg<K>;
    extern __shared__ uint8_t smem_raw[];
    tcr::Block<K, 1> blk(smem_raw);
    Policy<K> p(a, maps);
    if (blk.warp == C::kCopyW) {
        // raw blocks: the first steps' ahead of the dependency wait; the columns' scales behind it
        uint32_t s = 0, early = 0;
        auto load = [&](const tcr::Run& r, uint32_t u, uint32_t step) {
            if (C::kQ6) {
                const uint32_t row_bytes = a.units * 210;
                if (blk.lane == 0) {
                    *reinterpret_cast<volatile uint32_t*>(blk.base_p + C::kOffAt + 4 * (step % C::kW)) = (u * 210 & 15) | (row_bytes & 15) << 8;
                    mbar_expect_tx(blk.raw_bar(step), C::kWBytes);
                }
                __syncwarp();
                if (blk.lane < 8)
                    tma_load_2d(blk.raw(step) + blk.lane * (C::kWBytes / 8), r.map[0], (int32_t)((blk.lane * row_bytes + u * 210) & ~15u), r.row[0] / 8, blk.raw_bar(step));
            } else if (elect_one()) {
                mbar_expect_tx(blk.raw_bar(step), C::kWBytes + r.n * 4);
                tma_load_2d(blk.raw(step), r.map[0], (int32_t)(u * 136), r.row[0], blk.raw_bar(step));       // elements of two bytes
            }
            __syncwarp();
        };
        for (uint32_t i = p.begin(); i < p.end() && early < C::kW; i++) {
            const tcr::Run r = p.run(i);
            for (uint32_t u = r.u0; u < r.u1 && early < C::kW; u++) load(r, u, early++);
        }
        grid_dependency_wait();
        for (uint32_t i = p.begin(); i < p.end() && blk.ok; i++) {
            const tcr::Run r = p.run(i);
            for (uint32_t u = r.u0; u < r.u1; u++, s++) {
                if (s >= early) {
                    if (!blk.raw_free(s)) break;
                    load(r, u, s);
                }
                if (!C::kQ6 && elect_one()) bulk_load_1d(blk.scales(s), r.xs + (size_t)(u - r.u0) * r.n, r.n * 4, blk.raw_bar(s));
                __syncwarp();
            }
        }
        // whatever was requested arrives before the CTA leaves, whichever role gives up, and when (weights whose step's scales were never requested can only
        // be waited for until the limit)
        mbar_drain(blk.w_full, C::kW, s > early ? s : early);
    } else if (blk.warp == C::kCopyB && C::kQ6) {
        // One activation row is split here, a unit per step: block b into rows b, 8 + b (and 16 + b) of an image whose other values stay zeros.
        uint4* const images = reinterpret_cast<uint4*>(blk.base_p + C::kOffB);
        for (uint32_t i = blk.lane; i < C::kB * C::kBStage / 16; i += 32) images[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        const uint32_t steps = p.steps(), row = blk.lane >> 2;
        uint32_t unit = p.run(p.begin()).u0;
        float next[8];
        grid_dependency_wait();
        tcr::load8(a.x + (size_t)unit * 256 + 8 * blk.lane, true, next);
        for (uint32_t c = 0; c < steps; c++) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = next[i];
            if (++unit == a.units) unit = 0;
            tcr::load8(a.x + (size_t)unit * 256 + 8 * blk.lane, true, next);
            if (!blk.image_free(c)) break;
            uint8_t* const image = blk.base_p + C::kOffB + c % C::kB * C::kBStage;
            const float scale = tcr::split_column<K>(v, blk.lane, image, row, image, 8 + row, C::kPanel, nullptr, 0);
            if (blk.lane == 0) reinterpret_cast<float*>(blk.base_p + C::kOffXs)[c % C::kXs * C::kCols] = scale;
            fence_proxy_async();
            __syncwarp();
            if (blk.lane == 0) mbar_arrive(blk.image_bar(c));
        }
    } else if (blk.warp == C::kCopyB) {
        uint32_t c = 0;
        grid_dependency_wait();
        for (uint32_t i = p.begin(); i < p.end() && blk.ok; i++) {
            const tcr::Run r = p.run(i);
            for (uint32_t u = r.u0; u < r.u1; u++, c++) {
                if (!blk.image_free(c)) break;
                if (elect_one()) {
                    mbar_expect_tx(blk.image_bar(c), C::kBStage);
                    bulk_load_1d(blk.image(c), r.b + (size_t)(u - r.u0) * C::kBStage, C::kBStage, blk.image_bar(c));
                }
                __syncwarp();
            }
        }
        mbar_drain(blk.b_full, C::kB, c);
    } else {
        blk.work(p);
    }
    blk.leave(a.status);
}

// Shares, grid and the context's places; the pre-pass and the product as dependent launches.
template <tcr::Kind K> static int32_t launch(runit_ctx* ctx, const char* name, Args& a, const Maps& maps, const float* x, uint32_t k, uint32_t batch) {
    static bool configured[64] = {false};
    if (ctx->device >= 64 || !configured[ctx->device]) {
        RUNIT_CUDA_TRY(ctx, cudaFuncSetAttribute(gemv_tc_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, tcr::Cfg<K>::kSmem));
        if (ctx->device < 64) configured[ctx->device] = true;
    }
    // two units per share, ten shares at most: enough items for every SM at the sizes where a tile per CTA would leave most of them idle
    a.shares = (a.units + 1) / 2 < kMaxShares ? (a.units + 1) / 2 : kMaxShares;
    a.items *= a.shares;
    a.inverse = a.shares > 1 ? (uint32_t)((0x100000000ull + a.shares - 1) / a.shares) : 0;
    uint32_t grid = (uint32_t)ctx->sm_count;
    grid = grid < kMaxCtas ? grid : kMaxCtas;
    grid = grid < a.items ? grid : a.items;
    a.x = x;
    a.images = (const uint8_t*)ctx->d_xq;
    a.scales = (const float*)(a.images + (size_t)a.units * C::kBStage);
    a.tickets = (uint32_t*)ctx->d_tc;
    a.part = (float*)((uint8_t*)ctx->d_tc + kTicketBytes);
    a.status = ctx->d_status;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.stream = ctx->stream;
    cfg.attrs = attr;
    // The product requests weights as soon as the launch before it lets it start.  Where a kernel before the call may have written them, the call's
    // first launch is an ordinary one, which starts when all of it can be seen.
    cfg.numAttrs = !ctx->foreign_kernels && !ctx->weights_written && ctx->tune.pdl != 0 ? 1 : 0;
    ctx->weights_written = false;
    cudaError_t e;
    if (!tcr::Cfg<K>::kQ6) {
        cfg.gridDim = dim3(a.units);
        cfg.blockDim = dim3(256);
        e = cudaLaunchKernelEx(&cfg, split_kernel, x, (uint8_t*)ctx->d_xq, (float*)a.scales, k, batch);
        if (e != cudaSuccess) return runit_fail(ctx, RUNIT_ERR_LAUNCH, "launch of %s (split of the activations) failed: %s", name, cudaGetErrorString(e));
        const int32_t st = runit_after_launch(ctx, "gemv_split_x");
        if (st != RUNIT_OK) return st;
        cfg.numAttrs = 1;
    }
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(tcr::Cfg<K>::kThreads);
    cfg.dynamicSmemBytes = tcr::Cfg<K>::kSmem;
    e = cudaLaunchKernelEx(&cfg, gemv_tc_kernel<K>, maps, a);
    if (e != cudaSuccess) return runit_fail(ctx, RUNIT_ERR_LAUNCH, "launch of %s (tcgen05) failed: %s", name, cudaGetErrorString(e));
    return runit_after_launch(ctx, name);
}

}  // namespace tcg

// Where it is the faster one.  The packed f32 kernel takes a launch per matrix and power of two in the batch (3 = 2 + 1), 2 to 4 us each and then some 5e12
// multiply-adds a second; this one takes 4 to 7 us (the pre-pass and its hand-over) and 3.4e12 weights a second, whatever the batch.  So it wins with
// eight rows or three launches, with two nearly always, and against one from the sizes below on, which lie where the two meet (us, f32 / this: batch 2,
// K 256 8192 rows 2.8 / 4.5, 16384 5.1 / 4.6; K 1024 16384 9.2 / 11.1, 32768 15.3 / 13.3; K 2048 4096 6.2 / 7.7, 8192 12.1 / 10.5; K 3584 2048 6.4 / 7.7, 4096
// 12.3 / 10.4; K 12288 512 9.2 / 10.5, 1024 14.3 / 10.5; batch 4, K 1024 8192 6.1 / 7.4, 16384 12.1 / 11.2; K 2048 2048 6.3 / 7.5, but a step of width 2048 with it 231 / 225, 4096 7.7 / 7.7; K 3584 2048 7.8 / 7.8; K 8192 512 9.5 /
// 9.5; two launches, K 1024: two matrices of 2816, batch 2, 6.5 / 7.3; one of 1024, batch 3, 6.3 / 7.1, of 2048 7.6 / 7.2; batch 3 stays here throughout, because its third
// row would meet 16-bit activations there).
static bool gemv_tc_pays(uint32_t n_mats, uint64_t rows, uint32_t k, uint32_t batch) {
    const uint32_t launches = n_mats * (uint32_t)__builtin_popcount(batch);
    if (batch == 8 || launches > 2) return true;
    if (launches == 2) return batch != 2 || k < 512 || k > 1024 || rows >= 8192;
    if (batch == 2) return rows >= (k <= 512 ? 12288u : k <= 1024 ? 24576u : k <= 2048 ? 6144u : k <= 8192 ? 3072u : k <= 12288 ? 768u : 0u);
    return rows >= (k <= 512 ? 10240u : k <= 1024 ? 12288u : k <= 5120 ? 2048u : k <= 8192 ? 512u : 0u);
}

bool gemv_tc_applies(const runit_ctx* ctx, int fmt, uint32_t n_mats, const uint32_t* m, uint32_t k, uint32_t batch) {
    if (fmt != RUNIT_FMT_Q8_0 || batch < 2 || batch > 8 || k == 0 || k % 256 != 0 || ctx->tune.gemv_math == 1 || !ctx->encode_tiled || !ctx->d_xq || !ctx->d_tc) return false;
    if ((size_t)(k / 256) * (tcg::C::kBStage + 32) > ctx->xq_bytes) return false;
    uint64_t rows = 0;
    for (uint32_t i = 0; i < n_mats; i++) rows += m[i];
    return ctx->tune.gemv_tc == 1 || gemv_tc_pays(n_mats, rows, k, batch);
}

// n_mats (1..3) matrices over the same activations in one launch.
int32_t gemv_tc_multi(runit_ctx* ctx, uint32_t n_mats, const void* const* w, const float* x, float* const* y, const float* const* res, const uint32_t* m,
                      uint32_t k, uint32_t batch) {
    using namespace tcg;
    Args a{};
    Maps maps{};
    a.units = k / 256;
    a.batch = batch;
    a.nseg = n_mats;
    uint64_t tiles = 0;
    for (uint32_t i = 0; i < 3; i++) {
        const uint32_t s = i < n_mats ? i : 0;      // unused entries repeat segment 0 (never selected)
        a.y[i] = y[s];
        a.res[i] = res ? res[s] : nullptr;
        a.m[i] = m[s];
        a.tile0[i] = i < n_mats ? (uint32_t)tiles : 0xFFFFFFFFu;
        if (i < n_mats) {
            const int32_t st = runit_get_tmap(ctx, w[i], m[i], (uint64_t)a.units * 272, 128, 272, &maps.m[i]);
            if (st != RUNIT_OK) return st;
            tiles += ((uint64_t)m[i] + 127) / 128;
        } else {
            maps.m[i] = maps.m[0];
        }
    }
    a.items = (uint32_t)tiles;         // times ten shares: far below 2^32 / 10, where the quotient by shares ends, for matrices that fit a GPU
    return launch<kKind>(ctx, "gemv_batched_tc", a, maps, x, k, batch);
}

// Q6_K, one activation row; w 16-byte aligned.
bool gemv_q6k_tc_applies(const runit_ctx* ctx, const void* w, uint32_t m, uint32_t k) {
    return m >= 8 && k % 256 == 0 && runit_aligned(w, 16) && ctx->d_tc && ctx->encode_tiled;
}
int32_t gemv_q6k_tc(runit_ctx* ctx, const char* name, const void* w, const float* x, float* y, const float* res, uint32_t m, uint32_t k) {
    using namespace tcg;
    Args a{};
    Maps maps{};
    a.units = k / 256;
    a.batch = 1;
    // The boxes are made of groups of eight rows; the rows behind the last whole group are a tile of their own, whose map ends where the matrix does.
    const uint32_t whole = m & ~7u, row_bytes = a.units * 210;
    int32_t st = runit_get_tmap(ctx, w, whole / 8, (uint64_t)row_bytes * 8, 16, 240, &maps.m[0]);
    if (st == RUNIT_OK && whole < m) st = runit_get_tmap(ctx, (const uint8_t*)w + (size_t)whole * row_bytes, 1, (uint64_t)row_bytes * (m - whole), 16, 240, &maps.m[1]);
    if (st != RUNIT_OK) return st;
    a.nseg = whole < m ? 2 : 1;
    a.y[0] = y;
    a.y[1] = y + whole;
    a.res[0] = res;
    a.res[1] = res ? res + whole : nullptr;
    a.m[0] = whole;
    a.m[1] = m - whole;
    a.tile0[1] = (whole + 127) / 128;
    a.items = a.tile0[1] + a.nseg - 1;
    // Three parts of an activation where the kernel that this one replaces (one warp per row) multiplied f32 values; its others held them in three 8-bit limbs
    // per 32 (2.7e-7 against 64 bits at K = 3584, two parts here 1.0e-7; 5 % of 152064 x 3584's time are saved).
    return k < 2048 ? launch<tcr::Q6K_8R>(ctx, name, a, maps, x, k, 1) : launch<tcr::Q6K_8>(ctx, name, a, maps, x, k, 1);
}

}  // namespace runit
