// Binary convolution on activations kept as {0,1} bytes: TMA feeds tcgen05.mma kind::i8 directly.
//
// The engine in bcontract_tc5.cuh reads packed bits and spends its time expanding them to bytes in shared
// memory with eight producer warps.  Here the layer that produces an activation also writes it as one byte per
// channel (NHWC, 8x the packed size, a quarter of the fp32 copy that is written anyway), and then the pixel
// operand of a convolution tap is a rectangle of that tensor: for a tile of whole output rows,
//
//   A_tap[(row, ow)][c] = x8[img][row * s + ky - pad][ow * s + kx - pad][c]     (zero outside the image),
//
// which is one tiled TMA load per tap and 64-channel group, 64-byte-swizzled, landing in exactly the K-major
// layout tcgen05.mma reads.  Zero fill outside the image is the reference's padding (bit 0).  No thread touches
// the operand: one lane issues the loads, one lane issues the MMAs, the other warps are the epilogue.
//
//   cnt[p][n] = sum_k a_k xor b_k = sum_k a_k * (1 - 2 b_k) + sum_k b_k
//
// with a the activation bits as unsigned bytes {0,1} and the weights stored as signed bytes 1 - 2b = {+1,-1}: the
// MMA (unsigned x signed 8-bit, s32 accumulators) yields the first sum and the epilogue adds the weight row's
// popcount.  A zero-filled tap contributes b_k, the reference's count for a padded position.
//
// Tiles: OW <= 128.  If an image has more than 128 output pixels a tile is `rows` whole output rows of one image
// (rows * OW <= 128), else `imgs` whole images.  The M = 128 rows of the MMA beyond the tile's pixels hold stale
// bytes; their accumulator lanes are never read.  The input's tensor map has five dimensions (c, w, h, image,
// column parity): stride 1 uses parity 0 only; stride 2 views W as (W / 2, parity) and folds the row parity into
// the base address (two tensor maps), so that a tap is still a dense box.
//
// Where the weights are streamed, a unit of work is a pair of pixel tiles (M = 2 x 128) that share every weight
// stage, each with its own accumulator: half the weight bytes per MMA.
//
// Weights: expanded once (bconv_u8_expand_weights_kernel) into per-(channel block, K box) images in the
// SWIZZLE_NONE K-major core-matrix layout, streamed per stage by one bulk copy - or, when a channel block's
// weights are small (the 64-channel layers: 45 KB), loaded once per CTA and kept in shared memory, which takes
// them off the L2 -> shared-memory path that bounds this kernel.
//
// Every wait is bounded; a wait that gives up records a code in a status word, raises the CTA's abort flag,
// and the CTA frees its tensor memory and returns.
#pragma once
#include "bconv_epilogue.cuh"

namespace dabnn {

constexpr int U8_BOX_BYTES = 128 * 64;       // one K box of the pixel operand: 128 rows x 64 bytes
constexpr int U8_ACCS = 4;                   // TMEM accumulators of up to 128 columns
constexpr int U8_THREADS = 64 + EPI_THREADS;  // warp 0: loads, warp 1: MMA, then the epilogue warps (bconv_epilogue.cuh)
constexpr int U8_MAX_SMEM = 227 * 1024;

__device__ int g_u8_status;   // 0 = ok; 21 loader, 22 MMA (accumulator), 23 MMA (stage), 24 epilogue

struct U8Params {
    const unsigned char* w_img;   // expanded weights (bconv_u8_expand_weights_kernel)
    const float *a, *b;           // per-channel affine (both or neither)
    const float* shortcut;        // fp32 [M][N] added after the affine, or null
    float* out;                   // fp32 [M][N] or null
    unsigned char* out_u8;        // {0,1} bytes [M][N] or null
    uint64_t* out_bits;           // packed sign bits [M][N/64] or null
    int B, OH, OW, N;
    int kh, kw, pad_h, pad_w, stride, cw;
    int rows, imgs, tiles_per_img, ntiles;
    int G, stages, wb, nboxes;    // K boxes per stage, ring stages, rows of a weight box image, kh*kw*cw
    int resident;                 // the channel block's weights stay in shared memory (loaded once per CTA)
    int wide;                     // cin % 128 == 0: one TMA load covers two K boxes (128-byte rows, SWIZZLE_128B)
    int pair;                     // two pixel tiles share every weight stage (streamed weights: halves their bytes)
    int narrow;                   // see EpiOut
    int nbc;                      // output channels per CTA: TC5_MAX_N, or 64 / 32 when there are too few tiles to fill the SMs
                                  // (streamed weights only: a CTA then copies its rows out of every box image)
};

__host__ __device__ inline int u8_weight_rows(int N) { return min(N, TC5_MAX_N); }
__host__ __device__ inline size_t u8_weight_image_bytes(int N, int nboxes) {
    return (size_t)((N + TC5_MAX_N - 1) / TC5_MAX_N) * nboxes * u8_weight_rows(N) * 64;
}
__host__ __device__ inline size_t u8_weight_bytes(int N, int nboxes) {
    return u8_weight_image_bytes(N, nboxes) + (size_t)((N + TC5_MAX_N - 1) / TC5_MAX_N) * TC5_MAX_N * sizeof(int);
}

// grid (nboxes, channel blocks): the image of K box q (= packed word q) of one channel block: wb rows x 64 bytes,
// byte k of row n = 1 - 2 * bit k of the word (+1 or -1 as a signed byte), stored as 8-row x 16-byte core matrices
// ([row / 8][k / 16][row % 8][k % 16]); rows beyond the channel block are zero.
__global__ void __launch_bounds__(256) bconv_u8_expand_weights_kernel(const uint64_t* w, const long long ldw, const int N,
                                                                      const int nboxes, unsigned char* dst) {
    const int q = blockIdx.x, nb = blockIdx.y, wb = u8_weight_rows(N);
    const int n0 = nb * TC5_MAX_N, n_this = min(TC5_MAX_N, N - n0);
    unsigned char* img = dst + ((size_t)nb * nboxes + q) * wb * 64;
    for (int idx = threadIdx.x; idx < wb * 4; idx += blockDim.x) {
        const int row = idx >> 2, unit = idx & 3;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (row < n_this) {
            const uint32_t bits = (uint32_t)(__ldg(w + (long long)(n0 + row) * ldw + q) >> (unit * 16)) & 0xffffu;
            auto signed_bytes = [](uint32_t nibble) {   // four bits -> four bytes, 0 -> 0x01, 1 -> 0xff
                const uint32_t m = (nibble * 0x00204081u) & 0x01010101u;
                return (m * 0xffu) | (m ^ 0x01010101u);
            };
            v.x = signed_bytes(bits & 0xfu); v.y = signed_bytes((bits >> 4) & 0xfu);
            v.z = signed_bytes((bits >> 8) & 0xfu); v.w = signed_bytes((bits >> 12) & 0xfu);
        }
        *reinterpret_cast<uint4*>(img + (row >> 3) * 512 + unit * 128 + (row & 7) * 16) = v;
    }
    if (q == 0 && threadIdx.x < TC5_MAX_N) {
        int pc = 0;
        if ((int)threadIdx.x < n_this)
            for (int k = 0; k < nboxes; k++) pc += __popcll(__ldg(w + (long long)(n0 + threadIdx.x) * ldw + k));
        reinterpret_cast<int*>(dst + u8_weight_image_bytes(N, nboxes))[n0 + threadIdx.x] = pc;
    }
}

// fp32 -> {0,1} bytes (x > 0), 16 elements per thread step
__global__ void __launch_bounds__(256) binarize_u8_kernel(const float* __restrict__ in, unsigned char* __restrict__ out, const size_t n16,
                                                           const size_t count) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) {
        uint32_t wds[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 f = __ldg(reinterpret_cast<const float4*>(in) + i * 4 + j);
            wds[j] = (f.x > 0.f ? 1u : 0u) | (f.y > 0.f ? 0x100u : 0u) | (f.z > 0.f ? 0x10000u : 0u) | (f.w > 0.f ? 0x1000000u : 0u);
        }
        reinterpret_cast<uint4*>(out)[i] = make_uint4(wds[0], wds[1], wds[2], wds[3]);
    }
    if (blockIdx.x == 0)   // tail
        for (size_t i = n16 * 16 + threadIdx.x; i < count; i += blockDim.x) out[i] = in[i] > 0.f ? 1 : 0;
}

// K-major SWIZZLE_64B shared-memory descriptor: 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)4 << 61);
}
// K-major SWIZZLE_128B: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

template <bool PAIR>   // PAIR: a unit of work is two pixel tiles sharing the weight stages (p.pair)
__global__ void __launch_bounds__(U8_THREADS, 1)
    bconv_u8_kernel(const U8Params p, const __grid_constant__ CUtensorMap in_map0, const __grid_constant__ CUtensorMap in_map1) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t bar_full[8], bar_empty[8], bar_acc_full[U8_ACCS], bar_acc_empty[U8_ACCS], bar_w;
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_abort;
    __shared__ __align__(16) float pop[TC5_MAX_N];
    __shared__ __align__(16) float chan_a[TC5_MAX_N];
    __shared__ __align__(16) float chan_b[TC5_MAX_N];

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int n0 = blockIdx.y * p.nbc;
    const int n_this = min(p.nbc, p.N - n0);        // multiple of 16 (host-checked)
    const int n_mma = n_this;
    constexpr int np = PAIR ? 2 : 1;                // pixel tiles per unit of work (they share the unit's weight stages)
    const int nunits = (p.ntiles + np - 1) / np;
    const int a_bytes1 = p.G * U8_BOX_BYTES, a_bytes = np * a_bytes1;   // one tile's boxes of a stage, all of them
    const int gbox_bytes = p.wb * 64, wbox_bytes = min(p.nbc, p.wb) * 64;   // a box image in global / this CTA's rows of it
    const int stage_bytes = a_bytes + (p.resident ? 0 : p.G * wbox_bytes);
    unsigned char* wres = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    unsigned char* stage0 = wres + (p.resident ? p.nboxes * wbox_bytes : 0);   // a multiple of 1024 bytes further
    const int nst = (p.nboxes + p.G - 1) / p.G;     // stages per tile
    const int acc_cols = (n_mma + 31) & ~31;        // columns between accumulators: whole 32-column items
    int tmem_cols = 32;
    while (tmem_cols < U8_ACCS * acc_cols) tmem_cols <<= 1;
    const volatile int* abort_flag = &s_abort;
    const int ohw = p.OH * p.OW;
    const int box_px = p.rows * p.OW * p.imgs;      // pixels a tile's loads cover

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        for (int i = 0; i < p.stages; i++) { mbar_init(&bar_full[i], 1); mbar_init(&bar_empty[i], 1); }
        for (int i = 0; i < U8_ACCS; i++) { mbar_init(&bar_acc_full[i], 1); mbar_init(&bar_acc_empty[i], 4 * ((n_this + 31) >> 5)); }
        mbar_init(&bar_w, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::);
        s_abort = 0;
    }
    if (tid < TC5_MAX_N) {
        pop[tid] = epi_pop(tid < n_this ? __ldg(reinterpret_cast<const int*>(p.w_img + u8_weight_image_bytes(p.N, p.nboxes)) + n0 + tid) : 0);
        const bool have = p.a && tid < n_this;
        chan_a[tid] = have ? __ldg(p.a + n0 + tid) : 1.f;
        chan_b[tid] = have ? __ldg(p.b + n0 + tid) : 0.f;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    grid_launch_dependents();
    grid_dependency_wait();   // set-up touched constants only; activations come next

    if (warp == 0) {
        // =========================== loads: one lane ===========================
        if (lane == 0) {
            // this CTA's rows of its channel block's box images
            const unsigned char* wsrc = p.w_img + (size_t)(n0 / TC5_MAX_N) * p.nboxes * gbox_bytes + (size_t)(n0 % TC5_MAX_N) * 64;
            const uint32_t stage0_addr = smem_u32(stage0);
            const uint32_t box_tx = (uint32_t)box_px * 64u;   // a load always delivers its whole box (zeros outside the tensor)
            uint32_t s = 0, use = 0;
            bool ok = true;
            if (p.resident) {   // the whole channel block, once
                const uint32_t bytes = (uint32_t)(p.nboxes * wbox_bytes), bar = smem_u32(&bar_w);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(wres)), "l"(wsrc), "r"(bytes), "r"(bar) : "memory");
            }
            for (int unit = blockIdx.x; unit < nunits && ok; unit += gridDim.x) {
                int img0[2], oh0[2];   // a tile past the last one lies outside the tensor: its loads deliver zeros
                for (int t = 0; t < np; t++) {
                    const int tile = unit * np + t, tq = tile / p.tiles_per_img;
                    img0[t] = tq * p.imgs; oh0[t] = (tile - tq * p.tiles_per_img) * p.rows;
                }
                int cg = 0, ky = 0, kx = 0;
                for (int st = 0; st < nst; st++) {
                    if (use >= 1 && !mbar_wait<32>(&bar_empty[s], (use - 1) & 1, abort_flag)) {
                        atomicCAS(&g_u8_status, 0, 21);
                        s_abort = 1;
                        ok = false;
                        break;
                    }
                    const int nb = min(p.G, p.nboxes - st * p.G);
                    const uint32_t bar = smem_u32(&bar_full[s]), sa = stage0_addr + s * stage_bytes;
                    const uint32_t wbytes = p.resident ? 0u : (uint32_t)(nb * wbox_bytes);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(wbytes + np * nb * box_tx) : "memory");
                    if (!p.resident) {
                        if (wbox_bytes == gbox_bytes) {   // whole box images: the stage's boxes are one run
                            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                         ::"r"(sa + a_bytes), "l"(wsrc + (size_t)st * p.G * gbox_bytes), "r"(wbytes), "r"(bar) : "memory");
                        } else {
                            for (int b = 0; b < nb; b++)
                                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                             ::"r"(sa + a_bytes + b * wbox_bytes), "l"(wsrc + (size_t)(st * p.G + b) * gbox_bytes), "r"((uint32_t)wbox_bytes),
                                               "r"(bar) : "memory");
                        }
                    }
                    const int bstep = p.wide ? 2 : 1;   // a wide load fills two K boxes (16 KB: 128 rows of 128 bytes)
                    for (int b = 0; b < nb; b += bstep) {
                        const int dy = ky - p.pad_h, dx = kx - p.pad_w;
                        int c1 = 0, c2 = dx, c3 = dy;
                        const CUtensorMap* map = &in_map0;
                        if (p.stride == 2) {
                            const int hp = dy & 1, wp = dx & 1;
                            c1 = wp; c2 = (dx - wp) >> 1; c3 = (dy - hp) >> 1;
                            if (hp) map = &in_map1;
                        }
                        for (int t = 0; t < np; t++)
                            asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
                                         ::"r"(sa + t * a_bytes1 + b * U8_BOX_BYTES), "l"(reinterpret_cast<uint64_t>(map)), "r"(cg * 64), "r"(c2),
                                           "r"(oh0[t] + c3), "r"(img0[t]), "r"(c1), "r"(bar) : "memory");
                        if ((cg += bstep) == p.cw) { cg = 0; if (++kx == p.kw) { kx = 0; ky++; } }
                    }
                    if (++s == (uint32_t)p.stages) { s = 0; use++; }
                }
            }
        }
    } else if (warp == 1) {
        // =========================== MMA issue: the whole warp walks, one lane issues ===========================
        // instruction descriptor: D = s32, A = u8, B = s8, both K-major, N = n_mma, M = 128
        const uint32_t idesc = (2u << 4) | (1u << 10) | ((uint32_t)(n_mma >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t d_a = p.wide ? umma_desc_sw128(smem_u32(stage0)) : umma_desc_sw64(smem_u32(stage0));
        const uint64_t d_b = p.resident ? umma_desc(smem_u32(wres), 512) : umma_desc(smem_u32(stage0) + a_bytes, 512);
        const uint32_t stage_units = (uint32_t)stage_bytes >> 4, wbox_units = (uint32_t)wbox_bytes >> 4, a_step = (uint32_t)(a_bytes1 >> 4);
        const bool leader = elect_lane();
        bool ok = true;
        if (p.resident && !mbar_wait_warp(&bar_w, 0, abort_flag)) {
            atomicCAS(&g_u8_status, 0, 23);
            s_abort = 1;
            ok = false;
        }
        uint32_t s = 0, par = 0;
        int i = 0;   // tiles so far: tile i accumulates in accumulator i % U8_ACCS
        for (int unit = blockIdx.x; unit < nunits && ok; unit += gridDim.x, i += np) {
            for (int t = 0; t < np && ok; t++) {
                const int accbuf = (i + t) % U8_ACCS, accuse = (i + t) / U8_ACCS;
                if (accuse >= 1 && !mbar_wait_warp(&bar_acc_empty[accbuf], (accuse - 1) & 1, abort_flag)) {
                    atomicCAS(&g_u8_status, 0, 22);
                    s_abort = 1;
                    ok = false;
                }
            }
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d_tmem = tmem_base + (i % U8_ACCS) * acc_cols;   // the pair's second accumulator follows the first
            uint32_t accum = 0;
            for (int st = 0; st < nst; st++) {
                if (!mbar_wait_warp(&bar_full[s], par, abort_flag)) {
                    atomicCAS(&g_u8_status, 0, 23);
                    s_abort = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int nb = min(p.G, p.nboxes - st * p.G);
                const uint64_t ad = d_a + (uint64_t)(s * stage_units);
                const uint64_t bd = d_b + (uint64_t)(p.resident ? st * p.G * wbox_units : s * stage_units);
                // one MMA per 32 bytes of K: 32 bytes along the swizzled row of A, two 16-byte units (256 bytes) of B
                if (leader) {
                    if (p.wide) {   // a 128-byte row of A holds the K of two weight boxes; a stage is one such pair (G = 2)
                        const uint64_t bd2 = bd + wbox_units;
#pragma unroll
                        for (int t = 0; t < np; t++) {
                            const uint64_t at = ad + t * a_step;
                            mma_i8_ss(d_tmem + t * acc_cols, at, bd, idesc, accum);
                            mma_i8_ss(d_tmem + t * acc_cols, at + 2, bd + 16, idesc, 1u);
                            mma_i8_ss(d_tmem + t * acc_cols, at + 4, bd2, idesc, 1u);
                            mma_i8_ss(d_tmem + t * acc_cols, at + 6, bd2 + 16, idesc, 1u);
                        }
                    } else {
#pragma unroll
                        for (int b = 0; b < 4; b++) {   // (G is at most four)
                            if (b < nb) {
#pragma unroll
                                for (int t = 0; t < np; t++) {
                                    const uint64_t at = ad + t * a_step + b * (U8_BOX_BYTES >> 4), bt = bd + b * wbox_units;
                                    mma_i8_ss(d_tmem + t * acc_cols, at, bt, idesc, b ? 1u : accum);
                                    mma_i8_ss(d_tmem + t * acc_cols, at + 2, bt + 16, idesc, 1u);
                                }
                            }
                        }
                    }
                    umma_commit(&bar_empty[s]);
                }
                accum = 1u;
                if (++s == (uint32_t)p.stages) { s = 0; par ^= 1u; }
            }
            if (ok && leader)
                for (int t = 0; t < np; t++) umma_commit(&bar_acc_full[(i + t) % U8_ACCS]);
            __syncwarp();
        }
    } else {
        // =========================== epilogue ===========================
        const int ew = warp - 2, group = ew >> 2, r0 = (warp & 3) * 32;   // TMEM lane quarter of a warp = warp % 4
        EpiWarp e;
        e.init(smem_u32(stage0 + p.stages * stage_bytes), ew);
#pragma unroll
        for (int k = 0; k < 4; k++) e.set_row(k, r0 + e.row_of(k), p.N);   // accumulator rows are the tile's pixels in order
        const EpiOut o{p.out, p.out_u8, p.out_bits, p.narrow};
        const EpiChannels ch{pop, chan_a, chan_b};
        // Items: 32-channel chunks of this CTA's tiles in order, dealt to the warp groups in turn.
        const int nchunk = (n_this + 31) >> 5;
        const EpiDiv per_img(p.tiles_per_img, p.ntiles + (int)gridDim.x * 16);
        auto tile_of = [&](int k) { return (blockIdx.x + (k / np) * (int)gridDim.x) * np + k % np; };   // this CTA's k-th tile
        // first output pixel of a tile and how many of its pixels exist
        auto tile_span = [&](int tile, long long& base, int& nvalid) {
            const int tq = per_img(tile), img0 = tq * p.imgs, oh0 = (tile - tq * p.tiles_per_img) * p.rows;
            base = ((long long)img0 * p.OH + oh0) * p.OW;
            nvalid = p.imgs > 1 ? min(p.imgs, p.B - img0) * ohw : min(p.rows, p.OH - oh0) * p.OW;
        };
        auto element = [&](long long base, int chunk) { return (size_t)base * p.N + n0 + chunk * 32 + e.q * 8; };   // of a tile's first pixel, at the lane's channels
        auto limit_of = [&](int nvalid, int chunk) { return chunk * 32 + e.q * 8 < n_this ? (uint32_t)(nvalid * p.N) : 0u; };
        int k = group / nchunk, chunk = group - k * nchunk, tile = tile_of(k);
        long long base = 0;
        int nvalid = 0;
        if (tile < p.ntiles) {
            tile_span(tile, base, nvalid);
            if (p.shortcut) {
                const float* at = p.shortcut + element(base, chunk);
                const uint32_t limit = limit_of(nvalid, chunk);
#pragma unroll
                for (int s = 0; s < 4; s++) e.fetch(s, at, limit, p.narrow);
            }
        }
        while (tile < p.ntiles) {
            int k2 = k, chunk2 = chunk + EPI_GROUPS;   // the item after this one, for the shortcut's prefetch
            while (chunk2 >= nchunk) { chunk2 -= nchunk; k2++; }
            const int tile2 = tile_of(k2);
            long long base2 = 0;
            int nvalid2 = 0;
            const bool more = tile2 < p.ntiles;
            if (more) tile_span(tile2, base2, nvalid2);
            const int accbuf = k % U8_ACCS, cl = chunk * 32 + e.q * 8;
            if (!__all_sync(0xffffffffu, mbar_wait<64>(&bar_acc_full[accbuf], (k / U8_ACCS) & 1, abort_flag))) {
                atomicCAS(&g_u8_status, 0, 24);
                s_abort = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            e.take(tmem_base + ((uint32_t)r0 << 16) + accbuf * acc_cols + chunk * 32);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_acc_empty[accbuf]);   // this warp's share of the accumulator has been read
            if (p.shortcut)
                e.finish<true, false>(o, ch, cl < TC5_MAX_N ? cl : 0, element(base, chunk), limit_of(nvalid, chunk), p.shortcut + element(base2, chunk2), more ? limit_of(nvalid2, chunk2) : 0u);
            else
                e.finish<false, false>(o, ch, cl < TC5_MAX_N ? cl : 0, element(base, chunk), limit_of(nvalid, chunk), nullptr, 0u);
            k = k2; chunk = chunk2; tile = tile2; base = base2; nvalid = nvalid2;
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols));
    }
}

}  // namespace dabnn
