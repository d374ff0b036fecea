// 3x3 stride-1 binary convolution on {0,1}-byte activations in which every input byte enters the SM once per tile.
//
// bconv_u8_kernel loads one box of the tile's pixels per tap: nine copies of (nearly) the same bytes, and on the
// deep layers the weights again for every tile; it runs at the rate at which L2 can feed the SMs.  Here a tile's
// input arrives once, as the halo of the tile: (rows + 2) x (OW + 2) pixels x 64 channels, one tiled TMA load per
// 64-channel group (zero fill outside the image = the reference's padding), 64-byte-swizzled, pixel after pixel at a
// pitch of P = OW + 2.  The pixel operand of tap (ky, kx) is then that same buffer read from pixel ky * P + kx on: the
// K-major SWIZZLE_64B descriptor with its start address advanced by (ky * P + kx) * 64 bytes - the swizzle is a
// function of the final shared-memory address, so a start anywhere inside the swizzle atom reads the rows in order.
// Operand row m of the MMA is halo pixel m, i.e. output pixel (m / P, m % P): the two columns m % P >= OW of every
// output row are computed and never read (116 of 128 rows carry pixels for a 56-pixel row, as against 112 before).
//
// Weights as in bconv_u8.cuh (signed bytes 1 - 2b, per (tap, 64-channel group) box images): resident in shared memory
// when a channel block's nine taps fit, else streamed in stages of one window row (three taps) of one channel group,
// and then a unit of work is two pixel tiles that share every weight stage.  The loop order is channel group, window
// row, tile, tap, so a halo buffer is released after its 18 (36 with two tiles: each its own) MMAs and the ring refills
// while the other groups compute.
//
// Small images (7x7: the last stage of a ResNet) go two to a tile.  The pitch is then P = OW + 1: the zero column left of
// a row doubles as the zero column right of the row above, the second image's halo starts (OH + 1) * P pixels after
// the first one's - its top padding row is the first image's bottom padding row - and one zero pixel, written once at
// start-up, stands behind the second halo for the last pixel's lower right tap.  The two images' boxes are two TMA loads
// into one slot; 98 of the MMA's 128 rows carry pixels, and the nine taps of a pixel cost one load instead of nine.
//
// A block whose result also feeds a 2x2 stride-2 average pooling (the downsample shortcut of the next stage: reference
// layers/AvePool.cpp:84) can write the pooled tensor as well: tiles are then an even number of output rows, the
// four warps of an item leave their results in their buffers and, between two barriers of their own, fold pooled pixels x
// four channels out of them in the reference's tap order, sum first, then the division.
//
// Warps: 0 halo loads, 1 weight loads, 2 MMA issue (one lane each), 3 .. 14 epilogue (bconv_epilogue.cuh, with the
// accumulator row -> pixel mapping above).  Every wait is bounded; a wait that gives up records a code in the
// byte-activation engine's status word (21 halo loader, 25 weight loader, 22 / 23 / 26 MMA thread waiting for an
// accumulator / a halo / a weight stage, 24 epilogue), raises the CTA's abort flag, and the CTA frees its tensor
// memory and returns.
#pragma once
#include "bconv_u8.cuh"

namespace dabnn {

constexpr int HL_THREADS = 96 + EPI_THREADS;   // warps 0, 1, 2 + the epilogue warps
constexpr int HL_MAX_HSLOTS = 8, HL_MAX_WSTAGES = 8;   // (more than four weight stages only with narrow channel blocks)

struct HaloParams {
    const unsigned char* w_img;   // expanded weights (bconv_u8_expand_weights_kernel): box (tap * cw + cg)
    const float *a, *b;
    const float* shortcut;
    float* out;
    unsigned char* out_u8;
    uint64_t* out_bits;
    float* pool_out;              // or null: fp32 [B][OH / 2][OW / 2][N], the 2x2 stride-2 average pooling of `out` (OH, OW, rows even)
    int B, OH, OW, N;
    int cw;                       // 64-channel groups of the input
    int P;                        // halo pitch in pixels: OW + 2 (OW + 1 with two images per tile)
    int imgs, img_pitch;          // images per tile (1 or 2) and, with two, the accumulator rows between them: (OH + 1) * P
    int rows, tiles_per_img, ntiles;
    int hslots, halo_stride;      // halo ring: slots and bytes between them (a multiple of 1024)
    int wstages;                  // weight ring stages of three boxes (streamed weights)
    int wb;                       // rows of a weight box image
    int nb;                       // output channels per CTA: TC5_MAX_N, or 64 / 32 when there are too few tiles to fill the SMs
                                  // (streamed weights only: a CTA then copies its rows out of every box image)
    int resident, pair;
    int narrow;                   // see EpiOut
};

template <bool PAIR, bool POOL>
__global__ void __launch_bounds__(HL_THREADS, 1)
    bconv_halo_kernel(const HaloParams p, const __grid_constant__ CUtensorMap in_map) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t halo_full[HL_MAX_HSLOTS], halo_empty[HL_MAX_HSLOTS], w_full[HL_MAX_WSTAGES], w_empty[HL_MAX_WSTAGES];
    __shared__ __align__(8) uint64_t bar_acc_full[U8_ACCS], bar_acc_empty[U8_ACCS], bar_w;
    __shared__ uint32_t tmem_base_s;
    // epi_abort: POOL, one flag per epilogue group.  Written by the group's own warps between its second barrier and its first,
    // read between the first and the second: all four warps of a group read the same value and leave, or stay, together.
    __shared__ int s_abort, epi_abort[EPI_GROUPS];
    __shared__ __align__(16) float pop[TC5_MAX_N];
    __shared__ __align__(16) float chan_a[TC5_MAX_N];
    __shared__ __align__(16) float chan_b[TC5_MAX_N];

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int n0 = blockIdx.y * p.nb;
    const int n_this = min(p.nb, p.N - n0);        // multiple of 16 (host-checked)
    const int n_mma = n_this;
    constexpr int np = PAIR ? 2 : 1;
    const int nunits = (p.ntiles + np - 1) / np;
    const int nboxes = 9 * p.cw, gbox_bytes = p.wb * 64, wbox_bytes = min(p.nb, p.wb) * 64;   // a box image in global / this CTA's rows of it
    unsigned char* halo0 = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
    unsigned char* wbase = halo0 + p.hslots * p.halo_stride;                                   // resident weights or the weight ring
    unsigned char* epi_buf = wbase + (p.resident ? nboxes * wbox_bytes : p.wstages * 3 * wbox_bytes);   // a multiple of 1024 bytes further
    const int acc_cols = (n_mma + 31) & ~31;       // columns between accumulators: whole 32-column items
    int tmem_cols = 32;
    while (tmem_cols < U8_ACCS * acc_cols) tmem_cols <<= 1;
    const volatile int* abort_flag = &s_abort;
    const uint32_t halo_tx = (uint32_t)(p.imgs * (p.rows + 2) * p.P * 64);

    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        for (int i = 0; i < p.hslots; i++) { mbar_init(&halo_full[i], 1); mbar_init(&halo_empty[i], 1); }
        for (int i = 0; i < HL_MAX_WSTAGES; i++) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 1); }
        for (int i = 0; i < U8_ACCS; i++) { mbar_init(&bar_acc_full[i], 1); mbar_init(&bar_acc_empty[i], 4 * ((n_this + 31) >> 5)); }
        mbar_init(&bar_w, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::);
        s_abort = 0;
        for (int i = 0; i < EPI_GROUPS; i++) epi_abort[i] = 0;
    }
    if (p.imgs == 2 && tid < p.hslots * 4)   // the zero pixel behind the second image's halo (never written again)
        sts128(smem_u32(halo0) + (tid >> 2) * p.halo_stride + (p.img_pitch + (p.rows + 2) * p.P) * 64 + (tid & 3) * 16, 0u, 0u, 0u, 0u);
    if (tid < TC5_MAX_N) {
        pop[tid] = epi_pop(tid < n_this ? __ldg(reinterpret_cast<const int*>(p.w_img + u8_weight_image_bytes(p.N, nboxes)) + n0 + tid) : 0);
        const bool have = p.a && tid < n_this;
        chan_a[tid] = have ? __ldg(p.a + n0 + tid) : 1.f;
        chan_b[tid] = have ? __ldg(p.b + n0 + tid) : 0.f;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    // this CTA's rows of its channel block's box images
    const unsigned char* wsrc = p.w_img + (size_t)(n0 / TC5_MAX_N) * nboxes * gbox_bytes + (size_t)(n0 % TC5_MAX_N) * 64;
    grid_launch_dependents();
    if (warp != 1) grid_dependency_wait();   // the weight loader reads constants only and may run ahead of the previous kernel's end

    if (warp == 0) {
        // =========================== halo loads: one lane ===========================
        if (lane == 0) {
            const uint32_t halo0_addr = smem_u32(halo0);
            uint32_t hs = 0, huse = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < nunits && ok; unit += gridDim.x) {
                int img[2], oh0[2];   // a tile past the last one lies outside the tensor: its load delivers zeros
                for (int t = 0; t < np; t++) {
                    const int tile = unit * np + t;
                    if (p.imgs == 2) { img[t] = tile * 2; oh0[t] = 0; }
                    else { img[t] = tile / p.tiles_per_img; oh0[t] = (tile - img[t] * p.tiles_per_img) * p.rows; }
                }
                for (int cg = 0; cg < p.cw && ok; cg++)
                    for (int t = 0; t < np; t++) {
                        if (huse >= 1 && !mbar_wait<32>(&halo_empty[hs], (huse - 1) & 1, abort_flag)) {
                            atomicCAS(&g_u8_status, 0, 21);
                            s_abort = 1;
                            ok = false;
                            break;
                        }
                        const uint32_t bar = smem_u32(&halo_full[hs]);
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(halo_tx) : "memory");
                        for (int j = 0; j < p.imgs; j++)   // (an image past the last one lies outside the tensor: zeros)
                            asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
                                         ::"r"(halo0_addr + hs * p.halo_stride + j * p.img_pitch * 64), "l"(reinterpret_cast<uint64_t>(&in_map)), "r"(cg * 64), "r"(-1),
                                           "r"(oh0[t] - 1), "r"(img[t] + j), "r"(0), "r"(bar) : "memory");
                        if (++hs == (uint32_t)p.hslots) { hs = 0; huse++; }
                    }
            }
        }
    } else if (warp == 1) {
        // =========================== weight loads: one lane ===========================
        if (lane == 0) {
            if (p.resident) {   // the whole channel block, once
                const uint32_t bytes = (uint32_t)(nboxes * wbox_bytes), bar = smem_u32(&bar_w);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(wbase)), "l"(wsrc), "r"(bytes), "r"(bar) : "memory");
            } else {
                const uint32_t w0_addr = smem_u32(wbase);
                uint32_t ws = 0, wuse = 0;
                bool ok = true;
                for (int unit = blockIdx.x; unit < nunits && ok; unit += gridDim.x)
                    for (int cg = 0; cg < p.cw && ok; cg++)
                        for (int ky = 0; ky < 3; ky++) {
                            if (wuse >= 1 && !mbar_wait<32>(&w_empty[ws], (wuse - 1) & 1, abort_flag)) {
                                atomicCAS(&g_u8_status, 0, 25);
                                s_abort = 1;
                                ok = false;
                                break;
                            }
                            const uint32_t bar = smem_u32(&w_full[ws]), dst = w0_addr + ws * 3 * wbox_bytes;
                            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(3u * wbox_bytes) : "memory");
                            for (int kx = 0; kx < 3; kx++)   // the three taps of window row ky of this channel group
                                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                             ::"r"(dst + kx * wbox_bytes), "l"(wsrc + (size_t)((ky * 3 + kx) * p.cw + cg) * gbox_bytes), "r"((uint32_t)wbox_bytes),
                                               "r"(bar) : "memory");
                            if (++ws == (uint32_t)p.wstages) { ws = 0; wuse++; }
                        }
            }
        }
    } else if (warp == 2) {
        // =========================== MMA issue: the whole warp walks, one lane issues ===========================
        // instruction descriptor: D = s32, A = u8, B = s8, both K-major, N = n_mma, M = 128
        const uint32_t idesc = (2u << 4) | (1u << 10) | ((uint32_t)(n_mma >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t d_halo = umma_desc_sw64(smem_u32(halo0));
        const uint64_t d_w = umma_desc(smem_u32(wbase), 512);
        const uint32_t halo_units = (uint32_t)p.halo_stride >> 4, wbox_units = (uint32_t)wbox_bytes >> 4, row_units = (uint32_t)p.P * 4u;
        const bool leader = elect_lane();
        bool ok = true;
        if (p.resident && !mbar_wait_warp(&bar_w, 0, abort_flag)) {
            atomicCAS(&g_u8_status, 0, 26);
            s_abort = 1;
            ok = false;
        }
        uint32_t hs = 0, hpar = 0, ws = 0, wpar = 0;
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
            uint32_t d_tmem[np];
            for (int t = 0; t < np; t++) d_tmem[t] = tmem_base + ((i + t) % U8_ACCS) * acc_cols;
            uint32_t accum = 0;
            for (int cg = 0; cg < p.cw && ok; cg++) {
                uint32_t slot[np];
                for (int t = 0; t < np; t++) {   // this group's halo of every tile of the unit
                    if (!mbar_wait_warp(&halo_full[hs], hpar, abort_flag)) {
                        atomicCAS(&g_u8_status, 0, 23);
                        s_abort = 1;
                        ok = false;
                        break;
                    }
                    slot[t] = hs;
                    if (++hs == (uint32_t)p.hslots) { hs = 0; hpar ^= 1u; }
                }
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int ky = 0; ky < 3; ky++) {
                    uint64_t bd;
                    if (p.resident) {
                        bd = d_w + (uint64_t)((ky * 3 * p.cw + cg) * wbox_units);
                    } else {
                        if (!mbar_wait_warp(&w_full[ws], wpar, abort_flag)) {
                            atomicCAS(&g_u8_status, 0, 26);
                            s_abort = 1;
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        bd = d_w + (uint64_t)(ws * 3 * wbox_units);
                    }
                    const uint32_t bstep = p.resident ? (uint32_t)p.cw * wbox_units : wbox_units;   // from tap kx to tap kx + 1
                    if (leader) {
#pragma unroll
                        for (int t = 0; t < np; t++) {
                            // tap (ky, kx): the halo read from pixel ky * P + kx on; 32 bytes of K per MMA
                            const uint64_t ad = d_halo + (uint64_t)(slot[t] * halo_units + ky * row_units);
#pragma unroll
                            for (int kx = 0; kx < 3; kx++) {
                                mma_i8_ss(d_tmem[t], ad + kx * 4, bd + kx * bstep, idesc, kx ? 1u : accum);
                                mma_i8_ss(d_tmem[t], ad + kx * 4 + 2, bd + kx * bstep + 16, idesc, 1u);
                            }
                        }
                        if (!p.resident) umma_commit(&w_empty[ws]);
                    }
                    accum = 1u;
                    if (!p.resident && ++ws == (uint32_t)p.wstages) { ws = 0; wpar ^= 1u; }
                }
                if (ok && leader)
                    for (int t = 0; t < np; t++) umma_commit(&halo_empty[slot[t]]);
            }
            if (ok && leader)
                for (int t = 0; t < np; t++) umma_commit(&bar_acc_full[(i + t) % U8_ACCS]);
            __syncwarp();
        }
    } else {
        // =========================== epilogue ===========================
        // Accumulator row r is halo pixel r: output row r / P of the tile, column r % P; it has a pixel when the column is
        // below OW.
        const int ew = warp - 3, group = ew >> 2, r0 = (warp & 3) * 32;   // TMEM lane quarter of a warp = warp % 4
        EpiWarp e;
        const uint32_t epi_addr = smem_u32(epi_buf);
        e.init(epi_addr, ew);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int r = r0 + e.row_of(k);
            const int second = (p.imgs == 2 && r >= p.img_pitch) ? 1 : 0, rr = r - second * p.img_pitch;   // which image of the tile
            const int orow = rr / p.P, ocol = rr - orow * p.P;
            e.set_row(k, ocol < p.OW && orow < p.rows ? (second * p.rows + orow) * p.OW + ocol : -1, p.N);   // the pixel's index within the tile
        }
        const EpiOut o{p.out, p.out_u8, p.out_bits, p.narrow};
        const EpiChannels ch{pop, chan_a, chan_b};
        // Items: 32-channel chunks of this CTA's tiles in order, dealt to the warp groups in turn.
        const int nchunk = (n_this + 31) >> 5;
        const EpiDiv per_img(p.tiles_per_img, p.ntiles + (int)gridDim.x * 16);
        auto tile_of = [&](int k) { return (blockIdx.x + (k / np) * (int)gridDim.x) * np + k % np; };      // this CTA's k-th tile
        auto tile_span = [&](int tile, long long& base, int& nvalid) {
            if (p.imgs == 2) {   // whole images, the last tile may hold one
                base = (long long)tile * 2 * p.OH * p.OW;
                nvalid = max(0, min(2, p.B - tile * 2)) * p.OH * p.OW;
                return;
            }
            const int img = per_img(tile), oh0 = (tile - img * p.tiles_per_img) * p.rows;
            base = ((long long)img * p.OH + oh0) * p.OW;
            nvalid = min(p.rows, p.OH - oh0) * p.OW;
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
        // POOL: the group folds its item's 32 channels: a thread takes four of them (pool_quad) of the tile's pooled pixels
        // pool_px, pool_px + 16, ...
        const int tid_g = (ew & 3) * 32 + lane, pool_quad = tid_g & 7, pool_px = tid_g >> 3, pw = p.OW >> 1, pool_pixels = (p.rows >> 1) * pw;
        auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
        bool alive = true;
        while (alive && tile < p.ntiles) {
            const int ptile = tile, pchunk = chunk;
            // the item after this one, for the shortcut's prefetch
            int k2 = k, chunk2 = chunk + EPI_GROUPS;
            while (chunk2 >= nchunk) { chunk2 -= nchunk; k2++; }
            const int tile2 = tile_of(k2);
            long long base2 = 0;
            int nvalid2 = 0;
            const bool more = tile2 < p.ntiles;
            if (more) tile_span(tile2, base2, nvalid2);
            const int accbuf = k % U8_ACCS, cl = chunk * 32 + e.q * 8;
            alive = mbar_wait_warp<64>(&bar_acc_full[accbuf], (k / U8_ACCS) & 1, abort_flag);
            if (!alive) {
                atomicCAS(&g_u8_status, 0, 24);
                s_abort = 1;
                epi_abort[group] = 1;
            } else {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                e.take(tmem_base + ((uint32_t)r0 << 16) + accbuf * acc_cols + chunk * 32);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_acc_empty[accbuf]);   // this warp's share of the accumulator has been read
                if (p.shortcut)
                    e.finish<true, POOL>(o, ch, cl < TC5_MAX_N ? cl : 0, element(base, chunk), limit_of(nvalid, chunk), p.shortcut + element(base2, chunk2), more ? limit_of(nvalid2, chunk2) : 0u);
                else
                    e.finish<false, POOL>(o, ch, cl < TC5_MAX_N ? cl : 0, element(base, chunk), limit_of(nvalid, chunk), nullptr, 0u);
            }
            k = k2; chunk = chunk2; tile = tile2; base = base2; nvalid = nvalid2;
            if (POOL) {
                // 2x2 average pooling of the item
                group_sync();
                if (epi_abort[group]) break;
                if (pchunk * 32 + pool_quad * 4 < n_this) {
                    const int img = per_img(ptile), oh0 = (ptile - img * p.tiles_per_img) * p.rows;
                    for (int pp = pool_px; pp < pool_pixels; pp += 16) {
                        const int prow = pp / pw, pcol = pp - prow * pw;
                        if (oh0 + 2 * prow + 1 >= p.OH) break;
                        float4 x[4];
#pragma unroll
                        for (int tap = 0; tap < 4; tap++) {
                            const int r = (2 * prow + (tap >> 1)) * p.P + 2 * pcol + (tap & 1);   // the accumulator row: its warp is the one
                            const int w = group * 4 + ((r / 32 + 1) & 3);                         // whose index modulo four is r / 32
                            x[tap] = lds128f(epi_addr + w * EPI_WARP_BYTES + (r & 31) * 128 + ((pool_quad ^ (r & 7)) << 4));
                        }
                        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int tap = 0; tap < 4; tap++) {   // the reference's order: (0,0), (0,1), (1,0), (1,1)
                            acc.x = __fadd_rn(acc.x, x[tap].x); acc.y = __fadd_rn(acc.y, x[tap].y); acc.z = __fadd_rn(acc.z, x[tap].z); acc.w = __fadd_rn(acc.w, x[tap].w);
                        }
                        // (a quarter is a power of two: the product is the quotient)
                        const size_t d = ((((size_t)img * (p.OH >> 1) + (oh0 >> 1) + prow) * pw) + pcol) * p.N + n0 + pchunk * 32 + pool_quad * 4;
                        *reinterpret_cast<float4*>(p.pool_out + d) =
                            make_float4(__fmul_rn(acc.x, 0.25f), __fmul_rn(acc.y, 0.25f), __fmul_rn(acc.z, 0.25f), __fmul_rn(acc.w, 0.25f));
                    }
                }
                group_sync();   // the buffers may be overwritten
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols));
    }
}

}  // namespace dabnn
