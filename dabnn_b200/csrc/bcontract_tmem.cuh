// Binary contraction with the pixel operand in tensor memory: tcgen05.mma kind::i8, A from TMEM, B resident in shared memory.
//
//   cnt[p][n] = sum_k x[p][k] XOR w[n][k] = popc(w[n]) + sum_k x[p][k] * (1 - 2 w[n][k])
//
// with 1 - 2 w as +1 / -1 bytes.  The kernel of bcontract_tc5.cuh expands both operands into shared memory for every tile, and
// its shared-memory pipe is what runs out: per 32 bytes of K it writes 8 KB and the tensor core reads them back.  Here
//   * the CTA's filters are expanded once, before the first tile, and stay in shared memory (the channel block is narrowed
//     until they fit: tmem_plan in contraction.cu), or are streamed for four tiles at a time (second kernel below);
//   * the producers, thread = pixel row, write their expanded bytes with tcgen05.st straight to the tensor-memory columns that
//     the MMA reads as its A operand (lane = row, a column = four bytes of K): no shared-memory traffic at all;
//   * the +1 / -1 filters make the accumulator the count less popc(w): nothing per pixel row travels to the epilogue;
//   * the epilogue is the one of independent warps (bconv_epilogue.cuh).
// Both operands use the same bit -> K-slot permutation (expand32), which a contraction is blind to.
//
// What bounds it: the producers' instruction issue at long K, the epilogue (and HBM: the fp32 output and shortcut) at short K.
// Against the kernel of bcontract_tc5.cuh, us a launch: block of 256 x 28x28x128 -> 128 3x3 with shortcut 78.5 -> 53.6 (212 MB,
// 32 us at the copy rate), 256 x 56x56x64 -> 64 179 -> 98, 256 x 14x14x256 -> 256 72 -> 49; 256 x 14x14x256 -> 512 1x1 49 -> 27;
// 802816 x 64 x 576 GEMM 150 -> 87; 49 x 512 x 4608 25 -> 10.5.  Left shifts instead of right ones in the expansion: 14x14x256
// 54 -> 49, 7x7x512 at 32 channels 85 -> 75; groups of producers in turn instead of half a stage each: 72 -> 54.
//
// Tensor memory: columns 0 - 255 hold the accumulators, 256 - 511 four stages of 64 columns (256 bits of K).
// Every wait on an mbarrier is bounded, with the status codes of bcontract_tc5.cuh.
#pragma once
#include "bconv_epilogue.cuh"

namespace dabnn {

constexpr int TM_STAGES = 4, TM_WORDS = 4;           // ring stages, 64-bit words of K per stage
constexpr int TM_STAGE_COLS = TM_WORDS * 16, TM_A_COL = 256;
constexpr int TM_AHEAD = 3;                          // stages of its own that a producer's loads run ahead
constexpr int TM_WARPS = 16;                         // producers + epilogue
constexpr int TM_THREADS = TM_WARPS * 32 + 32;
constexpr int TM_MAX_ACCS = 4;
constexpr int TM_MAX_LD = 1 << 24;                   // output pitch (the epilogue's 32-bit offsets within a tile)

struct TmemPlan {
    int nbc;                                         // channels per CTA
    int producer_warps;                              // 4, 8 or 12
};
__host__ __device__ inline int tmem_smem_bytes(int nbc, int kwords, int producer_warps) {
    return kwords * nbc * 64 + (TM_WARPS - producer_warps) * EPI_WARP_BYTES + 128 /*alignment slack*/;
}

__device__ __forceinline__ void mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bd, uint32_t idesc, uint32_t accum) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(bd), "r"(idesc), "r"(accum), "r"(0), "r"(0), "r"(0), "r"(0) : "memory");
}
// One 64-bit word of the warp's 32 rows -> 16 tensor-memory columns, K slots as expand32 orders them.  A set bit becomes the byte
// 128: left shifts are multiplications and leave the logic pipe, which the masks alone keep busy.  The accumulator is scaled
// back, exactly, in the epilogue.
constexpr int TM_MAX_WORDS = (1 << 21) / 128 / 64 - 1;   // |accumulator| stays below 2^21 (EpiWarp::finish)
__device__ __forceinline__ void tmem_st_word(uint32_t t_addr, uint64_t word) {
    const uint32_t M = 0x80808080u, l = (uint32_t)word, h = (uint32_t)(word >> 32);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(t_addr), "r"((l << 7) & M), "r"((l << 6) & M), "r"((l << 5) & M), "r"((l << 4) & M), "r"((l << 3) & M), "r"((l << 2) & M),
                   "r"((l << 1) & M), "r"(l & M), "r"((h << 7) & M), "r"((h << 6) & M), "r"((h << 5) & M), "r"((h << 4) & M), "r"((h << 3) & M),
                   "r"((h << 2) & M), "r"((h << 1) & M), "r"(h & M)
                 : "memory");
}

// one word of a filter row -> its four 16-byte units of +1 / -1 bytes
__device__ __forceinline__ void expand_filter_word(uint32_t dst, uint64_t word) {
    auto sgn = [](uint32_t x) { const uint32_t m = x & 0x01010101u; return (m * 0xffu) | (m ^ 0x01010101u); };   // 0 -> +1, 1 -> -1
#pragma unroll
    for (int u = 0; u < 4; u++) {                        // unit u: bits s + 8 i of the half word, s = 4 (u & 1) ..
        const uint32_t half = (uint32_t)(word >> (u >= 2 ? 32 : 0)) >> (4 * (u & 1));
        sts128(dst + u * TC5_LBO, sgn(half), sgn(half >> 1), sgn(half >> 2), sgn(half >> 3));
    }
}
// WORDS (even) consecutive words of an operand row from word q on, d = their position; words beyond kwords are zero
template <int WORDS, class XOp>
__device__ __forceinline__ void load_words(uint64_t (&v)[WORDS], const XOp& xop, const RowCtx& row, typename XOp::Dec& d, int q, int kwords, bool pair) {
#pragma unroll
    for (int j = 0; j < WORDS; j += 2) {
        v[j] = 0; v[j + 1] = 0;
        if (q + j < kwords) {
            const uint64_t* p = xop.addr(row, d);
            if (pair && q + j + 1 < kwords) {            // two words of one tap on a 16-byte boundary
                if (p) {
                    const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2*>(p));
                    v[j] = t.x; v[j + 1] = t.y;
                }
                xop.advance(d, 2);
            } else {
                if (p) v[j] = __ldg(p);
                xop.advance(d, 1);
                if (q + j + 1 < kwords) {
                    p = xop.addr(row, d);
                    if (p) v[j + 1] = __ldg(p);
                }
                xop.advance(d, 1);
            }
        }
    }
}

// The epilogue warps' side of a CTA: items of 32 channels of its tiles in order, dealt to the groups of four warps in turn.
template <int EW>
__device__ __forceinline__ void tmem_epilogue(const EpilogueParams& ep, const EpiChannels& ch, const int ew, const uint32_t epi_smem,
                                              const uint32_t tmem_base, const int n0, const int n_this, const int M, const int ntiles_m,
                                              const int acc_cols, const int naccs, const int narrow, uint64_t* bar_acc_full,
                                              uint64_t* bar_acc_empty, int* s_abort) {
    constexpr int EGROUPS = EW / 4;
    const volatile int* abort_flag = s_abort;
    const int group = ew >> 2, r0 = ((threadIdx.x >> 5) & 3) * 32, ld = (int)ep.ld_out;   // TMEM lane quarter = warp % 4
    const float* const addsrc = ep.shortcut ? ep.shortcut : ep.accumulate ? ep.out : nullptr;
    EpiWarp e;
    e.init(epi_smem, ew);
#pragma unroll
    for (int k = 0; k < 4; k++) e.set_row(k, r0 + e.row_of(k), ld);
    const EpiOut o{ep.out, nullptr, ep.bits, narrow};
    const int nchunk = (n_this + 31) >> 5;
    auto element = [&](int tile, int chunk) { return (size_t)tile * 128 * ld + n0 + chunk * 32 + e.q * 8; };
    auto limit_of = [&](int tile, int chunk) { return chunk * 32 + e.q * 8 < n_this ? (uint32_t)(min(128, M - tile * 128) * ld) : 0u; };
    int k = 0, chunk = group;
    while (chunk >= nchunk) { chunk -= nchunk; k++; }
    int tile = blockIdx.x + k * gridDim.x;
    if (addsrc && tile < ntiles_m) {
        const float* at = addsrc + element(tile, chunk);
        const uint32_t limit = limit_of(tile, chunk);
#pragma unroll
        for (int s = 0; s < 4; s++) e.fetch(s, at, limit, narrow);
    }
    while (tile < ntiles_m) {
        int k2 = k, chunk2 = chunk + EGROUPS;   // the item after this one, for the shortcut's prefetch
        while (chunk2 >= nchunk) { chunk2 -= nchunk; k2++; }
        const int tile2 = blockIdx.x + k2 * gridDim.x;
        const int acc = k & (naccs - 1), cl = chunk * 32 + e.q * 8;
        if (!mbar_wait_warp<64>(&bar_acc_full[acc], (k / naccs) & 1, abort_flag)) {
            atomicCAS(&g_tc5_status, 0, 2);
            *s_abort = 1;
            break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        e.take(tmem_base + ((uint32_t)r0 << 16) + acc * acc_cols + chunk * 32);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (e.lane == 0) mbar_arrive(&bar_acc_empty[acc]);   // this warp's share of the accumulator has been read
        if (addsrc)
            e.finish<true, false, true>(o, ch, cl, element(tile, chunk), limit_of(tile, chunk), tile2 < ntiles_m ? addsrc + element(tile2, chunk2) : addsrc,
                                        tile2 < ntiles_m ? limit_of(tile2, chunk2) : 0u);
        else
            e.finish<false, false, true>(o, ch, cl, element(tile, chunk), limit_of(tile, chunk), nullptr, 0u);
        k = k2; chunk = chunk2; tile = tile2;
    }
}

// PW producer warps, the other 16 - PW are the epilogue.  The output pitch ep.ld_out is also the shortcut's; sign bits are
// written for ep.ld_out == N only (host-checked).
template <int PW, class XOp, class WOp>
__global__ void __launch_bounds__(TM_THREADS, 1)
    bcontract_tmem_kernel(const XOp xop, const WOp wop, const EpilogueParams ep, const int M, const int N, const int kwords, const int ntiles_m,
                          const int nbc, const int narrow, const int weights_first) {
    constexpr int EW = TM_WARPS - PW, PGROUPS = PW / 4;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t bar_full[TM_STAGES], bar_empty[TM_STAGES], bar_acc_full[TM_MAX_ACCS], bar_acc_empty[TM_MAX_ACCS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_abort, popw[TC5_MAX_N];
    __shared__ __align__(16) float pop[TC5_MAX_N];
    __shared__ __align__(16) float chan_a[TC5_MAX_N];
    __shared__ __align__(16) float chan_b[TC5_MAX_N];

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int n0 = blockIdx.y * nbc, n_this = min(nbc, N - n0);              // a multiple of 16 (host-checked)
    const int nchunks = (kwords + TM_WORDS - 1) / TM_WORDS;
    const int acc_cols = (n_this + 31) & ~31, naccs = acc_cols > 64 ? 2 : TM_MAX_ACCS;   // columns per accumulator: whole 32-column items
    const uint32_t wimg = (smem_u32(smem_dyn) + 127) & ~127u, wbox = (uint32_t)nbc * 64u;   // filters: [word][row / 8][unit][row % 8][16 bytes]
    const uint32_t epi_smem = wimg + (uint32_t)kwords * wbox;
    const volatile int* abort_flag = &s_abort;

    if (warp == TM_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base_s)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        for (int i = 0; i < TM_STAGES; i++) { mbar_init(&bar_full[i], 4); mbar_init(&bar_empty[i], 1); }
        for (int i = 0; i < TM_MAX_ACCS; i++) { mbar_init(&bar_acc_full[i], 1); mbar_init(&bar_acc_empty[i], 4 * ((n_this + 31) >> 5)); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::);
        s_abort = 0;
    }
    if (tid < TC5_MAX_N) popw[tid] = 0;
    // Filters that no kernel still running may be writing are read while that kernel drains (weights_first); otherwise after it.
    if (!weights_first) grid_dependency_wait();
    if (tid < TC5_MAX_N) {
        const bool have = ep.a && tid < n_this;
        chan_a[tid] = have ? __ldg(ep.a + n0 + tid) : 1.f;
        chan_b[tid] = have ? __ldg(ep.b + n0 + tid) : 0.f;
    }
    __syncthreads();
    {   // thread = channel (lanes) x word, eight loads in flight
        const int nlog = 31 - __clz(nbc);                                    // nbc is a power of two
        const int r = tid & (nbc - 1), per = TM_WARPS * 32 >> nlog;
        if (tid < TM_WARPS * 32 && r < n_this) {
            const RowCtx row = wop.make_row(n0 + r);
            const uint32_t dst = wimg + (r >> 3) * 512 + (r & 7) * 16;
            int pc = 0;
            for (int q0 = tid >> nlog; q0 < kwords; q0 += per * 8) {
                uint64_t w[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int q = q0 + j * per;
                    w[j] = 0;
                    if (q < kwords) w[j] = __ldg(wop.addr(row, wop.decode(q)));
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int q = q0 + j * per;
                    if (q < kwords) {
                        pc += __popcll(w[j]);
                        expand_filter_word(dst + (uint32_t)q * wbox, w[j]);
                    }
                }
            }
            atomicAdd(&popw[r], pc);
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads what was just written
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    if (weights_first) grid_dependency_wait();   // activations (and what is added to) come next

    if (warp < PW) {
        // =========================== producers: thread = operand row ===========================
        // The groups of four warps take the stages in turn, so that a group has several stages' time for the chain wait - write -
        // wait for the writes - hand over.  Its loads run TM_AHEAD of its stages ahead and do not stop at tile boundaries: the
        // cursor below walks (tile, stage).
        const int group = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t a_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + TM_A_COL;
        const bool pair = xop.pairable();
        struct Words { uint64_t w[TM_WORDS]; };
        int ltile = blockIdx.x, lchunk = group;
        while (lchunk >= nchunks) { lchunk -= nchunks; ltile += gridDim.x; }
        RowCtx xr = xop.make_row(ltile * 128 + r);
        typename XOp::Dec xd = xop.decode(lchunk * TM_WORDS);
        auto load_next = [&](Words& v) {
            if (ltile < ntiles_m) load_words(v.w, xop, xr, xd, lchunk * TM_WORDS, kwords, pair);
            lchunk += PGROUPS;
            if (lchunk < nchunks) {
                xop.advance(xd, (PGROUPS - 1) * TM_WORDS);
            } else {
                do { lchunk -= nchunks; ltile += gridDim.x; } while (lchunk >= nchunks);
                xr = xop.make_row(ltile * 128 + r);
                xd = xop.decode(lchunk * TM_WORDS);
            }
        };
        Words v[TM_AHEAD];
#pragma unroll
        for (int j = 0; j < TM_AHEAD; j++) load_next(v[j]);
        const int total = ((ntiles_m - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * nchunks;   // stages of this CTA
        bool ok = true;
        for (int i = group; i < total && ok;) {
#pragma unroll
            for (int j = 0; j < TM_AHEAD; j++, i += PGROUPS) {
                if (i >= total || !ok) break;
                const uint32_t s = i % TM_STAGES, use = i / TM_STAGES;
                if (use >= 1) ok = mbar_wait_warp(&bar_empty[s], (use - 1) & 1, abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");   // the MMAs that read this stage are complete
#pragma unroll
                for (int w = 0; w < TM_WORDS; w++) tmem_st_word(a_addr + s * TM_STAGE_COLS + w * 16, v[j].w[w]);   // (words beyond K: zeros that no MMA reads)
                load_next(v[j]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_full[s]);
            }
        }
        if (!ok) {
            atomicCAS(&g_tc5_status, 0, 1);
            s_abort = 1;
        }
    } else if (warp == TM_WARPS) {
        // =========================== MMA issue: the whole warp walks, one lane issues ===========================
        // instruction descriptor: D = s32, A = u8, B = s8, both K-major, N = n_this, M = 128
        const uint32_t idesc = (2u << 4) | (1u << 10) | ((uint32_t)(n_this >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t d_b = umma_desc(wimg, 512);
        const uint32_t wbox_units = wbox >> 4;
        const bool leader = elect_lane();
        uint32_t s = 0, par = 0;
        bool ok = true;
        int acc = 0, accpar = 0, first = 1;
        for (int tile = blockIdx.x; tile < ntiles_m && ok; tile += gridDim.x) {
            if (!first && !mbar_wait_warp(&bar_acc_empty[acc], accpar ^ 1, abort_flag)) {
                atomicCAS(&g_tc5_status, 0, 3);
                s_abort = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d_tmem = tmem_base + acc * acc_cols;
            uint64_t bd = d_b;
            for (int c = 0; c < nchunks; c++, bd += TM_WORDS * wbox_units) {
                if (!mbar_wait_warp(&bar_full[s], par, abort_flag)) {
                    atomicCAS(&g_tc5_status, 0, 4);
                    s_abort = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int words = min(TM_WORDS, kwords - c * TM_WORDS);
                const uint32_t at = tmem_base + TM_A_COL + s * TM_STAGE_COLS;
                if (leader) {   // one MMA per 32 bytes of K: eight columns of A, two 16-byte units (256 bytes) of B
#pragma unroll
                    for (int j = 0; j < TM_WORDS; j++)
                        if (j < words) {
                            mma_i8_ts(d_tmem, at + j * 16, bd + j * wbox_units, idesc, c + j ? 1u : 0u);
                            mma_i8_ts(d_tmem, at + j * 16 + 8, bd + j * wbox_units + 16, idesc, 1u);
                        }
                    umma_commit(&bar_empty[s]);
                }
                if (++s == TM_STAGES) { s = 0; par ^= 1u; }
            }
            if (ok && leader) umma_commit(&bar_acc_full[acc]);
            __syncwarp();
            if (++acc == naccs) { acc = 0; accpar ^= 1; first = 0; }
        }
    } else {
        // =========================== epilogue ===========================
        if (tid - PW * 32 < TC5_MAX_N) pop[tid - PW * 32] = epi_pop_scaled(popw[tid - PW * 32]);
        asm volatile("bar.sync 1, %0;" ::"n"(EW * 32) : "memory");
        tmem_epilogue<EW>(ep, EpiChannels{pop, chan_a, chan_b}, warp - PW, epi_smem, tmem_base, n0, n_this, M, ntiles_m, acc_cols, naccs, narrow,
                          bar_acc_full, bar_acc_empty, &s_abort);
    }

    // ---- everybody is past its last use of the tensor memory ----
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == TM_WARPS) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base));
    }
}

// ---- the same for K too long for the filters to stay in shared memory ----
// 64 channels per CTA and up to four pixel tiles at a time, each with an accumulator of its own: a stage of 256 bits of K of the
// filters is expanded once for the four tiles (by four warps of their own, into a ring of eight stages) and the steps run
// K-stage by K-stage, tile by tile.  A word of a tile then costs what it costs with resident filters of 64 channels; the next
// narrower resident block, 32 channels, expands every pixel row twice as often.  8 producer warps (tiles t = group, group + 2),
// 4 filter warps, 4 epilogue warps.  Bound by the producers' instruction issue, with a gap while the four accumulators are read.
// us against the kernel of bcontract_tc5.cuh: 12544 x 512 x 4608 58.8 -> 49.9, 64 x 28x28x384 -> 512 5x5 433 -> 353,
// 128 x 28x28x128 -> 64 5x5 87 -> 43, block of 256 x 7x7x512 -> 512 70.6 -> 58.0.
constexpr int TS_NBC = 64, TS_TILES = 4, TS_PW = 8, TS_FW = 4, TS_EW = 4, TS_BSTAGES = 8;
constexpr int TS_BSTAGE_BYTES = TM_WORDS * TS_NBC * 64;
constexpr int TS_SMEM_BYTES = TS_BSTAGES * TS_BSTAGE_BYTES + TS_EW * EPI_WARP_BYTES + 128;

template <class XOp, class WOp>
__global__ void __launch_bounds__(TM_THREADS, 1)
    bcontract_tmem_stream_kernel(const XOp xop, const WOp wop, const EpilogueParams ep, const int M, const int N, const int kwords, const int ntiles_m,
                                 const int narrow) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t bar_full[TM_STAGES], bar_empty[TM_STAGES], bar_bfull[TS_BSTAGES], bar_bempty[TS_BSTAGES];
    __shared__ __align__(8) uint64_t bar_acc_full[TS_TILES], bar_acc_empty[TS_TILES];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_abort, popw[TS_NBC];
    __shared__ __align__(16) float pop[TS_NBC];
    __shared__ __align__(16) float chan_a[TS_NBC];
    __shared__ __align__(16) float chan_b[TS_NBC];

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int n0 = blockIdx.y * TS_NBC, n_this = min(TS_NBC, N - n0);
    const int nchunks = (kwords + TM_WORDS - 1) / TM_WORDS;
    const int my_tiles = (ntiles_m - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const uint32_t bring = (smem_u32(smem_dyn) + 127) & ~127u, epi_smem = bring + TS_BSTAGES * TS_BSTAGE_BYTES;
    const volatile int* abort_flag = &s_abort;

    if (warp == TM_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base_s)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        for (int i = 0; i < TM_STAGES; i++) { mbar_init(&bar_full[i], 4); mbar_init(&bar_empty[i], 1); }
        for (int i = 0; i < TS_BSTAGES; i++) { mbar_init(&bar_bfull[i], TS_FW); mbar_init(&bar_bempty[i], 1); }
        for (int i = 0; i < TS_TILES; i++) { mbar_init(&bar_acc_full[i], 1); mbar_init(&bar_acc_empty[i], 4 * ((n_this + 31) >> 5)); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::);
        s_abort = 0;
    }
    if (tid < TS_NBC) {
        popw[tid] = 0;
        const bool have = ep.a && tid < n_this;
        chan_a[tid] = have ? __ldg(ep.a + n0 + tid) : 1.f;
        chan_b[tid] = have ? __ldg(ep.b + n0 + tid) : 0.f;
    }
    __syncthreads();
    if (tid < TM_WARPS * 32 && (tid & (TS_NBC - 1)) < n_this) {   // popcounts of the filter rows
        const RowCtx row = wop.make_row(n0 + (tid & (TS_NBC - 1)));
        int pc = 0;
#pragma unroll 8
        for (int q = tid / TS_NBC; q < kwords; q += TM_WARPS * 32 / TS_NBC) pc += __popcll(__ldg(wop.addr(row, wop.decode(q))));
        atomicAdd(&popw[tid & (TS_NBC - 1)], pc);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    auto tiles_of = [&](int g) { return min(TS_TILES, my_tiles - g * TS_TILES); };   // of the CTA's g-th group of tiles
    const int ngroups = (my_tiles + TS_TILES - 1) / TS_TILES;

    if (warp < TS_PW) {
        // =========================== producers: thread = operand row of tiles p and p + 2 of a group ===========================
        const int p = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t a_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + TM_A_COL;
        const bool pair = xop.pairable();
        RowCtx xr[2];
        int lg = 0, lc = 0, lt = 0;   // load cursor: group, K stage, which of the two tiles
        auto rows_of = [&](int g) {
#pragma unroll
            for (int t = 0; t < 2; t++) xr[t] = xop.make_row(((int)blockIdx.x + (g * TS_TILES + p + 2 * t) * (int)gridDim.x) * 128 + r);   // (beyond M: not valid)
        };
        rows_of(0);
        typename XOp::Dec xd = xop.decode(0);
        struct Words { uint64_t w[TM_WORDS]; };
        auto load_next = [&](Words& v) {
            if (lg >= ngroups) return;
            typename XOp::Dec d = xd;
            const RowCtx row = lt ? xr[1] : xr[0];
            load_words(v.w, xop, row, d, lc * TM_WORDS, kwords, pair);
            if (lt == 0 && p + 2 < tiles_of(lg)) { lt = 1; return; }
            lt = 0;
            if (++lc < nchunks) { xop.advance(xd, TM_WORDS); return; }
            lc = 0;
            lg++;
            while (lg < ngroups && p >= tiles_of(lg)) lg++;   // a last group of one tile has nothing for the second group of warps
            rows_of(lg);
            xd = xop.decode(0);
        };
        while (lg < ngroups && p >= tiles_of(lg)) lg++;
        Words v[TM_AHEAD];
#pragma unroll
        for (int j = 0; j < TM_AHEAD; j++) load_next(v[j]);
        int g = 0, c = 0, t = p, base = 0;   // this step; base: steps of the groups before
        while (g < ngroups && p >= tiles_of(g)) { base += tiles_of(g) * nchunks; g++; }
        bool ok = true;
        while (g < ngroups && ok) {
#pragma unroll
            for (int j = 0; j < TM_AHEAD; j++) {
                if (g >= ngroups || !ok) break;
                const int gt = tiles_of(g), i = base + c * gt + t;
                const uint32_t s = i % TM_STAGES, use = i / TM_STAGES;
                if (use >= 1) ok = mbar_wait_warp(&bar_empty[s], (use - 1) & 1, abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int w = 0; w < TM_WORDS; w++) tmem_st_word(a_addr + s * TM_STAGE_COLS + w * 16, v[j].w[w]);
                load_next(v[j]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_full[s]);
                t += 2;
                if (t >= gt) {
                    t = p;
                    if (++c == nchunks) {
                        c = 0;
                        base += gt * nchunks;
                        g++;
                        while (g < ngroups && p >= tiles_of(g)) { base += tiles_of(g) * nchunks; g++; }
                    }
                }
            }
        }
        if (!ok) {
            atomicCAS(&g_tc5_status, 0, 1);
            s_abort = 1;
        }
    } else if (warp < TS_PW + TS_FW) {
        // =========================== filters: thread = channel x half a stage's words ===========================
        const int x = tid - TS_PW * 32, r = x & (TS_NBC - 1), w0 = (x / TS_NBC) * 2;
        const RowCtx row = wop.make_row(n0 + (r < n_this ? r : 0));
        const uint32_t dst = bring + (r >> 3) * 512 + (r & 7) * 16;
        auto load = [&](int c, uint64_t& a, uint64_t& b) {
            const int q = c * TM_WORDS + w0;
            a = 0; b = 0;
            if (r < n_this && q < kwords) a = __ldg(wop.addr(row, wop.decode(q)));
            if (r < n_this && q + 1 < kwords) b = __ldg(wop.addr(row, wop.decode(q + 1)));
        };
        uint64_t a0, b0, a1, b1;   // this stage's words and the next one's
        load(0, a0, b0);
        load(nchunks > 1 ? 1 : 0, a1, b1);
        uint32_t s = 0, use = 0;
        bool ok = true;
        for (int g = 0; g < ngroups && ok; g++) {
            for (int c = 0; c < nchunks; c++) {
                uint64_t a2, b2;
                load((c + 2) % nchunks, a2, b2);   // (nchunks is at least two)
                if (use >= 1 && !mbar_wait_warp<32>(&bar_bempty[s], (use - 1) & 1, abort_flag)) {
                    atomicCAS(&g_tc5_status, 0, 1);
                    s_abort = 1;
                    ok = false;
                    break;
                }
                const uint32_t at = dst + s * TS_BSTAGE_BYTES + w0 * TS_NBC * 64;
                expand_filter_word(at, a0);
                expand_filter_word(at + TS_NBC * 64, b0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_bfull[s]);
                if (++s == TS_BSTAGES) { s = 0; use++; }
                a0 = a1; b0 = b1; a1 = a2; b1 = b2;
            }
        }
    } else if (warp == TM_WARPS) {
        // =========================== MMA issue: the whole warp walks, one lane issues ===========================
        const uint32_t idesc = (2u << 4) | (1u << 10) | ((uint32_t)(n_this >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // as above
        const uint64_t d_b = umma_desc(bring, 512);
        const bool leader = elect_lane();
        uint32_t s = 0, par = 0, bs = 0, bpar = 0;
        bool ok = true;
        for (int g = 0; g < ngroups && ok; g++) {
            const int gt = tiles_of(g);
            for (int c = 0; c < nchunks && ok; c++) {
                if (!mbar_wait_warp(&bar_bfull[bs], bpar, abort_flag)) ok = false;
                const int words = min(TM_WORDS, kwords - c * TM_WORDS);
                const uint64_t bd = d_b + (uint64_t)(bs * (TS_BSTAGE_BYTES >> 4));
                for (int t = 0; t < gt && ok; t++) {
                    if (c == 0 && g > 0 && !mbar_wait_warp(&bar_acc_empty[t], (g - 1) & 1, abort_flag)) ok = false;
                    if (ok && !mbar_wait_warp(&bar_full[s], par, abort_flag)) ok = false;
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t at = tmem_base + TM_A_COL + s * TM_STAGE_COLS, d_tmem = tmem_base + t * TS_NBC;
                    if (leader) {
#pragma unroll
                        for (int j = 0; j < TM_WORDS; j++)
                            if (j < words) {
                                mma_i8_ts(d_tmem, at + j * 16, bd + j * (TS_NBC * 4), idesc, c + j ? 1u : 0u);
                                mma_i8_ts(d_tmem, at + j * 16 + 8, bd + j * (TS_NBC * 4) + 16, idesc, 1u);
                            }
                        umma_commit(&bar_empty[s]);
                        if (c == nchunks - 1) umma_commit(&bar_acc_full[t]);
                        if (t == gt - 1) umma_commit(&bar_bempty[bs]);
                    }
                    __syncwarp();
                    if (++s == TM_STAGES) { s = 0; par ^= 1u; }
                }
                if (++bs == TS_BSTAGES) { bs = 0; bpar ^= 1u; }
            }
        }
        if (!ok) {
            atomicCAS(&g_tc5_status, 0, 4);
            s_abort = 1;
        }
    } else {
        // =========================== epilogue ===========================
        const int x = tid - (TS_PW + TS_FW) * 32;
        if (x < TS_NBC) pop[x] = epi_pop_scaled(popw[x]);
        asm volatile("bar.sync 1, %0;" ::"n"(TS_EW * 32) : "memory");
        tmem_epilogue<TS_EW>(ep, EpiChannels{pop, chan_a, chan_b}, warp - TS_PW - TS_FW, epi_smem, tmem_base, n0, n_this, M, ntiles_m, TS_NBC, TS_TILES,
                             narrow, bar_acc_full, bar_acc_empty, &s_abort);
    }

    // ---- everybody is past its last use of the tensor memory ----
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == TM_WARPS) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base));
    }
}

}  // namespace dabnn
