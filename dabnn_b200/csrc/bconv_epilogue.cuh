// Epilogue of the byte-activation convolutions: accumulators in tensor memory -> counts -> affine -> + shortcut -> fp32,
// {0,1} bytes, packed sign bits.
//
// A work item is 32 accumulator rows x 32 channels and belongs to one warp from the first load to the last store: no
// barrier between warps, no staging tile that a copy engine still reads.  The warp takes its rows with tcgen05.ld (lane =
// row), turns the block over in 4 KB of shared memory of its own (lane = eight channels of a row; both sides conflict-free
// through an XOR of the 16-byte column), and then works on coalesced rows: four lanes cover the 128 bytes of a row's 32
// channels with 32-byte accesses, eight rows per step.  The shortcut arrives in the same arrangement straight from global
// memory, fetched a whole item ahead into the registers that the current item has just used up.
//
// What bounds it: instruction issue (and HBM at large batches).  The form before let 16 warps meet at a barrier for every
// 128 x 64 block and wait for the tensor store of an earlier block to have read its staging tile: 3300 cycles per block,
// whether the data came from HBM or from L2.
#pragma once
#include "bcontract_tc5.cuh"

namespace dabnn {

constexpr int EPI_WARPS = 12;                    // (16 would leave 96 registers a thread, and the loop invariants would be spilled)
constexpr int EPI_THREADS = EPI_WARPS * 32;
constexpr int EPI_GROUPS = EPI_WARPS / 4;        // a group of four warps covers the 128 accumulator rows of one 32-channel item
constexpr int EPI_WARP_BYTES = 32 * 128;         // 32 rows x 32 channels of 32 bits
constexpr int EPI_SMEM_BYTES = EPI_WARPS * EPI_WARP_BYTES;

__device__ __forceinline__ uint4 lds128u(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
// 32-byte accesses of the lanes whose element offset lies below a limit.  Read-once data: no line of L1 is spent on it (and
// not .nc: the output may be the shortcut's own memory).
__device__ __forceinline__ void ldg256_below(float (&v)[8], const float* base, uint32_t off, uint32_t limit) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a;\n\tsetp.lt.u32 p, %9, %10;\n\tmad.wide.u32 a, %9, 4, %8;\n\t"
                 "@p ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [a];\n\t}"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]) : "l"(base), "r"(off), "r"(limit) : "memory");
}
__device__ __forceinline__ void stg256_below(float* base, uint32_t off, uint32_t limit, const float (&v)[8]) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a;\n\tsetp.lt.u32 p, %1, %2;\n\tmad.wide.u32 a, %1, 4, %0;\n\t"
                 "@p st.global.v8.f32 [a], {%3, %4, %5, %6, %7, %8, %9, %10};\n\t}"
                 ::"l"(base), "r"(off), "r"(limit), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// the same as two 16-byte accesses, for tensors that start on a 16-byte boundary only
__device__ __forceinline__ void ldg128x2_below(float (&v)[8], const float* base, uint32_t off, uint32_t limit) {
    if (off < limit) {
        const float4* p = reinterpret_cast<const float4*>(base + off);
        const float4 x = p[0], y = p[1];
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    }
}
__device__ __forceinline__ void stg128x2_below(float* base, uint32_t off, uint32_t limit, const float (&v)[8]) {
    if (off < limit) {
        float4* p = reinterpret_cast<float4*>(base + off);
        p[0] = make_float4(v[0], v[1], v[2], v[3]);
        p[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}
__device__ __forceinline__ void stg64_below(unsigned char* base, uint32_t off, uint32_t limit, uint32_t x, uint32_t y) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a;\n\tsetp.lt.u32 p, %1, %2;\n\tmad.wide.u32 a, %1, 1, %0;\n\t@p st.global.v2.b32 [a], {%3, %4};\n\t}"
                 ::"l"(base), "r"(off), "r"(limit), "r"(x), "r"(y) : "memory");
}
// four {0,1} bytes, byte i = v[i] > 0: the sign bit of 0 - v is set exactly then (0, -0 and NaN give 0); a byte permute in
// its sign-replicating mode turns two sign bits into two bytes
__device__ __forceinline__ uint32_t sign_pair(float a, float b) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, 0x00fb;" : "=r"(r) : "r"(__float_as_uint(__fsub_rn(0.f, a))), "r"(__float_as_uint(__fsub_rn(0.f, b))));
    return r;
}
__device__ __forceinline__ uint32_t sign_bytes(float a, float b, float c, float d) {
    return __byte_perm(sign_pair(a, b), sign_pair(c, d), 0x5410) & 0x01010101u;
}
// 16 accumulator columns of the warp's 32 rows: lane = row
__device__ __forceinline__ void tmem_ld16(uint32_t (&v)[16], uint32_t t_addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                   "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(t_addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// n / d for tile numbers: one multiplication where it is exact (n * d below 2^32 for every n in question)
struct EpiDiv {
    uint32_t d, inv;              // inv = 0: divide
    __device__ __forceinline__ EpiDiv(int d_, int n_max) : d((uint32_t)d_), inv(d_ > 1 && (unsigned long long)n_max * d_ < (1ull << 32) ? 0xffffffffu / (uint32_t)d_ + 1u : 0u) {}
    __device__ __forceinline__ int operator()(int n) const { return d == 1 ? n : inv ? (int)__umulhi((uint32_t)n, inv) : n / (int)d; }
};

struct EpiOut {
    float* out;                   // fp32 [pixels][N] or null
    unsigned char* out_u8;        // {0,1} bytes [pixels][N] or null
    uint64_t* out_bits;           // packed sign bits [pixels][N / 64] or null
    int narrow;                   // the shortcut or `out` starts on a 16-byte boundary only
};

// Per-channel constants as the epilogue reads them: popcount of the weight row as epi_pop or epi_pop_scaled gives it, affine.
struct EpiChannels {
    const float *pop, *a, *b;     // shared memory
};
constexpr float EPI_POP_BIAS = 12582912.f;   // 1.5 * 2^23
// An integer of less than 23 bits (a count is one) added to the bits of 2^23 is 2^23 + that integer as a float: the popcount
// is kept with those bits added, as an integer.  Accumulators of 128 a bit: an integer of less than 22 bits and a sign added to
// the bits of 1.5 * 2^23 is 1.5 * 2^23 + that integer; the popcount is kept less the bias, scaled alike.
__device__ __forceinline__ float epi_pop(int pop) { return __uint_as_float((uint32_t)pop + 0x4B000000u); }
__device__ __forceinline__ float epi_pop_scaled(int pop) { return (float)pop - EPI_POP_BIAS / 128.f; }

// One warp's side of the epilogue.
struct EpiWarp {
    uint32_t buf;                 // this warp's 4 KB
    int lane, q;                  // q: the lane's eight channels of the item
    // Element offsets (pixel within the tile * N) of the rows this lane meets after the turn-over (row step * 8 + lane / 4 of
    // the warp's 32), all ones where a row carries no pixel; the same for every tile.
    uint32_t off[4];
    float sc[4][8];               // shortcut of the item to come

    __device__ __forceinline__ void init(uint32_t epi_smem, int epi_warp) {
        lane = threadIdx.x & 31;
        q = lane & 3;
        buf = epi_smem + epi_warp * EPI_WARP_BYTES;
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int i = 0; i < 8; i++) sc[s][i] = 0.f;
    }
    __device__ __forceinline__ int row_of(int s) const { return s * 8 + (lane >> 2); }
    __device__ __forceinline__ void set_row(int s, int pixel, int N) { off[s] = pixel < 0 ? 0xffffffffu : (uint32_t)(pixel * N); }
    // fetches step s of an item's shortcut; at: the tile's first pixel at the lane's channels, limit: elements that exist
    __device__ __forceinline__ void fetch(int s, const float* at, uint32_t limit, int narrow) {
        if (narrow) ldg128x2_below(sc[s], at, off[s], limit);
        else ldg256_below(sc[s], at, off[s], limit);
    }
    // takes the item's 32 accumulator columns into the buffer (16 at a time: the registers also hold the shortcut to come)
    __device__ __forceinline__ void take(uint32_t t_addr) {
        __syncwarp();   // the item before has been read out of the buffer
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t v[16];
            tmem_ld16(v, t_addr + h * 16);
#pragma unroll
            for (int k = 0; k < 4; k++) sts128(buf + lane * 128 + (((h * 4 + k) ^ (lane & 7)) << 4), v[k * 4], v[k * 4 + 1], v[k * 4 + 2], v[k * 4 + 3]);
        }
    }
    // cl: the lane's first channel within the CTA's block (readable, whether or not the channels exist).  e0: the tile's first
    // pixel at the lane's first channel, limit: elements from there on that exist (0 where the channels do not).  next /
    // next_limit: what `fetch` needs for the item to come.  KEEP: the results also stay in the buffer, at the places the
    // accumulators had.
    template <bool SC, bool KEEP, bool SCALED = false>
    __device__ __forceinline__ void finish(const EpiOut& o, const EpiChannels& ch, int cl, size_t e0, uint32_t limit, const float* next, uint32_t next_limit) {
        __syncwarp();
        float pop[8], a[8], b[8];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float4 x = *reinterpret_cast<const float4*>(ch.pop + cl + h * 4), y = *reinterpret_cast<const float4*>(ch.a + cl + h * 4),
                         z = *reinterpret_cast<const float4*>(ch.b + cl + h * 4);
            pop[h * 4] = x.x; pop[h * 4 + 1] = x.y; pop[h * 4 + 2] = x.z; pop[h * 4 + 3] = x.w;
            a[h * 4] = y.x; a[h * 4 + 1] = y.y; a[h * 4 + 2] = y.z; a[h * 4 + 3] = y.w;
            b[h * 4] = z.x; b[h * 4 + 1] = z.y; b[h * 4 + 2] = z.z; b[h * 4 + 3] = z.w;
        }
        float* const po = o.out + e0;
        unsigned char* const p8 = o.out_u8 + e0;
        const uint32_t lim_out = o.out ? limit : 0u, lim_u8 = o.out_u8 ? limit : 0u;
        const uint32_t src = buf + (lane >> 2) * 128, c0 = ((2 * q) ^ (lane >> 2)) << 4, c1 = ((2 * q + 1) ^ (lane >> 2)) << 4;
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const uint4 t0 = lds128u(src + s * 1024 + c0), t1 = lds128u(src + s * 1024 + c1);
            const uint32_t t[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
            float y[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                // the count, exactly (see epi_pop)
                y[i] = SCALED ? __fmaf_rn(__uint_as_float(t[i] + 0x4B400000u), 1.f / 128.f, pop[i])
                              : __fsub_rn(__uint_as_float(t[i] + __float_as_uint(pop[i])), 8388608.f);
                y[i] = __fadd_rn(__fmul_rn(a[i], y[i]), b[i]);
                if (SC) y[i] = __fadd_rn(sc[s][i], y[i]);
            }
            if (SC) fetch(s, next, next_limit, o.narrow);
            if (KEEP) {
                sts128f(src + s * 1024 + c0, y[0], y[1], y[2], y[3]);
                sts128f(src + s * 1024 + c1, y[4], y[5], y[6], y[7]);
            }
            if (o.narrow) stg128x2_below(po, off[s], lim_out, y);
            else stg256_below(po, off[s], lim_out, y);
            const uint32_t w0 = sign_bytes(y[0], y[1], y[2], y[3]), w1 = sign_bytes(y[4], y[5], y[6], y[7]);
            stg64_below(p8, off[s], lim_u8, w0, w1);
            if (o.out_bits) {   // four flags -> a nibble, four lanes -> the 32 bits of the row's channels
                uint32_t bits = (((w0 * 0x01020408u) >> 24 & 0xfu) | ((w1 * 0x01020408u) >> 20 & 0xf0u)) << (8 * q);
                bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
                bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
                if (q == 0 && off[s] < limit) reinterpret_cast<uint32_t*>(o.out_bits)[(e0 + off[s]) >> 5] = bits;
            }
        }
    }
};

}  // namespace dabnn
