// Q4_K / Q5_K matmul of several activation rows on the 5th-generation tensor cores, at float accuracy in two half passes.
//
// The reference re-reads the weights for every 8 activation rows (q4k_matmul_batched8,
// runtime/kernels/quant_kq/q4k_matmul_batched8.wgsl:9-23).  Here one pass over the weights serves up to 128 rows, and the
// contraction is exact in the weights:
//
//   w = d*sc*q - dmin*mn = d * [ sc*(q - z) + (z*sc - (dmin/d)*mn) ]        (z = 8 for 4-bit codes, 16 for 5-bit codes)
//
// sc*(q - z) is an integer below 1024, exact in half precision, so ONE 16-bit weight operand serves an activation that
// is split into two halves (x*2^e = Xh + Xl, 22 bits; e per activation row).  The bracket's second term is constant
// over a sub-block of 32 weights: it multiplies the sub-block's mean activation, one more k-step of 16 per super-block
// (high and low half of the eight constants).  The accumulator of a super-block (256 weights) is drained to registers,
// where d is applied in float: the tensor core, whose additions truncate, never accumulates over more than a super-block.
// Error against 64 bits 2.9e-7..3.7e-7 to 32 rows (streaming kernel 3.3e-7..4.5e-7), 5.7e-7..6.3e-7 above (prefill kernel
// 1.2e-6..2.2e-6 from K = 1024 on).
//
// What bounds it.  To 48 rows the instructions of the dequantising warps (16 rows: 3,500 cycles a unit of 256 rows x 256
// weights, 1,470 at the DRAM rate; ncu: issue slots 55 % busy, ALU 41 %, DRAM 32 %); above, the hand-overs between
// dequantising, mma and drain (T = 128: 8,000 cycles a unit, the tensor pipe busy in 4,300 of them).  Whole call on B200, us, before | now (before: streaming kernel in
// slabs, prefill kernel with three passes), 128256 x 4096: 16 rows 201 | 105, 24 rows 302 | 115, 37 rows 348 | 147, 64 rows
// 348 | 159, 80 rows 350 | 195, 128 rows 387 | 267, 512 rows 1252 | 1166; 57344 x 8192, 512 rows: 1183 | 951.  The 48- and
// 128-row variants spill 52 and 112 bytes (128 rows: 2 % of its instructions).
//   * the dequantised operand lives in TENSOR MEMORY (tcgen05.st, A operand of tcgen05.mma); through shared memory its
//     write and re-read alone would cost 1.7 times the shared-memory bandwidth that streaming at the DRAM rate leaves;
//   * a CTA takes 256 weight rows at a time (two 128-lane row tiles share every activation tile);
//   * the work is one list of (row tile, activation tile, super-block) units over at most one CTA per SM, cut into equal
//     contiguous shares: every SM is busy whatever the shape.  A tile that is cut leaves partial sums in a workspace, which
//     are added in ascending order of k (deterministic): by the CTA that finishes last, or by rows_reduce_kernel.
//
// Roles (20 warps): warp 0 TMA loads of raw super-blocks (box 128 rows x 1 block), warp 1 (and 3) mma issue, warp 2 bulk
// copies of the activation tiles (laid out by rows_pack_kernel exactly as the mma reads them), warps 4-19 dequantise and
// drain (RowsPlan says which does what).
//
// Every wait is bounded: on a time-out the role raises the CTA's abort flag and the device status word, waits return
// at once from then on, the loops run out (so that all barriers stay matched), copies and mmas in flight are waited
// for, tensor memory is freed and the kernel returns.
#include <cuda.h>
#include <cuda_fp16.h>

#include <cstring>
#include <type_traits>

#include "kernels.h"
#include "q4k_common.cuh"

namespace bpq4k {

namespace {

constexpr uint32_t kWaitLimit = 1u << 21;
constexpr uint32_t kSuspendNs = 1000;                 // a waiting warp sleeps this long at most: polls take issue slots from the dequantising warps
constexpr uint32_t kMaxCtas = 160;                    // counters (one per CTA)
constexpr uint32_t kWorkers = 16;                     // warps that dequantise and drain
constexpr uint32_t kThreads = (4 + kWorkers) * 32;
constexpr uint32_t kTileRows = 256;                   // weight rows of a unit: two row tiles of 128 lanes
constexpr float kLowScale = 2048.f, kLowScaleInv = 1.f / 2048.f;  // of stacked low halves
constexpr uint32_t kASlotCols = 40;                   // tensor-memory columns of one dequantised group: 32 codes + 8 (constant term)

// T: activation rows of the tile.
//   up to 32   the high and the low halves of the activations are stacked into one mma of 2T columns, each half with its
//              own accumulator; above that they accumulate into the same T columns.  Stacked low halves carry a factor 2^11 of
//              their own (rows_pack_kernel)
//   up to 48   two accumulators per row tile: the next super-block accumulates while the last is drained
//   above      (WIDE) one accumulator per row tile (tensor memory holds two tiles' accumulators and the operand ring) and an issuing warp for each, the second two groups behind the
//              first, so that one accumulates while the other is drained.  The T partial sums of a weight row fill a
//              thread's registers, so eight warps dequantise and eight others drain: setmaxnreg 64 and 160.
template <int T, int QT>
struct RowsPlan {
    static constexpr bool STACK = T <= 32;
    static constexpr bool WIDE = T > 48;
    static constexpr uint32_t NBUF = WIDE ? 1u : 2u;
    static constexpr uint32_t N = STACK ? 2u * T : (uint32_t)T;   // columns of one accumulator
    static constexpr uint32_t ACC_COLS = 2u * NBUF * N;
    static constexpr uint32_t NA = (512u - ACC_COLS) / (2u * kASlotCols) > 5u ? 5u : (512u - ACC_COLS) / (2u * kASlotCols);
    static constexpr uint32_t BLOCK = QT == 1 ? 176u : 144u;
    static constexpr uint32_t RAW_BYTES = 128u * BLOCK;
    static constexpr uint32_t G_BYTES = T * 256u;                 // activations of a 64-weight group: 2T rows x 128 B
    static constexpr uint32_t S_BYTES = T * 64u;                  // sub-block sums of a super-block: 2T rows x 32 B, behind its last group
    static constexpr uint32_t SB_BYTES = 4u * G_BYTES + S_BYTES;
    // activation ring: a slot holds a super-block's four groups, or (one accumulator) one group
    static constexpr uint32_t BG = NBUF == 2u ? 4u : 1u;
    static constexpr uint32_t B_SLOT = (BG * G_BYTES + S_BYTES + 1023u) & ~1023u;
    static constexpr uint32_t NB = T <= 8 ? 4u : T <= 24 ? 3u : T <= 48 ? 2u : T <= 96 ? 5u : 4u;
    // barriers of the operand ring and of the accumulators: one set for both row tiles, or one each
    static constexpr uint32_t RB = NBUF == 2u ? 1u : 2u;
    static constexpr uint32_t BAR_BYTES = 1024u;
    static constexpr uint32_t S_RING = WIDE ? 4u * 256u * 4u : 0u;   // WIDE: the drain's scale of every weight row, four super-blocks deep
    static constexpr uint32_t NR = (226u * 1024u - 1024u - BAR_BYTES - S_RING - NB * B_SLOT) / RAW_BYTES > 10u
                                       ? 10u : (226u * 1024u - 1024u - BAR_BYTES - S_RING - NB * B_SLOT) / RAW_BYTES;
    static constexpr uint32_t SMEM_BYTES = 1024u + NB * B_SLOT + NR * RAW_BYTES + BAR_BYTES + S_RING;
    static_assert(NA >= 2 && NR >= 2 && NB >= 2, "rings too short");
};

struct RowsArgs {
    CUtensorMap tmap_w;       // [N rows][K/256 blocks] as 32-bit words, box 128 rows x 1 block
    const uint8_t* image;     // activation image (rows_pack_kernel)
    const float* inv;         // 2^-e per activation row
    const float* sb_scale;    // STACK: [super-block][T], read only if a word of `spread` is not zero
    const uint32_t* spread;
    uint32_t n_spread;
    const float* bias;
    float* Y;
    uint32_t M, N, nsb, u_base, u_extra;
    uint32_t tok_tiles, slot_rows;  // activation tiles; rows of a workspace slot (min(M, T))
    uint32_t defer;           // cut tiles are added up by rows_reduce_kernel
    float* part;              // [CTA][2][slot_rows][256]
    uint32_t* counters;       // one per CTA, cleared by rows_pack_kernel
    int* status;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return ok;
}
// Bounded wait; false once the CTA is aborting (then at once: the caller carries on so that barriers stay matched).
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status) {
    if (mbar_try_wait(bar, parity)) return true;
    for (uint32_t i = 0; i < kWaitLimit; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63u) == 0u && *abort_flag) return false;
    }
    *abort_flag = 1;
    if (status) atomicExch(status, kDeviceTimeout);
    return false;
}
// The same for what is still in flight at the end: also waits while the CTA aborts.
__device__ __forceinline__ void wait_in_flight(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kWaitLimit; i++)
        if (mbar_try_wait(bar, parity)) return;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tmap, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
// K-major shared-memory descriptors, version 1 (sm_100), LBO unused: rows of 128 B (128-byte swizzle, 8-row groups
// 1024 B apart) and rows of 32 B (32-byte swizzle, 8-row groups 256 B apart).
__device__ __forceinline__ uint64_t desc_128(uint32_t a) { return (uint64_t)((a >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61); }
__device__ __forceinline__ uint64_t desc_32(uint32_t a) { return (uint64_t)((a >> 4) & 0x3FFFu) | (1ull << 16) | (16ull << 32) | (1ull << 46) | (6ull << 61); }
// A from tensor memory, B from shared memory, half operands, float accumulator.  The whole warp comes here and one lane
// (`leader`) issues: the descriptors then stay in uniform registers (see the issuing warp).
__device__ __forceinline__ void umma_ts(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t leader, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(leader)
        : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
        "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void ldg128(const float* p, float* v) {
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p) : "memory");
}
template <int C>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t* v) {
    if constexpr (C == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                       "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(taddr));
    else if constexpr (C == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(taddr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                     : "r"(taddr));
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// (w & 0x00F000F0) | base in one instruction (the compiler makes two of the expression: 64 of 600 a warp and unit)
__device__ __forceinline__ uint32_t codes_of(uint32_t w, uint32_t base) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(0x00F000F0u), "r"(base));
    return r;
}
// (1024 + 16 q) * (sc/16) - (64 + z) * sc = sc * (q - z), exact: `biased` holds 0x6400 | 16 q in both halves
__device__ __forceinline__ uint32_t scale_codes(uint32_t biased, __half2 m, __half2 a) {
    const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&biased), m, a);
    return *reinterpret_cast<const uint32_t*>(&r);
}


// The scales of a row's super-block.  The drain applies s = d.  Where dmin is large beside d (blocks whose spread is small
// beside their offset) the constant term would not fit a half: s = d * 2^k and the codes carry f = 2^-k, which halves hold
// exactly up to k = 20.
struct BlockScales {
    uint32_t sc_lo, sc_hi, mn_lo, mn_hi;
    float s = 0.f, f, rho;
    bool any_wide;
    template <bool Q5>
    __device__ __forceinline__ void load(const uint4& w) {
        const BlockHeader h{w.x, w.y, w.z, w.w};
        const float d = half_bits_to_float(h.w0), dmin = half_bits_to_float(h.w0 >> 16);
        unpack_scales_packed(h, sc_lo, sc_hi, mn_lo, mn_hi);
        s = d, f = 1.f, rho = dmin / d;
        const bool wide = !(fabsf(dmin) < 16.f * fabsf(d));
        any_wide = __any_sync(0xFFFFFFFFu, wide);
        if (wide) {
            if (d == 0.f) {
                f = 0.f, s = dmin * 0.0625f, rho = 16.f;
            } else {
                const uint32_t e = (__float_as_uint(rho) >> 23) & 255u;  // at least 131
                f = __uint_as_float((257u - e) << 23);                   // rho * f in [8, 16)
                s = d * __uint_as_float((e - 3u) << 23);
                rho *= f;
            }
        }
    }
};
// A 64-weight group's two scales sc (even and odd sub-block) as the operands of scale_codes.
struct GroupScales {
    __half2 me, mo, ae, ao;
    __device__ __forceinline__ GroupScales(const BlockScales& h, uint32_t g, float z) {
        const uint32_t scw = (g >= 2u ? h.sc_hi : h.sc_lo) >> (16u * (g & 1u));
        // sc/16 in both halves of a register: 0x6400 | sc is 1024 + sc
        const uint32_t be = __byte_perm(scw, 0x64u, 0x4040), bo = __byte_perm(scw, 0x64u, 0x4141);
        const __half2 k16 = __float2half2_rn(0.0625f), k64 = __float2half2_rn(-64.f);
        me = __hfma2(*reinterpret_cast<const __half2*>(&be), k16, k64), mo = __hfma2(*reinterpret_cast<const __half2*>(&bo), k16, k64);
        if (h.any_wide) me = __float2half2_rn(__low2float(me) * h.f), mo = __float2half2_rn(__low2float(mo) * h.f);
        const __half2 kz = __float2half2_rn(-(64.f + z) * 16.f);
        ae = __hmul2(me, kz), ao = __hmul2(mo, kz);
    }
};
// Four code words (16 code bytes: 16 weights of the even and 16 of the odd sub-block of group g) -> 16 columns of the
// operand: per word the even sub-block's weights 4i, 4i+2 | 4i+1, 4i+3, then the odd one's.
template <bool Q5>
__device__ __forceinline__ void dequant_words(const uint4& code, const uint4& fifth, uint32_t g, const GroupScales& gs, uint32_t* v) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t w = i == 0 ? code.x : i == 1 ? code.y : i == 2 ? code.z : code.w;
        // codes 16 q under the half 1024; Q5_K: with the fifth bit above them
        uint32_t f0 = 0x64006400u, f1 = f0, f2 = f0, f3 = f0;
        if constexpr (Q5) {
            const uint32_t q = (i == 0 ? fifth.x : i == 1 ? fifth.y : i == 2 ? fifth.z : fifth.w) >> (2u * g);  // bits 0 and 1 of each byte
            auto fifth_of = [](uint32_t b) {
                uint32_t r;
                asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(b), "r"(0x01000100u), "r"(0x64006400u));
                return r;
            };
            f0 = fifth_of(q << 8), f1 = fifth_of(q), f2 = fifth_of(q << 7), f3 = fifth_of(q >> 1);
        }
        v[4 * i] = scale_codes(codes_of(w << 4, f0), gs.me, gs.ae);
        v[4 * i + 1] = scale_codes(codes_of(w >> 4, f1), gs.me, gs.ae);
        v[4 * i + 2] = scale_codes(codes_of(w, f2), gs.mo, gs.ao);
        v[4 * i + 3] = scale_codes(codes_of(w >> 8, f3), gs.mo, gs.ao);
    }
}
// The constant terms 32 * (z*sc*f - rho*mn) of the eight sub-blocks: four words of high halves, four of low ones.
template <bool Q5>
__device__ __forceinline__ void constant_terms(const BlockScales& h, uint32_t (&cw)[8]) {
    const float zf = 32.f * (Q5 ? 16.f : 8.f) * h.f, rf = -32.f * h.rho;
    // byte b of w as a float: 2^23 + byte is one permute away
    auto byte_f = [](uint32_t w, uint32_t b) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | b)) - 8388608.f; };
#pragma unroll
    for (uint32_t p = 0; p < 4; p++) {
        const uint32_t sw = p < 2 ? h.sc_lo : h.sc_hi, mw = p < 2 ? h.mn_lo : h.mn_hi, b = 2u * (p & 1u);
        const float ce = fmaf(rf, byte_f(mw, b), zf * byte_f(sw, b));
        const float co = fmaf(rf, byte_f(mw, b + 1u), zf * byte_f(sw, b + 1u));
        cw[p] = half2_bits(ce, co);
        const float2 cf = __half22float2(*reinterpret_cast<const __half2*>(&cw[p]));
        cw[4 + p] = half2_bits(ce - cf.x, co - cf.y);
    }
}

__device__ __forceinline__ uint32_t unit_begin(uint32_t cta, uint32_t base, uint32_t extra) { return cta * base + min(cta, extra); }
__device__ __forceinline__ uint32_t unit_owner(uint32_t u, uint32_t base, uint32_t extra) {
    const uint32_t cut = extra * (base + 1u);
    return u < cut ? u / (base + 1u) : extra + (u - cut) / base;
}

template <int T, int QT>
__global__ void __launch_bounds__(kThreads, 1) rows_tc_kernel(const __grid_constant__ RowsArgs a) {
    using P = RowsPlan<T, QT>;
    constexpr bool Q5 = QT == 1;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    auto b_slot = [&](uint32_t s) { return base + s * P::B_SLOT; };
    auto raw_slot = [&](uint32_t s) { return base + P::NB * P::B_SLOT + s * P::RAW_BYTES; };
    constexpr uint32_t OFF_BAR = P::NB * P::B_SLOT + P::NR * P::RAW_BYTES;
    const uint32_t bar0 = base + OFF_BAR;
    auto raw_full = [&](uint32_t s) { return bar0 + s * 8u; };
    auto raw_empty = [&](uint32_t s) { return bar0 + (P::NR + s) * 8u; };
    auto b_full = [&](uint32_t s) { return bar0 + (2u * P::NR + s) * 8u; };
    auto b_empty = [&](uint32_t s) { return bar0 + (2u * P::NR + P::NB + s) * 8u; };
    constexpr uint32_t A0 = 2u * P::NR + 2u * P::NB;
    auto a_full = [&](uint32_t rt, uint32_t s) { return bar0 + (A0 + (P::RB == 2u ? rt : 0u) * P::NA + s) * 8u; };
    auto a_empty = [&](uint32_t rt, uint32_t s) { return bar0 + (A0 + (2u + (P::RB == 2u ? rt : 0u)) * P::NA + s) * 8u; };
    constexpr uint32_t C0 = A0 + 4u * P::NA;
    auto acc_full = [&](uint32_t rt, uint32_t b) { return bar0 + (C0 + (P::RB == 2u ? rt * 2u : 0u) + b) * 8u; };
    auto acc_empty = [&](uint32_t rt, uint32_t b) { return bar0 + (C0 + 4u + (P::RB == 2u ? rt * 2u : 0u) + b) * 8u; };
    const uint32_t done_bar = bar0 + (C0 + 8u) * 8u;
    auto s_full = [&](uint32_t rt, uint32_t s) { return bar0 + (C0 + 11u + rt * 4u + s) * 8u; };  // (after done_bar and 16 bytes of flags)
    const uint32_t skew_bar = bar0 + (C0 + 19u) * 8u;
    static_assert((C0 + 20u) * 8u <= P::BAR_BYTES, "barrier area");
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + OFF_BAR + (C0 + 9u) * 8u);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + OFF_BAR + (C0 + 9u) * 8u + 4u);
    volatile uint32_t* last_flag = reinterpret_cast<volatile uint32_t*>(base_ptr + OFF_BAR + (C0 + 9u) * 8u + 8u);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t u0 = unit_begin(blockIdx.x, a.u_base, a.u_extra), u1 = unit_begin(blockIdx.x + 1u, a.u_base, a.u_extra);
    const uint32_t nu = u1 - u0;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < P::NR; s++) mbar_init(raw_full(s), 1), mbar_init(raw_empty(s), P::WIDE ? 4u : 8u);
        for (uint32_t s = 0; s < P::NB; s++) mbar_init(b_full(s), 1), mbar_init(b_empty(s), P::WIDE ? 2u : 1u);
        for (uint32_t rt = 0; rt < P::RB; rt++) {  // a group is dequantised by one of two sets of four warps per row tile
            for (uint32_t s = 0; s < P::NA; s++) mbar_init(a_full(rt, s), P::WIDE ? 4u : 8u), mbar_init(a_empty(rt, s), 1);
            for (uint32_t b = 0; b < P::NBUF; b++) mbar_init(acc_full(rt, b), 1), mbar_init(acc_empty(rt, b), P::WIDE ? 4u : 16u);
        }
        mbar_init(done_bar, P::WIDE ? 2u : 1u);
        if constexpr (P::WIDE) {
            for (uint32_t i = 0; i < 8; i++) mbar_init(s_full(i >> 2, i & 3u), 4);
            mbar_init(skew_bar, 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
    auto acc_col = [&](uint32_t rt, uint32_t b) { return (rt * P::NBUF + b) * P::N; };
    auto a_col = [&](uint32_t rt, uint32_t s) { return P::ACC_COLS + (rt * P::NA + s) * kASlotCols; };
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // WIDE: 20 warps are launched with 96 registers a thread, 61,440 in all; 8 x 32 x (64 + 160) + 4 x 32 x 32 is the same sum
    if (warp < 4) {
    if constexpr (P::WIDE) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp == 0) {
        // ---------------- raw super-blocks ----------------
        if (lane == 0) {
            uint32_t tile = u0 / a.nsb, b = u0 - tile * a.nsb, s = 0, it = 0, issued = 0, rtile = tile / a.tok_tiles;
            bool ok = true;
            for (uint32_t k = 0; k < nu && ok; k++) {
                for (uint32_t rt = 0; rt < 2 && ok; rt++) {
                    ok = it == 0 || wait_bar(raw_empty(s), (it - 1u) & 1u, abort_flag, a.status);
                    if (!ok) break;
                    if (!BPQ4K_CHECK(b < a.nsb && rtile * kTileRows < a.N && s < P::NR, a.status)) {
                        *abort_flag = 1, ok = false;
                        break;
                    }
                    mbar_expect_tx(raw_full(s), P::RAW_BYTES);
                    tma_load_2d(raw_slot(s), &a.tmap_w, b * (P::BLOCK / 4u), rtile * kTileRows + rt * 128u, raw_full(s));
                    issued++;
                    if (++s == P::NR) s = 0, it++;
                }
                if (++b == a.nsb) b = 0, tile++, rtile = tile / a.tok_tiles;
            }
            if (!ok)  // aborting: nothing may still be written to shared memory after the exit
                for (uint32_t i = issued > P::NR ? issued - P::NR : 0u; i < issued; i++) wait_in_flight(raw_full(i % P::NR), (i / P::NR) & 1u);
        }
    } else if (warp == 2) {
        // ---------------- activation tiles ----------------
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // the image is written by the kernel ahead of this one
            uint32_t tt = u0 / a.nsb, b = u0 - tt * a.nsb, s = 0, it = 0, issued = 0;
            tt %= a.tok_tiles;
            bool ok = true;
            for (uint32_t k = 0; k < nu && ok; k++) {
                const uint8_t* src = a.image + ((uint64_t)tt * a.nsb + b) * P::SB_BYTES;
                for (uint32_t g = 0; g < 4 && ok; g += P::BG) {
                    ok = it == 0 || wait_bar(b_empty(s), (it - 1u) & 1u, abort_flag, a.status);
                    if (!ok) break;
                    if (!BPQ4K_CHECK(tt < a.tok_tiles && b < a.nsb && s < P::NB, a.status)) {
                        *abort_flag = 1, ok = false;
                        break;
                    }
                    const uint32_t bytes = P::BG * P::G_BYTES + (g + P::BG == 4u ? P::S_BYTES : 0u);
                    mbar_expect_tx(b_full(s), bytes);
                    bulk_load(b_slot(s), src + g * P::G_BYTES, bytes, b_full(s));
                    issued++;
                    if (++s == P::NB) s = 0, it++;
                }
                if (++b == a.nsb) {
                    b = 0;
                    if (++tt == a.tok_tiles) tt = 0;
                }
            }
            if (!ok)
                for (uint32_t i = issued > P::NB ? issued - P::NB : 0u; i < issued; i++) wait_in_flight(b_full(i % P::NB), (i / P::NB) & 1u);
        }
    } else if (warp == 1 || P::WIDE) {
        // ---------------- mma issue ----------------
        // The whole warp walks the loop, one lane issues.  (With the loop under `lane == 0` every descriptor of every mma
        // was moved to uniform registers by itself: 110 cycles an mma, 5,100 cycles for the 34 small mmas of a unit.)
        {
            const uint32_t leader = elect_one();
            constexpr uint32_t idesc = (1u << 4) | ((P::N >> 3) << 17) | ((128u >> 4) << 24);  // f32 += f16 * f16, K-major, M = 128
            bool ok = true;
            // one group of one row tile: A slot at `ta`, activations at `bt`, the super-block's sums at `st` behind its last group
            auto group = [&](uint32_t d, uint32_t ta, uint32_t bt, uint32_t st, uint32_t g) {
                const uint64_t b_hi = desc_128(bt), b_lo = desc_128(bt + T * 128u);
                if constexpr (!P::STACK) {  // the small low halves first
#pragma unroll
                    for (uint32_t ks = 0; ks < 4; ks++) umma_ts(leader, d, ta + ks * 8u, b_lo + ks * 2u, idesc, (g | ks) ? 1u : 0u);
                }
#pragma unroll
                for (uint32_t ks = 0; ks < 4; ks++) umma_ts(leader, d, ta + ks * 8u, b_hi + ks * 2u, idesc, (!P::STACK || (g | ks)) ? 1u : 0u);
                if (g == 3) {
                    if constexpr (!P::STACK) umma_ts(leader, d, ta + 32u, desc_32(st + T * 32u), idesc, 1u);
                    umma_ts(leader, d, ta + 32u, desc_32(st), idesc, 1u);
                }
            };
            if constexpr (P::NBUF == 2u) {
                uint32_t sb = 0, itb = 0, sa = 0, ita = 0;
                for (uint32_t k = 0; k < nu && ok; k++) {
                    const uint32_t buf = k & 1u;
                    if (k >= 2u) ok = wait_bar(acc_empty(0, buf), ((k >> 1) - 1u) & 1u, abort_flag, a.status);
                    ok &= wait_bar(b_full(sb), itb & 1u, abort_flag, a.status);
                    const uint32_t bt = b_slot(sb);
#pragma unroll
                    for (uint32_t g = 0; g < 4; g++) {
                        ok &= wait_bar(a_full(0, sa), ita & 1u, abort_flag, a.status);
                        fence_after();
#pragma unroll
                        for (uint32_t rt = 0; rt < 2; rt++)
                            group(tmem + acc_col(rt, buf), tmem + a_col(rt, sa), bt + g * P::G_BYTES, bt + 4u * P::G_BYTES, g);
                        umma_commit(leader, a_empty(0, sa));
                        if (++sa == P::NA) sa = 0, ita++;
                    }
                    umma_commit(leader, acc_full(0, buf));
                    umma_commit(leader, b_empty(sb));
                    if (++sb == P::NB) sb = 0, itb++;
                }
            } else {
                // one issuing warp per row tile: while one waits for its accumulator to be drained the other keeps the tensor
                // core busy (one warp for both stood still in every drain: 11,300 cycles a unit at T = 128, 4,300 of them mmas)
                const uint32_t rt = warp >> 1;
                uint32_t sb = 0, itb = 0, sa = 0, ita = 0;
                if (rt == 1u) ok = wait_bar(skew_bar, 0, abort_flag, a.status);  // two groups behind: the drains alternate
                for (uint32_t k = 0; k < nu && ok; k++) {
                    if (k > 0) ok = wait_bar(acc_empty(rt, 0), (k - 1u) & 1u, abort_flag, a.status);
#pragma unroll
                    for (uint32_t g = 0; g < 4; g++) {
                        ok &= wait_bar(b_full(sb), itb & 1u, abort_flag, a.status);
                        ok &= wait_bar(a_full(rt, sa), ita & 1u, abort_flag, a.status);
                        fence_after();
                        const uint32_t bt = b_slot(sb);
                        group(tmem + acc_col(rt, 0), tmem + a_col(rt, sa), bt, bt + P::G_BYTES, g);
                        umma_commit(leader, a_empty(rt, sa));
                        umma_commit(leader, b_empty(sb));
                        if (g == 1 && k == 0 && rt == 0u) umma_commit(leader, skew_bar);
                        if (g == 3) umma_commit(leader, acc_full(rt, 0));
                        if (++sb == P::NB) sb = 0, itb++;
                        if (++sa == P::NA) sa = 0, ita++;
                    }
                }
            }
            umma_commit(leader, done_bar);  // every mma has read its operands before shared and tensor memory go away
            wait_in_flight(done_bar, 0);
        }
    }
    } else if constexpr (P::WIDE) {
        const uint32_t rt = ((warp - 4u) >> 2) & 1u, quad = warp & 3u;
        const uint32_t row = quad * 32u + lane;            // lane of the row tile
        const uint32_t tl = tmem + ((quad * 32u) << 16);   // this warp's lanes
        float* s_ring = reinterpret_cast<float*>(base_ptr + OFF_BAR + P::BAR_BYTES) + rt * 128u + row;  // [super-block & 3][256]
        if (warp < 12u) {
            // ---------------- dequantise: one weight row per thread ----------------
            asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
            uint32_t rs = rt, rit = 0, sa = 0, ita = 0;
            for (uint32_t k = 0; k < nu; k++) {
                wait_bar(raw_full(rs), rit & 1u, abort_flag, a.status);
                const uint32_t rp = raw_slot(rs) + row * P::BLOCK;
                BlockScales h;
                h.load<Q5>(lds128(rp));
                // (read four super-blocks from now at the earliest: the operand ring is shorter than one)
                s_ring[(k & 3u) * 256u] = h.s;
                __syncwarp();
                if (lane == 0) mbar_arrive(s_full(rt, k & 3u));
#pragma unroll
                for (uint32_t g = 0; g < 4; g++) {
                    const GroupScales gs(h, g, Q5 ? 16.f : 8.f);
                    const uint32_t ta = tl + a_col(rt, sa);
                    if (ita > 0) wait_bar(a_empty(rt, sa), (ita - 1u) & 1u, abort_flag, a.status);
                    __syncwarp();
                    fence_after();
#pragma unroll
                    for (uint32_t hf = 0; hf < 2; hf++) {
                        uint32_t v[16];
                        const uint4 code = lds128(rp + (Q5 ? 48u : 16u) + g * 32u + hf * 16u);
                        uint4 fifth = make_uint4(0, 0, 0, 0);
                        if constexpr (Q5) fifth = lds128(rp + 16u + hf * 16u);
                        dequant_words<Q5>(code, fifth, g, gs, v);
                        tmem_st16(ta + hf * 16u, v);
                    }
                    if (g == 3) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(raw_empty(rs));
                        rs += 2u;
                        if (rs >= P::NR) rs -= P::NR, rit++;
                        uint32_t cw[8];
                        constant_terms<Q5>(h, cw);
                        tmem_st8(ta + 32u, cw);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a_full(rt, sa));
                    if (++sa == P::NA) sa = 0, ita++;
                }
            }
        } else {
            // ---------------- drain: the T partial sums of one weight row per thread ----------------
            asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
            float y[T];
#pragma unroll
            for (int j = 0; j < T; j++) y[j] = 0.f;
            uint32_t tile = u0 / a.nsb, b = u0 - tile * a.nsb;
            bool seg_head = b == 0;
            for (uint32_t k = 0; k < nu; k++) {
                wait_bar(s_full(rt, k & 3u), (k >> 2) & 1u, abort_flag, a.status);
                const float sc = s_ring[(k & 3u) * 256u];
                wait_bar(acc_full(rt, 0), k & 1u, abort_flag, a.status);
                __syncwarp();
                fence_after();
                const uint32_t col = tl + acc_col(rt, 0);
#pragma unroll
                for (int c0 = 0; c0 < T; c0 += 16) {
                    uint32_t v[16];
                    tmem_ld<16>(col + c0, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c0 + 16 == T) {
                        fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(acc_empty(rt, 0));
                    }
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        y[c0 + j] = fmaf(sc, __uint_as_float(v[j]), y[c0 + j]);
                        asm volatile("" : "+f"(y[c0 + j]));  // (before the next load: else all T loaded values wait in registers)
                    }
                }
                const bool tile_end = b + 1u == a.nsb;
                if (tile_end || k + 1u == nu) {
                    // a whole tile goes to Y, a cut one to the workspace
                    asm volatile("griddepcontrol.wait;" ::: "memory");
                    const uint32_t rtile = tile / a.tok_tiles, tok0 = (tile - rtile * a.tok_tiles) * T;
                    const uint32_t n = rtile * kTileRows + rt * 128u + row, tok_n = min(a.M - tok0, (uint32_t)T);
                    const bool whole = tile_end && seg_head;
                    float* out = whole ? a.Y + (uint64_t)tok0 * a.N + n
                                       : a.part + ((uint64_t)blockIdx.x * 2u + (seg_head ? 1u : 0u)) * a.slot_rows * kTileRows + rt * 128u + row;
                    const uint32_t stride = whole ? a.N : kTileRows;
                    const float bias = whole && a.bias && n < a.N ? a.bias[n] : 0.f;
                    const bool row_ok = n < a.N || !whole;
                    // 2^-e of 32 activation rows a turn, one per lane: a load per value would cost the turn an L2 latency each
                    float iv = whole && lane < tok_n ? __ldcg(a.inv + tok0 + lane) : 1.f;
                    // 32 columns a turn, the rest moved down: the loop keeps the compiler from holding every column's address
                    // beside the sums (it spilled 114 of the 128), and leaves zeros behind
#pragma unroll 1
                    for (uint32_t c0 = 0; c0 < (uint32_t)T; c0 += 32) {
                        const float ivn = whole && c0 + 32u + lane < tok_n ? __ldcg(a.inv + tok0 + c0 + 32u + lane) : 1.f;
#pragma unroll
                        for (uint32_t j = 0; j < 32; j++) {
                            const float r = fmaf(y[j], __shfl_sync(0xFFFFFFFFu, iv, j), bias);
                            if (c0 + j < tok_n && row_ok &&
                                BPQ4K_CHECK(whole ? tok0 + c0 + j < a.M && n < a.N : c0 + j < a.slot_rows && blockIdx.x < kMaxCtas, a.status))
                                *out = r;
                            out += stride;
                        }
                        iv = ivn;
#pragma unroll
                        for (int j = 0; j < T; j++) y[j] = j + 32 < T ? y[j + 32 < T ? j + 32 : j] : 0.f;
                    }
                    seg_head = true;
                }
                if (tile_end) b = 0, tile++;
                else b++;
            }
            fence_before();
        }
    } else {
        // ---------------- dequantise, drain ----------------
        const uint32_t wk = warp - 4u, rt = wk >> 3, set = (wk >> 2) & 1u, quad = warp & 3u;
        const uint32_t row = quad * 32u + lane;            // lane of the row tile
        const uint32_t tl = tmem + ((quad * 32u) << 16);   // this warp's lanes
        constexpr int TH = T / 2;                          // columns this warp drains: [set*TH, set*TH + TH)
        constexpr int CH = TH % 16 == 0 ? 16 : TH % 8 == 0 ? 8 : 4;
        float y[TH];
#pragma unroll
        for (int j = 0; j < TH; j++) y[j] = 0.f;
        // The low halves' own sum, or one fma more a super-block: which is faster is the compiler's schedule (57344 x 8192, us,
        // two sums | one: 8 rows 86.4 | 87.7, 16 rows 95.7 | 89.9, 24 rows 95.1 | 97.8).
        constexpr bool TWO_SUMS = P::STACK && T <= 24 && T != 16;
        [[maybe_unused]] float yl[TWO_SUMS ? TH : 1];
        if constexpr (TWO_SUMS)
#pragma unroll
            for (int j = 0; j < TH; j++) yl[j] = 0.f;
        float s_prev = 0.f;
        uint32_t dtile = u0 / a.nsb, db = u0 - dtile * a.nsb;  // of the super-block that is drained next
        bool seg_head = db == 0;                             // its segment starts at its tile's first block
        uint32_t rs = rt, rit = 0;                          // raw ring position (stages alternate between the row tiles)
        uint32_t sa = set, ita = 0;                         // operand ring position (groups alternate between the sets)

        auto drain = [&](uint32_t kd, auto spread) {
            constexpr bool SPREAD = decltype(spread)::value;
            const uint32_t buf = kd % P::NBUF;
            wait_bar(acc_full(rt, buf), (kd / P::NBUF) & 1u, abort_flag, a.status);
            __syncwarp();
            fence_after();
            const uint32_t col = tl + acc_col(rt, buf) + set * TH;
            uint32_t hi[TH];
            [[maybe_unused]] uint32_t lo[P::STACK ? TH : 1];
#pragma unroll
            for (int c = 0; c < TH; c += CH) {
                tmem_ld<CH>(col + c, hi + c);
                if constexpr (P::STACK) tmem_ld<CH>(col + T + c, lo + c);
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(rt, buf));
            if constexpr (SPREAD) {  // (stacked, one activation tile)
#pragma unroll
                for (int c = 0; c < TH; c += 4) {
                    float f[4];
                    ldg128(a.sb_scale + db * T + set * TH + c, f);
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        y[c + j] = fmaf(s_prev, fmaf(__uint_as_float(lo[c + j]), kLowScaleInv, __uint_as_float(hi[c + j])) * f[j], y[c + j]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < TH; j++) {
                    if constexpr (TWO_SUMS) {
                        y[j] = fmaf(s_prev, __uint_as_float(hi[j]), y[j]);
                        yl[j] = fmaf(s_prev, __uint_as_float(lo[j]), yl[j]);
                    } else if constexpr (P::STACK) {
                        y[j] = fmaf(s_prev, fmaf(__uint_as_float(lo[j]), kLowScaleInv, __uint_as_float(hi[j])), y[j]);
                    } else {
                        y[j] = fmaf(s_prev, __uint_as_float(hi[j]), y[j]);
                    }
                }
            }
            const bool tile_end = db + 1u == a.nsb;
            if (tile_end || kd + 1u == nu) {
                // ---- end of a segment: a whole tile goes to Y, a cut one to the workspace ----
                if constexpr (TWO_SUMS) {
#pragma unroll
                    for (int j = 0; j < TH; j++) y[j] = fmaf(yl[j], kLowScaleInv, y[j]), yl[j] = 0.f;
                }
                asm volatile("griddepcontrol.wait;" ::: "memory");
                const uint32_t rtile = dtile / a.tok_tiles, tok0 = (dtile - rtile * a.tok_tiles) * T;
                const uint32_t n = rtile * kTileRows + rt * 128u + row;
                const uint32_t t0 = set * TH, tok_n = min(a.M - tok0, (uint32_t)T);
                bool write = true;
                if (!(tile_end && seg_head)) {
                    const uint64_t slot = (uint64_t)a.slot_rows * kTileRows;
                    float* mine = a.part + ((uint64_t)blockIdx.x * 2u + (seg_head ? 1u : 0u)) * slot + t0 * kTileRows + rt * 128u + row;
#pragma unroll
                    for (int j = 0; j < TH; j++)
                        if (t0 + j < tok_n && BPQ4K_CHECK(t0 + j < a.slot_rows && blockIdx.x < kMaxCtas, a.status)) mine[j * kTileRows] = y[j];
                    write = false;
                    if (!a.defer) {
                    const uint32_t c_first = unit_owner(dtile * a.nsb, a.u_base, a.u_extra);
                    const uint32_t c_last = unit_owner((dtile + 1u) * a.nsb - 1u, a.u_base, a.u_extra);
                    __threadfence();
                    asm volatile("bar.sync 1, %0;" ::"n"(kWorkers * 32) : "memory");
                    if (threadIdx.x == 4u * 32u) *last_flag = atomicInc(a.counters + c_first, c_last - c_first);
                    asm volatile("bar.sync 1, %0;" ::"n"(kWorkers * 32) : "memory");
                    write = *last_flag == c_last - c_first;  // this CTA is the tile's last: add the segments in order of k
                    if (write) {
                        __threadfence();
#pragma unroll
                        for (int j = 0; j < TH; j++) y[j] = 0.f;
                        for (uint32_t c = c_first; c <= c_last; c++) {
                            const float* p = a.part + ((uint64_t)c * 2u + (c == c_first ? 1u : 0u)) * slot + t0 * kTileRows + rt * 128u + row;
#pragma unroll
                            for (int j = 0; j < TH; j++) {
                                if (t0 + j < tok_n && BPQ4K_CHECK(t0 + j < a.slot_rows && c < gridDim.x, a.status)) y[j] += __ldcg(p + j * kTileRows);
                            }
                        }
                    }
                    asm volatile("bar.sync 1, %0;" ::"n"(kWorkers * 32) : "memory");  // last_flag may be written again
                    }
                }
                if (write && n < a.N) {
                    const float bias = a.bias ? a.bias[n] : 0.f;
                    float* out = a.Y + (uint64_t)(tok0 + t0) * a.N + n;
                    const float* inv = a.inv + tok0 + t0;
#pragma unroll
                    for (int j = 0; j < TH; j++) {
                        if (t0 + j < tok_n && BPQ4K_CHECK(tok0 + t0 + j < a.M, a.status)) *out = fmaf(y[j], __ldcg(inv + j), bias);
                        out += a.N;
                        if (j % 8 == 7) asm volatile("" ::: "memory");
                    }
                }
#pragma unroll
                for (int j = 0; j < TH; j++) y[j] = 0.f;
                seg_head = true;
            }
            if (tile_end) db = 0, dtile++;
            else db++;
        };

        auto turns = [&](uint32_t k0, uint32_t k1, auto spread) {
            for (uint32_t k = k0; k < k1; k++) {
            const bool more = k < nu;
            BlockScales h;
            if (more) {
                wait_bar(raw_full(rs), rit & 1u, abort_flag, a.status);
                const uint32_t rp = raw_slot(rs) + row * P::BLOCK;
                h.load<Q5>(lds128(rp));
#pragma unroll
                for (uint32_t gi = 0; gi < 2; gi++) {
                    const uint32_t g = set + 2u * gi;  // 64-weight group: sub-blocks 2g and 2g+1
                    const uint32_t cp = rp + (Q5 ? 48u : 16u) + g * 32u;
                    const GroupScales gs(h, g, Q5 ? 16.f : 8.f);
                    const uint32_t ta = tl + a_col(rt, sa);
                    const uint4 code[2] = {lds128(cp), lds128(cp + 16u)};
                    uint4 fifth[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
                    if constexpr (Q5) fifth[0] = lds128(rp + 16u), fifth[1] = lds128(rp + 32u);
                    if (gi == 1) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(raw_empty(rs));
                        rs += 2u;
                        if (rs >= P::NR) rs -= P::NR, rit++;
                    }
                    uint32_t v[32];
                    dequant_words<Q5>(code[0], fifth[0], g, gs, v);
                    dequant_words<Q5>(code[1], fifth[1], g, gs, v + 16);
                    if (ita > 0) wait_bar(a_empty(rt, sa), (ita - 1u) & 1u, abort_flag, a.status);
                    __syncwarp();
                    fence_after();
                    tmem_st16(ta, v);
                    tmem_st16(ta + 16u, v + 16);
                    if (gi == 1 && set == 1) {  // the last group of the super-block carries the constant terms of its eight sub-blocks
                        uint32_t cw[8];
                        constant_terms<Q5>(h, cw);
                        tmem_st8(ta + 32u, cw);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a_full(rt, sa));
                    sa += 2u;
                    if (sa >= P::NA) sa -= P::NA, ita++;
                }
            }
            if (k > 0) drain(k - 1u, spread);
            s_prev = h.s;
            }
        };
        if constexpr (P::STACK) {
            // the first drain needs to know whether some super-block of some row has a scale of its own
            turns(0, 1, std::false_type{});
            asm volatile("griddepcontrol.wait;" ::: "memory");
            uint32_t any = 0;
            for (uint32_t i = lane; i < a.n_spread; i += 32u) any |= __ldcg(a.spread + i);
            if (__any_sync(0xFFFFFFFFu, any != 0u)) turns(1, nu + 1u, std::true_type{});
            else turns(1, nu + 1u, std::false_type{});
        } else {
            turns(0, nu + 1u, std::false_type{});
        }
        fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Activations -> the image the matmul copies tile by tile.  Row t is scaled by a power of two that brings its largest
// magnitude into [2^14, 2^15) and split into halves.  Stacked (T <= 32): the low halves are scaled by 2^11 more, so that they
// have a half's whole range below them, and a super-block whose largest lies 2^4 or more below the row's is scaled by a power
// of its own (`spread` says that there is one; the drain then applies the powers, 3 to 5 % slower): a value keeps 22 bits down to
// 2^-24 of its super-block's largest, where the streaming kernel, which serves fewer rows, keeps 21 of the largest of 32.  Not
// stacked: 22 bits down to 2^-17 of the row's largest, 2^-39 of that below (the prefill kernel, which served these rows before,
// 2^-25 whatever the row).  Per activation tile and super-block four groups of T*256 bytes: rows
// 0..T-1 the high halves, T..2T-1 the low ones, 128 B each in the 128-byte swizzle, a 16-byte chunk i holding the
// activations of code word i in the order the dequantiser produces its weights (4i, 4i+2, 4i+1, 4i+3 of the even
// sub-block, then of the odd one); then the same rows with 32 B each: the mean of each of the eight sub-blocks, twice
// (both 16-byte chunks alike, so there is no swizzle to apply).
// A block serves one row; where the rows alone do not fill the machine several blocks share one, and each finds the
// row's maximum itself.  Rows past M are zeros.
// The matmul's counters are cleared here, in the order of the call's own stream, so that no call depends on what the memory
// held before it (a clear by another stream's memset would not be ordered against the kernel).
__global__ void __launch_bounds__(256) rows_pack_kernel(const float* __restrict__ X, uint32_t M, uint32_t K, uint32_t T,
                                                        uint8_t* __restrict__ image, float* __restrict__ inv,
                                                        float* __restrict__ sb_scale, uint32_t* __restrict__ spread,
                                                        uint32_t* __restrict__ counters, [[maybe_unused]] int* status) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ uint32_t red[8];
    const uint32_t row = blockIdx.y, tt = row / T, t = row - tt * T, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t nsb = K / kQK;
    const bool live = row < M;
    if (row == 0 && blockIdx.x == 0 && threadIdx.x < kMaxCtas) counters[threadIdx.x] = 0;
    const float4* x4 = reinterpret_cast<const float4*>(X + (uint64_t)row * K);
    const bool stack = T <= 32u;
    uint32_t e = 0;  // biased exponent of the row's scale
    if (live) {
        // magnitudes compare as integers; a NaN counts as larger than infinity and reaches every output of the row
        uint32_t mx = 0;
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < K / 4u; i += 256u) {
            const float4 v = __ldg(x4 + i);
            mx = max(max(mx, max(__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.y) & 0x7FFFFFFFu)),
                     max(__float_as_uint(v.z) & 0x7FFFFFFFu, __float_as_uint(v.w) & 0x7FFFFFFFu));
        }
        mx = __reduce_max_sync(0xFFFFFFFFu, mx);
        if (lane == 0) red[warp] = mx;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; i++) mx = max(mx, red[i]);
        e = min(268u - (mx >> 23), 253u);  // of 2^14 / 2^exponent(mx)
        if (blockIdx.x == 0 && threadIdx.x == 0) inv[row] = __uint_as_float((254u - e) << 23);
    }
    int spread_any = 0;
    const float low = stack ? kLowScale : 1.f;
    auto split = [low](float p, float q, uint32_t& h, uint32_t& l) {
        h = half2_bits(p, q);
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
        l = half2_bits((p - f.x) * low, (q - f.y) * low);
    };
    const uint32_t g = lane >> 3, i = lane & 7u;
    for (uint32_t sb = blockIdx.x * 8u + warp; sb < nsb; sb += gridDim.x * 8u) {
        float4 e4 = make_float4(0.f, 0.f, 0.f, 0.f), o4 = e4;
        if (live) {
            e4 = __ldg(x4 + sb * 64u + g * 16u + i);
            o4 = __ldg(x4 + sb * 64u + g * 16u + 8u + i);
        }
        uint32_t es = e;  // biased exponent of this super-block's scale
        if (stack) {
            auto mag = [](const float4& v) {
                return max(max(__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.y) & 0x7FFFFFFFu),
                           max(__float_as_uint(v.z) & 0x7FFFFFFFu, __float_as_uint(v.w) & 0x7FFFFFFFu));
            };
            const uint32_t mx = __reduce_max_sync(0xFFFFFFFFu, max(mag(e4), mag(o4))), own = min(268u - (mx >> 23), 253u);
            // (at most 2^100 beside the row's: the inverse stays an ordinary float)
            if (mx && own >= e + 4u) es = min(own, e + 100u), spread_any = 1;
        }
        if (live) {
            const float scale = __uint_as_float(es << 23);
            e4.x *= scale, e4.y *= scale, e4.z *= scale, e4.w *= scale;
            o4.x *= scale, o4.y *= scale, o4.z *= scale, o4.w *= scale;
        }
        uint4 hi, lo;
        split(e4.x, e4.z, hi.x, lo.x);
        split(e4.y, e4.w, hi.y, lo.y);
        split(o4.x, o4.z, hi.z, lo.z);
        split(o4.y, o4.w, hi.w, lo.w);
        if (!BPQ4K_CHECK((tt + 1u) * T <= gridDim.y && t < T && sb < nsb, status)) break;
        uint8_t* blk = image + ((uint64_t)tt * nsb + sb) * T * 1088u;
        if (stack && lane == 0) sb_scale[((uint64_t)tt * nsb + sb) * T + t] = live ? __uint_as_float((127u + e - es) << 23) : 0.f;
        auto put = [&](uint32_t r, const uint4& v) { *reinterpret_cast<uint4*>(blk + g * T * 256u + r * 128u + ((i ^ (r & 7u)) << 4)) = v; };
        put(t, hi);
        put(T + t, lo);
        float se = (e4.x + e4.y) + (e4.z + e4.w), so = (o4.x + o4.y) + (o4.z + o4.w);
#pragma unroll
        for (int m = 1; m < 8; m <<= 1) {
            se += __shfl_xor_sync(0xFFFFFFFFu, se, m);
            so += __shfl_xor_sync(0xFFFFFFFFu, so, m);
        }
        uint32_t sh, sl;
        split(0.03125f * se, 0.03125f * so, sh, sl);
        if (i < 4)  // two chunks of the high row, two of the low one
            *reinterpret_cast<uint32_t*>(blk + T * 1024u + (i < 2 ? t : T + t) * 32u + (i & 1u) * 16u + g * 4u) = i < 2 ? sh : sl;
    }
    if (stack) {
        spread_any = __syncthreads_or(spread_any);
        if (threadIdx.x == 0) spread[row * gridDim.x + blockIdx.x] = spread_any;
    }
}

// Cut tiles: the sum of the segments in ascending order of k, times 2^-e, plus the bias.  Where tiles are cut into many
// segments one CTA would add them with a chain of L2 latencies (1024 x 4096, 48 rows: 16 segments, 50 of 77 us); here
// a thread takes four weight rows of one activation row and the whole machine shares the work.
// One block: the tile that CTA blockIdx.x begins and others finish, four activation rows.
__global__ void __launch_bounds__(256) rows_reduce_kernel(const float* __restrict__ part, const float* __restrict__ inv,
                                                          const float* __restrict__ bias, float* __restrict__ Y, uint32_t M, uint32_t N,
                                                          uint32_t T, uint32_t tok_tiles, uint32_t slot_rows, uint32_t nsb, uint32_t u_base,
                                                          uint32_t u_extra, [[maybe_unused]] int* status) {
    const uint32_t tile = (unit_begin(blockIdx.x + 1u, u_base, u_extra) - 1u) / nsb;
    const uint32_t rtile = tile / tok_tiles, tok0 = (tile - rtile * tok_tiles) * T;
    const uint32_t t = blockIdx.y * 4u + (threadIdx.x >> 6), r4 = (threadIdx.x & 63u) * 4u, n = rtile * kTileRows + r4;
    const uint32_t c_first = unit_owner(tile * nsb, u_base, u_extra), c_last = unit_owner((tile + 1u) * nsb - 1u, u_base, u_extra);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (c_first != blockIdx.x || c_first == c_last || t >= slot_rows || tok0 + t >= M || n >= N) return;
    if (!BPQ4K_CHECK(c_last < gridDim.x && c_first < c_last, status)) return;
    const uint64_t slot = (uint64_t)slot_rows * kTileRows;
    const float* p = part + (uint64_t)c_first * 2u * slot + t * kTileRows + r4;
    float4 s = __ldcg(reinterpret_cast<const float4*>(p + slot));
#pragma unroll 8
    for (uint32_t c = c_first + 1u; c <= c_last; c++) {
        p += 2u * slot;
        const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
        s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
    }
    const float k = __ldcg(inv + tok0 + t);
    float* out = Y + (uint64_t)(tok0 + t) * N + n;
    const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
        if (n + i < N) out[i] = fmaf(v[i], k, bias ? bias[n + i] : 0.f);
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// Activation rows per tile: up to 128 rows one tile, above that the rows are shared out evenly over as few tiles of at
// most 128 as possible (T: see RowsPlan).
uint32_t rows_tile(uint32_t M) {
    const uint32_t tiles = (M + 127u) / 128u, per = (M + tiles - 1u) / tiles;
    return per <= 32u ? (per + 7u) & ~7u : per <= 48u ? 48u : (per + 15u) & ~15u;
}

template <int T, int QT>
cudaError_t launch_rows(const RowsArgs& ra, uint32_t grid, bool pdl, cudaStream_t stream) {
    using P = RowsPlan<T, QT>;
    static KernelConfig kcfg;
    if (cudaError_t e = kcfg.prepare(reinterpret_cast<const void*>(rows_tc_kernel<T, QT>), kThreads, P::SMEM_BYTES, nullptr)) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = P::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, rows_tc_kernel<T, QT>, ra);
}

template <int QT>
cudaError_t launch_rows_t(uint32_t T, const RowsArgs& ra, uint32_t grid, bool pdl, cudaStream_t stream) {
    switch (T) {
        case 8: return launch_rows<8, QT>(ra, grid, pdl, stream);
        case 16: return launch_rows<16, QT>(ra, grid, pdl, stream);
        case 24: return launch_rows<24, QT>(ra, grid, pdl, stream);
        case 32: return launch_rows<32, QT>(ra, grid, pdl, stream);
        case 48: return launch_rows<48, QT>(ra, grid, pdl, stream);
        case 64: return launch_rows<64, QT>(ra, grid, pdl, stream);
        case 80: return launch_rows<80, QT>(ra, grid, pdl, stream);
        case 96: return launch_rows<96, QT>(ra, grid, pdl, stream);
        case 112: return launch_rows<112, QT>(ra, grid, pdl, stream);
        default: return launch_rows<128, QT>(ra, grid, pdl, stream);
    }
}

}  // namespace

// Blocks of rows_pack_kernel that share a row: one from four blocks per SM on, else as many as the row has warps' work for.
static uint32_t pack_blocks(uint32_t rows, uint32_t nsb, uint32_t ctas) {
    const uint32_t want = 4u * ctas / rows, most = (nsb + 7u) / 8u;
    return want < 1u ? 1u : want < most ? want : most;
}
constexpr uint32_t kSpreadWords = 32u * (kRowsMaxK / kQK / 8u);

// Buffer of a call: the counters, the activation scales (2^-e), the image, (to 32 rows) the words of `spread` and the
// super-blocks' scales, two cut tiles per CTA.
constexpr size_t kCounterBytes = 1024;
static_assert(kCounterBytes >= kMaxCtas * 4u, "counters");
static size_t rows_head_bytes(uint32_t M) { return kCounterBytes + (((size_t)M * 4u + 127u + 256u) & ~(size_t)255u); }
static size_t rows_image_bytes(uint32_t M, uint32_t K) {
    const uint32_t T = rows_tile(M), tiles = (M + T - 1u) / T;
    return (size_t)tiles * T * (K / kQK) * 1088u + (((T <= 32u ? kSpreadWords * 4u + (size_t)T * (K / kQK) * 4u : 0u) + 255u) & ~(size_t)255u);
}
static size_t rows_part_bytes(uint32_t M) {
    const uint32_t T = rows_tile(M);
    return (size_t)kMaxCtas * 2u * (M < T ? M : T) * kTileRows * 4u;
}
size_t rows_buffer_bytes(uint32_t M, uint32_t K) { return rows_head_bytes(M) + rows_image_bytes(M, K) + rows_part_bytes(M); }

// Units of the busiest CTA (a unit's mmas grow with the tile, its dequantisation does not; Q5_K's fifth bit), the ends of its
// tiles, the segments of cut tiles that are written and read again, the packing of the activations.  Fitted, like the
// prefill kernel's, to 2,116 timed calls (65 to 2048 rows, weights from 64 x 1024 to 128256 x 4096 and 40960 x 28672, both
// types; 9 % rms).  The choice between the two misses the faster kernel by more than 6 % for 104 of them, by 20 % at most.
double rows_estimate_us(uint32_t M, uint32_t N, uint32_t K, int sm_count, int qtype) {
    const uint32_t T = rows_tile(M), ctas = (uint32_t)sm_count < kMaxCtas ? (uint32_t)sm_count : kMaxCtas;
    const uint64_t nsb = K / kQK, tiles = (uint64_t)((N + kTileRows - 1u) / kTileRows) * ((M + T - 1u) / T), units = tiles * nsb;
    const uint64_t grid = units < ctas ? units : ctas, per = (units + grid - 1u) / grid;
    const uint64_t cuts = units % (grid * nsb) == 0u ? 0u : grid - 1u, segments = cuts + (cuts < tiles ? cuts : tiles);
    const double t = T / 128.0;
    const bool q5 = qtype == 13;
    return 5.5 + (double)per * ((q5 ? 1.54 : 1.33) + (q5 ? 3.95 : 3.54) * t) + 7.3 * t * (double)((per + nsb - 1u) / nsb) +
           0.91e-6 * (double)segments * (M < T ? M : T) * kTileRows + 1.77e-6 * M * K;
}

cudaError_t launch_rows_tc(const MatmulArgs& m, void* buffer, size_t buffer_bytes, int* status_dev, int sm_count,
                           TmapCache* tmaps, bool pdl, cudaStream_t stream, int* launches, int qtype) {
    if (m.M == 0 || m.N == 0) return cudaSuccess;
    if ((qtype != 12 && qtype != 13) || m.n_slots || m.n_peers || m.prologue || m.residual || m.M > kRowsMaxM || m.K > kRowsMaxK ||
        !buffer || buffer_bytes < rows_buffer_bytes(m.M, m.K))
        return cudaErrorInvalidValue;
    const bool q5 = qtype == 13;
    const uint32_t nsb = m.K / kQK, block_words = q5 ? 44u : 36u, T = rows_tile(m.M);
    const uint32_t tok_tiles = (m.M + T - 1u) / T;
    const uint32_t ctas = (uint32_t)sm_count < kMaxCtas ? (uint32_t)sm_count : kMaxCtas;
    uint8_t* buf = static_cast<uint8_t*>(buffer);
    RowsArgs ra{};
    ra.counters = reinterpret_cast<uint32_t*>(buf);
    ra.inv = reinterpret_cast<const float*>(buf + kCounterBytes);
    ra.image = buf + rows_head_bytes(m.M);
    ra.spread = reinterpret_cast<const uint32_t*>(ra.image + (size_t)tok_tiles * T * nsb * 1088u);
    ra.sb_scale = reinterpret_cast<const float*>(ra.spread + kSpreadWords);
    ra.n_spread = T <= 32u ? pack_blocks(tok_tiles * T, nsb, ctas) * T : 0u;
    ra.part = reinterpret_cast<float*>(buf + rows_head_bytes(m.M) + rows_image_bytes(m.M, m.K));
    ra.tok_tiles = tok_tiles;
    ra.slot_rows = m.M < T ? m.M : T;
    ra.bias = m.bias;
    ra.Y = m.Y;
    ra.M = m.M;
    ra.N = m.N;
    ra.nsb = nsb;
    ra.status = status_dev;
    const uint64_t units64 = (uint64_t)((m.N + kTileRows - 1u) / kTileRows) * tok_tiles * nsb;
    if (units64 > 0x3FFFFFFFull) return cudaErrorInvalidValue;  // (group numbers stay below 2^32)
    const uint32_t units = (uint32_t)units64;
    const uint32_t grid = units < ctas ? units : ctas;
    ra.u_base = units / grid;
    ra.u_extra = units % grid;
    // a tile of nsb units is cut into at most (nsb - 2) / u_base + 2 segments; up to three the last CTA adds them itself
    ra.defer = T > 48u ? 1u : nsb > 1u && (nsb - 2u) / ra.u_base + 2u > 3u;
    const uint32_t key_nb = nsb | (q5 ? 0x50000000u : 0u), key_cb = 0x80u;  // apart from the streaming kernel's boxes of the same weights
    bool found = false;
    if (tmaps)
        for (const auto& en : tmaps->entries)
            if (en.W == m.W && en.rows == m.N && en.row_bytes == m.w_row_bytes && en.nb == key_nb && en.cb == key_cb) {
                std::memcpy(&ra.tmap_w, en.map, sizeof(CUtensorMap));
                found = true;
                break;
            }
    if (!found) {
        EncodeTiledFn enc = encode_fn();
        if (!enc) return cudaErrorNotSupported;
        const cuuint64_t gdim[2] = {(cuuint64_t)nsb * block_words, (cuuint64_t)m.N};
        const cuuint64_t gstride[1] = {(cuuint64_t)m.w_row_bytes};
        const cuuint32_t box[2] = {block_words, 128u};
        const cuuint32_t estr[2] = {1u, 1u};
        if (enc(&ra.tmap_w, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t*>(m.W), gdim, gstride, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
        if (tmaps) {
            auto& en = tmaps->entries[tmaps->next++ % TmapCache::kEntries];
            en.W = m.W, en.rows = m.N, en.row_bytes = m.w_row_bytes, en.nb = key_nb, en.cb = key_cb;
            std::memcpy(en.map, &ra.tmap_w, sizeof(CUtensorMap));
        }
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(pack_blocks(tok_tiles * T, nsb, ctas), tok_tiles * T);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, rows_pack_kernel, m.X, m.M, m.K, T, const_cast<uint8_t*>(ra.image), const_cast<float*>(ra.inv),
                                       const_cast<float*>(ra.sb_scale), const_cast<uint32_t*>(ra.spread), ra.counters, status_dev);
    if (launches) ++*launches;
    if (e != cudaSuccess) return e;
    e = q5 ? launch_rows_t<1>(T, ra, grid, pdl, stream) : launch_rows_t<0>(T, ra, grid, pdl, stream);
    if (launches) ++*launches;
    if (e != cudaSuccess || !ra.defer) return e;
    cfg.gridDim = dim3(grid, (ra.slot_rows + 3u) / 4u);
    e = cudaLaunchKernelEx(&cfg, rows_reduce_kernel, (const float*)ra.part, ra.inv, ra.bias, ra.Y, ra.M, ra.N, T, tok_tiles, ra.slot_rows, nsb,
                           ra.u_base, ra.u_extra, status_dev);
    if (launches) ++*launches;
    return e;
}

}  // namespace bpq4k
