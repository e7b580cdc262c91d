// Device building blocks shared by the tensor-core kernels: bounded mbarrier waits, TMA copies, tcgen05 forms, and the
// fixed-point requantisation of one accumulator with its per-column constants.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "requant.h"

namespace enn_b200 {
namespace {

constexpr int kBM = 128;            // rows per tile = UMMA M
constexpr int kBK = 128;            // bytes of K per stage = one 128B swizzle atom = 4 UMMA K steps
constexpr int kMaxBN = 256;         // UMMA N limit
constexpr uint32_t kSpinLimit = 1u << 24;

struct ColParam {   // per output column, 16 bytes
    int32_t mult;
    int32_t addend;   // stage-2 addend: 2^(e-1) + ((out_zp - act_min) << e)
    int32_t esh;      // right shift e >= 1 of the fused form; negative: general requantisation, `addend` = raw shift
    int32_t bias;     // folded bias'
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait of the single-thread roles (producers, MMA issuer).  Callers look at the barrier with the non-blocking
// test_wait first (the common case: already complete); what is left waits with try_wait, which parks the thread in
// hardware between looks instead of spinning through issue slots that the epilogue warps of the same scheduler need.
__device__ __forceinline__ bool mbar_wait_fast(uint32_t bar, uint32_t parity, volatile int *abort_flag, int32_t *err, int code,
                                               uint32_t looks = kSpinLimit >> 7) {
    for (uint32_t i = 0; i < looks; ++i) {       // by default 2^17 looks of up to 10 us: gives up after about a second
        // suspend-time hint (ns): stay parked until the phase completes instead of coming back every few hundred cycles
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(10000u)
            : "memory");
        if (ok) return true;
        if ((i & 63u) == 63u && *abort_flag) return false;
    }
    *abort_flag = 1;
    if (err) *reinterpret_cast<volatile int32_t *>(err) = code;
    return false;
}
// Bounded wait.  Returns false after the limit (or when another thread already aborted the CTA).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int32_t *err, int code) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023u) == 1023u && *abort_flag) return false;
    }
    *abort_flag = 1;
    if (err) *reinterpret_cast<volatile int32_t *>(err) = code;
    return false;
}

// A producer that gives up waits, with a limit, for its copies in flight before the shared memory is given back.  (stage, phase) is the
// next fill: stages before it were last filled in the ring's present round, the others in the round before (never filled: nothing to
// wait for).  Lanes that fill alternate stages pass theirs as first and step.
__device__ __forceinline__ void drain_stages(uint32_t full0, uint32_t nst, uint32_t stage, uint32_t phase, uint32_t first = 0, uint32_t step = 1) {
    for (uint32_t s = first; s < nst; s += step)
        for (uint32_t i = 0; i < (1u << 12); ++i)
            if (mbar_try_wait(full0 + 8 * s, s < stage ? phase : phase ^ 1)) break;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t c0, int32_t c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Arrives on the mbarrier once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- CTA-pair (cta_group::2) forms: two CTAs of a cluster compute one 256-row tile, each holding its own 128 rows of
// A, half of the B rows and its 128 accumulator lanes.  The MMA is issued by the rank-0 CTA only.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Address of the same shared-memory offset in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The tile lands in this CTA's shared memory; the bytes are counted on the rank-0 CTA's barrier (cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster, int32_t c0, int32_t c1) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t slot_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    const uint16_t mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask) : "memory");
}

// One k-block: KS (1, 2 or 4) MMAs over consecutive 32-byte K slices of the A tile at descriptor address `lo_a` and the
// B tile at `lo_b` (16-byte units; `desc_hi` = the constant upper descriptor word).  All descriptors are formed first, then
// the MMAs follow each other as one uninterrupted instruction run.  The first MMA overwrites the accumulator when
// `accumulate_first` is 0.
template <bool TWO, int KS>
__device__ __forceinline__ void umma_i8_run(uint32_t d_tmem, uint32_t desc_hi, uint32_t lo_a, uint32_t lo_b, uint32_t idesc,
                                            uint32_t accumulate_first) {
#define ENN_MMA_PAIR "tcgen05.mma.cta_group::2.kind::i8"
#define ENN_MMA_ONE "tcgen05.mma.cta_group::1.kind::i8"
#define ENN_DESC(I, OFF)                                                       \
    "add.u32 t, %2, " #OFF ";\n\tmov.b64 a" #I ", {t, %1};\n\t"                 \
    "add.u32 t, %3, " #OFF ";\n\tmov.b64 b" #I ", {t, %1};\n\t"
#define ENN_RUN_HEAD                                                                                  \
    "{\n\t.reg .pred p, q;\n\t.reg .b64 a0, a1, a2, a3, b0, b1, b2, b3;\n\t.reg .b32 t;\n\t"           \
    "setp.ne.b32 p, %5, 0;\n\t"                                                                       \
    "setp.eq.b32 q, %5, %5;\n\t"
#define ENN_RUN_ARGS ::"r"(d_tmem), "r"(desc_hi), "r"(lo_a), "r"(lo_b), "r"(idesc), "r"(accumulate_first) : "memory"
#define ENN_RUN(MMA)                                                                                                   \
    if (KS == 4)                                                                                                       \
        asm volatile(ENN_RUN_HEAD ENN_DESC(0, 0) ENN_DESC(1, 2) ENN_DESC(2, 4) ENN_DESC(3, 6)                         \
                     MMA " [%0], a0, b0, %4, p;\n\t" MMA " [%0], a1, b1, %4, q;\n\t" MMA " [%0], a2, b2, %4, q;\n\t" \
                     MMA " [%0], a3, b3, %4, q;\n\t}" ENN_RUN_ARGS);                                                   \
    else if (KS == 2)                                                                                                  \
        asm volatile(ENN_RUN_HEAD ENN_DESC(0, 0) ENN_DESC(1, 2)                                                       \
                     MMA " [%0], a0, b0, %4, p;\n\t" MMA " [%0], a1, b1, %4, q;\n\t}" ENN_RUN_ARGS);                   \
    else                                                                                                               \
        asm volatile(ENN_RUN_HEAD ENN_DESC(0, 0) MMA " [%0], a0, b0, %4, p;\n\t}" ENN_RUN_ARGS);
    if (TWO) { ENN_RUN(ENN_MMA_PAIR) } else { ENN_RUN(ENN_MMA_ONE) }
#undef ENN_RUN
#undef ENN_RUN_ARGS
#undef ENN_RUN_HEAD
#undef ENN_DESC
#undef ENN_MMA_ONE
#undef ENN_MMA_PAIR
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major operand tile in shared memory, 128-byte rows, 128B swizzle: rows are 128 bytes apart, groups of 8
// rows 1024 bytes apart (stride byte offset), descriptor version 1, layout type 2 (SWIZZLE_128B).
// `span` = bytes per row = swizzle span (128 / 64 / 32): groups of 8 rows are 8 * span bytes apart and the layout
// type is SWIZZLE_128B (2), SWIZZLE_64B (4) or SWIZZLE_32B (6).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t span = 128) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);        // start address, 16-byte units
    d |= static_cast<uint64_t>(1) << 16;                            // leading byte offset (unused for swizzled K-major)
    d |= static_cast<uint64_t>((8 * span) >> 4) << 32;              // stride byte offset
    d |= static_cast<uint64_t>(1) << 46;                            // descriptor version
    d |= static_cast<uint64_t>(span == 128 ? 2 : (span == 64 ? 4 : 6)) << 61;
    return d;
}

__device__ __forceinline__ uint32_t pack_sat_u8_tc(int32_t hi, int32_t lo, uint32_t upper) {
    uint32_t d;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(hi), "r"(lo), "r"(upper));
    return d;
}

// Epilogue modes (one kernel variant each; the planner picks the cheapest one every column of the operator allows):
//   kModeNudge   fused two-stage form below, every column a right shift e >= 1;
//   kModeGeneral as kModeNudge, but columns flagged esh < 0 take the general code (left shifts, e == 0, wide ranges);
//   kModeReluTwo lower clamp == output zero point (ReLU-type outputs): a negative stage-1 value ends at the clamp with or
//                without the tie correction, so the correction is dropped and the bias, both rounding terms and a left
//                shift ls fold into one 64-bit addend: q = acc * M0 + C, C = bias * M0 + 2^(30-ls) (+ 2^(e-1+31-ls) when
//                e >= 1); result = (q >> (31 - ls)) >> e.  Covers e == 0 and left shifts, which otherwise need the
//                general code.
//   kModeReluHi  the same with one shift, hi32(q) >> (e - 1), for operators whose columns all have e >= 1 and ls == 0
//                (two ALU instructions per output fewer; option no_relu_hi keeps the two-shift form).
// ColParam words: {mult, addend, esh, bias} for the first two modes, {C low, C high, mult, shifts} for the ReLU modes
// (shifts = e - 1 for kModeReluHi, (31 - ls) | e << 8 for kModeReluTwo).
constexpr int kModeNudge = 0, kModeGeneral = 1, kModeReluHi = 2, kModeReluTwo = 3;
// kModeReluHi for outputs whose clamp is the whole unsigned byte (lower clamp 0, upper clamp 255, unsigned bytes): the
// saturating byte pack is the clamp, so the min / max and the add of the lower clamp to the packed word are left out.
// A kernel template value only: the plan and the ColParam contents are those of kModeReluHi.
constexpr int kModeReluSat = 4;

// The constants of one column in registers.  The ReLU modes read {C, (M0, shifts)} as two 64-bit words, so that the
// 64-bit addend arrives as a register pair and need not be assembled from two 32-bit registers.
struct ColRegs {
    int4 v;
    int64_t cc;
};
// `p` points into shared memory (derived from the kernel's shared array, so the compiler emits shared loads with
// the constant part of the address as the instruction's immediate offset).
template <int MODE>
__device__ __forceinline__ void ld_col_shared(const uint8_t *p, ColRegs &c) {
    __builtin_assume(__isShared(p));
    if (MODE >= kModeReluHi) {
        const longlong2 v = *reinterpret_cast<const longlong2 *>(p);
        c.cc = v.x;
        asm("mov.b64 {%0, %1}, %2;" : "=r"(c.v.z), "=r"(c.v.w) : "l"(v.y));
    } else {
        c.v = *reinterpret_cast<const int4 *>(p);
    }
}

// Requantise one accumulator (bias not yet added) to (value - act_min) in [0, act_max - act_min]; kModeReluSat leaves
// the clamp to the caller's saturating pack.
// Fast form (esh = right shift e >= 1): stage 1 is one 32x32->64 multiply-add and a funnel shift, stage 2 is
// (x + addend - [x < 0]) >> e with addend = 2^(e-1) + ((out_zp - act_min) << e), i.e. RoundingDivideByPOT
// (ties away from zero) with the zero point and the lower clamp folded in.
template <int MODE>
__device__ __forceinline__ int32_t tc_requant(int32_t acc, const ColRegs &cr, int32_t hi_clamp, int32_t out_zp, int32_t act_min,
                                              int32_t act_max) {
    const int4 &c = cr.v;
    if (MODE >= kModeReluHi) {
        const int64_t q = static_cast<int64_t>(acc) * c.z + cr.cc;
        int32_t lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(q));
        int32_t v;
        if (MODE == kModeReluTwo) {
            const int32_t xa = static_cast<int32_t>(__funnelshift_r(static_cast<uint32_t>(lo), static_cast<uint32_t>(hi), static_cast<uint32_t>(c.w)));
            v = xa >> (c.w >> 8);
        } else {
            v = hi >> c.w;
        }
        if (MODE == kModeReluSat) return v;
        return __vimin_s32_relu(v, hi_clamp);
    }
    acc += c.w;
    if (MODE == kModeGeneral && c.z < 0) return enn_requant(acc, c.x, c.y, out_zp, act_min, act_max) - act_min;   // c.y = raw shift
    const int64_t p = static_cast<int64_t>(acc) * c.x + (1ll << 30);
    const int32_t x = static_cast<int32_t>(p >> 31);
    const int32_t v = (x + c.y - static_cast<int32_t>(static_cast<uint32_t>(x) >> 31)) >> c.z;
    return __vimin_s32_relu(v, hi_clamp);
}
// The same from the four 32-bit words of a ColParam.
template <int MODE>
__device__ __forceinline__ int32_t tc_requant(int32_t acc, const int4 &c, int32_t hi_clamp, int32_t out_zp, int32_t act_min,
                                              int32_t act_max) {
    ColRegs cr;
    cr.v = c;
    cr.cc = 0;
    if (MODE >= kModeReluHi) asm("mov.b64 %0, {%1, %2};" : "=l"(cr.cc) : "r"(c.x), "r"(c.y));
    return tc_requant<MODE>(acc, cr, hi_clamp, out_zp, act_min, act_max);
}

// Fused add: four requantised bytes and the four bytes of the other addend at the same place go through the quantized add
// exactly as add_kernel_vec computes it (kernels_direct.cu): stage 1 of either input from the operator's tables in shared
// memory, stage 2 computed.
struct FaddCtx {
    uint32_t lut_u32;       // 2 x 256 words in shared memory: input-0 table, input-1 table
    int32_t mo, so, out_off, act_min, act_max;
    bool swap;
};
__device__ __forceinline__ uint32_t fadd_word(uint32_t y, uint32_t r, const FaddCtx &f) {
    const uint32_t a = f.swap ? r : y, b = f.swap ? y : r;
    uint32_t word = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t ba = (a >> (8 * k)) & 0xff, bb = (b >> (8 * k)) & 0xff;
        int32_t x0, x1;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x0) : "r"(f.lut_u32 + ba * 4));
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x1) : "r"(f.lut_u32 + 1024 + bb * 4));
        int32_t o = enn_rdivpot(enn_srdhm(x0 + x1, f.mo), -f.so) + f.out_off;
        o = max(f.act_min, o);
        o = min(f.act_max, o);
        word |= (static_cast<uint32_t>(o) & 0xff) << (8 * k);
    }
    return word;
}
// ---------------------------------------------------------------------------------------------------------------------
// Epilogue of one accumulator tile, "quad" form.
//
// tcgen05.ld 16x256b hands a thread the two columns 2q, 2q + 1 (q = lane & 3) of every group of eight for the rows
// lane / 4 and lane / 4 + 8, so a warp's quarter of the tile (32 rows) gives a thread FOUR rows of the same columns.  The
// constants of a column are then loaded from shared memory once per four outputs instead of once per output: with one row
// per thread (32x32b) those 16-byte loads, two to four data cycles of the load-store unit each, were what bounded every
// epilogue (75 % of that unit's cycles in the 3x3 layer 256x56x56x64).  The planners permute the channels within groups of 32
// so that a thread's eight columns of a group are eight consecutive output channels: a quad stores whole 32-byte sectors.
//
// Channel c of an N tile of bn_data channels (bn_data % 16 == 0; a last group of 16 uses four channels per thread):
//   tile_row   row of the packed weights = accumulator column
//   tile_slot  position of its constants: the four threads of a quad read 64 consecutive bytes
// ---------------------------------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ int tile_row(int c, int bn_data) {
    const int g = c & ~31, r = c & 31;
    if (g + 32 <= bn_data) return g + 8 * ((r & 7) >> 1) + 2 * (r >> 3) + (r & 1);
    return g + 8 * ((r & 3) >> 1) + 2 * ((r >> 2) & 3) + (r & 1);
}
__host__ __device__ __forceinline__ int tile_slot(int c, int bn_data) {
    const int g = c & ~31, r = c & 31;
    return g + 32 <= bn_data ? g + 4 * (r & 7) + (r >> 3) : g + 4 * (r & 3) + ((r >> 2) & 3);
}

__device__ __forceinline__ void tmem_ld_16x256_x1(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
// 8 * NJ columns of 16 rows, NJ = 2 or 4: r[4 * j + 2 * h + s] = row lane / 4 + 8 * h, column 8 * j + 2 * (lane & 3) + s.
template <int NJ>
__device__ __forceinline__ void tmem_ld_16x256(uint32_t taddr, uint32_t (&r)[4 * NJ]) {
    if constexpr (NJ == 4)
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                       "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr)
                     : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr)
                     : "memory");
}

// What the epilogue of a kernel needs to know once.
struct EpiArgs {
    int32_t hi_clamp, out_zp, act_min, act_max;
    uint32_t lo_word, sign_word;    // lower clamp added back to the packed bytes, sign flip of signed outputs
    int align;                      // widest store every row start allows: 8, 4 or 1
    ptrdiff_t res_delta;            // fused add: the other addend relative to the output
    FaddCtx fadd;
};
// ... and once per tile.
struct EpiTile {
    uint8_t *row[4];        // first output byte of this thread's rows (tile column 0), rows lane / 4 + 8 * h of the quarter
    uint32_t live;          // bit h: row h exists
    int32_t asum[4];        // zw' * sum_k a of the rows
    int n_left;             // real columns of the tile
};

// P: the kernel's parameters.  Unsigned outputs: byte + act_min <= act_max <= 255, so a plain 32-bit add of the lower clamp never
// carries between bytes.  Signed outputs (act_min may be negative): the bytes get act_min + 128 (0..127, sums again <= 255)
// and the sign bit of every byte is flipped afterwards.
template <typename P>
__device__ __forceinline__ EpiArgs epi_args(const P &p, int64_t st_bits, ptrdiff_t res_delta, const FaddCtx &fadd) {
    EpiArgs e;
    e.hi_clamp = p.act_max - p.act_min;
    e.out_zp = p.out_zp; e.act_min = p.act_min; e.act_max = p.act_max;
    e.sign_word = p.a_signed ? 0x80808080u : 0u;
    e.lo_word = (static_cast<uint32_t>(p.act_min + (p.a_signed ? 128 : 0)) & 0xff) * 0x01010101u;
    e.align = (st_bits & 7) == 0 ? 8 : ((st_bits & 3) == 0 ? 4 : 1);
    e.res_delta = res_delta;
    e.fadd = fadd;
    return e;
}

// Requantises columns [c0, c0 + 8 * NJ) of the warp's 32 rows and stores them.  `t_row`: TMEM address of the tile's column
// 0 in the warp's lane quarter; `cols`: the tile's constants in shared memory.  FULL: every row and column is real and rows
// start on 8-byte boundaries; the general form's tests (per row and store width) cost as much as the requantisation itself.
template <int MODE, bool ASUM, bool FADD, int NJ, bool FULL>
__device__ __forceinline__ void epi_group(uint32_t t_row, const uint8_t *cols, int c0, const EpiTile &t, int lane, const EpiArgs &e) {
    constexpr bool kPlainPack = MODE == kModeReluSat;      // packed bytes are final: no lower clamp to add, no sign flip
    constexpr int kCh = 2 * NJ;                            // consecutive channels per thread: 8 or 4
    const int q = lane & 3;
    uint32_t r[2][4 * NJ];
    tmem_ld_16x256<NJ>(t_row + c0, r[0]);
    tmem_ld_16x256<NJ>(t_row + (16u << 16) + c0, r[1]);
    tmem_ld_wait();
    const uint8_t *cp = cols + (c0 + q) * 16;
    uint32_t w[4][kCh / 4];
#pragma unroll
    for (int i4 = 0; i4 < kCh / 4; ++i4) {
        int32_t y[4][4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int i = 4 * i4 + b;
            ColRegs cv;
            ld_col_shared<MODE>(cp + i * 64, cv);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                int32_t acc = static_cast<int32_t>(r[h >> 1][4 * (i >> 1) + 2 * (h & 1) + (i & 1)]);
                if (ASUM) acc -= t.asum[h];
                y[h][b] = tc_requant<MODE>(acc, cv, e.hi_clamp, e.out_zp, e.act_min, e.act_max);
            }
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const uint32_t hi = pack_sat_u8_tc(y[h][3], y[h][2], 0);
            const uint32_t pk = pack_sat_u8_tc(y[h][1], y[h][0], hi);
            w[h][i4] = kPlainPack ? pk : ((pk + e.lo_word) ^ e.sign_word);
        }
    }
    const int cb = c0 + kCh * q;                            // this thread's first column
    const int left = FULL ? kCh : t.n_left - cb;            // how many real ones from there on
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        if (!FULL && !(t.live >> h & 1)) continue;
        uint8_t *o = t.row[h] + cb;
        if constexpr (FADD) {                               // rows of 16-byte multiples only (plan)
            if (left >= kCh) {
                const uint8_t *res = o + e.res_delta;
#pragma unroll
                for (int k = 0; k < kCh / 4; ++k) w[h][k] = fadd_word(w[h][k], *reinterpret_cast<const uint32_t *>(res + 4 * k), e.fadd);
            }
        }
        if (FULL || (left >= kCh && e.align >= kCh)) {
            if constexpr (NJ == 4) *reinterpret_cast<uint2 *>(o) = make_uint2(w[h][0], w[h][1]);
            else *reinterpret_cast<uint32_t *>(o) = w[h][0];
        } else if (e.align >= 4 && (left & 3) == 0) {
#pragma unroll
            for (int k = 0; k < kCh / 4; ++k)
                if (4 * k < left) *reinterpret_cast<uint32_t *>(o + 4 * k) = w[h][k];
        } else {
#pragma unroll
            for (int b = 0; b < kCh; ++b)
                if (b < left) o[b] = static_cast<uint8_t>(w[h][b >> 2] >> (8 * (b & 3)));
        }
    }
}

// Column groups first, first + step, ... of a tile of bn_data columns for the warp's 32 rows.  cols_of(c0) returns the
// pointer the constants of columns c0 ... lie behind (at entry c0).
template <int MODE, bool ASUM, bool FADD, typename ColsOf>
__device__ __forceinline__ void epi_tile(uint32_t t_row, int first, int step, int bn_data, const EpiTile &t, int lane, const EpiArgs &e, ColsOf cols_of) {
    const bool rows_full = __all_sync(0xffffffffu, t.live == 15u) && e.align == 8;
    int c0 = first * 32;
    if (rows_full)
        for (; c0 + 32 <= t.n_left; c0 += 32 * step) epi_group<MODE, ASUM, FADD, 4, true>(t_row, cols_of(c0), c0, t, lane, e);
    for (; c0 < t.n_left; c0 += 32 * step) {
        if (c0 + 32 <= bn_data) epi_group<MODE, ASUM, FADD, 4, false>(t_row, cols_of(c0), c0, t, lane, e);
        else epi_group<MODE, ASUM, FADD, 2, false>(t_row, cols_of(c0), c0, t, lane, e);
    }
}

// zw' * sum_k a of this thread's four rows: accumulator column `col` of the extra group of 16.
__device__ __forceinline__ void epi_asum(uint32_t t_row, int col, int32_t zw_eff, int lane, int32_t (&asum)[4]) {
    uint32_t a[4], b[4];
    tmem_ld_16x256_x1(t_row + col, a);
    tmem_ld_16x256_x1(t_row + (16u << 16) + col, b);
    tmem_ld_wait();
    const int src = lane & ~3;      // column 0 of the group sits in the quad's first thread
    asum[0] = zw_eff * static_cast<int32_t>(__shfl_sync(0xffffffffu, a[0], src));
    asum[1] = zw_eff * static_cast<int32_t>(__shfl_sync(0xffffffffu, a[2], src));
    asum[2] = zw_eff * static_cast<int32_t>(__shfl_sync(0xffffffffu, b[0], src));
    asum[3] = zw_eff * static_cast<int32_t>(__shfl_sync(0xffffffffu, b[2], src));
}

}  // namespace
}  // namespace enn_b200
