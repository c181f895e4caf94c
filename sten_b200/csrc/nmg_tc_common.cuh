// Shared pieces of the tcgen05 kernels: tile constants, tile order, TMEM / MMA / descriptor primitives and the
// fp32-as-bf16-split tables.  Included by the fused expansion kernel and by the dense-operand kernel.
#pragma once
#include "nmg_common.cuh"

namespace nmg {

constexpr int TC_BM = 128;    // output features per CTA (MMA M)
constexpr int TC_BN = 256;    // tokens per CTA (MMA N)
constexpr int TC_BK = 64;     // reduction elements per stage: one 128-byte swizzle span of 16-bit data
constexpr int TC_STAGES = 4;
constexpr int TC_A_BYTES = TC_BM * TC_BK * 2;  // 16 KB
constexpr int TC_B_BYTES = TC_BN * TC_BK * 2;  // 32 KB
constexpr int TC_ACC_COLS = 256;    // one fp32 accumulator tile: 128 lanes x 256 columns

// Tile order: feature tiles are taken in bands of `band_w`; inside a band the CTA index runs over the band's feature
// tiles first, then over token tiles.  The CTAs that are resident together then cover a block of band_w x (CTAs / band_w)
// tiles and share its operand panels through L2; a wave reads band_w weight panels and CTAs / band_w activation
// panels from HBM, which is least when the block is square in bytes: 16 for one-CTA tiles (128 x 256, 148 CTAs), 8 for
// the 256 x 256 tiles of CTA pairs (74 pairs).
constexpr int TC_BAND = 16;
constexpr int TC_BAND_PAIR = 8;
__device__ __forceinline__ void tile_of_cta(int lin, int tiles_f, int tiles_t, int &tf, int &tt, int band_w = TC_BAND) {
    const int per_band = band_w * tiles_t;
    const int band = lin / per_band, within = lin - band * per_band;
    const int width = min(band_w, tiles_f - band * band_w);
    tt = within / width;
    tf = band * band_w + (within - tt * width);
}


// One lane of a converged warp.  The issuing warps run their loops with all lanes and issue under this predicate: their operands
// then stay in uniform registers, which is where the tensor-core instructions want them.  Under `if (lane == 0)` every operand
// is moved over per instruction, and a step of four MMAs took 460 ns whatever its width.
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void tmem_alloc(uint32_t *smem_slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the A operand in TMEM: lane = row, 32-bit column = two neighbouring reduction elements
__device__ __forceinline__ void tc_mma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// The same load without the wait, and the wait as a fence on the destination registers: between the two the load is
// in flight and the registers must not be read; the "+r" operands keep the compiler from moving a use above the wait.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_fence(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                   "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                   "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :: "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {  // completion: tmem_wait_st
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// One 16-byte store to a multicast address: NVSwitch writes it to the same offset on every GPU of the multicast group.
__device__ __forceinline__ void multimem_st_v4(void *mc_addr, uint4 v) {
    asm volatile("multimem.st.weak.global.v4.f32 [%0], {%1, %2, %3, %4};"
                 ::"l"(mc_addr), "f"(__uint_as_float(v.x)), "f"(__uint_as_float(v.y)), "f"(__uint_as_float(v.z)), "f"(__uint_as_float(v.w))
                 : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// ---- CTA pairs (thread-block cluster of 2, tcgen05 cta_group::2) -------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the two halves of the cluster barrier, for a rendezvous that is only waited for later
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// shared::cluster address of `local` (a shared::cta address of this CTA) in the CTA with the given cluster rank
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// Arrive on a barrier of the pair's other CTA (or this one) to say "my reads of the accumulator are done".  The reads are
// tcgen05.ld whose values are already in registers (tcgen05.wait::ld) when this runs, so the signal carries no data and
// needs no release: a release at cluster scope would first wait until every global store this thread has in flight --
// the tile's output -- is acknowledged by L2, once per tile and warp, which is what bounded the drain.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster_bounded(uint64_t *bar, uint32_t parity, int *status, int code) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try_wait_cluster(bar, parity)) return true;
        if (global_timer_ns() - t0 > kWaitLimitNs) break;
    }
    if (status) atomicExch(status, code);
    return false;
}
// 2-D tiled TMA load of a CTA pair, no multicast: the box lands in THIS CTA's shared memory, the bytes are reported to
// the mbarrier at `bar_cluster_addr`, which may live in the peer CTA.
__device__ __forceinline__ void tma_load_2d_pair(void *smem_dst, const CUtensorMap *map, int x, int y, uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr)
        : "memory");
}
// commit of the pair's MMAs: arrives at the barrier at this shared-memory offset in BOTH CTAs
__device__ __forceinline__ void tc2_commit_both(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t *smem_slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc2_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, rows of 128 bytes, 8-row groups 1024 bytes
// apart.  Fields: start address >> 4 (bits 0-13), leading byte offset >> 4 (16-29, unused for swizzled K-major,
// set to 1), stride byte offset >> 4 (32-45), descriptor version 1 (46-47), layout type 2 = SWIZZLE_128B (61-63).
__device__ __forceinline__ uint64_t make_sw128_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
// Instruction descriptor (kind::f16): D = fp32 (bits 4-5 = 1), A / B format (7-9, 10-12: 0 = f16, 1 = bf16), both
// K-major (15, 16 = 0), N >> 3 (17-22), M >> 4 (24-28).
template <typename T> __device__ __forceinline__ uint32_t make_idesc(int n_cols = TC_BN) {
    const uint32_t fmt = sizeof(T) == 2 && DT<T>::id == NMG_BF16 ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(n_cols >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

// Two fp32 values -> two 16-bit values in one word (first in the low half) with one packed conversion.
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<float>(float, float) { return 0; }  // never used: fp32 outputs are stored as words


// Exact (erf) GELU with a short erf: erf(x) = 1 - (a1 t + ... + a5 t^5) exp(-x^2), t = 1 / (1 + p x) for x >= 0 (Abramowitz &
// Stegun 7.1.26, absolute error 1.5e-7, i.e. below fp32 rounding of the result for |v| of order one).  With x = |v| / sqrt(2)
// and v * sign(v) = |v|, gelu(v) = v (1 + erf(v / sqrt 2)) / 2 collapses to max(v, 0) - |v| q(t) 2^(-v^2 log2(e) / 2) where q
// carries the halved coefficients: fifteen instructions, two of them on the special-function unit (flush-to-zero forms, which
// need no range fix-up), against the library erf's thirty.
__device__ __forceinline__ float gelu_erf(float v) {
    const float av = fabsf(fminf(v, 1e30f));  // +inf: the second factor below is 0 then, and the first must not be infinite
    float t, e;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.23164189f, av, 1.f)));   // p / sqrt(2)
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"((v * -0.72134752f) * v));          // log2(e) / 2
    const float q = fmaf(fmaf(fmaf(fmaf(0.5307027145f, t, -0.7265760135f), t, 0.7107068705f), t, -0.142248368f), t, 0.127414796f) * t;
    return fmaf(-(av * q), e, fmaxf(v, 0.f));
}

// Two neighbouring values at a time: the multiplications and additions are packed ones, one instruction for both with the same rounding
// (ten instructions per value where gelu_erf takes fifteen).  The drain warps of the two-pass product take about as long for a tile of
// K = 1024 as its MMAs: feed-forward pair 4096 x 1024 f16, 12288 tokens 200 -> 196.5 us, the same bits.
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ void gelu_erf_pair(uint32_t &ra, uint32_t &rb) {
    const float a = __uint_as_float(ra), b = __uint_as_float(rb);
    auto both = [](float c) { return pack_f32x2(c, c); };
    const uint64_t v = pack_f32x2(a, b), av = pack_f32x2(fabsf(fminf(a, 1e30f)), fabsf(fminf(b, 1e30f)));
    float x, y, ta, tb, ea, eb;
    unpack_f32x2(fma_f32x2(both(0.23164189f), av, both(1.f)), x, y);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ta) : "f"(x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(tb) : "f"(y));
    unpack_f32x2(mul_f32x2(mul_f32x2(v, both(-0.72134752f)), v), x, y);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ea) : "f"(x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(eb) : "f"(y));
    const uint64_t t = pack_f32x2(ta, tb);
    uint64_t q = fma_f32x2(both(-0.5307027145f), t, both(0.7265760135f));  // -q
    q = fma_f32x2(q, t, both(-0.7107068705f));
    q = fma_f32x2(q, t, both(0.142248368f));
    q = mul_f32x2(fma_f32x2(q, t, both(-0.127414796f)), t);
    unpack_f32x2(fma_f32x2(mul_f32x2(av, q), pack_f32x2(ea, eb), pack_f32x2(fmaxf(a, 0.f), fmaxf(b, 0.f))), x, y);
    ra = __float_as_uint(x);
    rb = __float_as_uint(y);
}

// ---- fp32 operands ---------------------------------------------------------------------------------------------------------
// The tensor core's fp32 accumulator truncates instead of rounding, which biases long sums: the relative error grows linearly with the
// number of additions to a sum that has its size already, by 2e-8 each.  fp32 products therefore keep a running sum outside the tensor
// core: after every chunk of k-blocks the partial tile is added to it with round-to-nearest FADDs (fused kernel: a second accumulator
// tile in TMEM, by all twelve warps; two-pass kernel: registers of the drain warps) and the MMAs restart from zero.  The error
// then does not depend on the length.
//
// fp32 operands run as exact sums of three bf16 pieces, x = xh + xm + xl, which have fp32's range: every value keeps its own precision,
// however far it lies below the others of its row.  Of the nine products of pieces six are computed, smallest first; the three left
// out are at most 2^-24 of the product each, the size of an fp32 rounding.
// Two fp16 pieces under one exponent per row take three products (3072 <- 768, 4096 tokens: 62.6 us against 84.1), but they lose
// what lies more than 2^-18 below the largest of its row, and outputs that meet only such values are wrong without a sign of it.
//
// Pieces below bf16's range: a value below 2^-110 loses its last bits.  An activation row that has no value of 2^-80 or more is
// split times 2^40, and its results are multiplied by 2^-40.
constexpr int SPLIT_PLANES = 3, SPLIT_TERMS = 6;
constexpr uint32_t TINY_ROW = (uint32_t)(127 - 80) << 23;  // magnitude bits: rows below are tiny
constexpr float TINY_SCALE = 0x1p40f, TINY_FACTOR = 0x1p-40f;
__device__ __forceinline__ bool not_tiny(float v) { return (__float_as_uint(v) & 0x7fffffffu) >= TINY_ROW; }  // infinities and NaN too
// Two values -> one word of each plane.  The largest magnitudes would round up to infinity: their first piece is the largest finite one.
__device__ __forceinline__ void split3_pair(float a, float b, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
    constexpr float TOP = 0x1.fep127f;
    const __nv_bfloat162 h = __floats2bfloat162_rn(fminf(fmaxf(a, -TOP), TOP), fminf(fmaxf(b, -TOP), TOP));
    const float ra = a - __low2float(h), rb = b - __high2float(h);
    const __nv_bfloat162 m = __floats2bfloat162_rn(ra, rb);
    const __nv_bfloat162 l = __floats2bfloat162_rn(ra - __low2float(m), rb - __high2float(m));
    hi = *reinterpret_cast<const uint32_t *>(&h);
    mid = *reinterpret_cast<const uint32_t *>(&m);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
__device__ __forceinline__ void split3(float f, __nv_bfloat16 (&piece)[3]) {
    uint32_t w[3];
    split3_pair(f, 0.f, w[0], w[1], w[2]);
#pragma unroll
    for (int c = 0; c < 3; c++) piece[c] = __ushort_as_bfloat16((unsigned short)(w[c] & 0xffffu));
}
// Planes of product t, the smallest products first
constexpr int split_w(int t) { return t == 1 ? 2 : t == 2 || t == 4 ? 1 : 0; }
constexpr int split_x(int t) { return t == 0 ? 2 : t == 2 || t == 3 ? 1 : 0; }
template <typename T> struct TcMode { using elem = T; };  // what the tensor cores multiply
template <> struct TcMode<float> { using elem = __nv_bfloat16; };

}  // namespace nmg
