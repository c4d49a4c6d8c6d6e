// ptx.cuh -- inline-PTX wrappers for sm_103a: mbarrier, TMA (cp.async.bulk.tensor), tcgen05
// (TMEM alloc, MMA, commit, load) and the shared-memory / instruction descriptors of tcgen05.mma.
// Written from the PTX ISA descriptions of these instructions.
#pragma once
#include <cuda.h>
#include <cstdint>

namespace tl {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---- mbarrier --------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One lane of a converged warp (elect.sync over the full mask); true in the elected lane only.
__device__ __forceinline__ bool elect_one()
{
    uint32_t elected;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(elected));
    return elected != 0;
}

// Programmatic dependent launch: block until the prerequisite grid has completed and its memory
// operations are visible (returns at once when the launch has no programmatic dependency).
__device__ __forceinline__ void grid_dep_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Allow the dependent grid to be scheduled once every CTA of this grid has issued this (or exited).
__device__ __forceinline__ void grid_dep_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait on the phase with the given parity: true once the phase has completed, false when
// `limit_ns` of %globaltimer time has passed (the caller records the timeout and leaves its loop).
// `bar` is a shared-memory address.  A phase that has completed, or completes while the hardware holds
// the first try_wait, costs one instruction and a predicate; the spin (one PTX block, so an issue loop that
// calls it carries no data-dependent inner loop of its own) is off that path.  Called by one lane it
// costs 36 clocks on a completed phase; by 32 lanes 130.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns)
{
    if (mbar_try_wait(bar, parity)) return true;
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .u64 t0, t1;\n\t"
        "mov.u64 t0, %%globaltimer;\n\t"
        "TL_WAIT_LOOP:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra TL_WAIT_DONE;\n\t"
        "mov.u64 t1, %%globaltimer;\n\t"
        "sub.u64 t1, t1, t0;\n\t"
        "setp.lt.u64 q, t1, %3;\n\t"
        "@q bra TL_WAIT_LOOP;\n\t"
        "TL_WAIT_DONE:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "l"(limit_ns)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns)
{
    return mbar_wait(smem_u32(bar), parity, limit_ns);
}

// Barrier 1 over the N threads of the epilogue warps.
template <int N>
__device__ __forceinline__ void named_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(N) : "memory");
}

// ---- TMA ---------------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tmap(const void* tmap)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}

// 3-D tiled load of one box into shared memory; completion is signalled as transaction bytes on
// `bar`.  The x coordinate times the element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const void* tmap, uint32_t bar, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_dst),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// ---- tcgen05 -------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* slot_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One k-block of D[tmem] (+)= A * B^T: four tcgen05.mma along k, issued by one thread.  A descriptor's
// high word is the same for every tile (sdesc_hi); its low word (sdesc_lo) advances by `a_step` /
// `b_step` (16-byte units) per k step.  `accumulate` 0 starts the accumulator with the first product.
// KIND 0: 16-bit inputs (f16 or bf16 per idesc); 1: E4M3.  CG 2: the pair MMA, issued by the leader CTA:
// A rows and B rows (N) are split between the two CTAs' shared memory at the same offsets; D rows
// 0-127 land in the leader's TMEM, 128-255 in the peer's.
// One block for the four, with the descriptors formed by a single add each: the issuing warp's
// instructions per k-block bound the main loop of tiles narrower than 256 columns (an MMA takes 64
// clocks at 128 columns and 49 at 64; with 64-bit descriptors built from their fields for every
// MMA a k-block took 500 clocks whatever its width).
#define TL_MMA4(GROUP, KINDSTR)                                                                          \
    asm volatile(                                                                                        \
        "{\n\t.reg .pred p, q;\n\t.reg .b32 al, bl;\n\t.reg .b64 ad, bd;\n\t"                                 \
        "setp.ne.b32 p, %5, 0;\n\tsetp.eq.u32 q, 0, 0;\n\t"                                                \
        "mov.b64 ad, {%1, %3};\n\t"                                                                      \
        "mov.b64 bd, {%2, %3};\n\t"                                                                      \
        "tcgen05.mma.cta_group::" GROUP ".kind::" KINDSTR " [%0], ad, bd, %4, p;\n\t"                     \
        "add.u32 al, %1, %6;\n\tadd.u32 bl, %2, %7;\n\t"                                                 \
        "mov.b64 ad, {al, %3};\n\tmov.b64 bd, {bl, %3};\n\t"                                             \
        "tcgen05.mma.cta_group::" GROUP ".kind::" KINDSTR " [%0], ad, bd, %4, q;\n\t"                     \
        "add.u32 al, al, %6;\n\tadd.u32 bl, bl, %7;\n\t"                                                 \
        "mov.b64 ad, {al, %3};\n\tmov.b64 bd, {bl, %3};\n\t"                                             \
        "tcgen05.mma.cta_group::" GROUP ".kind::" KINDSTR " [%0], ad, bd, %4, q;\n\t"                     \
        "add.u32 al, al, %6;\n\tadd.u32 bl, bl, %7;\n\t"                                                 \
        "mov.b64 ad, {al, %3};\n\tmov.b64 bd, {bl, %3};\n\t"                                             \
        "tcgen05.mma.cta_group::" GROUP ".kind::" KINDSTR " [%0], ad, bd, %4, q;\n\t}\n" ::"r"(d_tmem),    \
        "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate), "r"(a_step), "r"(b_step)               \
        : "memory")
template <int KIND, int CG>
__device__ __forceinline__ void mma_kblock(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                           uint32_t accumulate, uint32_t a_step, uint32_t b_step)
{
    if constexpr (KIND == 0 && CG == 1) TL_MMA4("1", "f16");
    else if constexpr (KIND == 0) TL_MMA4("2", "f16");
    else if constexpr (CG == 1) TL_MMA4("1", "f8f6f4");
    else TL_MMA4("2", "f8f6f4");
}
// One of the four (16-bit inputs).
template <int CG>
__device__ __forceinline__ void mma_k16(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                        uint32_t accumulate)
{
#define TL_MMA1(GROUP)                                                                                       \
    asm volatile(                                                                                            \
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\t"                                                        \
        "setp.ne.b32 p, %5, 0;\n\tmov.b64 ad, {%1, %3};\n\tmov.b64 bd, {%2, %3};\n\t"                         \
        "tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], ad, bd, %4, p;\n\t}\n" ::"r"(d_tmem),              \
        "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate)                                            \
        : "memory")
    if constexpr (CG == 1) TL_MMA1("1");
    else TL_MMA1("2");
#undef TL_MMA1
}
#undef TL_MMA4

// Arrive once on `bar` when every tcgen05 operation issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Warp-collective load of 32 consecutive fp32 columns of this warp's 32 TMEM lanes; waits for the
// load to complete inside the same asm statement so the outputs are valid on return.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// The same for 8 or 16 columns, as floats.
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&r)[N])
{
    static_assert(N == 8 || N == 16, "8 or 16 columns");
    if constexpr (N == 16)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
            "tcgen05.wait::ld.sync.aligned;\n"
            : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
              "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
            : "r"(taddr)
            : "memory");
    else
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
            "tcgen05.wait::ld.sync.aligned;\n"
            : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
            : "r"(taddr)
            : "memory");
}

// Shared-memory matrix descriptor for tcgen05.mma with 128-byte swizzling:
//   bits  0-13 start address >> 4, 16-29 leading-dimension byte offset >> 4,
//   bits 32-45 stride-dimension byte offset >> 4, bits 46-48 fixed 0b001,
//   bits 49-51 base offset (0: tiles are 1024-byte aligned), bits 61-63 swizzle mode (2 = 128B).
// K-major tiles: rows of 128 bytes, 8-row groups 1024 bytes apart (SBO); LBO unused.
// MN-major tiles: 128-byte rows along MN, one row per k; 8-k groups SBO apart, 64-element MN
// chunks LBO apart.
// The low word (start address, LBO) and the high word (SBO and the fixed fields) separately: a tile
// address below 256 KB leaves the LBO field alone when a low word is advanced by 16-byte units.
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t saddr, uint32_t lbo_bytes)
{
    return ((saddr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
__device__ __forceinline__ constexpr uint32_t sdesc_hi(uint32_t sbo_bytes)
{
    return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
}

// ---- clusters and the CTA pair (cta_group::2) ----------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_id_x()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t ncluster_x()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
    return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t cta_addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(cta_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on a barrier that may live in another CTA of the cluster.  Release at CTA scope (the default): it
// hands over TMEM (ordered by tcgen05.fence), not memory; at cluster scope it waits for every global
// store and register spill the thread has outstanding (ncu: 8 warps stalled on it per issued
// instruction of the shared-piece kernel).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load into this CTA's shared memory whose completion is signalled on an mbarrier that may live
// in the peer CTA of the pair (cluster address).
__device__ __forceinline__ void tma_load_3d_pair(uint32_t smem_dst, const void* tmap, uint32_t mbar_cluster_addr, int x,
                                                 int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_dst),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(mbar_cluster_addr), "r"(x), "r"(y), "r"(z)
        : "memory");
}
// The same load multicast to the CTAs in `cta_mask` (same shared-memory offset in each); each
// destination's completion is counted on the mbarrier at the given offset in its own pair's leader.
__device__ __forceinline__ void tma_load_3d_pair_mc(uint32_t smem_dst, const void* tmap, uint32_t mbar_cluster_addr,
                                                    uint16_t cta_mask, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.multicast::cluster"
        ".cta_group::2 [%0], [%1, {%4, %5, %6}], [%2], %3;" ::"r"(smem_dst),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(mbar_cluster_addr), "h"(cta_mask), "r"(x), "r"(y), "r"(z)
        : "memory");
}
__device__ __forceinline__ void st_shared_u16(uint32_t addr, uint16_t v)
{
    asm volatile("st.shared.b16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}
__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// 16-byte global -> shared copy without a register round trip (completion per thread, by group)
__device__ __forceinline__ void cp_async16(uint32_t smem_addr, const void* gptr)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr), "l"(gptr) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Collective over one warp in each CTA of the pair.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Arrive once on the mbarrier at this offset in every CTA of `cta_mask` when the pair MMAs issued so
// far by this thread have completed.
__device__ __forceinline__ void mma_commit_pair(uint32_t bar, uint16_t cta_mask)
{
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"(cta_mask)
        : "memory");
}

}  // namespace ptx
}  // namespace tl
