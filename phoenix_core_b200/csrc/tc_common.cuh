// Helpers shared by the TMA-fed tcgen05 kernels: TMA load wrappers, wide stores, the tensor-map encoder
// (fetched from the driver at run time, so the library does not link against libcuda), small host utilities.
#pragma once
#include "sm_share.h"
#include <cstdlib>

#include <cuda.h>

#include "common.cuh"
#include "umma.cuh"

namespace pcb {
extern int g_sm_margin;      // defined in api.cu
namespace tc {

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar) : "memory");
}

// Pairs of SMs (clusters of two CTAs, cta_group::2). One thread of the even CTA issues the MMAs of both; the operands of an MMA lie half in
// each CTA's shared memory at the same offsets, the accumulator rows half in each one's tensor memory.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Cluster address of the location `local_addr` (a shared::cta address of this CTA) in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Relaxed: the arrival orders nothing but the tensor-memory reads before it, which tcgen05.wait::ld and the tcgen05 fences on
// both sides already order; a cluster-scope release here made every arrival wait for the thread's outstanding stores.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA loads of one box into this CTA's shared memory whose bytes are counted by a barrier given by its cluster address
// (the even CTA's `full` barrier). One destination, no multicast.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar_cluster) : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar_cluster) : "memory");
}
__device__ __forceinline__ void tma_load_5d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar_cluster) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t slot_smem_addr, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem_addr), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t tmem_addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_addr), "r"(cols) : "memory");
}
// D[tmem of both CTAs] (+)= A * B for the pair; issued by one thread of the even CTA. Descriptors as two 32-bit words.
__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, {%7, %7, %7, %7, %7, %7, %7, %7}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void mma_tf32_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                              uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], da, db, %5, {%7, %7, %7, %7, %7, %7, %7, %7}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// Arrives on the barrier at the given cluster address once every MMA issued so far for the pair has completed.
__device__ __forceinline__ void mma_commit_pair(uint32_t bar_cluster) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster) : "memory");
}

// Programmatic dependent launch. A kernel launched with launch_chained may start while the kernel in front of it in the stream is
// still running, once every CTA of that one has called chain_next() (or ended); every thread calls chain_wait() before its first access
// to global memory, which returns when the kernel in front has completed and its writes are visible. What comes before that call
// (barriers, tensor memory, the launch itself) then overlaps the tail of the kernel in front: about 1.5 us per launch of a chain of small
// kernels. A kernel calls chain_next() once its own wait is over, so that only its direct successor sits beside it. A persistent kernel
// that takes the whole tensor memory must also ask for more than half of the shared memory (ONE_CTA_SMEM): beside the tail of another
// kernel the SMs become free one by one, and an SM that could hold two of its CTAs could be given two, the second one waiting for the
// first one's tensor memory.
constexpr size_t ONE_CTA_SMEM = 116 * 1024;
// Dynamic shared memory a CTA may have. Kernels whose need varies from call to call are given this limit whatever the call needs: the
// limit is state of the function, and another host thread could lower it between a thread's own setting and its launch.
constexpr int MAX_CTA_SMEM = 227 * 1024;
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Loads of a chained kernel behind chain_wait(): the grid is resident while the kernel in front still writes, so data may not go through the
// non-coherent path (__ldg, or const __restrict__ parameters), which is for data that nobody writes during the life of the grid.
// Not loaded, and zero, where `ok` is false.
__device__ __forceinline__ uint16_t ld_chained(const uint16_t* p, bool ok = true) {
    uint16_t v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u16 %0, 0;\n\t@q ld.global.u16 %0, [%1];\n\t}" : "=h"(v) : "l"(p), "r"((uint32_t)ok));
    return v;
}
__device__ __forceinline__ uint32_t ld_chained(const uint32_t* p, bool ok = true) {
    uint32_t v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u32 %0, 0;\n\t@q ld.global.u32 %0, [%1];\n\t}" : "=r"(v) : "l"(p), "r"((uint32_t)ok));
    return v;
}
__device__ __forceinline__ uint2 ld_chained(const uint2* p, bool ok = true) {
    uint2 v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t@q ld.global.v2.u32 {%0, %1}, [%2];\n\t}"
                 : "=r"(v.x), "=r"(v.y) : "l"(p), "r"((uint32_t)ok));
    return v;
}
__device__ __forceinline__ uint4 ld_chained(const uint4* p, bool ok = true) {
    uint4 v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
                 "@q ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "r"((uint32_t)ok));
    return v;
}
__device__ __forceinline__ float ld_chained(const float* p, bool ok = true) { return __uint_as_float(ld_chained(reinterpret_cast<const uint32_t*>(p), ok)); }
__device__ __forceinline__ float2 ld_chained(const float2* p, bool ok = true) {
    const uint2 v = ld_chained(reinterpret_cast<const uint2*>(p), ok);
    return make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
}
__device__ __forceinline__ float4 ld_chained(const float4* p, bool ok = true) {
    const uint4 v = ld_chained(reinterpret_cast<const uint4*>(p), ok);
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
// `cluster`: CTAs per cluster.
template <typename... Params, typename... Args>
cudaError_t launch_clusters(int cluster, bool chained, void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (chained) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster; attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
cudaError_t launch_chained_if(bool chained, void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, Args... args) {
    return launch_clusters(1, chained, kernel, grid, block, smem, stream, args...);
}
template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, Args... args) {
    return launch_chained_if(true, kernel, grid, block, smem, stream, args...);
}

// Whether a warp may store what the barrier it waits for announces: its own wait succeeds in every lane, and no wait of the call had
// expired when the status word was read, which is done in front of the wait to hide the read. (A wait that expires meanwhile leaves the
// barrier open: whoever gives up no longer signals.)
__device__ __forceinline__ int read_status(const int* status) { return *reinterpret_cast<const volatile int*>(status); }
__device__ __forceinline__ bool warp_may_store(bool ok, int status_before) { return __all_sync(0xffffffffu, ok && status_before == 0); }

// TMA store of one shared-memory box (written by ordinary stores, then fence_proxy_async) to global memory; elements of
// the box that fall outside the tensor are not written. Completion is tracked per thread in bulk groups.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
// Bulk copy of a contiguous shared-memory range to global memory (both 16-byte aligned, size a multiple of 16 bytes).
__device__ __forceinline__ void bulk_store_1d(void* dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Until the bulk stores committed so far by this thread have finished READING shared memory (the buffer may be reused).
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void st_shared_u16(uint32_t addr, uint16_t v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// 32-byte store: one full sector per thread and half as many store instructions as 16-byte stores.
__device__ __forceinline__ void st_global_v8(void* addr, const uint32_t* v) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void red_add_f32x4(float* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// A warp's block of 32 output rows (one per lane: a channel plane of an NCHW tensor) x 32 tile columns, for planes whose image rows
// are not 16-byte aligned. Stored from the registers, an instruction would write 2 to 8 bytes to each of 32 planes (32 sectors);
// through shared memory the lanes of an instruction write neighbouring pixels of 32 / V columns of one or a few planes. On
// 45 x 37 planes, 24 -> 40 channels, the 3x3 forward kernel went from 62 to 35 us with it.
//   packed    the lane's 32 16-bit columns in pairs;   buf: EPI_ROWS_BYTES of shared memory of this warp
//   row_off   element offset of the lane's plane, or -1 for a row that is not stored
//   pix_off   element offset of column (lane % (32 / V)) * V of the block inside a plane, or -1 if it lies outside the image
constexpr int EPI_ROWS_PITCH = 17;                               // words per row: odd, so rows start in different banks
constexpr int EPI_ROWS_BYTES = 32 * EPI_ROWS_PITCH * 4;
template <int V>
__device__ __forceinline__ void store_rows(uint32_t buf, const uint32_t (&packed)[16], uint16_t* out, int row_off, int pix_off, int lane) {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 16; ++e) asm volatile("st.shared.u32 [%0], %1;" ::"r"(buf + (uint32_t)(lane * EPI_ROWS_PITCH + e) * 4u), "r"(packed[e]) : "memory");
    __syncwarp();
    constexpr int LANES = 32 / V;                                // lanes per row
    const int sub = lane / LANES, col = (lane % LANES) * V;
    const uint32_t src = buf + (uint32_t)(sub * EPI_ROWS_PITCH * 4 + col * 2);
#pragma unroll 8
    for (int r = 0; r < 32; r += V) {                            // V rows per instruction
        const int ro = __shfl_sync(0xffffffffu, row_off, r + sub);
        const uint32_t a = src + (uint32_t)(r * EPI_ROWS_PITCH * 4);
        if (V == 1) {
            uint16_t h;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(a) : "memory");
            if (ro >= 0 && pix_off >= 0) out[(size_t)ro + pix_off] = h;
        } else if (V == 2) {
            uint32_t w;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(a) : "memory");
            if (ro >= 0 && pix_off >= 0) *reinterpret_cast<uint32_t*>(out + (size_t)ro + pix_off) = w;
        } else {
            uint2 w;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w.x) : "r"(a) : "memory");
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w.y) : "r"(a + 4) : "memory");
            if (ro >= 0 && pix_off >= 0) *reinterpret_cast<uint2*>(out + (size_t)ro + pix_off) = w;
        }
    }
}

// The same for fp32 results: 32 columns of floats per lane; `reduce`: added to the output instead of stored.
constexpr int EPI_ROWS_F32_PITCH = 33;
constexpr int EPI_ROWS_F32_BYTES = 32 * EPI_ROWS_F32_PITCH * 4;
template <int V>
__device__ __forceinline__ void store_rows_f32(uint32_t buf, const uint32_t (&v)[32], float* out, int row_off, int pix_off, int lane, bool reduce) {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 32; ++e) asm volatile("st.shared.u32 [%0], %1;" ::"r"(buf + (uint32_t)(lane * EPI_ROWS_F32_PITCH + e) * 4u), "r"(v[e]) : "memory");
    __syncwarp();
    constexpr int LANES = 32 / V;
    const int sub = lane / LANES, col = (lane % LANES) * V;
    const uint32_t src = buf + (uint32_t)(sub * EPI_ROWS_F32_PITCH + col) * 4u;
#pragma unroll 8
    for (int r = 0; r < 32; r += V) {
        const int ro = __shfl_sync(0xffffffffu, row_off, r + sub);
        float w[V];
#pragma unroll
        for (int e = 0; e < V; ++e) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(w[e]) : "r"(src + (uint32_t)(r * EPI_ROWS_F32_PITCH + e) * 4u) : "memory");
        if (ro < 0 || pix_off < 0) continue;
        float* dst = out + (size_t)ro + pix_off;
        if (reduce) {
            if (V == 4) red_add_f32x4(dst, w[0], w[V > 1 ? 1 : 0], w[V > 2 ? 2 : 0], w[V > 3 ? 3 : 0]);
            else {
#pragma unroll
                for (int e = 0; e < V; ++e) atomicAdd(dst + e, w[e]);
            }
        } else if (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(w[0], w[V > 1 ? 1 : 0], w[V > 2 ? 2 : 0], w[V > 3 ? 3 : 0]);
        else if (V == 2) *reinterpret_cast<float2*>(dst) = make_float2(w[0], w[V > 1 ? 1 : 0]);
        else *dst = w[0];
    }
}

// The same for tiles of at most 64 rows, where two to four of the eight epilogue warps have any: each of them is bound by the latency of its
// chain of shuffles, reads and stores, not by the stores. (Real-valued 8 -> 8 channels, 70 x 75, batch 105, 1 x 1: 139 us, as above
// 221. With all rows in use the bursts are slower: 8 -> 112 channels, 67 x 67, batch 125, two components, 578 / 453.)
template <int V>
__device__ __forceinline__ void store_rows_f32_few(uint32_t buf, const uint32_t (&v)[32], float* out, int row_off, int pix_off, int lane, bool reduce) {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 32; ++e) asm volatile("st.shared.u32 [%0], %1;" ::"r"(buf + (uint32_t)(lane * EPI_ROWS_F32_PITCH + e) * 4u), "r"(v[e]) : "memory");
    __syncwarp();
    constexpr int LANES = 32 / V;
    const int sub = lane / LANES, col = (lane % LANES) * V;
    const uint32_t src = buf + (uint32_t)(sub * EPI_ROWS_F32_PITCH + col) * 4u;
    // eight instructions' reads in flight before the first of their stores
#pragma unroll 1
    for (int r0 = 0; r0 < 32; r0 += 8 * V) {
        float w[8][V];
        int ro[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = r0 + i * V;
            ro[i] = __shfl_sync(0xffffffffu, row_off, r + sub);
#pragma unroll
            for (int e = 0; e < V; ++e) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(w[i][e]) : "r"(src + (uint32_t)(r * EPI_ROWS_F32_PITCH + e) * 4u));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (ro[i] < 0 || pix_off < 0) continue;
            float* dst = out + (size_t)ro[i] + pix_off;
            if (reduce) {
                if (V == 4) red_add_f32x4(dst, w[i][0], w[i][V > 1 ? 1 : 0], w[i][V > 2 ? 2 : 0], w[i][V > 3 ? 3 : 0]);
                else {
#pragma unroll
                    for (int e = 0; e < V; ++e) atomicAdd(dst + e, w[i][e]);
                }
            } else if (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(w[i][0], w[i][V > 1 ? 1 : 0], w[i][V > 2 ? 2 : 0], w[i][V > 3 ? 3 : 0]);
            else if (V == 2) *reinterpret_cast<float2*>(dst) = make_float2(w[i][0], w[i][V > 1 ? 1 : 0]);
            else *dst = w[i][0];
        }
    }
}

// Adds a warp's block of 32 accumulator rows (one per lane) x COLS columns to an fp32 result whose rows run along the columns. From the
// registers, an instruction would add 16 bytes to each of 32 rows; through shared memory its lanes add to whole runs of 128 (COLS 32) or
// 64 bytes of a few rows, so L2 sees a quarter of the lines per instruction. Whole training passes, from the registers / through shared
// memory, us: 1x1 16-bit 128 -> 128 channels, 14 x 14, batch 32 50.7 / 47.6; 24 -> 24, 57 x 57, batch 16 65.0 / 59.0; fp32 the same 156.5 / 147.3;
// 3x3 32 -> 32, 14 x 14, batch 4 16-bit 53.0 / 49.4, fp32 52.4 / 48.9. The narrow kernels keep their adds from the registers: their rows have
// 16 columns at most, and the detour costs more than it saves (8 -> 8, 56 x 56, batch 4: 37.6 / 40.0).
//   buf     ADD_ROWS_BYTES<COLS> of shared memory of this warp (the operand ring, once every MMA has read it)
//   QUADS   four columns per add (the rows' starts are multiples of four elements), else one
//   place   (row, &sign) -> where this lane's first column of the row goes, or null; called by the whole warp
template <bool B> struct Bool { static constexpr bool value = B; };
template <int COLS> constexpr int ADD_ROWS_BYTES = 32 * (COLS + 1) * 4;
template <int COLS, bool QUADS>
__device__ __forceinline__ int add_rows_column(int lane) { return QUADS ? (lane % (COLS / 4)) * 4 : lane % COLS; }
template <int COLS, bool QUADS, typename Place>
__device__ __forceinline__ void add_rows(uint32_t buf, const uint32_t (&v)[COLS], int lane, Place place) {
    constexpr int V = QUADS ? 4 : 1, LANES = COLS / V, ROWS = 32 / LANES;    // lanes per row, rows per instruction
    __syncwarp();
#pragma unroll
    for (int e = 0; e < COLS; ++e) asm volatile("st.shared.u32 [%0], %1;" ::"r"(buf + (uint32_t)(lane * (COLS + 1) + e) * 4u), "r"(v[e]) : "memory");
    __syncwarp();
    const int sub = lane / LANES;
    const uint32_t src = buf + (uint32_t)(sub * (COLS + 1) + add_rows_column<COLS, QUADS>(lane)) * 4u;
#pragma unroll 4
    for (int r = 0; r < 32; r += ROWS) {
        float sgn = 1.f;
        float* dst = place(r + sub, sgn);
        float w[V];
#pragma unroll
        for (int e = 0; e < V; ++e) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(w[e]) : "r"(src + (uint32_t)(r * (COLS + 1) + e) * 4u) : "memory");
        if (!dst) continue;
        if (V == 4) red_add_f32x4(dst, sgn * w[0], sgn * w[V > 1 ? 1 : 0], sgn * w[V > 2 ? 2 : 0], sgn * w[V > 3 ? 3 : 0]);
        else atomicAdd(dst, sgn * w[0]);
    }
}

// A tile of 16-byte units on its way from pixel-major rows of channels to channel-major rows of pixels (the staging kernels): U units
// per pixel, V pixels per load of a thread. The units' places are permuted inside 128 bytes so that neither side has bank conflicts.
constexpr int STAGE_THREADS = 256, STAGE_UNITS = 1024;
template <int V, int U>
__device__ __forceinline__ int stage_unit(int px, int g) {
    constexpr int LINE = 8 / U > V ? 8 / U : V;                    // pixels that share a permutation
    return (px * U + g) ^ ((px / LINE) & 7);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// Encodes a tiled tensor map with zero out-of-bounds fill; returns a pcb_status.
inline int make_tensor_map(CUtensorMap* map, CUtensorMapDataType dt, const void* ptr, int rank, const cuuint64_t* dims,
                           const cuuint64_t* strides_bytes, const cuuint32_t* box, const cuuint32_t* elem_strides,
                           CUtensorMapSwizzle swizzle, const char* what) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) { set_error("cuTensorMapEncodeTiled is not available from the driver"); return PCB_ERR_CUDA; }
    const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    const CUresult r = fn(map, dt, (cuuint32_t)rank, const_cast<void*>(ptr), dims, strides_bytes, box, elem_strides ? elem_strides : ones,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (%s) failed with code %d", what, (int)r); return PCB_ERR_CUDA; }
    return PCB_OK;
}

// SMs the persistent kernels size their grids for: the device's count minus the margin set through pcb_set_sm_margin (SMs left
// free so that another kernel, e.g. a collective's, can run beside them).
inline int device_sms() {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
            sms = 148;
    }
    return sms;
}
inline int sm_count() { return sms_beside(device_sms(), pcb::g_sm_margin); }
inline int sm_pairs() { return pairs_beside(device_sms(), pcb::g_sm_margin); }

// Whether a main kernel is chained to a prologue of that many CTAs: only behind a short one. Behind a longer prologue the gap does not
// matter, and the main kernel, started CTA by CTA beside the last wave, can be the slower for it. Chained / not, us: fp32 3x3, 128
// channels, 28 x 28, batch 128, forward 2196 / 2087; fp16 3x3 of the same size, filter gradient 482 / 446; the 7x7/2 stem, 224 x 224, batch 128,
// forward 350 / 245 (but 3x3 64 -> 64, 56 x 56, batch 64 228 / 228). Behind short ones: 3x3 64 -> 64, 56 x 56, batch 8, forward 40.9 / 43.3, 3x3
// 16 -> 16, 45 x 37, batch 32 26.8 / 29.0, 32 x 32, batch 16, forward 12.8 / 14.8, both gradients 31.4 / 37.3.
inline bool chain_behind(unsigned prologue_blocks, unsigned per_sm) { return prologue_blocks <= per_sm * (unsigned)sm_count(); }

// Whether a kernel of row tiles of 128 takes them two at a time on pairs of SMs (clusters of two): only where an SM has some 64 MMAs of
// 256 columns (8192 clocks) to issue. A cluster launch starts later than a plain one, which shallow layers pay for; the halved operand traffic is what it
// buys. No count of MMAs divides the two exactly. Forward, fp16, (MMAs per SM) single / pairs, us: 1x1, 256 -> 128, 14 x 14, batch 20 (27) 17.4 / 18.6; 64 -> 64,
// 30 x 30, batch 48 (37) 24.7 / 25.0; 3x3 stride 2, 48 -> 64, 40 x 40, batch 12 (37) 22.9 / 23.5; above the line 3x3, 512 -> 128, 7 x 7, batch 16 (95) 106.9 / 86.2;
// 48 -> 64, 45 x 37, batch 9 (114) 38.5 / 35.7; 24 -> 40, 45 x 37, batch 24 (152) 42.6 / 39.3. Misplaced by it: 3x3, 24 -> 40, 45 x 37, batch 10 (63) 25.6 / 25.0; 128 -> 128,
// 7 x 7, batch 30 (45) 39.0 / 34.7; 5x5, 20 -> 64, 37 x 41, batch 8 (128) 38.3 / 39.1; channels-last 3x3, 128 -> 128, 14 x 14, batch 24 (143) 37.1 / 38.4. Filter
// gradients, with the other passes: 3x3, 24 -> 40, 45 x 37, batch 24 123.9 / 120.0; 512 -> 128, 7 x 7, batch 16 191.0 / 192.8.
inline bool worth_pairs(double mmas) { return mmas >= 64.0 * sm_count(); }

inline int round_up(int v, int m) { return (v + m - 1) / m * m; }
// Number of slices to cut each of `items` work items of `steps` steps into when every CTA occupies a whole SM: as few clocks as possible
// over one to three rounds of the machine. Every round costs its CTAs' steps and their fixed part (tensor-memory allocation, pipeline
// fill, the adds of the accumulators: 8 us a round, which is some 24 steps of 64 pixels of the 16-bit kernels and 16 of 32 pixels of
// the fp32 one). 24 -> 88 channels, 3x3, 27 x 27, batch 5, 27 items of 60 steps: 66.6 us in one round of 5 slices, 83.5 in three
// of 16, which fill the machine 6 % better. A CTA takes at least two steps: the adds of twice as many accumulators cost more than the
// second step (56 -> 56 channels, 1 x 1, 30 x 30, batch 5: 35.1 us, one step each 44.4).
inline int split_count(int items, int sms, int steps, int fixed) {
    int best = 1;
    long long best_cost = -1;
    for (int splits = 1; splits <= (steps + 1) / 2 && (splits == 1 || (long long)splits * items <= 3LL * sms); ++splits) {
        const int per = (steps + splits - 1) / splits;
        const long long rounds = ((long long)items * splits + sms - 1) / sms, cost = rounds * (per + fixed);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = splits; }
    }
    return best;
}
inline int grid_cap(size_t work_items, int per_block, int blocks_per_sm) {
    const size_t want = (work_items + per_block - 1) / per_block, cap = (size_t)sm_count() * blocks_per_sm;
    return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

}  // namespace tc
}  // namespace pcb
