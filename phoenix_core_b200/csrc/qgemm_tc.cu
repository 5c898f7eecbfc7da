// Quaternion matrix products on the tensor cores straight from the caller's tensors: dense layers (forward, backward-data and
// filter gradient, any feature counts, fp16 / bf16 / fp32).
//
// One output tile of the product is 128 rows of one operand (A) by NT columns of the other (B) for all four output
// components: D[m][(c, n)] = sum over (kc, k) of A[kc][m][k] * s(kc, c) B[c ^ kc][n][k]. A is multiplied as it lies in memory;
// the signed / permuted quaternion block is expanded on B alone while its tile is written to shared memory: component
// c ^ kc of B, with its sign, goes to block c of the stage (kc, k chunk). So a stage is ONE real product 128 x (4 NT) x 64 and the
// expanded 4 x 4 block never exists in global memory. Roles:
//     forward        m = output feature, n = batch row, k = input feature:   A[kc] = w_kc,  B = x,  s = s(c ^ kc, c)
//     backward-data  m = input feature,  n = batch row, k = output feature:  A[kc] = w_kc,  B = dy, s = s(c, c ^ kc)
//     filter grad.   m = output feature, n = input feature, k = batch row:   A[kc] = dy_kc, B = x,  s = s(c ^ kc, kc)
// The rows m are contiguous in the output of every pass, so the 32 lanes of an epilogue warp store 32 consecutive elements.
// (replaces the 16 GEMM calls and accumulate passes of the reference, src/dense.hpp:21-379, src/backend/cudnn/dense.hpp:20-218.)
//
// Three groups of four warps load (plain loads: feature counts need no alignment, which a tensor map would ask for), expand and store
// the operands in the tcgen05 layouts, each group its own stages;
// one thread of a thirteenth warp issues the MMAs. fp32 operands are split into hi + lo TF32 numbers on their way
// (three MMAs per product). The reduced dimension of a tile is cut over the CTAs of a cluster, which add
// their partial tiles through distributed shared memory in a fixed order (results do not depend on timing, nothing is zeroed or
// cast in a second pass). What bounds a dense layer of a few hundred features is the latency of this chain (load, expand, MMA,
// exchange, store), not bandwidth: hence one kernel per call (its first CTA resets the call's status word), no staging
// kernels, and a cluster split that fills the machine.
// All mbarrier waits are bounded.
#include <atomic>

#include "tc_common.cuh"
#include "tensor_path.cuh"
#include "unaligned_chunk.h"

namespace pcb {
namespace {

using namespace umma;
using namespace tc;

constexpr int QM = 128;                               // rows of a tile
constexpr int Q_GROUP = 128, Q_GROUPS = 3;             // loader threads: groups that fill stages in turn
constexpr int Q_LOADERS = Q_GROUP * Q_GROUPS, Q_THREADS = Q_LOADERS + 32;
constexpr int Q_MAX_STAGES = 6;
constexpr int Q_ROW_BYTES = 128;                      // bytes of one K row of an operand tile: 64 16-bit or 32 fp32 elements
constexpr int ST_Q_LOADER = 0x1000, ST_Q_MMA = 0x2000, ST_Q_EPILOGUE = 0x4000;
// MMAs that may be added into one fp32 accumulator of the fp32 path (each truncates when it adds: conv_tf32.cu), and how many
// accumulators there are. 8 stages of 12 MMAs in each of 4 accumulators.
constexpr int Q_F32_STAGES_PER_ACC = 8, Q_F32_ACCS = 4;

// One operand: element (component, u, v) lies at component * cs + u + v * ld, u being the contiguous index.
struct QOperand {
    const void* p;
    int cs, ld;
    int nu, nv;          // extents of u and v
    int chunk;           // bytes per load: the largest of 16, 8, 4 that divides every row start; 2: unaligned chunks of 16
};
struct QProblem {
    QOperand a, b;
    void* out;
    const void* bias;    // [4][M] or null
    int M, N, K;
    int o_c, o_n;        // output element (c, n, m) at c * o_c + n * o_n + m
    int tiles_m, tiles_n;
    int stages;          // of a tile: four (one per component of A) for every K chunk of 64 (fp32: 32) elements
    int split;           // CTAs that share a tile, neighbours in a cluster: slices of the stages
    uint32_t neg;        // bit 4 * kc + c: component c ^ kc of B enters block c negated
};
struct QParams {
    QProblem prob[2];
    int first_blocks;    // CTAs of prob[0]; the rest work on prob[1]
    int cluster;         // CTAs of a cluster (the larger of the two splits)
    int fmt;             // 0 = fp16, 1 = bf16, 2 = fp32 as TF32
    int* clear;          // the call's status word, if this launch is to reset it
};

__device__ __forceinline__ uint32_t q_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void q_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t local_addr, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t local_addr, uint32_t rank) { return __float_as_uint(ld_cluster_f32(local_addr, rank)); }
__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

// ---- operand tiles ----------------------------------------------------------------------------------------------------------
// ROWS (m or n) x 128 bytes of K (64 16-bit or 32 fp32 elements), moved by the 128 threads of a loader group in chunks of CB = 16, 8 or 4 bytes.
//   KMAJ: u = k. Chunk i of thread t: row t / PER + i * STEP, byte (t % PER) * CB of that row's 128.
//   else: u = m or n, v = k. Chunk i: k row t / PER + i * STEP, byte (t % PER) * CB of the ROWS elements.
template <bool F32, bool KMAJ, int ROWS, int CB>
struct QChunks {
    static constexpr int EB = F32 ? 4 : 2;
    static constexpr int PER = (KMAJ ? Q_ROW_BYTES : ROWS * EB) / CB, STEP = Q_GROUP / PER;
    static constexpr int COUNT = ROWS * Q_ROW_BYTES / CB / Q_GROUP;
    static_assert(Q_GROUP % PER == 0 && COUNT >= 1, "chunks");
};
template <bool F32, bool KMAJ, int ROWS, int CB>
__device__ __forceinline__ void load_chunks(uint32_t (&r)[ROWS / 4], const QOperand& o, int comp, int row0, int k0, int t) {
    typedef QChunks<F32, KMAJ, ROWS, CB> C;
    const int u = (KMAJ ? k0 : row0) + (t % C::PER) * (CB / C::EB), v0 = (KMAJ ? row0 : k0) + t / C::PER;
    const bool u_ok = u < o.nu;
    const char* src = static_cast<const char*>(o.p) + ((size_t)comp * o.cs + (size_t)v0 * o.ld + u) * C::EB;
    const size_t step = (size_t)C::STEP * o.ld * C::EB;
#pragma unroll
    for (int i = 0; i < C::COUNT; ++i) {
        const bool ok = u_ok && v0 + i * C::STEP < o.nv;
        const char* q = src + i * step;
        if (CB == 16) {
            const uint4 w = ld_chained(reinterpret_cast<const uint4*>(q), ok);
            r[4 * i] = w.x; r[4 * i + 1] = w.y; r[4 * i + 2] = w.z; r[4 * i + 3] = w.w;
        } else if (CB == 8) {
            const uint2 w = ld_chained(reinterpret_cast<const uint2*>(q), ok);
            r[2 * i] = w.x; r[2 * i + 1] = w.y;
        } else {
            r[i] = ld_chained(reinterpret_cast<const uint32_t*>(q), ok);
        }
    }
}
__device__ __forceinline__ uint32_t tf32_hi(uint32_t x) { return x & 0xFFFFE000u; }
__device__ __forceinline__ uint32_t tf32_lo(uint32_t x) { return __float_as_uint(__uint_as_float(x) - __uint_as_float(x & 0xFFFFE000u)); }
// Writes the chunks to rows row_base .. of an operand tile, every element's sign flipped by `flip`; fp32: hi parts to `tile`, lo
// parts to `tile` + lo_ofs.
template <bool F32, bool KMAJ, int ROWS, int CB>
__device__ __forceinline__ void store_chunks(const uint32_t (&r)[ROWS / 4], uint32_t tile, uint32_t lo_ofs, int row_base, uint32_t flip, int t) {
    typedef QChunks<F32, KMAJ, ROWS, CB> C;
    const int ub = (t % C::PER) * CB, v0 = t / C::PER;
#pragma unroll
    for (int i = 0; i < C::COUNT; ++i) {
        const int v = v0 + i * C::STEP;
        uint32_t dst;
        if (KMAJ) {
            const int row = row_base + v;
            dst = tile + (uint32_t)row * Q_ROW_BYTES + (uint32_t)(((ub >> 4) ^ (row & 7)) << 4) + (uint32_t)(ub & 15);
        } else {
            // blocks of 128 bytes of rows, K rows of 128 bytes inside; 16-byte units swizzled over 8 K rows (16-bit elements),
            // 32-byte units over 4 K rows (fp32)
            const int b = row_base * C::EB + ub, in = b & 127;
            dst = tile + (uint32_t)(b >> 7) * (F32 ? 32 : 64) * Q_ROW_BYTES + (uint32_t)v * Q_ROW_BYTES +
                  (F32 ? (uint32_t)(((in >> 5) ^ (v & 3)) << 5) + (uint32_t)(in & 31) : (uint32_t)(((in >> 4) ^ (v & 7)) << 4) + (uint32_t)(in & 15));
        }
        uint32_t w[4], lo[4];
        constexpr int W = CB / 4;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            w[j] = r[W * i + j] ^ flip;
            if (F32) { lo[j] = tf32_lo(w[j]); w[j] = tf32_hi(w[j]); }
        }
        if (CB == 16) { st_shared_v4(dst, w[0], w[1], w[2], w[3]); if (F32) st_shared_v4(dst + lo_ofs, lo[0], lo[1], lo[2], lo[3]); }
        else if (CB == 8) { st_shared_v2(dst, w[0], w[1]); if (F32) st_shared_v2(dst + lo_ofs, lo[0], lo[1]); }
        else { st_shared_u32(dst, w[0]); if (F32) st_shared_u32(dst + lo_ofs, lo[0]); }
    }
}
// 16-bit rows that start at any element, in 16-byte chunks: the aligned 8-byte vectors that hold a chunk are loaded and shifted into
// place, elements past the row end are cleared. The tensor, four components, is a whole number of such vectors, so one that holds
// an element never reaches past its end. Against element loads (eight load and eight store instructions per chunk instead of
// three and one): 974 x 608 -> 431, fp16, forward + backward 231 -> 174 us. (With 4-byte aligned rows the plain 4-byte form is
// faster, 31 against 37 us for 128 -> 250 at batch 128, and so it is for fp32.)
template <bool KMAJ, int ROWS>
__device__ __forceinline__ void load_unaligned(uint32_t (&r)[ROWS / 4], const QOperand& o, int comp, int row0, int k0, int t) {
    typedef QChunks<false, KMAJ, ROWS, 16> C;
    const int u = (KMAJ ? k0 : row0) + (t % C::PER) * 8, v0 = (KMAJ ? row0 : k0) + t / C::PER;
    const int left = o.nu - u, total = 4 * o.cs;                       // valid elements of the chunk; elements of the tensor
    uint32_t mask[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) mask[j] = (2 * j < left ? 0xffffu : 0u) | (2 * j + 1 < left ? 0xffff0000u : 0u);
    const unsigned at0 = (unsigned)comp * o.cs + (unsigned)v0 * o.ld + u;  // (unsigned: rows past the last one may leave the 32-bit range)
#pragma unroll
    for (int i = 0; i < C::COUNT; ++i) {
        const bool ok = left > 0 && v0 + i * C::STEP < o.nv;
        const int at = (int)(at0 + (unsigned)(i * C::STEP) * o.ld), al = at & ~3, sh = at & 3;
        const int vectors = ok ? chunk_vectors(at, total) : 0;
        const uint2* q = reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(o.p) + al);
        const uint2 a = ld_chained(q, vectors > 0), b = ld_chained(q + 1, vectors > 1), c = ld_chained(q + 2, vectors > 2);
        uint32_t w[6] = {a.x, a.y, b.x, b.y, c.x, c.y};
#pragma unroll
        for (int j = 0; j < 5; ++j) w[j] = (sh & 2) ? w[j + 1] : w[j];
        const uint32_t sel = (sh & 1) ? 0x5432u : 0x3210u;
#pragma unroll
        for (int j = 0; j < 4; ++j) r[4 * i + j] = __byte_perm(w[j], w[j + 1], sel) & mask[j];
    }
}
template <bool F32, bool KMAJ, int ROWS>
__device__ __forceinline__ void load_tile(uint32_t (&r)[ROWS / 4], const QOperand& o, int comp, int row0, int k0, int t) {
    if (o.chunk == 16) load_chunks<F32, KMAJ, ROWS, 16>(r, o, comp, row0, k0, t);
    else if (o.chunk == 8) load_chunks<F32, KMAJ, ROWS, 8>(r, o, comp, row0, k0, t);
    else if (F32 || o.chunk == 4) load_chunks<F32, KMAJ, ROWS, 4>(r, o, comp, row0, k0, t);
    else load_unaligned<KMAJ, ROWS>(r, o, comp, row0, k0, t);
}
template <bool F32, bool KMAJ, int ROWS>
__device__ __forceinline__ void store_tile(const uint32_t (&r)[ROWS / 4], const QOperand& o, uint32_t tile, uint32_t lo_ofs, int row_base, uint32_t flip, int t) {
    if (o.chunk == 8) store_chunks<F32, KMAJ, ROWS, 8>(r, tile, lo_ofs, row_base, flip, t);
    else if (o.chunk == 4) store_chunks<F32, KMAJ, ROWS, 4>(r, tile, lo_ofs, row_base, flip, t);
    else store_chunks<F32, KMAJ, ROWS, 16>(r, tile, lo_ofs, row_base, flip, t);
}
// fp32 operand with its rows contiguous along m or n: blocks of 32 rows `block_bytes` apart, groups of 4 K rows 512 bytes apart.
__device__ __forceinline__ uint64_t make_desc_mn_f32(uint32_t addr, uint32_t block_bytes) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((block_bytes >> 4) & 0x3FFFu) << 16) | ((uint64_t)(512u >> 4) << 32) |
           DESC_VERSION_SM100 | (1ull << 61);
}

template <bool F32, int NT>
struct QLayout {
    static constexpr int N = 4 * NT;
    static constexpr uint32_t A_TILE = QM * Q_ROW_BYTES, B_TILE = N * Q_ROW_BYTES;
    static constexpr uint32_t STAGE = (A_TILE + B_TILE) * (F32 ? 2 : 1);
    static constexpr int STAGES_FIT = (int)((216 * 1024) / STAGE);
    static constexpr int STAGES = STAGES_FIT < Q_MAX_STAGES ? STAGES_FIT : Q_MAX_STAGES;
    static constexpr int ACCS = F32 ? Q_F32_ACCS : 2;                 // accumulators of N columns, used in turn
    static constexpr uint32_t PARTIAL = (uint32_t)N * QM * 4;         // the exchanged partial tile, in the stages' memory
    static constexpr uint32_t BODY = STAGES * STAGE > PARTIAL ? STAGES * STAGE : PARTIAL;
    static constexpr size_t SMEM = 1024 + BODY + 256;
    static_assert(ACCS * N <= 512, "tensor memory");
};

__device__ __forceinline__ void q_store(void* out, size_t at, float v, int fmt) {
    if (fmt == 2) static_cast<float*>(out)[at] = v;
    else if (fmt == 0) static_cast<__half*>(out)[at] = __float2half_rn(v);
    else static_cast<__nv_bfloat16*>(out)[at] = __float2bfloat16_rn(v);
}
__device__ __forceinline__ float q_bias(const void* bias, size_t at, int fmt) {
    if (fmt == 2) return ld_chained(static_cast<const float*>(bias) + at);
    const uint16_t raw = ld_chained(static_cast<const uint16_t*>(bias) + at);
    return fmt == 0 ? __half2float(__ushort_as_half(raw)) : __bfloat162float(__ushort_as_bfloat16(raw));
}

template <bool F32, int NT, bool AK, bool BK>
__device__ __forceinline__ void q_tile(const QProblem& p, int block, int cluster, int fmt, uint32_t tmem_base, uint32_t tiles, uint32_t full_bar,
                                       uint32_t empty_bar, uint32_t done_bar, int* status) {
    typedef QLayout<F32, NT> L;
    constexpr int KC = F32 ? 32 : 64;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int split = p.split, tile = block / split, rank = block - tile * split;
    const int m0 = (tile % p.tiles_m) * QM, n0 = (tile / p.tiles_m) * NT;
    const int per = (p.stages + split - 1) / split;
    const int s_beg = min(p.stages, rank * per), s_end = min(p.stages, s_beg + per);
    // stage s: chunk s / 4, component s % 4 of A. (The grid is padded to whole clusters: CTAs past the last tile do nothing.)
    const int n_stages = tile < p.tiles_m * p.tiles_n ? s_end - s_beg : 0;

    bool ok = true;
    if (t < Q_LOADERS) {
        // ------------------------------------------------------------------------------------------ loaders
        // group g fills stages g, g + Q_GROUPS, ...: while one group waits for its loads the others write theirs
        const int tg = t % Q_GROUP;
        constexpr int HALF = NT == 32 ? 4 : 2;                     // components of B in registers at a time
        for (int st = t / Q_GROUP; st < n_stages && ok; st += Q_GROUPS) {
            const int kc = (s_beg + st) & 3, k0 = ((s_beg + st) >> 2) * KC, s = st % L::STAGES;
            uint32_t ra[QM / 4], rb[HALF][NT / 4];
            load_tile<F32, AK, QM>(ra, p.a, kc, m0, k0, tg);
#pragma unroll
            for (int c = 0; c < HALF; ++c) load_tile<F32, BK, NT>(rb[c], p.b, c ^ kc, n0, k0, tg);
            ok = mbar_wait_bounded(empty_bar + 8 * s, (st / L::STAGES + 1) & 1, status, ST_Q_LOADER);
            if (ok) {
                const uint32_t a_tile = tiles + s * L::STAGE, b_tile = a_tile + L::A_TILE * (F32 ? 2 : 1);
                constexpr uint32_t SIGN = F32 ? 0x80000000u : 0x80008000u;
                const uint32_t neg = p.neg >> (4 * kc);
                store_tile<F32, AK, QM>(ra, p.a, a_tile, L::A_TILE, 0, 0u, tg);
#pragma unroll
                for (int h = 0; h < 4; h += HALF) {
                    if (h > 0) {
#pragma unroll
                        for (int c = 0; c < HALF; ++c) load_tile<F32, BK, NT>(rb[c], p.b, (h + c) ^ kc, n0, k0, tg);
                    }
#pragma unroll
                    for (int c = 0; c < HALF; ++c)
                        store_tile<F32, BK, NT>(rb[c], p.b, b_tile, L::B_TILE, (h + c) * NT, ((neg >> (h + c)) & 1u) ? SIGN : 0u, tg);
                }
                fence_proxy_async_smem();
            }
            ok = __all_sync(0xffffffffu, ok);
            if (ok && lane == 0) mbar_arrive(full_bar + 8 * s);    // (not after an expired wait: the MMA thread's own wait then runs out)
        }
    } else if (n_stages > 0) {
        // ------------------------------------------------------------------------------------------ MMA issuer
        const uint32_t idesc = make_idesc_f16(F32 ? 2 : fmt, QM, L::N, !AK, !BK);
        constexpr uint32_t KROWS = F32 ? 32 : 64, KSTEP = F32 ? 8 : 16;          // K rows of a stage, K of one MMA
        constexpr uint32_t AS = (AK ? 32 : KSTEP * Q_ROW_BYTES) >> 4, BS = (BK ? 32 : KSTEP * Q_ROW_BYTES) >> 4;
        auto desc = [](uint32_t addr, bool kmajor) {
            return kmajor ? make_desc_kmajor(addr) : (F32 ? make_desc_mn_f32(addr, KROWS * Q_ROW_BYTES) : make_desc_mnmajor(addr, KROWS * Q_ROW_BYTES));
        };
        const bool el = elect_one();
        int s = 0, phase = 0;
        for (int st = 0; st < n_stages; ++st) {
            if (!warp_wait_bounded(full_bar + 8 * s, phase, status, ST_Q_MMA)) break;
            tc_fence_after_sync();
            if (el) {
                const uint32_t a_tile = tiles + s * L::STAGE, b_tile = a_tile + L::A_TILE * (F32 ? 2 : 1);
                const uint64_t ah = desc(a_tile, AK), bh = desc(b_tile, BK);
                if (F32) {
                    // stage st adds into accumulator st mod 4; small terms first
                    const uint32_t d = tmem_base + (uint32_t)((st % L::ACCS) * L::N);
                    const uint64_t al = desc(a_tile + L::A_TILE, AK), bl = desc(b_tile + L::B_TILE, BK);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        mma_tf32_ss(d, al + AS * j, bh + BS * j, idesc, (st >= L::ACCS || j > 0) ? 1u : 0u);
                        mma_tf32_ss(d, ah + AS * j, bl + BS * j, idesc, 1u);
                        mma_tf32_ss(d, ah + AS * j, bh + BS * j, idesc, 1u);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)                            // two accumulators in turn
                        mma_f16_ss(tmem_base + (uint32_t)((j & 1) * L::N), ah + AS * j, bh + BS * j, idesc, (st > 0 || j > 1) ? 1u : 0u);
                }
                mma_commit(empty_bar + 8 * s);
                if (st == n_stages - 1) mma_commit(done_bar);
            }
            if (++s == L::STAGES) { s = 0; phase ^= 1; }
        }
    }
    __syncwarp();

    // ---------------------------------------------------------------------------------------------- epilogue
    const int q = warp & 3, half = warp >> 2;                          // TMEM lane quadrant, half of the columns (warps 0 .. 7)
    if (warp < 8) {
        if (n_stages > 0) ok = mbar_wait_bounded(done_bar, 0, status, ST_Q_EPILOGUE) && ok;
        const int seen = read_status(status);                          // the CTA's own word, in shared memory: asked after the wait
        ok = warp_may_store(ok, seen);
        tc_fence_after_sync();
        const int row = q * 32 + lane, m = m0 + row;
#pragma unroll 1
        for (int cb = 0; cb < L::N / 2; cb += 32) {
            const int col0 = half * (L::N / 2) + cb;
            float sum[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) sum[e] = 0.f;
            if (ok && n_stages > 0) {
#pragma unroll
                for (int acc = 0; acc < L::ACCS; ++acc) {
                    if (F32 && acc >= n_stages) break;                 // fewer stages than accumulators
                    uint32_t v[32];
                    tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * L::N) + col0, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) sum[e] += __uint_as_float(v[e]);
                }
            }
            if (split > 1) {
                // the stages are drained (every MMA has completed), their memory takes the partial tile [column][row]
#pragma unroll
                for (int e = 0; e < 32; ++e) st_shared_u32(tiles + (uint32_t)((col0 + e) * QM + row) * 4u, __float_as_uint(sum[e]));
            } else if (ok && m < p.M) {
                const int c = col0 / NT, nb = n0 + col0 - c * NT;      // 32 columns lie in one component
                const float badd = p.bias ? q_bias(p.bias, (size_t)c * p.M + m, fmt) : 0.f;
#pragma unroll
                for (int e = 0; e < 32; ++e)
                    if (nb + e < p.N) q_store(p.out, (size_t)c * p.o_c + (size_t)(nb + e) * p.o_n + m, sum[e] + badd, fmt);
            }
        }
        tc_fence_before_sync();
    }
    if (cluster > 1) {
        q_cluster_sync();
        if (split > 1 && t < Q_LOADERS) {
            // every CTA of the tile finishes N / split columns: the partial tiles are added in rank order, four columns at a time
            // so that their reads from the other SMs overlap
            const int row = t % QM, m = m0 + row, cols = L::N / split, col_beg = rank * cols;
            const uint32_t peer0 = q_cluster_rank() - (uint32_t)rank;
            bool good = true;                                          // no CTA of the tile has given up a wait
            for (int r = 0; r < split; ++r) good = good && ld_cluster_u32(smem_u32(status), peer0 + r) == 0u;
            constexpr int BATCH = 4;
            if (good && m < p.M) {
                for (int col = col_beg + (t / QM) * BATCH; col < col_beg + cols; col += Q_GROUPS * BATCH) {
                    float v[BATCH][8];
#pragma unroll
                    for (int e = 0; e < BATCH; ++e)
#pragma unroll
                        for (int r = 0; r < 8; ++r)
                            v[e][r] = r < split ? ld_cluster_f32(tiles + (uint32_t)((col + e) * QM + row) * 4u, peer0 + r) : 0.f;
                    const int c = col / NT;                            // cols and NT are multiples of BATCH: one component
                    const float badd = p.bias ? q_bias(p.bias, (size_t)c * p.M + m, fmt) : 0.f;
#pragma unroll
                    for (int e = 0; e < BATCH; ++e) {
                        const int n = n0 + col + e - c * NT;
                        float sum = badd;
#pragma unroll
                        for (int r = 0; r < 8; ++r) sum += v[e][r];
                        if (n < p.N) q_store(p.out, (size_t)c * p.o_c + (size_t)n * p.o_n + m, sum, fmt);
                    }
                }
            }
        }
        q_cluster_sync();                                              // nobody leaves while its partial tile is still read
    }
}

// PAIR: prob[0] has layouts (AK, BK), prob[1] (AK1, BK1) -- both gradients of a dense layer in one launch.
// The status word: every CTA keeps its own in shared memory (its waits look at no other; an epilogue asks those of all CTAs of its tile, so tiles of
// other clusters are stored after an expired wait), and ORs it into the call's word when it ends. The
// first CTA resets that word when it starts (p.clear), instead of a launch in front of this one, which cost 2 to 3 us of a call: a CTA
// has something to OR only after a wait of 2^31 clocks has run out, a second behind the start of its wave, and the first CTA is of the
// first wave.
template <bool F32, int NT, bool AK, bool BK, bool PAIR, bool AK1, bool BK1>
__global__ void __launch_bounds__(Q_THREADS, 1) qgemm_tc_kernel(const __grid_constant__ QParams p, int* __restrict__ status) {
    typedef QLayout<F32, NT> L;
    extern __shared__ uint8_t smem_raw[];
    const int t = threadIdx.x, warp = t >> 5;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + L::BODY);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * Q_MAX_STAGES + 1);
    int* own_status = reinterpret_cast<int*>(tmem_slot + 1);
    const uint32_t full_bar = smem_u32(bars), empty_bar = smem_u32(bars + Q_MAX_STAGES), done_bar = smem_u32(bars + 2 * Q_MAX_STAGES);
    if (t == 0) {
        *own_status = 0;
        for (int s = 0; s < L::STAGES; ++s) { mbar_init(full_bar + 8 * s, Q_GROUP / 32); mbar_init(empty_bar + 8 * s, 1); }
        mbar_init(done_bar, 1);
        fence_barrier_init();
    }
    if (warp == Q_LOADERS / 32) tmem_alloc(smem_u32(tmem_slot), L::ACCS * L::N);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    chain_wait();
    chain_next();
    const int block = blockIdx.x;
    if (block == 0 && t == 0 && p.clear) *p.clear = 0;
    if (!PAIR || block < p.first_blocks)
        q_tile<F32, NT, AK, BK>(p.prob[0], block, p.cluster, p.fmt, tmem_base, smem_u32(base), full_bar, empty_bar, done_bar, own_status);
    else
        q_tile<F32, NT, AK1, BK1>(p.prob[1], block - p.first_blocks, p.cluster, p.fmt, tmem_base, smem_u32(base), full_bar, empty_bar, done_bar, own_status);
    tc_fence_before_sync();
    __syncthreads();
    if (t == 0 && *own_status != 0) atomicOr(status, *own_status);
    if (warp == Q_LOADERS / 32) tmem_dealloc(tmem_base, L::ACCS * L::N);
}

template <bool F32, int NT, bool AK, bool BK, bool PAIR, bool AK1, bool BK1>
int q_launch(QParams p, int blocks, int* status, cudaStream_t stream, StatusClear& sc) {
    typedef QLayout<F32, NT> L;
    auto* kernel = qgemm_tc_kernel<F32, NT, AK, BK, PAIR, AK1, BK1>;
    PCB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(Q_THREADS);
    cfg.dynamicSmemBytes = L::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;    // as launch_chained
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    p.clear = nullptr;
    if (sc.pending) { p.clear = sc.word; sc.pending = false; }
    PCB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, status));
    return PCB_OK;
}

// Bytes per load of an operand whose rows start `ld` elements apart and whose components lie `cs` elements apart.
int q_chunk(const void* ptr, int ld, int cs, int es) {
    int c = 16;
    while (c > es && ((size_t)ld * es % c != 0 || (size_t)cs * es % c != 0 || reinterpret_cast<uintptr_t>(ptr) % c != 0)) c >>= 1;
    return c;
}
QOperand q_operand(const void* ptr, int cs, int ld, int nu, int nv, int f32) {
    QOperand o;
    o.p = ptr; o.cs = cs; o.ld = ld; o.nu = nu; o.nv = nv; o.chunk = q_chunk(ptr, ld, cs, f32 ? 4 : 2);
    return o;
}
void q_finish(QProblem& p, int NT, int f32, uint32_t neg) {
    p.tiles_m = (p.M + QM - 1) / QM;
    p.tiles_n = (p.N + NT - 1) / NT;
    p.stages = (p.K + (f32 ? 32 : 64) - 1) / (f32 ? 32 : 64) * 4;
    p.neg = neg;
}
uint32_t q_signs(Pass pass) {
    uint32_t neg = 0;
    for (int kc = 0; kc < 4; ++kc)
        for (int c = 0; c < 4; ++c) {
            const bool n = pass == PASS_FWD ? quat_negative(c ^ kc, c) : (pass == PASS_BWD_DATA ? quat_negative(c, c ^ kc) : quat_negative(c ^ kc, kc));
            if (n) neg |= 1u << (4 * kc + c);
        }
    return neg;
}
// SMs that clusters of `cl` CTAs of these kernels (one CTA per SM) fill at once. A cluster lies inside one group of 14 to 20 SMs, and how many SMs a group has
// differs between devices, so the runtime is asked: 16 clusters of 8 did not fit a device of 148 SMs, and the layers that were cut into 16 of them
// took two rounds (forward in 16 bits, 144 -> 946 features at batch 42, as two rounds of 8 / one of 4: 14.7 / 8.4 us). Beside an SM margin, a cluster less for
// each SM of it.
int q_slots(int cl) {
    static std::atomic<int> clusters[4];                               // of 1, 2, 4 and 8 CTAs, plus one; 0: not asked yet
    if (cl == 1) return sm_count();
    std::atomic<int>& known = clusters[cl == 2 ? 1 : (cl == 4 ? 2 : 3)];
    int n = known.load(std::memory_order_relaxed) - 1;
    if (n < 0) {
        auto* kernel = qgemm_tc_kernel<false, 32, false, true, false, false, false>;
        const size_t smem = QLayout<false, 32>::SMEM;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(device_sms() / cl * cl));
        cfg.blockDim = dim3(Q_THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)cl; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();                                        // (no device, as where only a route is asked for: an estimate, not kept)
            n = (cl > 2 ? device_sms() * 7 / 8 : device_sms()) / cl;
        } else {
            known.store(n + 1, std::memory_order_relaxed);
        }
    }
    return (n - g_sm_margin) * cl;
}
// Picks the slices of the stages of the one or two problems of a launch, and the cluster that holds them: powers of
// two up to 8 (a portable cluster). The cost of a choice is rounds of the machine x (stages of the longest CTA + the fixed part
// of a CTA, about as long as 6 stages). fp32: every slice short enough for its accumulators.
int q_plan(QParams& p, bool two, int f32) {
    long long best = -1;
    int blocks = 0;
    QProblem &a = p.prob[0], &b = p.prob[1];
    const int most = Q_F32_STAGES_PER_ACC * Q_F32_ACCS;                // stages of an fp32 slice
    const int ta = a.tiles_m * a.tiles_n, tb = two ? b.tiles_m * b.tiles_n : 0;
    int sa_best = 1, sb_best = 1;
    for (int sa = 1; sa <= 8; sa *= 2)
        for (int sb = 1; sb <= (two ? 8 : 1); sb *= 2) {
            const int la = (a.stages + sa - 1) / sa, lb = two ? (b.stages + sb - 1) / sb : 0;
            if ((sa > 1 && sa > a.stages) || (two && sb > 1 && sb > b.stages)) continue;
            if (f32 && (la > most || lb > most)) continue;
            const int cl = sa > sb ? sa : sb;
            const int na = round_up(ta * sa, cl), nb = round_up(tb * sb, cl), slots = q_slots(cl);
            if (slots < cl) continue;
            const long long cost = (long long)((na + nb + slots - 1) / slots) * ((la > lb ? la : lb) + 6 + (cl > 1 ? 1 : 0));
            if (best < 0 || cost < best) { best = cost; sa_best = sa; sb_best = sb; p.cluster = cl; p.first_blocks = na; blocks = na + nb; }
        }
    a.split = sa_best;
    b.split = sb_best;
    return blocks;
}

QProblem dense_problem(Pass pass, const Geom& g, const void* x, const void* w, const void* dy, const void* bias, void* out, int NT, int f32) {
    QProblem p;
    const int I = g.Ci, O = g.Co, B = g.Nb;
    p.out = out; p.bias = nullptr;
    if (pass == PASS_FWD) {
        p.M = O; p.N = B; p.K = I;
        p.a = g.w_io ? q_operand(w, I * O, O, O, I, f32) : q_operand(w, I * O, I, I, O, f32);
        p.b = q_operand(x, B * I, I, I, B, f32);
        p.o_c = B * O; p.o_n = O;
        p.bias = g.has_bias ? bias : nullptr;
    } else if (pass == PASS_BWD_DATA) {
        p.M = I; p.N = B; p.K = O;
        p.a = g.w_io ? q_operand(w, I * O, O, O, I, f32) : q_operand(w, I * O, I, I, O, f32);
        p.b = q_operand(dy, B * O, O, O, B, f32);
        p.o_c = B * I; p.o_n = I;
    } else {
        p.M = O; p.N = I; p.K = B;
        p.a = q_operand(dy, B * O, O, O, B, f32);
        p.b = q_operand(x, B * I, I, I, B, f32);
        p.o_c = I * O; p.o_n = O;
    }
    p.split = 1;
    q_finish(p, NT, f32, q_signs(pass));
    return p;
}
int q_tiles(const QProblem& p) { return p.tiles_m * p.tiles_n; }

}  // namespace

// fp32: a slice of the reduced dimension is at most 8 chunks of 32 long (q_plan), and there are at most 8 slices.
bool dense_tc_supported(int dtype, int variant, const Geom& g) {
    if (variant != PCB_VARIANT_16_PRODUCT || g.nc != 4 || g.real_in) return false;
    if (g.H != 1 || g.W != 1 || g.KH != 1 || g.KW != 1 || !g.dw_io || g.groups != 1) return false;
    const int most = 8 * Q_F32_STAGES_PER_ACC * Q_F32_ACCS / 4 * 32;
    if (dtype == PCB_F32 && (g.Ci > most || g.Co > most || g.Nb > most)) return false;
    // A wide fp32 layer runs faster from staged hi / lo operands: here every tile splits its operands again. This kernel against the
    // staged ones, us: forward 2048 x 2048 x 2048 2069 / 1829, 1024 x 2048 x 2048 1051 / 1036 (not for a forward pass that is longer than
    // wide, 2048 x 1024 x 1536 720 / 830, but one line serves both directions and backward is the longer one: preferred_route).
    if (dtype == PCB_F32 && (long long)g.Nb * g.Ci * g.Co > (1ll << 31)) return false;
    return true;
}

namespace {
// What a call launches; blocks == 0: no cut of the reduced dimensions fits the machine.
struct DensePlan {
    QParams p;
    int blocks, wide;
};
DensePlan plan_fwd(int dtype, const Geom& g, const void* x, const void* w, const void* bias, void* y) {
    const int f32 = dtype == PCB_F32;
    DensePlan d;
    d.p.fmt = f32 ? 2 : (dtype == PCB_F16 ? 0 : 1);
    d.p.prob[0] = dense_problem(PASS_FWD, g, x, w, nullptr, bias, y, 32, f32);
    d.wide = !f32 && q_tiles(d.p.prob[0]) > sm_count();
    if (d.wide) d.p.prob[0] = dense_problem(PASS_FWD, g, x, w, nullptr, bias, y, 64, f32);
    d.p.prob[1] = d.p.prob[0];
    d.blocks = q_plan(d.p, false, f32);
    return d;
}
DensePlan plan_bwd(int dtype, const Geom& g, const void* x, const void* w, const void* dy, void* dw, void* dx, bool both) {
    const int f32 = dtype == PCB_F32;
    DensePlan d;
    d.p.fmt = f32 ? 2 : (dtype == PCB_F16 ? 0 : 1);
    auto build = [&](int NT) {
        d.p.prob[0] = dense_problem(PASS_BWD_FILTER, g, x, w, dy, nullptr, dw, NT, f32);
        d.p.prob[1] = both ? dense_problem(PASS_BWD_DATA, g, x, w, dy, nullptr, dx, NT, f32) : d.p.prob[0];
        return q_tiles(d.p.prob[0]) + (both ? q_tiles(d.p.prob[1]) : 0);
    };
    d.wide = !f32 && build(32) > sm_count();
    build(d.wide ? 64 : 32);
    d.blocks = q_plan(d.p, both, f32);
    return d;
}
// These grids are not persistent: with an SM margin they are taken only where all their CTAs fit beside it at once.
bool plan_fits(const DensePlan& d) { return d.blocks > 0 && (g_sm_margin == 0 || d.blocks <= sm_count()); }
}  // namespace

// Where the staged kernels are the faster ones. They pay once for the copies and for the expanded filter matrix (16 products of I x O,
// whatever the batch) and then read their operands by TMA; here every tile loads, splits (fp32) or shifts (odd rows) its operands
// again. So they win for large batches of wide layers, earlier in fp32 and for rows that are not a whole number of load units, and
// for the filter gradient, whose reduction is the batch, where its few tiles leave it on as many CTAs. Batch x I x O, this kernel / staged,
// us:
//   forward        fp16  4096 x 2048 x 2048   641 /  772    8192 x 1536 x 1024   629 /  577    16384 x 512 x 512   219 /  261
//                  fp16  1024 x  511 x  333    42 /   48    4096 x  511 x  333   112 /   82     2048 x 1001 x 999   216 /  139
//                  fp32  1536 x 2048 x  512   398 /  449    2048 x 2048 x  512   543 /  521     1536 x 611 x 703   242 /  207
//   both gradients fp16  2048 x 2048 x 2048   657 /  959    4096 x 3072 x  768   981 /  927    16384 x 511 x 333   766 /  692
//                  fp32  1024 x 1024 x 1024   472 /  515    1536 x  768 x  768   478 /  397     2048 x 1024 x 1024 1029 /  845
//   dw alone       fp16  8192 x 2048 x 2048  1421 / 1496   16384 x  768 x  768   589 /  552     8192 x 511 x 333   327 /  260
//                  fp32  1024 x  256 x  256    38 /   56    1280 x  512 x  512   108 /   77     2048 x 1024 x 1024  526 /  370
// Both gradients of a large 16-bit layer are faster apart, dw here and dx staged: 4096 x 2048 x 1024 866 -> 710, 8192 x 1024 x 1024
// 926 -> 640 (both staged: 780).
DenseRoute preferred_route(int dtype, const Geom& g, bool backward, bool need_dx) {
    const long long B = g.Nb, I = g.Ci, O = g.Co, IO = I * O, P = B * IO;
    if (dtype == PCB_F32) {
        bool staged;                               // (rows of O alone that are not a whole number of 16-byte units: 1000 x 768 x 1001 forward 217 / 250)
        if (backward && !need_dx) staged = (B >= 1280 && P >= 180000000) || (B >= 768 && P >= 400000000);
        else if (I % 4 != 0 && (!backward || O % 4 != 0)) staged = P >= 500000000;
        else if (backward) staged = (B >= 1280 && P >= 720000000) || P >= 2000000000;
        else staged = B >= 1792 && I >= 2 * O && P >= 1500000000;
        return staged ? DENSE_STAGED : DENSE_DIRECT;
    }
    if (I % 2 != 0 || O % 2 != 0) {
        const bool both = I % 2 != 0 && O % 2 != 0, wide = IO >= 1 << 17;
        bool staged;
        if (backward && !need_dx) staged = (B >= 4096 && wide) || (B >= 65536 && IO >= 1 << 15);
        else if (backward) staged = (B >= 8192 && wide && (both || P >= 3000000000)) || (IO >= 500000 && B >= (both ? 2048 : 4096));
        else staged = (B >= 4096 && wide) || (B >= 1024 && I % 2 != 0 && IO >= 900000);
        return staged ? DENSE_STAGED : DENSE_DIRECT;
    }
    if (IO < 1 << 19) return DENSE_DIRECT;
    if (!backward) return B >= 6144 && P >= 6000000000 ? DENSE_STAGED : DENSE_DIRECT;
    // (dw of up to one tile per SM at a long reduction: 128 CTAs with a thousand stages each)
    if (B >= 16384 && IO <= 148ll * 128 * 32) return DENSE_STAGED;
    return need_dx && (B >= 6144 || (B >= 3072 && I >= 2 * O)) ? DENSE_FILTER_DIRECT : DENSE_DIRECT;
}

DenseRoute dense_tc_route(int dtype, const Geom& g, bool backward, bool need_dx) {
    const DenseRoute route = preferred_route(dtype, g, backward, need_dx);
    if (route == DENSE_STAGED) return route;
    const bool both = need_dx && route == DENSE_DIRECT;
    const bool fits = plan_fits(backward ? plan_bwd(dtype, g, nullptr, nullptr, nullptr, nullptr, nullptr, both) : plan_fwd(dtype, g, nullptr, nullptr, nullptr, nullptr));
    return fits ? route : DENSE_STAGED;
}

int dense_tc_fwd(int dtype, const Geom& g, const void* x, const void* w, const void* bias, void* y, int* status, cudaStream_t stream,
                 StatusClear& sc) {
    const DensePlan d = plan_fwd(dtype, g, x, w, bias, y);
    if (d.blocks == 0) { set_error("no split of this dense layer"); return PCB_ERR_UNSUPPORTED; }
    if (d.p.fmt == 2) return g.w_io ? q_launch<true, 32, false, true, false, false, false>(d.p, d.blocks, status, stream, sc)
                                    : q_launch<true, 32, true, true, false, false, false>(d.p, d.blocks, status, stream, sc);
    if (d.wide) return g.w_io ? q_launch<false, 64, false, true, false, false, false>(d.p, d.blocks, status, stream, sc)
                              : q_launch<false, 64, true, true, false, false, false>(d.p, d.blocks, status, stream, sc);
    return g.w_io ? q_launch<false, 32, false, true, false, false, false>(d.p, d.blocks, status, stream, sc)
                  : q_launch<false, 32, true, true, false, false, false>(d.p, d.blocks, status, stream, sc);
}

// dw, and dx unless it is null, in one launch.
int dense_tc_bwd(int dtype, const Geom& g, const void* x, const void* w, const void* dy, void* dw, void* dx, int* status, cudaStream_t stream,
                 StatusClear& sc) {
    const DensePlan d = plan_bwd(dtype, g, x, w, dy, dw, dx, dx != nullptr);
    if (d.blocks == 0) { set_error("no split of this dense layer"); return PCB_ERR_UNSUPPORTED; }
    const bool f32 = d.p.fmt == 2;
    if (!dx) {
        if (f32) return q_launch<true, 32, false, false, false, false, false>(d.p, d.blocks, status, stream, sc);
        return d.wide ? q_launch<false, 64, false, false, false, false, false>(d.p, d.blocks, status, stream, sc)
                      : q_launch<false, 32, false, false, false, false, false>(d.p, d.blocks, status, stream, sc);
    }
    if (f32) return g.w_io ? q_launch<true, 32, false, false, true, true, true>(d.p, d.blocks, status, stream, sc)
                           : q_launch<true, 32, false, false, true, false, true>(d.p, d.blocks, status, stream, sc);
    if (d.wide) return g.w_io ? q_launch<false, 64, false, false, true, true, true>(d.p, d.blocks, status, stream, sc)
                              : q_launch<false, 64, false, false, true, false, true>(d.p, d.blocks, status, stream, sc);
    return g.w_io ? q_launch<false, 32, false, false, true, true, true>(d.p, d.blocks, status, stream, sc)
                  : q_launch<false, 32, false, false, true, false, true>(d.p, d.blocks, status, stream, sc);
}

}  // namespace pcb
