// Tiled persistent PCG: one CTA per SM keeps every solver vector of its rows
// on the SM for the whole solve and streams nothing but the matrix.
//
// The streamed kernel (pcg_persistent.cuh) re-reads z, p, x, r, A p of every
// row each iteration and gathers each neighbour's z and old p from L2: 32 B
// per entry on top of the entry's own 28, so its iteration at 1024 x 1024 rows
// (96 us, block-Jacobi) is bound by L2 traffic (~0.7 GB), not by the 0.4 GB
// that must come from HBM.  Here
//   * p of the CTA's rows and of its halo (the other CTAs' rows that its
//     entries reach) lies in shared memory, and entries carry 16-bit indices
//     into it, so a gather is a shared-memory read;
//   * x, r and A p (then z in the same place) lie in tensor memory, used as
//     plain storage: 9 columns of one warp's 32 lanes per 32-row slice, 512
//     columns, i.e. 7 slices per warp and up to 224 (7,168 rows) per SM;
//   * x takes alpha p one iteration later, when p is at hand anyway;
//   * the blocks of a warp's next slice are already on their way: each warp
//     owns a stage in shared memory that the copy engine fills (cp.async.bulk)
//     while the warp works on, across the barriers too, so the stream does not
//     stop for the reductions (801 x 643: 25 -> 21 us per iteration; not with
//     the coarse level, whose rows of A_c^-1 live in the L1 that the stages
//     would take: 1024 x 1024 went from 96 to 117 ms with them);
//   * only z of rows in another CTA's halo goes through global memory: the
//     owner writes it with the update, every CTA forms the halo's p = z +
//     beta p itself, with the arithmetic of the owner (identical values).
// Per iteration a row costs its blocks and 16-bit columns (26 B each), D'
// and M^-1 (48 B), and 32 B of coarse weights with the coarse level.
// Measured on B200, streamed against tiled: 801 x 643 rows, 50 iterations,
// 2.88 against 1.30 ms (53 against 21 us per iteration); 1024 x 1024 96
// against 44 us per iteration, with the coarse level 118 against 56; a batch of
// 128 grids of 16 to 128 a side 105 against 47.  Their arithmetic per row is
// the same; only the FP64 sums run in another order.
//
// Phases, per-instance logic, preconditioner (block-Jacobi, or with a coarse
// level: CO = 1 dense, CO = 2 batched) and stopping rules are those of
// pcg_persistent_kernel, synchronisation by the counter barrier.  ONE: a
// single instance, whose per-row sums are kept per thread and added once per
// phase.  MODE 0 streams symmetric blocks, 1 general ones (bending); MODE 2
// first copies the CTA's blocks of either kind, their columns, D' and M^-1
// into shared memory, for systems whose rows are too wide for registers but
// whose matrix fits the SMs: their iteration is latency, not bytes.  CLU
// (MODE 2): the grid is one thread-block cluster, whose barrier and shared
// memory carry the reductions, as in the resident kernel's cluster build.
// A 61 x 47 garment with bending (18 neighbours a row, 16 CTAs): 11.9 us per
// iteration streamed, 4.6 as a cluster.
#pragma once

#include "pcg_persistent.cuh"

namespace chysx_b200 {

constexpr int kTileThreads = 1024;
constexpr int kTileWarps = kTileThreads / 32;
// threads per CTA: 512 where the matrix lies in shared memory (a few slices
// per CTA, the rest is synchronisation: the 61 x 47 garment 4.6 us per
// iteration against 5.0 with 1024)
__host__ __device__ constexpr int tile_threads(int mode) { return mode == 2 ? 512 : kTileThreads; }
constexpr int kTileCols = 9;          // TMEM columns per slice: x, r, A p / z
constexpr int kTileMaxSlices = 224;   // 7 per warp: 8 warps per lane quarter x 7 slices x 9 columns <= 512

struct TileArgs {
    const unsigned short* lcol;       // [ELL entries] own row (< the CTA's rows) or rows + halo index
    const int* halo_off;              // [grid + 1]
    const int* halo_row;              // internal row of every halo entry
    const unsigned short* halo_li;    // its instance, relative to the CTA's first
    const unsigned* bmask;            // [n_slices] rows in some halo, one bit per lane
    int tmem_cols;                    // columns allocated (power of two >= 32)
    int max_slices;                   // per CTA
    int max_halo;
    int max_entries;                  // ELL entries of a CTA (MODE 2; else 0)
    int ow;                           // floats per block (MODE 2)
    int max_blk;                      // coarse blocks of a CTA
    int stage;                        // blocks of a slice that a warp's stage holds (MODE 0; 0: no stages)
};
// Coarse values of one of the CTA's blocks, per phase and state: A_c^-1 R^T of
// r (kCU), of the new r (kCN), of b and of r0 (start only).
constexpr int kTileCoarseW = 48, kTcB = 24, kTc0 = 36;
static_assert(kCU == 0 && kCN == 12 && kInstCoarseW == 24, "the first two are the batched level's");

// Dynamic shared memory: slice partials, instance records, coarse values,
// slice offsets / masks / instances, halo rows and instances, p.
__host__ __device__ inline size_t tile_align(size_t v) { return (v + 15) & ~static_cast<size_t>(15); }
struct TileSmem {
    size_t li, vbuf, blk, soff, mask, sli, hrow, hli, p, mat, diag, col, stage, bytes;
};
__host__ __device__ inline TileSmem tile_smem(int parts, int max_inst, size_t coarse_bytes, int max_blk,
                                              int max_slices, int max_halo, int max_entries, int ow, int stage) {
    TileSmem s;
    s.li = (size_t)parts * kSlotW * sizeof(double);
    s.vbuf = tile_align(s.li + (size_t)max_inst * sizeof(LocalInst));
    s.blk = tile_align(s.vbuf + coarse_bytes);  // per block: values, first slice (+ 1), instance
    s.soff = tile_align(s.blk + (size_t)max_blk * (kTileCoarseW + 2) * sizeof(float) + sizeof(int));
    s.mask = s.soff + (size_t)(max_slices + 1) * sizeof(int);
    s.sli = s.mask + (size_t)max_slices * sizeof(unsigned);
    s.hrow = tile_align(s.sli + (size_t)max_slices * 2 * sizeof(unsigned short));  // instance, coarse block
    s.hli = s.hrow + (size_t)max_halo * sizeof(int);
    s.p = tile_align(s.hli + (size_t)max_halo * sizeof(unsigned short));
    s.mat = tile_align(s.p + (size_t)3 * (32 * (size_t)max_slices + max_halo) * sizeof(float));
    // MODE 2: blocks, D' and M^-1 (192 floats each per slice; copied in 16-byte
    // pieces, as the blocks), columns
    s.diag = tile_align(s.mat + (size_t)max_entries * ow * sizeof(float));
    s.col = s.diag + (max_entries ? (size_t)384 * max_slices * sizeof(float) : 0);
    s.stage = (s.col + (size_t)max_entries * sizeof(unsigned short) + 127) & ~static_cast<size_t>(127);
    s.bytes = s.stage + (size_t)stage * (kTileThreads / 32) * 192 * sizeof(float);
    return s;
}

// ---- tensor memory as storage: this warp's 32 lanes, consecutive columns ----
__device__ __forceinline__ void tm_ld1(uint32_t a, float& x) {
    uint32_t u;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(u) : "r"(a) : "memory");
    x = __uint_as_float(u);
}
__device__ __forceinline__ void tm_ld2(uint32_t a, float& x, float& y) {
    uint32_t u, v;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(u), "=r"(v) : "r"(a) : "memory");
    x = __uint_as_float(u);
    y = __uint_as_float(v);
}
__device__ __forceinline__ void tm_ld4(uint32_t a, float& x, float& y, float& z, float& w) {
    uint32_t u, v, s, t;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(u), "=r"(v), "=r"(s), "=r"(t)
                 : "r"(a)
                 : "memory");
    x = __uint_as_float(u);
    y = __uint_as_float(v);
    z = __uint_as_float(s);
    w = __uint_as_float(t);
}
// the loads above have arrived in a and b (which pass through, so no use moves ahead of the wait)
__device__ __forceinline__ void tm_wait_ld(float3& a, float3& b) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(a.x), "+f"(a.y), "+f"(a.z), "+f"(b.x), "+f"(b.y), "+f"(b.z)
                 :
                 : "memory");
}
__device__ __forceinline__ void tm_st1(uint32_t a, float x) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(a), "r"(__float_as_uint(x)) : "memory");
}
__device__ __forceinline__ void tm_st2(uint32_t a, float x, float y) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(a), "r"(__float_as_uint(x)),
                 "r"(__float_as_uint(y))
                 : "memory");
}
__device__ __forceinline__ void tm_st4(uint32_t a, float x, float y, float z, float w) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(__float_as_uint(x)),
                 "r"(__float_as_uint(y)), "r"(__float_as_uint(z)), "r"(__float_as_uint(w))
                 : "memory");
}
__device__ __forceinline__ void tm_wait_st() {
    __syncwarp();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_ld3(uint32_t a, float3& v) {
    __syncwarp();  // .sync.aligned: the warp must have reconverged
    tm_ld2(a, v.x, v.y);
    tm_ld1(a + 2, v.z);
}
__device__ __forceinline__ void tm_st3(uint32_t a, float3 v) {
    __syncwarp();
    tm_st2(a, v.x, v.y);
    tm_st1(a + 2, v.z);
}
// columns of a slice
constexpr uint32_t kTmX = 0, kTmR = 3, kTmQ = 6;

// streaming loads: read once per phase, not worth an L1 line
__device__ __forceinline__ float ld_na(const float* p) {
    float v;
    asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ S6 ld6_na(const float* p) {
    return S6{ld_na(p), ld_na(p + 32), ld_na(p + 64), ld_na(p + 96), ld_na(p + 128), ld_na(p + 160)};
}
__device__ __forceinline__ int ld_na(const unsigned short* p) {
    unsigned short v;
    asm volatile("ld.global.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

// ---- a warp's stage: one bulk copy at a time, completion on its mbarrier ----
__device__ __forceinline__ void stage_fetch(uint32_t dst, const float* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// waits for the copy of phase `parity`, at most kBarrierTimeoutNs
__device__ __forceinline__ bool stage_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    unsigned long long t0 = 0;
    for (unsigned spins = 0;; ++spins) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (spins == 0) t0 = global_ns();
        else if ((spins & 63u) == 0 && global_ns() - t0 > kBarrierTimeoutNs) return false;
    }
}

template <bool ONE, int CO, int MODE = 0, bool CLU = false>
__global__ void __launch_bounds__(tile_threads(MODE), 1)
pcg_tiled_kernel(DevTopo t, Vecs v, BatchPlan bp, SolverCfg cfg, int warm, const TileArgs* ta, void*) {
    constexpr int SYNC = 0;  // slot_set: two sets by parity
    constexpr int BLOCK = tile_threads(MODE), kW = BLOCK / 32;
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ int s_flag, s_exit;
    __shared__ uint32_t s_tmem;
    constexpr bool STG = MODE == 0 && CO == 0;
    __shared__ __align__(8) uint64_t s_mbar[STG ? kW : 1];
    __shared__ float s_tmp[CO ? BLOCK : 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = bp.cta_slice[blockIdx.x], s1 = bp.cta_slice[blockIdx.x + 1], ns = s1 - s0;
    const int il0 = bp.cta_inst_lo[blockIdx.x], il1 = bp.cta_inst_hi[blockIdx.x];
    const int nloc = il1 - il0 + 1;
    const TileArgs T = *ta;
    const int h0 = T.halo_off[blockIdx.x], nh = T.halo_off[blockIdx.x + 1] - h0;
    const int nown = ns * 32;
    const bool coarse = CO == 1 && bp.cg != nullptr && bp.cg->on && bp.cg->dense && *(volatile int*)bp.cg->fail == 0;
    const bool coarse_b =
        CO == 2 && !warm && bp.cg != nullptr && bp.cg->on && bp.cg->batched && *(volatile int*)bp.cg->fail == 0;
    const bool any_c = coarse || coarse_b;
    const size_t cbytes = CO == 1 && bp.cg ? (size_t)bp.cg->m * sizeof(float) + 16 : 0;
    const TileSmem lay = tile_smem(ONE ? kW : T.max_slices, bp.max_inst_per_cta, cbytes, T.max_blk,
                                   T.max_slices, T.max_halo, T.max_entries, T.ow, T.stage);
    __shared__ double s_cslot[CLU ? 2 : 1][kClusterMax][CLU ? kSlotW : 1];
    double* spart = reinterpret_cast<double*>(s_raw);
    LocalInst* li = reinterpret_cast<LocalInst*>(s_raw + lay.li);
    float* c_vbuf = reinterpret_cast<float*>(s_raw + lay.vbuf);
    float* c_blk = reinterpret_cast<float*>(s_raw + lay.blk);                  // [max_blk][kTileCoarseW]
    int* s_bk0 = reinterpret_cast<int*>(c_blk + (size_t)T.max_blk * kTileCoarseW);  // first slice of every block
    int* s_binst = s_bk0 + T.max_blk + 1;                                      // its instance, relative
    int* s_off = reinterpret_cast<int*>(s_raw + lay.soff);
    unsigned* s_mask = reinterpret_cast<unsigned*>(s_raw + lay.mask);
    unsigned short* s_sli = reinterpret_cast<unsigned short*>(s_raw + lay.sli);
    unsigned short* s_slb = s_sli + T.max_slices;
    int* s_hrow = reinterpret_cast<int*>(s_raw + lay.hrow);
    unsigned short* s_hli = reinterpret_cast<unsigned short*>(s_raw + lay.hli);
    float* s_p = reinterpret_cast<float*>(s_raw + lay.p);
    float* s_mat = reinterpret_cast<float*>(s_raw + lay.mat);
    float* s_diag = reinterpret_cast<float*>(s_raw + lay.diag);
    unsigned short* s_col = reinterpret_cast<unsigned short*>(s_raw + lay.col);
    unsigned target = 0;
    int ph = 0;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&s_tmem))),
                     "r"(T.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        s_flag = 0;
        s_exit = 0;
    }
    if (STG && lane == 0)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tfence.mbarrier_init.release.cluster;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&s_mbar[STG ? warp : 0])))
                     : "memory");
    init_local(bp, li, s0, s1, il0, il1);
    for (int k = tid; k <= ns; k += BLOCK) s_off[k] = t.slice_off[s0 + k];
    for (int k = tid; k < ns; k += BLOCK) {
        s_mask[k] = T.bmask[s0 + k];
        s_sli[k] = (unsigned short)(bp.slice_inst[s0 + k] - il0);
    }
    // the CTA's coarse blocks (runs of its slices)
    // (their parameters wait in shared memory: registers are short)
    __shared__ struct {
        const float4* w;
        const float* ainv;
        float* vals;
        const int *inst_blk, *inst_aoff;
        int m, g, nv, B0, nbl;  // nv: values per set
    } co;
    if (tid == 0) {
        co.nbl = 1;
        if (any_c) {
            const CoarseArgs& cg = *bp.cg;
            co.w = cg.w;
            co.ainv = cg.ainv;
            co.vals = cg.cvals;
            co.inst_blk = cg.inst_blk;
            co.inst_aoff = cg.inst_aoff;
            co.m = cg.m;
            co.g = cg.g;
            co.nv = 12 * cg.cta_blk[gridDim.x];
            co.B0 = cg.cta_blk[blockIdx.x];
            co.nbl = cg.cta_blk[blockIdx.x + 1] - co.B0;
        }
    }
    __syncthreads();
    if (any_c) {
        const int B0 = co.B0, nbl = co.nbl;
        for (int q = tid; q <= nbl; q += BLOCK) {
            s_bk0[q] = bp.cg->blk_row0[B0 + q] / 32 - s0;
            if (q < nbl) s_binst[q] = ONE ? 0 : bp.cg->blk_inst[B0 + q] - il0;
        }
        for (int x = tid; x < nbl * kTileCoarseW; x += BLOCK) c_blk[x] = 0.0f;
    }
    for (int h = tid; h < nh; h += BLOCK) {
        s_hrow[h] = T.halo_row[h0 + h];
        s_hli[h] = ONE ? 0 : T.halo_li[h0 + h];
    }
    if (MODE == 2) {
        const int e0 = t.slice_off[s0], ne = t.slice_off[s1] - e0;
        const float4* src = reinterpret_cast<const float4*>(t.val + (size_t)e0 * T.ow);
        for (int x = tid; x < ne * T.ow / 4; x += BLOCK) reinterpret_cast<float4*>(s_mat)[x] = src[x];
        const float4* d = reinterpret_cast<const float4*>(t.dnl + (size_t)s0 * 192);
        const float4* mi = reinterpret_cast<const float4*>(t.minv + (size_t)s0 * 192);
        for (int x = tid; x < ns * 48; x += BLOCK) {
            reinterpret_cast<float4*>(s_diag)[x] = d[x];
            reinterpret_cast<float4*>(s_diag)[ns * 48 + x] = mi[x];
        }
        for (int x = tid; x < ne; x += BLOCK) s_col[x] = T.lcol[e0 + x];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (CLU) cluster_sync_all();  // the other CTAs' shared memory is live before any store into it
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ONE && tid == 0) {  // the partials are per warp
        li[0].seg_lo = 0;
        li[0].seg_hi = kW;
    }
    if (any_c)
        for (int q = warp; q < co.nbl; q += kW)
            for (int k = s_bk0[q] + lane; k < s_bk0[q + 1]; k += 32) s_slb[k] = (unsigned short)q;
    __syncthreads();
    // The warp's stage: blocks of slice `staged` (-1: none under way)
    float* s_stage = reinterpret_cast<float*>(s_raw + lay.stage) + (size_t)warp * T.stage * 192;
    const uint32_t mbar = static_cast<uint32_t>(__cvta_generic_to_shared(&s_mbar[STG ? warp : 0]));
    const int n_stage = STG ? T.stage : 0;
    int staged = -1;
    uint32_t stage_par = 0;
    auto stage_blocks = [&](int k) { return min((s_off[k + 1] - s_off[k]) >> 5, n_stage); };
    // every lane's reads of the stage come before the copy that overwrites it:
    // plain reads and the copy engine's writes go through different proxies,
    // which __syncwarp alone does not order
    auto stage_slice = [&](int k) {
        const int c = stage_blocks(k);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (c == 0) return;
        staged = k;
        if (lane == 0)
            stage_fetch(static_cast<uint32_t>(__cvta_generic_to_shared(s_stage)), t.val + (size_t)s_off[k] * 6,
                        (uint32_t)c * 768u, mbar);
    };
    auto stage_done = [&]() {
        if (staged < 0) return;
        staged = -1;
        if (!stage_wait(mbar, stage_par)) {
            s_flag = 1;
            *(volatile int*)&bp.bar->error = 1;
        }
        stage_par ^= 1u;
    };
    // the next slice of this warp whose instance is not done
    auto next_k = [&](int k) {
        k += kW;
        while (!ONE && k < ns && li[s_sli[k]].done) k += kW;
        return k;
    };
    // tensor memory of the warp's j-th slice
    const uint32_t tm0 = s_tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(kTileCols * (warp >> 2));
    constexpr uint32_t kTmStep = kTileCols * (kW / 4);
    bool ok = true;
    auto no_step = [](LocalInst&, const double*) {};
    auto cw = [&](int i) { return __ldg(co.w + i); };  // four fields per block always
    auto cblk = [&](int k) { return c_blk + (ONE ? 0 : (int)s_slb[k]) * kTileCoarseW; };
    auto inst_of = [&](int k) { return ONE ? 0 : (int)s_sli[k]; };
    auto ldp = [&](int j) { return f3(s_p[3 * j], s_p[3 * j + 1], s_p[3 * j + 2]); };
    auto stp = [&](int j, float3 a) {
        s_p[3 * j] = a.x;
        s_p[3 * j + 1] = a.y;
        s_p[3 * j + 2] = a.z;
    };
    // restriction of a slice's vector into its partial (spart entry `part`)
    auto restrict_part = [&](float3 a, float4 w4, int part) { warp_restrict(4, a, w4, slice_cpart(spart, part)); };
    // the CTA's restrictions, 12 values per block, into this phase's set: P
    // threads per value add every P-th partial, then one adds the P sums
    auto publish_coarse = [&]() {
        float* dst = co.vals + (size_t)slot_set(ph) * co.nv + 12 * co.B0;
        const int nv = ONE ? 12 : co.nbl * 12;
        const int P = min(8, max(1, BLOCK / nv));
        for (int x = tid; x < nv * P; x += BLOCK) {
            const int h = x % P, qu = x / P, q = qu / 12, u = qu - 12 * q;
            const int lo = ONE ? 0 : s_bk0[q], hi = ONE ? kW : s_bk0[q + 1];
            float acc = 0.0f;
            for (int sl = lo + h; sl < hi; sl += P) acc += slice_cpart(spart, sl)[u];
            if (P > 1) s_tmp[x] = acc;
            else dst[qu] = acc;
        }
        if (P > 1) {
            __syncthreads();
            for (int x = tid; x < nv; x += BLOCK) {
                float acc = 0.0f;
                for (int h = 0; h < P; ++h) acc += s_tmp[x * P + h];
                dst[x] = acc;
            }
        }
        __syncthreads();
    };
    // y = A_c^-1 v on the CTA's own blocks, v the values of `set`: into entry
    // `off`, or (with_alpha) kCN = kCU - alpha y.  Ends with a __syncthreads.
    auto apply_coarse = [&](int set, int off, bool with_alpha) {
        const float* src = co.vals + (size_t)set * co.nv;
        const int nbl = co.nbl;
        if (CO == 1) {
            const int c_m = co.m, c_g = co.g;
            // v of every block (G CTAs each where they are small), then half
            // a row of A_c^-1 per warp, 16-byte pieces
            if (c_g == 1) {
                for (int x = tid; x < c_m / 4; x += BLOCK)
                    reinterpret_cast<float4*>(c_vbuf)[x] = __ldcg(reinterpret_cast<const float4*>(src) + x);
            } else {
                for (int x = tid; x < c_m / 4; x += BLOCK) {
                    const int B = x / 3, q = x - 3 * B;
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int c = B * c_g; c < min((B + 1) * c_g, (int)gridDim.x); ++c) {
                        const float4 v4 = __ldcg(reinterpret_cast<const float4*>(src + 12 * c) + q);
                        acc.x += v4.x;
                        acc.y += v4.y;
                        acc.z += v4.z;
                        acc.w += v4.w;
                    }
                    reinterpret_cast<float4*>(c_vbuf)[x] = acc;
                }
            }
            __syncthreads();
            constexpr int rows = 12, parts = 2;
            const int m4 = c_m / 4;
            const float4* A = reinterpret_cast<const float4*>(co.ainv + (size_t)(12 * (co.B0 / c_g)) * c_m);
            for (int x = warp; x < rows * parts; x += kW) {
                const int r = x / parts, h = x - r * parts;
                const float4* a4 = A + (size_t)r * m4;
                float acc = 0.0f;
#pragma unroll 4
                for (int j = h * 32 + lane; j < m4; j += 32 * parts) {
                    const float4 av = __ldg(a4 + j), vv = reinterpret_cast<const float4*>(c_vbuf)[j];
                    acc = fmaf(av.x, vv.x, fmaf(av.y, vv.y, fmaf(av.z, vv.z, fmaf(av.w, vv.w, acc))));
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                if (lane == 0) s_tmp[x] = acc;
            }
            __syncthreads();
            if (tid < rows) {
                const float y = s_tmp[2 * tid] + s_tmp[2 * tid + 1];
                float* o = c_blk + tid;
                if (with_alpha) o[kCN] = fmaf(-li[0].alpha, y, o[kCU]);
                else o[off] = y;
            }
        }
        if (CO == 2) {
            // a warp per block: the instance's values (at most 160, five per
            // lane) times the block's 12 rows of the instance's inverse
            for (int q = warp; q < nbl; q += kW) {
                const LocalInst& L = li[s_binst[q]];
                if (L.done) continue;
                const int I0 = co.inst_blk[L.b], m = 12 * (co.inst_blk[L.b + 1] - I0);
                const float* A = co.ainv + co.inst_aoff[L.b] + (size_t)(12 * (co.B0 + q - I0)) * m;
                float c[5], prod[16];
#pragma unroll
                for (int z = 0; z < 5; ++z) c[z] = lane + 32 * z < m ? __ldcg(src + 12 * I0 + lane + 32 * z) : 0.0f;
#pragma unroll
                for (int r = 0; r < 16; ++r) prod[r] = 0.0f;
#pragma unroll
                for (int z = 0; z < 5; ++z)
                    if (lane + 32 * z < m) {
#pragma unroll
                        for (int r = 0; r < 12; ++r)
                            prod[r] = fmaf(__ldg(A + (size_t)r * m + lane + 32 * z), c[z], prod[r]);
                    }
                const float y = warp_sum16(prod);
                const int u = lane >> 1;
                float* o = c_blk + q * kTileCoarseW;
                if ((lane & 1) == 0 && u < 12) {
                    if (with_alpha) o[kCN + u] = fmaf(-L.alpha, y, o[kCU + u]);
                    else o[off + u] = y;
                }
            }
        }
        __syncthreads();
    };
    // One reduction phase, after the partials and a __syncthreads: a warp per
    // instance publishes the CTA's segment, thread 0 meets the other CTAs, a
    // warp per instance reads the totals and applies `step`.
    auto phase = [&](auto nv, bool exit_test, auto&& step) {
        constexpr int NV = decltype(nv)::value;
        const int set = slot_set(ph);
        if constexpr (CLU) {
            cluster_phase<NV>(spart, li, 1, s_cslot, set, step);
        } else {
            for (int q = warp; q < nloc; q += kW) {
                const LocalInst& L = li[q];
                if (L.done) continue;
                double acc[NV];
#pragma unroll
                for (int u = 0; u < NV; ++u) acc[u] = 0.0;
                for (int sl = L.seg_lo + lane; sl < L.seg_hi; sl += 32) {
#pragma unroll
                    for (int u = 0; u < NV; ++u) acc[u] += spart[sl * kSlotW + u];
                }
#pragma unroll
                for (int u = 0; u < NV; ++u) {
                    acc[u] = warp_sum(acc[u]);
                    if (lane == 0) bp.slots[((size_t)set * bp.n_slots + L.own_slot) * kSlotW + u] = acc[u];
                }
            }
            __syncthreads();
            if (tid == 0) {
                if (!barrier_arrive_wait(bp.bar, target)) s_flag = 1;
                else if (exit_test) s_exit = *(volatile unsigned*)&bp.bar->ndone >= (unsigned)bp.n_inst;
            }
            __syncthreads();
            if (!s_flag) {
                for (int q = warp; q < nloc; q += kW) {
                    LocalInst& L = li[q];
                    if (L.done) continue;
                    constexpr int KP = 5;  // one pass covers 160 CTAs
                    double tot[NV];
#pragma unroll
                    for (int u = 0; u < NV; ++u) tot[u] = 0.0;
                    for (int c0 = L.slot_lo; c0 < L.slot_hi; c0 += 32 * KP) {
                        constexpr int NP = NV > 2 ? 2 : NV;  // values in flight together (registers)
#pragma unroll
                        for (int u0 = 0; u0 < NV; u0 += NP) {
                            double val[KP][NP];
#pragma unroll
                            for (int j = 0; j < KP; ++j)
#pragma unroll
                                for (int u = 0; u < NP; ++u) {
                                    const int k = c0 + j * 32 + lane;
                                    val[j][u] = k < L.slot_hi
                                                    ? __ldcg(bp.slots + ((size_t)set * bp.n_slots + k) * kSlotW + u0 + u)
                                                    : 0.0;
                                }
#pragma unroll
                            for (int j = 0; j < KP; ++j)
#pragma unroll
                                for (int u = 0; u < NP; ++u) tot[u0 + u] += val[j][u];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < NV; ++u) tot[u] = warp_sum(tot[u]);
                    if (lane == 0) step(L, tot);
                    __syncwarp();
                }
            }
        }
        ++ph;
        __syncthreads();
    };
    using N1 = std::integral_constant<int, 1>;
    using N2 = std::integral_constant<int, 2>;
    using N8 = std::integral_constant<int, kStartW>;
    // one exchange phase carrying only the restriction in the partials
    auto coarse_exchange = [&](int off) {
        __syncthreads();
        publish_coarse();
        const int set = slot_set(ph);
        phase(N1{}, false, no_step);
        if (!s_flag) apply_coarse(set, off, false);
        ok = s_flag == 0;
    };
    // (A p)_i = D'_i p_i + sum_j A_ij (p_j - p_i) of row `lane` of slice k, p in shared memory
    auto row_product = [&](int k, float3 pi) {
        const int s = s0 + k;
        const int so = s_off[k], w = (s_off[k + 1] - so) >> 5;
        float3 acc = f3(0.f, 0.f, 0.f);
        if constexpr (MODE == 2) {
            const int sl = so - s_off[0];
            const float* vb = s_mat + (size_t)sl * T.ow + lane;
            const unsigned short* lc = s_col + sl + lane;
            if (s * 32 + lane < t.n) acc = mul(ld6(s_diag + k * 192 + lane), pi);
            const int nsym = T.ow == 9;
#pragma unroll 2
            for (int e = 0; e < w; ++e) acc = acc + mul_off(vb + e * T.ow * 32, nsym, ldp(lc[e * 32]) - pi);
            return acc;
        }
        const unsigned short* lc = T.lcol + so + lane;
        if (s * 32 + lane < t.n) acc = mul(ld6_na(t.dnl + (size_t)s * 192 + lane), pi);
        if constexpr (MODE == 1) {
            const float* vb = t.val + (size_t)so * 9 + lane;
            for (int e = 0; e < w; ++e) {
                const float* q = vb + e * 288;
                const float3 d = ldp(ld_na(lc + e * 32)) - pi;
                acc = acc + f3(ld_na(q) * d.x + ld_na(q + 32) * d.y + ld_na(q + 64) * d.z,
                               ld_na(q + 96) * d.x + ld_na(q + 128) * d.y + ld_na(q + 160) * d.z,
                               ld_na(q + 192) * d.x + ld_na(q + 224) * d.y + ld_na(q + 256) * d.z);
            }
            return acc;
        }
        const float* vb = t.val + (size_t)so * 6 + lane;
        if (!STG || n_stage == 0) {
            if (w == 6) {
#pragma unroll
                for (int e = 0; e < 6; ++e) acc = acc + mul(ld6_na(vb + e * 192), ldp(ld_na(lc + e * 32)) - pi);
            } else {
                for (int e = 0; e < w; ++e) acc = acc + mul(ld6_na(vb + e * 192), ldp(ld_na(lc + e * 32)) - pi);
            }
            return acc;
        }
        if (staged != k) {  // first use, or another slice's instance has finished since
            stage_done();
            stage_slice(k);
        }
        const int c = min(w, n_stage);
        if (w == 6) {
            int col[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) col[e] = ld_na(lc + e * 32);
            stage_done();
            if (c == 6) {
#pragma unroll
                for (int e = 0; e < 6; ++e) acc = acc + mul(ld6(s_stage + e * 192 + lane), ldp(col[e]) - pi);
            } else {
#pragma unroll
                for (int e = 0; e < 6; ++e)
                    acc = acc + mul(e < c ? ld6(s_stage + e * 192 + lane) : ld6_na(vb + e * 192), ldp(col[e]) - pi);
            }
        } else {
            stage_done();
            for (int e = 0; e < w; ++e)
                acc = acc + mul(e < c ? ld6(s_stage + e * 192 + lane) : ld6_na(vb + e * 192),
                                ldp(ld_na(lc + e * 32)) - pi);
        }
        // the warp's next slice, of the next iteration after the last one
        int kn = next_k(k);
        if (kn >= ns) kn = next_k(warp - kW);
        if (kn < ns) stage_slice(kn);
        return acc;
    };
    // per-thread sums of a phase: added over the warp once (ONE) or per slice
    struct Sums {
        double a, b;
        float3 c[4];
    };
    auto zero_sums = [](Sums& q) {
        q.a = q.b = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) q.c[u] = f3(0.f, 0.f, 0.f);
    };
    auto add_restrict = [](Sums& q, float3 a, float4 w4) {
        q.c[0] = q.c[0] + a;
        q.c[1] = f3(fmaf(w4.x, a.x, q.c[1].x), fmaf(w4.x, a.y, q.c[1].y), fmaf(w4.x, a.z, q.c[1].z));
        q.c[2] = f3(fmaf(w4.y, a.x, q.c[2].x), fmaf(w4.y, a.y, q.c[2].y), fmaf(w4.y, a.z, q.c[2].z));
        q.c[3] = f3(fmaf(w4.z, a.x, q.c[3].x), fmaf(w4.z, a.y, q.c[3].y), fmaf(w4.z, a.z, q.c[3].z));
    };
    auto put_restrict = [&](const Sums& q) {  // the warp's 12 sums into its partial
        const float a[16] = {q.c[0].x, q.c[0].y, q.c[0].z, q.c[1].x, q.c[1].y, q.c[1].z, q.c[2].x, q.c[2].y,
                             q.c[2].z, q.c[3].x, q.c[3].y, q.c[3].z, 0.f, 0.f, 0.f, 0.f};
        const float y = warp_sum16(a);
        const int u = lane >> 1;
        if ((lane & 1) == 0 && u < 12) slice_cpart(spart, warp)[u] = y;
    };
    // restriction of a per-row vector get(k, i) into the partials
    auto restrict_all = [&](auto&& get) {
        Sums sm;
        zero_sums(sm);
        uint32_t tm = tm0;
        for (int k = warp; k < ns; k += kW, tm += kTmStep) {
            const int i = (s0 + k) * 32 + lane;
            const float3 a = get(tm, i);
            const float4 w4 = i < t.n ? cw(i) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (ONE) add_restrict(sm, a, w4);
            else {
                if (lane == 0) spart[k * kSlotW] = 0.0;
                restrict_part(a, w4, k);
            }
        }
        if (ONE) {
            if (lane == 0) spart[warp * kSlotW] = 0.0;
            put_restrict(sm);
        }
    };
    auto load_b = [&](uint32_t, int i) { return i < t.n ? xyz(v.b[i]) : f3(0.f, 0.f, 0.f); };
    auto load_minv = [&](int s, int i) {
        S6 m{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (i < t.n)
            m = MODE == 2 ? ld6(s_diag + (ns + s - s0) * 192 + lane) : ld6_na(t.minv + (size_t)s * 192 + lane);
        return m;
    };
    auto publish_z = [&](int k, int i, float3 z) {
        if ((s_mask[k] >> lane) & 1u) __stcg(v.z + i, f4(z));
    };

    // ---- start: r = b - A x0, z = M^-1 r, the instances' start values -------
    if (any_c) {
        restrict_all(load_b);
        coarse_exchange(kTcB);  // A_c^-1 R^T b
    }
    if (ok && warm) {
        uint32_t tm = tm0;
        for (int k = warp; k < ns; k += kW, tm += kTmStep) {
            const int i = (s0 + k) * 32 + lane;
            stp(k * 32 + lane, i < t.n ? xyz(v.x[i]) : f3(0.f, 0.f, 0.f));
        }
        for (int h = tid; h < nh; h += BLOCK) stp(nown + h, xyz(ldcg4(v.x + s_hrow[h])));
        __syncthreads();
        tm = tm0;
        for (int k = warp; k < ns; k += kW, tm += kTmStep) {
            const int i = (s0 + k) * 32 + lane;
            const float3 ax = row_product(k, ldp(k * 32 + lane));
            tm_st3(tm + kTmR, load_b(0u, i) - ax);
        }
        tm_wait_st();
        if (coarse) {
            restrict_all([&](uint32_t tm, int) {
                float3 r, d = f3(0.f, 0.f, 0.f);
                tm_ld3(tm + kTmR, r);
                tm_wait_ld(r, d);
                return r;
            });
            coarse_exchange(kTc0);  // A_c^-1 R^T r0
        }
    }
    auto zb_of = [&](int k, int i, const S6& Mi, float3 b, float4 w4) {
        float3 zb = mul(Mi, b);
        if (any_c) zb = zb + coarse_prolong(4, cblk(k) + kTcB, w4);
        return zb;
    };
    if (ok) {
        double tot[kStartW];
#pragma unroll
        for (int u = 0; u < kStartW; ++u) tot[u] = 0.0;
        uint32_t tm = tm0;
        for (int k = warp; k < ns; k += kW, tm += kTmStep) {
            const int i = (s0 + k) * 32 + lane;
            const S6 Mi = load_minv(s0 + k, i);
            const float4 w4 = any_c && i < t.n ? cw(i) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float3 b = load_b(0u, i), zb = zb_of(k, i, Mi, b, w4);
            float3 x0 = f3(0.f, 0.f, 0.f), r = b, z = zb;
            if (warm) {
                float3 d = f3(0.f, 0.f, 0.f);
                tm_ld3(tm + kTmR, r);
                tm_wait_ld(r, d);
                x0 = ldp(k * 32 + lane);
                z = mul(Mi, r);
                if (coarse) z = z + coarse_prolong(4, cblk(k) + kTc0, w4);
            } else {
                tm_st3(tm + kTmX, x0);
                tm_st3(tm + kTmR, r);
                tm_st3(tm + kTmQ, z);
                publish_z(k, i, z);
            }
            const double q8[kStartW] = {dot3d(r, z), dot3d(r, r), dot3d(b, b), dot3d(b, zb),
                                        dot3d(x0, b), dot3d(x0, r), dot3d(b, z), dot3d(b, r)};
            if (ONE) {
#pragma unroll
                for (int u = 0; u < kStartW; ++u) tot[u] += q8[u];
            } else {
#pragma unroll
                for (int u = 0; u < kStartW; ++u) {
                    const double y = warp_sum(q8[u]);
                    if (lane == 0) spart[k * kSlotW + u] = y;
                }
            }
        }
        tm_wait_st();
        if (ONE) {
#pragma unroll
            for (int u = 0; u < kStartW; ++u) {
                const double y = warp_sum(tot[u]);
                if (lane == 0) spart[warp * kSlotW + u] = y;
            }
        }
        __syncthreads();
        phase(N8{}, false, [&](LocalInst& L, const double* q) { step_start(bp, L, q, cfg, warm); });
        ok = s_flag == 0;
    }
    if (ok && warm) {
        // the scaled guess, or the zero guess where the instance fell back
        uint32_t tm = tm0;
        for (int k = warp; k < ns; k += kW, tm += kTmStep) {
            const int i = (s0 + k) * 32 + lane;
            const S6 Mi = load_minv(s0 + k, i);
            const float4 w4 = any_c && i < t.n ? cw(i) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float3 b = load_b(0u, i);
            float3 x = ldp(k * 32 + lane), r, z, d = f3(0.f, 0.f, 0.f);
            tm_ld3(tm + kTmR, r);
            tm_wait_ld(r, d);
            const LocalInst& L = li[inst_of(k)];
            if (coarse) {
                z = mul(Mi, r) + coarse_prolong(4, cblk(k) + kTc0, w4);
                start_row_linear(L, b, zb_of(k, i, Mi, b, w4), x, r, z);
            } else {
                start_row(L, b, Mi, x, r, z);
            }
            tm_st3(tm + kTmX, x);
            tm_st3(tm + kTmR, r);
            tm_st3(tm + kTmQ, z);
            publish_z(k, i, z);
        }
        tm_wait_st();
        // a data-free phase orders the new z before any halo read
        for (int q = tid; q < (ONE ? kW : ns); q += BLOCK) spart[q * kSlotW] = 0.0;
        __syncthreads();
        phase(N1{}, false, no_step);
        ok = s_flag == 0;
    }
    if (any_c && ok) {
        // A_c^-1 R^T r of the start: of r0, of the scaled mix of r0 and b, or of b
        const bool from_r0 = coarse && warm && !li[0].fallback;
        for (int x = tid; x < 12 * co.nbl; x += BLOCK) {
            float* o = c_blk + (x / 12) * kTileCoarseW + x % 12;
            o[kCU] = from_r0 ? fmaf(li[0].scale, o[kTc0], li[0].scale_b * o[kTcB]) : o[kTcB];
        }
        __syncthreads();
    }

    // ---- iterations ---------------------------------------------------------
    const int iter_cap = cfg.max_iter + 2;
    for (int guard = 0; ok && guard < iter_cap; ++guard) {
        if (ONE && li[0].done) break;  // uniform over the grid: every CTA forms the same totals
        // p = z + beta p of the own rows and, from the published z, of the
        // halo; x takes the previous iteration's alpha p
        uint32_t tm = tm0;
        for (int k = warp; k < ns; k += kW, tm += kTmStep) {
            const LocalInst& L = li[inst_of(k)];
            if (L.done) continue;
            float3 z, x = f3(0.f, 0.f, 0.f);
            tm_ld3(tm + kTmQ, z);
            if (L.iter > 0) {
                tm_ld3(tm + kTmX, x);
                const float3 p = ldp(k * 32 + lane);
                const float al = L.alpha, be = L.beta;
                tm_wait_ld(z, x);
                tm_st3(tm + kTmX, f3(fmaf(al, p.x, x.x), fmaf(al, p.y, x.y), fmaf(al, p.z, x.z)));
                z = f3(fmaf(be, p.x, z.x), fmaf(be, p.y, z.y), fmaf(be, p.z, z.z));
            } else {
                tm_wait_ld(z, x);
            }
            stp(k * 32 + lane, z);
        }
        for (int h = tid; h < nh; h += BLOCK) {
            const LocalInst& L = li[ONE ? 0 : s_hli[h]];
            if (L.done) continue;
            float3 z = xyz(ldcg4(v.z + s_hrow[h]));
            if (L.iter > 0) {
                const float3 p = ldp(nown + h);
                const float be = L.beta;
                z = f3(fmaf(be, p.x, z.x), fmaf(be, p.y, z.y), fmaf(be, p.z, z.z));
            }
            stp(nown + h, z);
        }
        __syncthreads();
        // A p, sigma = p.A p (and the restriction of A p); M^-1 of the update's
        // first slice comes in behind the barrier (registers permitting)
        S6 mi_n{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        auto fetch_diag = [&](int k) {
            if (k >= ns) return;
            const int i = (s0 + k) * 32 + lane;
            mi_n = load_minv(s0 + k, i);
        };
        {
            Sums sm;
            zero_sums(sm);
            uint32_t tm = tm0;
            for (int k = warp; k < ns; k += kW, tm += kTmStep) {
                const LocalInst& L = li[inst_of(k)];
                if (L.done) continue;
                const int i = (s0 + k) * 32 + lane;
                const float4 w4 = any_c && i < t.n ? cw(i) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float3 pi = ldp(k * 32 + lane);
                const float3 acc = row_product(k, pi);
                tm_st3(tm + kTmQ, acc);
                const double sig = (double)pi.x * acc.x + (double)pi.y * acc.y + (double)pi.z * acc.z;
                if (ONE) {
                    sm.a += sig;
                    if (CO == 1) add_restrict(sm, acc, w4);
                } else {
                    const double y = warp_sum(sig);
                    if (lane == 0) spart[k * kSlotW] = y;
                    if (coarse_b) restrict_part(acc, w4, k);
                }
            }
            if (ONE) {
                const double y = warp_sum(sm.a);
                if (lane == 0) spart[warp * kSlotW] = y;
                if (CO == 1) put_restrict(sm);
            }
            tm_wait_st();
        }
        if (STG) fetch_diag(next_k(warp - kW));
        __syncthreads();
        if (any_c) publish_coarse();
        const int set1 = slot_set(ph);
        phase(N1{}, !ONE, [&](LocalInst& L, const double* q) { step_alpha(L, q); });
        if (s_flag) {
            ok = false;
            break;
        }
        // every CTA reads ndone between the same two barriers, where it does not change
        if (!ONE && s_exit) break;
        if (any_c) apply_coarse(set1, 0, true);
        // r -= alpha A p; z = M^-1 r (+ its coarse part)
        {
            Sums sm;
            zero_sums(sm);
            int kn = 0;
            for (int k = next_k(warp - kW); k < ns; k = kn) {
                const LocalInst& L = li[inst_of(k)];
                const uint32_t tm = tm0 + kTmStep * (uint32_t)(k / kW);
                const int i = (s0 + k) * 32 + lane;
                float3 r, ap;
                __syncwarp();
                tm_ld4(tm + kTmR, r.x, r.y, r.z, ap.x);
                tm_ld2(tm + kTmQ + 1, ap.y, ap.z);
                kn = next_k(k);
                if (!STG) fetch_diag(k);
                const S6 Mi = mi_n;
                const float4 w4 = any_c && i < t.n ? cw(i) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float al = L.alpha;
                if (STG) fetch_diag(kn);
                tm_wait_ld(r, ap);
                const float3 rn = f3(fmaf(-al, ap.x, r.x), fmaf(-al, ap.y, r.y), fmaf(-al, ap.z, r.z));
                float3 zn = mul(Mi, rn);
                if (any_c) zn = zn + coarse_prolong(4, cblk(k) + kCN, w4);
                __syncwarp();
                tm_st4(tm + kTmR, rn.x, rn.y, rn.z, zn.x);
                tm_st2(tm + kTmQ + 1, zn.y, zn.z);
                publish_z(k, i, zn);
                const double rz = dot3d(rn, zn), rr = dot3d(rn, rn);
                if (ONE) {
                    sm.a += rz;
                    sm.b += rr;
                    if (CO == 1) add_restrict(sm, rn, w4);
                } else {
                    const double y = warp_sum(rz), y2 = warp_sum(rr);
                    if (lane == 0) {
                        spart[k * kSlotW] = y;
                        spart[k * kSlotW + 1] = y2;
                    }
                    if (coarse_b) restrict_part(rn, w4, k);
                }
            }
            if (ONE) {
                const double y = warp_sum(sm.a), y2 = warp_sum(sm.b);
                if (lane == 0) {
                    spart[warp * kSlotW] = y;
                    spart[warp * kSlotW + 1] = y2;
                }
                if (CO == 1) put_restrict(sm);
            }
            tm_wait_st();
        }
        __syncthreads();
        if (any_c) publish_coarse();
        const int set2 = slot_set(ph);
        phase(N2{}, false, [&](LocalInst& L, const double* q) { step_beta(bp, L, q, cfg); });
        if (s_flag) {
            ok = false;
            break;
        }
        // the coarse part restarts from R^T r_new (no recurrence drift)
        if (any_c) apply_coarse(set2, kCU, false);
    }
    // x with the last iteration's alpha p
    uint32_t tm = tm0;
    for (int k = warp; k < ns; k += kW, tm += kTmStep) {
        const LocalInst& L = li[inst_of(k)];
        const int i = (s0 + k) * 32 + lane;
        float3 x, d = f3(0.f, 0.f, 0.f);
        tm_ld3(tm + kTmX, x);
        tm_wait_ld(x, d);
        if (L.iter > 0) {
            const float3 p = ldp(k * 32 + lane);
            x = f3(fmaf(L.alpha, p.x, x.x), fmaf(L.alpha, p.y, x.y), fmaf(L.alpha, p.z, x.z));
        }
        if (i < t.n) v.x[i] = f4(x);
    }
    if (!ok) instances_fail(bp, li, nloc);
    stage_done();  // the copy for the iteration that does not come
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(T.tmem_cols) : "memory");
}

}  // namespace chysx_b200
