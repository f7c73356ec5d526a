// MXFP4 GEMM for skinny M (decode shapes, M <= 64, batch 1): C[M,N] = A @ B^T, optionally c_a * (A @ B^T) + c_b.
//
// HBM-bound on the weight stream like the FP8 kernel of gemm_fp8_skinny.cu, whose schedule it shares: N is cut into
// 16-column units that are dealt out as (rounds) x (number of SMs) tiles of up to 240 columns, so that every SM streams
// the same number of weight rows; consecutive CTAs start their walk over K at different blocks.
//
// What is new here are the scale factors.  tcgen05.cp moves whole 512-byte atoms of 128 rows, and the MMA can only start
// at an even 32-row group of one, so a tile cut at a 16-column unit cannot use the atoms as they lie in memory.  Staging
// warps therefore gather each row's scale words with 4-byte cp.async and lay them down as atoms that start at the
// tile's own first row.  The gather reads either form -- the tensor-core layout or the caller's row-major [rows, K/32]
// bytes -- so row-major calls need no re-layout pass and no scratch either.
//
// 16 x 28672 x 8192, cold L2: 24.5 us (5.1 TB/s) with tensor-core scales and 26.3 with row-major ones; the one-CTA kernel on
// 128 x 128 tiles (224 of them, 1.5 waves) takes 37.4, and 6.6 for the pre-pass on top.
//
// Roles: warp 0 TMA producer, warp 1 TMEM allocator + MMA issuer, warps 2-5 epilogue (two accumulators),
// warps 6.. scale staging.  Bounded waits and teardown as in gemm_fp8.cu.
#include "tc_common.cuh"

namespace hkb {
namespace {

constexpr int kMaxStages = 24;
constexpr int kBarBytes = 1024;           // barriers + tmem slot + abort flag live in the first KB
constexpr int kTailPad = 16 * 1024;       // the MMA reads 128 rows x 128 B from every A base
constexpr int kSmemLimit = 232448;        // 227 KB
constexpr int kMaxUnits = 15;             // 240 columns: 2 x 240 accumulator columns + 24 of scale factors in TMEM
constexpr int kSfBytes = 3 * 1024;        // per stage: two atoms of A, two K atoms x two row blocks of B
constexpr int kStagers = 5;               // warps (<= stages: 240 columns and 64 rows leave five)

struct SkinnyMxParams {
    int M, N, K;
    int a_box_rows, a_bytes;              // rows of A fetched per stage (multiple of 8, <= 64); smem reserved for them
    int tiles, base, rem;                 // tile t is base + (t < rem) units wide and starts at unit t*base + min(t, rem)
    int stages, stage_bytes, sf_off;      // sf_off: scale atoms inside a stage
    int rot;                              // K blocks by which consecutive CTAs are offset in their walk over K
    int katoms, katoms_tc;                // K / 128, and rounded up to even (row pitch of the tensor-core layout in atoms)
    const uint8_t* sfa;
    const uint8_t* sfb;
    int sfa_tc, sfb_tc;                   // layout of each scale array: 1 = tensor-core, 0 = row-major [rows, K/32]
    __nv_bfloat16* C;
    const __nv_bfloat16* c_a;             // fused multiply-add, or null
    const __nv_bfloat16* c_b;
    uint32_t* status;
};

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&p);
}
// Byte offset of row r's word of K atom 0, and the distance to the next K atom's word.
__device__ __forceinline__ size_t sf_row_offset(int r, bool tc, int katoms, int katoms_tc) {
    return tc ? (size_t)(r >> 7) * katoms_tc * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4 : (size_t)r * katoms * 4;
}
// Byte offset of row r's word inside consecutive atoms of 128 rows.
__device__ __forceinline__ uint32_t sf_smem_offset(int r) { return (uint32_t)((r >> 7) * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4); }
// Four bytes global -> shared, zeros when !valid (the source is then not read).
__device__ __forceinline__ void cp_async4(uint32_t dst, const uint8_t* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

#define TILE_WIDTH(t) (p.base + ((t) < p.rem ? 1 : 0))
#define TILE_COL0(t) (((t) * p.base + min((t), p.rem)) * 16)

__global__ void __launch_bounds__(192 + 32 * kStagers, 1)
gemm_mxfp4_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB128,
                         const __grid_constant__ CUtensorMap tmB64, const __grid_constant__ CUtensorMap tmB16,
                         const SkinnyMxParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t bar_base = smem_u32(smem);
    const uint32_t ring_base = bar_base + kBarBytes;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + 2 + a); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + 8 * (2 * kMaxStages + 4));
    volatile uint32_t* abort_flag = tmem_slot + 1;
    // TMEM columns: accumulators at 0 and 256 (240 each), A's scales at 240 (2 K atoms x 4), B's at 496 (2 x 8)
    constexpr uint32_t TMEM_COLS = 512, TMEM_SFA = 240, TMEM_SFB = 496;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int kstages = (p.K + 255) / 256;            // a 128-element tail reads zero-filled data and zero scales
    const int ks0 = (int)(((long long)blockIdx.x * p.rot) % kstages);

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full_bar(s), 2);                // the producer's expect_tx arrive + the staging warp's
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 4);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS);
    pdl_wait();      // nothing in global memory is touched before this
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {
            prefetch_tmap(&tmA);
            prefetch_tmap(&tmB128);
            prefetch_tmap(&tmB64);
            prefetch_tmap(&tmB16);
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
                const int w = TILE_WIDTH(t);
                const int n0 = TILE_COL0(t);
                const uint32_t stage_tx = (uint32_t)p.a_box_rows * 128 + (uint32_t)w * 2048;
                int ks = ks0;
                for (int i = 0; i < kstages; ++i, ks = (ks + 1 == kstages ? 0 : ks + 1)) {
                    if (!mbar_wait(empty_bar(s), ph ^ 1, abort_flag, p.status, kErrWaitProducer)) { ok = false; break; }
                    mbar_arrive_expect_tx(full_bar(s), stage_tx);
                    const uint32_t st = ring_base + s * p.stage_bytes;
                    tma_load_3d(st, &tmA, full_bar(s), ks * 128, 0, 0);
                    const uint32_t sb = st + p.a_bytes;
                    int r = 0;
                    for (; r + 8 <= w; r += 8) tma_load_3d(sb + r * 2048, &tmB128, full_bar(s), ks * 128, n0 + r * 16, 0);
                    for (; r + 4 <= w; r += 4) tma_load_3d(sb + r * 2048, &tmB64, full_bar(s), ks * 128, n0 + r * 16, 0);
                    for (; r < w; ++r) tma_load_3d(sb + r * 2048, &tmB16, full_bar(s), ks * 128, n0 + r * 16, 0);
                    if (++s == p.stages) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            int acc = 0;
            uint32_t acc_ph = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
                const uint32_t n = 16u * TILE_WIDTH(t);
                const int sfb_blocks = n > 128 ? 2 : 1;
                if (!mbar_wait(tempty_bar(acc), acc_ph ^ 1, abort_flag, p.status, kErrWaitMma)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * 256;
                for (int i = 0; i < kstages; ++i) {     // accumulation order follows the producer's walk
                    if (!mbar_wait(full_bar(s), ph, abort_flag, p.status, kErrWaitMma)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t st = ring_base + s * p.stage_bytes;
                    const uint64_t da = smem_desc_sw128(st);
                    const uint64_t db = smem_desc_sw128(st + p.a_bytes);
                    const uint32_t sf = st + p.sf_off;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {       // the two K atoms of this stage
                        tc_cp_sf(tmem_base + TMEM_SFA + h * 4, smem_desc_sf(sf + h * 512));
                        for (int r = 0; r < sfb_blocks; ++r)
                            tc_cp_sf(tmem_base + TMEM_SFB + (h * 2 + r) * 4, smem_desc_sf(sf + 1024 + (h * 2 + r) * 512));
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {       // 4 x K=64 (32 bytes of each 128-byte row)
                        const uint32_t h = k >> 1, sf_id = (k & 1) * 2;
                        mma_mxf4(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc_mxf4(128, n, sf_id, sf_id),
                                 tmem_base + TMEM_SFA + h * 4, tmem_base + TMEM_SFB + h * 8, (i | k) != 0);
                    }
                    tc_commit(empty_bar(s));
                    if (++s == p.stages) { s = 0; ph ^= 1; }
                }
                if (ok) {
                    tc_commit(tfull_bar(acc));
                    if (++acc == 2) { acc = 0; acc_ph ^= 1; }
                }
            }
        }
    } else if (warp < 6) {
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const bool row_ok = row < p.M;
        const bool warp_has_rows = quarter * 32 < p.M;       // warp-uniform: quarters past M read no TMEM
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const int64_t row_off = (int64_t)(row_ok ? row : 0) * p.N;
        int acc = 0;
        uint32_t acc_ph = 0;
        for (int t = blockIdx.x; t < p.tiles; t += gridDim.x) {
            const int w = TILE_WIDTH(t);
            const int n0 = TILE_COL0(t);
            if (p.c_a && row_ok)
                for (int c = 0; c < w * 16; c += 64) {
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.c_a + row_off + n0 + c));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.c_b + row_off + n0 + c));
                }
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(tfull_bar(acc), acc_ph, abort_flag, p.status, kErrWaitEpilogue))) break;
            tc_fence_after();
            if (warp_has_rows) {
                const uint32_t t_addr = tmem_base + lane_addr + acc * 256;
                for (int u = 0; u < w; ++u) {
                    uint32_t r[16];
                    tmem_ld16(t_addr + u * 16, r);
                    const int64_t off = row_off + n0 + u * 16;
                    uint4 ca0, ca1, cb0, cb1;
                    if (p.c_a) {                             // row 0 stands in for rows past M
                        ca0 = __ldg(reinterpret_cast<const uint4*>(p.c_a + off)); ca1 = __ldg(reinterpret_cast<const uint4*>(p.c_a + off + 8));
                        cb0 = __ldg(reinterpret_cast<const uint4*>(p.c_b + off)); cb1 = __ldg(reinterpret_cast<const uint4*>(p.c_b + off + 8));
                    }
                    tmem_ld_wait();
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                    if (p.c_a) {
                        float a[16], b[16];
                        unpack8(ca0, *reinterpret_cast<float(*)[8]>(a)); unpack8(ca1, *reinterpret_cast<float(*)[8]>(a + 8));
                        unpack8(cb0, *reinterpret_cast<float(*)[8]>(b)); unpack8(cb1, *reinterpret_cast<float(*)[8]>(b + 8));
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = __fmaf_rn(a[j], v[j], b[j]);
                    }
                    if (row_ok) {
                        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                                     ::"l"(p.C + off), "r"(pack2(v[0], v[1])), "r"(pack2(v[2], v[3])), "r"(pack2(v[4], v[5])),
                                       "r"(pack2(v[6], v[7])), "r"(pack2(v[8], v[9])), "r"(pack2(v[10], v[11])),
                                       "r"(pack2(v[12], v[13])), "r"(pack2(v[14], v[15])) : "memory");
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(acc));
            if (++acc == 2) { acc = 0; acc_ph ^= 1; }
        }
    } else {
        // ================= scale staging =================
        // Warp g takes every kStagers-th stage from start to end: copies out, wait, fence, arrive.  So as many stages are
        // in flight as there are warps.  (Two warps that kept several stages' copies in flight each did no better than
        // one stage at a time: the proxy fence waits for all of a thread's copies.)
        const int g = warp - 6;
        const size_t a_step = p.sfa_tc ? 512 : 4, b_step = p.sfb_tc ? 512 : 4;     // to the next K atom's word
        int s = g;                                           // g < kStagers <= stages
        uint32_t ph = 0;
        int i = g;                                           // K step of the tile, in the producer's order
        bool ok = true;
        for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
            const int rows = TILE_WIDTH(t) * 16;
            const int n0 = TILE_COL0(t);
            for (; i < kstages; i += kStagers) {
                if (!__all_sync(0xFFFFFFFFu, mbar_wait(empty_bar(s), ph ^ 1, abort_flag, p.status, kErrWaitProducer))) { ok = false; break; }
                const uint32_t sf = ring_base + s * p.stage_bytes + p.sf_off;
                const int ks = ks0 + i < kstages ? ks0 + i : ks0 + i - kstages;
                const bool in1 = 2 * ks + 1 < p.katoms;      // the second K atom of an odd K / 128 is zeros
                for (int r = lane; r < rows; r += 32) {
                    const uint8_t* src = p.sfb + sf_row_offset(n0 + r, p.sfb_tc, p.katoms, p.katoms_tc) + 2 * ks * b_step;
                    const uint32_t dst = sf + 1024 + sf_smem_offset(r);
                    cp_async4(dst, src, true);
                    cp_async4(dst + 1024, in1 ? src + b_step : src, in1);
                }
                for (int r = lane; r < p.M; r += 32) {
                    const uint8_t* src = p.sfa + sf_row_offset(r, p.sfa_tc, p.katoms, p.katoms_tc) + 2 * ks * a_step;
                    const uint32_t dst = sf + sf_smem_offset(r);
                    cp_async4(dst, src, true);
                    cp_async4(dst + 512, in1 ? src + a_step : src, in1);
                }
                asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
                fence_proxy_async_smem();                    // tcgen05.cp reads these generic-proxy writes
                __syncwarp();
                if (lane == 0) mbar_arrive(full_bar(s));
                s += kStagers;
                if (s >= p.stages) { s -= p.stages; ph ^= 1; }
            }
            i -= kstages;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (*abort_flag) {
            const uint64_t t0 = globaltimer_ns();
            while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

#undef TILE_WIDTH
#undef TILE_COL0

}  // namespace

// Host side: called by gemm_mxfp4_impl for M <= 64, batch == 1, N % 16 == 0 (arguments already validated).
int launch_gemm_mxfp4_skinny(const void* A, const void* B, void* C, const void* sfa, const void* sfb, bool sfa_tc, bool sfb_tc,
                             const void* c_a, const void* c_b, int64_t M, int64_t N, int64_t K, uint32_t* status, cudaStream_t st) {
    const int sms = sm_count();
    HKB_REQUIRE(sms > 0, HKB_ERR_CUDA, "no CUDA device");
    SkinnyMxParams p{};
    p.M = (int)M; p.N = (int)N; p.K = (int)K;
    p.katoms = (int)(K / 128); p.katoms_tc = (p.katoms + 1) & ~1;
    p.sfa = (const uint8_t*)sfa; p.sfb = (const uint8_t*)sfb; p.sfa_tc = sfa_tc; p.sfb_tc = sfb_tc;
    p.C = (__nv_bfloat16*)C; p.c_a = (const __nv_bfloat16*)c_a; p.c_b = (const __nv_bfloat16*)c_b; p.status = status;
    p.a_box_rows = (int)((M + 7) / 8 * 8);
    p.a_bytes = (p.a_box_rows * 128 + 1023) / 1024 * 1024;
    const int64_t units = N / 16;
    const int64_t rounds = (units + (int64_t)kMaxUnits * sms - 1) / ((int64_t)kMaxUnits * sms);
    p.tiles = (int)(units < rounds * sms ? units : rounds * sms);
    p.base = (int)(units / p.tiles);
    p.rem = (int)(units % p.tiles);
    const int maxw = p.base + (p.rem ? 1 : 0);
    HKB_REQUIRE(maxw >= 1 && maxw <= kMaxUnits, HKB_ERR_UNSUPPORTED, "gemm_mxfp4 (skinny): internal tile width %d out of range", maxw);
    p.sf_off = p.a_bytes + maxw * 2048;
    p.stage_bytes = p.sf_off + kSfBytes;
    p.stages = (kSmemLimit - 1024 - kBarBytes - kTailPad) / p.stage_bytes;
    if (p.stages > kMaxStages) p.stages = kMaxStages;
    HKB_REQUIRE(p.stages >= kStagers, HKB_ERR_UNSUPPORTED, "gemm_mxfp4 (skinny): not enough shared memory");
    p.rot = 17;      // as in the FP8 kernel
    const int smem = 1024 + kBarBytes + p.stages * p.stage_bytes + kTailPad;
    CUtensorMap tmA, tmB128, tmB64, tmB16;
    int rc = make_tmap_bytes(&tmA, A, (uint64_t)K / 2, (uint64_t)M, 1, (uint32_t)p.a_box_rows);
    if (rc != HKB_OK) return rc;
    rc = make_tmap_bytes(&tmB128, B, (uint64_t)K / 2, (uint64_t)N, 1, 128);
    if (rc != HKB_OK) return rc;
    rc = make_tmap_bytes(&tmB64, B, (uint64_t)K / 2, (uint64_t)N, 1, 64);
    if (rc != HKB_OK) return rc;
    rc = make_tmap_bytes(&tmB16, B, (uint64_t)K / 2, (uint64_t)N, 1, 16);
    if (rc != HKB_OK) return rc;
    // the limit is the kernel's, not the call's: every call sets the same one, whatever its own size (calls may overlap)
    HKB_CUDA(cudaFuncSetAttribute(gemm_mxfp4_skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    const int grid = p.tiles < sms ? p.tiles : sms;
    HKB_CUDA(launch_dependent(true, gemm_mxfp4_skinny_kernel, grid, 192 + 32 * kStagers, smem, 0, st, tmA, tmB128, tmB64, tmB16, p));
    return check_launch("gemm_mxfp4_skinny_kernel");
}

}  // namespace hkb
