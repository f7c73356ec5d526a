// Block-scale FP8 GEMM for skinny M (decode shapes, M <= 32): C[m,n] = sum_kb (A @ B^T)[kb] * sa[m,kb] * sb[kb,n/128],
// optionally c_a * that + c_b.
//
// The weight stream B[N,K] should bound it.  The block-scale kernel of gemm_fp8.cu does not get there: 128-column tiles
// leave SMs idle (N = 14336: 112 tiles on 148 SMs), its TMA fetches 128 rows of A of which M exist, and all accumulators
// of up to 32 tokens sit in the registers of one warp.  So the operands trade places:
//
//  * The weights are the MMA's 128 rows, the tokens (16 or 32) its N columns.  Eight epilogue warps promote a partial
//    product with one weight row and half of the tokens per thread.
//  * N is cut into 16-row units that are dealt out as (rounds) x (number of SMs) tiles of up to 128 rows; a tile's rows
//    come with ONE TMA box of exactly that height (two tensor maps: base and base + 1 units).  A tile may straddle two
//    128-row scale groups: each thread picks its row's group.
//  * Staging warps transpose the activation scales, eight K blocks at a time, into shared memory ([K block][token]), where
//    the epilogue reads them as broadcasts.
//  * What bounds it is the MMA thread and the hand-off, at about 0.3 us per K block and tile with one K block per
//    stage and two commits for each.  So a stage holds two K blocks, one commit publishes both partial products, and the
//    epilogue returns the operands: 24 x 14336 x 4096 takes 16.2 us, 18.0 with one K block per stage (and 20.3 with four
//    instead of eight epilogue warps; the MMAs of two K blocks interleaved: no difference).
//
// Every K block is promoted in order with the same fused multiply-adds as in the large kernel, so the two give the same
// bits.  Cold L2, us, large kernel / this one: 24 x 14336 x 4096 24.8 / 16.2, 32 x 28672 x 8192 53.8 / 44.7 (5.3 TB/s),
// 16 x 57344 x 4096 75.2 / 39.5 (6.0 TB/s), 32 x 1024 x 8192 26.8 / 20.3, 8 x 4096 x 4096 16.0 / 11.3, 1 x 1024 x 1024
// 7.9 / 6.0.  With multiply-add, quantizer included: 17 x 1024 x 1024 19.5 / 13.3, 17 x 4096 x 4096 27.6 / 19.5,
// 17 x 28672 x 8192 78.9 / 62.5 (c_a and c_b loaded token by token behind the stores instead: 21.5, 27.7, 76.8).  With 64
// tokens the epilogue's scale reads take over (64 x 28672 x 8192 57.4 / 64.6): those stay there.
//
// Roles: warp 0 TMA producer, warp 1 TMEM allocator + MMA issuer, warps 2-9 epilogue, warps 10-11 scale staging.  Bounded
// waits and teardown as in gemm_fp8.cu.
#include "tc_common.cuh"

namespace hkb {
namespace {

constexpr int kMaxStages = 16;
constexpr int kStep = 2;                  // K blocks per pipeline stage, hand-off and commit
constexpr int kAccs = 8;                  // accumulator sets in TMEM, kStep partial products of 32 columns each
constexpr int kSlots = 4;                 // ring of staged scales
constexpr int kChunk = 8;                 // K blocks per slot
constexpr int kPitch = 36;                // floats per K block: 32 token scales, then the weight scales of two groups
constexpr int kSlotBytes = kChunk * kPitch * 4;
constexpr int kHeadBytes = 1024 * ((1024 + kSlots * kSlotBytes + 1023) / 1024);      // barriers (first KB), then the scale ring
constexpr int kTailPad = 16 * 1024;       // the MMA reads 128 weight rows from every stage base
constexpr int kSmemLimit = 232448;        // 227 KB
constexpr int kMaxUnits = 8;              // 128 weight rows
constexpr int kEpiWarps = 8;             // two per TMEM lane quarter, half of the token columns each
constexpr int kThreads = 32 * (4 + kEpiWarps);

struct BsSkinnyParams {
    int M, N, K;
    int64_t ldc;
    int a_box_rows;                       // rows of A fetched per stage (multiple of 8, <= 32)
    int tiles, base, rem;                 // tile t is base + (t < rem) units high and starts at unit t*base + min(t, rem)
    int stages, sub_bytes, a_off;         // one K block inside a stage; its activation rows
    const float* sa;
    const float* sb;
    __nv_bfloat16* C;
    const __nv_bfloat16* c_a;             // fused multiply-add (both [M, N]), or null
    const __nv_bfloat16* c_b;
    uint32_t* status;
};

// 8 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
#define TILE_UNITS(t) (p.base + ((t) < p.rem ? 1 : 0))
#define TILE_ROW0(t) (((t) * p.base + min((t), p.rem)) * 16)

// NT: token columns (16 or 32).
template <int NT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_fp8_blockscale_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB0,
                                  const __grid_constant__ CUtensorMap tmB1, const BsSkinnyParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t bar_base = smem_u32(smem);
    const uint32_t ring_base = bar_base + kHeadBytes;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + kAccs + a); };
    auto sfull_bar = [&](int i) { return bar_base + 8u * (2 * kMaxStages + 2 * kAccs + i); };
    auto sempty_bar = [&](int i) { return bar_base + 8u * (2 * kMaxStages + 2 * kAccs + kSlots + i); };
    constexpr int kNumBars = 2 * kMaxStages + 2 * kAccs + 2 * kSlots;
    static_assert(kNumBars * 8 + 8 <= 1024, "barrier area");
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + kNumBars * 8);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    float* const scales = reinterpret_cast<float*>(smem + 1024);          // [kSlots][kChunk][kPitch]
    constexpr uint32_t TMEM_COLS = 512;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int kblocks = p.K / 128;
    const int ksteps = (kblocks + kStep - 1) / kStep;       // an odd last block is followed by zero-filled data and zero scales
    const uint32_t stage_bytes = kStep * p.sub_bytes;
    const int nchunks = (kblocks + kChunk - 1) / kChunk;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < kAccs; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), kEpiWarps);
        }
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(sfull_bar(i), 1);
            mbar_init(sempty_bar(i), kEpiWarps);
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
            prefetch_tmap(&tmB0);
            prefetch_tmap(&tmB1);
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
                const CUtensorMap* const tmB = t < p.rem ? &tmB1 : &tmB0;
                const int n0 = TILE_ROW0(t);
                const uint32_t stage_tx = kStep * ((uint32_t)p.a_box_rows * 128 + (uint32_t)TILE_UNITS(t) * 2048);
                for (int ks = 0; ks < ksteps; ++ks) {
                    if (!mbar_wait(empty_bar(s), ph ^ 1, abort_flag, p.status, kErrWaitProducer)) { ok = false; break; }
                    mbar_arrive_expect_tx(full_bar(s), stage_tx);
                    const uint32_t st = ring_base + s * stage_bytes;
#pragma unroll
                    for (int i = 0; i < kStep; ++i) {
                        tma_load_3d(st + i * p.sub_bytes, tmB, full_bar(s), (ks * kStep + i) * 128, n0, 0);
                        tma_load_3d(st + i * p.sub_bytes + p.a_off, &tmA, full_bar(s), (ks * kStep + i) * 128, 0, 0);
                    }
                    if (++s == p.stages) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t IDESC = idesc_f8(128, NT);
            int s = 0;
            uint32_t ph = 0;
            int acc = 0;
            uint32_t acc_ph = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
                for (int ks = 0; ks < ksteps; ++ks) {
                    if (!mbar_wait(full_bar(s), ph, abort_flag, p.status, kErrWaitMma)) { ok = false; break; }
                    if (!mbar_wait(tempty_bar(acc), acc_ph ^ 1, abort_flag, p.status, kErrWaitMma)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t st = ring_base + s * stage_bytes;
                    const uint64_t dw = smem_desc_sw128(st);
                    const uint64_t dx = smem_desc_sw128(st + p.a_off);
                    const uint64_t sub = (uint64_t)(p.sub_bytes >> 4);
                    const uint32_t d = tmem_base + acc * (kStep * 32);
#pragma unroll
                    for (int i = 0; i < kStep; ++i)
#pragma unroll
                        for (int k = 0; k < 4; ++k) mma_f8(d + i * 32, dw + i * sub + (uint64_t)(k * 2), dx + i * sub + (uint64_t)(k * 2), IDESC, k != 0);
                    tc_commit(tfull_bar(acc));              // the only commit: the epilogue hands the stage back
                    if (++acc == kAccs) { acc = 0; acc_ph ^= 1; }
                    if (++s == p.stages) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp < 2 + kEpiWarps) {
        // ================= epilogue: one weight row per thread =================
        constexpr int NC = NT / 2;                           // token columns of this warp: col0 .. col0 + NC - 1
        const int col0 = ((warp - 2) >> 2) * NC;
        const int quarter = warp & 3;
        const int row_in_tile = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        int acc = 0, slot = 0, s = 0;
        uint32_t acc_ph = 0, slot_ph = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
            const int rows = TILE_UNITS(t) * 16;
            const int n0 = TILE_ROW0(t);
            const bool row_ok = row_in_tile < rows;
            const bool warp_has_rows = quarter * 32 < rows;              // warp-uniform
            const int n = n0 + (row_ok ? row_in_tile : 0);
            const int group = (n >> 7) - (n0 >> 7);                      // 0 or 1
            if (p.c_a && warp_has_rows && col0 + (lane & (NC - 1)) < p.M) {      // this warp's part of c_a and c_b, into L2
                const int64_t off = (int64_t)(col0 + (lane & (NC - 1))) * p.N + n0 + quarter * 32;
                asm volatile("prefetch.global.L2 [%0];" ::"l"((lane < 16 ? p.c_a : p.c_b) + off));
            }
            float2 acc2[NC / 2];
#pragma unroll
            for (int j = 0; j < NC / 2; ++j) acc2[j] = make_float2(0.0f, 0.0f);
            for (int ch = 0; ch < nchunks && ok; ++ch) {
                if (!__all_sync(0xFFFFFFFFu, mbar_wait(sfull_bar(slot), slot_ph, abort_flag, p.status, kErrWaitEpilogue))) { ok = false; break; }
                const int ks_end = min(ksteps - ch * (kChunk / kStep), kChunk / kStep);
                for (int kk = 0; kk < ks_end; ++kk) {
                    const float* const sc = scales + (slot * kChunk + kk * kStep) * kPitch;
                    // the scales come before the wait, so that their latency passes with it
                    float2 f[kStep][NC / 2];
#pragma unroll
                    for (int i = 0; i < kStep; ++i) {
                        const float sb = sc[i * kPitch + 32 + group];
                        const float2 sb2 = make_float2(sb, sb);
#pragma unroll
                        for (int j = 0; j < NC; j += 4) {
                            const float4 s4 = *reinterpret_cast<const float4*>(sc + i * kPitch + col0 + j);
                            f[i][j / 2] = __fmul2_rn(make_float2(s4.x, s4.y), sb2);
                            f[i][j / 2 + 1] = __fmul2_rn(make_float2(s4.z, s4.w), sb2);
                        }
                    }
                    if (!__all_sync(0xFFFFFFFFu, mbar_wait(tfull_bar(acc), acc_ph, abort_flag, p.status, kErrWaitEpilogue))) { ok = false; break; }
                    if (warp == 2 && lane == 0) mbar_arrive(empty_bar(s));       // these MMAs are done with their operands
                    if (++s == p.stages) s = 0;
                    tc_fence_after();
                    uint32_t r[kStep][NC];
                    if (warp_has_rows) {
                        const uint32_t t_addr = tmem_base + lane_addr + acc * (kStep * 32) + col0;
#pragma unroll
                        for (int i = 0; i < kStep; ++i)
#pragma unroll
                            for (int c = 0; c < NC; c += 16) {
                                if constexpr (NC % 16) tmem_ld8(t_addr + i * 32 + c, r[i] + c);
                                else tmem_ld16(t_addr + i * 32 + c, *reinterpret_cast<uint32_t(*)[16]>(r[i] + c));
                            }
                        tmem_ld_wait();
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty_bar(acc));
                    if (++acc == kAccs) { acc = 0; acc_ph ^= 1; }
                    if (warp_has_rows) {
#pragma unroll
                        for (int i = 0; i < kStep; ++i)
#pragma unroll
                            for (int j = 0; j < NC; j += 2)
                                acc2[j / 2] = __ffma2_rn(make_float2(__uint_as_float(r[i][j]), __uint_as_float(r[i][j + 1])), f[i][j / 2], acc2[j / 2]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(sempty_bar(slot));
                if (++slot == kSlots) { slot = 0; slot_ph ^= 1; }
            }
            if (ok && row_ok) {
                float v[NC];
#pragma unroll
                for (int j = 0; j < NC; ++j) v[j] = (j & 1) ? acc2[j / 2].y : acc2[j / 2].x;
                if (p.c_a) {
                    // All loads go out before the first store: C may be c_a or c_b, so the compiler cannot move them up, and one
                    // round trip per token is longer than the whole K loop of a small layer.
                    __nv_bfloat16 ca[NC], cb[NC];
#pragma unroll
                    for (int j = 0; j < NC; ++j) {
                        const int64_t off = (int64_t)min(col0 + j, p.M - 1) * p.N + n;
                        ca[j] = p.c_a[off];
                        cb[j] = p.c_b[off];
                    }
#pragma unroll
                    for (int j = 0; j < NC; ++j) v[j] = __fmaf_rn(__bfloat162float(ca[j]), v[j], __bfloat162float(cb[j]));
                }
#pragma unroll
                for (int j = 0; j < NC; ++j)
                    if (col0 + j < p.M) p.C[(int64_t)(col0 + j) * p.ldc + n] = __float2bfloat16_rn(v[j]);
            }
        }
    } else {
        // ================= scale staging: warp g fills every second slot =================
        const int g = warp - 2 - kEpiWarps;
        const int nsb = p.N / 128;
        const bool vec = (kblocks & 3) == 0 && (reinterpret_cast<uintptr_t>(p.sa) & 15) == 0;
        int slot = g, ch = g;                                // ch: chunk of the tile, in the epilogue's order
        uint32_t ph = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
            const int g0 = TILE_ROW0(t) >> 7;
            for (; ch < nchunks; ch += 2) {
                const int kb0 = ch * kChunk;
                const int kn = min(kblocks - kb0, kChunk);
                float v[kChunk];
                const float* const src = p.sa + (int64_t)lane * kblocks + kb0;
#pragma unroll
                for (int k = 0; k < kChunk; k += 4) {
                    if (lane < p.M && vec && k < kn) {       // kblocks % 4 == 0: whole vectors
                        const float4 f = __ldg(reinterpret_cast<const float4*>(src + k));
                        v[k] = f.x; v[k + 1] = f.y; v[k + 2] = f.z; v[k + 3] = f.w;
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) v[k + i] = (lane < p.M && k + i < kn) ? __ldg(src + k + i) : 0.0f;
                    }
                }
                const int wk = lane >> 1, wg = min(g0 + (lane & 1), nsb - 1);
                const float wsc = wk < kn ? __ldg(p.sb + (int64_t)(kb0 + wk) * nsb + wg) : 0.0f;
                if (!__all_sync(0xFFFFFFFFu, mbar_wait(sempty_bar(slot), ph ^ 1, abort_flag, p.status, kErrWaitProducer))) { ok = false; break; }
                float* const dst = scales + slot * kChunk * kPitch;
#pragma unroll
                for (int k = 0; k < kChunk; ++k) dst[k * kPitch + lane] = v[k];
                if (wk < kChunk) dst[wk * kPitch + 32 + (lane & 1)] = wsc;
                __syncwarp();
                if (lane == 0) mbar_arrive(sfull_bar(slot));
                slot += 2;
                if (slot >= kSlots) { slot -= kSlots; ph ^= 1; }
            }
            ch -= nchunks;
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

#undef TILE_UNITS
#undef TILE_ROW0

template <int NT>
int launch(const CUtensorMap& tmA, const CUtensorMap& tmB0, const CUtensorMap& tmB1, const BsSkinnyParams& p, int smem, int grid, cudaStream_t st) {
    // the limit is the kernel's, not the call's: every call sets the same one, whatever its own size (calls may overlap)
    HKB_CUDA(cudaFuncSetAttribute(gemm_fp8_blockscale_skinny_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    HKB_CUDA(launch_dependent(true, gemm_fp8_blockscale_skinny_kernel<NT>, grid, kThreads, smem, 0, st, tmA, tmB0, tmB1, p));
    return check_launch("gemm_fp8_blockscale_skinny_kernel");
}

}  // namespace

// Host side: called by gemm_fp8_blockscale_impl for M <= 32 and 128-column weight-scale groups (arguments already validated).
int launch_gemm_fp8_blockscale_skinny(const void* A, const void* B, void* C, const float* sa, const float* sb, const void* c_a, const void* c_b,
                                      int64_t M, int64_t N, int64_t K, int64_t ldc, uint32_t* status, cudaStream_t st) {
    const int sms = sm_count();
    HKB_REQUIRE(sms > 0, HKB_ERR_CUDA, "no CUDA device");
    BsSkinnyParams p{};
    p.M = (int)M; p.N = (int)N; p.K = (int)K; p.ldc = ldc;
    p.sa = sa; p.sb = sb; p.C = (__nv_bfloat16*)C; p.c_a = (const __nv_bfloat16*)c_a; p.c_b = (const __nv_bfloat16*)c_b; p.status = status;
    p.a_box_rows = (int)((M + 7) / 8 * 8);
    const int nt = (int)((M + 15) / 16 * 16);
    const int64_t units = N / 16;
    const int64_t rounds = (units + (int64_t)kMaxUnits * sms - 1) / ((int64_t)kMaxUnits * sms);
    p.tiles = (int)(units < rounds * sms ? units : rounds * sms);
    p.base = (int)(units / p.tiles);
    p.rem = (int)(units % p.tiles);
    const int maxu = p.base + (p.rem ? 1 : 0);
    HKB_REQUIRE(maxu >= 1 && maxu <= kMaxUnits, HKB_ERR_UNSUPPORTED, "gemm_fp8_blockscale (skinny): internal tile height %d out of range", maxu);
    p.a_off = maxu * 2048;
    p.sub_bytes = p.a_off + nt * 128;
    p.stages = (kSmemLimit - 1024 - kHeadBytes - kTailPad) / (kStep * p.sub_bytes);
    if (p.stages > kMaxStages) p.stages = kMaxStages;
    const int smem = 1024 + kHeadBytes + p.stages * kStep * p.sub_bytes + kTailPad;
    CUtensorMap tmA, tmB0, tmB1;
    int rc = make_tmap_bytes(&tmA, A, (uint64_t)K, (uint64_t)M, 1, (uint32_t)p.a_box_rows);
    if (rc != HKB_OK) return rc;
    rc = make_tmap_bytes(&tmB0, B, (uint64_t)K, (uint64_t)N, 1, (uint32_t)p.base * 16);
    if (rc != HKB_OK) return rc;
    rc = make_tmap_bytes(&tmB1, B, (uint64_t)K, (uint64_t)N, 1, (uint32_t)maxu * 16);
    if (rc != HKB_OK) return rc;
    const int grid = p.tiles < sms ? p.tiles : sms;
    if (nt == 16) return launch<16>(tmA, tmB0, tmB1, p, smem, grid, st);
    return launch<32>(tmA, tmB0, tmB1, p, smem, grid, st);
}

}  // namespace hkb
