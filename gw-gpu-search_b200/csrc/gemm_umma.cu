// Reconstruction GEMM with fused |z|^2 and blocked argmax on the tcgen05 tensor cores (sm_100a).
//
// Replaces fp_gemm.gemm_absmax / fused_peaks (pipeline/fp_gemm.py:14-44): z_re = Are @ Z, z_im = Aim @ Z; per
// template row and per 128-sample block the maximum of z_re^2 + z_im^2 and its first sample index. The reference
// writes one (max, index) per block; here a row can also be reduced over `group` consecutive blocks (a 1 s cluster
// window is 16 blocks at 2048 Hz), which fuses the window reduction of fp_filter.py:745-746 into the epilogue.
//
// Design (one persistent CTA per SM, 10 warps):
//   warp 0      TMA producer: loads the whole A operand once (Are/Aim rows of up to two 128-row M blocks, kept
//               resident in shared memory), then streams Z tiles of 128 samples x K through a ring of stages.
//   warp 1      MMA issuer: one elected thread issues tcgen05.mma (M=128, N=128, K=16 steps) into TMEM. Work item =
//               (time tile, M block); accumulators for re and im sit in 256 TMEM columns, double buffered (512).
//   warps 2-9   epilogue: two groups of four warps, group g takes the items of accumulator buffer g (every other
//               item; with two M blocks, always M block g), so a group has two items' time for one and no barrier per
//               item. A warp reads its 32 rows' re and im by tcgen05.ld, 32 samples at a time, the next 32 in flight
//               while these are compared; the maximum runs as four chains of eight (one chain of 32 compares waits for
//               its own latency: it, and not the tensor cores, set the time of an item). Only (max, index) per row and
//               output group reaches global memory.
// Work split: gridDim.x CTAs (or, where whole groups would divide unevenly, pairs of CTAs) take contiguous runs of
// output groups; the two CTAs of a pair (a cluster) halve their run at a tile, and a group cut there is merged through
// distributed shared memory at the end. 448 windows over 148 CTAs are 3.03 each, 4 at most; over 74 pairs 7 for two.
// Measured with the warp-wide issue loop below: 256 x 64 split bf16 by 917,504 samples, 1 s windows, 247 -> 159 us a call
// (209 with a one-lane loop; kernel 141, 1,282 TFLOP/s issued); 1,024 x 128 fp16 by 2^20, 636 -> 511 (615; 1,266).
// Operands: A is K-major (row = template, K contiguous), Z is MN-major (K rows, samples contiguous); both are staged
// by TMA with the 128-byte swizzle. No multicast. Every wait is bounded (one second) and records GWB_ERR_TIMEOUT.
#include "common.cuh"

namespace gwb {
namespace {

constexpr int kTile = 128;                      // samples per block (the reference's BN)
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + 32 * kEpiWarps;   // 320
constexpr int kATileBytes = 128 * 128;          // 128 rows x 64 two-byte elements
constexpr int kTmemCols = 512;

enum Form { kF16 = 0, kBF16x3 = 1 };

struct __align__(64) UmmaArgs {
    CUtensorMap tA[4];   // re (hi), im (hi), re lo, im lo
    CUtensorMap tZ[2];   // Z (hi), Z lo
    float* V;
    int32_t* I;
    long long ldv;
    long long Tn;
    int M, K, ntiles, group, nout, stages, pair;
    DeviceError* err;
};

template <int FORM>
struct FormCfg {
    static constexpr int NA = FORM == kF16 ? 2 : 4;      // A tiles per (M block, K chunk)
    static constexpr int NZ = FORM == kF16 ? 1 : 2;      // Z operands per stage
    static constexpr int NPROD = FORM == kF16 ? 1 : 3;   // products accumulated per (re|im)
    static constexpr uint32_t FMT = FORM == kF16 ? 0u : 1u;
};

struct SmemLayout {
    uint32_t a_off, z_off, stage_bytes, x_off, bar_off, total;
};

__host__ __device__ inline SmemLayout smem_layout(int na, int nz, int nkc, int K, int stages) {
    SmemLayout L;
    L.a_off = 0;
    L.z_off = 2u * na * nkc * kATileBytes;
    L.stage_bytes = (uint32_t)nz * 2u * (uint32_t)K * 128u;
    L.x_off = L.z_off + (uint32_t)stages * L.stage_bytes;
    L.bar_off = L.x_off + 3u * 2u * 128u * 8u;
    L.total = L.bar_off + (uint32_t)(2 * stages + 6) * 8u + 16u;
    return L;
}

template <int FORM>
__global__ void __launch_bounds__(kThreads, 1) umma_absmax_kernel(const __grid_constant__ UmmaArgs args) {
    using C = FormCfg<FORM>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);

    const int K = args.K, nkc = K / 64, S = args.stages;
    const SmemLayout L = smem_layout(C::NA, C::NZ, nkc, K, S);
    uint8_t* sA = smem + L.a_off;
    uint8_t* sZ = smem + L.z_off;
    // maxima that cross warps: [0], [1] the two epilogue groups' (one M block), by window parity; [2] the cut window's
    float (*xv)[2][128] = reinterpret_cast<float (*)[2][128]>(smem + L.x_off);
    int (*xi)[2][128] = reinterpret_cast<int (*)[2][128]>(smem + L.x_off + 3072);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L.bar_off);
    uint64_t* full = bars;
    uint64_t* empty = bars + S;
    uint64_t* tfull = bars + 2 * S;
    uint64_t* tempty = tfull + 2;
    uint64_t* barA = tempty + 2;
    uint64_t* done = barA + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * 256;
    const int MBe = min(2, (args.M - m0 + 127) / 128);
    const int pair = args.pair, rank = pair ? (int)(blockIdx.x & 1) : 0;
    const int runs = (int)gridDim.x >> pair, run = (int)blockIdx.x >> pair;
    const long long o0 = (long long)run * args.nout / runs;
    const long long o1 = (long long)(run + 1) * args.nout / runs;
    const int r_begin = (int)(o0 * args.group);
    const int r_end = (int)min(o1 * (long long)args.group, (long long)args.ntiles);
    const int r_mid = r_begin + (r_end - r_begin + 1) / 2;            // where a pair's run is cut
    const int t_begin = rank ? r_mid : r_begin, t_end = pair && !rank ? r_mid : r_end;
    const int ntl = t_end - t_begin;
    // the cut falls inside a group: rank 1 hands its part's maximum to rank 0
    const bool cut = pair && r_mid < r_end && r_mid % args.group != 0;
    if (!pair && (ntl <= 0 || MBe <= 0)) return;   // uniform across the CTA
    const bool live = ntl > 0 && MBe > 0;          // a pair's CTA without tiles still meets the other at the end

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], kEpiWarps / 2);
        }
        mbar_init(barA, 1);
        mbar_init(done, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (!live) {
    } else if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            for (int a = 0; a < C::NA; ++a) prefetch_tmap(&args.tA[a]);
            for (int z = 0; z < C::NZ; ++z) prefetch_tmap(&args.tZ[z]);
            mbar_arrive_expect_tx(barA, (uint32_t)(MBe * C::NA * nkc * kATileBytes));
            for (int mb = 0; mb < MBe; ++mb)
                for (int a = 0; a < C::NA; ++a)
                    for (int kc = 0; kc < nkc; ++kc)
                        tma_load_2d(sA + ((mb * C::NA + a) * nkc + kc) * kATileBytes, &args.tA[a], barA, kc * 64,
                                    m0 + mb * 128);
            for (int i = 0; i < ntl; ++i) {
                const int s = i % S;
                const uint32_t n = (uint32_t)(i / S);
                if (*abort_flag) break;
                if (!mbar_wait_bounded(&empty[s], (n & 1) ^ 1)) {
                    record_error(args.err, GWB_ERR_TIMEOUT, 101, blockIdx.x, i);
                    *abort_flag = 1;
                    break;
                }
                mbar_arrive_expect_tx(&full[s], L.stage_bytes);
                const int x = (t_begin + i) * kTile;
                for (int z = 0; z < C::NZ; ++z)
                    for (int h = 0; h < 2; ++h)
                        tma_load_2d(sZ + s * L.stage_bytes + (z * 2 + h) * K * 128, &args.tZ[z], &full[s],
                                    x + 64 * h, 0);
            }
            // make sure no copy is still landing in shared memory when the CTA exits
            mbar_wait_bounded(barA, 0);
            for (int s = 0; s < S && s < ntl; ++s) {
                const int nfill = (ntl - s + S - 1) / S;
                mbar_wait_bounded(&full[s], (uint32_t)((nfill - 1) & 1));
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp runs the loop and one elected lane issues: descriptors, TMEM addresses and loop state are then
        // warp-uniform and stay in the uniform registers that tcgen05.mma reads (in a one-lane branch each operand of
        // each MMA was moved there first, and the issue loop, not the MMAs, set the time of a tile).
        const bool el = elect_lane();
        const uint32_t tm = (uint32_t)warp_uniform((int)tmem);
        const uint32_t idesc = instr_desc(128, 128, C::FMT, C::FMT, 0, 1);
        const uint32_t a_base = smem_u32(sA), z_base = smem_u32(sZ);
        bool ok = mbar_wait_warp(barA, 0);
        if (!ok) {
            record_error(args.err, GWB_ERR_TIMEOUT, 102, blockIdx.x, 0);
            *abort_flag = 1;
        }
        tc_fence_after();
        int s = 0;
        uint32_t ph = 0;                                   // stage and its phase
        for (int i = 0; i < ntl && ok; ++i) {
            ok = __all_sync(0xffffffffu, *abort_flag == 0) && mbar_wait_warp(&full[s], ph);
            if (!ok) {
                record_error(args.err, GWB_ERR_TIMEOUT, 103, blockIdx.x, i);
                *abort_flag = 1;
                break;
            }
            tc_fence_after();
            for (int mb = 0; mb < MBe; ++mb) {
                const int j = i * MBe + mb, b = j & 1;
                ok = mbar_wait_warp(&tempty[b], (uint32_t)(((j >> 1) & 1) ^ 1));
                if (!ok) {
                    record_error(args.err, GWB_ERR_TIMEOUT, 104, blockIdx.x, i);
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after();
                for (int ri = 0; ri < 2; ++ri) {
                    const uint32_t d = tm + (uint32_t)(b * 256 + ri * 128);
                    uint32_t acc = 0;
#pragma unroll
                    for (int pr = 0; pr < C::NPROD; ++pr) {
                        // products: (A hi, Z hi), (A hi, Z lo), (A lo, Z hi)
                        const int a = (pr == 2 ? 2 : 0) + ri;
                        const int z = (pr == 1) ? 1 : 0;
                        // descriptors advance by K steps of 16: 32 bytes of a 64-wide A box, 2048 of Z
                        uint64_t ad = smem_desc(a_base + (mb * C::NA + a) * nkc * kATileBytes, 16, 1024, 2);
                        uint64_t bd = smem_desc(z_base + s * L.stage_bytes + (z * 2) * K * 128, (uint32_t)K * 128u, 1024,
                                                2);
                        for (int kc = 0; kc < nkc; ++kc) {
                            if (el) {
                                umma_f16(d, ad, bd, idesc, acc);
                                umma_f16(d, ad + (32 >> 4), bd + (2048 >> 4), idesc, 1);
                                umma_f16(d, ad + (64 >> 4), bd + (4096 >> 4), idesc, 1);
                                umma_f16(d, ad + (96 >> 4), bd + (6144 >> 4), idesc, 1);
                            }
                            acc = 1;
                            ad += kATileBytes >> 4;
                            bd += 4 * 2048 >> 4;
                        }
                    }
                }
                if (el) umma_commit(&tfull[b]);
            }
            if (!ok) break;
            if (el) umma_commit(&empty[s]);
            if (++s == S) {
                s = 0;
                ph ^= 1;
            }
        }
        __syncwarp();
        if (el) umma_commit(done);
        __syncwarp();
        mbar_wait_bounded(done, 0);
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        const int q = warp & 3, g = (warp - 2) >> 2;
        const int rl = 32 * q + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(g * 256);
        const int G = args.group;
        // maximum of item j (tile t): waits for the accumulators, frees them once they are in registers
        auto item = [&](int j, int t, float& best, int& bi) {
            best = -1.f;
            bi = 0;
            if (*abort_flag || !mbar_wait_bounded(&tfull[g], (uint32_t)((j >> 1) & 1))) {
                record_error(args.err, GWB_ERR_TIMEOUT, 105, blockIdx.x, j);
                *abort_flag = 1;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty[g]);
                return;
            }
            tc_fence_after();
            const long long left = args.Tn - (long long)t * kTile;     // samples of the tile inside the row
            uint32_t re[2][32], im[2][32];
            tmem_ld_32x32b_x32(lane_base, re[0]);
            tmem_ld_32x32b_x32(lane_base + 128, im[0]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                tmem_ld_wait();
                // tie every value to the wait so no use is scheduled above it
#pragma unroll
                for (int jj = 0; jj < 32; ++jj) asm volatile("" : "+r"(re[c & 1][jj]), "+r"(im[c & 1][jj]));
                if (c < 3) {
                    tmem_ld_32x32b_x32(lane_base + 32 * (c + 1), re[(c + 1) & 1]);
                    tmem_ld_32x32b_x32(lane_base + 128 + 32 * (c + 1), im[(c + 1) & 1]);
                } else {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&tempty[g]);
                }
                if (left >= kTile)
                    best_of_32<true>(re[c & 1], im[c & 1], 32, 32 * c, best, bi);
                else
                    best_of_32<false>(re[c & 1], im[c & 1], (int)min(32ll, max(0ll, left - 32 * c)), 32 * c, best, bi);
            }
            bi += t * kTile;
        };
        // the maximum (wb, wi) of the part of group o that this CTA holds, of M block mb: rank 1's part of a cut group
        // goes to shared memory, rank 0 keeps its own in registers (returns true), all others go out
        auto put = [&](int o, int mb, float wb, int wi) {
            if (cut && o == r_mid / G) {
                if (rank == 0) return true;
                xv[2][mb][rl] = wb;
                xi[2][mb][rl] = wi;
                return false;
            }
            const int row = m0 + mb * 128 + rl;
            if (row < args.M) {
                args.V[(long long)row * args.ldv + o] = wb;
                args.I[(long long)row * args.ldv + o] = wi;
            }
            return false;
        };
        float wb = -2.f;                                   // below any tile's maximum (at least -1)
        int wi = 0;
        bool held = false;                                 // (wb, wi) is rank 0's part of the cut group
        if (MBe == 2) {                                    // group g: M block g of every tile
            for (int i = 0; i < ntl; ++i) {
                const int t = t_begin + i;
                float best;
                int bi;
                item(2 * i + g, t, best, bi);
                if (best > wb) {
                    wb = best;
                    wi = bi;
                }
                if ((t + 1) % G == 0 || t + 1 == t_end) {
                    held = put(t / G, g, wb, wi);
                    if (!held) wb = -2.f;
                }
            }
        } else if (G == 1) {                               // one M block, every tile an output: tiles by parity
            for (int i = g; i < ntl; i += 2) {
                float best;
                int bi;
                item(i, t_begin + i, best, bi);
                put(t_begin + i, 0, best, bi);
            }
        } else {                                           // one M block: the two groups meet at every output
            int par = 0;
            for (int t = t_begin; t < t_end; par ^= 1) {
                const int o = t / G, te = min((o + 1) * G, t_end);
                wb = -2.f;
                wi = 0;
                for (; t < te; ++t) {
                    const int i = t - t_begin;
                    if ((i & 1) != g) continue;
                    float best;
                    int bi;
                    item(i, t, best, bi);
                    if (best > wb) {
                        wb = best;
                        wi = bi;
                    }
                }
                if (g == 1) {
                    xv[par][0][rl] = wb;
                    xi[par][0][rl] = wi;
                }
                named_bar_sync(1, 32 * kEpiWarps);         // the slots take turns: written again two outputs on
                if (g == 0) {
                    const float ob = xv[par][0][rl];
                    const int oi = xi[par][0][rl];
                    if (ob > wb || (ob == wb && oi < wi)) {
                        wb = ob;
                        wi = oi;
                    }
                    held = put(o, 0, wb, wi);
                }
            }
        }
        if (cut) {
            // rank 1's part lies after rank 0's: it replaces only where it is larger
            cluster_sync_all();
            if (held) {
                const int mb = MBe == 2 ? g : 0;
                float ob;
                int oi;
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(ob) : "r"(mapa_shared(smem_u32(&xv[2][mb][rl]), 1)));
                asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(oi) : "r"(mapa_shared(smem_u32(&xi[2][mb][rl]), 1)));
                if (ob > wb) {
                    wb = ob;
                    wi = oi;
                }
                const int row = m0 + mb * 128 + rl;
                if (row < args.M) {
                    args.V[(long long)row * args.ldv + r_mid / G] = wb;
                    args.I[(long long)row * args.ldv + r_mid / G] = wi;
                }
            }
        }
    }
    if (cut) {
        // every thread of both CTAs: the epilogue warps met once above (rank 1's part is in shared memory); all meet
        // again here, so that rank 1 does not leave while its shared memory may be read
        if (!live || warp < 2) cluster_sync_all();
        __syncwarp();
        cluster_sync_all();
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

template <int FORM>
int launch_umma(const uint16_t* const* A, const uint16_t* const* Zp, long long lda, long long ldz, int M, int K,
                long long Tn, int group, float* V, int32_t* I, long long ldv, cudaStream_t stream) {
    using C = FormCfg<FORM>;
    GWB_CHECK_ARG(M > 0 && Tn > 0 && group > 0, GWB_ERR_SHAPE, "fused_peaks: M=%d Tn=%lld group=%d", M, Tn, group);
    GWB_CHECK_ARG(K > 0 && K % 64 == 0 && K <= 256, GWB_ERR_SHAPE, "fused_peaks: K=%d must be a multiple of 64, <= 256",
                  K);
    GWB_CHECK_ARG(lda >= K && ldz >= Tn, GWB_ERR_SHAPE, "fused_peaks: lda=%lld < K or ldz=%lld < Tn", lda, ldz);
    GWB_CHECK_ARG(lda % 8 == 0 && ldz % 8 == 0, GWB_ERR_ALIGN, "fused_peaks: lda=%lld and ldz=%lld must be multiples of 8",
                  lda, ldz);
    for (int a = 0; a < C::NA; ++a)
        GWB_CHECK_ARG(A[a] != nullptr && aligned(A[a], 16), GWB_ERR_ALIGN, "fused_peaks: A operand %d misaligned", a);
    for (int z = 0; z < C::NZ; ++z)
        GWB_CHECK_ARG(Zp[z] != nullptr && aligned(Zp[z], 16), GWB_ERR_ALIGN, "fused_peaks: Z operand %d misaligned", z);
    GWB_CHECK_ARG(V != nullptr && I != nullptr, GWB_ERR_ARG, "fused_peaks: null output");
    const long long ntiles = cdiv(Tn, kTile);
    GWB_CHECK_ARG(ntiles * kTile < (1ll << 31), GWB_ERR_SHAPE, "fused_peaks: Tn too large for int32 indices");
    const long long nout = cdiv(ntiles, group);
    GWB_CHECK_ARG(ldv >= nout, GWB_ERR_SHAPE, "fused_peaks: ldv=%lld < outputs per row %lld", ldv, nout);

    UmmaArgs args;
    memset(&args, 0, sizeof(args));
    const CUtensorMapDataType dt = FORM == kF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    for (int a = 0; a < C::NA; ++a) {
        int r = encode_tmap_2d(&args.tA[a], dt, A[a], (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, 64, 128,
                               CU_TENSOR_MAP_SWIZZLE_128B);
        if (r) return r;
    }
    for (int z = 0; z < C::NZ; ++z) {
        int r = encode_tmap_2d(&args.tZ[z], dt, Zp[z], (uint64_t)Tn, (uint64_t)K, (uint64_t)ldz * 2, 64, (uint32_t)K,
                               CU_TENSOR_MAP_SWIZZLE_128B);
        if (r) return r;
    }
    const int nkc = K / 64;
    const int mgroups = (M + 255) / 256;
    const int max_smem = 227 * 1024;
    int stages = 8;
    while (stages > 1 && smem_layout(C::NA, C::NZ, nkc, K, stages).total + 1024 > (uint32_t)max_smem) --stages;
    {   // the launch table may ask for a shallower Z ring (forms 4: stacked fp16, 5: stacked split bf16; kh = K)
        int pair = 0, st = 0, order = 0;
        if (tune_lookup(FORM == kF16 ? 4 : 5, K, &pair, &st, &order) && st >= 2) stages = std::min(stages, st);
    }
    const uint32_t smem = smem_layout(C::NA, C::NZ, nkc, K, stages).total + 1024;
    GWB_CHECK_ARG(smem <= (uint32_t)max_smem, GWB_ERR_SHAPE, "fused_peaks: K=%d needs %u bytes of shared memory", K,
                  smem);
    args.V = V;
    args.I = I;
    args.ldv = ldv;
    args.Tn = Tn;
    args.M = M;
    args.K = K;
    args.ntiles = (int)ntiles;
    args.group = group;
    args.nout = (int)nout;
    args.stages = stages;
    args.err = device_error_ptr();

    auto kern = umma_absmax_kernel<FORM>;
    GWB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int gx = (int)std::max(1ll, std::min(nout, (long long)std::max(1, num_sms() / mgroups)));
    // pairs of CTAs where whole groups of several tiles would divide unevenly (a CTA would hold 16 or fewer): the run
    // with the most groups then holds at most half a group more than the mean per CTA, not a whole one
    args.pair = group > 1 && gx > 1 && nout <= 16ll * gx && nout % gx != 0;
    if (args.pair) gx &= ~1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gx, mgroups);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = args.pair ? 1 : 0;
    GWB_CUDA(cudaLaunchKernelEx(&cfg, kern, args));
    GWB_LAUNCH_CHECK("umma_absmax_kernel");
    return GWB_OK;
}

}  // namespace
}  // namespace gwb

extern "C" {

int gwb_fused_peaks_f16(const uint16_t* Are, const uint16_t* Aim, long long lda, const uint16_t* Z, long long ldz,
                        int M, int K, long long Tn, int group, float* V, int32_t* I, long long ldv, void* stream) {
    const uint16_t* A[2] = {Are, Aim};
    const uint16_t* Zs[1] = {Z};
    return gwb::launch_umma<gwb::kF16>(A, Zs, lda, ldz, M, K, Tn, group, V, I, ldv, (cudaStream_t)stream);
}

int gwb_fused_peaks_bf16x3(const uint16_t* Are_hi, const uint16_t* Are_lo, const uint16_t* Aim_hi,
                           const uint16_t* Aim_lo, long long lda, const uint16_t* Z_hi, const uint16_t* Z_lo,
                           long long ldz, int M, int K, long long Tn, int group, float* V, int32_t* I,
                           long long ldv, void* stream) {
    const uint16_t* A[4] = {Are_hi, Aim_hi, Are_lo, Aim_lo};
    const uint16_t* Zs[2] = {Z_hi, Z_lo};
    return gwb::launch_umma<gwb::kBF16x3>(A, Zs, lda, ldz, M, K, Tn, group, V, I, ldv, (cudaStream_t)stream);
}

}  // extern "C"
