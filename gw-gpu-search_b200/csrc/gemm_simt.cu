// Plain-fp32 form of the reconstruction GEMM with fused |z|^2 and blocked argmax, on the fp32 pipe.
//
// Same contract as gwb_fused_peaks_f16 (pipeline/fp_gemm.py:14-44 semantics) with fp32 operands: the reference only
// has an fp16 GEMM, so this is the full-precision form that the mixed forms are compared against. Two kernels with the same
// sums: simt_absmax_packed_kernel, which runs (64 template rows x part of an output group of `group` 128-sample blocks per
// CTA of 128 threads, paired FMAs, asynchronous copies), and simt_absmax_kernel, which runs where gwb_f32_set_async(0) asks
// for it or there are more than 65,535 blocks of 64 rows (128 rows x one output group per CTA of 256 threads as 16 x 16).
// In both a thread owns 8 rows x 8 samples for re and im, and K is staged through shared memory 16 at a time.
#include <cooperative_groups.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace gwb {
namespace {

constexpr int BM = 128, BN = 128, BK = 16;

__device__ __forceinline__ void better(float ov, int oi, float& v, int& i) {
    if (ov > v || (ov == v && oi < i)) {
        v = ov;
        i = oi;
    }
}

__global__ void __launch_bounds__(256) simt_absmax_kernel(const float* __restrict__ Are, const float* __restrict__ Aim,
                                                          long long lda, const float* __restrict__ Z, long long ldz,
                                                          int M, int K, long long Tn, int ntiles, int group,
                                                          float* __restrict__ V, int32_t* __restrict__ I,
                                                          long long ldv) {
    __shared__ __align__(16) float sAr[BK][BM];
    __shared__ __align__(16) float sAi[BK][BM];
    __shared__ __align__(16) float sZ[BK][BN];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM;
    const int o = blockIdx.x;
    const int t0 = o * group, t1 = min(t0 + group, ntiles);
    float wb[8];
    int wi[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        wb[i] = -1.f;
        wi[i] = 0;
    }
    for (int t = t0; t < t1; ++t) {
        const long long c0 = (long long)t * BN;
        float ar[8][8], ai[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) ar[i][j] = ai[i][j] = 0.f;
        for (int k0 = 0; k0 < K; k0 += BK) {
            // A tiles: 128 rows x 16 k, stored k-major; each thread moves 8 values of each
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int e = tid + 256 * r;       // 0..2047
                const int row = e >> 4, kk = e & 15;
                const int gr = m0 + row, gk = k0 + kk;
                const bool ok = gr < M && gk < K;
                sAr[kk][row] = ok ? Are[(long long)gr * lda + gk] : 0.f;
                sAi[kk][row] = ok ? Aim[(long long)gr * lda + gk] : 0.f;
            }
            // Z tile: 16 k x 128 samples
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int e = tid + 256 * r;
                const int kk = e >> 7, cc = e & 127;
                const long long gc = c0 + cc;
                const int gk = k0 + kk;
                sZ[kk][cc] = (gk < K && gc < Tn) ? Z[(long long)gk * ldz + gc] : 0.f;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a_r[8], a_i[8], z[8];
                const float4* pr = reinterpret_cast<const float4*>(&sAr[kk][ty * 8]);
                const float4* pi = reinterpret_cast<const float4*>(&sAi[kk][ty * 8]);
                const float4* pz = reinterpret_cast<const float4*>(&sZ[kk][tx * 8]);
                float4 v;
                v = pr[0]; a_r[0] = v.x; a_r[1] = v.y; a_r[2] = v.z; a_r[3] = v.w;
                v = pr[1]; a_r[4] = v.x; a_r[5] = v.y; a_r[6] = v.z; a_r[7] = v.w;
                v = pi[0]; a_i[0] = v.x; a_i[1] = v.y; a_i[2] = v.z; a_i[3] = v.w;
                v = pi[1]; a_i[4] = v.x; a_i[5] = v.y; a_i[6] = v.z; a_i[7] = v.w;
                v = pz[0]; z[0] = v.x; z[1] = v.y; z[2] = v.z; z[3] = v.w;
                v = pz[1]; z[4] = v.x; z[5] = v.y; z[6] = v.z; z[7] = v.w;
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        ar[i][j] = fmaf(a_r[i], z[j], ar[i][j]);
                        ai[i][j] = fmaf(a_i[i], z[j], ai[i][j]);
                    }
            }
            __syncthreads();
        }
        // |z|^2, max and first index per row over this thread's 8 samples, then over the 16 threads of the row
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float best = -1.f;
            int bi = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int cc = tx * 8 + j;
                const float p = (c0 + cc < Tn) ? fmaf(ar[i][j], ar[i][j], ai[i][j] * ai[i][j]) : -1.f;
                if (p > best) {
                    best = p;
                    bi = cc;
                }
            }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, off, 16);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, off, 16);
                better(ob, oi, best, bi);
            }
            const int gi = (int)(c0 + bi);
            if (t == t0 || best > wb[i]) {
                wb[i] = best;
                wi[i] = gi;
            }
        }
    }
    if (tx == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = m0 + ty * 8 + i;
            if (row < M) {
                V[(long long)row * ldv + o] = wb[i];
                I[(long long)row * ldv + o] = wi[i];
            }
        }
    }
}

// The same product, packed and pipelined: the kernel that runs unless gwb_f32_set_async(0) asks for the one above.
// It is bound by the fp32 pipe (128 FMA lanes per SM; 69 TFLOP/s measured with independent FMAs), and what kept the
// one-FMA-per-instruction form at 35 TFLOP/s was the issue of everything else beside the FMAs with two warps per
// scheduler. So:
//  - FMAs go in pairs (fma.rn.f32x2: two samples of a row per instruction, each rounded as fmaf), which halves the
//    issue slots they take and leaves the others for shared-memory reads and the duplicated A values;
//  - operand tiles are copied by cp.async through a ring of AS_ST stages while earlier ones are multiplied (Z in 16-byte
//    copies where ldz and the base allow, else 4-byte ones: the arithmetic is the same);
//  - CTAs of 128 threads own 64 rows, two per SM, so one's barriers and epilogue pass under the other's FMAs and a
//    row count is padded to 64, not 128;
//  - a window is shared out over a cluster of SPL CTAs (each walks its part of the blocks; rank 0 merges the maxima
//    in block order through distributed shared memory), so that the last wave is a quarter of a window long.
// Sums run over k in order with one rounding per FMA, so results are bit-identical to the kernel above.
// Measured, 248 x 192 by 192 x 458,700, 1 s windows: 2,526 -> 1,728 us (50.6 TFLOP/s; 1,759 with each copy's address
// taken anew from its step; 1,935 with pairs along samples, 16 duplicated A values per k; 1,915 with no duplicated value
// but pairs (row, sample), (row + 1, sample + 1) and the crossed ones: three operands of 64 bits an instruction, which the
// register file presumably does not read in its two cycles); 64 templates x 118 rows of K by 475,136 samples: 855 ->
// 326 us (half the rows were padding). The FMA pipe is 78 % busy while a CTA runs; the waits of two warps per scheduler
// for each other's operand steps and the last wave are the rest.
// Pairs run along rows: A lies k-major in shared memory (4-byte copies), so a pair of rows is one register pair as read,
// and only the 8 samples of a k are duplicated, not 16 A values. Thread (tx, ty) owns rows 8 ty .. 8 ty + 7 and samples
// 4 tx + j, 64 + 4 tx + j (j < 4): a warp's A reads are two broadcast float4, its Z reads two runs of 256 bytes.
constexpr int AS_ST = 3, AS_BM = 64, AS_NT = 128, AS_MAXSPL = 4;
constexpr int AS_LD = AS_BM + 4;                 // floats per k of an A tile (k-major; rows on 16-byte boundaries)
constexpr int AS_STAGE = (2 * AS_LD + BN) * BK;  // floats per stage: A re, A im (BK x AS_LD), Z (BK x BN)

// N bytes (16 or 4) to shared memory, zero past the first src_bytes
template <int N>
__device__ __forceinline__ void cp_async_zfill(float* smem, const float* gmem, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (N == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gmem), "r"(src_bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(gmem), "r"(src_bytes) : "memory");
}

using pair32 = unsigned long long;               // two floats, the lower one in the low word

__device__ __forceinline__ pair32 dup(float a) {
    pair32 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ void fma2(pair32& c, pair32 a, pair32 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 unpack(pair32 p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}

template <int SPL, bool VEC>
__global__ void __launch_bounds__(AS_NT, 2) simt_absmax_packed_kernel(
    const float* __restrict__ Are, const float* __restrict__ Aim, long long lda, const float* __restrict__ Z,
    long long ldz, int M, int K, long long Tn, int ntiles, int group, float* __restrict__ V, int32_t* __restrict__ I,
    long long ldv) {
    static_assert(BN == 128 && BK == 16 && AS_BM == 64 && AS_NT == 128, "tile shape");
    extern __shared__ __align__(16) float smf[];
    __shared__ float s_best[AS_BM];
    __shared__ int s_idx[AS_BM];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * AS_BM;
    const int o = blockIdx.x / SPL, rank = blockIdx.x % SPL;
    // this CTA's blocks: its share of the window [o group, min(o group + group, ntiles)); the last ranks may have none
    const int w0 = o * group, w1 = min(w0 + group, ntiles);
    const int share = (group + SPL - 1) / SPL;
    const int t0 = min(w0 + rank * share, w1), t1 = min(t0 + share, w1);
    const int nk = (K + BK - 1) / BK;
    const int nsteps = (t1 - t0) * nk;
    // Copies of the next step's tiles: (lt, lk) is its block and its place along K, ls its stage. A thread copies one k of
    // the rows row0 + 8 r (rows past M are read as the last one: nothing is written for them) and samples zc .. of the
    // k's zk + ZS r; pointers go on by a constant, and k's past K or samples past Tn are zero-filled.
    constexpr int E = VEC ? 4 : 1, ZT = BN / E, ZS = AS_NT / ZT;  // samples per copy; threads and k's per round of copies
    const int ak = tid % BK, row0 = tid / BK, rows = M - m0;
    const int zk = tid / ZT, zc = tid % ZT * E;
    const float* a_re = Are + (long long)(m0 + min(row0, rows - 1)) * lda;
    const float* a_im = Aim + (long long)(m0 + min(row0, rows - 1)) * lda;
    int lt = t0, lk = 0, ls = 0;
    auto load = [&]() {
        float* sA = smf + ls * AS_STAGE;
        const int k0 = lk * BK;
        {
            const int kc = min(k0 + ak, K - 1), nb = k0 + ak < K ? 4 : 0;
            const float* pr = a_re + kc;
            const float* pi = a_im + kc;
            float* d = sA + ak * AS_LD + row0;
#pragma unroll
            for (int r = 0; r < AS_BM * BK / AS_NT; ++r) {       // A: 64 rows x 16 k, transposed
                cp_async_zfill<4>(d + 8 * r, pr, nb);
                cp_async_zfill<4>(d + 8 * r + AS_LD * BK, pi, nb);
                if (row0 + 8 * (r + 1) < rows) {
                    pr += 8 * lda;
                    pi += 8 * lda;
                }
            }
        }
        {
            const long long gc = (long long)lt * BN + zc;
            const int nc = gc < Tn ? (int)min((long long)(4 * E), (Tn - gc) * 4) : 0;
            const float* pz = Z + (nc ? (long long)(k0 + zk) * ldz + gc : 0);
            float* d = sA + 2 * AS_LD * BK + zk * BN + zc;
#pragma unroll
            for (int r = 0; r < BK / ZS; ++r) {                  // Z: 16 k x 128 samples
                const int nb = k0 + zk + ZS * r < K ? nc : 0;
                cp_async_zfill<4 * E>(d + ZS * r * BN, nb ? pz : Z, nb);
                pz += ZS * ldz;
            }
        }
        if (++lk == nk) {
            lk = 0;
            ++lt;
        }
        ls = ls + 1 == AS_ST ? 0 : ls + 1;
    };
    float wb[8];
    int wi[8];
    pair32 ar[4][8], ai[4][8];                   // rows (2 i, 2 i + 1), samples 4 tx + j, 64 + 4 tx + j
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        wb[i] = -2.f;                            // below every block's maximum (at least -1)
        wi[i] = 0;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) ar[i][j] = ai[i][j] = 0ull;
#pragma unroll
    for (int s = 0; s < AS_ST - 1; ++s) {
        if (s < nsteps) load();
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int t = t0, k = 0, st = 0;                   // this step's block, place along K and stage
    for (int step = 0; step < nsteps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(AS_ST - 2) : "memory");
        __syncthreads();                         // this step's tiles are in; every thread is done with step - 1's
        if (step + AS_ST - 1 < nsteps) load();
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* sAr = smf + st * AS_STAGE;
        const float* sAi = sAr + AS_LD * BK;
        const float* sZ = sAi + AS_LD * BK;
        st = st + 1 == AS_ST ? 0 : st + 1;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 z0 = *reinterpret_cast<const float4*>(sZ + kk * BN + 4 * tx);
            const float4 z1 = *reinterpret_cast<const float4*>(sZ + kk * BN + 64 + 4 * tx);
            const pair32 z[8] = {dup(z0.x), dup(z0.y), dup(z0.z), dup(z0.w), dup(z1.x), dup(z1.y), dup(z1.z), dup(z1.w)};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const ulonglong2 r2 = *reinterpret_cast<const ulonglong2*>(sAr + kk * AS_LD + 8 * ty + 4 * h);
                const ulonglong2 i2 = *reinterpret_cast<const ulonglong2*>(sAi + kk * AS_LD + 8 * ty + 4 * h);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    fma2(ar[2 * h][j], r2.x, z[j]);
                    fma2(ar[2 * h + 1][j], r2.y, z[j]);
                    fma2(ai[2 * h][j], i2.x, z[j]);
                    fma2(ai[2 * h + 1][j], i2.y, z[j]);
                }
            }
        }
        if (++k == nk) {
            // |z|^2, max and first index per row over this thread's 8 samples (increasing order), then over the 16
            // threads of the row; then the running window maximum
            const long long c0 = (long long)t * BN;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float best = -1.f;
                int bi = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float2 re = unpack(ar[i / 2][j]), im = unpack(ai[i / 2][j]);
                    const float xr = i & 1 ? re.y : re.x, xi = i & 1 ? im.y : im.x;
                    const int cc = (j < 4 ? 4 * tx + j : 64 + 4 * tx + (j - 4));
                    const float p = (c0 + cc < Tn) ? fmaf(xr, xr, xi * xi) : -1.f;
                    if (p > best) {
                        best = p;
                        bi = cc;
                    }
                }
#pragma unroll
                for (int off = 8; off > 0; off >>= 1) {
                    const float ob = __shfl_xor_sync(0xffffffffu, best, off, 16);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, off, 16);
                    better(ob, oi, best, bi);
                }
                if (best > wb[i]) {
                    wb[i] = best;
                    wi[i] = (int)(c0 + bi);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) ar[i][j] = ai[i][j] = 0ull;
            k = 0;
            ++t;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if constexpr (SPL > 1) {
        // rank 0 takes the other ranks' maxima in block order (a later block replaces only where it is larger)
        if (tx == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                s_best[8 * ty + i] = wb[i];
                s_idx[8 * ty + i] = wi[i];
            }
        }
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        if (rank == 0 && tid < AS_BM && m0 + tid < M) {
            float b = s_best[tid];
            int bi = s_idx[tid];
#pragma unroll
            for (int r = 1; r < SPL; ++r) {
                const float ob = *cl.map_shared_rank(&s_best[tid], r);
                const int oi = *cl.map_shared_rank(&s_idx[tid], r);
                if (ob > b) {
                    b = ob;
                    bi = oi;
                }
            }
            V[(long long)(m0 + tid) * ldv + o] = b;
            I[(long long)(m0 + tid) * ldv + o] = bi;
        }
        cl.sync();                               // no CTA leaves while rank 0 may read its shared memory
    } else if (tx == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = m0 + 8 * ty + i;
            if (row < M) {
                V[(long long)row * ldv + o] = wb[i];
                I[(long long)row * ldv + o] = wi[i];
            }
        }
    }
}

template <int SPL, bool VEC>
int launch_packed(const float* Are, const float* Aim, long long lda, const float* Z, long long ldz, int M, int K,
                  long long Tn, int ntiles, int group, long long nout, float* V, int32_t* I, long long ldv,
                  cudaStream_t stream) {
    auto kern = simt_absmax_packed_kernel<SPL, VEC>;
    const int smem = AS_ST * AS_STAGE * (int)sizeof(float);
    GWB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nout * SPL), (unsigned)cdiv(M, AS_BM));
    cfg.blockDim = dim3(AS_NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = SPL;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = SPL > 1 ? 1 : 0;
    GWB_CUDA(cudaLaunchKernelEx(&cfg, kern, Are, Aim, lda, Z, ldz, M, K, Tn, ntiles, group, V, I, ldv));
    GWB_LAUNCH_CHECK("simt_absmax_packed_kernel");
    return GWB_OK;
}

std::atomic<int> g_f32_async{1};   // 0: the synchronous kernel only (gwb_f32_set_async)

}  // namespace
}  // namespace gwb

extern "C" int gwb_f32_set_async(int on) {
    using namespace gwb;
    GWB_CHECK_ARG(on == 0 || on == 1, GWB_ERR_ARG, "f32_set_async: on=%d (0 or 1)", on);
    g_f32_async.store(on);
    return GWB_OK;
}

extern "C" int gwb_fused_peaks_f32(const float* Are, const float* Aim, long long lda, const float* Z, long long ldz,
                                   int M, int K, long long Tn, int group, float* V, int32_t* I, long long ldv,
                                   void* stream) {
    using namespace gwb;
    GWB_CHECK_ARG(M > 0 && K > 0 && Tn > 0 && group > 0, GWB_ERR_SHAPE, "fused_peaks_f32: M=%d K=%d Tn=%lld group=%d",
                  M, K, Tn, group);
    GWB_CHECK_ARG(lda >= K && ldz >= Tn, GWB_ERR_SHAPE, "fused_peaks_f32: lda or ldz too small");
    GWB_CHECK_ARG(Are && Aim && Z && V && I, GWB_ERR_ARG, "fused_peaks_f32: null pointer");
    const long long ntiles = cdiv(Tn, BN);
    GWB_CHECK_ARG(ntiles * BN < (1ll << 31), GWB_ERR_SHAPE, "fused_peaks_f32: Tn too large for int32 indices");
    const long long nout = cdiv(ntiles, group);
    GWB_CHECK_ARG(ldv >= nout, GWB_ERR_SHAPE, "fused_peaks_f32: ldv=%lld < outputs per row %lld", ldv, nout);
    GWB_CHECK_ARG(nout < (1ll << 31), GWB_ERR_SHAPE, "fused_peaks_f32: too many outputs");
    group = (int)std::min<long long>(group, ntiles);        // one output at most: the kernels' sums of it stay in range
    if (g_f32_async.load() && cdiv(M, AS_BM) <= 65535) {
        const bool vec = ldz % 4 == 0 && aligned(Z, 16);        // 16-byte copies of Z
        // windows are shared out over clusters while whole windows would leave the last of few waves nearly empty
        // (two CTAs per SM; from 32 waves on it is a thirty-second at most) and a part still holds two blocks
        const long long items = nout * cdiv(M, AS_BM);
        const bool whole = items >= 32ll * 2 * num_sms() || nout * AS_MAXSPL >= (1ll << 31);
        const int spl = whole ? 1 : group >= 8 ? 4 : group >= 4 ? 2 : 1;
        auto go = [&](auto v) {
            constexpr bool VEC = decltype(v)::value;
            cudaStream_t st = (cudaStream_t)stream;
            const int nt = (int)ntiles;
            if (spl == 4) return launch_packed<4, VEC>(Are, Aim, lda, Z, ldz, M, K, Tn, nt, group, nout, V, I, ldv, st);
            if (spl == 2) return launch_packed<2, VEC>(Are, Aim, lda, Z, ldz, M, K, Tn, nt, group, nout, V, I, ldv, st);
            return launch_packed<1, VEC>(Are, Aim, lda, Z, ldz, M, K, Tn, nt, group, nout, V, I, ldv, st);
        };
        return vec ? go(std::true_type{}) : go(std::false_type{});
    }
    dim3 grid((unsigned)nout, (unsigned)cdiv(M, BM));
    simt_absmax_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(Are, Aim, lda, Z, ldz, M, K, Tn, (int)ntiles, group, V,
                                                                I, ldv);
    GWB_LAUNCH_CHECK("simt_absmax_kernel");
    return GWB_OK;
}
