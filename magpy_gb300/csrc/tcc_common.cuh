// tcc_common.cuh -- what the two kernels for clusters of more than 64 particles
// share (sllg_tcc.cu: D streamed; sllg_tcr.cu: D resident in tensor memory): the
// split of particles over a cluster's CTAs, the layouts of D, B and the
// accumulators, and the launches.
#pragma once
#include <cuda_fp16.h>
#include "common.cuh"
#include "plan.hpp"
#include "tc_cluster.cuh"
#include "tc_ptx.cuh"

namespace magpy {

namespace {

constexpr int PPC = 42;           // particles per CTA
constexpr int RT = 128;           // rows of D per CTA (one MMA tile)
constexpr int KC = 64;            // K elements per chunk of D
constexpr int PAIRS = PPC / 2;    // particle pairs per CTA
constexpr int EPI_WARPS = 8;      // epilogue warps (0..7)
constexpr uint32_t DRAIN_LIMIT = 1u << 24;
constexpr int32_t ST_WATCHDOG = 16;

__host__ __device__ inline size_t tcc_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Accumulator columns the MMAs write: [main NB | corr NB] from the main MMA,
// and the correction MMA's N = NB rounded up to a multiple of 16 from column
// NB (for NB = 40, eight columns past 2 NB).
__host__ __device__ constexpr int tcc_acc_cols(int nb) { return nb + (nb + 15) / 16 * 16; }

// Instruction descriptors of the two MMAs of a k-step, and B's layout.
template <int NB> struct Idesc {
    static constexpr uint32_t MAIN = tc::idesc_f16_f32(RT, 2 * NB);
    // D_lo B_hi into [NB, NB + NC): N a multiple of 16 (for NB = 40 the
    // last 8 columns multiply the first B_lo rows into accumulator
    // columns that nothing reads)
    static constexpr uint32_t CORR = tc::idesc_f16_f32(RT, tcc_acc_cols(NB) - NB);
    static constexpr uint32_t B_LBO = (2 * NB / 8) * 128;  // between K-adjacent core matrices of B
};

// Accumulators from column `acc` -> field tile F[row][member], row stride NB + 4
// (epilogue warps 0..7: lane quarter warp % 4, member half warp / 4).
template <int NB>
__device__ inline void tcc_field_tile(uint32_t acc, float *F, int warp, int lane)
{
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t lanes = (uint32_t)(32 * quarter) << 16;
    const int row = 32 * quarter + lane;
    constexpr int HALF = NB / 2;  // member columns per warp (a multiple of 4)
#pragma unroll
    for (int cb = 0; cb < HALF / 8; cb++) {
        const int col = half * HALF + 8 * cb;
        float vm[8], vc[8];
        tc::tmem_ld8(acc + lanes + (uint32_t)col, vm);
        tc::tmem_ld8(acc + lanes + (uint32_t)(NB + col), vc);
        tc::tmem_ld_wait();
        float4 *dst = reinterpret_cast<float4 *>(F + row * (NB + 4) + col);
        dst[0] = make_float4(fmaf(vc[0], 1.0f / tc::SPLIT_SCALE, vm[0]),
                             fmaf(vc[1], 1.0f / tc::SPLIT_SCALE, vm[1]),
                             fmaf(vc[2], 1.0f / tc::SPLIT_SCALE, vm[2]),
                             fmaf(vc[3], 1.0f / tc::SPLIT_SCALE, vm[3]));
        dst[1] = make_float4(fmaf(vc[4], 1.0f / tc::SPLIT_SCALE, vm[4]),
                             fmaf(vc[5], 1.0f / tc::SPLIT_SCALE, vm[5]),
                             fmaf(vc[6], 1.0f / tc::SPLIT_SCALE, vm[6]),
                             fmaf(vc[7], 1.0f / tc::SPLIT_SCALE, vm[7]));
    }
    if constexpr (HALF % 8 == 4) {  // the last four columns (NB = 40)
        const int col = half * HALF + HALF - 4;
        float vm[4], vc[4];
        tc::tmem_ld4(acc + lanes + (uint32_t)col, vm);
        tc::tmem_ld4(acc + lanes + (uint32_t)(NB + col), vc);
        tc::tmem_ld_wait();
        *reinterpret_cast<float4 *>(F + row * (NB + 4) + col) =
            make_float4(fmaf(vc[0], 1.0f / tc::SPLIT_SCALE, vm[0]),
                        fmaf(vc[1], 1.0f / tc::SPLIT_SCALE, vm[1]),
                        fmaf(vc[2], 1.0f / tc::SPLIT_SCALE, vm[2]),
                        fmaf(vc[3], 1.0f / tc::SPLIT_SCALE, vm[3]));
    }
}

// One particle's sample: x = (hi + lo) sc, o its index in a component's
// [S][P] planes.  Not inlined, as field_block is not: what a step rarely runs
// is kept out of the step loop's code.
__device__ __noinline__ void tcc_write_sample(double *mx, double *my, double *mz, int64_t o,
                                              double sc, float xh, float xl, float yh, float yl,
                                              float zh, float zl)
{
    mx[o] = ((double)xh + (double)xl) * sc;
    my[o] = ((double)yh + (double)yl) * sc;
    mz[o] = ((double)zh + (double)zl) * sc;
}

// D tile (global, [chunk][split][128 x KC, row groups outermost]) into tensor
// memory for the MMAs' A operand: row r in lane r, split sp's K element k in
// column dcol + sp K/2 + k/2 (two 16-bit elements per column, the even K in
// the low half).  Warps 0..7: lane quarter warp % 4, split warp / 4.  Ends
// with the stores complete; a CTA barrier must follow before the first MMA.
__device__ inline void tcc_load_d_tmem(uint32_t dcol, int K, const __half *dtile, int warp, int lane)
{
    if (warp >= 8) return;
    const int quarter = warp & 3, sp = warp >> 2;
    const uint32_t row = (uint32_t)(32 * quarter + lane);
    const uint32_t lanes = (uint32_t)(32 * quarter) << 16;
    for (int c0 = 0; c0 < K / 2; c0 += 8) {
        uint32_t v[8];
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int k = 2 * (c0 + c), kc = k / KC, kk = k % KC;
            const __half *src = dtile + (size_t)(2 * kc + sp) * RT * KC +
                                tc::cm_offset_rows(row, (uint32_t)kk, KC);
            v[c] = *reinterpret_cast<const uint32_t *>(src);
        }
        tc::tmem_st8(dcol + lanes + (uint32_t)(sp * (K / 2) + c0), v);
    }
    tc::tmem_st_wait();
    tc::fence_before_sync();
}

// The OR over the cluster of a word of each CTA (every thread gets it).  No CTA
// may write its word before every CTA has read it.
__device__ inline int cluster_or(const int *word, int T)
{
    __shared__ int any;
    if (threadIdx.x == 0) {
        int a = 0;
        const uint32_t base = tc::smem_addr(word);
        for (int r = 0; r < T; r++) a |= tc::ld_cluster_s32(tc::mapa(base, (uint32_t)r));
        any = a;
    }
    __syncthreads();
    return any;
}

// A check of the step loop: whether any CTA of the cluster was marked before it,
// the same answer in every CTA.  A CTA that is ahead enters the step, and may mark
// itself there, while another still reads: so each publishes its error word as it
// stands before the barrier, in one of two words by the check's number (the word
// is written again two checks later, past the next check's barrier, at which
// every CTA arrives after its reads).
__device__ inline int cluster_check(const int *sErr, int T, int64_t number)
{
    __shared__ int marked[2];
    __syncthreads();  // this CTA's earlier marks
    int *word = &marked[number & 1];
    if (threadIdx.x == 0) *word = *(const volatile int *)sErr;
    tc::cluster_sync();
    return cluster_or(word, T);
}

// The check after the last step, past which no CTA marks itself: a wait that ran
// out after the last check of the loop is reported too.
__device__ inline int cluster_last_check(const int *sErr, int T)
{
    tc::cluster_sync();
    return cluster_or(sErr, T);
}

template <class Kern>
cudaError_t tcc_prepare(Kern kern, int T, size_t smem)
{
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem);
    if (err == cudaSuccess && T > 8)
        err = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return err;
}

template <class Kern, class... Args>
cudaError_t tcc_launch(Kern kern, int T, size_t smem, int threads, int64_t tiles,
                       cudaStream_t stream, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * T));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)T;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // the stream's scheduling priority, carried into a captured graph node
    // (a batch gives its longest group the highest)
    int prio = 0;
    if (cudaStreamGetPriority(stream, &prio) != cudaSuccess) prio = 0;
    attr[1].id = cudaLaunchAttributePriority;
    attr[1].val.priority = prio;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace

}  // namespace magpy
