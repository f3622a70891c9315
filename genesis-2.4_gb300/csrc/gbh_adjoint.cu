// gbh_adjoint.cu -- launchers of the adjoint kernels (compiled with
// --fmad=false so the per-step recomputation reproduces the FP64 step bit
// for bit).
#include "gbh_adjoint.cuh"

namespace gbh {

namespace {
cudaError_t smem_attr(const void *fn, size_t smem)
{
    if (smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}
}  // namespace

cudaError_t launch_adj_copy(const AdjView &v, int ntiles, int maxrows, int c, int dir, bool to_tape,
                            cudaStream_t st)
{
    if (ntiles <= 0 || maxrows <= 0) return cudaSuccess;
    const dim3 grid(ntiles, (maxrows + ADJ_COPY_ROWS - 1) / ADJ_COPY_ROWS);
    k_adj_copy<<<grid, dim3(LANES, ADJ_COPY_ROWS), 0, st>>>(v, c, dir, to_tape ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_adj_ck_to_tape(const AdjView &v, int ntiles, int maxrows, int c0, int nk, cudaStream_t st)
{
    if (ntiles <= 0 || maxrows <= 0 || nk <= 0) return cudaSuccess;
    const dim3 grid(ntiles, (maxrows + ADJ_COPY_ROWS - 1) / ADJ_COPY_ROWS, nk);
    k_adj_ck_to_tape<<<grid, dim3(LANES, ADJ_COPY_ROWS), 0, st>>>(v, c0);
    return cudaGetLastError();
}

cudaError_t launch_adj_linearize(const AdjView &v, int ntiles, int smax, int nk, cudaStream_t st)
{
    if (ntiles <= 0 || nk <= 0) return cudaSuccess;
    const size_t smem = (size_t)2 * smax * LANES * sizeof(double);
    cudaError_t ce = smem_attr((const void *)k_adj_eliminate, smem);
    if (ce != cudaSuccess) return ce;
    k_adj_linearize<<<dim3(ntiles, nk), LANES, 0, st>>>(v);
    k_adj_eliminate<<<dim3(ntiles, nk), LANES, smem, st>>>(v, smax);
    return cudaGetLastError();
}

size_t adj_reverse_smem(int n, int nch, int nslots, int hmax)
{
    return sizeof(double) * (6 * (size_t)n + 2) + sizeof(int2) * ((size_t)nch + n) + 2 * sizeof(int) * (size_t)n +
           (size_t)nslots * sizeof(AdjSlot) + (size_t)hmax * sizeof(AdjChan);
}

cudaError_t launch_adj_reverse(const AdjView &v, const AdjPlan &pl, int ngroups, int warps, size_t smem, int hmax, int nk,
                               int step0, cudaStream_t st)
{
    if (ngroups <= 0 || nk <= 0) return cudaSuccess;
    cudaError_t ce = smem_attr((const void *)k_adj_reverse, smem);
    if (ce != cudaSuccess) return ce;
    k_adj_reverse<<<ngroups, warps * LANES, smem, st>>>(v, pl, hmax, nk, step0);
    return cudaGetLastError();
}

cudaError_t launch_adj_reduce(const AdjView &v, int ntiles, int smax, int nk, cudaStream_t st)
{
    if (ntiles <= 0 || nk <= 0) return cudaSuccess;
    k_adj_reduce<<<dim3(ntiles, smax), LANES, 0, st>>>(v, nk);
    return cudaGetLastError();
}

}  // namespace gbh
