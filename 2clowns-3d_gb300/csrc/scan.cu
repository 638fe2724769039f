// scan.cu -- where the set positions of a bit mask go: the exclusive scan of the
// counts per 1024-bit tile (the masks and counts come from the kernel that decides
// the bits, the kernel that uses them ranks a bit inside its tile; grid_index.cuh).
#include "grid_index.cuh"

namespace clowns {

// One block scans the tiles' counts in place, NV interleaved lists at once; totals[k]
// is list k's sum.
template <int NV>
__global__ void __launch_bounds__(1024) k_scan_tiles(int* __restrict__ sums, int nt, int* __restrict__ totals) {
    __shared__ int sm[NV][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int per = (nt + 1023) / 1024, lo = threadIdx.x * per;
    int s[NV], x[NV];
    for (int k = 0; k < NV; k++) s[k] = 0;
    for (int q = lo; q < min(nt, lo + per); q++)
        for (int k = 0; k < NV; k++) s[k] += sums[NV * q + k];
    for (int k = 0; k < NV; k++) {
        x[k] = s[k];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x[k], o);
            if (lane >= o) x[k] += y;
        }
        if (lane == 31) sm[k][wid] = x[k];
    }
    __syncthreads();
    if (wid < NV) {                        // warp k: list k's warp totals
        int w = sm[wid][lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        sm[wid][lane] = w;
        if (lane == 31) totals[wid] = w;
    }
    __syncthreads();
    for (int k = 0; k < NV; k++) x[k] += (wid ? sm[k][wid - 1] : 0) - s[k];
    for (int q = lo; q < min(nt, lo + per); q++)
        for (int k = 0; k < NV; k++) {
            const int v = sums[NV * q + k];
            sums[NV * q + k] = x[k];
            x[k] += v;
        }
}

int scan_tiles_dev(int lists, int* sums, long n, int* totals, cudaStream_t s) {
    const int nt = (int)((n + kBitTile - 1) / kBitTile);
    if (lists == 1) k_scan_tiles<1><<<1, 1024, 0, s>>>(sums, nt, totals);
    else k_scan_tiles<2><<<1, 1024, 0, s>>>(sums, nt, totals);
    CLOWNS_CUDA_TRY(cudaGetLastError());
    return CLOWNS_OK;
}

}  // namespace clowns
