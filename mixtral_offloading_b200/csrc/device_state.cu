// Device-side error flag of the library and the pass from fp32 sums to bf16 rows that the 3-bit GEMM ends with.
#include "common.cuh"
#include "kernels.cuh"

namespace hqm {

// Device-side failure flag of the bounded waits (read by hqm_device_error()).
static __device__ int g_tc_error = 0;
int* tc_error_ptr() {
    static int* ptrs[MAX_DEVICES];                 // the flag of the current device (one copy per device)
    int*& ptr = ptrs[current_device_slot()];
    if (!ptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_tc_error) == cudaSuccess) ptr = (int*)p;
    }
    return ptr;
}

__global__ void rows_from_sums_kernel(uint16_t* __restrict__ y, const float* __restrict__ sums,
                                      const uint16_t* __restrict__ bias, int64_t MN, int N) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < MN; i += (int64_t)gridDim.x * blockDim.x) {
        float v = sums[i];
        if (bias) v += bf16_bits_to_float(bias[i % N]);
        y[i] = float_to_bf16_bits(v);
    }
}

int launch_rows_from_sums(uint16_t* y, const float* sums, const uint16_t* bias, int64_t M, int N, cudaStream_t st) {
    int64_t b = (M * N + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    rows_from_sums_kernel<<<(int)(b < 1 ? 1 : b), 256, 0, st>>>(y, sums, bias, M * N, N);
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

}  // namespace hqm

// Reads and clears the device-side failure flag (see the header); synchronises the device.  Not part of
// the per-token path.
extern "C" int hqm_device_error(void) {
    int v = 0;
    int* p = hqm::tc_error_ptr();
    if (!p) return -1;
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    if (cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (v != 0 && cudaMemset(p, 0, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
