// ensemble.cu -- host-side geometry of the persistent ensemble kernel (ensemble.cuh);
// the kernel itself is instantiated in ensemble_all.cu and ensemble_part*.cu.
#include <algorithm>

#include "ensemble_kernel.cuh"
#include "obl.h"

namespace obl {

bool ens_length_supported(int n)
{
    switch (n) {
#define OBL_C(N) case N: return true;
        OBL_ENS_FOR_EACH_N(OBL_C)
#undef OBL_C
    }
    return false;
}

int ens_lines_of(int n)
{
    switch (n) {
#define OBL_C(N) case N: return ens_lines<N>();
        OBL_ENS_FOR_EACH_N(OBL_C)
#undef OBL_C
    }
    return 1;
}

// ----------------------------------------------------------------------------- self-test
// One CTA through the grid barrier with its arrival counter preset: 0 releases at once;
// any other value never reaches the release count (nothing else arrives), so the bounded
// wait gives up and raises the error flag, as a lost CTA of a real launch would.
__global__ void k_barrier_selftest(unsigned *bar, int *passed)
{
    const bool ok = ens_barrier(bar, reinterpret_cast<int *>(bar + 2));
    if (threadIdx.x == 0) *passed = ok ? 1 : 0;
}

int ens_barrier_selftest(bool never_released, cudaStream_t s, std::string &err)
{
    unsigned *bar = nullptr;   // arrivals, generation, error flag, passed
    if (cudaMalloc(&bar, 4 * sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        err = "barrier self-test: allocation failed";
        return OBL_ERR_NOMEM;
    }
    const unsigned init[4] = {never_released ? 1u : 0u, 0u, 0u, 0u};
    cudaError_t e = cudaMemcpyAsync(bar, init, sizeof init, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        k_barrier_selftest<<<1, 128, 0, s>>>(bar, reinterpret_cast<int *>(bar + 3));
        e = cudaGetLastError();
    }
    unsigned out[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, bar, sizeof out, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(bar);
    if (e != cudaSuccess) {
        err = std::string("barrier self-test: ") + cudaGetErrorString(e);
        return OBL_ERR_CUDA;
    }
    if (out[2]) {
        err = "barrier self-test: the grid-barrier wait gave up";
        return OBL_ERR_TIMEOUT;
    }
    return out[3] ? OBL_OK : OBL_ERR_TIMEOUT;
}

// ----------------------------------------------------------------------------- host side
template <typename T> long long EnsGeoHost<T>::rows_units(int n, long long npairs)
{
    const int w = ens_lines_of(n);
    return (npairs + w - 1) / w;
}

template <typename T> long long EnsGeoHost<T>::pinv_rows_units(int n, long long npairs) { return 4 * rows_units(n, npairs); }

template <typename T, int N> static size_t ens_smem_rows() { return TpRows<T, N, ens_lines<N>()>::smem_fwd3_seq; }
template <typename T, int N, int OP> static size_t ens_smem_col()
{
    return sizeof(C2<T>) * (size_t)TpLine<N, OP>::ROWS * ens_lines<N>();
}
template <typename T, int N> static size_t ens_smem_cols()
{
    return std::max({ens_smem_col<T, N, OP_PAD>(), ens_smem_col<T, N, OP_DERIV>(), ens_smem_col<T, N, OP_FWD>(),
                     TpPinv<T, N, ens_lines<N>()>::smem});
}
template <typename T, int N> static size_t ens_smem_pinv_rows()
{
    using G = TpRows<T, N, ens_lines<N>()>;
    return sizeof(C2<T>) * (size_t)G::WB * G::LF;
}

template <typename T> size_t EnsGeoHost<T>::smem(int nx, int ny, int pb, int pe)
{
    size_t m = 0;
    const bool rows = pb <= 0 && pe > 0, mid = pb <= 3 && pe > 1, tail = pb <= 4 && pe > 4;
    switch (nx) {
#define OBL_C(N)                                                                                         \
    case N:                                                                                              \
        if (rows) m = std::max(m, ens_smem_rows<T, N>());                                                \
        if (tail) m = std::max(m, ens_smem_pinv_rows<T, N>());                                           \
        break;
        OBL_ENS_FOR_EACH_N(OBL_C)
#undef OBL_C
    }
    switch (ny) {
#define OBL_C(N) case N: if (mid) m = std::max(m, ens_smem_cols<T, N>()); break;
        OBL_ENS_FOR_EACH_N(OBL_C)
#undef OBL_C
    }
    return m;
}

template struct EnsGeoHost<float>;
template struct EnsGeoHost<double>;

} // namespace obl
