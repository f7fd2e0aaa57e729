// multi.cuh -- the row and column line kernels over several fields of one shape in one
// launch (see launch_rows_multi / launch_cols_multi in lines.cuh).  The per-line work is
// tp_row_unit / tp_cols_unit unchanged; only the field of each unit is looked up first.
#pragma once
#include "lines_dispatch.cuh"

namespace obl {

template <typename T, int N, int OP>
__global__ void __launch_bounds__(TpRows<T, N>::NT, TpRows<T, N>::minb) 
    k_tp_rows_multi(RowArgs<T> a0, const __grid_constant__ MultiPtr<T> m, int nb)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int f = blockIdx.x / nb;   // nb CTAs per field
    RowArgs<T> a = a0;
    a.src = m.src[f];
    a.dst = m.dst[f];
    tp_row_unit<T, N, OP>(a, (long long)(blockIdx.x - f * nb) * TpRows<T, N>::WB, reinterpret_cast<C2<T> *>(smraw));
}

template <typename T, int N, int OP, bool REAL>
__global__ void __launch_bounds__(TpGeo<T, N, OP>::NT, TpGeo<T, N, OP>::minb) 
    k_tp_cols_multi(ColArgs<T> a0, const __grid_constant__ MultiPtr<T> m)
{
    using G = TpGeo<T, N, OP>;
    extern __shared__ __align__(128) unsigned char smraw[];
    const int f = blockIdx.y / a0.nlev, z = blockIdx.y - f * a0.nlev;
    ColArgs<T> a = a0;
    a.src = m.src[f];
    a.dst = m.dst[f];
    tp_cols_unit<T, N, OP, REAL, G::NT, G::WB>(a, blockIdx.x, z, reinterpret_cast<C2<T> *>(smraw));
}

template <typename T, int N, int OP>
static cudaError_t rows_multi_t(const RowArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    using G = TpRows<T, N>;
    static bool inits[kMaxDevices] = {};
    constexpr size_t sm = sizeof(C2<T>) * (size_t)G::WB * G::template line_elems<OP>();
    auto kern = k_tp_rows_multi<T, N, OP>;
    const int ds = device_slot();
    if (ds < 0 || !inits[ds]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        if (ds >= 0) inits[ds] = true;
    }
    const long long nb = (a.npairs + G::WB - 1) / G::WB;
    if (nb < 1) return cudaSuccess;
    kern<<<(unsigned)(nb * nf), G::NT, sm, s>>>(a, m, (int)nb);
    return cudaGetLastError();
}

template <typename T, int N, int OP, bool REAL>
static cudaError_t cols_multi_t(const ColArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    static bool inits[kMaxDevices] = {};
    constexpr int WB = TpGeo<T, N, OP>::WB, NT = TpGeo<T, N, OP>::NT;
    const size_t sm = tp_cols_smem<T, N, OP>();
    auto kern = k_tp_cols_multi<T, N, OP, REAL>;
    const int ds = device_slot();
    if (ds < 0 || !inits[ds]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        if (ds >= 0) inits[ds] = true;
    }
    ColArgs<T> b = a;
    b.pf_ahead = 0;
    const int nlines = REAL ? b.ncols / 2 : b.ncols;
    dim3 grid((nlines + WB - 1) / WB, (unsigned)(b.nlev * nf));
    if (grid.x < 1 || grid.y < 1) return cudaSuccess;
    kern<<<grid, NT, sm, s>>>(b, m);
    return cudaGetLastError();
}

template <typename T, int N>
static cudaError_t rows_multi_n(int op, const RowArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    switch (op) {
    case OP_DERIV: return rows_multi_t<T, N, OP_DERIV>(a, m, nf, s);
    case OP_PAD: return rows_multi_t<T, N, OP_PAD>(a, m, nf, s);
    case OP_UNPAD: return rows_multi_t<T, N, OP_UNPAD>(a, m, nf, s);
    }
    return cudaErrorInvalidValue;
}

template <typename T, int N>
static cudaError_t cols_multi_n(int op, const ColArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    switch (op) {
    case OP_DERIV: return cols_multi_t<T, N, OP_DERIV, true>(a, m, nf, s);
    case OP_PAD: return cols_multi_t<T, N, OP_PAD, true>(a, m, nf, s);
    case OP_UNPAD: return cols_multi_t<T, N, OP_UNPAD, true>(a, m, nf, s);
    }
    return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_rows_multi_real(int op, int n, const RowArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return rows_multi_n<T, N>(op, a, m, nf, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_cols_multi_real(int op, int n, const ColArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return cols_multi_n<T, N>(op, a, m, nf, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_rows_multi_fwd(int n, const RowArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return rows_multi_t<T, N, OP_FWD>(a, m, nf, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

// (complex columns)
template <typename T>
cudaError_t launch_cols_multi_fwd(int n, const ColArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return cols_multi_t<T, N, OP_FWD, false>(a, m, nf, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

} // namespace obl
