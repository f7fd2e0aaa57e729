// fused_launch.cuh -- launchers of the step's multi-output kernels (fused.cuh), in units of
// compilation by precision (fused_*.cu, pinv_*.cu; see launch_cols in lines.cuh).
#pragma once
#include "fused.cuh"
#include "lines_dispatch.cuh"

namespace obl {

template <typename K> static cudaError_t allow_smem(K kern, size_t sm, bool (&inits)[kMaxDevices])
{
    const int ds = device_slot();
    if (ds >= 0 && inits[ds]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e == cudaSuccess && ds >= 0) inits[ds] = true;
    return e;
}

template <typename T, int N> static cudaError_t rows3_run_n(const RowsFwd3Args<T> &a, cudaStream_t s)
{
    using G = TpRows<T, N>;
    static bool inits[kMaxDevices] = {};
    cudaError_t e = allow_smem(k_tp_rows_fwd3<T, N>, G::smem_fwd3, inits);
    if (e != cudaSuccess) return e;
    const long long grid = (a.npairs + G::WB - 1) / G::WB;
    if (grid < 1) return cudaSuccess;
    k_tp_rows_fwd3<T, N><<<(unsigned)grid, G::NT, G::smem_fwd3, s>>>(a);
    return cudaGetLastError();
}

template <typename T, int N>
static cudaError_t rows3_multi_n(const RowsFwd3Args<T> &a, const RowsFwd3Fields<T> &m, int nf, cudaStream_t s)
{
    using G = TpRows<T, N>;
    static bool inits[kMaxDevices] = {};
    cudaError_t e = allow_smem(k_tp_rows_fwd3_multi<T, N>, G::smem_fwd3, inits);
    if (e != cudaSuccess) return e;
    const long long nb = (a.npairs + G::WB - 1) / G::WB;
    if (nb < 1) return cudaSuccess;
    k_tp_rows_fwd3_multi<T, N><<<(unsigned)(nb * nf), G::NT, G::smem_fwd3, s>>>(a, m, (int)nb);
    return cudaGetLastError();
}

template <typename T, int N> struct TpColsFwd {
    using G = TpGeo<T, N, OP_PAD>;   // one middle butterfly a thread in all three
    static constexpr int NT = TwoPass<N>::R0 * G::WB;
    static constexpr size_t smem = sizeof(C2<T>) * (size_t)G::WB * TpLine<N, OP_PAD>::ROWS;
    static_assert(TpLine<N, OP_DERIV>::ROWS <= TpLine<N, OP_PAD>::ROWS && TpLine<N, OP_FWD>::ROWS <= TpLine<N, OP_PAD>::ROWS, "one exchange for all");
};
template <typename T, int N>
__global__ void __launch_bounds__(TpColsFwd<T, N>::NT, TpGeo<T, N, OP_PAD>::minb)
    k_tp_cols_fwd(const __grid_constant__ ColsFwdArgs<T> a, int npad, int nddy)
{
    constexpr int WB = TpGeo<T, N, OP_PAD>::WB, NT = TpColsFwd<T, N>::NT;
    extern __shared__ __align__(128) unsigned char smraw[];
    C2<T> *buf = reinterpret_cast<C2<T> *>(smraw);
    // unit u of one of the three lists: field, plane, line group
    auto run = [&](auto op, const ColArgs<T> &c0, const MultiPtr<T> &m, int nlines, int u) {
        constexpr int OP = decltype(op)::value;
        const int nbx = (nlines + WB - 1) / WB, f = u / (nbx * c0.nlev), v = u - f * nbx * c0.nlev, z = v / nbx;
        ColArgs<T> c = c0;
        c.src = m.src[f];
        c.dst = m.dst[f];
        tp_cols_unit<T, N, OP, OP != OP_FWD, NT, WB>(c, v - z * nbx, z, buf);
    };
    const int u = blockIdx.x;
    if (u < npad) run(std::integral_constant<int, OP_PAD>{}, a.pad, a.mpad, a.pad.ncols / 2, u);
    else if (u < npad + nddy) run(std::integral_constant<int, OP_DERIV>{}, a.ddy, a.mddy, a.ddy.ncols / 2, u - npad);
    else run(std::integral_constant<int, OP_FWD>{}, a.fwd, a.mfwd, a.fwd.ncols, u - npad - nddy);
}

template <typename T, int N> static cudaError_t cols_fwd_n(const ColsFwdArgs<T> &a, cudaStream_t s)
{
    using G = TpColsFwd<T, N>;
    constexpr int WB = TpGeo<T, N, OP_PAD>::WB;
    static bool inits[kMaxDevices] = {};
    cudaError_t e = allow_smem(k_tp_cols_fwd<T, N>, G::smem, inits);
    if (e != cudaSuccess) return e;
    auto units = [&](const ColArgs<T> &c, int nlines, int nf) { return (long long)((nlines + WB - 1) / WB) * c.nlev * nf; };
    const long long npad = units(a.pad, a.pad.ncols / 2, a.nf), nddy = units(a.ddy, a.ddy.ncols / 2, a.nf),
                    nfwd = units(a.fwd, a.fwd.ncols, a.nfwd);
    k_tp_cols_fwd<T, N><<<(unsigned)(npad + nddy + nfwd), G::NT, G::smem, s>>>(a, (int)npad, (int)nddy);
    return cudaGetLastError();
}

template <typename T> cudaError_t ColsFwdLaunch<T>::run(int n, const ColsFwdArgs<T> &a, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return cols_fwd_n<T, N>(a, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorNotSupported;
}

template <typename T>
cudaError_t RowsFwd3Launch<T>::run_multi(int n, const RowsFwd3Args<T> &a, const RowsFwd3Fields<T> &m, int nf, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return rows3_multi_n<T, N>(a, m, nf, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorNotSupported;
}

template <typename T> cudaError_t RowsFwd3Launch<T>::run(int n, const RowsFwd3Args<T> &a, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return rows3_run_n<T, N>(a, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorNotSupported;
}


template <typename T, int N> static cudaError_t pinv_cols_n(const PinvColArgs<T> &a, int nlev, cudaStream_t s)
{
    using G = TpPinv<T, N>;
    static bool inits[kMaxDevices] = {};
    cudaError_t e = allow_smem(k_tp_cols_pinv<T, N>, G::smem, inits);
    if (e != cudaSuccess) return e;
    const int nbx = (a.lhx + G::WB - 1) / G::WB;
    dim3 grid(a.dph ? nbx + (nbx + 1) / 2 : nbx, nlev);
    k_tp_cols_pinv<T, N><<<grid, G::NT, G::smem, s>>>(a);
    return cudaGetLastError();
}

template <typename T, int N> static cudaError_t pinv_rows_n(const PinvRowArgs<T> &a, cudaStream_t s)
{
    using G = TpRows<T, N>;
    static bool inits[kMaxDevices] = {};
    constexpr size_t sm = sizeof(C2<T>) * (size_t)G::WB * G::LF;
    cudaError_t e = allow_smem(k_tp_rows_pinv<T, N>, sm, inits);
    if (e != cudaSuccess) return e;
    const long long grid = (a.dpdz ? 4 : 3) * ((a.npairs + G::WB - 1) / G::WB);
    if (grid < 1) return cudaSuccess;
    k_tp_rows_pinv<T, N><<<(unsigned)grid, G::NTI, sm, s>>>(a);
    return cudaGetLastError();
}

template <typename T> cudaError_t PinvLaunch<T>::cols(int n, const PinvColArgs<T> &a, int nlev, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return pinv_cols_n<T, N>(a, nlev, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorNotSupported;
}
template <typename T> cudaError_t PinvLaunch<T>::rows(int n, const PinvRowArgs<T> &a, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return pinv_rows_n<T, N>(a, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorNotSupported;
}

} // namespace obl
