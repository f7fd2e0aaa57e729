// lines_dispatch.cuh -- runtime-length dispatch of the row / column kernels.
// Supported base lengths n (and their 3/2 partners): the grid sizes of the
// reference's production namelists and of the benchmark workloads.
#pragma once
#include <cmath>
#include <vector>

#include "lines.cuh"

#define OBL_FOR_EACH_N(X) \
    X(32) X(48) X(64) X(80) X(96) X(128) X(160) X(192) X(240) X(256) X(320) X(384) X(512) X(640)

namespace obl {

template <typename T, int N>
cudaError_t rows_n(int op, const RowArgs<T> &a, cudaStream_t s)
{
    switch (op) {
    case OP_DERIV: return launch_rows_t<T, N, OP_DERIV>(a, s);
    case OP_PAD: return launch_rows_t<T, N, OP_PAD>(a, s);
    case OP_UNPAD: return launch_rows_t<T, N, OP_UNPAD>(a, s);
    case OP_FWD: return launch_rows_t<T, N, OP_FWD>(a, s);
    case OP_INV: return launch_rows_t<T, N, OP_INV>(a, s);
    }
    return cudaErrorInvalidValue;
}

template <typename T, int N>
cudaError_t cols_real_n(int op, const ColArgs<T> &a, cudaStream_t s)
{
    switch (op) {
    case OP_DERIV: return launch_cols_t<T, N, OP_DERIV, true>(a, s);
    case OP_PAD: return launch_cols_t<T, N, OP_PAD, true>(a, s);
    case OP_UNPAD: return launch_cols_t<T, N, OP_UNPAD, true>(a, s);
    }
    return cudaErrorInvalidValue;
}
template <typename T, int N>
cudaError_t cols_cplx_n(int op, const ColArgs<T> &a, cudaStream_t s)
{
    switch (op) {
    case OP_FWD: return launch_cols_t<T, N, OP_FWD, false>(a, s);
    case OP_INV: return launch_cols_t<T, N, OP_INV, false>(a, s);
    case OP_FILT: return launch_cols_t<T, N, OP_FILT, false>(a, s);
    }
    return cudaErrorInvalidValue;
}

template <typename T> cudaError_t launch_rows(int op, int n, const RowArgs<T> &a, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return rows_n<T, N>(op, a, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

template <typename T> cudaError_t launch_cols_real(int op, int n, const ColArgs<T> &a, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return cols_real_n<T, N>(op, a, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}
template <typename T> cudaError_t launch_cols_cplx(int op, int n, const ColArgs<T> &a, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return cols_cplx_n<T, N>(op, a, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------- host twiddle tables
template <class P> struct PlanVec;
template <int... Rs> struct PlanVec<RPlan<Rs...>> {
    static std::vector<int> get() { return {Rs...}; }
};

// w_N^m = exp(-2 pi i m / N), m < N, interleaved re, im
inline std::vector<double> plan_roots(int N)
{
    const double pi = 3.14159265358979323846264338327950288;
    std::vector<double> out(2 * (size_t)N);
    for (int m = 0; m < N; ++m) {
        const double ang = -2.0 * pi * (double)m / (double)N;
        out[2 * m] = std::cos(ang);
        out[2 * m + 1] = std::sin(ang);
    }
    return out;
}
inline std::vector<double> plan_table_for(int N, const std::vector<double> &roots, const std::vector<int> &radices)
{
    std::vector<double> out;
    out.reserve(4 * (size_t)N);
    int NS = 1;
    for (int R : radices) {
        if (NS > 1) {
            const int tws = N / (NS * R);
            for (int r = 0; r < R; ++r)
                for (int k = 0, m = 0; k < NS; ++k, m = (m + r * tws) % N) {   // m = r*k*tws mod N
                    out.push_back(roots[2 * m]);
                    out.push_back(roots[2 * m + 1]);
                }
        }
        NS *= R;
    }
    return out;
}

// The tables of base length N by role (no three-radix kernel transforms 3N/2 forward).  The
// roots of N and of 3N/2 are computed once and gathered: with a cosine and a sine for every
// entry of every table the context of a 640x320 FP64 grid took 537 us to create, now 461.
template <int N> std::vector<std::vector<double>> plan_tables_n()
{
    constexpr int M = 3 * N / 2, R0 = TwoPass<N>::R0, R1 = TwoPass<N>::R1, RP = 3 * R1 / 2;
    const std::vector<double> a = plan_roots(N), b = plan_roots(M);
    std::vector<std::vector<double>> t(2 * ROLE_TP);
    t[ROLE_FWD] = plan_table_for(N, a, PlanVec<FwdPlan<N>>::get());
    t[ROLE_BWD] = plan_table_for(N, a, PlanVec<BwdPlan<N>>::get());
    t[ROLE_PADBWD] = plan_table_for(M, b, PlanVec<PadBwdPlan<N>>::get());
    t[ROLE_TP + ROLE_FWD] = plan_table_for(N, a, {R0, R1});
    t[ROLE_TP + ROLE_BWD] = plan_table_for(N, a, {R1, R0});
    t[ROLE_TP + ROLE_PADFWD] = plan_table_for(M, b, {R0, RP});
    t[ROLE_TP + ROLE_PADBWD] = plan_table_for(M, b, {RP, R0});
    return t;
}

} // namespace obl
