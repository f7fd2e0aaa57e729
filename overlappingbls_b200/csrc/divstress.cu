// divstress.cu -- the stress-divergence row pass (see divstress.cuh).
#include "divstress.cuh"
#include "lines_dispatch.cuh"

namespace obl {

constexpr int kFillPer = 4096;   // elements of a BOGUS plane per CTA

// ddx of WB row pairs by two passes, the other terms added at the store.  The addends are
// asked into L2 when the unit starts and read in groups of four elements a row, so that a
// group's loads (up to 24) are in flight together.
template <typename T, int N>
__global__ void __launch_bounds__(TpRows<T, N>::NT, TpRows<T, N>::minb)
    k_tp_rows_divt(RowArgs<T> a, const __grid_constant__ DivRows<T> e, int nb, int nfill)
{
    using C = C2<T>;
    using G = TpRows<T, N>;
    constexpr int R0 = G::R0, R1 = G::R1, WB = G::WB, NT = G::NT, LS = G::LF > G::LD ? G::LF : G::LD;
    extern __shared__ __align__(16) unsigned char smraw[];
    C *buf = reinterpret_cast<C *>(smraw);
    const int tid = threadIdx.x;
    if ((int)blockIdx.x >= nb) {
        const int u = blockIdx.x - nb, p = u / nfill;
        const long long i0 = (long long)(u - p * nfill) * kFillPer;
        for (long long i = i0 + tid; i < i0 + kFillPer && i < e.plane; i += NT) e.bogus[p][i] = e.bogus_value;
        return;
    }
    const long long base = (long long)blockIdx.x * WB;
    auto active = [&](int ln) {
        const long long p = base + ln;
        // checked build: the pair lies in the launch's rows and on one level
        return p < a.npairs && ck_in(2 * p + 1, 2 * a.npairs, CK_DIVT_ROW) && ck_in((2 * p) % e.ny + 1, e.ny, CK_DIVT_ROW);
    };
    const long long dz = e.fwd ? e.plane : -e.plane;      // the other tz plane
    {
        constexpr int EL = 128 / sizeof(T), PL = (N + EL - 1) / EL;
        for (int i = tid; i < 6 * PL * WB; i += NT) {
            const int ln = i / (6 * PL), k = (i / PL) % 6;
            if (!active(ln)) continue;
            const long long r = 2 * (base + ln) + (k & 1), z = r / e.ny, o = z * e.plane + (r - z * e.ny) * a.src_stride + (i % PL) * EL;
            if (k >= 2 && (z < e.zlo || z > e.zhi)) continue;
            const T *p = k < 2 ? e.out + o : e.tz + o + (k >= 4 ? dz : 0);
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        }
    }
    auto src = [&](int ln, const T *&A, const T *&B) {
        if (!active(ln)) return false;
        A = reinterpret_cast<const T *>(a.src) + 2 * (base + ln) * a.src_stride;
        B = A + a.src_stride;
        return true;
    };
    tp_rows_first<T, R0, R1, WB, NT, LS>(src, a.scale, buf);
    __syncthreads();
    const int line = tid / R0, j = tid % R0;
    C v[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) v[r] = buf[line * LS + r * G::PF + j];
#pragma unroll
    for (int r = 1; r < R1; ++r) v[r] = cmul(v[r], __ldg(a.twF + r * R0 + j));
    Dft<R1, true>::run(v);
    __syncthreads();
    tp_deriv<T, N, R0, R1>(v, a.ktab, j);
    Dft<R1, false>::run(v);
#pragma unroll
    for (int r = 0; r < R1; ++r) buf[line * LS + j * G::PD + r] = v[r];
    __syncthreads();
    tp_rows_last<T, R0, R1, WB, NT, LS>(tid, buf, a.twB, [&](int ln, int jj, const C(&x)[R0]) {
        if (!active(ln)) return;
        const long long r0 = 2 * (base + ln), z = r0 / e.ny, o = z * e.plane + (r0 - z * e.ny) * a.src_stride + jj;
        T *A = e.out + o, *B = A + a.src_stride;
        const T *H = e.tz + o + (e.fwd ? e.plane : 0), *L = e.tz + o - (e.fwd ? 0 : e.plane);
        const bool vert = z >= e.zlo && z <= e.zhi;
#pragma unroll
        for (int r = 0; r < R0; r += 4) {
            T da[4], db[4], ha[4], hb[4], la[4], lb[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = (r + k) * R1;
                da[k] = A[i];
                db[k] = B[i];
                ha[k] = vert ? H[i] : (T)0;
                hb[k] = vert ? H[a.src_stride + i] : (T)0;
                la[k] = vert ? L[i] : (T)0;
                lb[k] = vert ? L[a.src_stride + i] : (T)0;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = (r + k) * R1;
                T sa = x[r + k].x + da[k], sb = x[r + k].y + db[k];
                if (vert) {
                    sa += e.rdz * (ha[k] - la[k]);
                    sb += e.rdz * (hb[k] - lb[k]);
                }
                A[i] = sa;
                B[i] = sb;
            }
        }
        if (jj < 2) A[N] = B[N] = (T)0;
    });
}

template <typename T, int N>
static cudaError_t launch_divt_n(const RowArgs<T> &a, const DivRows<T> &e0, cudaStream_t s)
{
    using G = TpRows<T, N>;
    static bool inits[kMaxDevices] = {};
    constexpr size_t sm = sizeof(C2<T>) * (size_t)G::WB * (G::LF > G::LD ? G::LF : G::LD);
    auto kern = k_tp_rows_divt<T, N>;
    const int ds = device_slot();
    if (ds < 0 || !inits[ds]) {
        cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (err != cudaSuccess) return err;
        if (ds >= 0) inits[ds] = true;
    }
    DivRows<T> e = e0;
    if (!e.bogus[0]) { e.bogus[0] = e.bogus[1]; e.bogus[1] = nullptr; }
    const int np = (e.bogus[0] ? 1 : 0) + (e.bogus[1] ? 1 : 0), nfill = (int)((e.plane + kFillPer - 1) / kFillPer);
    const long long nb = (a.npairs + G::WB - 1) / G::WB;
    if (nb + np < 1) return cudaSuccess;
    kern<<<(unsigned)(nb + (long long)np * nfill), G::NT, sm, s>>>(a, e, (int)nb, nfill);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_rows_divt(int n, const RowArgs<T> &a, const DivRows<T> &e, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return launch_divt_n<T, N>(a, e, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}
template cudaError_t launch_rows_divt<float>(int, const RowArgs<float> &, const DivRows<float> &, cudaStream_t);
template cudaError_t launch_rows_divt<double>(int, const RowArgs<double> &, const DivRows<double> &, cudaStream_t);

} // namespace obl
