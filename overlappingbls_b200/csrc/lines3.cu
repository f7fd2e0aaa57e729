// lines3.cu -- see lines3.cuh.
#include "lines3.cuh"
#include "lines_dispatch.cuh"

namespace obl {

// A complex value whose arithmetic is scalar: cadd, csub, ... of fft.cuh pack float2 only
struct alignas(8) S2 {
    float x, y;
};
__device__ __forceinline__ S2 s2(float x, float y) { return S2{x, y}; }

constexpr int kRows3Warps = 8;

// One warp takes the LPW row pairs from base; LL lanes a line, the exchange in shared memory.
template <int N, int OP> __global__ void __launch_bounds__(32 * kRows3Warps) k_rows3(RowArgs<float> a)
{
    using C = S2;
    using D = LineDerived<N, OP>;
    constexpr int LL = D::LL, LPW = D::LPW, VR = D::VR;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane / LL, t = lane % LL;
    LineScratch<C> sc{reinterpret_cast<C *>(smraw) + (warp * LPW + g) * scratch_len(N)};
    const long long pr = ((long long)blockIdx.x * kRows3Warps + warp) * LPW + g;
    const bool act = pr < a.npairs;
    const long long r0 = 2 * (act ? pr : 0);
    C v[VR];
    if constexpr (OP == OP_INV) {
        // two Hermitian half spectra -> Z = A + iB on all N bins; Im of DC and Nyquist ignored
        using G = Geo<N, D::RB0, LL>;
        const C *A = reinterpret_cast<const C *>(a.src) + r0 * a.src_stride;
        const C *B = A + a.src_stride;
#pragma unroll
        for (int b = 0; b < G::PER; ++b) {
            const int j = t + LL * b;
#pragma unroll
            for (int r = 0; r < D::RB0; ++r) {
                const int i = j + r * G::NB;
                C z = s2(0, 0);
                if (act && (G::FULL || j < G::NB)) {
                    const bool lo = i <= N / 2;
                    const int k = lo ? i : N - i;
                    C av = A[k], bv = B[k];
                    if (k == 0 || k == N / 2) { av.y = 0; bv.y = 0; }
                    z = lo ? s2(av.x - bv.y, av.y + bv.x) : s2(av.x + bv.y, bv.x - av.y);
                }
                v[b * D::RB0 + r] = z;
            }
        }
        fft_regs<N, typename D::PB, LL, false>(v, sc, reinterpret_cast<const C *>(a.twB), t);
        using GL = Geo<N, D::RBL, LL>;
        float *Ao = reinterpret_cast<float *>(a.dst) + r0 * a.dst_stride;
        float *Bo = Ao + a.dst_stride;
        if (!act) return;
#pragma unroll
        for (int b = 0; b < GL::PER; ++b) {
            const int j = t + LL * b;
            if (GL::FULL || j < GL::NB)
#pragma unroll
                for (int r = 0; r < D::RBL; ++r) {
                    Ao[j + r * GL::NB] = v[b * D::RBL + r].x;
                    Bo[j + r * GL::NB] = v[b * D::RBL + r].y;
                }
        }
    } else {
        using G = Geo<N, D::RF0, LL>;
        const float *A = reinterpret_cast<const float *>(a.src) + r0 * a.src_stride;
        const float *B = A + a.src_stride;
        float ca = 0, cb = 0;
        if (act) { ca = A[0]; cb = B[0]; }
#pragma unroll
        for (int b = 0; b < G::PER; ++b) {
            const int j = t + LL * b;
#pragma unroll
            for (int r = 0; r < D::RF0; ++r) {
                const int i = j + r * G::NB;
                C z = s2(0, 0);
                if (act && (G::FULL || j < G::NB)) z = s2((A[i] - ca) * a.scale, (B[i] - cb) * a.scale);
                v[b * D::RF0 + r] = z;
            }
        }
        fft_regs<N, typename D::PF, LL, true>(v, sc, reinterpret_cast<const C *>(a.twF), t);
        // the half spectra of both rows; the x-Nyquist is zeroed (203_fftn_mpi.f90:25) and the
        // subtracted constants return in the DC bins
        using GL = Geo<N, D::RFL, LL>;
#pragma unroll
        for (int b = 0; b < GL::PER; ++b) {
            const int j = t + LL * b;
            if (GL::FULL || j < GL::NB)
#pragma unroll
                for (int r = 0; r < D::RFL; ++r) sc.st(j + r * GL::NB, v[b * D::RFL + r]);
        }
        __syncwarp();
        C *Ao = reinterpret_cast<C *>(a.dst) + r0 * a.dst_stride;
        C *Bo = Ao + a.dst_stride;
        constexpr int H = N / 2;
        for (int k = t; k <= H; k += LL) {
            C ao = s2(0, 0), bo = s2(0, 0);
            if (k < H) {
                const C z = sc.ld(k), zc = cconj(sc.ld(k == 0 ? 0 : N - k));
                const C s = cadd(z, zc), d = csub(z, zc);
                ao = s2(0.5f * s.x, 0.5f * s.y);
                bo = s2(0.5f * d.y, -0.5f * d.x);
                if (k == 0) {
                    ao.x += ca * a.scale * (float)N;
                    bo.x += cb * a.scale * (float)N;
                }
            }
            if (act) {
                Ao[k] = ao;
                Bo[k] = bo;
            }
        }
    }
}

// WB adjacent complex columns of one plane per CTA, line-minor (see k_cols_gform)
constexpr int kCols3Warps = 8, kCols3Lines = 8;
template <int N, int OP> __global__ void __launch_bounds__(32 * kCols3Warps) k_cols3(ColArgs<float> a, int kmul)
{
    using C = S2;
    using D = LineDerived<N, OP>;
    constexpr int WB = kCols3Lines, LL = (32 / WB) * kCols3Warps;
    constexpr bool FWD = OP == OP_FWD;
    using P = typename std::conditional<FWD, typename D::PF, typename D::PB>::type;
    constexpr int VR = Regs<N, LL, P>::v, R0 = PlanInfo<P>::first, RL = PlanInfo<P>::last;
    using G0 = Geo<N, R0, LL>;
    using GL = Geo<N, RL, LL>;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, z = blockIdx.y;
    const int line = lane % WB, t = lane / WB + (32 / WB) * warp;
    const int gl = blockIdx.x * WB + line;
    const bool act = gl < a.ncols;
    const int glc = act ? gl : 0;
    const C *src = reinterpret_cast<const C *>(a.src) + (long long)z * a.src_plane;
    C *dst = reinterpret_cast<C *>(a.dst) + (long long)z * a.dst_plane;
    LineMinor<C, WB> sc{reinterpret_cast<C *>(smraw), line};
    // the checked build tests each element's level, column and plane offset
    auto ok = [&](int i, int col, long long row, long long plane, int site) {
        return ck_in(z, a.nlev, site) && ck_in(col, row, site) && ck_in((long long)i * row + col, plane, site);
    };
    C v[VR];
#pragma unroll
    for (int b = 0; b < G0::PER; ++b) {
        const int j = t + LL * b;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int i = j + r * G0::NB;
            C x = s2(0, 0);
            if (act && (G0::FULL || j < G0::NB)) {
                if (!OBL_CHECK || ok(i, glc, a.src_row, a.src_plane, CK_COL_LOAD)) x = src[(long long)i * a.src_row + glc];
                if (!FWD && kmul) {
                    const float kk = (float)(kmul == 1 ? a.ktab[glc] : a.ktab[i]);
                    x = s2(-kk * x.y, kk * x.x);
                }
                x.x *= a.scale;
                x.y *= a.scale;
            }
            v[b * R0 + r] = x;
        }
    }
    fft_regs<N, P, LL, FWD, true>(v, sc, reinterpret_cast<const C *>(FWD ? a.twF : a.twB), t);
    if (!act) return;
#pragma unroll
    for (int b = 0; b < GL::PER; ++b) {
        const int j = t + LL * b;
        if (GL::FULL || j < GL::NB)
#pragma unroll
            for (int r = 0; r < RL; ++r) {
                const int i = j + r * GL::NB;
                C x = v[b * RL + r];
                if (FWD && a.zero_nyq && i == N / 2) x = s2(0, 0);
                if (!OBL_CHECK || ok(i, gl, a.dst_row, a.dst_plane, CK_COL_STORE)) dst[(long long)i * a.dst_row + gl] = x;
            }
    }
}

template <int N, int OP> static cudaError_t rows3_n(const RowArgs<float> &a, cudaStream_t s)
{
    using D = LineDerived<N, OP>;
    constexpr size_t sm = sizeof(S2) * (size_t)kRows3Warps * D::LPW * scratch_len(N);
    static_assert(sm <= 48 * 1024, "no opt-in shared memory");
    const long long per = (long long)kRows3Warps * D::LPW, grid = (a.npairs + per - 1) / per;
    if (grid < 1) return cudaSuccess;
    k_rows3<N, OP><<<(unsigned)grid, 32 * kRows3Warps, sm, s>>>(a);
    return cudaGetLastError();
}

template <int N, int OP> static cudaError_t cols3_n(const ColArgs<float> &a, int kmul, cudaStream_t s)
{
    constexpr size_t sm = sizeof(S2) * (size_t)N * kCols3Lines;
    static_assert(sm <= 48 * 1024, "no opt-in shared memory");
    dim3 grid((a.ncols + kCols3Lines - 1) / kCols3Lines, a.nlev);
    if (grid.x < 1 || grid.y < 1) return cudaSuccess;
    k_cols3<N, OP><<<grid, 32 * kCols3Warps, sm, s>>>(a, kmul);
    return cudaGetLastError();
}

cudaError_t launch_rows3(int op, int n, const RowArgs<float> &a, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return op == OP_FWD ? rows3_n<N, OP_FWD>(a, s) : rows3_n<N, OP_INV>(a, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_cols3(int op, int n, const ColArgs<float> &a, int kmul, cudaStream_t s)
{
    switch (n) {
#define OBL_CASE(N) case N: return op == OP_FWD ? cols3_n<N, OP_FWD>(a, kmul, s) : cols3_n<N, OP_INV>(a, kmul, s);
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return cudaErrorInvalidValue;
}

} // namespace obl
