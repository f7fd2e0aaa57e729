// gform.cu -- the pressure RHS in G form: one y-transform for the x- and z-parts.
//
// The right-hand side of press_stag_array (109_press_stag_array.f90:203-225) per mode is
//     i*(kx*H_x + ky*H_y) + (H_z(z+1) - H_z(z) [+ H_z(0) at z = 1])/dz,
// with H = the 2D transform (x r2c, then y c2c) of the scaled u, v, w.  kx and the
// z-difference are constant along y, so by linearity of the y-transform
//     G = i*kx*H_x + (H_z(z+1) - H_z(z) [+ H_z(0)])/dz
// can be formed from the x-spectra before it: one y-transform of G (written over H_x)
// replaces those of H_x and H_z, and the solve forms G + i*ky*H_y.  H_z is still
// transformed at level 0 (the Neumann ghost p_hat(0) = p_hat(1) - dz*H_z(0), :313-315)
// and, at levels 1..L, in the line group of kx = 0 only: the (0,0) mode's RHS is H_z
// itself (:219-221).
#include "lines_dispatch.cuh"
#include "press.cuh"

namespace obl {

// G of level z + 1 (z = the launch's plane index); FIRST: the launch of level 1 alone,
// whose z-difference also takes H_z(0)
template <typename T, bool FIRST> struct GSrc {
    const C2<T> *Hx, *Hz;
    const double *kx;
    long long S;
    int lhx, lv0;
    T idz;
    __device__ __forceinline__ C2<T> operator()(int z, int i, int gl) const
    {
        const long long lv = lv0 + z;
        const long long q = (long long)i * lhx + gl;
        if (!ck_in(q, S, CK_GFORM_LOAD)) return mk<T>(0, 0);
        const C2<T> hx = __ldcg(Hx + S * lv + q), hzc = __ldcg(Hz + S * lv + q), hzn = __ldcg(Hz + S * (lv + 1) + q);
        C2<T> dh = csub(hzn, hzc);
        if constexpr (FIRST) dh = cadd(dh, __ldcg(Hz + q));
        const T k = (T)kx[gl];
        return mk<T>(-k * hx.y + dh.x * idz, k * hx.x + dh.y * idz);
    }
};

// A CTA owns WB adjacent complex columns of one plane.  Lane l % WB is the line, the other
// lane bits and the warp index are the butterfly slot (LL slots), and the exchange is
// line-minor; a three-radix plan (fft2.cuh).  The two-pass columns measured slower here: G
// takes three loads an element, which a radix-32 butterfly's registers do not leave in
// flight (512 lines FP64, 64 levels: 138 us against 224).  FP32 lines of 256 and more read
// their twiddles through L1, with the registers bounded for 4 CTAs an SM.
constexpr int kGformWarps = 8;
template <typename T> struct GformGeo {
    static constexpr int WB = sizeof(T) == 4 ? 8 : 4, LL = (32 / WB) * kGformWarps;
};
template <typename T, int N> constexpr bool gform_tw_global() { return sizeof(T) == 4 && N >= 256; }

template <typename T, int N, bool FIRST>
__global__ void __launch_bounds__(32 * kGformWarps, gform_tw_global<T, N>() ? 4 : 1) k_cols_gform(ColArgs<T> a, GSrc<T, FIRST> g)
{
    using C = C2<T>;
    using D = LineDerived<N, OP_FWD>;
    constexpr int WB = GformGeo<T>::WB, LL = GformGeo<T>::LL, VR = Regs<N, LL, typename D::PF>::v;
    using G0 = Geo<N, D::RF0, LL>;
    using GL = Geo<N, D::RFL, LL>;
    extern __shared__ __align__(16) unsigned char smraw[];
    C *buf = reinterpret_cast<C *>(smraw);
    const C *tw = a.twF;
    if constexpr (!gform_tw_global<T, N>()) {
        C *s = buf;
        buf += D::TF;
        for (int i = threadIdx.x; i < D::TF; i += blockDim.x) s[i] = a.twF[i];
        __syncthreads();
        tw = s;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, z = blockIdx.y;
    const int line = lane % WB, t = lane / WB + (32 / WB) * warp, gl = blockIdx.x * WB + line;
    const bool act = gl < a.ncols;
    LineMinor<C, WB> sc{buf, line};
    C v[VR];
#pragma unroll
    for (int b = 0; b < G0::PER; ++b) {
        const int j = t + LL * b;
#pragma unroll
        for (int r = 0; r < D::RF0; ++r)
            v[b * D::RF0 + r] = act && (G0::FULL || j < G0::NB) ? g(z, j + r * G0::NB, gl) : mk<T>(0, 0);
    }
    fft_regs<N, typename D::PF, LL, true, true>(v, sc, tw, t);
    if (!act) return;
    C *dst = reinterpret_cast<C *>(a.dst) + (long long)z * a.dst_plane;
#pragma unroll
    for (int b = 0; b < GL::PER; ++b) {
        const int j = t + LL * b;
        if (GL::FULL || j < GL::NB)
#pragma unroll
            for (int r = 0; r < D::RFL; ++r) {
                const int i = j + r * GL::NB;
                // the checked build tests each element's level, column and plane offset
                if (!(ck_in(z, a.nlev, CK_COL_STORE) && ck_in(gl, a.dst_row, CK_COL_STORE) &&
                      ck_in((long long)i * a.dst_row + gl, a.dst_plane, CK_COL_STORE)))
                    continue;
                dst[(long long)i * a.dst_row + gl] = a.zero_nyq && i == N / 2 ? mk<T>(0, 0) : v[b * D::RFL + r];
            }
    }
}

template <typename T, int N, bool FIRST>
static cudaError_t gform_launch(const ColArgs<T> &a, const GSrc<T, FIRST> &g, cudaStream_t s)
{
    using D = LineDerived<N, OP_FWD>;
    constexpr int WB = GformGeo<T>::WB;
    const size_t sm = sizeof(C2<T>) * ((gform_tw_global<T, N>() ? 0 : (size_t)D::TF) + (size_t)N * WB);
    auto kern = k_cols_gform<T, N, FIRST>;
    static bool inits[kMaxDevices] = {};
    const int ds = device_slot();
    if (ds < 0 || !inits[ds]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        if (ds >= 0) inits[ds] = true;
    }
    dim3 grid((a.ncols + WB - 1) / WB, a.nlev);
    if (grid.x < 1 || grid.y < 1) return cudaSuccess;
    kern<<<grid, 32 * kGformWarps, sm, s>>>(a, g);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_gform_cols(int ny, C2<T> *Hx, const C2<T> *Hz, const double *kx, long long S, int lhx, int L,
                              double dz, const C2<T> *twF, cudaStream_t s)
{
    // level 1 (with H_z(0)), then levels 2..L; G of level lv is written over H_x(lv)
    for (int part = 0; part < 2; ++part) {
        const int lv0 = part == 0 ? 1 : 2, nlev = part == 0 ? 1 : L - 1;
        if (nlev < 1) continue;
        ColArgs<T> a{};
        a.src = Hx + S * lv0;
        a.dst = Hx + S * lv0;
        a.src_row = a.dst_row = lhx;
        a.src_plane = a.dst_plane = S;
        a.ncols = lhx;
        a.nlev = nlev;
        a.scale = (T)1;
        a.twF = twF;
        a.zero_nyq = 1;   // 203_fftn_mpi.f90:33
        cudaError_t e = cudaErrorInvalidValue;
        if (part == 0) {
            GSrc<T, true> g{Hx, Hz, kx, S, lhx, lv0, (T)(1.0 / dz)};
            switch (ny) {
#define OBL_CASE(N) case N: e = gform_launch<T, N, true>(a, g, s); break;
                OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
            }
        } else {
            GSrc<T, false> g{Hx, Hz, kx, S, lhx, lv0, (T)(1.0 / dz)};
            switch (ny) {
#define OBL_CASE(N) case N: e = gform_launch<T, N, false>(a, g, s); break;
                OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
            }
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template cudaError_t launch_gform_cols<float>(int, C2<float> *, const C2<float> *, const double *, long long, int, int,
                                              double, const C2<float> *, cudaStream_t);
template cudaError_t launch_gform_cols<double>(int, C2<double> *, const C2<double> *, const double *, long long, int,
                                               int, double, const C2<double> *, cudaStream_t);

} // namespace obl
