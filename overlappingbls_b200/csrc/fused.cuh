// fused.cuh -- cluster-fused plane kernels of the projection-plus-derivative step.
//
// The separable line kernels move every intermediate through HBM: the x-padded plane of
// zero_padding, the x spectrum of the pressure RHS, and a second read of each field for
// ddy.  Here one thread-block cluster owns one (field, level) plane at a time:
//
//   row phase    each row pair is read once and transformed once along x; from that one
//                spectrum the warp produces ddx (written out), the x-padded rows and the
//                scaled x half-spectra of the RHS (both into the cluster's scratch slot);
//   cluster.sync
//   column phase column tiles of the x-padded plane are y-padded (written out), column
//                tiles of the field give ddy (the plane was just read, so it comes from L2),
//                and column tiles of the x spectrum are y-transformed into H_x, H_y, H_z;
//   cluster.sync before the slot is reused for the next plane.
//
// The scratch slot of a cluster (x-padded plane + x spectrum, ~2.5 MB for a 512^2 FP32
// plane) is rewritten before it is read on every plane and stays in L2 while the
// cluster works on it, so only the compulsory reads and writes reach HBM: this is the
// on-GPU replacement of the pencil transposes of zero_padding and fftn_mpi
// (108_01_padd.f90:114,129; 203_fftn_mpi.f90:27).
#pragma once
#include <cooperative_groups.h>

#include "lines.cuh"

namespace obl {

namespace cg = cooperative_groups;

template <typename T> struct FwdFusedArgs {
    const T *f[4];          // u, v, w, theta: (ldx, ny, nlev)
    T *d[8];                // dudx, dudy, dvdx, dvdy, dwdx, dwdy, dtdx, dtdy
    T *big[4];              // (nx2, ny2, nlev)
    C2<T> *H[3];            // RHS spectra of u, v, w: (lhx, ny, nlev), levels 1..L written
    unsigned char *scr;     // cluster scratch slots
    long long slot_bytes;
    int ldx, nlev, L, nfields;
    double sc_press;        // const/(tadv1*dt) (109_press_stag_array.f90:166-168)
    const double *kx;       // kx(lhx) (ddx)
    const double *ky;       // ky(lhy) (ddy)
    const C2<T> *twF, *twB, *twPB;   // plans: forward N, backward N, padded backward 3N/2
};

// fused row work of one row pair: ddx, x-pad and (optionally) the scaled half spectra
template <typename T, int N>
__device__ __forceinline__ void row_fwd_fused(const T *A, const T *B, T *dA, T *dB, T *pA, T *pB, C2<T> *sA,
                                              C2<T> *sB, bool act, bool spec, double sc_press,
                                              const double *kx, const C2<T> *twF, const C2<T> *twB,
                                              const C2<T> *twPB, C2<T> *scr_line, int t)
{
    using C = C2<T>;
    using DD = LineDerived<N, OP_DERIV>;
    using DP = LineDerived<N, OP_PAD>;
    constexpr int LL = DD::LL;
    static_assert(DP::LL == LL, "deriv and pad chains must share the lane layout");
    constexpr int VD = DD::VR, VP = DP::VR;
    constexpr int RF0 = DD::RF0, RFL = DD::RFL, RPL = DP::RBL;
    constexpr int N2 = 3 * N / 2;
    LineScratch<C> sc{scr_line};
    const T scale = (T)1 / (T)N;

    T ca = 0, cb = 0;
    if (act) { ca = A[0]; cb = B[0]; }
    C v[VD > VP ? VD : VP];
    {
        using G = Geo<N, RF0, LL>;
#pragma unroll
        for (int b = 0; b < G::PER; ++b) {
            const int j = t + LL * b;
#pragma unroll
            for (int r = 0; r < RF0; ++r) {
                const int i = j + r * G::NB;
                C z = mk<T>(0, 0);
                if (act && (G::FULL || j < G::NB)) z = mk<T>((A[i] - ca) * scale, (B[i] - cb) * scale);
                v[b * RF0 + r] = z;
            }
        }
    }
    fft_regs<N, typename DD::PF, LL, true>(v, sc, twF, t);   // v = FFT((x - c)/N), layout D(RFL)

    // (1) half spectra of the RHS: FFT(sc * x) = N*sc*v + sc*c*N at DC, x-Nyquist zeroed
    if (spec) {
        using G = Geo<N, RFL, LL>;
#pragma unroll
        for (int b = 0; b < G::PER; ++b) {
            const int j = t + LL * b;
            if (G::FULL || j < G::NB)
#pragma unroll
                for (int r = 0; r < RFL; ++r) sc.st(j + r * G::NB, v[b * RFL + r]);
        }
        __syncwarp();
        const T f = (T)((double)N * sc_press);
        constexpr int H = N / 2;
        for (int k = t; k <= H; k += LL) {
            C ao = mk<T>(0, 0), bo = mk<T>(0, 0);
            if (k < H) {
                const C z = sc.ld(k), zc = cconj(sc.ld(k == 0 ? 0 : N - k));
                const C s = cadd(z, zc), d = csub(z, zc);
                ao = mk<T>((T)0.5 * f * s.x, (T)0.5 * f * s.y);
                bo = mk<T>((T)0.5 * f * d.y, (T)-0.5 * f * d.x);
                if (k == 0) {
                    ao.x += (T)(sc_press * (double)N) * ca;
                    bo.x += (T)(sc_press * (double)N) * cb;
                }
            }
            if (act) {
                sA[k] = ao;
                sB[k] = bo;
            }
        }
        __syncwarp();
    }
    // (2) x-pad to 3N/2 (108_01_padd.f90:100-112)
    {
        C w[VP];
        reg_pad<T, N, RFL, LL>(v, w, t);
        fft_regs<N2, typename DP::PB, LL, false>(w, sc, twPB, t);
        using G = Geo<N2, RPL, LL>;
        if (act) {
#pragma unroll
            for (int b = 0; b < G::PER; ++b) {
                const int j = t + LL * b;
                if (G::FULL || j < G::NB)
#pragma unroll
                    for (int r = 0; r < RPL; ++r) {
                        const int i = j + r * G::NB;
                        pA[i] = w[b * RPL + r].x + ca;
                        pB[i] = w[b * RPL + r].y + cb;
                    }
            }
        }
    }
    // (3) ddx (004_derivatives.f90:33-39)
    {
        reg_deriv<T, N, RFL, LL>(v, kx, t);
        fft_regs<N, typename DD::PB, LL, false>(v, sc, twB, t);
        using G = Geo<N, DD::RBL, LL>;
        if (act) {
#pragma unroll
            for (int b = 0; b < G::PER; ++b) {
                const int j = t + LL * b;
                if (G::FULL || j < G::NB)
#pragma unroll
                    for (int r = 0; r < DD::RBL; ++r) {
                        const int i = j + r * G::NB;
                        dA[i] = v[b * DD::RBL + r].x;
                        dB[i] = v[b * DD::RBL + r].y;
                    }
            }
        }
    }
}

template <typename T, int N> struct FwdFusedGeo {
    using C = C2<T>;
    static constexpr int N2 = 3 * N / 2, LH = N / 2 + 1;
    using DD = LineDerived<N, OP_DERIV>;
    using DP = LineDerived<N, OP_PAD>;
    static constexpr int LPW = DD::LPW;
    static constexpr int TF = DD::TF, TB = DD::TB, TPB = DP::TB;
    static constexpr size_t row_scr = sizeof(C) * (size_t)8 * LPW * scratch_len(N2);
    static constexpr size_t tile_pad = sizeof(T) * (size_t)tile_rows(N2) * ColTile<T, true, DP::LPW>::S;
    static constexpr size_t tile_der = sizeof(T) * (size_t)tile_rows(N) * ColTile<T, true, DD::LPW>::S;
    static constexpr size_t tile_cpx = sizeof(C) * (size_t)tile_rows(N) * ColTile<T, false, DD::LPW>::S;
    static constexpr size_t work = row_scr > tile_pad ? (row_scr > tile_der ? (row_scr > tile_cpx ? row_scr : tile_cpx)
                                                                             : (tile_der > tile_cpx ? tile_der : tile_cpx))
                                                      : (tile_pad > tile_der ? (tile_pad > tile_cpx ? tile_pad : tile_cpx)
                                                                             : (tile_der > tile_cpx ? tile_der : tile_cpx));
    static constexpr size_t smem = sizeof(C) * ((size_t)TF + TB + TPB) + work;
    // scratch slot: x-padded plane (N2 x N reals) + x half spectrum (LH x N complex)
    static size_t slot_bytes() { return ((sizeof(T) * (size_t)N2 * N + 255) / 256) * 256 + sizeof(C) * (size_t)LH * N; }
};

template <typename T, int N>
__global__ void __launch_bounds__(256, 2) k_fwd_fused(FwdFusedArgs<T> a)
{
    using C = C2<T>;
    using GG = FwdFusedGeo<T, N>;
    using DD = typename GG::DD;
    using DP = typename GG::DP;
    constexpr int N2 = GG::N2, LH = GG::LH, LPW = GG::LPW;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), csize = (int)cl.num_blocks();
    const int cid = blockIdx.x / csize, ncl = gridDim.x / csize;

    extern __shared__ __align__(16) unsigned char smraw[];
    C *twF = reinterpret_cast<C *>(smraw);
    C *twB = twF + GG::TF;
    C *twPB = twB + GG::TB;
    unsigned char *work = reinterpret_cast<unsigned char *>(twPB + GG::TPB);
    for (int i = threadIdx.x; i < GG::TF; i += blockDim.x) twF[i] = a.twF[i];
    for (int i = threadIdx.x; i < GG::TB; i += blockDim.x) twB[i] = a.twB[i];
    for (int i = threadIdx.x; i < GG::TPB; i += blockDim.x) twPB[i] = a.twPB[i];
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane / DD::LL, t = lane % DD::LL;
    const long long pl = (long long)a.ldx * N, plb = (long long)N2 * N2, sp = (long long)LH * N;
    T *xpad = reinterpret_cast<T *>(a.scr + (long long)cid * a.slot_bytes);
    C *xspec = reinterpret_cast<C *>(a.scr + (long long)cid * a.slot_bytes +
                                      ((sizeof(T) * (size_t)N2 * N + 255) / 256) * 256);
    const int nitems = a.nfields * a.nlev;

    for (int item = cid; item < nitems; item += ncl) {
        const int fi = item / a.nlev, z = item - fi * a.nlev;
        const bool spec = fi < 3 && z >= 1 && z <= a.L;
        const T *fz = a.f[fi] + pl * z;
        // ---- row phase: pairs distributed over the warps of the cluster
        {
            C *scr_line = reinterpret_cast<C *>(work) + (warp * LPW + g) * scratch_len(N2);
            const int wg = rank * 8 + warp, nwg = csize * 8;
            for (int p0 = wg * LPW; p0 < N / 2; p0 += nwg * LPW) {
                const int p = p0 + g;
                const bool act = p < N / 2;
                const int y0 = 2 * (act ? p : 0);
                const T *A = fz + (long long)y0 * a.ldx;
                T *dA = a.d[2 * fi] + pl * z + (long long)y0 * a.ldx;
                T *pA = xpad + (long long)y0 * N2;
                C *sA = xspec + (long long)y0 * LH;
                row_fwd_fused<T, N>(A, A + a.ldx, dA, dA + a.ldx, pA, pA + N2, sA, sA + LH, act, spec, a.sc_press,
                                    a.kx, twF, twB, twPB, scr_line, t);
            }
        }
        cl.sync();
        // ---- column phase: y-pad tiles, ddy tiles, RHS y-transform tiles
        {
            constexpr int WP = ColTile<T, true, DP::LPW>::W, WD = ColTile<T, true, DD::LPW>::W;
            constexpr int WC = ColTile<T, false, DD::LPW>::W;
            const int np = (N2 + WP - 1) / WP, nd = (N + WD - 1) / WD, ns = spec ? (LH + WC - 1) / WC : 0;
            for (int task = rank; task < np + nd + ns; task += csize) {
                if (task < np) {
                    ColArgs<T> ca{};
                    ca.src = xpad; ca.dst = a.big[fi] + plb * z; ca.src_row = N2; ca.dst_row = N2;
                    ca.ncols = N2; ca.nlev = 1; ca.scale = (T)1 / (T)N;
                    ca.twF = twF; ca.twB = twPB;
                    col_unit<T, N, OP_PAD, true>(ca, 0, task, twF, twPB, reinterpret_cast<T *>(work));
                } else if (task < np + nd) {
                    ColArgs<T> ca{};
                    ca.src = fz; ca.dst = a.d[2 * fi + 1] + pl * z; ca.src_row = a.ldx; ca.dst_row = a.ldx;
                    ca.ncols = N; ca.nlev = 1; ca.scale = (T)1 / (T)N; ca.ktab = a.ky;
                    col_unit<T, N, OP_DERIV, true>(ca, 0, task - np, twF, twB, reinterpret_cast<T *>(work));
                } else {
                    ColArgs<T> ca{};
                    ca.src = xspec; ca.dst = a.H[fi] + sp * z; ca.src_row = LH; ca.dst_row = LH;
                    ca.ncols = LH; ca.nlev = 1; ca.scale = (T)1; ca.zero_nyq = 1;
                    col_unit<T, N, OP_FWD, false>(ca, 0, task - np - nd, twF, twB, reinterpret_cast<C *>(work));
                }
            }
        }
        cl.sync();
    }
}

// ----------------------------------------------------------------------------- multi-output rows
// One read of each row pair of a field yields ddx, the x-padded rows (zero_padding's
// first half, into the intermediate xpad) and, on levels 1..L of u, v, w, the scaled x
// half-spectra of the pressure RHS (written straight into H; the y transform then runs
// in place).  Replaces three separate row passes over the same field.
template <typename T> struct RowsFwd3Args {
    const T *src;          // field (ldx, ny, nlev)
    T *dfdx;               // (ldx, ny, nlev)
    T *xpad;               // (nx2, ny, nlev), xgap more elements between the levels
    C2<T> *H;              // (lhx, ny, nlev) or nullptr (theta)
    long long npairs;      // ny*nlev/2
    long long xgap;
    int ldx, ny, L;
    int z0;                // level of the first row pair (src, dfdx, H start there; a chunk of levels)
    double sc_press;
    const double *kx;
    const C2<T> *twF, *twB, *twPB;
};

// Unit u of the multi-output row pass: the WB row pairs from u*WB.  One forward transform;
// its spectrum stays in registers (16 values a thread at N = 512) until both backward
// transforms have made their first pass into exchanges of their own, so that the last
// passes of ddx and of the padded rows share one phase and no register holds the spectrum
// through them.
// SEQ: the two backward transforms share one exchange, one after the other, with the
// spectrum held through the first (the persistent ensemble kernel, whose CTAs per SM the
// larger shared memory would cut).
template <typename T, int N, int WB_ = 0, bool SEQ = false>
__device__ __forceinline__ void tp_rows_fwd3_unit(const RowsFwd3Args<T> &a, long long u, C2<T> *buf)
{
    using C = C2<T>;
    using G = TpRows<T, N, WB_>;
    constexpr int R0 = G::R0, R1 = G::R1, RP = G::RP, WB = G::WB, NT = G::NT, N2 = G::N2, LH = G::LH;
    constexpr int LP = G::LPF;      // the forward exchange shares the padded one's memory
    C *bufP = buf, *bufD = SEQ ? buf : buf + WB * LP;
    const long long base = u * WB;
    const int tid = threadIdx.x;
    auto active = [&](int ln) {
        const long long p = base + ln;
        // checked build: the pair lies in the launch's rows and on one level
        return p < a.npairs && ck_in(2 * p + 1, 2 * a.npairs, CK_ROWS3_ROW) && ck_in((2 * p) % a.ny + 1, a.ny, CK_ROWS3_ROW);
    };
    auto src = [&](int ln, const T *&A, const T *&B) {
        if (!active(ln)) return false;
        A = a.src + 2 * (base + ln) * a.ldx;
        B = A + a.ldx;
        return true;
    };
    const T scale = (T)1 / (T)N;
    tp_rows_first<T, R0, R1, WB, NT, LP>(src, scale, bufP);
    __syncthreads();
    const int line = tid / R0, j = tid % R0;
    C v[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) v[r] = bufP[line * LP + r * G::PF + j];
#pragma unroll
    for (int r = 1; r < R1; ++r) v[r] = cmul(v[r], __ldg(a.twF + r * R0 + j));
    Dft<R1, true>::run(v);                                 // FFT((x - c)/N), bins j + r*R0
    __syncthreads();                                       // the forward exchange is read
    // (1) half spectra of the RHS on levels 1..L: FFT(sc*x) = N*sc*v + sc*c*N at DC, x-Nyquist zeroed
    if (a.H) {
        const bool act = active(line);
        const long long r0 = 2 * (base + (act ? line : 0));
        const int z = a.z0 + (int)(r0 / a.ny);
        const bool spec = act && z >= 1 && z <= a.L && ck_in(r0 + 1, (long long)(a.L + 1 - a.z0) * a.ny, CK_ROWS3_SPEC);
        const T s1 = (T)((double)N * a.sc_press), h = (T)0.5 * s1;
        C *sA = a.H + r0 * LH, *sB = sA + LH;
        const T *A = a.src + r0 * a.ldx;
        auto put = [&](int k, C s, C d) {
            C ao = cscale(s, h), bo = cscale(d, h);
            if (spec) {
                if (k == 0) {
                    ao.x += s1 * A[0];
                    bo.x += s1 * A[a.ldx];
                }
                sA[k] = ao;
                sB[k] = bo;
            }
        };
        if constexpr (32 % R0 == 0) {
            tp_split_spectra<T, R0, R1>(v, j, put);
        } else {
#pragma unroll
            for (int r = 0; r < R1; ++r) bufP[line * LP + j + r * R0] = v[r];
            __syncthreads();
            tp_split_spectra_smem<T, N, R0, R1>(v, j, bufP + line * LP, put);
            __syncthreads();
        }
        if (spec && j == 0) sA[N / 2] = sB[N / 2] = mk<T>(0, 0);
    }
    // (2) first passes of the x-pad to 3N/2 (108_01_padd.f90:100-112) and of ddx
    // (004_derivatives.f90:33-39), (3) their last passes.  The loops of the two last passes
    // deal their butterflies from opposite ends, so the warps without a padded one start
    // with ddx
    auto pad_first = [&]() {
        if (j == 0) v[R1 / 2] = mk<T>(0, 0);               // the source's Nyquist bin (0 for ddx too)
        DftPad<R1>::run(v, [&](auto ic, C x) { bufP[line * LP + j * G::PP + decltype(ic)::value] = x; });
    };
    auto ddx_first = [&]() {
        tp_deriv<T, N, R0, R1>(v, a.kx, j);
        Dft<R1, false>::run(v);
#pragma unroll
        for (int r = 0; r < R1; ++r) bufD[line * G::LD + j * G::PD + r] = v[r];
    };
    auto pad_last = [&]() {
        tp_rows_last<T, R0, RP, WB, NT, LP>(tid, bufP, a.twPB, [&](int ln, int jj, const C(&x)[R0]) {
            if (!active(ln)) return;
            const long long r0 = 2 * (base + ln);
            const T ca = a.src[r0 * a.ldx], cb = a.src[(r0 + 1) * a.ldx];
            T *A = a.xpad + (a.xgap ? r0 * N2 + (r0 / a.ny) * a.xgap : r0 * N2), *B = A + N2;
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                A[jj + r * RP] = x[r].x + ca;
                B[jj + r * RP] = x[r].y + cb;
            }
        });
    };
    auto ddx_last = [&]() {
        tp_rows_last<T, R0, R1, WB, NT, G::LD>(NT - 1 - tid, bufD, a.twB, [&](int ln, int jj, const C(&x)[R0]) {
            if (!active(ln)) return;
            T *A = a.dfdx + 2 * (base + ln) * a.ldx, *B = A + a.ldx;
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                A[jj + r * R1] = x[r].x;
                B[jj + r * R1] = x[r].y;
            }
        });
    };
    pad_first();
    if constexpr (SEQ) {
        __syncthreads();
        pad_last();
        __syncthreads();
        ddx_first();
        __syncthreads();
    } else {
        ddx_first();
        __syncthreads();
        pad_last();
    }
    ddx_last();
}

template <typename T, int N>
__global__ void __launch_bounds__(TpRows<T, N>::NT, TpRows<T, N>::minb) k_tp_rows_fwd3(RowsFwd3Args<T> a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    tp_rows_fwd3_unit<T, N>(a, blockIdx.x, reinterpret_cast<C2<T> *>(smraw));
}

// The same for several fields in one launch: field f's pointers replace src, dfdx, xpad, H.
// (__grid_constant__: indexing the by-value argument made every thread copy it to local
// memory first)
template <typename T> struct RowsFwd3Fields {
    const T *src[4];
    T *dfdx[4], *xpad[4];
    C2<T> *H[4];
};
template <typename T, int N>
__global__ void __launch_bounds__(TpRows<T, N>::NT, TpRows<T, N>::minb) 
    k_tp_rows_fwd3_multi(const __grid_constant__ RowsFwd3Args<T> a0, const __grid_constant__ RowsFwd3Fields<T> m, int nb)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int f = blockIdx.x / nb;   // nb CTAs per field
    RowsFwd3Args<T> a = a0;
    a.src = m.src[f];
    a.dfdx = m.dfdx[f];
    a.xpad = m.xpad[f];
    a.H = m.H[f];
    tp_rows_fwd3_unit<T, N>(a, blockIdx.x - f * nb, reinterpret_cast<C2<T> *>(smraw));
}

template <typename T> struct RowsFwd3Launch {
    static cudaError_t run(int n, const RowsFwd3Args<T> &a, cudaStream_t s);
    static cudaError_t run_multi(int n, const RowsFwd3Args<T> &a, const RowsFwd3Fields<T> &m, int nf, cudaStream_t s);
};

// The forward pass's column work of all fields in one launch: units of the y-pad, of ddy and
// of the RHS y-transform, one after the other in blockIdx.x.
template <typename T> struct ColsFwdArgs {
    ColArgs<T> pad, ddy, fwd;
    MultiPtr<T> mpad, mddy, mfwd;
    int nf, nfwd;                         // fields; spectra
};
template <typename T> struct ColsFwdLaunch {
    static cudaError_t run(int n, const ColsFwdArgs<T> &a, cudaStream_t s);
};

// ----------------------------------------------------------------------------- fused inverse
// y-inverse of the pressure solution: one load of p_hat(z) gives the y-inverses of p_hat
// and i*ky*p_hat (109_press_stag_array.f90:231-238), one load of the dpdz spectrum gives
// its y-inverse; i*kx*p_hat is formed from the y-inverse of p_hat by the row pass.  Level
// 0 only needs p.  Line-minor column layout.
template <typename T> struct PinvColArgs {
    const C2<T> *ph, *dph;                // (lhx, ny, 0..L) spectra
    C2<T> *Xp, *Xdy, *Xdz;                // y-inverses of p_hat, i*ky*p_hat, dpdz spectrum
    long long S;                          // lhx*ny
    int lhx;
    const double *kx, *ky;                // kx(lhx), ky_2d row (ny)
    const C2<T> *twB;
};

// One CTA unit of the y-inverse: two transforms of level z, WB lines each, one middle
// butterfly per thread.  Units u < nbx take line group u of p_hat and make both of its
// transforms (p_hat and i*ky*p_hat, one load); the others take two line groups of the dpdz
// spectrum.  Both transforms make their first passes into exchanges of their own and share
// the last phase, in which radix-32 butterflies of one line group would leave half of the
// threads idle.
template <typename T, int N, int WB_ = 0> struct TpPinv {
    static constexpr int R0 = TwoPass<N>::R0, R1 = TwoPass<N>::R1, WB = WB_ ? WB_ : TpGeo<T, N, OP_INV>::WB, NT = R0 * WB;
    static constexpr int PO = tp_pitch(R1), LE = R0 * PO * WB;     // one exchange
    static constexpr size_t smem = sizeof(C2<T>) * 2 * (size_t)LE;
    // resident warps per SM (512 lines, 64 levels, FP32: 16 warps 89 us, 24 105 us, the three
    // radix kernel 103; FP64: 162, 187 before; 128 lines: FP32 29 -> 23, FP64 80 -> 41)
    static constexpr int wsm = sizeof(T) == 4 ? (R0 >= 24 ? 16 : 24) : (R0 == 32 ? 8 : 12);
    static constexpr int minb = wsm * 32 / NT > 0 ? wsm * 32 / NT : 1;
};
template <typename T, int N, int WB_ = 0>
__device__ __forceinline__ void tp_pinv_cols_unit(const PinvColArgs<T> &a, int u, int z, C2<T> *buf)
{
    using C = C2<T>;
    using G = TpPinv<T, N, WB_>;
    constexpr int R0 = G::R0, R1 = G::R1, WB = G::WB, NT = G::NT, PO = G::PO, LE = G::LE;
    const int tid = threadIdx.x, line = tid % WB, j = tid / WB;
    const int nbx = (a.lhx + WB - 1) / WB;
    const bool pp = u < nbx;                        // p_hat's unit
    if (!pp && z == 0) return;                      // level 0 needs p only
    const int g0 = pp ? u : 2 * (u - nbx), g1 = pp ? u : g0 + 1;
    const int nt = pp ? (z == 0 ? 1 : 2) : (g1 < nbx ? 2 : 1);   // (p_hat alone: a grid of nbx units)
    auto load = [&](const C *src, int g, C(&v)[R1]) {
        const int gl = g * WB + line;
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const long long q = (long long)(j + r * R0) * a.lhx + gl;
            v[r] = gl < a.lhx && ck_in(q, a.S, CK_PINV_COL_LOAD) ? __ldcg(src + a.S * z + q) : mk<T>(0, 0);
        }
    };
    auto first = [&](C(&v)[R1], C *b) {
        Dft<R1, false>::run(v);
#pragma unroll
        for (int r = 0; r < R1; ++r) b[(j * PO + r) * WB + line] = v[r];
    };
    {
        C v[R1], w[R1];
        load(pp ? a.ph : a.dph, g0, v);
        if (pp) {
            // i*kx p_hat needs no transform of its own: kx is constant along y, so its
            // y-inverse is i*kx times that of p_hat, applied by the x-inverse row pass
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                const T kyv = (T)a.ky[j + r * R0];
                w[r] = mk<T>(-kyv * v[r].y, kyv * v[r].x);
            }
        } else if (nt > 1) {
            load(a.dph, g1, w);
        }
        first(v, buf);
        if (nt > 1) first(w, buf + LE);
    }
    __syncthreads();
#pragma unroll 1
    for (int f = tid; f < nt * R1 * WB; f += NT) {
        const int q = f / (R1 * WB), jj = (f / WB) % R1;
        const C *b = buf + q * LE;
        C *dst = pp ? (q == 0 ? a.Xp : a.Xdy) : a.Xdz;
        const int gl = (q == 0 ? g0 : g1) * WB + line;
        C x[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) x[r] = b[(r * PO + jj) * WB + line];
#pragma unroll
        for (int r = 1; r < R0; ++r) x[r] = cmulc(x[r], __ldg(a.twB + r * R1 + jj));
        Dft<R0, false>::run(x);
        if (gl < a.lhx) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const long long i = (long long)(jj + r * R1) * a.lhx + gl;
                if (ck_in(i, a.S, CK_PINV_COL_STORE)) dst[a.S * z + i] = x[r];
            }
        }
    }
}

template <typename T, int N> __global__ void __launch_bounds__(TpPinv<T, N>::NT, TpPinv<T, N>::minb) k_tp_cols_pinv(PinvColArgs<T> a)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    tp_pinv_cols_unit<T, N>(a, blockIdx.x, blockIdx.y, reinterpret_cast<C2<T> *>(smraw));
}

// x-inverse of the four y-inverses and the projection (110_project.f90:16-40) in one
// pass over the rows: p at levels 0..L, dpdx/dpdy/dpdz at 1..L (slot z-1), and
// u,v (levels 1..L) and w (levels 2..L) += dt*(-tadv1*grad p).
template <typename T> struct PinvRowArgs {
    const C2<T> *Xp, *Xdy, *Xdz;          // (lhx, ny, 0..L); dpdx's is i*kx*Xp
    const double *kx;                     // kx(lhx), Nyquist entry 0
    T *p, *dpdx, *dpdy, *dpdz;            // p (ldx, ny, 0:nz); d* (ldx, ny, 1:nz); dpdz optional
    T *u, *v, *w;                         // updated in place (ldx, ny, 0:nz); u = nullptr: no project()
    long long npairs;                     // ny*(L+1)/2
    int ldx, ny, lhx;
    T dt_tadv1;                           // dt*tadv1
    const C2<T> *twF;                     // two-pass table of nx
    int w_from_1;                         // 0: w updated from level 2 (bottom rank, jz_min = 2);
                                          // 1: from level 1 (the z-slab of a rank above it)
    int L, zero_bc;                       // zero_bc: also w(1) = w(nz) = 0 (110_project.f90:55-60), nz = L+1
};

// Unit: component q (0: p; 1: dpdx and u; 2: dpdy and v; 3: dpdz and w) of the WB row pairs
// from base.
template <typename T, int N, int WB_ = 0>
__device__ __forceinline__ void tp_pinv_rows_unit(const PinvRowArgs<T> &a, int q, long long base, C2<T> *buf)
{
    using C = C2<T>;
    using G = TpRows<T, N, WB_>;
    constexpr int R0 = G::R0, R1 = G::R1;
    const long long pl = (long long)a.ldx * a.ny;
    // levels of the unit's pairs: level 0 holds p only
    auto row0 = [&](int ln) { return 2 * (base + ln); };
    auto active = [&](int ln) {
        const long long p = base + ln;
        if (p >= a.npairs || (q > 0 && 2 * p < a.ny)) return false;
        // checked build: the pair lies in the launch's rows and on one level
        return ck_in(2 * p + 1, 2 * a.npairs, CK_PINV_ROW) && ck_in((2 * p) % a.ny + 1, a.ny, CK_PINV_ROW);
    };
    const C *X = q <= 1 ? a.Xp : q == 2 ? a.Xdy : a.Xdz;
    auto src = [&](int ln, const C *&A, const C *&B) {
        if (!active(ln)) return false;
        A = X + row0(ln) * a.lhx;
        B = A + a.lhx;
        return true;
    };
    // dpdx: i*kx times the y-inverse of p_hat.  On the two Hermitian rows packed as
    // Z = A + iB that is i*k_signed*Z (k_signed = kx(k) for bins k <= N/2, -kx(N-k) above)
    auto op = [&](int j, C(&x)[R0]) {
        if (q != 1) return;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int k = j + r * R1;
            const T kk = k <= N / 2 ? (T)a.kx[k] : -(T)a.kx[N - k];
            x[r] = mk<T>(-kk * x[r].y, kk * x[r].x);
        }
    };
    T fa[R1], fb[R1];
    T *f = nullptr, *out = nullptr, *bc = nullptr;
    bool act = false, proj = false;
    // the rows of the field to update are on their way while the exchange is read
    auto pre = [&](int ln, int j) {
        act = active(ln);
        const long long r0 = row0(act ? ln : 0);
        const int z = (int)(r0 / a.ny);
        const long long off = (r0 % a.ny) * a.ldx + j;
        proj = act && a.u && (q == 1 || q == 2 || (q == 3 && z >= (a.w_from_1 ? 1 : 2)));   // jz_min for w
        f = (q == 1 ? a.u : q == 2 ? a.v : a.w) + pl * z + off;
        out = q == 0 ? a.p + pl * z + off : (q == 1 ? a.dpdx : q == 2 ? a.dpdy : a.dpdz) + pl * (z - 1) + off;
        bc = act && q == 3 && a.zero_bc && (z == 1 || z == a.L) ? a.w + pl * (z == 1 ? 1 : z + 1) + off : nullptr;
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            fa[r] = proj ? f[r * R0] : (T)0;
            fb[r] = proj ? f[a.ldx + r * R0] : (T)0;
        }
    };
    // the update's rows into L2 before the first pass: one 128-byte line per lane
    if (q > 0 && a.u) {
        constexpr int EL = 128 / sizeof(T), PL = (N + EL - 1) / EL;
        for (int i = threadIdx.x; i < 2 * PL * G::WB; i += G::NTI) {
            const int ln = i / (2 * PL);
            if (!active(ln)) continue;
            const long long r0 = row0(ln);
            const T *p = (q == 1 ? a.u : q == 2 ? a.v : a.w) + pl * (r0 / a.ny) + (r0 % a.ny + (i / PL) % 2) * a.ldx + (i % PL) * EL;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        }
    }
    tp_rows_inv<T, N, WB_>(src, op, buf, a.twF, pre, [&](int, int j, const C(&x)[R1]) {
        if (!act) return;
        if (bc) {   // whole rows, pads included
#pragma unroll
            for (int r = 0; r < R1; ++r) bc[r * R0] = bc[a.ldx + r * R0] = (T)0;
            if (j < 2) bc[N] = bc[a.ldx + N] = (T)0;
        }
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            out[r * R0] = x[r].x;
            out[a.ldx + r * R0] = x[r].y;
            if (proj) {   // 110_project.f90:16-40: u = u + dt*(-tadv1*dpdx)
                f[r * R0] = fa[r] + (-a.dt_tadv1 * x[r].x);
                f[a.ldx + r * R0] = fb[r] + (-a.dt_tadv1 * x[r].y);
            }
        }
    });
}

template <typename T, int N>
__global__ void __launch_bounds__(TpRows<T, N>::NTI, TpRows<T, N>::minbI) k_tp_rows_pinv(PinvRowArgs<T> a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const unsigned nq = a.dpdz ? 4 : 3;
    tp_pinv_rows_unit<T, N>(a, (int)(blockIdx.x % nq), (long long)(blockIdx.x / nq) * TpRows<T, N>::WB, reinterpret_cast<C2<T> *>(smraw));
}

template <typename T> struct PinvLaunch {
    static cudaError_t cols(int n, const PinvColArgs<T> &a, int nlev, cudaStream_t s);
    static cudaError_t rows(int n, const PinvRowArgs<T> &a, cudaStream_t s);
};

template <typename T> struct FwdFusedLaunch {
    // returns cudaErrorNotSupported for lengths without an instantiation
    static cudaError_t run(int n, const FwdFusedArgs<T> &a, int nclusters, int csize, cudaStream_t s);
    static size_t slot_bytes(int n);
    static int max_clusters(int n, int csize);
};

} // namespace obl
