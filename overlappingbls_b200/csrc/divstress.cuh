// divstress.cuh -- stress divergence: divt = ddx(tx) + ddy(ty) + dz(tz).
//
// divstress_uv / divstress_w (SBL/code/107_divstress.f90:4-104) add three derivative
// fields.  ddy(ty) is the plain column pass into divt; the row pass of ddx(tx) then adds
// the stored ddy and the vertical difference of tz as it stores (the reference forms the
// same sum, :36-37, :85-98), writes the two x pad columns as 0 (:40, :95) and fills the
// BOGUS levels.  Adding in the row pass rather than in the column pass: its reads and
// stores are whole rows, and no hook's registers sit beside a column butterfly.
#pragma once
#include "lines.cuh"

namespace obl {

template <typename T> struct DivRows {
    T *out;             // divt at level z0 (holds ddy(ty) when the rows run)
    const T *tz;        // tz at level z0
    long long plane;
    int ny;
    T rdz;              // 1/dz
    int fwd;            // 1: (tz(k+1) - tz(k)) / dz (ddz_w); 0: (tz(k) - tz(k-1)) / dz (ddz_uv)
    int zlo, zhi;       // planes of the pass that take the vertical term
    T *bogus[2];        // planes to fill (nullptr: none)
    T bogus_value;
};

// a: rows of tx, twF/twB and ktab of nx; a.dst is not used
template <typename T>
cudaError_t launch_rows_divt(int n, const RowArgs<T> &a, const DivRows<T> &e, cudaStream_t s);

} // namespace obl
