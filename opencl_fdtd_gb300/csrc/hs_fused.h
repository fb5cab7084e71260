// Arguments and launcher of the H kernel of fdtd_run (hs_fused.cu): H, optionally the Poynting
// vector of the step and the E update of the next one, in one launch.
#pragma once

#include "yee_common.cuh"
#include "monitors.h"

namespace fdtd {

// Threads of a block, one cell each; two blocks per SM. With the next step's E, 512 (64 registers a
// thread) ran a step of the 395x345x73 grid in 0.191 ms, 448 (72 registers) in 0.200; without it 448
// is the faster one, and with it where dt/mu or spacing tables take registers too (512 spills).
constexpr int hs_threads(bool ahead, bool mu, int dxmode) { return ahead && !mu && dxmode != 2 ? 512 : 448; }

// CPML faces of one axis, for the H update and for the next step's E update
template <typename R>
struct HSAxis {
    int32_t Tn, Tp;
    FacePsi<R> h, e;
};

template <typename R>
struct HSK {
    const R *E;            // E after this step's update and sources (read-only here)
    const R *HA;           // H before the update
    R *HB;                 // H after the update
    R *S, *oS;             // S every launch (with Poynting); oS only when write_oS
    const R *cm;           // dt/mu, NULL without mu
    R *EB;                 // E after the next step's update and sources (the E-ahead form)
    const R *ce;           // dt/eps
    uint32_t sx, sy, sz, syz;
    uint64_t N;
    R dt, inv_d, sf;
    const R *inv_de[3], *inv_dh[3];
    HSAxis<R> ax[3];
    // tiles of a plane: rows own rows by seglen own columns (a z row is nseg segments)
    uint32_t rows, seglen, nseg, ntile;
    uint32_t xchunk, nchunk;   // x planes per block, x chunks (ceil(sx / xchunk))
    int32_t write_oS;
    int32_t reverse;       // 1: the x chunks in descending order
    int32_t dft_on;        // 1: one extra block (the last) takes the step's DFT sample of E
    // point sources of the next step (E-ahead), as in YeeK
    int32_t nsrc, src_t, src_stride;
    const R *src_values;
    uint32_t src_x[YEE_SRC], src_j[YEE_SRC];
    int32_t src_c[YEE_SRC], src_col[YEE_SRC];
    R src_val[YEE_SRC];           // the step's values when src_values is NULL
    DftK<R> dft;
};

// Which form: MU, the spacing mode (0 dx = 1, 1 uniform, 2 tables), Poynting, E of the next step
struct HSForm {
    bool mu, poynting, ahead;
    int dxmode;
};

template <typename R>
bool hs_form_exists(const HSForm &f);
// pdl: launched with programmatic stream serialization
template <typename R>
cudaError_t launch_hs(const HSK<R> &k, const HSForm &f, bool pdl, cudaStream_t st);

}  // namespace fdtd
