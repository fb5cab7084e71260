// Device helpers shared by the per-update kernels (yee_kernels.cu) and the H kernel of fdtd_run
// (hs_fused.cu): read-only loads, CPML depth lookup and the per-face CPML arithmetic.
#pragma once

#include "yee_common.cuh"

namespace fdtd {

// Coefficient tables, which no launch writes.
template <typename T>
__device__ __forceinline__ T ldg(const T *p) { return __ldg(p); }

// Fields, psi and what else the launch before may write, where the kernel itself does not write it: a
// coherent load that stays behind the wait of a dependent launch (grid_dependency_sync). Such a launch runs
// beside the one that writes them, while ld.global.nc, which __ldg and const restrict pointers become, is for
// data that stays as it is as long as the kernel lives. As an instruction that stays where it is written the
// load costs nothing (a step of 395x345x73 cells 0.196 ms either way); left to the compiler as *p the next
// plane's loads came too late (0.340 ms).
__device__ __forceinline__ float ldf(const float *p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ double ldf(const double *p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Depth index of the cell inside the face's slab, or -1 (update_e.cl:81-90). A 'p' face
// thicker than its axis never applies (the reference's unsigned s - T wraps).
__device__ __forceinline__ int pml_ir(int pol, int T, uint32_t s, uint32_t c)
{
    if (pol == 0) return (c < (uint32_t)T) ? (int)c : -1;
    if ((uint32_t)T <= s && c >= s - (uint32_t)T) return (int)(s - 1u - c);
    return -1;
}

// psi_u advances with the derivative of the v component along r and psi_v with that of the
// u component (update_e.cl:93-96); both derivatives along r are first scaled by p2 = 1/kappa.
// E-type kernels fold (psi_u, psi_v) into (P_u, P_v) with signs (-, +) for r in {x, z} and
// (+, -) for r = y (update_e.cl:73-77, 97-98); H-type kernels use the mirrored signs
// (update_h.cl:113-114). Returns the new (psi_u, psi_v).
template <typename R, bool ETYPE, int AX>
__device__ __forceinline__ void face_update(R p0, R p1, R p2, R su_old, R sv_old, R &su, R &sv,
                                            R &d_xy, R &d_xz, R &d_yx, R &d_yz, R &d_zx, R &d_zy,
                                            R &px, R &py, R &pz)
{
    R &dv = (AX == 0) ? d_zx : (AX == 1) ? d_zy : d_yz;
    R &du = (AX == 0) ? d_yx : (AX == 1) ? d_xy : d_xz;
    dv = dv * p2;
    du = du * p2;
    su = p0 * su_old + p1 * dv;
    sv = p0 * sv_old + p1 * du;
    R &pu = (AX == 0) ? py : px;
    R &pv = (AX == 2) ? py : pz;
    const bool plus_u = ETYPE ? (AX == 1) : (AX != 1);
    if (plus_u) { pu = pu + su; pv = pv - sv; }
    else        { pu = pu - su; pv = pv + sv; }
}

// psi index of cell (x, y, z) at depth ir of a face of axis AX with thickness T
template <int AX>
__device__ __forceinline__ uint32_t psi_index(uint32_t ir, uint32_t T, uint32_t x, uint32_t y,
                                              uint32_t z, uint32_t sy, uint32_t sz)
{
    if (AX == 0) return (ir * sy + y) * sz + z;
    if (AX == 1) return (x * T + ir) * sz + z;
    return (x * sy + y) * T + ir;
}

// CPML face of one axis for a coordinate: depth ir (-1 outside) and side (0 = 'n', 1 = 'p').
struct FaceAt {
    int ir, side;
};

__device__ __forceinline__ FaceAt face_at(int Tn, int Tp, uint32_t s, uint32_t c)
{
    FaceAt f;
    f.ir = -1;
    f.side = 0;
    if (c < (uint32_t)Tn) {
        f.ir = (int)c;
    } else if (Tp && c >= s - (uint32_t)Tp) {
        f.ir = (int)(s - 1u - c);
        f.side = 1;
    }
    return f;
}

// coefficient c (p0, p1, p2) at the face's depth; psi arrays read and written
template <typename R>
__device__ __forceinline__ R face_tab(const FacePsi<R> &a, const FaceAt &f, int c)
{
    return ldg((f.side ? a.tab[1][c] : a.tab[0][c]) + f.ir);
}

template <typename R>
__device__ __forceinline__ const R *face_A(const FacePsi<R> &a, const FaceAt &f, int c)
{
    return f.side ? a.A[1][c] : a.A[0][c];
}

template <typename R>
__device__ __forceinline__ R *face_B(const FacePsi<R> &a, const FaceAt &f, int c)
{
    return f.side ? a.B[1][c] : a.B[0][c];
}

// Per-thread view of one axis's CPML faces for a coordinate that stays fixed during the march
// (y or z): depth index (ir < 0 outside both faces), thickness, coefficients and psi arrays. AWAY:
// psi is written to other arrays than it is read from.
template <typename R, bool AWAY>
struct FixedFace {
    int ir;
    uint32_t T;
    R p0, p1, p2;
    R *pu, *pv;                 // written, and read unless AWAY
    const R *ru, *rv;

    __device__ __forceinline__ R u(uint32_t i) const { return AWAY ? ru[i] : pu[i]; }
    __device__ __forceinline__ R v(uint32_t i) const { return AWAY ? rv[i] : pv[i]; }
};

template <typename R, bool AWAY>
__device__ __forceinline__ FixedFace<R, AWAY> fixed_face(const AxisK<R> &a, uint32_t s, uint32_t c, bool act)
{
    FixedFace<R, AWAY> f;
    f.ir = -1;
    f.T = 0;
    f.p0 = f.p1 = f.p2 = R(0);
    f.pu = f.pv = nullptr;
    f.ru = f.rv = nullptr;
    const FaceAt at = face_at(a.Tn, a.Tp, s, c);
    if (act && at.ir >= 0) {
        f.ir = at.ir;
        f.T = (uint32_t)(at.side ? a.Tp : a.Tn);
        f.p0 = face_tab(a.f, at, 0);
        f.p1 = face_tab(a.f, at, 1);
        f.p2 = face_tab(a.f, at, 2);
        f.pu = face_B(a.f, at, 0);
        f.pv = face_B(a.f, at, 1);
        if (AWAY) {
            f.ru = face_A(a.f, at, 0);
            f.rv = face_A(a.f, at, 1);
        }
    }
    return f;
}

// True when an x face covers a plane of [xa, xb): what a block asks once, before its march.
template <typename R>
__device__ __forceinline__ bool x_faces(const AxisK<R> &a, uint32_t sx, uint32_t xa, uint32_t xb)
{
    return xa < (uint32_t)a.Tn || (a.Tp && xb > sx - (uint32_t)a.Tp);
}

}  // namespace fdtd
