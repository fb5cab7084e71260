// Batched stepping of many independent cavity variants.
//
// All variants' work is cut into tiles of BATCH_THREADS consecutive (y, z) cells times a chunk
// of x planes. Two schedules run the same tile code:
//   * per half-step: launches of one block per tile, one for E and one for H per step: of the tiles of all
//     variants that share launches, or of one variant, whose descriptor is then among the arguments
//     (k_batch_e1 / h1; large float32 variants). A launch starts while the one before drains;
//   * persistent: a cooperative grid of resident blocks takes the tiles of every variant
//     from a device work counter for the E half-step, synchronises the grid, does the same for
//     the H half-step, synchronises again, and repeats -- one launch advances the whole sweep by
//     nsteps steps.
// Point sources are added and monitor points recorded by the thread that updates the cell.
//
// Storage: E, H and dt/eps in float32, or in bfloat16 / float16 with float32 arithmetic. In
// 16-bit storage every tile (one component of the BATCH_TILE cells one warp updates in one x
// plane) carries a power-of-two exponent e: stored value = value * 2^-e, chosen when the tile
// is written so that the tile's largest magnitude lands in [2^13, 2^14) -- inside float16's
// normal range with headroom, whatever the field's absolute level (a ringdown decays through
// many decades). The warp reduces the new values' maximum with shuffles before it stores them
// (no barrier); tiles of a field are only rewritten in that field's half-step, when no other
// tile reads them.
//
// The float32 arithmetic and its order are those of the per-update kernels (this translation
// unit is compiled with --fmad=false), so float32 storage gives results bit-identical to
// stepping each variant on its own.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "batch.h"
#include "yee_device.cuh"

namespace cg = cooperative_groups;

namespace fdtd {

namespace {

template <int ST>
struct Store;

template <>
struct Store<BATCH_F32> {
    using T = float;
    static constexpr bool scaled = false;
    __device__ static float dec(T v) { return v; }
    __device__ static T enc(float v) { return v; }
};

template <>
struct Store<BATCH_BF16> {
    using T = __nv_bfloat16;
    static constexpr bool scaled = true;
    __device__ static float dec(T v) { return __bfloat162float(v); }
    __device__ static T enc(float v) { return __float2bfloat16_rn(v); }
};

template <>
struct Store<BATCH_F16> {
    using T = __half;
    static constexpr bool scaled = true;
    __device__ static float dec(T v) { return __half2float(v); }
    __device__ static T enc(float v) { return __float2half_rn(v); }
};

template <>
struct Store<BATCH_BF16U> {
    using T = __nv_bfloat16;
    static constexpr bool scaled = false;
    __device__ static float dec(T v) { return __bfloat162float(v); }
    __device__ static T enc(float v) { return __float2bfloat16_rn(v); }
};

// 2^e for e in [-126, 127] (exact)
__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }

// exponent of a tile whose largest magnitude is m: m * 2^-e in [2^13, 2^14)
__device__ __forceinline__ int tile_exp(float m)
{
    if (!(m > 0.f) || !isfinite(m)) return 0;
    int E;
    frexpf(m, &E);
    return max(-100, min(100, E - 14));
}

// exponent word of plane x, tile jt (= cell j / BATCH_TILE): the three components' exponents
// e_c as bytes e_c + 128 in bits 8c .. 8c + 7
__device__ __forceinline__ uint32_t texp_index(const BVar &v, uint32_t x, uint32_t jt)
{
    return x * v.ntl + jt;
}

__device__ __forceinline__ int xe(int32_t word, int c) { return (int)(((uint32_t)word >> (8 * c)) & 0xffu) - 128; }

__device__ __forceinline__ int32_t xpack(int e0, int e1, int e2)
{
    return (int32_t)((uint32_t)(e0 + 128) | ((uint32_t)(e1 + 128) << 8) | ((uint32_t)(e2 + 128) << 16));
}

// Largest magnitude of each of three values over the warp (all 32 lanes take part; idle lanes
// pass 0): the tile exponents, identical in every lane. The bit patterns of non-negative floats
// order like the values, so one integer warp reduction per component finds the maximum.
__device__ __forceinline__ void warp_exps(float a, float b, float c, int &ea, int &eb, int &ec)
{
    const uint32_t ma = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(a)));
    const uint32_t mb = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(b)));
    const uint32_t mc = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(c)));
    ea = tile_exp(__uint_as_float(ma));
    eb = tile_exp(__uint_as_float(mb));
    ec = tile_exp(__uint_as_float(mc));
}

// CPML face of one axis fixed for the thread (y or z) of update H (0: E, 1: H): depth, coefficients,
// thickness and psi. A store may alias the descriptor, so what is read through it is loaded again for
// every plane: KEEP holds thickness and psi in registers instead.
template <int H, bool KEEP>
struct BFix {
    const BAxis &a;
    int ir, side;
    float p0, p1, p2;
    uint32_t T_;
    float *u_, *v_;

    __device__ __forceinline__ uint32_t T() const { return KEEP ? T_ : (uint32_t)(side ? a.Tp : a.Tn); }
    __device__ __forceinline__ float *u() const { return KEEP ? u_ : a.psi[H][side][0]; }
    __device__ __forceinline__ float *v() const { return KEEP ? v_ : a.psi[H][side][1]; }
};

template <int h, bool KEEP>
__device__ __forceinline__ BFix<h, KEEP> bfix(const BAxis &a, uint32_t s, uint32_t c, bool act)
{
    BFix<h, KEEP> f = {a, -1, 0, 0.f, 0.f, 0.f, 0u, nullptr, nullptr};
    const FaceAt at = face_at(a.Tn, a.Tp, s, c);
    if (act && at.ir >= 0) {
        f.ir = at.ir;
        f.side = at.side;
        f.T_ = (uint32_t)(at.side ? a.Tp : a.Tn);
        f.p0 = ldg(a.tab[h][at.side][0] + at.ir);
        f.p1 = ldg(a.tab[h][at.side][1] + at.ir);
        f.p2 = ldg(a.tab[h][at.side][2] + at.ir);
        f.u_ = a.psi[h][at.side][0];
        f.v_ = a.psi[h][at.side][1];
    }
    return f;
}

// decode of a stored value with its tile exponent (no scaling at all in float32 storage)
template <int ST>
__device__ __forceinline__ float dv(typename Store<ST>::T v, int e)
{
    return Store<ST>::scaled ? Store<ST>::dec(v) * pow2(e) : Store<ST>::dec(v);
}

// ---- E half-step of one tile (update_e.cl:39-107 per cell) ------------------------------------
// Values one E plane reads (stored form and tile exponents).
template <typename T>
struct BELoad {
    T hx, hy, hz, nxy, nxz, nyz, nzy, ex, ey, ez, cx, cy, cz;
    int32_t gh, gy, gz, ge;        // exponent words: own H tile, H at y-1, H at z-1, own E tile
    float xu, xv, yu, yv, zu, zv;
};

template <int ST, bool KEEP, bool LATE = false>
__device__ void batch_e_tile(const BVar &v, int4 tl, const int64_t *counter, int t, int64_t rows)
{
    using SS = Store<ST>;
    using T = typename SS::T;
    const uint32_t sx = v.sx, sy = v.sy, sz = v.sz, syz = v.syz;
    const uint64_t N = v.N;
    const uint32_t xa = (uint32_t)tl.y, xb = (uint32_t)tl.z, jb = (uint32_t)tl.w;
    const uint32_t j = jb * BATCH_THREADS + threadIdx.x;
    const bool act = j < syz;
    const uint32_t y = act ? v.dsz.div(j) : 0u;
    const uint32_t z = act ? j - y * sz : 0u;
    const T *const Hx = (const T *)v.H, *const Hy = Hx + N, *const Hz = Hx + 2 * N;
    T *const Ex = (T *)v.E, *const Ey = Ex + N, *const Ez = Ex + 2 * N;
    const T *const Cx = (const T *)v.ce, *const Cy = Cx + N, *const Cz = Cx + 2 * N;
    const int32_t *const hexp = v.hexp;
    int32_t *const eexp = v.eexp;
    // minus neighbours with periodic wrap (common.cl:75-81), 32-bit modular offsets
    const uint32_t dmy = y ? 0u - sz : (sy - 1u) * sz;
    const uint32_t dmz = z ? 0xffffffffu : sz - 1u;
    const uint32_t jt = j / BATCH_TILE;                          // own exponent tile
    const uint32_t jby = (j + dmy) / BATCH_TILE, jbz = (j + dmz) / BATCH_TILE;
    if (LATE) grid_dependency_sync();                            // the tables are the caller's
    const BFix<0, KEEP> fy = bfix<0, KEEP>(v.ax[1], sy, y, act);
    const BFix<0, KEEP> fz = bfix<0, KEEP>(v.ax[2], sz, z, act);
    // what the march needs of the descriptor in registers: a store may alias it, and a value read
    // through it would be loaded again for every plane
    const float inv = v.inv_d;
    const bool scale = v.dxmode != 0;
    const BAxis &ax0 = v.ax[0];
    const int Tn = ax0.Tn, Tp = ax0.Tp;
    const bool xf = xa < (uint32_t)Tn || (Tp && xb > sx - (uint32_t)Tp);   // an x face covers a plane of the tile
    // a point source, a monitor point in this tile (block-uniform)
    bool srcs = false, mons = false;
    const int64_t step = *counter + t;
    if (step < rows) {
        for (int s = 0; s < v.nsrc; ++s)
            srcs |= v.src_j[s] / BATCH_THREADS == jb && v.src_x[s] >= xa && v.src_x[s] < xb;
        for (int m = 0; m < v.nmon; ++m)
            mons |= v.mon_j[m] / BATCH_THREADS == jb && v.mon_x[m] >= xa && v.mon_x[m] < xb;
    }

    auto load = [&](uint32_t x, uint32_t i) {
        BELoad<T> q;
        const uint32_t imy = i + dmy, imz = i + dmz;   // 32-bit wrap arithmetic
        q.hx = Hx[i]; q.hy = Hy[i]; q.hz = Hz[i];
        q.nxy = Hx[imy]; q.nzy = Hz[imy];
        q.nxz = Hx[imz]; q.nyz = Hy[imz];
        q.ex = Ex[i]; q.ey = Ey[i]; q.ez = Ez[i];
        q.cx = Cx[i]; q.cy = Cy[i]; q.cz = Cz[i];
        if (SS::scaled) {
            q.gh = hexp[texp_index(v, x, jt)];
            q.gy = hexp[texp_index(v, x, jby)];
            q.gz = hexp[texp_index(v, x, jbz)];
            q.ge = eexp[texp_index(v, x, jt)];
        }
        q.xu = q.xv = q.yu = q.yv = q.zu = q.zv = 0.f;
        if (xf) {
            const FaceAt fx = face_at(Tn, Tp, sx, x);
            if (fx.ir >= 0) {
                const uint32_t ip = (uint32_t)fx.ir * syz + j;
                q.xu = ax0.psi[0][fx.side][0][ip]; q.xv = ax0.psi[0][fx.side][1][ip];
            }
        }
        if (fy.ir >= 0) {
            const uint32_t ip = (x * fy.T() + (uint32_t)fy.ir) * sz + z;
            q.yu = fy.u()[ip]; q.yv = fy.v()[ip];
        }
        if (fz.ir >= 0) {
            const uint32_t ip = (x * sy + y) * fz.T() + (uint32_t)fz.ir;
            q.zu = fz.u()[ip]; q.zv = fz.v()[ip];
        }
        return q;
    };

    float hy_m = 0.f, hz_m = 0.f;
    if (act) {
        const uint32_t xm = xa ? xa - 1u : sx - 1u;
        const uint32_t im = xm * syz + j;
        const int32_t wm = SS::scaled ? hexp[texp_index(v, xm, jt)] : 0;
        hy_m = dv<ST>(Hy[im], xe(wm, 1));
        hz_m = dv<ST>(Hz[im], xe(wm, 2));
    }
    uint32_t i = xa * syz + j;
    for (uint32_t x = xa; x < xb; ++x, i += syz) {
        float nx = 0.f, ny = 0.f, nz = 0.f, hy = 0.f, hz = 0.f;
        if (act) {
            const BELoad<T> cur = load(x, i);
            const float hx = dv<ST>(cur.hx, xe(cur.gh, 0));
            hy = dv<ST>(cur.hy, xe(cur.gh, 1));
            hz = dv<ST>(cur.hz, xe(cur.gh, 2));
            // backward differences (update_e.cl:39-46), times 1/dx
            float d_xy = hx - dv<ST>(cur.nxy, xe(cur.gy, 0));
            float d_xz = hx - dv<ST>(cur.nxz, xe(cur.gz, 0));
            float d_yx = hy - hy_m;
            float d_yz = hy - dv<ST>(cur.nyz, xe(cur.gz, 1));
            float d_zx = hz - hz_m;
            float d_zy = hz - dv<ST>(cur.nzy, xe(cur.gy, 2));
            if (scale) {
                d_xy = d_xy * inv; d_xz = d_xz * inv; d_yx = d_yx * inv;
                d_yz = d_yz * inv; d_zx = d_zx * inv; d_zy = d_zy * inv;
            }
            // CPML (update_e.cl:64-100): at most one face per axis
            float px = 0.f, py = 0.f, pz = 0.f;
            if (xf) {
                const FaceAt fx = face_at(Tn, Tp, sx, x);
                if (fx.ir >= 0) {
                    float su, sv;
                    face_update<float, true, 0>(ldg(ax0.tab[0][fx.side][0] + fx.ir), ldg(ax0.tab[0][fx.side][1] + fx.ir),
                                              ldg(ax0.tab[0][fx.side][2] + fx.ir), cur.xu, cur.xv, su, sv,
                                              d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
                    const uint32_t ip = (uint32_t)fx.ir * syz + j;
                    ax0.psi[0][fx.side][0][ip] = su;
                    ax0.psi[0][fx.side][1][ip] = sv;
                }
            }
            if (fy.ir >= 0) {
                float su, sv;
                face_update<float, true, 1>(fy.p0, fy.p1, fy.p2, cur.yu, cur.yv, su, sv,
                                          d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
                const uint32_t ip = (x * fy.T() + (uint32_t)fy.ir) * sz + z;
                fy.u()[ip] = su;
                fy.v()[ip] = sv;
            }
            if (fz.ir >= 0) {
                float su, sv;
                face_update<float, true, 2>(fz.p0, fz.p1, fz.p2, cur.zu, cur.zv, su, sv,
                                          d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
                const uint32_t ip = (x * sy + y) * fz.T() + (uint32_t)fz.ir;
                fz.u()[ip] = su;
                fz.v()[ip] = sv;
            }
            // update_e.cl:105-107
            nx = dv<ST>(cur.ex, xe(cur.ge, 0)) + SS::dec(cur.cx) * ((d_zy - d_yz) + px);
            ny = dv<ST>(cur.ey, xe(cur.ge, 1)) + SS::dec(cur.cy) * ((d_xz - d_zx) + py);
            nz = dv<ST>(cur.ez, xe(cur.ge, 2)) + SS::dec(cur.cz) * ((d_yx - d_xy) + pz);
            // point sources after the update (fdtd.py:168-169: E[ind] += value)
            if (srcs) {
                for (int s = 0; s < v.nsrc; ++s) {
                    if (v.src_x[s] != x || v.src_j[s] != j) continue;
                    const float val = v.src_values[step * v.nsrc + s];
                    if (v.src_c[s] == 0) nx = nx + val;
                    else if (v.src_c[s] == 1) ny = ny + val;
                    else nz = nz + val;
                }
            }
        }
        int e0 = 0, e1 = 0, e2 = 0;
        if (SS::scaled) {
            warp_exps(nx, ny, nz, e0, e1, e2);
            if ((threadIdx.x & 31u) == 0 && jt < v.ntl) eexp[texp_index(v, x, jt)] = xpack(e0, e1, e2);
        }
        if (act) {
            const T wx = SS::enc(SS::scaled ? nx * pow2(-e0) : nx);
            const T wy = SS::enc(SS::scaled ? ny * pow2(-e1) : ny);
            const T wz = SS::enc(SS::scaled ? nz * pow2(-e2) : nz);
            Ex[i] = wx;
            Ey[i] = wy;
            Ez[i] = wz;
            if (mons) {
                for (int m = 0; m < v.nmon; ++m) {
                    if (v.mon_x[m] != x || v.mon_j[m] != j) continue;
                    const int c = v.mon_c[m];
                    const T w = c == 0 ? wx : c == 1 ? wy : wz;
                    v.series[step * v.nmon + m] = (double)dv<ST>(w, c == 0 ? e0 : c == 1 ? e1 : e2);
                }
            }
            hy_m = hy;
            hz_m = hz;
        }
    }
}

// ---- H half-step of one tile (update_h.cl:36-131 per cell; Poynting off) ----------------------
template <typename T>
struct BHLoad {
    T ex1, ey1, ez1, rxy, rxz, ryz, rzy, hx, hy, hz;
    int32_t ge, gy, gz, gh;        // exponent words: E at x+1, E at y+1, E at z+1, own H tile
    float xu, xv, yu, yv, zu, zv;
};

template <int ST, bool KEEP, bool LATE = false>
__device__ void batch_h_tile(const BVar &v, int4 tl)
{
    using SS = Store<ST>;
    using T = typename SS::T;
    const uint32_t sx = v.sx, sy = v.sy, sz = v.sz, syz = v.syz;
    const uint64_t N = v.N;
    const uint32_t xa = (uint32_t)tl.y, xb = (uint32_t)tl.z, jb = (uint32_t)tl.w;
    const uint32_t j = jb * BATCH_THREADS + threadIdx.x;
    const bool act = j < syz;
    const uint32_t y = act ? v.dsz.div(j) : 0u;
    const uint32_t z = act ? j - y * sz : 0u;
    const T *const Ex = (const T *)v.E, *const Ey = Ex + N, *const Ez = Ex + 2 * N;
    T *const Hx = (T *)v.H, *const Hy = Hx + N, *const Hz = Hx + 2 * N;
    int32_t *const hexp = v.hexp;
    const int32_t *const eexp = v.eexp;
    // plus neighbours with periodic wrap (common.cl:82-84)
    const uint32_t dpy = (y + 1u < sy) ? sz : 0u - (sy - 1u) * sz;
    const uint32_t dpz = (z + 1u < sz) ? 1u : 0u - (sz - 1u);
    const uint32_t jt = j / BATCH_TILE;
    const uint32_t jby = (j + dpy) / BATCH_TILE, jbz = (j + dpz) / BATCH_TILE;
    if (LATE) grid_dependency_sync();                            // the tables are the caller's
    const BFix<1, KEEP> fy = bfix<1, KEEP>(v.ax[1], sy, y, act);
    const BFix<1, KEEP> fz = bfix<1, KEEP>(v.ax[2], sz, z, act);
    const float inv = v.inv_d, dt = v.dt;
    const bool scale = v.dxmode != 0;
    const BAxis &ax0 = v.ax[0];
    const int Tn = ax0.Tn, Tp = ax0.Tp;
    const bool xf = xa < (uint32_t)Tn || (Tp && xb > sx - (uint32_t)Tp);

    auto load = [&](uint32_t x, uint32_t i) {
        BHLoad<T> q;
        const uint32_t x1 = (x + 1u < sx) ? x + 1u : 0u;
        const uint32_t i1 = x1 * syz + j;
        const uint32_t ipy = i + dpy, ipz = i + dpz;   // 32-bit wrap arithmetic
        q.ex1 = Ex[i1]; q.ey1 = Ey[i1]; q.ez1 = Ez[i1];
        q.rxy = Ex[ipy]; q.rzy = Ez[ipy];
        q.rxz = Ex[ipz]; q.ryz = Ey[ipz];
        q.hx = Hx[i]; q.hy = Hy[i]; q.hz = Hz[i];
        if (SS::scaled) {
            q.ge = eexp[texp_index(v, x1, jt)];
            q.gy = eexp[texp_index(v, x, jby)];
            q.gz = eexp[texp_index(v, x, jbz)];
            q.gh = hexp[texp_index(v, x, jt)];
        }
        q.xu = q.xv = q.yu = q.yv = q.zu = q.zv = 0.f;
        if (xf) {
            const FaceAt fx = face_at(Tn, Tp, sx, x);
            if (fx.ir >= 0) {
                const uint32_t ip = (uint32_t)fx.ir * syz + j;
                q.xu = ax0.psi[1][fx.side][0][ip]; q.xv = ax0.psi[1][fx.side][1][ip];
            }
        }
        if (fy.ir >= 0) {
            const uint32_t ip = (x * fy.T() + (uint32_t)fy.ir) * sz + z;
            q.yu = fy.u()[ip]; q.yv = fy.v()[ip];
        }
        if (fz.ir >= 0) {
            const uint32_t ip = (x * sy + y) * fz.T() + (uint32_t)fz.ir;
            q.zu = fz.u()[ip]; q.zv = fz.v()[ip];
        }
        return q;
    };

    float ex = 0.f, ey = 0.f, ez = 0.f;
    if (act) {
        const uint32_t i = xa * syz + j;
        const int32_t wa = SS::scaled ? eexp[texp_index(v, xa, jt)] : 0;
        ex = dv<ST>(Ex[i], xe(wa, 0));
        ey = dv<ST>(Ey[i], xe(wa, 1));
        ez = dv<ST>(Ez[i], xe(wa, 2));
    }
    uint32_t i = xa * syz + j;
    for (uint32_t x = xa; x < xb; ++x, i += syz) {
        float nx = 0.f, ny = 0.f, nz = 0.f, ex1 = 0.f, ey1 = 0.f, ez1 = 0.f;
        if (act) {
            const BHLoad<T> cur = load(x, i);
            ex1 = dv<ST>(cur.ex1, xe(cur.ge, 0));
            ey1 = dv<ST>(cur.ey1, xe(cur.ge, 1));
            ez1 = dv<ST>(cur.ez1, xe(cur.ge, 2));
            // forward differences (update_h.cl:36-43), times 1/dx
            float d_xy = dv<ST>(cur.rxy, xe(cur.gy, 0)) - ex;
            float d_xz = dv<ST>(cur.rxz, xe(cur.gz, 0)) - ex;
            float d_yx = ey1 - ey;
            float d_yz = dv<ST>(cur.ryz, xe(cur.gz, 1)) - ey;
            float d_zx = ez1 - ez;
            float d_zy = dv<ST>(cur.rzy, xe(cur.gy, 2)) - ez;
            if (scale) {
                d_xy = d_xy * inv; d_xz = d_xz * inv; d_yx = d_yx * inv;
                d_yz = d_yz * inv; d_zx = d_zx * inv; d_zy = d_zy * inv;
            }
            float px = 0.f, py = 0.f, pz = 0.f;
            if (xf) {
                const FaceAt fx = face_at(Tn, Tp, sx, x);
                if (fx.ir >= 0) {
                    float su, sv;
                    face_update<float, false, 0>(ldg(ax0.tab[1][fx.side][0] + fx.ir), ldg(ax0.tab[1][fx.side][1] + fx.ir),
                                              ldg(ax0.tab[1][fx.side][2] + fx.ir), cur.xu, cur.xv, su, sv,
                                              d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
                    const uint32_t ip = (uint32_t)fx.ir * syz + j;
                    ax0.psi[1][fx.side][0][ip] = su;
                    ax0.psi[1][fx.side][1][ip] = sv;
                }
            }
            if (fy.ir >= 0) {
                float su, sv;
                face_update<float, false, 1>(fy.p0, fy.p1, fy.p2, cur.yu, cur.yv, su, sv,
                                          d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
                const uint32_t ip = (x * fy.T() + (uint32_t)fy.ir) * sz + z;
                fy.u()[ip] = su;
                fy.v()[ip] = sv;
            }
            if (fz.ir >= 0) {
                float su, sv;
                face_update<float, false, 2>(fz.p0, fz.p1, fz.p2, cur.zu, cur.zv, su, sv,
                                          d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
                const uint32_t ip = (x * sy + y) * fz.T() + (uint32_t)fz.ir;
                fz.u()[ip] = su;
                fz.v()[ip] = sv;
            }
            // update_h.cl:129-131
            nx = dv<ST>(cur.hx, xe(cur.gh, 0)) - dt * ((d_zy - d_yz) - px);
            ny = dv<ST>(cur.hy, xe(cur.gh, 1)) - dt * ((d_xz - d_zx) - py);
            nz = dv<ST>(cur.hz, xe(cur.gh, 2)) - dt * ((d_yx - d_xy) - pz);
        }
        int e0 = 0, e1 = 0, e2 = 0;
        if (SS::scaled) {
            warp_exps(nx, ny, nz, e0, e1, e2);
            if ((threadIdx.x & 31u) == 0 && jt < v.ntl) hexp[texp_index(v, x, jt)] = xpack(e0, e1, e2);
        }
        if (act) {
            Hx[i] = SS::enc(SS::scaled ? nx * pow2(-e0) : nx);
            Hy[i] = SS::enc(SS::scaled ? ny * pow2(-e1) : ny);
            Hz[i] = SS::enc(SS::scaled ? nz * pow2(-e2) : nz);
            ex = ex1;
            ey = ey1;
            ez = ez1;
        }
    }
}

template <int ST>
__device__ __forceinline__ void batch_e_item(const BatchK &k, uint32_t ti, int t)
{
    const int4 tl = k.tiles[ti];
    batch_e_tile<ST, false>(k.vars[tl.x], tl, k.step, t, k.rows);
}

template <int ST>
__device__ __forceinline__ void batch_h_item(const BatchK &k, uint32_t ti)
{
    const int4 tl = k.tiles[ti];
    batch_h_tile<ST, false>(k.vars[tl.x], tl);
}

// next tile of the half-step whose counter is `ctr` (>= ntiles: none left)
__device__ __forceinline__ uint32_t next_tile(uint32_t *ctr, uint32_t *slot)
{
    __syncthreads();                                     // every thread has read the last one
    if (threadIdx.x == 0) *slot = atomicAdd(ctr, 1u);
    __syncthreads();
    return *slot;
}

// Persistent form: the E and H tile bodies together at four resident blocks per SM (64 registers; the
// descriptor is read again where it is used).
constexpr int BATCH_PERSIST_BLOCKS = 4;

template <int ST>
__global__ void __launch_bounds__(BATCH_THREADS, BATCH_PERSIST_BLOCKS) k_batch(const BatchK k)
{
    __shared__ uint32_t item;
    cg::grid_group grid = cg::this_grid();
    const int64_t step0 = *k.step;
    for (int t = 0; t < k.nsteps; ++t) {
        // half-step 2t uses counter 0, 2t + 1 counter 1; a counter is cleared right after the
        // grid barrier that ends its half-step, two barriers before its next use
        for (uint32_t ti = next_tile(&k.work[0], &item); ti < k.ntiles; ti = next_tile(&k.work[0], &item))
            batch_e_item<ST>(k, ti, t);
        grid.sync();
        if (blockIdx.x == 0 && threadIdx.x == 0) k.work[0] = 0u;
        for (uint32_t ti = next_tile(&k.work[1], &item); ti < k.ntiles; ti = next_tile(&k.work[1], &item))
            batch_h_item<ST>(k, ti);
        grid.sync();
        if (blockIdx.x == 0 && threadIdx.x == 0) k.work[1] = 0u;
    }
    // every block read the step counter before its first grid barrier
    if (blockIdx.x == 0 && threadIdx.x == 0) *k.step = step0 + k.nsteps;
}

// One tile per block, all variants' tiles in one launch per half-step. Both bodies wait on memory, so
// what counts is resident warps and a march without reloads: with the next plane loaded ahead (three
// blocks per SM) and the descriptor's pointers, limits and source list read again for every plane, the
// march was 261 (E) and 220 (H) instructions per warp and plane and a step of 8 variants (14.7 M cells)
// took 0.389 ms in float32, 0.420 in bfloat16 without exponents and 0.619 with; now 184 and 163 and 0.331,
// 0.297 and 0.406. E in float32 spills 56 bytes at five blocks and still gains (0.208 to 0.184 ms, four to
// five); H loses there (0.146 to 0.163), and so does E with tile exponents. Six blocks: 0.211 and 0.174.
// A call's last H launch advances the step counter.
template <int ST>
constexpr int batch_e_blocks() { return Store<ST>::scaled ? 4 : 5; }

template <int ST>
__global__ void __launch_bounds__(BATCH_THREADS, batch_e_blocks<ST>()) k_batch_e(const BatchK k)
{
    const int4 tl = k.tiles[blockIdx.x];
    grid_dependency_sync();
    batch_e_tile<ST, true>(k.vars[tl.x], tl, k.step, k.t, k.rows);
}

template <int ST>
__global__ void __launch_bounds__(BATCH_THREADS, 4) k_batch_h(const BatchK k)
{
    const int4 tl = k.tiles[blockIdx.x];
    grid_dependency_sync();
    batch_h_tile<ST, true>(k.vars[tl.x], tl);
    // the last launch of a call: the E launches, which read the counter, have completed
    if (k.advance && blockIdx.x == 0 && threadIdx.x == 0) *k.step += k.advance;
}

// One variant per launch, its descriptor among the kernel's arguments (five blocks per SM: 0.317 ms a step
// instead of 0.306); index arithmetic stands before the wait (0.304), chunks by fit_xchunk (0.279).
constexpr int BATCH_ONE_BLOCKS = 4;

__global__ void __launch_bounds__(BATCH_THREADS, BATCH_ONE_BLOCKS) k_batch_e1(const __grid_constant__ BatchOne k)
{
    const uint32_t xa = blockIdx.y * k.xchunk;
    const int4 tl = make_int4(0, (int)xa, (int)min(xa + k.xchunk, k.v.sx), (int)blockIdx.x);
    batch_e_tile<BATCH_F32, true, true>(k.v, tl, k.step, k.t, k.rows);
}

__global__ void __launch_bounds__(BATCH_THREADS, BATCH_ONE_BLOCKS) k_batch_h1(const __grid_constant__ BatchOne k)
{
    const uint32_t xa = blockIdx.y * k.xchunk;
    const int4 tl = make_int4(0, (int)xa, (int)min(xa + k.xchunk, k.v.sx), (int)blockIdx.x);
    batch_h_tile<BATCH_F32, true, true>(k.v, tl);
    if (k.advance && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *k.step += k.advance;
}

// one block per (column jb of BATCH_THREADS cells, plane x): float32 <-> storage, all three
// components of a cell per thread, one exponent word per warp tile
template <int ST>
__global__ void __launch_bounds__(BATCH_THREADS) k_batch_encode(const BVar v, int field, const float *src)
{
    using SS = Store<ST>;
    using T = typename SS::T;
    const uint32_t jb = blockIdx.x, x = blockIdx.y;
    const uint32_t j = jb * BATCH_THREADS + threadIdx.x;
    const bool act = j < v.syz;
    const uint64_t i = (uint64_t)x * v.syz + j;
    float val[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) val[c] = act ? src[(uint64_t)c * v.N + i] : 0.f;
    int e[3] = {0, 0, 0};
    if (SS::scaled) warp_exps(val[0], val[1], val[2], e[0], e[1], e[2]);
    T *dst = (T *)(field ? v.H : v.E);
    if (act) {
#pragma unroll
        for (int c = 0; c < 3; ++c) dst[(uint64_t)c * v.N + i] = SS::enc(SS::scaled ? val[c] * pow2(-e[c]) : val[c]);
    }
    const uint32_t jt = j / BATCH_TILE;
    if (SS::scaled && (threadIdx.x & 31u) == 0 && jt < v.ntl)
        (field ? v.hexp : v.eexp)[texp_index(v, x, jt)] = xpack(e[0], e[1], e[2]);
}

template <int ST>
__global__ void __launch_bounds__(BATCH_THREADS) k_batch_decode(const BVar v, int field, float *dst)
{
    using SS = Store<ST>;
    using T = typename SS::T;
    const uint32_t jb = blockIdx.x, x = blockIdx.y;
    const uint32_t j = jb * BATCH_THREADS + threadIdx.x;
    if (j >= v.syz) return;
    const uint64_t i = (uint64_t)x * v.syz + j;
    const T *src = (const T *)(field ? v.H : v.E);
    const int32_t w = SS::scaled ? (field ? v.hexp : v.eexp)[texp_index(v, x, j / BATCH_TILE)] : 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) dst[(uint64_t)c * v.N + i] = dv<ST>(src[(uint64_t)c * v.N + i], xe(w, c));
}

}  // namespace

template <int ST>
int batch_max_blocks_per_sm()
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_batch<ST>, BATCH_THREADS, 0) != cudaSuccess) return 0;
    return n;
}

template <int ST>
cudaError_t launch_batch(const BatchK &k, int blocks, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks, 1, 1);
    cfg.blockDim = dim3(BATCH_THREADS, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_batch<ST>, k);
}

template <int ST>
cudaError_t launch_batch_steps(const BatchK &kk, const BVar *const *groups, int n, uint32_t xchunk, cudaStream_t st)
{
    BatchK k = kk;
    BatchOne o;
    o.step = k.step;
    o.rows = k.rows;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    for (int g = 0; g < n; ++g) {
        const BVar *const one = groups[g];
        dim3 grid(k.ntiles, 1, 1);
        if (one) {
            o.v = *one;
            o.xchunk = xchunk ? xchunk : fit_xchunk(one->njb, one->sx, (uint64_t)sms * BATCH_ONE_BLOCKS);
            // the chunks are the grid's y extent, at most 65535
            const uint32_t least = (one->sx + 65534u) / 65535u;
            if (o.xchunk < least) o.xchunk = least;
            grid = dim3(one->njb, (one->sx + o.xchunk - 1) / o.xchunk, 1);
        }
        for (int t = 0; t < kk.nsteps && e == cudaSuccess; ++t) {
            const int advance = g == n - 1 && t == kk.nsteps - 1 ? kk.nsteps : 0;
            k.t = o.t = t;
            k.advance = o.advance = advance;
            // a block's launch overlaps the tail of the launch before: 8 variants of 1.8 M cells 0.337 to 0.331
            // ms a step, two of 0.1 M 19 to 14 us (the set-up before the wait as well: 0.355 ms and 12 us)
            if (one) {
                if constexpr (ST == BATCH_F32) {             // launched_alone
                    e = launch_dependent(k_batch_e1, grid, BATCH_THREADS, st, true, o);
                    if (e == cudaSuccess) e = launch_dependent(k_batch_h1, grid, BATCH_THREADS, st, true, o);
                }
            } else {
                e = launch_dependent(k_batch_e<ST>, grid, BATCH_THREADS, st, true, k);
                if (e == cudaSuccess) e = launch_dependent(k_batch_h<ST>, grid, BATCH_THREADS, st, true, k);
            }
        }
    }
    return e;
}

cudaError_t launch_batch_encode(int store, const BVar &v, int field, const float *src, cudaStream_t st)
{
    const dim3 g(v.njb, v.sx, 1);
    if (store == BATCH_BF16) k_batch_encode<BATCH_BF16><<<g, BATCH_THREADS, 0, st>>>(v, field, src);
    else if (store == BATCH_F16) k_batch_encode<BATCH_F16><<<g, BATCH_THREADS, 0, st>>>(v, field, src);
    else if (store == BATCH_BF16U) k_batch_encode<BATCH_BF16U><<<g, BATCH_THREADS, 0, st>>>(v, field, src);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_batch_decode(int store, const BVar &v, int field, float *dst, cudaStream_t st)
{
    const dim3 g(v.njb, v.sx, 1);
    if (store == BATCH_BF16) k_batch_decode<BATCH_BF16><<<g, BATCH_THREADS, 0, st>>>(v, field, dst);
    else if (store == BATCH_F16) k_batch_decode<BATCH_F16><<<g, BATCH_THREADS, 0, st>>>(v, field, dst);
    else if (store == BATCH_BF16U) k_batch_decode<BATCH_BF16U><<<g, BATCH_THREADS, 0, st>>>(v, field, dst);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

template cudaError_t launch_batch<BATCH_F32>(const BatchK &, int, cudaStream_t);
template cudaError_t launch_batch<BATCH_BF16>(const BatchK &, int, cudaStream_t);
template cudaError_t launch_batch<BATCH_F16>(const BatchK &, int, cudaStream_t);
template cudaError_t launch_batch_steps<BATCH_F32>(const BatchK &, const BVar *const *, int, uint32_t, cudaStream_t);
template cudaError_t launch_batch_steps<BATCH_BF16>(const BatchK &, const BVar *const *, int, uint32_t, cudaStream_t);
template cudaError_t launch_batch_steps<BATCH_F16>(const BatchK &, const BVar *const *, int, uint32_t, cudaStream_t);
template int batch_max_blocks_per_sm<BATCH_F32>();
template int batch_max_blocks_per_sm<BATCH_BF16>();
template int batch_max_blocks_per_sm<BATCH_F16>();
template cudaError_t launch_batch<BATCH_BF16U>(const BatchK &, int, cudaStream_t);
template cudaError_t launch_batch_steps<BATCH_BF16U>(const BatchK &, const BVar *const *, int, uint32_t, cudaStream_t);
template int batch_max_blocks_per_sm<BATCH_BF16U>();

}  // namespace fdtd
