// The H kernel of fdtd_run: the H update of a step and, in the same launch, its Poynting vector
// and the E update of the next step.
//
// Per-update kernels move every field once per update: E and H are read twice per step, and the
// six Poynting products go through memory (update_h.cl:142-155, update_s.cl:21-36). Here H is read
// from one buffer and written to another (ping-pong, with the H-side CPML arrays), so every value
// this launch reads is read-only, and a cell that a neighbour's result needs can be evaluated again:
//   * S at (x, y, z) takes the products of its own cell and of x-1, y-1 and z-1; the next E update
//     takes H_new at exactly the same four cells. One halo feeds both: the plane before the chunk,
//     a row and a column before the tile.
//   * with the next step's E in the launch (AHEAD; E ping-pongs too), a step reads E, H and dt/eps
//     once and writes E, H and S once: 72 B per cell in float32, 32 B per absorbing cell of a face,
//     against 96 B for update_E and H+S in two launches. Without it (the last step of a call, and
//     steps whose E needs a learned boundary's fix-up first) the launch leaves E alone.
//
// What bounds it: a step of the 395x345x73 grid with six 8-cell faces takes 0.189 ms (update_E and
// H+S in two launches: 0.231), 813 MB at 4.3 TB/s; without faces 0.150 ms. Plain copies of the same
// nine read and nine written streams take 0.115-0.139 ms there, so what is left is instruction issue:
// about 290 instructions per warp and plane, 60 of them arithmetic, and the absorbing columns' code
// on top (0.204 ms before the tile's face columns were given threads of their own). 200^3 cells:
// 0.153 ms (0.244 in two or three launches); 300^3: 0.444 (0.736).
//
// Measured and left out (0.150 / 0.204 ms without and with faces at the time): strips of rows per
// thread with shuffles and no barrier (0.151 / 0.211: 4 warps per scheduler, every instruction of the
// face code exposed), a separate copy of the march for warps without faces (spills: 0.175 / 0.370),
// code per face side (spills: 0.172 / 0.258), staging by per-thread asynchronous copies (0.215).
//
// Per-cell arithmetic and its order are those of update_H, update_S and update_E (compiled with
// --fmad=false), so fields and S are bit-identical to the per-call loop.
#include "yee_common.cuh"
#include "yee_device.cuh"
#include "hs_fused.h"

namespace fdtd {

// Everything one H evaluation at (x, y, z) reads besides E at the cell.
template <typename R>
struct HLoads {
    R ex1, ey1, ez1;              // E at x+1 (wrapped): the next plane's own
    R rxy, rzy;                   // E_x, E_z at y+1 (wrapped)
    R rxz, ryz;                   // E_x, E_y at z+1 (wrapped)
    R hx, hy, hz;                 // old H at the cell
    R cx, cy, cz;                 // dt/mu at the cell
    R xu, xv, yu, yv, zu, zv;     // old psi_H of the faces the cell is in
};

// psi index of a cell at plane x in the face of axis AX it is in
template <int AX>
__device__ __forceinline__ uint32_t psi_at(const FaceAt &f, uint32_t Tn, uint32_t Tp, uint32_t x, uint32_t y, uint32_t z,
                                           uint32_t sy, uint32_t sz)
{
    return psi_index<AX>((uint32_t)f.ir, f.side ? Tp : Tn, x, y, z, sy, sz);
}

// A block marches a chunk of x planes with a tile of the (y, z) plane, one cell per thread: a row
// and a column of halo cells (owned by other tiles, evaluated from the same read-only inputs,
// never written) before its own rows and columns. After each plane's H update the values that
// neighbours need (products, H_new) go to shared memory in slots that alternate by plane, so one
// barrier per plane suffices; x - 1 values stay in registers. The next plane's loads are issued
// before the barrier. The columns inside the z faces take the block's last threads, so that few warps
// hold absorbing cells; the others skip the CPML code.
template <typename R, int DX, bool MU, bool AHEAD>
__global__ void __launch_bounds__(hs_threads(AHEAD, MU, DX), 2) k_tile_h(const __grid_constant__ HSK<R> k)
{
    // values exchanged: products xy, zy (to y + 1), xz, yz (to z + 1); H_new x, y, z
    constexpr int XY = 0, ZY = 1, XZ = 2, YZ = 3, HX = 4, HY = 5, HZ = 6, NV = AHEAD ? 7 : 4;
    constexpr uint32_t HS_THREADS = (uint32_t)hs_threads(AHEAD, MU, DX);
    __shared__ R sV[2][NV][HS_THREADS];
    __shared__ R sC[AHEAD ? 6 : 3][HS_THREADS];   // z-face coefficients of each thread: H, then E
    const uint32_t t = threadIdx.x;
    const uint32_t chunk0 = blockIdx.x / k.ntile;
    if (chunk0 >= k.nchunk) {
        // the step's DFT sample: E is not written by this launch
        grid_dependency_sync();
        const int nq = k.dft.npoint * (k.dft.nfreq > 0 ? k.dft.nfreq : 1);
        for (int q = (int)t; q < nq; q += (int)HS_THREADS) dft_sample(k.dft, q);
        return;
    }
    const uint32_t sx = k.sx, sy = k.sy, sz = k.sz, syz = k.syz;
    const uint64_t N = k.N;
    const uint32_t tile = blockIdx.x - chunk0 * k.ntile;
    const uint32_t yt = tile / k.nseg, seg = tile - yt * k.nseg;
    const uint32_t y0 = yt * k.rows, z0 = seg * k.seglen;
    const uint32_t nrow = min(k.rows, sy - y0), len = min(k.seglen, sz - z0), ext = k.seglen + 1u;
    // columns 0 (the halo, z0 - 1) .. len of the tile: a leading and a trailing run lies in the z
    // faces, [ca, cb) between them does not
    const uint32_t Tn = (uint32_t)k.ax[2].Tn, Tp = (uint32_t)k.ax[2].Tp;
    uint32_t ca = 0u, cb = len + 1u;
    if (Tn + Tp) {
        const uint32_t halo = z0 ? z0 - 1u : sz - 1u, past = z0 + len;
        if (z0 < Tn) ca = min(Tn - z0, len) + 1u;
        else if (z0 >= sz - Tp && halo >= sz - Tp) ca = len + 1u;
        else if (halo < Tn || halo >= sz - Tp) ca = 1u;
        if (past > sz - Tp && ca <= len) cb = len + 1u - min(past - (sz - Tp), len + 1u - ca);
    }
    const uint32_t nin = cb - ca, nface = len + 1u - nin, ins = nin * (nrow + 1u);
    uint32_t w, c;
    if (t < ins) {
        w = t / nin;
        c = ca + t - w * nin;
    } else {
        const uint32_t u = t - ins;
        w = nface ? u / nface : nrow + 1u;
        c = u - w * nface;
        c = c < ca ? c : c + nin;
    }
    const bool act = w <= nrow && c <= len;
    const bool own = act && w > 0u && c > 0u;
    // The thread's place in the exchange. Threads beyond the tile share the last place, which no cell
    // has when there are such threads and nobody reads (stores under a condition made the compiler spill).
    const uint32_t p = act ? w * ext + c : HS_THREADS - 1u;
    const uint32_t y = act ? (w ? y0 + w - 1u : (y0 ? y0 - 1u : sy - 1u)) : y0;
    const uint32_t z = act ? (c ? z0 + c - 1u : (z0 ? z0 - 1u : sz - 1u)) : z0;
    const uint32_t j = y * sz + z;
    const uint32_t chunk = k.reverse ? k.nchunk - 1u - chunk0 : chunk0;
    const uint32_t xa = chunk * k.xchunk;
    const uint32_t xb = min(xa + k.xchunk, sx);
    // plus neighbours (common.cl:82-84) in 32-bit wrap arithmetic
    const uint32_t dpy = (y + 1u < sy) ? sz : 0u - (sy - 1u) * sz;
    const uint32_t dpz = (z + 1u < sz) ? 1u : 0u - (sz - 1u);
    FaceAt fy = face_at(k.ax[1].Tn, k.ax[1].Tp, sy, y), fz = face_at(k.ax[2].Tn, k.ax[2].Tp, sz, z);
    if (!act) fy.ir = fz.ir = -1;
    const bool wf = __any_sync(0xffffffffu, fy.ir >= 0 || fz.ir >= 0) != 0;
    if (fz.ir >= 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            sC[q][t] = face_tab(k.ax[2].h, fz, q);
            if (AHEAD) sC[3 + q][t] = face_tab(k.ax[2].e, fz, q);
        }
    }
    bool srcs = false;                                           // a point source of the next step in the tile
    if (AHEAD) {
        for (int s = 0; s < k.nsrc; ++s) srcs |= own && k.src_j[s] == j;
        srcs = __any_sync(0xffffffffu, srcs) != 0;
    }
    grid_dependency_sync();
    R iy = k.inv_d, iz = k.inv_d, iyh = k.inv_d, izh = k.inv_d;
    if (DX == 2) {
        iy = ldf(k.inv_de[1] + y);
        iz = ldf(k.inv_de[2] + z);
        if (AHEAD) { iyh = ldf(k.inv_dh[1] + y); izh = ldf(k.inv_dh[2] + z); }
    }
    const R *const E0 = k.E, *const E1 = k.E + N, *const E2 = k.E + 2 * N;
    const R *const H0 = k.HA, *const H1 = k.HA + N, *const H2 = k.HA + 2 * N;

    const bool xf = xa < (uint32_t)k.ax[0].Tn + 1u || (k.ax[0].Tp && (xa == 0u || xb > sx - (uint32_t)k.ax[0].Tp));
    auto load = [&](uint32_t x, uint32_t i, uint32_t i1, HLoads<R> &v) {
        const uint32_t ipy = i + dpy, ipz = i + dpz;             // 32-bit wrap arithmetic
        v.ex1 = ldf(E0 + i1); v.ey1 = ldf(E1 + i1); v.ez1 = ldf(E2 + i1);
        v.rxy = ldf(E0 + ipy); v.rzy = ldf(E2 + ipy);
        v.rxz = ldf(E0 + ipz); v.ryz = ldf(E1 + ipz);
        v.hx = ldf(H0 + i); v.hy = ldf(H1 + i); v.hz = ldf(H2 + i);
        if (MU) { v.cx = ldf(k.cm + i); v.cy = ldf(k.cm + N + i); v.cz = ldf(k.cm + 2 * N + i); }
        if (wf && fz.ir >= 0) {
            const uint32_t ip = psi_at<2>(fz, k.ax[2].Tn, k.ax[2].Tp, x, y, z, sy, sz);
            v.zu = ldf(face_A(k.ax[2].h, fz, 0) + ip); v.zv = ldf(face_A(k.ax[2].h, fz, 1) + ip);
        }
        if (wf && fy.ir >= 0) {
            const uint32_t ip = psi_at<1>(fy, k.ax[1].Tn, k.ax[1].Tp, x, y, z, sy, sz);
            v.yu = ldf(face_A(k.ax[1].h, fy, 0) + ip); v.yv = ldf(face_A(k.ax[1].h, fy, 1) + ip);
        }
        FaceAt fx;
        fx.ir = -1;
        fx.side = 0;
        if (xf) fx = face_at(k.ax[0].Tn, k.ax[0].Tp, sx, x);
        if (fx.ir >= 0) {
            const uint32_t ip = (uint32_t)fx.ir * syz + j;
            v.xu = ldf(face_A(k.ax[0].h, fx, 0) + ip); v.xv = ldf(face_A(k.ax[0].h, fx, 1) + ip);
        }
    };

    // The march evaluates plane xa - 1 first, without writing: its products and H_new are the x - 1
    // neighbours of the chunk's first plane.
    uint32_t x = xa ? xa - 1u : sx - 1u;
    uint32_t i = x * syz + j;
    R ex = ldf(E0 + i), ey = ldf(E1 + i), ez = ldf(E2 + i);
    R p_yx = R(0), p_zx = R(0), p_hy = R(0), p_hz = R(0);
    HLoads<R> v;
    uint32_t i1 = xa * syz + j;
    load(x, i, i1, v);
    const uint32_t nv = xb - xa + 1u;
    for (uint32_t n = 0; n < nv; ++n) {
        const bool wr = own && n > 0u;
        FaceAt fx;
        fx.ir = -1;
        fx.side = 0;
        if (xf) fx = face_at(k.ax[0].Tn, k.ax[0].Tp, sx, x);
        // what the E update after the barrier reads
        R c0, c1, c2, exu, exv, eyu, eyv, ezu, ezv;
        if (AHEAD) {
            c0 = ldf(k.ce + i); c1 = ldf(k.ce + N + i); c2 = ldf(k.ce + 2 * N + i);
            if (wf && fz.ir >= 0) {
                const uint32_t ip = psi_at<2>(fz, k.ax[2].Tn, k.ax[2].Tp, x, y, z, sy, sz);
                ezu = ldf(face_A(k.ax[2].e, fz, 0) + ip); ezv = ldf(face_A(k.ax[2].e, fz, 1) + ip);
            }
            if (wf && fy.ir >= 0) {
                const uint32_t ip = psi_at<1>(fy, k.ax[1].Tn, k.ax[1].Tp, x, y, z, sy, sz);
                eyu = ldf(face_A(k.ax[1].e, fy, 0) + ip); eyv = ldf(face_A(k.ax[1].e, fy, 1) + ip);
            }
            if (fx.ir >= 0) {
                const uint32_t ip = (uint32_t)fx.ir * syz + j;
                exu = ldf(face_A(k.ax[0].e, fx, 0) + ip); exv = ldf(face_A(k.ax[0].e, fx, 1) + ip);
            }
        }
        // ---- H (update_h.cl): forward differences (36-43)
        R d_xy = v.rxy - ex;
        R d_xz = v.rxz - ex;
        R d_yx = v.ey1 - ey;
        R d_yz = v.ryz - ey;
        R d_zx = v.ez1 - ez;
        R d_zy = v.rzy - ez;
        if (DX != 0) {
            const R ix = DX == 2 ? ldf(k.inv_de[0] + x) : k.inv_d;
            d_xy = d_xy * iy; d_xz = d_xz * iz; d_yx = d_yx * ix;
            d_yz = d_yz * iz; d_zx = d_zx * ix; d_zy = d_zy * iy;
        }
        // CPML (80-116): at most one face per axis
        R px = R(0), py = R(0), pz = R(0);
        if (fx.ir >= 0) {
            R su, sv;
            face_update<R, false, 0>(face_tab(k.ax[0].h, fx, 0), face_tab(k.ax[0].h, fx, 1), face_tab(k.ax[0].h, fx, 2),
                                     v.xu, v.xv, su, sv, d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
            if (wr) {
                const uint32_t ip = (uint32_t)fx.ir * syz + j;
                face_B(k.ax[0].h, fx, 0)[ip] = su;
                face_B(k.ax[0].h, fx, 1)[ip] = sv;
            }
        }
        if (wf && fy.ir >= 0) {
            R su, sv;
            face_update<R, false, 1>(face_tab(k.ax[1].h, fy, 0), face_tab(k.ax[1].h, fy, 1), face_tab(k.ax[1].h, fy, 2),
                                     v.yu, v.yv, su, sv, d_xy, d_xz, d_yx, d_yz, d_zx, d_zy, px, py, pz);
            if (wr) {
                const uint32_t ip = psi_at<1>(fy, k.ax[1].Tn, k.ax[1].Tp, x, y, z, sy, sz);
                face_B(k.ax[1].h, fy, 0)[ip] = su;
                face_B(k.ax[1].h, fy, 1)[ip] = sv;
            }
        }
        if (wf && fz.ir >= 0) {
            R su, sv;
            face_update<R, false, 2>(sC[0][t], sC[1][t], sC[2][t], v.zu, v.zv, su, sv, d_xy, d_xz, d_yx, d_yz, d_zx, d_zy,
                                     px, py, pz);
            if (wr) {
                const uint32_t ip = psi_at<2>(fz, k.ax[2].Tn, k.ax[2].Tp, x, y, z, sy, sz);
                face_B(k.ax[2].h, fz, 0)[ip] = su;
                face_B(k.ax[2].h, fz, 1)[ip] = sv;
            }
        }
        // 129-131
        const R hx = v.hx - (MU ? v.cx : k.dt) * ((d_zy - d_yz) - px);
        const R hy = v.hy - (MU ? v.cy : k.dt) * ((d_xz - d_zx) - py);
        const R hz = v.hz - (MU ? v.cz : k.dt) * ((d_yx - d_xy) - pz);
        R(*const sv)[HS_THREADS] = sV[n & 1u];
        R s0, s1, s2, o_yx, o_zx;                                // S from the cell's own and the x - 1 products
        // products (63-70, 135-155)
        const R ahx = hx + v.hx, ahy = hy + v.hy, ahz = hz + v.hz;
        const R o_xy = (v.ey1 + ey) * ahz;
        const R o_xz = (-(v.ez1 + ez)) * ahy;
        const R o_yz = (v.rzy + ez) * ahx;
        o_yx = (-(v.rxy + ex)) * ahz;
        o_zx = (v.rxz + ex) * ahy;
        const R o_zy = (-(v.ryz + ey)) * ahx;
        sv[XY][p] = o_xy;
        sv[ZY][p] = o_zy;
        sv[XZ][p] = o_xz;
        sv[YZ][p] = o_yz;
        s0 = o_xy + o_xz;
        s1 = o_yz + o_yx;
        s2 = (o_zx + o_zy) + p_zx;
        if (!AHEAD && wr && k.write_oS) {
            k.oS[i] = o_xy;
            (k.oS + N)[i] = o_yz;
            (k.oS + 2 * N)[i] = o_zx;
            (k.oS + 3 * N)[i] = o_xz;
            (k.oS + 4 * N)[i] = o_yx;
            (k.oS + 5 * N)[i] = o_zy;
        }
        if (AHEAD) {
            sv[HX][p] = hx;
            sv[HY][p] = hy;
            sv[HZ][p] = hz;
        }
        const R ox = ex, oy = ey, oz = ez;                       // E at the cell, for its update
        ex = v.ex1;
        ey = v.ey1;
        ez = v.ez1;
        // the next plane's loads fly during the barrier and what follows it
        const uint32_t xn = n ? x + 1u : xa;
        const uint32_t in = i1;
        i1 = xn + 1u == sx ? j : in + syz;
        if (n + 1u < nv) load(xn, in, i1, v);
        __syncthreads();
        if (wr) {
            k.HB[i] = hx;
            (k.HB + N)[i] = hy;
            (k.HB + 2 * N)[i] = hz;
            if (k.S) {
                // S (update_s.cl:33-36)
                k.S[i] = ((s0 + sv[XY][p - ext]) + sv[XZ][p - 1u]) * k.sf;
                (k.S + N)[i] = ((s1 + sv[YZ][p - 1u]) + p_yx) * k.sf;
                (k.S + 2 * N)[i] = (s2 + sv[ZY][p - ext]) * k.sf;
            }
            if (AHEAD) {
                // ---- the next step's E (update_e.cl): backward differences (39-46)
                R e_xy = hx - sv[HX][p - ext];
                R e_xz = hx - sv[HX][p - 1u];
                R e_yx = hy - p_hy;
                R e_yz = hy - sv[HY][p - 1u];
                R e_zx = hz - p_hz;
                R e_zy = hz - sv[HZ][p - ext];
                if (DX != 0) {
                    const R ix = DX == 2 ? ldf(k.inv_dh[0] + x) : k.inv_d;
                    e_xy = e_xy * iyh; e_xz = e_xz * izh; e_yx = e_yx * ix;
                    e_yz = e_yz * izh; e_zx = e_zx * ix; e_zy = e_zy * iyh;
                }
                // CPML (64-100)
                R qx = R(0), qy = R(0), qz = R(0);
                if (fx.ir >= 0) {
                    R su, sw;
                    face_update<R, true, 0>(face_tab(k.ax[0].e, fx, 0), face_tab(k.ax[0].e, fx, 1), face_tab(k.ax[0].e, fx, 2),
                                            exu, exv, su, sw, e_xy, e_xz, e_yx, e_yz, e_zx, e_zy, qx, qy, qz);
                    const uint32_t ip = (uint32_t)fx.ir * syz + j;
                    face_B(k.ax[0].e, fx, 0)[ip] = su;
                    face_B(k.ax[0].e, fx, 1)[ip] = sw;
                }
                if (wf && fy.ir >= 0) {
                    R su, sw;
                    face_update<R, true, 1>(face_tab(k.ax[1].e, fy, 0), face_tab(k.ax[1].e, fy, 1), face_tab(k.ax[1].e, fy, 2),
                                            eyu, eyv, su, sw, e_xy, e_xz, e_yx, e_yz, e_zx, e_zy, qx, qy, qz);
                    const uint32_t ip = psi_at<1>(fy, k.ax[1].Tn, k.ax[1].Tp, x, y, z, sy, sz);
                    face_B(k.ax[1].e, fy, 0)[ip] = su;
                    face_B(k.ax[1].e, fy, 1)[ip] = sw;
                }
                if (wf && fz.ir >= 0) {
                    R su, sw;
                    face_update<R, true, 2>(sC[3][t], sC[4][t], sC[5][t], ezu, ezv, su, sw, e_xy, e_xz, e_yx, e_yz, e_zx,
                                            e_zy, qx, qy, qz);
                    const uint32_t ip = psi_at<2>(fz, k.ax[2].Tn, k.ax[2].Tp, x, y, z, sy, sz);
                    face_B(k.ax[2].e, fz, 0)[ip] = su;
                    face_B(k.ax[2].e, fz, 1)[ip] = sw;
                }
                // 105-107
                R nx = ox + c0 * ((e_zy - e_yz) + qx);
                R ny = oy + c1 * ((e_xz - e_zx) + qy);
                R nz = oz + c2 * ((e_yx - e_xy) + qz);
                if (srcs) {
                    // point sources in list order (fdtd.py:168-169)
                    for (int s = 0; s < k.nsrc; ++s) {
                        if (k.src_x[s] != x || k.src_j[s] != j) continue;
                        const R val = k.src_values ? k.src_values[(int64_t)k.src_t * k.src_stride + k.src_col[s]] : k.src_val[s];
                        if (k.src_c[s] == 0) nx = nx + val;
                        else if (k.src_c[s] == 1) ny = ny + val;
                        else nz = nz + val;
                    }
                }
                k.EB[i] = nx;
                (k.EB + N)[i] = ny;
                (k.EB + 2 * N)[i] = nz;
            }
        }
        p_yx = o_yx;
        p_zx = o_zx;
        if (AHEAD) {
            p_hy = hy;
            p_hz = hz;
        }
        x = xn;
        i = in;
    }
}

// Double precision is bound by its arithmetic units, for which evaluating the halo again costs more
// than the memory passes saved: only the form without the next step's E exists there. With the next
// step's E, Poynting may be off (S NULL: the products are formed and S is not written).
template <typename R, int DX, bool MU>
static void (*hs_kernel_mu(const HSForm &f))(HSK<R>)
{
    if constexpr (sizeof(R) == 4)
        if (f.ahead) return k_tile_h<R, DX, MU, true>;
    return f.poynting && !f.ahead ? k_tile_h<R, DX, MU, false> : nullptr;
}

template <typename R, int DX>
static void (*hs_kernel_dx(const HSForm &f))(HSK<R>)
{
    return f.mu ? hs_kernel_mu<R, DX, true>(f) : hs_kernel_mu<R, DX, false>(f);
}

template <typename R>
static void (*hs_kernel(const HSForm &f))(HSK<R>)
{
    return f.dxmode == 0 ? hs_kernel_dx<R, 0>(f) : f.dxmode == 1 ? hs_kernel_dx<R, 1>(f) : hs_kernel_dx<R, 2>(f);
}

template <typename R>
bool hs_form_exists(const HSForm &f)
{
    return hs_kernel<R>(f) != nullptr;
}

template <typename R>
cudaError_t launch_hs(const HSK<R> &k, const HSForm &f, bool pdl, cudaStream_t st)
{
    const dim3 g(k.ntile * k.nchunk + (k.dft_on ? 1u : 0u), 1, 1);
    return launch_dependent(hs_kernel<R>(f), g, (unsigned)hs_threads(f.ahead, f.mu, f.dxmode), st, pdl, k);
}

template bool hs_form_exists<float>(const HSForm &);
template bool hs_form_exists<double>(const HSForm &);
template cudaError_t launch_hs<float>(const HSK<float> &, const HSForm &, bool, cudaStream_t);
template cudaError_t launch_hs<double>(const HSK<double> &, const HSForm &, bool, cudaStream_t);

}  // namespace fdtd
