// Elastic stress divergence of one RK stage for unrotated cubic materials
// (FP64 and FP32), the path every deck without frame rotation, surface
// traction or ny < nz takes; k_elastic_tile (gf_elastic.cuh) is the general
// form.
//
// With the cubic stiffness pattern the stress a cell contributes to one of
// its faces is affine in the face's own gradient g (g_a = d u_a / d x_D):
//     sigma_a = c_a g_a + K_a(D),   c_D = c11, c_a = c44 otherwise,
// where K_a(D) collects everything that is the cell's alone: with
// T[d][a] = g_a(-d face) + g_a(+d face) and the eigenstrain e0
//     K_D(D) = c12 (T[b][b] + T[c][c]) / 2 - (c11 e0_D + c12 (e0_b + e0_c)),
//     K_a(D) = c44 T[a][D] / 2 - 2 c44 e0_aD
// (get_dv_RK*, elastic_dynamic_solver.cpp:876-1289, whose face stress is the
// mean of the two cells' rows C (strain - e0)).  So a cell forms nine K once,
// its six neighbours take three each, and a face stress component costs one
// fused multiply-add and an addition: ~130 FP operations per cell, where the
// row-by-row evaluation of both sides of every face took several hundred and
// was bound by instruction issue at 10 % of DRAM bandwidth.
//
// A block owns a tile of (j, k) columns plus a ring of halo columns, one
// thread per column, and marches along x.  u of the plane and the K of the
// y- and z-faces pass between columns through shared memory: u in a ring of
// three planes filled by cp.async two planes ahead, K in two slots that
// alternate by plane, so a plane needs one barrier; everything along x stays
// in the column's registers, with the next plane's p or m already being
// loaded.  The stencil is one cell wide (the 19-point
// neighbourhood), so the halo is one column and the only x-halo work is the
// K of the planes next to the chunk.  A free face (open end or vacuum on
// either side) reads the column itself in the neighbour's place, so its
// gradient is 0, and its stress is selected to 0.
//
// Every multiply-add is written as fma() and every other product as a
// rounded multiply, so a cell's result does not depend on the instantiation
// or tile shape (the batched phase kernels run the same body).
#pragma once

#include <algorithm>

#include "gf_elastic.cuh"

namespace gf {

// elastic and eigenstrain constants of one material
template <class R>
struct ColMat {
    R c11, c12, c44;
    R l100_15, l111_15, Q11, Q12, Q44;
    R l100a1_075, l100a2_075, l111a1_075, l111a2_075;
    R F11, F12, F44h;
    uint32_t flags;
    int pad_;
};
template <class R>
__host__ __device__ inline ColMat<R> col_mat(const DevMatT<R>& d) {
    ColMat<R> m;
    m.c11 = d.cij[0][0]; m.c12 = d.cij[0][1]; m.c44 = d.cij[3][3];
    m.l100_15 = d.l100_15; m.l111_15 = d.l111_15; m.Q11 = d.Q11; m.Q12 = d.Q12; m.Q44 = d.Q44;
    m.l100a1_075 = d.l100a1_075; m.l100a2_075 = d.l100a2_075; m.l111a1_075 = d.l111a1_075; m.l111a2_075 = d.l111a2_075;
    m.F11 = d.F11; m.F12 = d.F12; m.F44h = d.F44h;
    m.flags = d.flags; m.pad_ = 0;
    return m;
}

// Tile of one block: W x H columns (k fastest) of which the inner ones (all
// but hk columns at each end and one row at each end) are its own; hk = 0
// when one tile spans an open z axis, whose ends are free faces.
struct ColGeom {
    int W, H, hk;
    int own_k, own_j;      // W - 2 hk, H - 2
    int tk, tj;            // tiles along k and j
    int chunk;             // x-planes per block
    int threads;           // W H rounded up to whole warps
};
// Threads of the per-engine kernel, and the blocks per SM its registers
// allow: the column's state must not spill (us per launch on the 128^3
// ferroelectric grid / the 128x128x96 film of several materials, before the
// tile shape was chosen by col_geom and the material by template: FP64 384 x 1
// block, 168 registers, 72 / 80; 512 x 1, 128 registers, 86 / 127; 256 x 2,
// 104 / 132; 256 x 3, 145 / 191.  FP32 384 x 2, 80 registers, 56 / 67; 256 x 3
// 56 / 68; 512 x 2, 64 registers, 65 / 94; 256 x 4 65 / 89.  Now 61 / 66 in FP64
// and 43 / 50 in FP32; the general tile took 255 / 183 and 159 / 99).
#ifndef GF_ECOL_T_F32
#define GF_ECOL_T_F32 384
#endif
#ifndef GF_ECOL_T_F64
#define GF_ECOL_T_F64 384
#endif
#ifndef GF_ECOL_MINB_F32
#define GF_ECOL_MINB_F32 2
#endif
#ifndef GF_ECOL_MINB_F64
#define GF_ECOL_MINB_F64 1
#endif
template <class R> constexpr int kColMaxThreads = is_mixed<R>::value ? GF_ECOL_T_F32 : GF_ECOL_T_F64;
template <class R> constexpr int kColMinBlocks = is_mixed<R>::value ? GF_ECOL_MINB_F32 : GF_ECOL_MINB_F64;
constexpr int kColBatchThreads = 256;    // of a batched work item

// which fields the dynamic eigenstrain reads: p only, m only, or whatever
// the run has (also antiferromagnets, flexoelectricity, static eigenstrain,
// none), read without prefetch
enum ColEig : int { CE_P = 1, CE_M = 2, CE_ANY = 3 };

// shared memory of a block whose arrays have `pitch` words per plane (a
// compile-time constant: neighbours and components are then fixed offsets)
template <class R>
inline size_t col_smem_bytes(int pitch, int nmat) {
    return ((size_t)pitch * (21 * sizeof(R) + 2) + 15) / 16 * 16 + (size_t)nmat * sizeof(ColMat<R>);
}

// March of column tile (bx, by) over x-chunk bz for the vector field op.u:
// f = sum_d (s(+d face) - s(-d face)) / (2 h_d), s_a = (c_a + c_a') g_a + K_a + K_a'
// with K_D(D) = c12 (T[b][b] + T[c][c]) / 2 - EN_D, K_a(D) = c44 T[a][D] / 2 - ES_aD
// (EN, ES: a cell's own terms, in the stress divergence its eigenstress).
// Op:
//   u[3]               the field
//   fetch(c) / next()  start loading the cell data of c / make it current
//   early(c, cl)       start loading what cell(c) and done(cl) will need
//   own_terms(c, solid, cm, EN, ES)   from the current cell data; ES = yz, xz, xy
//   cell(c, solid, cm, Tx, Ty, Tz)    an own cell, with its gradient sums
//   done(c, solid, f)                 an own cell, with its f (0 in vacuum)
template <class R, bool UNI, int NT, class Op>
__device__ __forceinline__ void col_march(const Params& P, const ColGeom& G, const uint8_t* __restrict__ mid,
                                          const DevMatT<R>* __restrict__ mats, int nmat, const ColMat<R>& um, Op& op, int bx, int by,
                                          int bz, unsigned char* smem_raw) {
    R* su = reinterpret_cast<R*>(smem_raw);            // [3][3][NT]
    R* sk = su + 9 * NT;                               // [2][6][NT]: y-face K, z-face K
    uint8_t* sid = reinterpret_cast<uint8_t*>(sk + 12 * NT);   // [2][NT]
    ColMat<R>* smat = reinterpret_cast<ColMat<R>*>(smem_raw + ((size_t)NT * (21 * sizeof(R) + 2) + 15) / 16 * 16);

    const int W = G.W, live_n = G.W * G.H;
    // threads past the tile repeat its last column (same values, no output)
    const int t = min((int)threadIdx.x, live_n - 1);
    const int row = t / W, col = t - row * W;
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    int j = by * G.own_j + row - 1, k = bx * G.own_k + col - G.hk;
    const bool own = (int)threadIdx.x < live_n && row >= 1 && row < G.H - 1 && j < ny && col >= G.hk && col < W - G.hk && k < nz;
    j = j < 0 ? j + ny : j % ny;
    k = k < 0 ? k + nz : k % nz;
    const int nyz = ny * nz, cjk = j * nz + k;
    const int i0 = bz * G.chunk, L = min(i0 + G.chunk, nx) - i0;

    if constexpr (!UNI) {
        for (int q = threadIdx.x; q < nmat; q += blockDim.x) smat[q] = col_mat(mats[q]);
    }
    // neighbour columns in the tile; at its edge the column itself (those
    // values are not used: an edge column only provides the K of the face
    // towards the tile)
    const bool fym = (j == 0 && !P.per_y) || row == 0, fyp = (j == ny - 1 && !P.per_y) || row == G.H - 1;
    const bool fzm = (k == 0 && !P.per_z) || col == 0, fzp = (k == nz - 1 && !P.per_z) || col == W - 1;
    R rdx, rdy, rdz;
    if constexpr (is_mixed<R>::value) { rdx = P.f.rdx; rdy = P.f.rdy; rdz = P.f.rdz; }
    else { rdx = P.rdx; rdy = P.rdy; rdz = P.rdz; }
    const R hx = R(0.5) * rdx, hyx = rdy / rdx, hzx = rdz / rdx;
    const R* const u0 = op.u.c[0];
    const R* const u1 = op.u.c[1];
    const R* const u2 = op.u.c[2];
    const auto c_of = [&](int p) { return wrapm(p, nx) * nyz + cjk; };

    // planes i0-1 and i0
    R uc[3];
    uint8_t id = 1, idn = 1;
    auto stage = [&](int slot, int pl) {
        const int cf = c_of(pl);
        R* d = su + 3 * slot * NT + t;
        cp_async_elem(d, u0 + cf); cp_async_elem(d + NT, u1 + cf); cp_async_elem(d + 2 * NT, u2 + cf);
        cp_async_commit();
    };
    {
        const int c0 = c_of(i0 - 1), c1 = c_of(i0);
        stage(1, i0);
        uc[0] = u0[c0]; uc[1] = u1[c0]; uc[2] = u2[c0];
        op.fetch(c0);
        if constexpr (!UNI) { id = mid[c0]; idn = mid[c1]; sid[t] = id; }
#pragma unroll
        for (int a = 0; a < 3; a++) su[a * NT + t] = uc[a];
        op.next();
    }
    __syncthreads();

    ColMat<R> cm;                    // constants of the column's current material
    int cm_id = -1;
    if constexpr (UNI) cm = um;
    // carried along x: gradient of x-face p, K of the cell below it, and what
    // the cell below it still lacks its upper x-face's stress for, as a stress:
    // the two x-faces' difference is formed before its product with hx, so that a
    // stress uniform along x has exactly no divergence (carried as a force,
    // w = rest - sx hx and f = sx hx + w contracted, it left the rounding error of
    // one product; the lower face's stress carried beside w took three more
    // registers, 128x128x96 film FP32 0.659 -> 0.686 ms per step)
    R gxm[3] = {R(0.), R(0.), R(0.)}, kxp[3] = {R(0.), R(0.), R(0.)}, w[3] = {R(0.), R(0.), R(0.)};
    int s3 = 0;                      // ring slot of plane p
    R c11p = R(0.), c44p = R(0.);    // constants of the cell below the x-face
    bool solid_p = UNI;
    if constexpr (UNI) { c11p = um.c11; c44p = um.c44; }

    for (int q = 0; q <= L + 1; q++) {
        const int p = i0 - 1 + q;
        const int s = q & 1;
        const int c = c_of(p);
        // next loads: u two planes ahead (into the slot of plane p-1, whose
        // readers are behind the last barrier), the cell data one plane ahead
        uint8_t idf = 1;
        const int s3n = s3 == 2 ? 0 : s3 + 1;
        if (q < L) {
            stage(s3n == 2 ? 0 : s3n + 1, p + 2);
            if constexpr (!UNI) idf = mid[c_of(p + 2)];
        } else {
            cp_async_commit();
        }
        if (q <= L) op.fetch(c_of(p + 1));
        if (own) op.early(q >= 1 && q <= L ? c : -1, q >= 2 ? (p - 1) * nyz + cjk : -1);
        const bool solid = UNI || id != 0;
        bool ym = !fym, yp = !fyp, zm = !fzm, zp = !fzp;      // face carries stress
        uint8_t iym = 1, iyp = 1, izm = 1, izp = 1;
        if constexpr (!UNI) {
            const uint8_t* ids = sid + s * NT;
            iym = ids[ym ? t - W : t]; iyp = ids[yp ? t + W : t]; izm = ids[zm ? t - 1 : t]; izp = ids[zp ? t + 1 : t];
            ym = ym && solid && iym != 0; yp = yp && solid && iyp != 0;
            zm = zm && solid && izm != 0; zp = zp && solid && izp != 0;
            if (id != cm_id) {
                cm_id = id;
                if (id != 0) cm = smat[id - 1];
                else cm = ColMat<R>{};
            }
        }
        const int oym = ym ? t - W : t, oyp = yp ? t + W : t, ozm = zm ? t - 1 : t, ozp = zp ? t + 1 : t;
        const R* us = su + 3 * s3 * NT;
        // the column's own u of plane p+1 has landed (all but the newest group)
        cp_async_wait_one();
        R gym[3], gyp[3], gzm[3], gzp[3], gxp[3], Tx[3], Ty[3], Tz[3];
        const bool xp = !(p == nx - 1 && !P.per_x) && !(p == -1 && !P.per_x) && (UNI || (solid && idn != 0));
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const R v = uc[a];
            uc[a] = su[(3 * s3n + a) * NT + t];
            gym[a] = mul_rn(v - us[a * NT + oym], rdy); gyp[a] = mul_rn(us[a * NT + oyp] - v, rdy);
            gzm[a] = mul_rn(v - us[a * NT + ozm], rdz); gzp[a] = mul_rn(us[a * NT + ozp] - v, rdz);
            gxp[a] = xp ? mul_rn(uc[a] - v, rdx) : R(0.);
            Tx[a] = gxm[a] + gxp[a]; Ty[a] = gym[a] + gyp[a]; Tz[a] = gzm[a] + gzp[a];
        }
        // the nine K of the cell
        const R c11 = cm.c11, c44 = cm.c44, c12h = R(0.5) * cm.c12, c44h = R(0.5) * cm.c44;
        R EN[3], ES[3], kx[3], ky[3], kz[3];
        op.own_terms(c, solid, cm, EN, ES);
        kx[0] = fma_rn(c12h, Ty[1] + Tz[2], -EN[0]);
        kx[1] = fma_rn(c44h, Ty[0], -ES[2]);
        kx[2] = fma_rn(c44h, Tz[0], -ES[1]);
        ky[0] = fma_rn(c44h, Tx[1], -ES[2]);
        ky[1] = fma_rn(c12h, Tx[0] + Tz[2], -EN[1]);
        ky[2] = fma_rn(c44h, Tz[1], -ES[0]);
        kz[0] = fma_rn(c44h, Tx[2], -ES[1]);
        kz[1] = fma_rn(c44h, Ty[2], -ES[0]);
        kz[2] = fma_rn(c12h, Tx[0] + Ty[1], -EN[2]);
        R* ks = sk + 6 * s * NT;
#pragma unroll
        for (int a = 0; a < 3; a++) { ks[a * NT + t] = ky[a]; ks[(3 + a) * NT + t] = kz[a]; }
        // the next plane's ids
        if constexpr (!UNI) sid[(s ^ 1) * NT + t] = idn;
        R sx[3] = {R(0.), R(0.), R(0.)};
        // x-face p: stress, and the cell below it is complete
        if (q >= 1) {
            const bool xm = !((p == 0 || p == nx) && !P.per_x) && (UNI || (solid && solid_p));
            const R s11 = c11p + c11, s44 = c44p + c44;
#pragma unroll
            for (int a = 0; a < 3; a++) sx[a] = xm ? fma_rn(a == 0 ? s11 : s44, gxm[a], kxp[a] + kx[a]) : R(0.);
            if (q >= 2 && own) {
                R f[3];
#pragma unroll
                for (int a = 0; a < 3; a++) f[a] = mul_rn(sx[a] + w[a], hx);
                op.done((p - 1) * nyz + cjk, solid_p, f);
            }
        }
        __syncthreads();
        // y- and z-faces of an own cell
        if (q >= 1 && q <= L && own) {
            R sm[3], sp[3];
            R y11m = c11 + c11, y44m = c44 + c44, y11p = y11m, y44p = y44m, z11m = y11m, z44m = y44m, z11p = y11m, z44p = y44m;
            if constexpr (!UNI) {
                if (ym && iym != id) { y11m = smat[iym - 1].c11 + c11; y44m = smat[iym - 1].c44 + c44; }
                if (yp && iyp != id) { y11p = smat[iyp - 1].c11 + c11; y44p = smat[iyp - 1].c44 + c44; }
                if (zm && izm != id) { z11m = smat[izm - 1].c11 + c11; z44m = smat[izm - 1].c44 + c44; }
                if (zp && izp != id) { z11p = smat[izp - 1].c11 + c11; z44p = smat[izp - 1].c44 + c44; }
            }
            R dy[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                sm[a] = ym ? fma_rn(a == 1 ? y11m : y44m, gym[a], ks[a * NT + oym] + ky[a]) : R(0.);
                sp[a] = yp ? fma_rn(a == 1 ? y11p : y44p, gyp[a], ky[a] + ks[a * NT + oyp]) : R(0.);
                dy[a] = sp[a] - sm[a];
            }
#pragma unroll
            for (int a = 0; a < 3; a++) {
                sm[a] = zm ? fma_rn(a == 2 ? z11m : z44m, gzm[a], ks[(3 + a) * NT + ozm] + kz[a]) : R(0.);
                sp[a] = zp ? fma_rn(a == 2 ? z11p : z44p, gzp[a], kz[a] + ks[(3 + a) * NT + ozp]) : R(0.);
                w[a] = fma_rn(dy[a], hyx, mul_rn(sp[a] - sm[a], hzx)) - sx[a];
            }
            op.cell(c, solid, cm, Tx, Ty, Tz);
        }
        op.next();
#pragma unroll
        for (int a = 0; a < 3; a++) { gxm[a] = gxp[a]; kxp[a] = kx[a]; }
        s3 = s3n;
        if constexpr (!UNI) { c11p = c11; c44p = c44; solid_p = solid; id = idn; idn = idf; }
    }
}

// The stage's stress divergence: u in, the force of every material cell and
// the crystal-frame strain of the cells whose LLG kernel reads it out.
template <class R, int PM>
struct ColForce {
    const Params& P;
    const StageIOT<R>& io;
    F3T<R> u;
    R cur[3], nxt[3];
    bool back, want;
    __device__ __forceinline__ ColForce(const Params& p, const StageIOT<R>& s) : P(p), io(s), u(s.u_in) {
        back = p.elasto_back;
        want = s.strain_c[0] != nullptr;
#pragma unroll
        for (int a = 0; a < 3; a++) cur[a] = nxt[a] = R(0.);
    }
    __device__ __forceinline__ void fetch(int c) {
        if constexpr (PM == CE_P) { nxt[0] = io.p_in.c[0][c]; nxt[1] = io.p_in.c[1][c]; nxt[2] = io.p_in.c[2][c]; }
        else if constexpr (PM == CE_M) { nxt[0] = io.m_in.c[0][c]; nxt[1] = io.m_in.c[1][c]; nxt[2] = io.m_in.c[2][c]; }
    }
    __device__ __forceinline__ void next() { cur[0] = nxt[0]; cur[1] = nxt[1]; cur[2] = nxt[2]; }
    __device__ __forceinline__ void early(int, int) const {}
    // eigenstress: EN_D = c11 e_D + c12 (e_b + e_c), ES_ab = 2 c44 e_ab of the
    // dynamic eigenstrain e (get_eigenstrain_dynamic)
    __device__ __forceinline__ void own_terms(int c, bool solid, const ColMat<R>& cm, R EN[3], R ES[3]) const {
        R e[6] = {R(0.), R(0.), R(0.), R(0.), R(0.), R(0.)};
        const R x = cur[0], y = cur[1], z = cur[2];
        if constexpr (PM == CE_P) {
            const R x2 = mul_rn(x, x), y2 = mul_rn(y, y), z2 = mul_rn(z, z);
            e[0] = fma_rn(cm.Q12, y2 + z2, mul_rn(cm.Q11, x2));
            e[1] = fma_rn(cm.Q12, x2 + z2, mul_rn(cm.Q11, y2));
            e[2] = fma_rn(cm.Q12, x2 + y2, mul_rn(cm.Q11, z2));
            e[3] = mul_rn(mul_rn(cm.Q44, y), z); e[4] = mul_rn(mul_rn(cm.Q44, x), z); e[5] = mul_rn(mul_rn(cm.Q44, y), x);
        } else if constexpr (PM == CE_M) {
            const R third = R(1.) / R(3.);
            e[0] = mul_rn(cm.l100_15, fma_rn(x, x, -third));
            e[1] = mul_rn(cm.l100_15, fma_rn(y, y, -third));
            e[2] = mul_rn(cm.l100_15, fma_rn(z, z, -third));
            e[3] = mul_rn(mul_rn(cm.l111_15, y), z); e[4] = mul_rn(mul_rn(cm.l111_15, x), z); e[5] = mul_rn(mul_rn(cm.l111_15, y), x);
        } else {
            if (back && solid) eigen_glb_m(P, io, (long)c, cm, e);
        }
        EN[0] = fma_rn(cm.c12, e[1] + e[2], mul_rn(cm.c11, e[0]));
        EN[1] = fma_rn(cm.c12, e[0] + e[2], mul_rn(cm.c11, e[1]));
        EN[2] = fma_rn(cm.c12, e[0] + e[1], mul_rn(cm.c11, e[2]));
        const R c442 = R(2.) * cm.c44;
        ES[0] = mul_rn(c442, e[3]); ES[1] = mul_rn(c442, e[4]); ES[2] = mul_rn(c442, e[5]);
    }
    __device__ __forceinline__ void cell(int c, bool solid, const ColMat<R>& cm, const R Tx[3], const R Ty[3], const R Tz[3]) const {
        if (!(want && solid && (cm.flags & (MF_FM | MF_AFM)))) return;
        io.strain_c[0][c] = R(0.5) * Tx[0];
        io.strain_c[1][c] = R(0.5) * Ty[1];
        io.strain_c[2][c] = R(0.5) * Tz[2];
        io.strain_c[3][c] = R(0.25) * (Tz[1] + Ty[2]);
        io.strain_c[4][c] = R(0.25) * (Tz[0] + Tx[2]);
        io.strain_c[5][c] = R(0.25) * (Ty[0] + Tx[1]);
    }
    __device__ __forceinline__ void done(int c, bool solid, const R f[3]) const {
        if (!solid) return;
#pragma unroll
        for (int a = 0; a < 3; a++) io.force.c[a][c] = f[a];
    }
};

template <class R, bool UNI, int PM, int NT>
__device__ __forceinline__ void elastic_col_body(const Params& P, const StageIOT<R>& io, const ColGeom& G, int nmat,
                                                 const ColMat<R>& um, int bx, int by, int bz, unsigned char* smem_raw) {
    ColForce<R, PM> op(P, io);
    col_march<R, UNI, NT>(P, G, io.mid, io.mats, nmat, um, op, bx, by, bz, smem_raw);
}

template <class R, bool UNI, int PM>
__global__ void __launch_bounds__(kColMaxThreads<R>, kColMinBlocks<R>)
    k_elastic_col(const __grid_constant__ Params P, const __grid_constant__ StageIOT<R> io, const __grid_constant__ ColGeom G, int nmat,
                  const __grid_constant__ ColMat<R> um) {
    GF_EXTERN_SMEM(unsigned char, smem_raw);
    elastic_col_body<R, UNI, PM, kColMaxThreads<R>>(P, io, G, nmat, um, blockIdx.x, blockIdx.y, blockIdx.z, smem_raw);
}

// Tile shape and x-chunk for a grid: the shape with at most max_threads
// columns, and the chunk, with the least estimated time.  A chunk of L planes
// marches L + 2; an SM with b resident blocks of T threads takes, per plane,
// the latency of one plane (barriers, loads: ~2600 cycles) or the issue time
// of b T columns (3.3 cycles each in FP32, 6.6 in FP64), whichever is longer
// (both from the timed launches: 128^3 FP32 43 us, 128x128x96 FP32 with one
// resident block 78 us); short rows cost partly used 32-byte sectors.
// slots(threads) gives the resident blocks of the chip.
template <class R, class F>
inline ColGeom col_geom(const Params& P, int max_threads, long sms, F slots, int fixed_chunk = 0) {
    constexpr double kPlaneLatency = 2600., kColumnIssue = is_mixed<R>::value ? 3.3 : 6.6;
    ColGeom best{};
    double best_cost = -1.;
    const int max_k = (P.nz + 7) / 8;
    for (int tk = 1; tk <= max_k; tk++) {
        ColGeom g{};
        g.own_k = (P.nz + tk - 1) / tk;
        g.tk = (P.nz + g.own_k - 1) / g.own_k;
        if (g.tk != tk) continue;
        g.hk = (tk == 1 && !P.per_z) ? 0 : 1;
        g.W = g.own_k + 2 * g.hk;
        for (int H = 3; H * g.W <= max_threads && H <= P.ny + 2; H++) {
            g.own_j = H - 2;
            g.tj = (P.ny + g.own_j - 1) / g.own_j;
            g.H = H;
            g.threads = (g.W * H + 31) / 32 * 32;
            const long b = slots(g.threads) / sms;
            if (b < 1) continue;
            auto plane = [&](long blocks) { return blocks < 1 ? 0. : std::max(kPlaneLatency, kColumnIssue * (double)(blocks * g.threads)); };
            for (int L = 1; L <= P.nx; L++) {
                if (fixed_chunk > 0 && L != fixed_chunk) continue;
                const int nc = (P.nx + L - 1) / L;
                if (fixed_chunk <= 0 && (P.nx + nc - 1) / nc != L) continue;
                const long per_sm = ((long)g.tk * g.tj * nc + sms - 1) / sms;
                const double sectors = 1. + 0.3 * 32. / (double)(g.W * sizeof(R));
                const double cost = (L + 2) * sectors * ((double)(per_sm / b) * plane(b) + plane(per_sm % b));
                if (best_cost < 0. || cost < best_cost) { best_cost = cost; best = g; best.chunk = L; }
            }
        }
    }
    return best;
}

}  // namespace gf
