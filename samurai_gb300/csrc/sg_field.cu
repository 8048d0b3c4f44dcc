// FP64 kernels of the MR advection step on the dense level slabs:
// update_ghost_mr (outer ghosts, projection, prediction), wavelet details,
// keep/coarsen/refine criteria, tag finalisation, update_fields and the
// first-order upwind step.  Built with --fmad=false: every FP64 operation is
// rounded on its own, in the reference's association order, so that the
// detail thresholds take the same decisions as the CPU implementation.
#include <algorithm>
#include <cstring>
#include <functional>
#include <type_traits>

#include "sg_phase_dev.cuh"

namespace sg
{
    // the mesh's device error word (Geom::err), read and cleared
    int device_error(Ctx& c)
    {
        int v = 0;
        if (read_device_error(c, &v) != cudaSuccess)
        {
            return check(c, "device_error");
        }
        if (v)
        {
            c.err = "a kernel addressed a cell outside the stored level box (invalid mesh)";
            return SG_ERR_STATE;
        }
        return SG_OK;
    }

    int graduate(Ctx& c, DeviceMesh& m, DeviceMesh& nm, int* iterations);
    int ensure_details(Ctx& c, int n);

    namespace
    {
        // The transposes of one projection and one prediction, written out instead of through linear forms: the
        // weights are those the forms would carry (2^-dim for each child; +-8^-k for each tap of the order-1
        // stencil, the signs and k as in predict_one), so the adjoint is the same operator, without building a form
        // in local memory per item.  lam[e] (e the written element) is read, scattered and, in place, cleared.
        template <int DIM, int CAP>
        __device__ __forceinline__ void project_transpose(const Geom& g, const RevAcc<CAP>& u, long long e, int lf, int x, int y, int z)
        {
            const double ld = u.lam_in[e];
            if (u.in_place)
            {
                u.lam_in[e] = 0.;
            }
            if (ld == 0.)
            {
                return;
            }
            const double wch = ld * (1.0 / static_cast<double>(1 << DIM));
            const Box3 bx    = box_at<DIM>(g, lf, 2 * x, 2 * y, 2 * z, 2);
            for (int sz = 0; sz < (DIM == 3 ? 2 : 1); ++sz)
            {
                for (int sy = 0; sy < 2; ++sy)
                {
                    const long long b = bx.base + sy * bx.sy + sz * bx.sz;
                    atomicAdd(u.lam_out + b, wch);
                    atomicAdd(u.lam_out + b + 1, wch);
                }
            }
        }

        template <int DIM, int CAP>
        __device__ __forceinline__ void predict_transpose(const Geom& g, const RevAcc<CAP>& u, long long e, int l, int x, int y, int z, int order)
        {
            const double ld = u.lam_in[e];
            if (u.in_place)
            {
                u.lam_in[e] = 0.;
            }
            if (ld == 0.)
            {
                return;
            }
            const int px = x >> 1, py = y >> 1, pz = z >> 1;
            if (order == 0)
            {
                atomicAdd(u.lam_out + elem_at(g, l - 1, px, py, pz), ld);
                return;
            }
            const int qx = x & 1, qy = y & 1, qz = z & 1;
            const Box3 bx = box_at<DIM>(g, l - 1, px - 1, py - 1, pz - 1, 3);
            for (int sz = 0; sz < (DIM == 3 ? 3 : 1); ++sz)
            {
                for (int sy = 0; sy < 3; ++sy)
                {
                    const long long base = bx.base + sy * bx.sy + sz * bx.sz;
                    for (int sx = 0; sx < 3; ++sx)
                    {
                        const int k    = (sx != 1) + (sy != 1) + (DIM == 3 && sz != 1);
                        const bool neg = ((sx == 0 && qx) || (sx == 2 && !qx)) ^ ((sy == 0 && qy) || (sy == 2 && !qy))
                                         ^ (DIM == 3 && ((sz == 0 && qz) || (sz == 2 && !qz)));
                        const double w = (k == 0 ? 1.0 : (k == 1 ? 0.125 : (k == 2 ? 0.015625 : 0.001953125))) * (neg ? -1.0 : 1.0);
                        atomicAdd(u.lam_out + base + sx, w * ld);
                    }
                }
            }
        }

        // The launches of the transposed ghost update: one per level and role, so
        // that no launch reads what it writes.
        // top-down, level l: corners (parts 1), faces and the projection onto level l-1; or the corners'
        // projection below alone (parts 2)
        template <int DIM, int CAP>
        __global__ void k_ghost_reverse(const __grid_constant__ Geom gp, int l, int parts, int nb, int has_bc, MeshPtrs m, RevAcc<CAP> u)
        {
            const Geom& g = gp;
            if (static_cast<int>(blockIdx.x) < nb)
            {
                const int total = static_cast<int>((parts & 1) ? boundary_count<DIM>(g, l) : corner_slots<DIM>(g, l));
                for (int t = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x); t < total; t += nb * static_cast<int>(blockDim.x))
                {
                    boundary_item<DIM, false>(g, l, t, m, u, has_bc != 0, 0., parts);
                }
                return;
            }
            project_items<false>(g, l, m, grid_team(nb), 1,
                          [&](long long w, int b, const Cell& c, int) { project_transpose<DIM>(g, u, 32 * w + b, l, c.x, c.y, c.z); });
        }

        template <int DIM, int CAP>
        __global__ void k_predict_reverse(const __grid_constant__ Geom gp, int l, int order, MeshPtrs m, RevAcc<CAP> u)
        {
            const Geom& g = gp;
            predict_items<false>(g, l, m, grid_team(), 1,
                          [&](long long w, int b, const Cell& c, int) { predict_transpose<DIM>(g, u, 32 * w + b, l, c.x, c.y, c.z, order); });
        }

        // the transpose of update_fields (op_update_fields): every reference entry of the new field hands its adjoint
        // to what it was copied, projected or predicted from
        template <int DIM, class A>
        __global__ void k_update_fields_reverse(const __grid_constant__ Geom gp, int order, const int* wl, const long long* lo, const uint32_t* nref,
                                        const uint32_t* ncells, const uint32_t* oref, const uint32_t* ocells, const uint32_t* ohc, A uo, A un)
        {
            const Geom& g = gp;
            block_items(wl, static_cast<int>(lo[LO_REF]), static_cast<int>(lo[LO_REF + g.nlev]), grid_team(), 1, [&](int w) { return nref[w]; },
                      [&](bool valid, int w_, int b, int)
                      {
                          if (!valid)
                          {
                              return;
                          }
                          const long long w = w_;
                          const long long e = 32 * w + b;
                          typename A::V v   = A::konst(0.);
                          if ((ncells[w] >> b) & 1u)
                          {
                              const int l  = level_of(g, w);
                              const Cell c = cell_of(g, l, w, b);
                              if ((ohc[w] >> b) & 1u)
                              {
                                  v = project_one<DIM>(g, uo, l + 1, c.x, c.y, c.z);
                              }
                              else if (l >= 1 && test(ocells, g, l - 1, c.x >> 1, c.y >> 1, c.z >> 1))
                              {
                                  v = predict_one<DIM>(g, uo, l, c.x, c.y, c.z, order);
                              }
                              else if ((oref[w] >> b) & 1u)
                              {
                                  v = uo.get(e);
                              }
                          }
                          un.put(e, v);
                      });
        }

        // -------------------------------------------------------- upwind
        // 2^l as a double from its exponent bits (no FP64 instruction)
        __device__ __forceinline__ double pow2(int l)
        {
            return __longlong_as_double(static_cast<long long>(1023 + l) << 52);
        }

        // x * 2^l (l >= 0), exactly, by raising the exponent when x and the
        // product are normal numbers; zeros keep their bits; otherwise the
        // multiplication
        __device__ __forceinline__ double scale2(double x, int l)
        {
            const long long b = __double_as_longlong(x);
            const int e       = static_cast<int>((b >> 52) & 0x7FF);
            if (e > 0 && e + l < 0x7FF)
            {
                return __longlong_as_double(b + (static_cast<long long>(l) << 52));
            }
            if ((static_cast<unsigned long long>(b) << 1) == 0)
            {
                return x;
            }
            return x * pow2(l);
        }

        struct UpwindArgs
        {
            double ha[3]; // .5 * a_d, as the reference's flux forms it
            double hb[3]; // .5 * |a_d|
            double fl[3]; // the flux form's coefficients of the left and the right value: (a, 0) or (0, a)
            double fr[3];
            bool zero_l[3], zero_r[3]; // which of them are zero
            double dt;
            int scheme;
        };

        // unp1 = u - dt * upwind(a, u) (stencil_field.hpp:38-44, 91-97;
        // demos/FiniteVolume/advection_2d.cpp:144) or the README lambda
        // (README.md:144-153).  Same-level neighbours are reference cells at
        // fixed offsets in the dense slabs.  On GB300 the FP64 pipe, not HBM,
        // bounds this kernel, so FP64 work is cut without changing a rounding:
        //  - the x-face flux between two leaf cells of a word is computed once
        //    (lane b's right flux is lane b+1's left flux: same operands, same
        //    operations, same bits) and passed by a shuffle;
        //  - /dx and dt/dx use dx = 2^-l exactly: x / 2^-l == x * 2^l.
        template <int DIM>
        __global__ void k_upwind(const __grid_constant__ Geom gp, const int* __restrict__ wl, const long long* __restrict__ lo, const uint32_t* __restrict__ cells, const double* __restrict__ u,
                                 double* __restrict__ unp1, UpwindArgs p)
        {
            const Geom& g  = gp;
            const int lane = threadIdx.x & 31;
            // consecutive threads hold consecutive leaf cells (block_items); a cell's left
            // flux is its left neighbour's right flux when that neighbour is the
            // previous lane's cell (the same face, the same expression)
            block_items(wl, static_cast<int>(lo[LO_CELLS]), static_cast<int>(lo[LO_CELLS + g.nlev]), grid_team(), 1, [&](int w) { return __ldg(cells + w); },
                           [&](bool valid, int w, int b, int)
                           {
                               int l = 0;
                               long long e = 0, sy = 0, sz = 0;
                               double uc = 0., rf = 0.;
                               if (valid)
                               {
                                   l                  = level_down(g, w, 0, g.max_level);
                                   const LevelGeom& L = g.lv[l];
                                   e                  = 32LL * w + b;
                                   sy                 = 32LL * L.W;
                                   sz                 = sy * L.R;
                                   uc                 = u[e];
                               }
                               if (p.scheme == 1)
                               {
                                   if (valid)
                                   {
                                       double s = uc - u[e - 1];
                                       s        = s + uc;
                                       s        = s - u[e - sy];
                                       if (DIM == 3)
                                       {
                                           s = s + uc;
                                           s = s - u[e - sz];
                                       }
                                       unp1[e] = uc - (p.dt * pow2(l)) * s;
                                   }
                                   return;
                               }
                               if (valid)
                               {
                                   const double ur = u[e + 1];
                                   rf              = p.ha[0] * (uc + ur) + p.hb[0] * (uc - ur);
                               }
                               const double rf_left = __shfl_up_sync(FULL_MASK, rf, 1);
                               const int wl_        = __shfl_up_sync(FULL_MASK, w, 1);
                               const int bl         = __shfl_up_sync(FULL_MASK, valid ? b : -2, 1);
                               if (!valid)
                               {
                                   return;
                               }
                               double lf;
                               if (lane > 0 && wl_ == w && bl == b - 1)
                               {
                                   lf = rf_left;
                               }
                               else
                               {
                                   const double ul = u[e - 1];
                                   lf              = p.ha[0] * (ul + uc) + p.hb[0] * (ul - uc);
                               }
                               const double ud = u[e - sy], uu = u[e + sy];
                               const double df = p.ha[1] * (ud + uc) + p.hb[1] * (ud - uc);
                               const double uf = p.ha[1] * (uc + uu) + p.hb[1] * (uc - uu);
                               double s        = -lf + rf;
                               s               = s + -df;
                               s               = s + uf;
                               if (DIM == 3)
                               {
                                   const double uf2 = u[e - sz], ub2 = u[e + sz];
                                   const double ff  = p.ha[2] * (uf2 + uc) + p.hb[2] * (uf2 - uc);
                                   const double bf  = p.ha[2] * (uc + ub2) + p.hb[2] * (uc - ub2);
                                   s                = s + -ff;
                                   s                = s + bf;
                               }
                               const double up = scale2(s, l); // s / dx with dx = 2^-l
                               unp1[e]         = uc - p.dt * up;
                           });
        }


        // ---------------------------------------------- flux-form convection
        // unp1 = u - dt * conv(u) with conv = make_convection_upwind<Field>(a)
        // (schemes/fv/operators/convection_lin.hpp:16-89), explicit application
        // (explicit_flux_based_scheme__lin_hom.hpp:39-319).  The reference
        // visits interfaces (same level by level, then level jumps, then the
        // boundary, direction by direction) and adds each face's contributions
        // to both cells; one thread per leaf cell here gathers the same terms
        // in the order they reach that cell:
        //  same level   d = 0: [+lc0 u_X], [+rc0 u_X-e], [+lc1 u_X+e], [+rc1 u_X]
        //               (X left / right of a same-level face, one x-interval);
        //               d > 0: the face below (previous row) first: [+rc0 u_X-e,
        //               +rc1 u_X] then [+lc0 u_X, +lc1 u_X+e];
        //  jumps, X fine (iteration level-1): coarse on the left, then coarse on
        //               the right, neighbour values from the ghosts at X's level;
        //  jumps, X coarse (iteration level): fine on the right, then on the
        //               left, row by row; a face along x adds one term per
        //               fine row, other faces add the pair sum of the two fine
        //               cells of a row (the i.size()==1 / pair branches);
        //  boundary:    +(2^l f) terms with the outer ghost.
        // Coefficients: face length^(dim-1) / cell volume times the upwind flux
        // coefficients (a, 0) for a >= 0, (0, a) otherwise; every factor is a
        // power of two.
        // Bound by the FP64 pipe, so only the terms that can change the sum are
        // formed: one of the two flux coefficients is zero, and a term 0 * v adds
        // +-0 to a sum that starts at +0 and is never -0, which leaves its bits as
        // they are unless v is infinite or NaN (tested on the exponent).  Products
        // with 2^l move the exponent, same-level neighbours sit at fixed strides.

        // acc + c * v; zero: c is zero
        __device__ __forceinline__ double add_term(double acc, double c, bool zero, double v)
        {
            if (zero && ((__double2hiint(v) >> 20) & 0x7FF) != 0x7FF)
            {
                return acc;
            }
            return acc + c * v;
        }

        // acc + (c * v + c * w)
        __device__ __forceinline__ double add_pair(double acc, double c, bool zero, double v, double w)
        {
            if (zero && ((__double2hiint(v) >> 20) & 0x7FF) != 0x7FF && ((__double2hiint(w) >> 20) & 0x7FF) != 0x7FF)
            {
                return acc;
            }
            return acc + (c * v + c * w);
        }

        // 64 registers: the level-jump branches want 90, which leaves two blocks of 256 on an SM
        template <int DIM>
        __global__ void __launch_bounds__(ITEM_BLOCK, 2) k_convection(const __grid_constant__ Geom gp, const int* __restrict__ wl, const long long* __restrict__ lo,
                                     const uint32_t* __restrict__ cells, const double* __restrict__ u, double* __restrict__ unp1, UpwindArgs p)
        {
            const Geom& g = gp;
            block_items(
                wl, static_cast<int>(lo[LO_CELLS]), static_cast<int>(lo[LO_CELLS + g.nlev]), grid_team(), 1, [&](int w) { return __ldg(cells + w); },
                [&](bool valid, int w_, int b, int)
                {
                    if (!valid)
                    {
                        return;
                    }
                    const long long w  = w_;
                    const int m        = level_down(g, w_, 0, g.max_level);
                    const Cell cc      = cell_of(g, m, w, b);
                    const int c[3]     = {cc.x, cc.y, cc.z};
                    const long long eX = 32 * w + b;
                    const long long strides[3] = {1, 32LL * g.lv[m].W, 32LL * g.lv[m].W * g.lv[m].R};
                    const double uX    = u[eX];
                    const int nm       = 1 << m;
                    auto leaf          = [&](int l, const int* q)
                    {
                        const Pos at = l >= 0 && l <= g.max_level ? pos_of(g, l, q[0], q[1], DIM == 3 ? q[2] : 0) : Pos{-1, 0};
                        return at.w >= 0 && ((__ldg(cells + at.w) >> at.b) & 1u);
                    };
                    auto val = [&](int l, const int* q) { return u[elem_at(g, l, q[0], q[1], DIM == 3 ? q[2] : 0)]; };
                    // a same-level leaf at element e
                    auto leaf_elem = [&](long long e) { return (__ldg(cells + (e >> 5)) >> (e & 31)) & 1u; };
                    double um[DIM], up[DIM];
                    bool ls_[DIM], rs_[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d)
                    {
                        um[d]  = u[eX - strides[d]];
                        up[d]  = u[eX + strides[d]];
                        ls_[d] = leaf_elem(eX - strides[d]);
                        rs_[d] = leaf_elem(eX + strides[d]);
                    }
                    double acc = 0.;
#pragma unroll
                    for (int d = 0; d < DIM; ++d)
                    {
                        // (a, 0) or (0, a): the coefficient of the left and of the right value
                        const double fl = p.fl[d], fr = p.fr[d];
                        const bool zl = p.zero_l[d], zr = p.zero_r[d];
                        const double lc0 = scale2(fl, m), lc1 = scale2(fr, m);
                        const double rc0 = -lc0, rc1 = -lc1;
                        const bool rs = rs_[d], ls = ls_[d];
                        // same level
                        if (d == 0)
                        {
                            if (rs) acc = add_term(acc, lc0, zl, uX);
                            if (ls) acc = add_term(acc, rc0, zl, um[d]);
                            if (rs) acc = add_term(acc, lc1, zr, up[d]);
                            if (ls) acc = add_term(acc, rc1, zr, uX);
                        }
                        else
                        {
                            if (ls)
                            {
                                acc = add_term(acc, rc0, zl, um[d]);
                                acc = add_term(acc, rc1, zr, uX);
                            }
                            if (rs)
                            {
                                acc = add_term(acc, lc0, zl, uX);
                                acc = add_term(acc, lc1, zr, up[d]);
                            }
                        }
                        if (rs && ls)
                        {
                            continue; // no other face along d
                        }
                        int xp[3] = {c[0], c[1], c[2]}, xm[3] = {c[0], c[1], c[2]};
                        ++xp[d];
                        --xm[d];
                        const bool out_r = xp[d] >= nm, out_l = xm[d] < 0;
                        // level jumps with X the fine cell
                        int pp[3] = {xp[0] >> 1, xp[1] >> 1, xp[2] >> 1}, pm[3] = {xm[0] >> 1, xm[1] >> 1, xm[2] >> 1};
                        const bool lcoarse = !ls && !out_l && m >= 1 && leaf(m - 1, pm);
                        const bool rcoarse = !rs && !out_r && m >= 1 && leaf(m - 1, pp);
                        if (lcoarse)
                        {
                            acc = add_term(acc, rc0, zl, um[d]);
                            acc = add_term(acc, rc1, zr, uX);
                        }
                        if (rcoarse)
                        {
                            acc = add_term(acc, lc0, zl, uX);
                            acc = add_term(acc, lc1, zr, up[d]);
                        }
                        // level jumps with X the coarse cell: its face children at m+1
                        int ch[3]        = {2 * c[0], 2 * c[1], 2 * c[2]};
                        ch[d]            = 2 * c[d] + 2;
                        const bool rfine = !rs && !rcoarse && !out_r && leaf(m + 1, ch);
                        ch[d]            = 2 * c[d] - 1;
                        const bool lfine = !ls && !lcoarse && !out_l && leaf(m + 1, ch);
                        // fine rows of the face in row order (z outer, y inner); a face
                        // normal to y or z has the pair of fine cells within each row
                        const int nrow = (d == 0) ? (DIM == 3 ? 4 : 2) : (DIM == 3 ? 2 : 1);
                        const double sf = pow2(m - DIM + 1);
                        if (rfine)
                        {
                            const double j0 = sf * fl, j1 = sf * fr;
                            for (int r = 0; r < nrow; ++r)
                            {
                                int q[3] = {2 * c[0], 2 * c[1], 2 * c[2]};
                                q[d]     = 2 * c[d] + 1;
                                if (d == 0)
                                {
                                    q[1] += r & 1;
                                    if (DIM == 3)
                                    {
                                        q[2] += r >> 1;
                                    }
                                    int qe[3] = {q[0] + 1, q[1], q[2]};
                                    acc       = add_term(acc, j0, zl, val(m + 1, q));
                                    acc       = add_term(acc, j1, zr, val(m + 1, qe));
                                }
                                else
                                {
                                    if (DIM == 3)
                                    {
                                        q[d == 1 ? 2 : 1] += r;
                                    }
                                    int qb[3] = {q[0] + 1, q[1], q[2]};
                                    int qe[3] = {q[0], q[1], q[2]}, qbe[3] = {qb[0], qb[1], qb[2]};
                                    ++qe[d];
                                    ++qbe[d];
                                    acc = add_pair(acc, j0, zl, val(m + 1, q), val(m + 1, qb));
                                    acc = add_pair(acc, j1, zr, val(m + 1, qe), val(m + 1, qbe));
                                }
                            }
                        }
                        if (lfine)
                        {
                            const double j0 = -sf * fl, j1 = -sf * fr;
                            for (int r = 0; r < nrow; ++r)
                            {
                                int q[3] = {2 * c[0], 2 * c[1], 2 * c[2]}; // Q, inside X on its left face
                                if (d == 0)
                                {
                                    q[1] += r & 1;
                                    if (DIM == 3)
                                    {
                                        q[2] += r >> 1;
                                    }
                                    int qm[3] = {q[0] - 1, q[1], q[2]};
                                    acc       = add_term(acc, j0, zl, val(m + 1, qm));
                                    acc       = add_term(acc, j1, zr, val(m + 1, q));
                                }
                                else
                                {
                                    if (DIM == 3)
                                    {
                                        q[d == 1 ? 2 : 1] += r;
                                    }
                                    int qb[3] = {q[0] + 1, q[1], q[2]};
                                    int qm[3] = {q[0], q[1], q[2]}, qbm[3] = {qb[0], qb[1], qb[2]};
                                    --qm[d];
                                    --qbm[d];
                                    acc = add_pair(acc, j0, zl, val(m + 1, qm), val(m + 1, qbm));
                                    acc = add_pair(acc, j1, zr, val(m + 1, q), val(m + 1, qb));
                                }
                            }
                        }
                        // boundary interfaces
                        if (out_r)
                        {
                            acc = add_term(acc, lc0, zl, uX);
                            acc = add_term(acc, lc1, zr, up[d]);
                        }
                        if (out_l)
                        {
                            acc = add_term(acc, -lc0, zl, um[d]);
                            acc = add_term(acc, -lc1, zr, uX);
                        }
                    }
                    unp1[eX] = uX - p.dt * acc;
                });
        }

        // --------------------------------------------------- layout moves
        // Each warp takes MOVE_WORDS listed words at a time: their bits and ranks are loaded by one lane each, then
        // the words' values move together, all loads in flight at once (a warp per word waits for list entry,
        // bits, rank and value in turn, word after word).
        constexpr int MOVE_WORDS = 8;

        template <class LoadF, class StoreF>
        __device__ __forceinline__ void move_words(const int* __restrict__ wl, const long long* __restrict__ lo, int nlev, const uint32_t* __restrict__ ref,
                                                   const int* __restrict__ rank, LoadF load, StoreF store)
        {
            const int lane  = threadIdx.x & 31;
            const int begin = static_cast<int>(lo[LO_REF]), end = static_cast<int>(lo[LO_REF + nlev]);
            for (int c0 = begin + static_cast<int>(warp_id()) * MOVE_WORDS; c0 < end; c0 += static_cast<int>(warp_count()) * MOVE_WORDS)
            {
                int w      = 0, r = 0;
                uint32_t m = 0u;
                if (lane < MOVE_WORDS && c0 + lane < end)
                {
                    w = wl[c0 + lane];
                    m = ref[w];
                    r = rank[w];
                }
                double v[MOVE_WORDS];
#pragma unroll
                for (int k = 0; k < MOVE_WORDS; ++k)
                {
                    const long long e   = 32LL * __shfl_sync(FULL_MASK, w, k) + lane;
                    const uint32_t bits = __shfl_sync(FULL_MASK, m, k);
                    const int at        = __shfl_sync(FULL_MASK, r, k) + __popc(bits & ((1u << lane) - 1u));
                    v[k]                = ((bits >> lane) & 1u) ? load(e, at) : 0.;
                }
#pragma unroll
                for (int k = 0; k < MOVE_WORDS; ++k)
                {
                    const long long e   = 32LL * __shfl_sync(FULL_MASK, w, k) + lane;
                    const uint32_t bits = __shfl_sync(FULL_MASK, m, k);
                    const int at        = __shfl_sync(FULL_MASK, r, k) + __popc(bits & ((1u << lane) - 1u));
                    if ((bits >> lane) & 1u)
                    {
                        store(e, at, v[k]);
                    }
                }
            }
        }

        __global__ void k_gather(const int* wl, const long long* lo, int nlev, const uint32_t* ref, const int* rank, const double* __restrict__ dense,
                                 double* __restrict__ compact)
        {
            move_words(wl, lo, nlev, ref, rank, [&](long long e, int) { return dense[e]; }, [&](long long, int at, double v) { compact[at] = v; });
        }

        __global__ void k_scatter(const int* wl, const long long* lo, int nlev, const uint32_t* ref, const int* rank, const double* __restrict__ compact,
                                  double* __restrict__ dense)
        {
            move_words(wl, lo, nlev, ref, rank, [&](long long, int at) { return compact[at]; }, [&](long long e, int, double v) { dense[e] = v; });
        }

        // details in the reference numbering: a cell whose parent the pass did not examine has none (0)
        __global__ void k_gather_details(MeshPtrs m, int nlev, const uint32_t* exam, const double* det, double* compact)
        {
            warp_list(m.wl_ref, m.lo[LO_REF], m.lo[LO_REF + nlev], warp_id(), warp_count(), [&](long long w) { return m.ref[w]; },
                      [&](long long w, int b)
                      { compact[ref_index(m.ref, m.rank, Pos{w, b})] = ((exam[w] >> b) & 1u) ? det[32 * w + b] : 0.; });
        }

        __global__ void k_tag_bytes(MeshPtrs m, int nlev, const uint32_t* tk, const uint32_t* tc, const uint32_t* tr, uint8_t* compact)
        {
            warp_list(m.wl_ref, m.lo[LO_REF], m.lo[LO_REF + nlev], warp_id(), warp_count(), [&](long long w) { return m.ref[w]; },
                      [&](long long w, int b)
                      {
                          const uint32_t t = ((tk[w] >> b) & 1u) | (((tc[w] >> b) & 1u) << 1) | (((tr[w] >> b) & 1u) << 2);
                          compact[ref_index(m.ref, m.rank, Pos{w, b})] = static_cast<uint8_t>(t);
                      });
        }

        __global__ void k_fill(const int* __restrict__ wl, const long long* __restrict__ lo, int nlev, const uint32_t* __restrict__ ref, double* dense,
                               double v)
        {
            const int lane  = threadIdx.x & 31;
            const int begin = static_cast<int>(lo[LO_REF]), end = static_cast<int>(lo[LO_REF + nlev]);
            for (int c0 = begin + static_cast<int>(warp_id()) * MOVE_WORDS; c0 < end; c0 += static_cast<int>(warp_count()) * MOVE_WORDS)
            {
                int w      = 0;
                uint32_t m = 0u;
                if (lane < MOVE_WORDS && c0 + lane < end)
                {
                    w = wl[c0 + lane];
                    m = ref[w];
                }
#pragma unroll
                for (int k = 0; k < MOVE_WORDS; ++k)
                {
                    const long long e   = 32LL * __shfl_sync(FULL_MASK, w, k) + lane;
                    const uint32_t bits = __shfl_sync(FULL_MASK, m, k);
                    if ((bits >> lane) & 1u)
                    {
                        dense[e] = v;
                    }
                }
            }
        }
    } // namespace

    namespace
    {
        // blocks of c.block threads: one warp per word of levels l0..l1, at most
        // max_blocks blocks of 8 warps' worth of warps
        int blocks_words(const Ctx& c, int l0, int l1)
        {
            if (l1 < l0)
            {
                return 1;
            }
            const Geom& g          = c.g;
            const long long wpb    = c.block / 32;
            const long long nb     = (g.lv[l1].woff + g.lv[l1].nwords - g.lv[l0].woff + wpb - 1) / wpb;
            const long long cap    = std::max(1LL, c.max_blocks * 8 / wpb);
            return static_cast<int>(nb < 1 ? 1 : (nb > cap ? cap : nb));
        }
    } // namespace

    cudaError_t launch_gather(Ctx& c, const DeviceMesh& m, const double* dense, double* compact)
    {
        k_gather<<<blocks_words(c, 0, c.g.nlev - 1), c.block, 0, c.stream>>>(m.wl_ref, m.d_lo, c.g.nlev, m.ref, m.rank, dense, compact);
        launched(c, "gather");
        return cudaGetLastError();
    }

    int gather_compact(Ctx& c, const DeviceMesh& m, const double* dense, double* compact)
    {
        if (launch_gather(c, m, dense, compact) != cudaSuccess)
        {
            c.err = "gather: kernel launch failed";
            return SG_ERR_CUDA;
        }
        return SG_OK;
    }

    int gather_details(Ctx& c, const DeviceMesh& m, double* compact)
    {
        k_gather_details<<<blocks_words(c, 0, c.g.nlev - 1), c.block, 0, c.stream>>>(mesh_ptrs(m), c.g.nlev, c.exam, c.detail, compact);
        launched(c, "gather");
        return check(c, "gather_details");
    }

    int tag_bytes(Ctx& c, const DeviceMesh& m, uint8_t* compact)
    {
        k_tag_bytes<<<blocks_words(c, 0, c.g.nlev - 1), c.block, 0, c.stream>>>(mesh_ptrs(m), c.g.nlev, c.tk, c.tc, c.tr, compact);
        launched(c, "gather");
        return check(c, "tag_bytes");
    }

    cudaError_t read_device_error(Ctx& c, int* v)
    {
        *v            = 0;
        cudaError_t e = cudaMemcpyAsync(v, c.g.err, sizeof(int), cudaMemcpyDeviceToHost, c.stream);
        if (e == cudaSuccess)
        {
            e = cudaStreamSynchronize(c.stream);
        }
        if (e == cudaSuccess && *v)
        {
            e = cudaMemsetAsync(c.g.err, 0, sizeof(int), c.stream);
        }
        return e;
    }

    int scatter_compact(Ctx& c, const DeviceMesh& m, const double* compact, double* dense)
    {
        k_scatter<<<blocks_words(c, 0, c.g.nlev - 1), c.block, 0, c.stream>>>(m.wl_ref, m.d_lo, c.g.nlev, m.ref, m.rank, compact, dense);
        launched(c, "scatter");
        return check(c, "scatter");
    }

    int fill_ref(Ctx& c, const DeviceMesh& m, double* dense, double value)
    {
        k_fill<<<blocks_words(c, 0, c.g.nlev - 1), c.block, 0, c.stream>>>(m.wl_ref, m.d_lo, c.g.nlev, m.ref, dense, value);
        launched(c, "fill");
        return check(c, "fill");
    }

    // --------------------------------------------------------------- graphs
    // The launch sequences below depend only on the level geometry and on
    // the buffers they touch: list sizes and level ranges are read on the
    // device.  Each is captured once per buffer combination into a CUDA graph
    // and replayed.
    template <class F>
    int run_cached(Ctx& c, unsigned long long k0, unsigned long long k1, unsigned long long k2, unsigned long long k3, F seq)
    {
        if (!c.use_graphs || c.timers.enabled)
        {
            if (c.trace.enabled)
            {
                trace_mark(c, nullptr);
            }
            return seq();
        }
        // a traced sequence carries its trace events as graph nodes (a head event first): a graph of its own
        if (c.trace.enabled)
        {
            k0 |= 1ull << 63;
        }
        for (auto& e : c.graphs)
        {
            if (e.key[0] == k0 && e.key[1] == k1 && e.key[2] == k2 && e.key[3] == k3)
            {
                if (cudaGraphLaunch(e.exec, c.stream) != cudaSuccess)
                {
                    return check(c, "cudaGraphLaunch");
                }
                c.n_launches += e.kernels;
                if (c.trace.enabled)
                {
                    for (const auto& mk : e.marks)
                    {
                        for (const auto& seen : c.trace.marks)
                        {
                            c.trace.reused = c.trace.reused || seen.second == mk.second;
                        }
                        c.trace.marks.push_back(mk);
                    }
                }
                return SG_OK;
            }
        }
        if (cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        {
            return check(c, "cudaStreamBeginCapture");
        }
        const int before      = c.n_launches;
        const size_t marks0   = c.trace.marks.size();
        if (c.trace.enabled)
        {
            trace_mark(c, nullptr);
        }
        int st                = seq();
        cudaGraph_t graph     = nullptr;
        cudaError_t e         = cudaStreamEndCapture(c.stream, &graph);
        // the trace events recorded during the capture belong to the graph
        std::vector<std::pair<const char*, cudaEvent_t>> marks(c.trace.marks.begin() + static_cast<long>(std::min(marks0, c.trace.marks.size())),
                                                               c.trace.marks.end());
        c.trace.marks.resize(std::min(marks0, c.trace.marks.size()));
        if (st || e != cudaSuccess)
        {
            if (graph)
            {
                cudaGraphDestroy(graph);
            }
            for (const auto& mk : marks)
            {
                give_event(c, mk.second);
            }
            if (!st)
            {
                c.err = std::string("graph capture: ") + cudaGetErrorString(e);
                st    = SG_ERR_CUDA;
            }
            cudaGetLastError();
            return st;
        }
        cudaGraphExec_t exec = nullptr;
        e                    = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess)
        {
            for (const auto& mk : marks)
            {
                give_event(c, mk.second);
            }
            return check(c, "cudaGraphInstantiate");
        }
        if (c.graphs.size() >= 64)
        {
            cudaGraphExecDestroy(c.graphs.front().exec);
            for (const auto& mk : c.graphs.front().marks)
            {
                give_event(c, mk.second);
            }
            c.graphs.erase(c.graphs.begin());
        }
        const int kernels = c.n_launches - before;
        c.graphs.push_back({{k0, k1, k2, k3}, exec, kernels, marks});
        c.trace.marks.insert(c.trace.marks.end(), marks.begin(), marks.end());
        if (cudaGraphLaunch(exec, c.stream) != cudaSuccess)
        {
            return check(c, "cudaGraphLaunch");
        }
        return SG_OK;
    }

    namespace
    {
        // A captured chain of kernel launches (one stream, no other node types) rebuilt with its kernels in the
        // opposite order.  The kernel parameters are copied from the captured nodes.
        cudaError_t reverse_chain(cudaGraph_t in, cudaGraph_t* out)
        {
            *out     = nullptr;
            size_t n = 0, nr = 0;
            cudaError_t e = cudaGraphGetNodes(in, nullptr, &n);
            if (e == cudaSuccess)
            {
                e = cudaGraphGetRootNodes(in, nullptr, &nr);
            }
            if (e != cudaSuccess)
            {
                return e;
            }
            std::vector<cudaGraphNode_t> order;
            if (n > 0)
            {
                if (nr != 1)
                {
                    return cudaErrorInvalidValue;
                }
                cudaGraphNode_t cur = nullptr;
                if ((e = cudaGraphGetRootNodes(in, &cur, &nr)) != cudaSuccess)
                {
                    return e;
                }
                while (order.size() <= n)
                {
                    order.push_back(cur);
                    size_t nd = 0;
                    if ((e = cudaGraphNodeGetDependentNodes(cur, nullptr, nullptr, &nd)) != cudaSuccess)
                    {
                        return e;
                    }
                    if (nd == 0)
                    {
                        break;
                    }
                    if (nd != 1 || (e = cudaGraphNodeGetDependentNodes(cur, &cur, nullptr, &nd)) != cudaSuccess)
                    {
                        return nd != 1 ? cudaErrorInvalidValue : e;
                    }
                }
                if (order.size() != n)
                {
                    return cudaErrorInvalidValue;
                }
            }
            if ((e = cudaGraphCreate(out, 0)) != cudaSuccess)
            {
                return e;
            }
            cudaGraphNode_t prev = nullptr;
            for (auto it = order.rbegin(); it != order.rend(); ++it)
            {
                cudaGraphNodeType t;
                cudaKernelNodeParams kp{};
                cudaGraphNode_t node = nullptr;
                if ((e = cudaGraphNodeGetType(*it, &t)) != cudaSuccess || t != cudaGraphNodeTypeKernel
                    || (e = cudaGraphKernelNodeGetParams(*it, &kp)) != cudaSuccess
                    || (e = cudaGraphAddKernelNode(&node, *out, prev ? &prev : nullptr, prev ? 1 : 0, &kp)) != cudaSuccess)
                {
                    cudaGraphDestroy(*out);
                    *out = nullptr;
                    return e != cudaSuccess ? e : cudaErrorInvalidValue;
                }
                prev = node;
            }
            return cudaSuccess;
        }
    } // namespace

    // run_cached for a launch sequence whose launches must run in the opposite order (the transpose of a chain of
    // linear operators): captured once per key, reversed, cached and replayed.  Always a graph (the reversal needs
    // the captured chain), and with no trace events inside.
    template <class F>
    int run_reversed(Ctx& c, unsigned long long k0, unsigned long long k1, unsigned long long k2, unsigned long long k3, F seq)
    {
        k0 |= 1ull << 62;
        for (auto& e : c.graphs)
        {
            if (e.key[0] == k0 && e.key[1] == k1 && e.key[2] == k2 && e.key[3] == k3)
            {
                c.n_launches += e.kernels;
                return cudaGraphLaunch(e.exec, c.stream) != cudaSuccess ? check(c, "cudaGraphLaunch") : SG_OK;
            }
        }
        const bool traced = c.trace.enabled;
        c.trace.enabled   = false;
        if (cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        {
            c.trace.enabled = traced;
            return check(c, "cudaStreamBeginCapture");
        }
        const int before  = c.n_launches;
        int st            = seq();
        cudaGraph_t graph = nullptr;
        cudaError_t e     = cudaStreamEndCapture(c.stream, &graph);
        c.trace.enabled   = traced;
        cudaGraph_t rev   = nullptr;
        if (!st && e == cudaSuccess)
        {
            e = reverse_chain(graph, &rev);
        }
        if (graph)
        {
            cudaGraphDestroy(graph);
        }
        if (st || e != cudaSuccess)
        {
            if (!st)
            {
                c.err = std::string("reversed graph: ") + cudaGetErrorString(e);
                st    = SG_ERR_CUDA;
            }
            cudaGetLastError();
            return st;
        }
        cudaGraphExec_t exec = nullptr;
        e                    = cudaGraphInstantiate(&exec, rev, 0);
        cudaGraphDestroy(rev);
        if (e != cudaSuccess)
        {
            return check(c, "cudaGraphInstantiate");
        }
        if (c.graphs.size() >= 64)
        {
            cudaGraphExecDestroy(c.graphs.front().exec);
            for (const auto& mk : c.graphs.front().marks)
            {
                give_event(c, mk.second);
            }
            c.graphs.erase(c.graphs.begin());
        }
        c.graphs.push_back({{k0, k1, k2, k3}, exec, c.n_launches - before, {}});
        return cudaGraphLaunch(exec, c.stream) != cudaSuccess ? check(c, "cudaGraphLaunch") : SG_OK;
    }

    namespace
    {
        // the setup of one pass baked into a captured graph (the host computes
        // it exactly as for the staged copy of the per-pass path)
        __global__ void k_pass_setup(PassSetup p, PassSetup* d)
        {
            for (int i = threadIdx.x; i < 3 * MAXLEV; i += blockDim.x)
            {
                d->eps[i] = p.eps[i];
            }
            if (threadIdx.x == 0)
            {
                d->ite = p.ite;
            }
        }

        // the condition of a conditional graph node from a device word
        __global__ void k_cond_set(cudaGraphConditionalHandle h, const int* flag, int invert)
        {
            cudaGraphSetConditional(h, ((*flag != 0) ? 1u : 0u) ^ static_cast<unsigned>(invert));
        }

        // end of a loop body: repeat while *flag is set, at most limit times
        // (the count at *iter, reset before the loop); past the limit the
        // mesh's error word records it and the loop stops
        __global__ void k_loop_next(cudaGraphConditionalHandle h, const int* flag, int* iter, int limit, int* err)
        {
            const int n = ++*iter;
            bool go     = *flag != 0;
            if (go && n >= limit)
            {
                atomicOr(err, 4);
                go = false;
            }
            cudaGraphSetConditional(h, go ? 1u : 0u);
        }

        // after the passes: which final buffers (parity of the transitions) and whether the ghosts need updating
        __global__ void k_step_flags(int* a)
        {
            const int trans = a[A_TRANS];
            a[A_PAR0]       = (trans & 1) == 0;
            a[A_PAR1]       = (trans & 1) == 1;
            a[A_NEEDG]      = a[A_PASSES] == trans;
        }

        // the leaf bitmap of a transition into recording slot a[A_TRANS] (before the count moves on)
        __global__ void k_record_bits(const uint32_t* cells, uint32_t* slots, const int* a, long long words)
        {
            uint32_t* dst = slots + static_cast<long long>(a[A_TRANS]) * words;
            for (long long w = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; w < words; w += static_cast<long long>(gridDim.x) * blockDim.x)
            {
                dst[w] = cells[w];
            }
        }

        __global__ void k_adapt_words(int* a, int slot, const int* src, int value, int add)
        {
            // a[slot] = src ? *src : value, or += when add
            const int v = src ? *src : value;
            a[slot]     = add ? a[slot] + v : v;
        }

        // Appends to the graph captured on c.stream a conditional node (IF:
        // its body runs once when the condition holds; WHILE: while it holds)
        // whose condition is set by set_cond(handle) just before the node and
        // whose body is captured from body(handle) on a capture stream of its
        // own.  Conditional bodies hold kernels, memsets and copies only.
        template <class SetCond, class Body>
        int capture_conditional(Ctx& c, cudaGraphConditionalNodeType type, SetCond set_cond, Body body)
        {
            cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
            cudaGraph_t graph          = nullptr;
            if (cudaStreamGetCaptureInfo(c.stream, &cs, nullptr, &graph) != cudaSuccess || cs != cudaStreamCaptureStatusActive)
            {
                c.err = "conditional node outside a capture";
                return SG_ERR_STATE;
            }
            if (c.cap_depth >= Ctx::CAPTURE_DEPTH || !c.cap_streams[c.cap_depth])
            {
                c.err = "conditional nodes nested too deep";
                return SG_ERR_STATE;
            }
            cudaGraphConditionalHandle h{};
            if (cudaGraphConditionalHandleCreate(&h, graph, 0, cudaGraphCondAssignDefault) != cudaSuccess)
            {
                return check(c, "cudaGraphConditionalHandleCreate");
            }
            set_cond(h);
            const cudaGraphNode_t* deps = nullptr;
            size_t nd                   = 0;
            if (cudaStreamGetCaptureInfo(c.stream, &cs, nullptr, &graph, &deps, nullptr, &nd) != cudaSuccess)
            {
                return check(c, "cudaStreamGetCaptureInfo");
            }
            cudaGraphNodeParams np{};
            np.type                 = cudaGraphNodeTypeConditional;
            np.conditional.handle   = h;
            np.conditional.type     = type;
            np.conditional.size     = 1;
            cudaGraphNode_t node    = nullptr;
            if (cudaGraphAddNode(&node, graph, deps, nullptr, nd, &np) != cudaSuccess)
            {
                return check(c, "cudaGraphAddNode (conditional)");
            }
            cudaGraph_t bodyg = np.conditional.phGraph_out[0];
            if (cudaStreamUpdateCaptureDependencies(c.stream, &node, nullptr, 1, cudaStreamSetCaptureDependencies) != cudaSuccess)
            {
                return check(c, "cudaStreamUpdateCaptureDependencies");
            }
            cudaStream_t s2 = c.cap_streams[c.cap_depth];
            if (cudaStreamBeginCaptureToGraph(s2, bodyg, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
            {
                return check(c, "cudaStreamBeginCaptureToGraph");
            }
            ++c.cap_depth;
            std::swap(c.stream, s2);
            int st = body(h);
            std::swap(c.stream, s2);
            --c.cap_depth;
            cudaGraph_t out = nullptr;
            const cudaError_t e = cudaStreamEndCapture(s2, &out);
            if (!st && e != cudaSuccess)
            {
                c.err = std::string("conditional body capture: ") + cudaGetErrorString(e);
                st    = SG_ERR_CUDA;
            }
            return st;
        }

        template <class Body>
        int capture_if(Ctx& c, const int* flag, Body body)
        {
            return capture_conditional(
                c, cudaGraphCondTypeIf,
                [&](cudaGraphConditionalHandle h)
                {
                    k_cond_set<<<1, 1, 0, c.stream>>>(h, flag, 0);
                    launched(c, "cond_set");
                },
                [&](cudaGraphConditionalHandle) { return body(); });
        }

        unsigned long long bits_of(double v)
        {
            unsigned long long b;
            std::memcpy(&b, &v, sizeof(b));
            return b;
        }

        unsigned long long ptr_key(const void* p)
        {
            return static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(p));
        }

        // update_ghost_mr / update_ghost_mr_aggregated (algorithm/update_ghost_mr.hpp:195-270)
        // of the sequence's fields.  update_ghost_periodic runs after the boundary
        // conditions of a level and after its prediction
        // (update_ghost_mr.hpp:205-234); the copy the reference also makes before
        // the boundary conditions is overwritten by this one before anything
        // reads it: the boundary conditions of a serial run read and write no
        // ghost across a periodic axis.
        void ghost_phases(Sequence& s)
        {
            const Geom& g  = s.c.g;
            const int lmin = g.min_level >= 2 ? g.min_level - 2 : 0; // no reference cell below min_level-2
            auto periodic  = [&](int l)
            {
                for (int d = 0; d < g.dim; ++d)
                {
                    if ((g.periodic >> d) & 1)
                    {
                        s.add(OP_PERIODIC_COPY, l, l, d); // a later axis reads the ghosts an earlier one wrote
                    }
                }
            };
            for (int l = g.max_level; l >= lmin; --l)
            {
                s.add(OP_GHOST, l, 0);
                periodic(l);
            }
            for (int l = std::max(lmin, 1); l <= g.max_level; ++l)
            {
                s.add(OP_PREDICT, l, l);
                periodic(l);
            }
        }

        // threads per block of the transposed launches, whose linear forms take up to 96 (2D) and 255 (3D) registers:
        // 65536 registers of an SM hold no larger block
        int reverse_block(const Ctx& c)
        {
            return std::min(c.block, c.g.dim == 3 ? 256 : 512);
        }

        // the same transposed, launch by launch in forward order (run_reversed turns the captured chain round)
        template <int DIM>
        int ghost_reverse_launches(Ctx& c, const DeviceMesh& dm, double* lam, int* overflow, bool has_bc)
        {
            const Geom& g    = c.g;
            const MeshPtrs m = mesh_ptrs(dm);
            const RevAcc<FormCap<DIM>::value> u{lam, lam, overflow, 1};
            const int lmin  = g.min_level >= 2 ? g.min_level - 2 : 0;
            const int block = reverse_block(c);
            for (int l = g.max_level; l >= lmin; --l)
            {
                const int nb = static_cast<int>(std::min(16384LL, (boundary_count<DIM>(g, l) + block - 1) / block));
                const int np = l > lmin ? blocks_words(c, l - 1, l - 1) : 0;
                if (nb + np > 0)
                {
                    k_ghost_reverse<DIM><<<nb + np, block, 0, c.stream>>>(c.g, l, 1, nb, has_bc ? 1 : 0, m, u);
                    launched(c, "ghost_level");
                }
                if (l >= g.min_level)
                {
                    const int ncb = static_cast<int>(std::min(16384LL, (corner_count<DIM>(g, l) + block - 1) / block));
                    k_ghost_reverse<DIM><<<ncb, block, 0, c.stream>>>(c.g, l, 2, ncb, has_bc ? 1 : 0, m, u);
                    launched(c, "ghost_corner_projection");
                }
            }
            for (int l = std::max(lmin, 1); l <= g.max_level; ++l)
            {
                k_predict_reverse<DIM><<<blocks_words(c, l, l), block, 0, c.stream>>>(c.g, l, c.cfg.prediction_radius, m, u);
                launched(c, "predict");
            }
            return check(c, "update_ghost_mr (transpose)");
        }

        FieldSlot slot_of(const DeviceField& f)
        {
            return {f.data, f.spare, f.bc_value, f.has_bc ? 1 : 0};
        }

        std::vector<FieldSlot> slots_of(const std::vector<DeviceField*>& fs)
        {
            std::vector<FieldSlot> v;
            for (const DeviceField* f : fs)
            {
                v.push_back(slot_of(*f));
            }
            return v;
        }

        // body(first, n) on groups of at most PHASE_FIELDS fields
        template <class Body>
        void field_groups(Sequence& s, const std::vector<FieldSlot>& fs, Body body)
        {
            for (int k = 0; k < static_cast<int>(fs.size()); k += PHASE_FIELDS)
            {
                s.fields(fs.data(), k, std::min(PHASE_FIELDS, static_cast<int>(fs.size()) - k));
                body();
            }
        }

        int seq_ghost(Ctx& c, DeviceMesh& m, double* u, bool has_bc, double bcv)
        {
            ScopedTimer timer(c, T_GHOST);
            Sequence s(c, m, m);
            const FieldSlot f{u, nullptr, bcv, has_bc ? 1 : 0};
            s.fields(&f, 0, 1);
            ghost_phases(s);
            return s.done("update_ghost_mr");
        }

        // Adapt::harten up to the fixed-point test (mr/adapt.hpp:276-375):
        // ghost update, details, tags, new cells, graduation and the comparison
        // with the current cells.  Reads the pass setup staged in pinned memory;
        // leaves the flags in pinned memory.  No host synchronisation.
        // The fields fs drive the criteria, one detail component each, the
        // components stored one dense slab after the other.
        int seq_front(Ctx& c, DeviceMesh& m, DeviceMesh& nm, const std::vector<DeviceField*>& fs, const PassSetup* graphed = nullptr)
        {
            const Geom& g  = c.g;
            const int minl = g.min_level;
            const int maxl = g.max_level;
            if (graphed)
            {
                k_pass_setup<<<1, 128, 0, c.stream>>>(*graphed, c.d_setup);
                launched(c, "pass_setup");
            }
            const std::vector<FieldSlot> slots = slots_of(fs);
            Sequence s(c, m, nm);
            s.env.setup_host = graphed ? nullptr : c.h_setup;
            s.fields(slots.data(), 0, std::min(PHASE_FIELDS, static_cast<int>(slots.size())));
            s.add(OP_PASS_BEGIN);
            s.timer_start(T_GHOST);
            field_groups(s, slots, [&]() { ghost_phases(s); });
            s.timer_stop(T_GHOST);

            s.timer_start(T_DETAIL);
            const int dl0 = minl > 0 ? minl - 1 : 0;
            const int dl1 = maxl - 1;
            if (dl1 >= dl0)
            {
                field_groups(s, slots,
                             [&]()
                             {
                                 if (c.rel_detail)
                                 {
                                     s.add(OP_ABSMAX_INIT);
                                     s.add(OP_ABSMAX);
                                 }
                                 s.add(OP_DETAIL, dl0, dl1);
                             });
            }
            s.timer_stop(T_DETAIL);

            s.timer_start(T_TAG);
            s.add(OP_CRITERIA);
            s.timer_stop(T_TAG);

            // children at levels maxl .. min_level: below min_level no parent has a leaf child, so the operator has
            // nothing to do there; periodic axes: update_tag_periodic before each level's operator, and on the
            // levels below too (mr/adapt.hpp:348-357)
            s.timer_start(T_FINALIZE);
            for (int l = maxl; l >= 1; --l)
            {
                for (int d = 0; d < g.dim; ++d)
                {
                    if (!((g.periodic >> d) & 1))
                    {
                        continue;
                    }
                    if (g.lv[l].n >= 2 * g.ghost_width)
                    {
                        s.add(OP_PERIODIC_TAG, l, l, 4 * d + 3);
                        continue;
                    }
                    s.add(OP_PERIODIC_TAG, l, l, 4 * d + 1);
                    s.add(OP_PERIODIC_TAG, l, l, 4 * d + 2);
                }
                if (l >= std::max(1, minl))
                {
                    s.add(OP_MAXIMUM, l, l);
                }
            }
            s.timer_stop(T_FINALIZE);

            s.timer_start(T_MESH_UPDATE);
            // the second graduation pass runs on the device only if the first one refined
            s.add(OP_NEW_CELLS, minl, maxl);
            grad_pass_phases(s, F_GRAD0, -1);
            if (!graphed)
            {
                grad_pass_phases(s, F_GRAD1, F_GRAD0);
            }
            else
            {
                // make_graduation to its fixed point on the device: further passes while the last one refined
                // (at most 64, as on the host path)
                s.flush();
                k_adapt_words<<<1, 1, 0, c.stream>>>(c.d_adapt, A_LOOP, c.d_flags + F_GRAD0, 0, 0);
                k_adapt_words<<<1, 1, 0, c.stream>>>(c.d_adapt, A_ITER, nullptr, 0, 0);
                launched(c, "adapt_words", 2);
                const int st = capture_conditional(
                    c, cudaGraphCondTypeWhile,
                    [&](cudaGraphConditionalHandle h)
                    {
                        k_cond_set<<<1, 1, 0, c.stream>>>(h, c.d_adapt + A_LOOP, 0);
                        launched(c, "cond_set");
                    },
                    [&](cudaGraphConditionalHandle h)
                    {
                        cudaMemsetAsync(c.d_flags + F_GRADX, 0, sizeof(int), c.stream);
                        Sequence s2(c, m, nm);
                        grad_pass_phases(s2, F_GRADX, -1);
                        const int st2 = s2.done("graduation");
                        if (!st2)
                        {
                            k_adapt_words<<<1, 1, 0, c.stream>>>(c.d_adapt, A_LOOP, c.d_flags + F_GRADX, 0, 0);
                            k_loop_next<<<1, 1, 0, c.stream>>>(h, c.d_adapt + A_LOOP, c.d_adapt + A_ITER, 64, c.g.err);
                            launched(c, "loop_next", 2);
                        }
                        return st2;
                    });
                if (st)
                {
                    return st;
                }
            }
            s.report(graphed ? nullptr : c.h_flags);
            s.add(OP_COMPARE);
            s.timer_stop(T_MESH_UPDATE);
            return s.done("harten front");
        }

        // new mesh from the new cells and update_fields (mr/adapt.hpp:380-386)
        // for the adapted fields fs and the fields os carried along (their
        // ghosts are updated first, mr/adapt.hpp:383)
        // ahead: launched before the host knows whether the pass changed the mesh;
        // the phases hang on the pass's flag.  The pass's front left the union of the
        // new mesh empty.
        int seq_back(Ctx& c, DeviceMesh& m, DeviceMesh& nm, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os,
                     bool ahead = false)
        {
            Sequence s(c, m, nm);
            s.guard(ahead ? c.d_flags + F_AHEAD : nullptr);
            if (!os.empty())
            {
                s.timer_start(T_GHOST);
                field_groups(s, slots_of(os), [&]() { ghost_phases(s); });
                s.timer_stop(T_GHOST);
            }
            std::vector<DeviceField*> all(fs);
            all.insert(all.end(), os.begin(), os.end());
            const std::vector<FieldSlot> slots = slots_of(all);
            s.fields(slots.data(), 0, std::min(PHASE_FIELDS, static_cast<int>(slots.size())));
            s.timer_start(T_CONSTRUCTION);
            build_mesh_phases(s, false);
            s.timer_stop(T_CONSTRUCTION);
            s.timer_start(T_FIELDS_UPDATE);
            field_groups(s, slots, [&]() { s.add(OP_UPDATE_FIELDS); });
            s.timer_stop(T_FIELDS_UPDATE);
            return s.done("update_fields");
        }

        // graph-cache key of a list of fields: their buffers and boundary values
        unsigned long long fields_key(const std::vector<DeviceField*>& fs, bool spares)
        {
            unsigned long long h = 1469598103934665603ull;
            auto mix             = [&](unsigned long long v)
            {
                h ^= v;
                h *= 1099511628211ull;
            };
            for (const DeviceField* f : fs)
            {
                mix(ptr_key(spares ? f->spare : f->data));
                mix(f->has_bc ? bits_of(f->bc_value) : 1ull);
            }
            return h;
        }
    } // namespace

    int update_ghost_mr(Ctx& c, DeviceField& f)
    {
        if (c.cfg.ghost_width > 2)
        {
            c.err = "update_ghost_mr: ghost widths 1 and 2 are implemented";
            return SG_ERR_ARG;
        }
        if (f.ghosts_valid && f.ghost_version == c.mesh_version)
        {
            return SG_OK;
        }
        DeviceMesh& m = c.m();
        double* u     = f.data;
        int st        = run_cached(c, 1, static_cast<unsigned long long>(c.cur), ptr_key(u), f.has_bc ? bits_of(f.bc_value) : 1ull,
                                   [&]() { return seq_ghost(c, m, u, f.has_bc, f.bc_value); });
        if (!st)
        {
            f.ghosts_valid  = true;
            f.ghost_version = c.mesh_version;
        }
        return st;
    }

    // Adapt::harten (mr/adapt.hpp:276-389) for one field, in two halves:
    // harten_begin launches everything up to the fixed-point test without
    // waiting; harten_end waits for it, finishes the graduation if needed and
    // launches the new mesh and update_fields.  Between the two halves the
    // host may launch other meshes' work (batched mode).
    int harten_begin(Ctx& c, DeviceField& f, int ite, double eps, double regularity, bool relative_detail)
    {
        return harten_begin_fields(c, {&f}, {}, ite, eps, regularity, relative_detail);
    }

    namespace
    {
        // the criteria thresholds of Harten pass ite (mr/adapt.hpp:325-339,
        // mr/criteria.hpp:20-113): per level eps_l, 2^(reg+dim) eps_l and that
        // over 2^dim, zero on the levels the pass does not examine
        void pass_thresholds(const Ctx& c, int ite, double eps, double regularity, double* out)
        {
            const int minl = c.cfg.min_level, maxl = c.cfg.max_level, dim = c.g.dim;
            for (int l = 0; l < 3 * MAXLEV; ++l)
            {
                out[l] = 0.;
            }
            for (int l = minl; l <= maxl - ite; ++l)
            {
                const int exponent     = dim * (maxl - l);
                out[l]                 = eps / (1 << exponent);
                out[MAXLEV + l]        = std::pow(2.0, regularity + dim) * out[l];
                out[2 * MAXLEV + l]    = out[MAXLEV + l] / (1 << dim);
            }
        }
    } // namespace

    namespace
    {
        // the second half of a pass, from its graph
        int launch_back(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, bool ahead)
        {
            DeviceMesh& m  = c.m();
            DeviceMesh& nm = c.spare();
            const unsigned long long kind = ahead ? 1ull << 40 : 0ull;
            if (fs.size() == 1 && os.empty())
            {
                DeviceField& f = *fs[0];
                return run_cached(c, 3 | kind, static_cast<unsigned long long>(c.cur), ptr_key(f.data), ptr_key(f.spare),
                                  [&]() { return seq_back(c, m, nm, fs, os, ahead); });
            }
            std::vector<DeviceField*> all(fs);
            all.insert(all.end(), os.begin(), os.end());
            return run_cached(c, (7 + 16 * fs.size()) | kind, static_cast<unsigned long long>(c.cur), fields_key(all, false), fields_key(all, true),
                              [&]() { return seq_back(c, m, nm, fs, os, ahead); });
        }
    } // namespace

    int harten_begin_fields(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, int ite, double eps, double regularity,
                            bool relative_detail)
    {
        if (c.cfg.ghost_width > 2)
        {
            c.err = "harten: ghost widths 1 and 2 are implemented";
            return SG_ERR_ARG;
        }
        if (int st = ensure_details(c, static_cast<int>(fs.size())))
        {
            return st;
        }
        DeviceMesh& m  = c.m();
        DeviceMesh& nm = c.spare();
        // the pinned inputs staged here were consumed by the previous pass,
        // which ended with harten_end's synchronisation
        c.h_setup->ite = ite;
        pass_thresholds(c, ite, eps, regularity, c.h_setup->eps);
        // the captured front differs with relative details and with the
        // number of fields: keys of their own
        c.rel_detail = relative_detail;
        // boundary cells are kept in the captured front only with --refine-boundary
        const unsigned long long rb = c.refine_boundary ? 256ull : 0ull;
        int st;
        if (fs.size() == 1)
        {
            DeviceField& f = *fs[0];
            st             = run_cached(c, (relative_detail ? 4 : 2) | rb, static_cast<unsigned long long>(c.cur), ptr_key(f.data),
                                        f.has_bc ? bits_of(f.bc_value) : 1ull, [&]() { return seq_front(c, m, nm, fs); });
        }
        else
        {
            st = run_cached(c, (relative_detail ? 6 : 5) | rb, static_cast<unsigned long long>(c.cur), fields_key(fs, false), fs.size(),
                            [&]() { return seq_front(c, m, nm, fs); });
        }
        // The first pass of an adaptation usually changes the mesh: its second half is queued before the host
        // hears of it, so the GPU does not wait for the round trip.  It hangs on a flag of the pass that is set only
        // when the pass's cells are final and differ: a pass that keeps its mesh, or whose graduation goes on from
        // the host, changes nothing more, the ghosts of the fields carried along included.
        c.back_ahead = !st && ite == 0 && !c.timers.enabled; // the named timers count the halves that run
        if (c.back_ahead)
        {
            st = launch_back(c, fs, os, true);
        }
        return st;
    }

    int harten_end(Ctx& c, DeviceField& f, bool* converged)
    {
        return harten_end_fields(c, {&f}, {}, converged);
    }

    int harten_end_fields(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, bool* converged)
    {
        DeviceMesh& m    = c.m();
        DeviceMesh& nm   = c.spare();
        bool back_queued = c.back_ahead;
        int st;
        if (cudaStreamSynchronize(c.stream) != cudaSuccess)
        {
            return check(c, "harten front sync");
        }
        if (!m.host_valid && (st = counts_arrived(c, m)))
        {
            return st;
        }
        for (DeviceField* f : fs)
        {
            f->ghosts_valid  = true; // the front's ghost update ran on the current mesh
            f->ghost_version = c.mesh_version;
        }
        if (c.h_flags[F_GRAD1])
        {
            // graduation still refining after two passes: finish the fixed
            // point with host-tested passes, then compare again (a second half
            // queued ahead did not run)
            back_queued = false;
            if ((st = graduate(c, m, nm, nullptr)))
            {
                return st;
            }
            cudaMemsetAsync(c.d_flags + F_DIFFER, 0, sizeof(int), c.stream);
            Sequence s(c, m, nm);
            s.add(OP_COMPARE);
            if ((st = s.done("harten compare")))
            {
                return st;
            }
            cudaMemcpyAsync(c.h_flags + F_DIFFER, c.d_flags + F_DIFFER, sizeof(int), cudaMemcpyDeviceToHost, c.stream);
            if (cudaStreamSynchronize(c.stream) != cudaSuccess)
            {
                return check(c, "harten compare sync");
            }
        }
        if (!c.h_flags[F_DIFFER])
        {
            *converged = true;
            return SG_OK;
        }
        *converged = false;
        if (!back_queued && (st = launch_back(c, fs, os, false)))
        {
            return st;
        }
        nm.host_valid = false; // a replayed graph refreshed the counters without host code
        for (const auto* list : {&fs, &os})
        {
            for (DeviceField* f : *list)
            {
                std::swap(f->data, f->spare);
                f->ghosts_valid = false;
            }
        }
        c.cur = 1 - c.cur;
        ++c.mesh_version;
        return SG_OK;
    }

    // The error word of an adaptation: a last pass that kept the mesh reported it with its flags, and nothing
    // that can raise it ran after that (further graduation and the comparison only move bits); otherwise it is
    // read from the device.
    int pass_error(Ctx& c, bool converged)
    {
        return converged && c.h_flags[F_ERR] == 0 ? SG_OK : device_error(c);
    }

    // No synchronisation before the pass: the pinned thresholds it rewrites
    // were consumed before the previous pass's harten_end returned, and its
    // launches queue behind whatever the stream still runs.
    int harten(Ctx& c, DeviceField& f, int ite, double eps, double regularity, bool* converged, bool relative_detail)
    {
        int st = harten_begin(c, f, ite, eps, regularity, relative_detail);
        if (st)
        {
            return st;
        }
        return harten_end(c, f, converged);
    }

    // ---------------------------------------------------------------
    // Operators of one step on a given (frozen) mesh, for the replay and the
    // adjoint: the ghost update and update_fields applied (value) or
    // transposed (reverse: the RevAcc accessor, launches in reverse order).
    int ghost_value(Ctx& c, DeviceMesh& m, double* u, bool has_bc, double bcv)
    {
        Sequence s(c, m, m);
        const FieldSlot f{u, nullptr, bcv, has_bc ? 1 : 0};
        s.fields(&f, 0, 1);
        ghost_phases(s);
        return s.done("update_ghost_mr");
    }

    // lam := G^T lam for the ghost update G of mesh m, in place.  The launch sequence is the one that separates
    // every read from every write (corner projections in launches of their own), captured once per mesh buffer
    // and adjoint array and replayed backwards.
    int ghost_reverse(Ctx& c, DeviceMesh& m, double* lam, int* overflow, bool has_bc)
    {
        const unsigned long long kind = 40ull | (has_bc ? 256ull : 0ull);
        return run_reversed(c, kind, ptr_key(m.ref), ptr_key(lam), ptr_key(overflow),
                            [&]()
                            {
                                return c.g.dim == 2 ? ghost_reverse_launches<2>(c, m, lam, overflow, has_bc)
                                                    : ghost_reverse_launches<3>(c, m, lam, overflow, has_bc);
                            });
    }

    int update_fields_value(Ctx& c, DeviceMesh& m, DeviceMesh& nm, const double* uo, double* un)
    {
        Sequence s(c, m, nm);
        const FieldSlot f{const_cast<double*>(uo), un, 0., 0};
        s.fields(&f, 0, 1);
        s.add(OP_UPDATE_FIELDS);
        return s.done("update_fields");
    }

    // lam_old += T^T lam_new for update_fields T from mesh m to mesh nm (lam_old is not cleared here)
    int update_fields_reverse(Ctx& c, DeviceMesh& m, DeviceMesh& nm, double* lam_new, double* lam_old, int* overflow)
    {
        if (c.g.dim == 2)
        {
            const RevAcc<FormCap<2>::value> r{lam_new, lam_old, overflow, 0};
            k_update_fields_reverse<2><<<blocks_words(c, 0, c.g.nlev - 1), reverse_block(c), 0, c.stream>>>(c.g, c.cfg.prediction_radius, nm.wl_ref, nm.d_lo, nm.ref,
                                                                                              nm.cells, m.ref, m.cells, m.hc, r, r);
        }
        else
        {
            const RevAcc<FormCap<3>::value> r{lam_new, lam_old, overflow, 0};
            k_update_fields_reverse<3><<<blocks_words(c, 0, c.g.nlev - 1), reverse_block(c), 0, c.stream>>>(c.g, c.cfg.prediction_radius, nm.wl_ref, nm.d_lo, nm.ref,
                                                                                              nm.cells, m.ref, m.cells, m.hc, r, r);
        }
        launched(c, "update_fields");
        return check(c, "update_fields (transpose)");
    }

    namespace
    {
        // The whole adaptation (Adapt::operator(), mr/adapt.hpp:147-195) as one
        // captured graph: Harten pass i (at most max_level - min_level of them)
        // runs under a conditional node that holds while the previous pass
        // changed the mesh, and its second half (new mesh, update_fields) under
        // one that holds when this pass changed it; graduation iterates in a
        // conditional loop.  Pass i works on mesh buffer (cur + i) mod 2 and on
        // the field buffers that many swaps away, all known when capturing.
        struct StepTail
        {
            DeviceField* u;    // the adapted field (fs[0])
            DeviceField* unp1; // the upwind's output
            double a[3];
            double dt;
            int scheme;
        };

        int seq_adapt(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, double eps, double regularity,
                      const StepTail* tail = nullptr)
        {
            const int passes = c.cfg.max_level - c.cfg.min_level;
            std::vector<DeviceField> fa, oa; // the fields as they stand at each pass (buffers swapped per transition)
            for (DeviceField* f : fs)
            {
                fa.push_back(*f);
            }
            for (DeviceField* f : os)
            {
                oa.push_back(*f);
            }
            cudaMemsetAsync(c.d_adapt, 0, A_COUNT * sizeof(int), c.stream);
            k_adapt_words<<<1, 1, 0, c.stream>>>(c.d_adapt, A_GO, nullptr, 1, 0);
            launched(c, "adapt_words");
            int st = SG_OK;
            for (int i = 0; i < passes && !st; ++i)
            {
                const int cur = (c.cur + i) & 1;
                DeviceMesh& m  = c.mesh[cur];
                DeviceMesh& nm = c.mesh[1 - cur];
                std::vector<DeviceField*> fp, op;
                for (auto& f : fa)
                {
                    fp.push_back(&f);
                }
                for (auto& f : oa)
                {
                    op.push_back(&f);
                }
                PassSetup ps{};
                pass_thresholds(c, i, eps, regularity, ps.eps);
                ps.ite    = i;
                auto pass = [&]()
                {
                    int s1 = seq_front(c, m, nm, fp, &ps);
                    if (s1)
                    {
                        return s1;
                    }
                    k_adapt_words<<<1, 1, 0, c.stream>>>(c.d_adapt, A_PASSES, nullptr, i + 1, 0);
                    k_adapt_words<<<1, 1, 0, c.stream>>>(c.d_adapt, A_GO, c.d_flags + F_DIFFER, 0, 0);
                    launched(c, "adapt_words", 2);
                    return capture_if(c, c.d_flags + F_DIFFER,
                                      [&]()
                                      {
                                          int s2 = seq_back(c, m, nm, fp, op);
                                          if (c.rec_slots)
                                          {
                                              k_record_bits<<<grid_for(c.g.total_words), 256, 0, c.stream>>>(nm.cells, c.rec_slots, c.d_adapt,
                                                                                                              c.g.total_words);
                                              launched(c, "record_bits");
                                          }
                                          k_adapt_words<<<1, 1, 0, c.stream>>>(c.d_adapt, A_TRANS, nullptr, 1, 1);
                                          launched(c, "adapt_words");
                                          return s2;
                                      });
                };
                st = i == 0 ? pass() : capture_if(c, c.d_adapt + A_GO, pass);
                for (auto* list : {&fa, &oa})
                {
                    for (auto& f : *list)
                    {
                        std::swap(f.data, f.spare);
                    }
                }
            }
            if (!st && tail)
            {
                // the rest of the time step on the final mesh: the mesh buffer and the field's buffer depend on the
                // parity of the number of transitions, the ghost update on whether the last pass changed the mesh
                // (when it kept it, its own ghost update left the ghosts valid)
                k_step_flags<<<1, 1, 0, c.stream>>>(c.d_adapt);
                launched(c, "adapt_words");
                for (int par = 0; par < 2 && !st; ++par)
                {
                    const int cur    = (c.cur + par) & 1;
                    DeviceMesh& mf   = c.mesh[cur];
                    double* ud       = par ? tail->u->spare : tail->u->data;
                    const bool bc    = tail->u->has_bc;
                    const double bcv = tail->u->bc_value;
                    st               = capture_if(c, c.d_adapt + (par ? A_PAR1 : A_PAR0),
                                                  [&]()
                                                  {
                                                      int s1 = capture_if(c, c.d_adapt + A_NEEDG,
                                                                          [&]() { return ghost_value(c, mf, ud, bc, bcv); });
                                                      return s1 ? s1 : upwind_on(c, mf, ud, tail->unp1->data, tail->a, tail->dt, tail->scheme);
                                                  });
                }
            }
            if (!st)
            {
                cudaMemcpyAsync(c.h_adapt, c.d_adapt, A_COUNT * sizeof(int), cudaMemcpyDeviceToHost, c.stream);
            }
            return st ? st : check(c, "adaptation graph");
        }

        bool graph_applies(const Ctx& c)
        {
            return c.graphed_adapt && c.use_graphs && !c.timers.enabled && !c.trace.enabled && c.cfg.max_level != c.cfg.min_level;
        }

        // launches seq_adapt's graph (captured on first use) without waiting
        int adapt_graph_launch(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, double eps, double regularity,
                               bool relative_detail, const StepTail* tail)
        {
            if (c.cfg.ghost_width > 2)
            {
                c.err = "harten: ghost widths 1 and 2 are implemented";
                return SG_ERR_ARG;
            }
            if (int st = ensure_details(c, static_cast<int>(fs.size())))
            {
                return st;
            }
            c.rel_detail = relative_detail;
            std::vector<DeviceField*> all(fs);
            all.insert(all.end(), os.begin(), os.end());
            unsigned long long kind = 9ull | (relative_detail ? 16ull : 0ull) | (c.refine_boundary ? 256ull : 0ull)
                                      | (static_cast<unsigned long long>(fs.size()) << 20);
            unsigned long long thr  = bits_of(eps) * 0x9E3779B97F4A7C15ull ^ bits_of(regularity);
            unsigned long long bufs = fields_key(all, false) ^ (fields_key(all, true) << 1) ^ (ptr_key(c.rec_slots) * 0x9E3779B97F4A7C15ull);
            if (tail)
            {
                kind |= (static_cast<unsigned long long>(tail->scheme) + 1) << 10;
                bufs ^= ptr_key(tail->unp1->data) * 0xC2B2AE3D27D4EB4Full;
                for (double v : {tail->a[0], tail->a[1], tail->a[2], tail->dt})
                {
                    thr = (thr ^ bits_of(v)) * 0x100000001B3ull;
                }
            }
            return run_cached(c, kind, static_cast<unsigned long long>(c.cur), bufs, thr, [&]() { return seq_adapt(c, fs, os, eps, regularity, tail); });
        }

        // waits for a launched adaptation graph and applies its outcome on the host: the buffer swaps of the
        // transitions, the current mesh, ghost validity and the step's own swap
        int adapt_graph_finish(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, const StepTail* tail,
                               int* n_harten)
        {
            if (cudaStreamSynchronize(c.stream) != cudaSuccess)
            {
                return check(c, "adaptation sync");
            }
            std::vector<DeviceField*> all(fs);
            all.insert(all.end(), os.begin(), os.end());
            const int passes = c.h_adapt[A_PASSES], trans = c.h_adapt[A_TRANS];
            for (int t = 0; t < trans; ++t)
            {
                for (DeviceField* f : all)
                {
                    std::swap(f->data, f->spare);
                }
                c.cur = 1 - c.cur;
                ++c.mesh_version;
            }
            if (trans > 0)
            {
                c.mesh[0].host_valid = c.mesh[1].host_valid = false;
            }
            // the last pass's ghost update ran on the final mesh when that pass kept it
            for (DeviceField* f : all)
            {
                f->ghosts_valid = false;
            }
            if (passes > trans || tail)
            {
                // the last pass kept the mesh, or the step's tail updated the ghosts
                for (DeviceField* f : fs)
                {
                    f->ghosts_valid  = true;
                    f->ghost_version = c.mesh_version;
                }
            }
            if (tail)
            {
                // unp1 = u - dt * upwind(a, u) then std::swap(u.array(), unp1.array())
                std::swap(tail->u->data, tail->unp1->data);
                tail->u->ghosts_valid    = false;
                tail->unp1->ghosts_valid = false;
            }
            if (n_harten)
            {
                *n_harten = passes;
            }
            return device_error(c);
        }

        // the adaptation (and the rest of the step when tail is given) through
        // the graph; false when that path does not apply (graphs off, timers or
        // the kernel trace on)
        bool adapt_graphed(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, double eps, double regularity,
                           bool relative_detail, int* n_harten, int* status, const StepTail* tail = nullptr)
        {
            if (!graph_applies(c))
            {
                return false;
            }
            *status = adapt_graph_launch(c, fs, os, eps, regularity, relative_detail, tail);
            if (!*status)
            {
                *status = adapt_graph_finish(c, fs, os, tail, n_harten);
            }
            return true;
        }

        StepTail make_tail(const Ctx& c, DeviceField& u, DeviceField& unp1, const double* a, double dt, int scheme)
        {
            StepTail t{};
            t.u    = &u;
            t.unp1 = &unp1;
            for (int d = 0; d < c.g.dim; ++d)
            {
                t.a[d] = a[d];
            }
            t.dt     = dt;
            t.scheme = scheme;
            return t;
        }
    } // namespace

    bool step_graph_applies(const Ctx& c)
    {
        return graph_applies(c);
    }

    // the time step's graph in two halves (batched mode: launch every instance's, then wait for each);
    // step_launch returns SG_ERR_NOTFOUND when the graph path does not apply to this mesh
    int step_launch(Ctx& c, DeviceField& u, DeviceField& unp1, double eps, double regularity, const double* a, double dt, int scheme)
    {
        if (!graph_applies(c))
        {
            return SG_ERR_NOTFOUND;
        }
        const StepTail t = make_tail(c, u, unp1, a, dt, scheme);
        return adapt_graph_launch(c, {&u}, {}, eps, regularity, false, &t);
    }

    int step_finish(Ctx& c, DeviceField& u, DeviceField& unp1, int* n_harten)
    {
        const double zero[3] = {0., 0., 0.};
        const StepTail t     = make_tail(c, u, unp1, zero, 0., 0);
        return adapt_graph_finish(c, {&u}, {}, &t, n_harten);
    }

    // One iteration of the demo's time loop (demos/FiniteVolume/advection_2d.cpp:140-147): MRadaptation(eps,
    // regularity), update_ghost_mr(u), unp1 = u - dt * upwind(a, u) (or the flux form / README scheme),
    // std::swap(u.array(), unp1.array()) — one captured graph and one synchronisation when graphs apply,
    // otherwise the separate calls.
    int step(Ctx& c, DeviceField& u, DeviceField& unp1, double eps, double regularity, const double* a, double dt, int scheme, int* n_harten)
    {
        const StepTail t = make_tail(c, u, unp1, a, dt, scheme);
        int st           = SG_OK;
        {
            ScopedTimer timer(c, T_ADAPT);
            if (adapt_graphed(c, {&u}, {}, eps, regularity, false, n_harten, &st, &t))
            {
                return st;
            }
        }
        if ((st = adapt(c, u, eps, regularity, n_harten, false)) || (st = update_ghost_mr(c, u)) || (st = upwind(c, u, unp1, a, dt, scheme)))
        {
            return st;
        }
        std::swap(u.data, unp1.data);
        u.ghosts_valid    = false;
        unp1.ghosts_valid = false;
        return SG_OK;
    }

    // Adapt<Fields...>::operator()(mra_config, other_fields...) (mr/adapt.hpp:147-195)
    int adapt_fields(Ctx& c, const std::vector<DeviceField*>& fs, const std::vector<DeviceField*>& os, double eps, double regularity,
                     bool relative_detail, int* n_harten)
    {
        ScopedTimer timer(c, T_ADAPT);
        int gst = SG_OK;
        if (adapt_graphed(c, fs, os, eps, regularity, relative_detail, n_harten, &gst))
        {
            return gst;
        }
        const int minl = c.cfg.min_level, maxl = c.cfg.max_level;
        int it         = 0;
        bool conv      = false;
        for (int i = 0; minl != maxl && i < maxl - minl; ++i)
        {
            ++it;
            conv      = false;
            int st    = harten_begin_fields(c, fs, os, i, eps, regularity, relative_detail);
            if (!st)
            {
                st = harten_end_fields(c, fs, os, &conv);
            }
            if (st)
            {
                return st;
            }
            if (conv)
            {
                break;
            }
        }
        if (n_harten)
        {
            *n_harten = it;
        }
        return pass_error(c, conv);
    }

    // Adapt::operator() (mr/adapt.hpp:147-195)
    int adapt(Ctx& c, DeviceField& f, double eps, double regularity, int* n_harten, bool relative_detail)
    {
        ScopedTimer timer(c, T_ADAPT);
        int gst = SG_OK;
        if (adapt_graphed(c, {&f}, {}, eps, regularity, relative_detail, n_harten, &gst))
        {
            return gst;
        }
        const int minl = c.cfg.min_level, maxl = c.cfg.max_level;
        int it         = 0;
        bool conv      = false;
        if (minl != maxl)
        {
            for (int i = 0; i < maxl - minl; ++i)
            {
                ++it;
                conv      = false;
                int st    = harten(c, f, i, eps, regularity, &conv, relative_detail);
                if (st)
                {
                    return st;
                }
                if (conv)
                {
                    break;
                }
            }
        }
        if (n_harten)
        {
            *n_harten = it;
        }
        return pass_error(c, conv);
    }

    // the upwind step on mesh m from the values at ud into unp1d
    int upwind_on(Ctx& c, const DeviceMesh& m, const double* ud, double* unp1d, const double* a, double dt, int scheme)
    {
        const Geom& g = c.g;
        UpwindArgs p{};
        for (int d = 0; d < g.dim; ++d)
        {
            p.fl[d] = a[d] >= 0 ? a[d] : 0.;
            p.fr[d] = a[d] >= 0 ? 0. : a[d];
            p.zero_l[d] = p.fl[d] == 0.;
            p.zero_r[d] = p.fr[d] == 0.;
            p.ha[d] = .5 * a[d];
            p.hb[d] = .5 * std::fabs(a[d]);
        }
        p.dt     = dt;
        p.scheme = scheme;
        const int nb    = blocks_words(c, 0, g.nlev - 1);
        const int block = std::min(c.block, ITEM_BLOCK);
        if (scheme == 2)
        {
            if (g.dim == 2)
            {
                k_convection<2><<<nb, block, 0, c.stream>>>(c.g, m.wl_cells, m.d_lo, m.cells, ud, unp1d, p);
            }
            else
            {
                k_convection<3><<<nb, block, 0, c.stream>>>(c.g, m.wl_cells, m.d_lo, m.cells, ud, unp1d, p);
            }
        }
        else if (g.dim == 2)
        {
            k_upwind<2><<<nb, c.block, 0, c.stream>>>(c.g, m.wl_cells, m.d_lo, m.cells, ud, unp1d, p);
        }
        else
        {
            k_upwind<3><<<nb, c.block, 0, c.stream>>>(c.g, m.wl_cells, m.d_lo, m.cells, ud, unp1d, p);
        }
        launched(c, scheme == 2 ? "convection" : "upwind");
        return check(c, "upwind");
    }

    int upwind(Ctx& c, DeviceField& u, DeviceField& unp1, const double* a, double dt, int scheme)
    {
        ScopedTimer timer(c, T_UPWIND);
        return upwind_on(c, c.m(), u.data, unp1.data, a, dt, scheme);
    }
} // namespace sg
