// The phases of a step (sg_phase.cuh): device code, their kernels, and the
// sequences that launch them alone or chained.
#include <algorithm>
#include <cstring>
#include <utility>

#include "sg_phase_dev.cuh"

namespace sg
{
    namespace
    {
        // every reference word of mesh m: one thread per list entry
        template <class F>
        __device__ __forceinline__ void team_ref_words(const Env& E, const MeshPtrs& m, const Team& T, F f)
        {
            const long long b = m.lo[LO_REF], e = m.lo[LO_REF + E.g.nlev];
            for (long long i = b + T.tid; i < e; i += T.nthr)
            {
                f(m.wl_ref[i]);
            }
        }

        __device__ __forceinline__ void raise(int* flag)
        {
            if (*static_cast<volatile int*>(flag) == 0) // set once, read by many words
            {
                atomicOr(flag, 1);
            }
        }

        // ---------------------------------------------------------- pass begin
        // the threshold bitmaps of the reference words and the flags of the pass
        __device__ __forceinline__ void op_pass_begin(const Env& E, const Team& T)
        {
            if (T.tid < F_COUNT)
            {
                E.flags[T.tid] = 0;
            }
            if (E.setup_host)
            {
                for (int k = T.tid; k < 3 * MAXLEV; k += T.nthr)
                {
                    E.setup->eps[k] = E.setup_host->eps[k];
                }
                if (T.tid == 0)
                {
                    E.setup->ite = E.setup_host->ite;
                }
            }
            team_ref_words(E, E.m, T,
                           [&](int w)
                           {
                               E.above[w]     = 0u;
                               E.ref_above[w] = 0u;
                               E.par_above[w] = 0u;
                           });
        }

        // ---------------------------------------------------------- ghosts
        // One level of the top-down pass of update_ghost_mr
        // (algorithm/update_ghost_mr.hpp:206-222).  Within a level the
        // reference's operations touch disjoint cells and read only cells
        // finalised earlier, so they run side by side: corners and faces from
        // item b of nb threads, the projection onto level l-1 from warp0 of nwarps.
        template <int DIM, bool PDL>
        __device__ __forceinline__ void ghost_boundary(const Env& E, int l, int b, int nb)
        {
            const int per   = static_cast<int>(boundary_count<DIM>(E.g, l));
            const int total = per * E.nf;
            for (int t = b; t < total; t += nb)
            {
                int f = 0, k = t;
                while (k >= per)
                {
                    k -= per;
                    ++f;
                }
                boundary_item<DIM, PDL>(E.g, l, k, E.m, ValAcc{E.f[f].u}, E.f[f].has_bc != 0, E.f[f].bcv, 3);
            }
        }

        template <int DIM, bool PDL>
        __device__ __forceinline__ void ghost_project(const Env& E, int l, const Team& T)
        {
            project_items<PDL>(E.g, l, E.m, T, E.nf,
                          [&](long long w, int b, const Cell& c, int f)
                          {
                              double* u     = E.f[f].u;
                              u[32 * w + b] = project_one<DIM>(E.g, ValAcc{u}, l, c.x, c.y, c.z);
                          });
        }

        __device__ __forceinline__ int lowest_level(const Geom& g)
        {
            return g.min_level >= 2 ? g.min_level - 2 : 0; // no reference cell below min_level - 2
        }

        // in a chain: the boundary items go to the last blocks first, the projection to the first
        template <int DIM>
        __device__ __forceinline__ void op_ghost(const Env& E, int l, const Team& T)
        {
            const int back = T.nblocks - 1 - T.block; // whole warps stay together
            ghost_boundary<DIM, false>(E, l, back * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x), T.nthr);
            if (l > lowest_level(E.g))
            {
                ghost_project<DIM, false>(E, l, T);
            }
        }

        template <int DIM, bool PDL>
        __device__ __forceinline__ void op_predict(const Env& E, int l, const Team& T)
        {
            predict_items<PDL>(E.g, l, E.m, T, E.nf,
                          [&](long long w, int b, const Cell& c, int f)
                          {
                              double* u     = E.f[f].u;
                              u[32 * w + b] = predict_one<DIM>(E.g, ValAcc{u}, l, c.x, c.y, c.z, E.order);
                          });
        }

        // ---------------------------------------------------------- details
        // compute_relative_detail (mr/rel_detail.hpp:75-111), per field: max |u| over the leaf cells (the bits
        // of non-negative doubles order like the doubles, so an integer atomic max is exact and independent
        // of the order); the details are then multiplied by 1 / max (1 when max is below the machine epsilon)
        __device__ __forceinline__ void op_absmax_init(const Env& E, const Team& T)
        {
            if (T.tid < E.nf)
            {
                E.absmax[T.tid] = static_cast<unsigned long long>(__double_as_longlong(2.2250738585072014e-308)); // numeric_limits<double>::min()
            }
        }

        __device__ __forceinline__ void op_absmax(const Env& E, const Team& T)
        {
            const int lane    = threadIdx.x & 31;
            const long long b = E.m.lo[LO_CELLS], e = E.m.lo[LO_CELLS + E.g.nlev];
            for (int f = 0; f < E.nf; ++f)
            {
                unsigned long long best = 0;
                for (long long i = b + T.warp0(); i < e; i += T.nwarps())
                {
                    const long long w = E.m.wl_cells[i];
                    if ((E.m.cells[w] >> lane) & 1u)
                    {
                        const unsigned long long v = static_cast<unsigned long long>(__double_as_longlong(fabs(E.f[f].u[32 * w + lane])));
                        best                       = v > best ? v : best;
                    }
                }
                for (int o = 16; o > 0; o >>= 1)
                {
                    const unsigned long long x = __shfl_xor_sync(FULL_MASK, best, o);
                    best                       = x > best ? x : best;
                }
                if (lane == 0 && best)
                {
                    atomicMax(E.absmax + f, best);
                }
            }
        }

        // compute_detail_op (mr/operators.hpp:139-540) on
        // intersection(all_cells[l], union(cells[l+1], cells[l+2])).on(l), levels l0 .. min(l1, max_level - ite - 1)
        // (mr/adapt.hpp:310-317).  A detail is compared with the thresholds of the criteria
        // (mr/criteria.hpp:31-111) as it is formed, once per child instead of being read back by each of the
        // kernels that ask: bit e of `above` (coarsening, eps_l), of `ref_above` (refinement) and of
        // `par_above` (as the parent of level l + 1's cells), each the OR over the adapted fields.
        // Bound by the FP64 pipe: 3^DIM additions per child.
        template <int DIM>
        __device__ __forceinline__ void op_detail(const Env& E, int l0, int l1, const Team& T)
        {
            const Geom& g = E.g;
            const int ite = E.setup->ite;
            const int le  = min(l1, g.max_level - ite - 1);
            if (le < l0)
            {
                return;
            }
            const double* eps   = E.setup->eps;
            const uint32_t* ref = E.m.ref;
            const uint32_t* hc  = E.m.hc;
            const uint32_t* hc2 = E.m.hc2;
            block_items(
                E.m.wl_ref, static_cast<int>(E.m.lo[LO_REF + l0]), static_cast<int>(E.m.lo[LO_REF + le + 1]), T, E.nf,
                [&](int w) { return ref[w] & (hc[w] | hc2[w]); },
                [&](bool valid, int w_, int b, int f)
                {
                    if (!valid)
                    {
                        return;
                    }
                    const long long w = w_;
                    const int l   = level_down(g, w_, l0, le);
                    const Cell c  = cell_of(g, l, w, b);
                    const Box3 cb = box_at<DIM>(g, l + 1, 2 * c.x, 2 * c.y, 2 * c.z, 2);
                    const Box3 sb = E.order ? box_at<DIM>(g, l, c.x - 1, c.y - 1, c.z - 1, 3) : Box3{0, 0, 0};
                    const double t_above = eps[l + 1], t_ref = eps[MAXLEV + l + 1];
                    const double t_par   = l + 1 < g.max_level ? eps[2 * MAXLEV + l + 2] : 0.;
                    uint32_t fa = 0u, fr = 0u, fp = 0u; // one bit per child
                    {
                        const double* u = E.f[f].u;
                        double* det     = E.det + f * E.capacity;
                        double d[1 << DIM];
#pragma unroll
                        for (int ch = 0; ch < (1 << DIM); ++ch)
                        {
                            d[ch] = u[cb.base + (ch & 1) + ((ch >> 1) & 1) * cb.sy + ((ch >> 2) & 1) * cb.sz];
                        }
                        if (E.order == 0)
                        {
                            const double uc = u[32 * w + b];
#pragma unroll
                            for (int ch = 0; ch < (1 << DIM); ++ch)
                            {
                                d[ch] = d[ch] - uc;
                            }
                        }
                        else
                        {
                            // d -= cf * src with cf = prod interp1 = +-8^-k (k = axes with
                            // an off-centre tap): cf * src is +-(src * 8^-k) bit for bit
                            // (power-of-two scaling is exact), and d - (-m) is d + m, so
                            // one product per source serves all children
#pragma unroll
                            for (int sz = 0; sz < (DIM == 3 ? 3 : 1); ++sz)
                            {
#pragma unroll
                                for (int sy = 0; sy < 3; ++sy)
                                {
                                    const long long base = sb.base + sy * sb.sy + sz * sb.sz;
#pragma unroll
                                    for (int sx = 0; sx < 3; ++sx)
                                    {
                                        const double src = u[base + sx];
                                        const int k      = (sx != 1) + (sy != 1) + (DIM == 3 && sz != 1);
                                        const double m   = k == 0 ? src : scale8(src, k);
#pragma unroll
                                        for (int ch = 0; ch < (1 << DIM); ++ch)
                                        {
                                            // interp1(parity, t) < 0: t == 0 on odd children, t == 2 on even ones
                                            const int px = ch & 1, py = (ch >> 1) & 1, pz = (ch >> 2) & 1;
                                            const bool neg = ((sx == 0 && px) || (sx == 2 && !px)) ^ ((sy == 0 && py) || (sy == 2 && !py))
                                                             ^ (DIM == 3 && ((sz == 0 && pz) || (sz == 2 && !pz)));
                                            d[ch]          = neg ? d[ch] + m : d[ch] - m;
                                        }
                                    }
                                }
                            }
                        }
                        if (E.relative)
                        {
                            double mx = __longlong_as_double(static_cast<long long>(E.absmax[f]));
                            if (mx < 2.220446049250313e-16) // numeric_limits<double>::epsilon()
                            {
                                mx = 1.0;
                            }
                            const double inv = 1. / mx;
#pragma unroll
                            for (int ch = 0; ch < (1 << DIM); ++ch)
                            {
                                d[ch] = d[ch] * inv;
                            }
                        }
#pragma unroll
                        for (int ch = 0; ch < (1 << DIM); ++ch)
                        {
                            det[cb.base + (ch & 1) + ((ch >> 1) & 1) * cb.sy + ((ch >> 2) & 1) * cb.sz] = d[ch];
                            fa |= (fabs(d[ch]) > t_above ? 1u : 0u) << ch;
                            fr |= (fabs(d[ch]) > t_ref ? 1u : 0u) << ch;
                            fp |= (fabs(d[ch]) > t_par ? 1u : 0u) << ch;
                        }
                    }
                    // the pair of children of each row: two neighbouring bits of one word
#pragma unroll
                    for (int s = 0; s < (1 << (DIM - 1)); ++s)
                    {
                        const long long e = cb.base + (s & 1) * cb.sy + (s >> 1) * cb.sz;
                        const long long v = e >> 5;
                        const int bit     = static_cast<int>(e & 31);
                        const uint32_t a2 = (fa >> (2 * s)) & 3u, r2 = (fr >> (2 * s)) & 3u, p2 = (fp >> (2 * s)) & 3u;
                        if (a2)
                        {
                            atomicOr(E.above + v, a2 << bit);
                        }
                        if (r2)
                        {
                            atomicOr(E.ref_above + v, r2 << bit);
                        }
                        if (p2)
                        {
                            atomicOr(E.par_above + v, p2 << bit);
                        }
                    }
                });
        }

        // ---------------------------------------------------------- tags
        // mr_criteria_op (mr/criteria.hpp:20-113) on intersection(cells[l], all_cells[l-1]).on(l-1), fine levels
        // min_level .. max_level - ite (mr/adapt.hpp:325-339), and keep_boundary_refined (mr/adapt.hpp:245-274):
        // the tags of the 32 cells of a reference word from the threshold bits, one thread per word.
        //  - a leaf starts tagged keep;
        //  - the children of a parent that is not above its own threshold and has no child above theirs are
        //    tagged coarsen (only);
        //  - the cells above the refinement threshold are tagged refine.
        // Cells of the word outside the reference keep what an earlier pass left them, as they do in samurai's
        // numbering: a mesh read after it changed shows the last pass that knew the cell.
        template <int DIM>
        __device__ __forceinline__ void op_criteria(const Env& E, const Team& T)
        {
            const Geom& g = E.g;
            const int le  = g.max_level - E.setup->ite;
            team_ref_words(
                E, E.m, T,
                [&](int w)
                {
                    const int l = level_down(g, w, 0, g.max_level);
                    uint32_t k = E.m.cells[w], c = 0u, r = 0u, examined = 0u;
                    // what the word holds outside the reference, loaded here: behind the stores the loads would wait
                    // for each other
                    const uint32_t other = ~E.m.ref[w];
                    const uint32_t was_k = E.tk[w] & other, was_c = E.tc[w] & other, was_r = E.tr[w] & other, was_e = E.exam[w] & other;
                    if (l >= g.min_level && l <= le)
                    {
                        const Word p   = word_at<DIM>(g, l, w);
                        const Parent q = parent_of<DIM>(g, p);
                        if (q.w >= 0)
                        {
                            // the 16 parents of the word's cells
                            const uint32_t pref = E.m.ref[q.w], phc = E.m.hc[q.w];
                            const uint32_t par  = ((pref & phc) >> q.shift) & 0xFFFFu;
                            examined            = spread16((pref & (phc | E.m.hc2[q.w])) >> q.shift);
                            if (par)
                            {
                                if (l > g.min_level)
                                {
                                    // any child above: the word and its sibling rows
                                    const LevelGeom& L = g.lv[l];
                                    const int sib_y    = ((p.ry - PY) & 1) ? -L.W : L.W;
                                    uint32_t any       = E.above[w] | E.above[w + sib_y];
                                    if (DIM == 3)
                                    {
                                        const int sib_z = ((p.rz - PY) & 1) ? -L.W * L.R : L.W * L.R;
                                        any |= E.above[w + sib_z] | E.above[w + sib_z + sib_y];
                                    }
                                    const uint32_t quiet = par & ~(E.par_above[q.w] >> q.shift) & ~(compress_pairs(any, 0u) & 0xFFFFu);
                                    const uint32_t sel   = spread16(quiet);
                                    k &= ~sel;
                                    c |= sel;
                                }
                                if (l < g.max_level)
                                {
                                    r = E.ref_above[w] & spread16(par);
                                }
                            }
                        }
                    }
                    if (E.refine_boundary && l == g.max_level)
                    {
                        // the leaves of max_level within max_stencil_radius cells of the boundary are tagged keep
                        // (the tag is overwritten)
                        const uint32_t edge = E.m.cells[w] & ~box_bits<DIM>(g, word_at<DIM>(g, l, w), -E.radius, -E.radius);
                        k |= edge;
                        c &= ~edge;
                        r &= ~edge;
                    }
                    E.tk[w]   = was_k | k;
                    E.tc[w]   = was_c | c;
                    E.tr[w]   = was_r | r;
                    E.exam[w] = was_e | examined;
                });
        }

        // maximum_op (mr/operators.hpp:22-96), children at level l: a kept child keeps its siblings and its
        // parent; children all tagged coarsen make their parent keep; otherwise no child coarsens.  One thread
        // per parent word, whose child words no other thread touches.
        template <int DIM>
        __device__ __forceinline__ void op_maximum(const Env& E, int l, const Team& T)
        {
            team_words<DIM>(E.g, T, l - 1, l - 1,
                            [&](const Word& p)
                            {
                                const uint32_t m = E.m.ref[p.w] & E.m.hc[p.w];
                                if (!m)
                                {
                                    return;
                                }
                                constexpr int ROWS = 1 << (DIM - 1);
                                uint32_t klo = 0u, khi = 0u, clo = 0xFFFFFFFFu, chi = 0xFFFFFFFFu;
                                uint32_t kw[2 * ROWS], cw[2 * ROWS];
                                int at[2 * ROWS];
#pragma unroll
                                for (int s = 0; s < 2 * ROWS; ++s)
                                {
                                    at[s] = -1;
                                }
                                child_words<DIM>(E.g, p,
                                                 [&](int s, int a, int b)
                                                 {
                                                     at[2 * s]     = a;
                                                     at[2 * s + 1] = b;
                                                 });
#pragma unroll
                                for (int s = 0; s < 2 * ROWS; ++s)
                                {
                                    kw[s] = at[s] >= 0 ? E.tk[at[s]] : 0u;
                                    cw[s] = at[s] >= 0 ? E.tc[at[s]] : 0u;
                                    if (s & 1)
                                    {
                                        khi |= kw[s];
                                        chi &= cw[s];
                                    }
                                    else
                                    {
                                        klo |= kw[s];
                                        clo &= cw[s];
                                    }
                                }
                                const uint32_t keep = m & compress_pairs(klo, khi);
                                const uint32_t allc = m & ~compress_pairs(~clo, ~chi);
                                const uint32_t none = m & ~keep & ~allc;
                                const uint32_t pk   = keep | allc;
                                if (pk)
                                {
                                    E.tk[p.w] |= pk;
                                }
#pragma unroll
                                for (int s = 0; s < 2 * ROWS; ++s)
                                {
                                    const uint32_t kk = spread16((s & 1) ? keep >> 16 : keep), nn = spread16((s & 1) ? none >> 16 : none);
                                    if (kk & ~kw[s])
                                    {
                                        E.tk[at[s]] = kw[s] | kk;
                                    }
                                    if (nn & cw[s])
                                    {
                                        E.tc[at[s]] = cw[s] & ~nn;
                                    }
                                }
                            });
        }

        // update_cell_array_from_tag (algorithm/graduation.hpp:743-842): leaves tagged refine are replaced by
        // their children, leaves tagged coarsen and not keep by their parent (at the even child)
        template <int DIM>
        __device__ __forceinline__ void op_new_cells(const Env& E, const Team& T)
        {
            const Geom& g         = E.g;
            const uint32_t* cells = E.m.cells;
            auto refined          = [&](int w, int l) { return l < g.max_level && cells[w] ? cells[w] & E.tr[w] : 0u; };
            auto coarsened        = [&](int w, int l)
            {
                const uint32_t c = l > g.min_level ? cells[w] : 0u;
                return c ? c & E.tc[w] & ~E.tk[w] & ~(l < g.max_level ? E.tr[w] : 0u) : 0u;
            };
            // the union of the next mesh starts empty
            for (int w = T.tid; w < static_cast<int>(g.total_words); w += T.nthr)
            {
                E.n.uni[w] = 0u;
            }
            team_words<DIM>(g, T, g.min_level, g.max_level,
                            [&](const Word& p)
                            {
                                uint32_t v = cells[p.w];
                                if (v)
                                {
                                    v = v & ~refined(p.w, p.l) & ~coarsened(p.w, p.l);
                                }
                                if (p.l > g.min_level)
                                {
                                    const Parent q = parent_of<DIM>(g, p);
                                    if (q.w >= 0)
                                    {
                                        v |= spread16(refined(q.w, p.l - 1) >> q.shift);
                                    }
                                }
                                if (p.l < g.max_level && E.m.hc[p.w])
                                {
                                    // parent of the coarsened (even) child: the first child row only, and only
                                    // under cells with a leaf child
                                    const LevelGeom& F = g.lv[p.l + 1];
                                    const int fy = 2 * p.ry - PY, fz = 2 * p.rz - PY;
                                    if (fy >= 0 && fy < F.R && (DIM == 2 || (fz >= 0 && fz < F.R)))
                                    {
                                        const int k = 2 * p.wi - 1, base = row_base<DIM>(F, fy, fz);
                                        const uint32_t lo = k >= 0 && k < F.W ? coarsened(base + k, p.l + 1) : 0u;
                                        const uint32_t hi = k + 1 < F.W ? coarsened(base + k + 1, p.l + 1) : 0u;
                                        if (lo | hi)
                                        {
                                            v |= compress_even(lo, hi);
                                        }
                                    }
                                }
                                E.n.cells[p.w] = v;
                            });
        }

        // ---------------------------------------------------------- graduation
        // One pass of make_graduation (algorithm/graduation.hpp:573-726, 245-330): the cells of level l that lie
        // under the (2*grad_width)-expansion of a leaf cell two or more levels finer are refined.
        // A pass that finds nothing leaves the cells unchanged.
        //  1. t0 = cells[l+1].on(l), and the marks (t2) cleared
        template <int DIM>
        __device__ __forceinline__ void op_grad_coarsen(const Env& E, const Team& T)
        {
            const Geom& g  = E.g;
            const int dlo = g.min_level, dtop = g.max_level - 2;
            team_words<DIM>(g, T, dlo, dtop + 1,
                            [&](const Word& p)
                            {
                                if (p.l > dlo)
                                {
                                    E.t0[p.w] = coarsen<DIM>(g, E.n.cells, p);
                                }
                                if (p.l <= dtop)
                                {
                                    E.t2[p.w] = 0u;
                                }
                            });
        }

        //  2. the expansion e of t0 marks its ancestors in t2: d[l] = (e[l+1] | d[l+1]).on(l)
        //     (graduation.hpp:628-723) is the set of the cells with a cell of e among their descendants.
        //     dilate_2gw(cells[l+1]).on(l) is computed as dilate_gw(cells[l+1].on(l)): per axis the parents of
        //     [a - 2gw, b + 2gw] are [a/2 - gw, b/2 + gw], so both give the same set, and the dilation then
        //     runs on the coarser level.
        template <int DIM>
        __device__ __forceinline__ void grad_mark(const Env& E, const Word& p, uint32_t e)
        {
            if (e)
            {
                const Parent q = parent_of<DIM>(E.g, p);
                if (q.w >= 0)
                {
                    const uint32_t bits = (compress_pairs(e, 0u) & 0xFFFFu) << q.shift;
                    if ((E.t2[q.w] & bits) != bits && (atomicOr(E.t2 + q.w, bits) & bits) != bits)
                    {
                        const Word pw{p.l - 1, q.w, q.ry, q.rz, q.wi};
                        const WordLoc at = loc_of<DIM>(E.g, pw);
                        mark_ancestors(E.g, E.t2, p.l - 1, at.row, at.wi, bits, E.g.min_level);
                    }
                }
            }
        }

        template <int DIM>
        __device__ __forceinline__ void op_grad_expand(const Env& E, const Team& T, int part)
        {
            const Geom& g  = E.g;
            const int elo = g.min_level + 1, ehi = g.max_level - 1;
            team_words<DIM>(g, T, elo, ehi,
                            [&](const Word& p)
                            {
                                const bool live = live_row<DIM>(g, p);
                                if (part == OP_GRAD_EXPAND_XY)
                                {
                                    E.t3[p.w] = live ? dilate_xy<DIM>(g, E.t0, p, E.grad_width) : 0u;
                                    return;
                                }
                                uint32_t e = 0u;
                                if (live)
                                {
                                    e = part == OP_GRAD_EXPAND_Z ? dilate_z(g, E.t3, p, E.grad_width) : dilate_xy<DIM>(g, E.t0, p, E.grad_width);
                                }
                                if (g.periodic)
                                {
                                    E.t1[p.w] = e;
                                }
                                else
                                {
                                    grad_mark<DIM>(E, p, e);
                                }
                            });
        }

        // with periodic axes the finer cells also act through their translates (graduation.hpp:309-318): the
        // expansion gains its translates within the domain (translation commutes with the dilation and with
        // on(), so the chain below carries them down)
        template <int DIM>
        __device__ __forceinline__ void op_grad_periodic(const Env& E, const Team& T)
        {
            const Geom& g = E.g;
            team_words<DIM>(g, T, g.min_level + 1, g.max_level - 1,
                            [&](const Word& p)
                            {
                                const WordLoc at = loc_of<DIM>(g, p);
                                E.t0[p.w] = E.t1[p.w] | (periodic_translates(g, E.t1, p.l, at.row, at.wi) & box_mask(g, p.l, at.row, at.wi, 0, 0));
                            });
        }

        // d[l] = (e[l+1] | d[l+1]).on(l) level by level (periodic axes)
        template <int DIM>
        __device__ __forceinline__ void op_grad_down(const Env& E, int l, int slot, const Team& T)
        {
            const Geom& g = E.g;
            team_words<DIM>(g, T, l, l,
                            [&](const Word& p)
                            {
                                const uint32_t dv = coarsen<DIM>(g, E.t0, p) | (l + 1 <= g.max_level - 2 ? coarsen<DIM>(g, E.t2, p) : 0u);
                                E.t2[p.w]         = dv;
                                const uint32_t rv = dv & E.n.cells[p.w];
                                E.t3[p.w]         = rv;
                                if (rv)
                                {
                                    raise(E.flags + slot);
                                }
                            });
        }

        // list_interval_to_refine_for_contiguous_boundary_cells for a max_stencil_radius of 2
        // (algorithm/graduation.hpp:370-497): in each non-periodic Cartesian direction t, a leaf P of level lc is
        // refined when a leaf b of level lc + 1 on the boundary the direction points to has b - 2 t among P's
        // children, i.e. P sits at coordinate n - 2 (t = +e) or 1 (t = -e) along the axis and one of its children's
        // neighbours across the boundary layer is a leaf.  The bits of word p to refine.
        template <int DIM>
        __device__ __forceinline__ uint32_t contiguous_boundary(const Geom& g, const uint32_t* nc, const Word& p)
        {
            const uint32_t v = nc[p.w];
            if (!v)
            {
                return 0u;
            }
            const LevelGeom& C = g.lv[p.l];
            const LevelGeom& F = g.lv[p.l + 1];
            const int y = p.ry - PY, z = DIM == 3 ? p.rz - PY : 0;
            const int x0   = 32 * p.wi - PX;
            const int nz   = DIM == 3 ? 2 : 1;
            uint32_t out   = 0u;
            auto fine_word = [&](int fy, int fz, int k) -> uint32_t
            {
                const int ry = fy + PY, rz = fz + PY;
                if (ry < 0 || ry >= F.R || (DIM == 3 && (rz < 0 || rz >= F.R)) || k < 0 || k >= F.W)
                {
                    return 0u;
                }
                return nc[row_base<DIM>(F, ry, rz) + k];
            };
            for (int d = 0; d < DIM; ++d)
            {
                if ((g.periodic >> d) & 1)
                {
                    continue;
                }
                for (int sgn = 1; sgn >= -1; sgn -= 2)
                {
                    const int q  = sgn > 0 ? C.n - 2 : 1; // coordinate of P along d
                    const int bf = sgn > 0 ? F.n - 1 : 0; // coordinate of b along d
                    if (d == 0)
                    {
                        const int bit = q - x0;
                        if (bit < 0 || bit >= 32 || !((v >> bit) & 1u))
                        {
                            continue;
                        }
                        const int xb = bf + PX;
                        bool hit     = false;
                        for (int sz = 0; sz < nz && !hit; ++sz)
                        {
                            for (int sy = 0; sy < 2 && !hit; ++sy)
                            {
                                hit = (fine_word(2 * y + sy, 2 * z + sz, xb >> 5) >> (xb & 31)) & 1u;
                            }
                        }
                        out |= hit ? (1u << bit) : 0u;
                    }
                    else
                    {
                        if ((d == 1 ? y : z) != q)
                        {
                            continue;
                        }
                        // the fine boundary row (or plane) under the word's cells: any of a cell's two x children
                        for (int s2 = 0; s2 < nz; ++s2)
                        {
                            const int fy = d == 1 ? bf : 2 * y + s2;
                            const int fz = d == 1 ? 2 * z + s2 : bf;
                            out |= compress_pairs(fine_word(fy, fz, 2 * p.wi - 1), fine_word(fy, fz, 2 * p.wi));
                        }
                    }
                }
            }
            return out & v;
        }

        //  3. t3 = the leaves to refine
        template <int DIM>
        __device__ __forceinline__ void op_grad_refine(const Env& E, int l0, int l1, int slot, const Team& T)
        {
            const Geom& g = E.g;
            const int dt  = g.max_level - 2;
            team_words<DIM>(g, T, l0, l1,
                            [&](const Word& p)
                            {
                                uint32_t rv = 0u;
                                if (p.l <= dt)
                                {
                                    rv = g.periodic ? E.t3[p.w] : (E.n.cells[p.w] & E.t2[p.w]);
                                }
                                if (E.radius == 2)
                                {
                                    rv |= contiguous_boundary<DIM>(g, E.n.cells, p);
                                }
                                E.t3[p.w] = rv;
                                if (rv)
                                {
                                    raise(E.flags + slot);
                                }
                            });
        }

        //  4. refined: levels l0 .. l1 change, t3 holds flags on l0 .. l1 - 1
        template <int DIM>
        __device__ __forceinline__ void op_grad_apply(const Env& E, int l0, int l1, const Team& T)
        {
            const Geom& g = E.g;
            uint32_t* nc  = E.n.cells;
            team_words<DIM>(g, T, l0, l1,
                            [&](const Word& p)
                            {
                                const uint32_t r = p.l < l1 ? E.t3[p.w] : 0u;
                                uint32_t add     = 0u;
                                if (p.l > l0)
                                {
                                    const Parent q = parent_of<DIM>(g, p);
                                    add            = q.w >= 0 ? spread16(E.t3[q.w] >> q.shift) : 0u;
                                }
                                if (r | add)
                                {
                                    nc[p.w] = (nc[p.w] & ~r) | add;
                                }
                            });
        }

        template <int DIM>
        __device__ __forceinline__ void op_compare(const Env& E, const Team& T)
        {
            const int begin = static_cast<int>(E.g.lv[E.g.min_level].woff), end = static_cast<int>(E.g.total_words);
            bool differ     = false;
#pragma unroll 4
            for (int w = begin + T.tid; w < end; w += T.nthr)
            {
                differ |= E.n.cells[w] != E.m.cells[w];
            }
            if (differ)
            {
                raise(E.flags + F_DIFFER);
            }
            if (!E.report)
            {
                return;
            }
            // the last block leaves the flags and the mesh's error word with the host, and settles the flag that a
            // second half queued ahead hangs on
            __shared__ bool last;
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0)
            {
                last = atomicAdd(E.flags + F_DONE, 1) == T.nblocks - 1;
            }
            __syncthreads();
            if (last && threadIdx.x < F_COUNT)
            {
                __threadfence();
                const int k = static_cast<int>(threadIdx.x);
                const int v = *static_cast<volatile int*>(k == F_ERR ? E.g.err : E.flags + k);
                constexpr unsigned SLOTS = (1u << F_COUNT) - 1u;
                const bool differ = __shfl_sync(SLOTS, v, F_DIFFER) != 0, final = __shfl_sync(SLOTS, v, F_GRAD1) == 0;
                if (k == F_AHEAD)
                {
                    E.flags[F_AHEAD] = differ && final;
                }
                E.report[k] = v;
            }
        }

        constexpr int SCAN_CHUNK = SCAN_WORDS;

        struct Pair
        {
            unsigned long long pop; // cells: reference in the low, leaves in the high 32 bits
            unsigned long long nz;  // non-empty words, likewise
        };

        __device__ __forceinline__ Pair warp_sum(Pair v)
        {
            for (int o = 16; o > 0; o >>= 1)
            {
                v.pop += __shfl_xor_sync(FULL_MASK, v.pop, o);
                v.nz += __shfl_xor_sync(FULL_MASK, v.nz, o);
            }
            return v;
        }

        __device__ __forceinline__ Pair word_counts(uint32_t r, uint32_t c)
        {
            return {static_cast<unsigned long long>(__popc(r)) | (static_cast<unsigned long long>(__popc(c)) << 32),
                    static_cast<unsigned long long>(r != 0u) | (static_cast<unsigned long long>(c != 0u) << 32)};
        }

        // sums of SCAN_GROUP chunks follow those of the chunks
        constexpr int SCAN_GROUP = 64;

        __device__ __forceinline__ int scan_chunks(const Geom& g)
        {
            return (static_cast<int>(g.total_words) + SCAN_CHUNK - 1) / SCAN_CHUNK;
        }

        __device__ __forceinline__ void add_sums(const Env& E, int ch, const Pair& t)
        {
            unsigned long long* sums = reinterpret_cast<unsigned long long*>(E.block_sums);
            const int chunks         = scan_chunks(E.g);
            atomicAdd(sums + 2 * ch, t.pop);
            atomicAdd(sums + 2 * ch + 1, t.nz);
            if (chunks > SCAN_GROUP) // nobody asks for the only group's
            {
                const int grp = chunks + ch / SCAN_GROUP;
                atomicAdd(sums + 2 * grp, t.pop);
                atomicAdd(sums + 2 * grp + 1, t.nz);
            }
        }

        // ---------------------------------------------------------- mesh construction
        __device__ __forceinline__ void op_clear_union(const Env& E, const Team& T)
        {
            for (int w = T.tid; w < static_cast<int>(E.g.total_words); w += T.nthr)
            {
                E.n.uni[w] = 0u;
            }
        }

        // hc = cells[l+1].on(l) (levels min-1 .. max-1: cells with a leaf child), the union's marks
        // (construct_union, mesh.hpp:1231-1262: every cell with a leaf among its descendants), and the expansion
        // of the cells by the stencil radius (cells_and_ghosts, levels min .. max; in 3D its xy part)
        template <int DIM>
        __device__ __forceinline__ void op_hc_cag(const Env& E, const Team& T)
        {
            const Geom& g  = E.g;
            const int minl = g.min_level, maxl = g.max_level;
            const int hlo  = max(minl - 1, 0), hhi = maxl - 1;
            uint32_t* cxy  = DIM == 2 ? E.n.cag : E.t0;
            const int chunks = scan_chunks(g);
            for (int k = T.tid; k < 2 * (chunks + (chunks + SCAN_GROUP - 1) / SCAN_GROUP); k += T.nthr)
            {
                E.block_sums[k] = 0; // the scan's totals
            }
            team_words<DIM>(g, T, min(hlo, minl), maxl,
                            [&](const Word& p)
                            {
                                if (p.l >= hlo && p.l <= hhi)
                                {
                                    const uint32_t h = coarsen<DIM>(g, E.n.cells, p);
                                    E.n.hc[p.w]      = h;
                                    if (h && (atomicOr(E.n.uni + p.w, h) & h) != h)
                                    {
                                        const WordLoc at = loc_of<DIM>(g, p);
                                        mark_ancestors(g, E.n.uni, p.l, at.row, at.wi, h, 0);
                                    }
                                }
                                if (p.l >= minl)
                                {
                                    cxy[p.w] = live_row<DIM>(g, p) ? dilate_xy<DIM>(g, E.n.cells, p, E.radius) : 0u;
                                }
                            });
        }

        // hc2 = hc.on(l) (cells with a leaf grandchild, levels min-2 .. max-2) with, in 2D, t1 =
        // cells_and_ghosts.on(l) (min-1 .. max-1) and, in 3D, the z part of cells_and_ghosts
        template <int DIM>
        __device__ __forceinline__ void op_hc2_cag(const Env& E, int l0, int l1, const Team& T)
        {
            const Geom& g  = E.g;
            const int minl = g.min_level, maxl = g.max_level;
            const int h2lo = max(minl - 2, 0), h2hi = maxl - 2;
            const int t1lo = max(minl - 1, 0), t1hi = maxl - 1;
            const bool multi = maxl != minl;
            team_words<DIM>(g, T, l0, l1,
                            [&](const Word& p)
                            {
                                if (p.l >= h2lo && p.l <= h2hi)
                                {
                                    E.n.hc2[p.w] = coarsen<DIM>(g, E.n.hc, p);
                                }
                                if (DIM == 2)
                                {
                                    if (multi && p.l >= t1lo && p.l <= t1hi)
                                    {
                                        E.t1[p.w] = coarsen<DIM>(g, E.n.cag, p);
                                    }
                                }
                                else if (p.l >= minl)
                                {
                                    E.n.cag[p.w] = live_row<DIM>(g, p) ? dilate_z(g, E.t0, p, E.radius) : 0u;
                                }
                            });
        }

        template <int DIM>
        __device__ __forceinline__ void op_cag_on(const Env& E, int l0, int l1, const Team& T)
        {
            team_words<DIM>(E.g, T, l0, l1, [&](const Word& p) { E.t1[p.w] = coarsen<DIM>(E.g, E.n.cag, p); });
        }

        // The reference before the children of the projection cells (mr/mesh.hpp:222-455): cells_and_ghosts,
        // the prediction ghosts cells_and_ghosts[l+1].on(l) expanded by p within the expanded domain and
        // cells[l+2].on(l) expanded by p, into scratch (rf) or, with periodic axes, the reference itself
        template <int DIM>
        __device__ __forceinline__ void op_ref0(const Env& E, const Team& T, int part)
        {
            const Geom& g  = E.g;
            const int minl = g.min_level, maxl = g.max_level;
            const int h2lo = max(minl - 2, 0), h2hi = maxl - 2;
            const int t1lo = max(minl - 1, 0), t1hi = maxl - 1;
            const int pr   = E.order; // prediction radius
            uint32_t* ref0 = g.periodic ? E.n.ref : E.rf;
            team_words<DIM>(g, T, lowest_level(g), maxl,
                            [&](const Word& p)
                            {
                                const bool live = live_row<DIM>(g, p);
                                const bool in1 = live && p.l >= t1lo && p.l <= t1hi, in2 = live && p.l >= h2lo && p.l <= h2hi;
                                if (part == OP_REF0_XY)
                                {
                                    E.t2[p.w] = in1 ? dilate_xy<DIM>(g, E.t1, p, pr) : 0u;
                                    E.t3[p.w] = in2 ? dilate_xy<DIM>(g, E.n.hc2, p, pr) : 0u;
                                    return;
                                }
                                uint32_t v = E.n.cag[p.w];
                                uint32_t a = 0u;
                                if (in1)
                                {
                                    a = DIM == 2 ? dilate_xy<DIM>(g, E.t1, p, pr) : dilate_z(g, E.t2, p, pr);
                                    if (a)
                                    {
                                        v |= a & box_bits<DIM>(g, p, pr, pr);
                                    }
                                }
                                uint32_t b = 0u;
                                if (in2)
                                {
                                    b = DIM == 2 ? dilate_xy<DIM>(g, E.n.hc2, p, pr) : dilate_z(g, E.t3, p, pr);
                                }
                                ref0[p.w] = v | b;
                            });
        }

        // periodic parts of the reference (mr/mesh.hpp:294-317, 356-368): the translates of cells_and_ghosts
        // within the domain expanded by the stencil radius, and those of the two prediction-ghost sets (written
        // in full into scratch first) within the domain; translate commutes with on() and the dilations
        template <int DIM>
        __device__ __forceinline__ void op_ref_periodic_src(const Env& E, const Team& T)
        {
            const Geom& g  = E.g;
            const int t1lo = max(g.min_level - 1, 0), t1hi = g.max_level - 1;
            team_words<DIM>(g, T, lowest_level(g), g.max_level,
                            [&](const Word& p)
                            {
                                const bool live = live_row<DIM>(g, p);
                                if (DIM == 2)
                                {
                                    E.t0[p.w] = live && p.l >= t1lo && p.l <= t1hi ? dilate_xy<DIM>(g, E.t1, p, E.order) : 0u;
                                    E.t2[p.w] = live ? dilate_xy<DIM>(g, E.n.hc2, p, E.order) : 0u;
                                }
                                else
                                {
                                    E.t0[p.w] = live ? dilate_z(g, E.t2, p, E.order) : 0u;
                                    E.t1[p.w] = live ? dilate_z(g, E.t3, p, E.order) : 0u;
                                }
                            });
        }

        template <int DIM>
        __device__ __forceinline__ void op_ref_periodic(const Env& E, const Team& T)
        {
            const Geom& g      = E.g;
            const bool multi   = g.max_level != g.min_level;
            const uint32_t* pb = DIM == 2 ? E.t2 : E.t1;
            team_words<DIM>(g, T, multi ? lowest_level(g) : g.min_level, g.max_level,
                            [&](const Word& p)
                            {
                                const WordLoc at = loc_of<DIM>(g, p);
                                uint32_t v       = multi ? E.n.ref[p.w] : E.n.cag[p.w];
                                if (p.l >= g.min_level)
                                {
                                    v |= periodic_translates(g, E.n.cag, p.l, at.row, at.wi) & box_mask(g, p.l, at.row, at.wi, E.radius, E.radius);
                                }
                                if (multi)
                                {
                                    v |= (periodic_translates(g, E.t0, p.l, at.row, at.wi) | periodic_translates(g, pb, p.l, at.row, at.wi))
                                         & box_mask(g, p.l, at.row, at.wi, 0, 0);
                                }
                                E.n.ref[p.w] = v;
                            });
        }

        // Children of the projection cells: reference[l+1] |= (reference[l] & union[l]) refined, in one pass
        // instead of level by level: the parent of a union cell is a union cell, so a cell whose parent p is in
        // the union joins the reference exactly when p or one of p's ancestors (down to the reference's first
        // level) is in ref0; and proj = reference & union.  Most words have no parent in the union, and the walk
        // up stops as soon as every candidate parent has been found.
        template <int DIM>
        __device__ __forceinline__ void op_ref_children(const Env& E, int l0, int l1, const Team& T)
        {
            const Geom& g      = E.g;
            const uint32_t* r0 = E.rf;
            team_words<DIM>(g, T, l0, l1,
                            [&](const Word& p)
                            {
                                uint32_t v = r0[p.w];
                                if (p.l > l0)
                                {
                                    const Parent q = parent_of<DIM>(g, p);
                                    if (q.w >= 0)
                                    {
                                        const uint32_t cand = (E.n.uni[q.w] >> q.shift) & 0xFFFFu;
                                        if (cand)
                                        {
                                            uint32_t got = (r0[q.w] >> q.shift) & cand; // parents themselves in ref0
                                            // ancestors of the 16 parents at level l - 1 - k: 16 >> k cells of one word
                                            const int y = p.ry - PY, z = p.rz - PY, x0 = 32 * p.wi - PX;
                                            for (int k = 1; p.l - 1 - k >= l0 && got != cand; ++k)
                                            {
                                                const LevelGeom& A = g.lv[p.l - 1 - k];
                                                const int ry = (y >> (k + 1)) + PY, rz = DIM == 3 ? (z >> (k + 1)) + PY : PY;
                                                if (ry < 0 || ry >= A.R || (DIM == 3 && (rz < 0 || rz >= A.R)))
                                                {
                                                    continue;
                                                }
                                                const int pos       = (x0 >> (k + 1)) + PX;
                                                const uint32_t word = r0[row_base<DIM>(A, ry, rz) + (pos >> 5)] >> (pos & 31);
                                                uint32_t bits;
                                                if (k >= 4)
                                                {
                                                    bits = (word & 1u) ? 0xFFFFu : 0u;
                                                }
                                                else
                                                {
                                                    bits = word & ((1u << (16 >> k)) - 1u);
                                                    for (int s = 0; s < k; ++s)
                                                    {
                                                        bits = spread16(bits);
                                                    }
                                                }
                                                got |= bits & cand;
                                            }
                                            v |= spread16(got);
                                        }
                                    }
                                }
                                E.n.ref[p.w] = v;
                                if (p.l < g.max_level)
                                {
                                    E.n.proj[p.w] = v ? v & E.n.uni[p.w] : 0u;
                                }
                                // the scan's totals of the word's chunk, a leaf word being a reference word
                                const unsigned lanes = __activemask();
                                if (__any_sync(lanes, v != 0u))
                                {
                                    const int ch    = p.w / SCAN_CHUNK;
                                    const Pair t    = word_counts(v, v ? E.n.cells[p.w] : 0u);
                                    const int first = __ffs(lanes) - 1;
                                    if (lanes == FULL_MASK && __all_sync(lanes, ch == __shfl_sync(lanes, ch, first)))
                                    {
                                        const Pair sum = warp_sum(t);
                                        if ((threadIdx.x & 31) == 0)
                                        {
                                            add_sums(E, ch, sum);
                                        }
                                    }
                                    else if (v)
                                    {
                                        add_sums(E, ch, t);
                                    }
                                }
                            });
        }

        // the same level by level (periodic axes: their translates enter between the levels); level l from l-1
        template <int DIM>
        __device__ __forceinline__ void op_ref_children_level(const Env& E, int l, const Team& T)
        {
            const Geom& g = E.g;
            team_words<DIM>(g, T, l, l,
                            [&](const Word& p)
                            {
                                const Parent q = parent_of<DIM>(g, p);
                                if (q.w < 0)
                                {
                                    return;
                                }
                                const uint32_t pc = E.n.ref[q.w] & E.n.uni[q.w];
                                // proj_cells of the coarse level, final now; the fine words of one coarse word
                                // all write this same value
                                E.n.proj[q.w]      = pc;
                                const uint32_t add = spread16(pc >> q.shift);
                                if (add)
                                {
                                    E.n.ref[p.w] |= add;
                                }
                            });
        }

        // a mesh of one level: no coarser reference, no projection
        __device__ __forceinline__ void op_single_level(const Env& E, const Team& T)
        {
            for (int w = T.tid; w < static_cast<int>(E.g.total_words); w += T.nthr)
            {
                E.n.ref[w]  = E.n.cag[w];
                E.n.proj[w] = 0u;
            }
        }

        // ---------------------------------------------------------- scan
        // Rank (exclusive popcount prefix of the reference), the lists of the non-empty reference and leaf words
        // and the counters, in two phases over chunks of SCAN_CHUNK words: the chunks' totals, then each chunk
        // adds up the totals before it and writes its words, 32 consecutive words per warp and step (every load
        // and store coalesced).
        // the block's sum of v, on every thread
        __device__ __forceinline__ Pair block_sum(Pair v)
        {
            __shared__ Pair part[32];
            v = warp_sum(v);
            __syncthreads();
            if ((threadIdx.x & 31) == 0)
            {
                part[threadIdx.x >> 5] = v;
            }
            __syncthreads();
            Pair t{0, 0};
            for (int k = 0; k < static_cast<int>(blockDim.x >> 5); ++k)
            {
                t.pop += part[k].pop;
                t.nz += part[k].nz;
            }
            return t;
        }

        __device__ __forceinline__ void op_scan_sums(const Env& E)
        {
            const int n  = static_cast<int>(E.g.total_words);
            const int nc = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
            for (int ch = blockIdx.x; ch < nc; ch += gridDim.x)
            {
                Pair v{0, 0};
                for (int w = ch * SCAN_CHUNK + threadIdx.x; w < min(n, (ch + 1) * SCAN_CHUNK); w += blockDim.x)
                {
                    const Pair t = word_counts(E.n.ref[w], E.n.cells[w]);
                    v.pop += t.pop;
                    v.nz += t.nz;
                }
                const Pair t = block_sum(v);
                if (threadIdx.x == 0)
                {
                    add_sums(E, ch, t);
                }
            }
        }

        // Also the prediction ghosts of every word (update_ghost_mr.hpp:224-233): reference cells inside the
        // box that are neither leaves nor projections and have a parent in the reference.
        template <int DIM>
        __device__ __forceinline__ void op_scan_write(const Env& E)
        {
            const Geom& g      = E.g;
            const MeshPtrs& M  = E.n;
            const int n        = static_cast<int>(g.total_words);
            const int nc       = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
            const int lane     = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
            const int per_warp = SCAN_CHUNK / nwarp; // a multiple of 32: blocks of at most SCAN_CHUNK threads, a power of two
            __shared__ Pair tot[32];
            for (int ch = blockIdx.x; ch < nc; ch += gridDim.x)
            {
                // whole groups before the chunk's, then the chunks of its group
                Pair before{0, 0};
                const int grp = ch / SCAN_GROUP;
                for (int k = threadIdx.x; k < grp + ch - grp * SCAN_GROUP; k += blockDim.x)
                {
                    const int at = k < grp ? nc + k : grp * SCAN_GROUP + (k - grp);
                    before.pop += static_cast<unsigned long long>(E.block_sums[2 * at]);
                    before.nz += static_cast<unsigned long long>(E.block_sums[2 * at + 1]);
                }
                before            = block_sum(before);
                const Pair prefix = before;
                const int w0 = ch * SCAN_CHUNK + warp * per_warp;
                Pair mine{0, 0};
                for (int w = w0 + lane; w < min(n, w0 + per_warp); w += 32)
                {
                    const Pair t = word_counts(M.ref[w], M.cells[w]);
                    mine.pop += t.pop;
                    mine.nz += t.nz;
                }
                mine = warp_sum(mine);
                __syncthreads();
                if (lane == 0)
                {
                    tot[warp] = mine;
                }
                __syncthreads();
                for (int k = 0; k < warp; ++k)
                {
                    before.pop += tot[k].pop;
                    before.nz += tot[k].nz;
                }
                for (int s = w0; s < min(n, w0 + per_warp); s += 32)
                {
                    const int w       = s + lane;
                    const bool in     = w < n;
                    const uint32_t r  = in ? M.ref[w] : 0u, c = in ? M.cells[w] : 0u;
                    const uint32_t br = __ballot_sync(FULL_MASK, r != 0u), bc = __ballot_sync(FULL_MASK, c != 0u);
                    const int l       = in ? level_down(g, w, 0, g.max_level) : 0;
                    if ((br | bc) == 0u)
                    {
                        // 32 empty words (most of a 3D mesh): no cell is looked up in them, so no rank
                        if (in)
                        {
                            M.pred[w] = 0u;
                            if (w == static_cast<int>(g.lv[l].woff))
                            {
                                M.lo[LO_REF + l]   = static_cast<unsigned>(before.nz);
                                M.lo[LO_CELLS + l] = static_cast<unsigned>(before.nz >> 32);
                            }
                        }
                        continue;
                    }
                    const Pair t      = word_counts(r, c);
                    unsigned pr       = static_cast<unsigned>(t.pop); // inclusive prefix of the reference cells
                    for (int o = 1; o < 32; o <<= 1)
                    {
                        const unsigned x = __shfl_up_sync(FULL_MASK, pr, o);
                        pr += lane >= o ? x : 0u;
                    }
                    const uint32_t lower = (1u << lane) - 1u;
                    const unsigned ir = static_cast<unsigned>(before.nz) + __popc(br & lower);
                    const unsigned ic = static_cast<unsigned>(before.nz >> 32) + __popc(bc & lower);
                    if (in)
                    {
                        M.rank[w] = static_cast<int>(static_cast<unsigned>(before.pop) + pr - static_cast<unsigned>(t.pop));
                        if (r)
                        {
                            M.wl_ref[ir] = w;
                        }
                        if (c)
                        {
                            M.wl_cells[ic] = w;
                        }
                        uint32_t pd = r & ~c;
                        pd          = pd ? pd & ~M.proj[w] : 0u;
                        if (pd)
                        {
                            const Word p = word_at<DIM>(g, l, w);
                            pd &= box_bits<DIM>(g, p, 0, 0);
                            if (pd)
                            {
                                const Parent q = l >= 1 ? parent_of<DIM>(g, p) : Parent{-1, 0, 0, 0, 0};
                                pd             = q.w >= 0 ? pd & spread16(M.ref[q.w] >> q.shift) : 0u;
                            }
                        }
                        M.pred[w] = pd;
                        if (w == static_cast<int>(g.lv[l].woff))
                        {
                            M.lo[LO_REF + l]   = ir;
                            M.lo[LO_CELLS + l] = ic;
                        }
                    }
                    before.pop += static_cast<unsigned long long>(__shfl_sync(FULL_MASK, pr, 31));
                    before.nz += static_cast<unsigned long long>(__popc(br)) | (static_cast<unsigned long long>(__popc(bc)) << 32);
                    // leaf cells are counted at the end only
                }
                if (ch == nc - 1)
                {
                    const Pair all = block_sum(mine);
                    if (threadIdx.x == 0)
                    {
                        // mine is per warp and the same on its lanes: all sums each warp 32 times
                        const unsigned long long pop = prefix.pop + all.pop / 32, nz = prefix.nz + all.nz / 32;
                        M.lo[0]                 = static_cast<long long>(pop & 0xFFFFFFFFull);
                        M.lo[1]                 = static_cast<long long>(nz & 0xFFFFFFFFull);
                        M.lo[2]                 = static_cast<long long>(pop >> 32);
                        M.lo[3]                 = static_cast<long long>(nz >> 32);
                        M.lo[LO_REF + g.nlev]   = M.lo[1];
                        M.lo[LO_CELLS + g.nlev] = M.lo[3];
                        for (int k = 0; k < 4; ++k)
                        {
                            M.host_lo[k] = M.lo[k];
                        }
                    }
                }
            }
        }

        // ---------------------------------------------------------- fields
        // update_fields (algorithm/update_fields.hpp:27-127): copy on
        // reference & new cells, projection on coarsened cells, prediction on
        // refined cells; every other reference entry of the new field is 0.
        template <int DIM>
        __device__ __forceinline__ void op_update_fields(const Env& E, const Team& T)
        {
            const Geom& g = E.g;
            block_items(E.n.wl_ref, static_cast<int>(E.n.lo[LO_REF]), static_cast<int>(E.n.lo[LO_REF + g.nlev]), T, E.nf, [&](int w) { return E.n.ref[w]; },
                        [&](bool valid, int w, int b, int f)
                        {
                            if (!valid)
                            {
                                return;
                            }
                            const long long e    = 32LL * w + b;
                            const uint32_t cells = E.n.cells[w], hc = E.m.hc[w], ref = E.m.ref[w];
                            const ValAcc uo{E.f[f].u};
                            double v = 0.;
                            if ((cells >> b) & 1u)
                            {
                                const int l  = level_down(g, w, 0, g.max_level);
                                const Cell c = cell_of(g, l, w, b);
                                if ((hc >> b) & 1u)
                                {
                                    v = project_one<DIM>(g, uo, l + 1, c.x, c.y, c.z);
                                }
                                else if (l >= 1 && test(E.m.cells, g, l - 1, c.x >> 1, c.y >> 1, c.z >> 1))
                                {
                                    v = predict_one<DIM>(g, uo, l, c.x, c.y, c.z, E.order);
                                }
                                else if ((ref >> b) & 1u)
                                {
                                    v = uo.get(e);
                                }
                            }
                            E.f[f].un[e] = v;
                        });
        }

        // ---------------------------------------------------------- periodic axes
        // iterate_over_periodic_ghosts (algorithm/update_periodic.hpp:27-140) on
        // axis d, one side: side 0 pairs the ghosts of [n, n + gw) with [0, gw),
        // side 1 those of [-gw, 0) with [n - gw, n); the other axes span
        // [-gw, n + gw).  Only pairs of two reference cells count.  Work item t
        // of the side: gw * (n + 2 gw)^(dim-1) of them.
        __device__ __forceinline__ bool periodic_pair(const Geom& g, int l, int d, int side, unsigned t, const uint32_t* ref, Pos* pg, Pos* pi)
        {
            const int n = g.lv[l].n, gw = g.ghost_width; // 1 or 2
            const int on     = (side == 0 ? n : -gw) + static_cast<int>(gw == 2 ? t & 1u : 0u);
            const unsigned r = gw == 2 ? t >> 1 : t;
            const unsigned span = static_cast<unsigned>(n + 2 * gw);
            const unsigned hi   = g.dim == 3 ? r / span : 0u;
            const int a = static_cast<int>(r - hi * span) - gw, b = static_cast<int>(hi) - gw; // the other axes, in order
            const int x = d == 0 ? on : a, y = d == 1 ? on : (d == 0 ? a : b), z = g.dim == 3 ? (d == 2 ? on : b) : 0;
            const int back = side == 0 ? -n : n;
            *pg = pos_of(g, l, x, y, z);
            *pi = pos_of(g, l, x + (d == 0 ? back : 0), y + (d == 1 ? back : 0), z + (d == 2 ? back : 0));
            const bool rg = test(ref, *pg), ri = test(ref, *pi);
            return rg && ri;
        }

        __host__ __device__ inline long long periodic_side_items(const Geom& g, int l)
        {
            const long long span = g.lv[l].n + 2 * g.ghost_width;
            return g.ghost_width * (g.dim == 2 ? span : span * span);
        }

        // update_ghost_periodic(level, field) (algorithm/update_periodic.hpp:19-25)
        // on one axis: both sides at once (they read inner cells and write
        // outer ghosts, so no item reads what another writes)
        __device__ __forceinline__ void op_periodic_copy(const Env& E, int l, int d, const Team& T)
        {
            const unsigned per = static_cast<unsigned>(periodic_side_items(E.g, l));
            for (unsigned t = T.tid; t < 2 * per; t += T.nthr)
            {
                const int side = t >= per ? 1 : 0;
                Pos pg, pi;
                if (periodic_pair(E.g, l, d, side, t - side * per, E.m.ref, &pg, &pi))
                {
                    for (int f = 0; f < E.nf; ++f)
                    {
                        E.f[f].u[elem(pg)] = E.f[f].u[elem(pi)];
                    }
                }
            }
        }

        // update_tag_periodic(level, tag) (algorithm/update_periodic.hpp:178-300)
        // on one axis: both cells of a pair take the union of their tags, side after side.  The two sides touch
        // different cells where the box is at least two ghost widths wide and then run together (sides 3).
        __device__ __forceinline__ void op_periodic_tag(const Env& E, int l, int d, int sides, const Team& T)
        {
            const unsigned per = static_cast<unsigned>(periodic_side_items(E.g, l));
            for (unsigned t = T.tid; t < (sides == 3 ? 2 * per : per); t += T.nthr)
            {
                const int side = sides == 3 ? (t >= per ? 1 : 0) : sides - 1;
                Pos pg, pi;
                if (!periodic_pair(E.g, l, d, side, t >= per ? t - per : t, E.m.ref, &pg, &pi))
                {
                    continue;
                }
                for (uint32_t* bm : {E.tk, E.tc, E.tr})
                {
                    const bool a = (bm[pg.w] >> pg.b) & 1u, b = (bm[pi.w] >> pi.b) & 1u;
                    if (a && !b)
                    {
                        atomicOr(bm + pi.w, 1u << pi.b);
                    }
                    else if (b && !a)
                    {
                        atomicOr(bm + pg.w, 1u << pg.b);
                    }
                }
            }
        }

        // ---------------------------------------------------------- dispatch
        template <int DIM, int OP, bool PDL>
        __device__ __forceinline__ void run_op(const Env& E, const Phase& p, const Team& T)
        {
            const int slot = p.aux & 7;
            if constexpr (OP == OP_PASS_BEGIN) op_pass_begin(E, T);
            if constexpr (OP == OP_GHOST) op_ghost<DIM>(E, p.l0, T);
            if constexpr (OP == OP_PREDICT) op_predict<DIM, PDL>(E, p.l0, T);
            if constexpr (OP == OP_ABSMAX_INIT) op_absmax_init(E, T);
            if constexpr (OP == OP_ABSMAX) op_absmax(E, T);
            if constexpr (OP == OP_DETAIL) op_detail<DIM>(E, p.l0, p.l1, T);
            if constexpr (OP == OP_CRITERIA) op_criteria<DIM>(E, T);
            if constexpr (OP == OP_MAXIMUM) op_maximum<DIM>(E, p.l0, T);
            if constexpr (OP == OP_NEW_CELLS) op_new_cells<DIM>(E, T);
            if constexpr (OP == OP_GRAD_COARSEN) op_grad_coarsen<DIM>(E, T);
            if constexpr (OP == OP_GRAD_EXPAND || OP == OP_GRAD_EXPAND_XY || OP == OP_GRAD_EXPAND_Z) op_grad_expand<DIM>(E, T, OP);
            if constexpr (OP == OP_GRAD_PERIODIC) op_grad_periodic<DIM>(E, T);
            if constexpr (OP == OP_GRAD_DOWN) op_grad_down<DIM>(E, p.l0, slot, T);
            if constexpr (OP == OP_GRAD_REFINE) op_grad_refine<DIM>(E, p.l0, p.l1, slot, T);
            if constexpr (OP == OP_GRAD_APPLY) op_grad_apply<DIM>(E, p.l0, p.l1, T);
            if constexpr (OP == OP_COMPARE) op_compare<DIM>(E, T);
            if constexpr (OP == OP_CLEAR_UNION) op_clear_union(E, T);
            if constexpr (OP == OP_HC_CAG) op_hc_cag<DIM>(E, T);
            if constexpr (OP == OP_HC2_CAG) op_hc2_cag<DIM>(E, p.l0, p.l1, T);
            if constexpr (OP == OP_CAG_ON) op_cag_on<DIM>(E, p.l0, p.l1, T);
            if constexpr (OP == OP_REF0 || OP == OP_REF0_XY || OP == OP_REF0_Z) op_ref0<DIM>(E, T, OP);
            if constexpr (OP == OP_REF_PERIODIC_SRC) op_ref_periodic_src<DIM>(E, T);
            if constexpr (OP == OP_REF_PERIODIC) op_ref_periodic<DIM>(E, T);
            if constexpr (OP == OP_REF_CHILDREN) op_ref_children<DIM>(E, p.l0, p.l1, T);
            if constexpr (OP == OP_REF_CHILDREN_LEVEL) op_ref_children_level<DIM>(E, p.l0, T);
            if constexpr (OP == OP_SINGLE_LEVEL) op_single_level(E, T);
            if constexpr (OP == OP_SCAN_SUMS) op_scan_sums(E);
            if constexpr (OP == OP_SCAN_WRITE) op_scan_write<DIM>(E);
            if constexpr (OP == OP_UPDATE_FIELDS) op_update_fields<DIM>(E, T);
            if constexpr (OP == OP_PERIODIC_COPY) op_periodic_copy(E, p.l0, p.aux, T);
            if constexpr (OP == OP_PERIODIC_TAG) op_periodic_tag(E, p.l0, p.aux >> 2, p.aux & 3, T);
        }

        // graduation phases may hang on a flag of an earlier one (bits 3.. of aux: its slot + 1)
        __device__ __forceinline__ bool guarded_off(const Env& E, const Phase& p)
        {
            if (p.op < OP_GRAD_COARSEN || p.op > OP_GRAD_APPLY)
            {
                return false;
            }
            const int guard = p.aux >> 3;
            return guard != 0 && E.flags[guard - 1] == 0; // one line of L1 per SM: settled before the launch or the last barrier
        }

        template <int DIM, int OP>
        __global__ void k_phase(const __grid_constant__ Env E, const __grid_constant__ Phase p)
        {
            // Launches are programmatic dependents of each other: the next one's blocks come in while this one runs and
            // wait for its end.  A level of the ghost update that follows another (FOLLOWS) goes further: it reads
            // nothing but the mesh's bitmaps until its items are handed out, and waits just before the first value.
            // It may also let its successor in before its own wait, since a first level has waited for whatever
            // wrote the bitmaps before it let anyone in.
            constexpr bool LEVEL = OP == OP_GHOST || OP == OP_PREDICT;
            if (!LEVEL || !(p.aux & FOLLOWS))
            {
                dependency_wait<true>();
            }
            asm volatile("griddepcontrol.launch_dependents;");
            if ((OP >= OP_GRAD_COARSEN && OP <= OP_GRAD_APPLY && guarded_off(E, p)))
            {
                return;
            }
            if (E.guard)
            {
                if (LEVEL)
                {
                    dependency_wait<true>(); // the flag may be older than the bitmaps, but never let a block end unwaited
                }
                if (*E.guard == 0)
                {
                    return;
                }
            }
            if constexpr (OP == OP_GHOST)
            {
                // the first l1 blocks take the boundary, the others the projection
                const int nb = p.l1;
                if (static_cast<int>(blockIdx.x) < nb)
                {
                    ghost_boundary<DIM, true>(E, p.l0, static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x), nb * static_cast<int>(blockDim.x));
                }
                else
                {
                    ghost_project<DIM, true>(E, p.l0, grid_team(nb));
                }
            }
            else
            {
                run_op<DIM, OP, true>(E, p, grid_team());
            }
            if constexpr (OP == OP_GHOST || OP == OP_PREDICT)
            {
                dependency_wait<true>(); // a block without items must not end before the launch it follows
            }
        }

        template <class... Params, class... Args>
        void launch_dependent(Ctx& c, bool overlap, void (*kernel)(Params...), int grid, int block, int cluster, Args&&... args)
        {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim  = dim3(static_cast<unsigned>(grid));
            cfg.blockDim = dim3(static_cast<unsigned>(block));
            cfg.stream   = c.stream;
            cudaLaunchAttribute at[2] = {};
            if (cluster > 1)
            {
                at[cfg.numAttrs].id               = cudaLaunchAttributeClusterDimension;
                at[cfg.numAttrs].val.clusterDim.x = static_cast<unsigned>(cluster);
                at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
                ++cfg.numAttrs;
            }
            // not inside conditional bodies, nor where the kernel trace puts an event after every launch
            if (overlap && c.overlap_launches && c.cap_depth == 0 && !c.trace.enabled)
            {
                at[cfg.numAttrs].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
                at[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
                ++cfg.numAttrs;
            }
            cfg.attrs = at;
            cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...); // the caller checks the last error
        }

        template <int DIM, int OP>
        void launch_one(Ctx& c, const Env& e, const Phase& p, int grid, int block)
        {
            // The field phases over all levels stay behind a full boundary: their waiting blocks would hold the
            // shared memory and registers that the launch before them still wants (three components, 2D levels 3
            // to 9, relative details: 379 us a step without them, 470 with them overlapped too).
            constexpr bool overlap = OP != OP_DETAIL && OP != OP_UPDATE_FIELDS && OP != OP_ABSMAX && OP != OP_ABSMAX_INIT;
            launch_dependent(c, overlap, k_phase<DIM, OP>, grid, block, 1, e, p);
        }

        // ---------------------------------------------------------- chain
        // PERIODIC: the phases of meshes with periodic axes too (a chain fetches its instructions as it goes: the
        // other meshes' kernel leaves them out)
        template <int DIM, bool PERIODIC>
        __device__ __forceinline__ void run_any(const Env& E, const Phase& p, const Team& T)
        {
            if constexpr (PERIODIC)
            {
                switch (p.op)
                {
#define SG_OP(op)                        \
    case op:                             \
        run_op<DIM, op, false>(E, p, T); \
        return;
                    SG_OP(OP_GRAD_PERIODIC)
                    SG_OP(OP_GRAD_DOWN)
                    SG_OP(OP_REF_PERIODIC_SRC)
                    SG_OP(OP_REF_PERIODIC)
                    SG_OP(OP_REF_CHILDREN_LEVEL)
                    SG_OP(OP_PERIODIC_COPY)
                    SG_OP(OP_PERIODIC_TAG)
#undef SG_OP
                    default: break;
                }
            }
            switch (p.op)
            {
#define SG_OP(op)                    \
    case op:                         \
        run_op<DIM, op, false>(E, p, T); \
        break;
                SG_OP(OP_PASS_BEGIN)
                SG_OP(OP_GHOST)
                SG_OP(OP_PREDICT)
                SG_OP(OP_ABSMAX_INIT)
                SG_OP(OP_ABSMAX)
                SG_OP(OP_DETAIL)
                SG_OP(OP_CRITERIA)
                SG_OP(OP_MAXIMUM)
                SG_OP(OP_NEW_CELLS)
                SG_OP(OP_GRAD_COARSEN)
                SG_OP(OP_GRAD_EXPAND)
                SG_OP(OP_GRAD_EXPAND_XY)
                SG_OP(OP_GRAD_EXPAND_Z)
                SG_OP(OP_GRAD_REFINE)
                SG_OP(OP_GRAD_APPLY)
                SG_OP(OP_COMPARE)
                SG_OP(OP_CLEAR_UNION)
                SG_OP(OP_HC_CAG)
                SG_OP(OP_HC2_CAG)
                SG_OP(OP_CAG_ON)
                SG_OP(OP_REF0)
                SG_OP(OP_REF0_XY)
                SG_OP(OP_REF0_Z)
                SG_OP(OP_REF_CHILDREN)
                SG_OP(OP_SINGLE_LEVEL)
                SG_OP(OP_SCAN_SUMS)
                SG_OP(OP_SCAN_WRITE)
                SG_OP(OP_UPDATE_FIELDS)
#undef SG_OP
                default: break;
            }
        }

        // Consecutive small phases in one launch of one thread-block cluster, a
        // hardware cluster barrier between them.  A phase of a small level is
        // bound by latency: its few dependent loads and what separates it from
        // the next.  As graph nodes the phases measure 2.4 to 6.7 us each on a
        // mesh of 8 levels (device time, warm), of which 0.9 us is the boundary
        // between two nodes and most of the rest launch, cold instructions and
        // ramp-up; a cluster barrier takes 0.25 us (16 blocks of 512 threads),
        // a barrier over the whole grid 1.3 us.  Levels of the ghost update chain
        // only where periodic exchanges stand between them, or in batches whose
        // launches do not overlap: as overlapping launches of their own they take
        // less (2D levels 2 to 8: 256 -> 217 us a step).  A cluster barrier that has to
        // wait for the blocks' stores takes 0.8 us, though, and every load after it
        // comes from L2 (0.2 us).  With periodic axes the exchanges between the
        // levels double the phases, most of them nearly empty: there the phases of
        // the smallest levels run in the first block alone, block barriers between
        // them, and only the end of such a run is a cluster barrier (2D levels 3 to
        // 9: 566 -> 522 us a step when it came in; without periodic axes the lone block loses what
        // the barriers save).
        template <int DIM, bool PERIODIC>
        __global__ void __launch_bounds__(CHAIN_THREADS, 1) k_chain(const __grid_constant__ Env Ep, const __grid_constant__ PhaseList L)
        {
            dependency_wait<true>();
            asm volatile("griddepcontrol.launch_dependents;");
            // the environment is read at every step of every phase: from shared memory, not from parameter
            // lines that each block would fetch one miss after the other
            __shared__ __align__(16) unsigned char store[sizeof(Env)];
            {
                const int* src = reinterpret_cast<const int*>(&Ep);
                for (int k = threadIdx.x; k < static_cast<int>(sizeof(Env) / sizeof(int)); k += blockDim.x)
                {
                    reinterpret_cast<int*>(store)[k] = src[k];
                }
                __syncthreads();
            }
            const Env& E = *reinterpret_cast<const Env*>(store);
            if (E.guard && *E.guard == 0)
            {
                return; // the whole cluster: the flag was settled before the launch
            }
            const Team all  = grid_team();
            const Team solo = {static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x), 0, 1};
            for (int i = 0; i < L.n; ++i)
            {
                Phase p          = L.p[i];
                const bool alone = PERIODIC && (p.op & PHASE_SOLO) != 0;
                if (PERIODIC)
                {
                    p.op &= static_cast<short>(~PHASE_SOLO);
                }
                if (guarded_off(E, p))
                {
                    continue; // the same on every thread: the flag was settled before the last barrier
                }
                if (!alone || blockIdx.x == 0)
                {
                    run_any<DIM, PERIODIC>(E, p, alone ? solo : all);
                }
                if (alone)
                {
                    __syncthreads();
                    if (i + 1 < L.n && (L.p[i + 1].op & PHASE_SOLO) != 0)
                    {
                        continue; // the other blocks wait at the end of the run
                    }
                }
                __syncwarp();
                asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
            }
        }

        using LaunchFn = void (*)(Ctx&, const Env&, const Phase&, int, int);

        template <int DIM, int... OPS>
        const LaunchFn* launch_table(std::integer_sequence<int, OPS...>)
        {
            static const LaunchFn table[] = {launch_one<DIM, OPS>...};
            return table;
        }

        const char* const OP_NAMES[OP_COUNT] = {
            "pass_begin",     "ghost_level",  "predict",       "absmax_init",  "absmax",       "detail",       "criteria",   "maximum",
            "new_cells",      "grad_coarsen", "grad_expand",   "grad_expand_xy", "grad_expand_z", "grad_periodic", "grad_down", "grad_refine",
            "grad_apply",     "compare",      "clear_union",   "hc_cag",       "hc2_cag",      "cag_on",       "ref0",       "ref0_xy",
            "ref0_z",         "ref_periodic_src", "ref_periodic", "ref_children", "ref_children", "single_level", "scan_sums",
            "scan_write",     "update_fields", "periodic_copy", "periodic_tag"};

        enum class Shape
        {
            WORDS, // a thread per bitmap word
            LIST,  // a thread per reference word
            ITEMS, // blocks that hand out the cells of their words
            SCAN,
            OTHER
        };

        Shape shape_of(int op)
        {
            switch (op)
            {
                case OP_PASS_BEGIN:
                case OP_CRITERIA: return Shape::LIST;
                case OP_GHOST:
                case OP_PREDICT:
                case OP_ABSMAX:
                case OP_DETAIL:
                case OP_UPDATE_FIELDS: return Shape::ITEMS;
                case OP_SCAN_SUMS:
                case OP_SCAN_WRITE: return Shape::SCAN;
                case OP_ABSMAX_INIT:
                case OP_PERIODIC_COPY:
                case OP_PERIODIC_TAG: return Shape::OTHER;
                default: return Shape::WORDS;
            }
        }

        long long range_words(const Geom& g, int l0, int l1)
        {
            return l1 < l0 ? 0 : g.lv[l1].woff + g.lv[l1].nwords - g.lv[l0].woff;
        }
    } // namespace

    const char* phase_name(int op)
    {
        return OP_NAMES[op];
    }

    // the bitmap words a phase walks
    long long phase_words(const Geom& g, const Phase& p)
    {
        switch (p.op)
        {
            case OP_GHOST: return range_words(g, std::max(p.l0 - 1, 0), p.l0);
            case OP_PREDICT:
            case OP_PERIODIC_COPY:
            case OP_PERIODIC_TAG:
            case OP_GRAD_DOWN:
            case OP_REF_CHILDREN_LEVEL: return range_words(g, p.l0, p.l0);
            case OP_MAXIMUM: return range_words(g, p.l0 - 1, p.l0 - 1);
            case OP_ABSMAX_INIT: return 1;
            default: return g.total_words;
        }
    }

    int launch_phase_alone(Ctx& c, const Env& e, const Phase& ph)
    {
        const Geom& g = c.g;
        Phase p       = ph;
        int block     = 256;
        long long grid = 1;
        // blocks that hand out the items of `words` words: a block per 16 words, at most max_blocks blocks of 256 threads
        auto items = [&](long long words)
        {
            block               = std::min(c.block, ITEM_BLOCK);
            const long long cap = std::max(1LL, c.max_blocks * 256 / block);
            return std::min(cap, std::max(1LL, (words + 15) / 16));
        };
        switch (shape_of(p.op))
        {
            case Shape::WORDS:
            {
                long long words = g.total_words;
                if (p.l0 <= p.l1 && p.l1 > 0)
                {
                    words = range_words(g, p.l0, p.l1);
                }
                if (p.op == OP_MAXIMUM)
                {
                    words = phase_words(g, p);
                }
                // the comparison's blocks sign off one by one at a counter (level 9 in 3D: 4864 of them took 27 us, 609 take 14)
                grid = std::min((p.op == OP_COMPARE ? c.max_blocks / 2 + 1 : 4LL * c.max_blocks), (words + block - 1) / block);
                break;
            }
            case Shape::LIST:
                // the list holds the non-empty words, far fewer than all
                grid = std::min(c.max_blocks, (g.total_words + block - 1) / block);
                break;
            case Shape::ITEMS:
                if (p.op == OP_GHOST)
                {
                    const long long nproj = p.l0 > (g.min_level >= 2 ? g.min_level - 2 : 0) ? items(g.lv[p.l0 - 1].nwords) : 0;
                    block                 = std::min(c.block, ITEM_BLOCK);
                    const long long edge  = (g.dim == 2 ? boundary_count<2>(g, p.l0) : boundary_count<3>(g, p.l0)) * e.nf;
                    const long long nb    = std::min(16384LL, (edge + block - 1) / block);
                    p.l1                  = static_cast<short>(nb);
                    grid                  = nb + nproj;
                }
                else if (p.op == OP_PREDICT)
                {
                    grid = items(g.lv[p.l0].nwords);
                }
                else
                {
                    grid = items(p.l0 <= p.l1 && p.l1 > 0 ? range_words(g, p.l0, p.l1) : g.total_words);
                }
                break;
            case Shape::SCAN: grid = (g.total_words + SCAN_WORDS - 1) / SCAN_WORDS; break;
            case Shape::OTHER:
                grid = p.op == OP_ABSMAX_INIT ? 1 : (2 * periodic_side_items(g, p.l0) + block - 1) / block;
                break;
        }
        if (grid < 1)
        {
            return SG_OK;
        }
        const auto ops        = std::make_integer_sequence<int, OP_COUNT>{};
        const LaunchFn* table = g.dim == 2 ? launch_table<2>(ops) : launch_table<3>(ops);
        table[p.op](c, e, p, static_cast<int>(grid), block);
        launched(c, phase_name(p.op));
        return check(c, phase_name(p.op));
    }

    namespace
    {
        auto chain_kernel(const Geom& g)
        {
            return g.dim == 2 ? (g.periodic ? k_chain<2, true> : k_chain<2, false>) : (g.periodic ? k_chain<3, true> : k_chain<3, false>);
        }
    } // namespace

    // The largest cluster a chain may use on this device: 16 blocks where the
    // device grants that (above the portable 8), 0 where it grants none.
    int chain_blocks(const Geom& g)
    {
        const void* k = reinterpret_cast<const void*>(chain_kernel(g));
        const bool big = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        cudaGetLastError();
        for (int n = big ? 16 : 8; n >= 2; n /= 2)
        {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim  = dim3(static_cast<unsigned>(n));
            cfg.blockDim = dim3(CHAIN_THREADS);
            cudaLaunchAttribute at{};
            at.id               = cudaLaunchAttributeClusterDimension;
            at.val.clusterDim.x = static_cast<unsigned>(n);
            at.val.clusterDim.y = at.val.clusterDim.z = 1;
            cfg.attrs    = &at;
            cfg.numAttrs = 1;
            int active   = 0;
            if (cudaOccupancyMaxActiveClusters(&active, k, &cfg) == cudaSuccess && active > 0)
            {
                return n;
            }
            cudaGetLastError();
        }
        return 0;
    }

    namespace
    {
        int launch_chain(Ctx& c, const Env& e, const std::vector<Phase>& ps)
        {
            PhaseList list{};
            list.n = static_cast<int>(ps.size());
            std::copy(ps.begin(), ps.end(), list.p);
            launch_dependent(c, true, chain_kernel(c.g), c.chain_blocks, CHAIN_THREADS, c.chain_blocks, e, list);
            launched(c, "chain");
            return check(c, "chain");
        }
    } // namespace

    // ------------------------------------------------------------ sequences
    MeshPtrs mesh_ptrs(const DeviceMesh& m)
    {
        return {m.cells, m.cag, m.proj, m.uni, m.ref, m.hc, m.hc2, m.pred, m.rank, m.wl_ref, m.wl_cells, m.d_lo, m.h_lo};
    }

    Sequence::Sequence(Ctx& ctx, const DeviceMesh& m, const DeviceMesh& n)
        : c(ctx)
    {
        std::memset(&env, 0, sizeof(env));
        env.g               = c.g;
        env.m               = mesh_ptrs(m);
        env.n               = mesh_ptrs(n);
        env.t0              = c.t0;
        env.t1              = c.t1;
        env.t2              = c.t2;
        env.t3              = c.t3;
        env.rf              = c.rf;
        env.tk              = c.tk;
        env.tc              = c.tc;
        env.tr              = c.tr;
        env.above           = c.above;
        env.ref_above       = c.ref_above;
        env.par_above       = c.par_above;
        env.exam            = c.exam;
        env.det             = c.detail;
        env.capacity        = c.capacity;
        env.setup           = c.d_setup;
        env.absmax          = c.d_absmax;
        env.flags           = c.d_flags;
        env.block_sums      = c.block_sums;
        env.order           = c.cfg.prediction_radius;
        env.radius          = c.cfg.max_stencil_radius;
        env.grad_width      = c.cfg.graduation_width;
        env.refine_boundary = c.refine_boundary ? 1 : 0;
        env.relative        = c.rel_detail ? 1 : 0;
    }

    void Sequence::fields(const FieldSlot* fs, int first, int nf)
    {
        if (env.nf == nf && std::memcmp(env.f, fs + first, static_cast<size_t>(nf) * sizeof(FieldSlot)) == 0)
        {
            return; // the fields the sequence already works on
        }
        flush();
        env.nf = nf;
        for (int k = 0; k < nf; ++k)
        {
            env.f[k] = fs[first + k];
        }
        env.det    = c.detail ? c.detail + static_cast<long long>(first) * c.capacity : nullptr;
        env.absmax = c.d_absmax + first;
    }

    // the pending phases have no use for it
    void Sequence::report(int* host)
    {
        env.report = host;
    }

    void Sequence::guard(const int* flag)
    {
        if (flag != env.guard)
        {
            flush();
            env.guard = flag;
        }
    }

    // A phase joins the pending chain when it walks few enough words for one
    // cluster to keep up with the whole chip (limits per kind in Ctx).  The
    // kernel trace times every phase as a launch of its own.
    void Sequence::add(int op, int l0, int l1, int aux)
    {
        if (status)
        {
            return;
        }
        const Phase p{static_cast<short>(op), static_cast<short>(l0), static_cast<short>(l1), static_cast<short>(aux)};
        long long words = phase_words(c.g, p);
        long long limit = c.fuse_words_mesh;
        switch (op)
        {
            case OP_GHOST:
            case OP_PREDICT:
            case OP_ABSMAX:
            case OP_DETAIL:
            case OP_UPDATE_FIELDS:
                words *= std::max(1, env.nf);
                limit = c.fuse_words_field;
                break;
            case OP_MAXIMUM:
            case OP_PERIODIC_COPY:
            case OP_PERIODIC_TAG: limit = c.fuse_words_max; break;
            default: break;
        }
        if (c.chain_blocks > 0 && !c.trace.enabled && words <= limit)
        {
            chain.push_back(p);
            switch (op)
            {
                case OP_GHOST:
                case OP_PREDICT:
                case OP_MAXIMUM:
                case OP_PERIODIC_COPY:
                case OP_PERIODIC_TAG:
                case OP_GRAD_DOWN:
                case OP_REF_CHILDREN_LEVEL:
                    if (c.g.periodic && words <= (c.g.dim == 2 ? SOLO_WORDS_2D : SOLO_WORDS_3D))
                    {
                        chain.back().op |= PHASE_SOLO;
                    }
                    break;
                default: break;
            }
            if (chain.size() == CHAIN_MAX)
            {
                flush();
            }
            return;
        }
        flush();
        if (!status)
        {
            // a level of the ghost update right behind another one's launch
            Phase q = p;
            if ((op == OP_GHOST || op == OP_PREDICT) && (last_alone == OP_GHOST || last_alone == OP_PREDICT || last_alone == OP_PERIODIC_COPY))
            {
                q.aux = FOLLOWS;
            }
            last_alone = op;
            status     = launch_phase_alone(c, env, q);
        }
    }

    void Sequence::flush()
    {
        if (!status && !chain.empty())
        {
            last_alone = -1;
            if (chain.size() == 1)
            {
                chain[0].op &= static_cast<short>(~PHASE_SOLO);
                status = launch_phase_alone(c, env, chain[0]);
            }
            else
            {
                status = launch_chain(c, env, chain);
            }
        }
        chain.clear();
    }

    // the named timers bracket launches: a chain ends where one starts or stops
    void Sequence::timer_start(int id)
    {
        if (c.timers.enabled)
        {
            flush();
        }
        sg::timer_start(c, id);
    }

    void Sequence::timer_stop(int id)
    {
        if (c.timers.enabled)
        {
            flush();
        }
        sg::timer_stop(c, id);
    }

    int Sequence::done(const char* what)
    {
        flush();
        return status ? status : check(c, what);
    }
} // namespace sg
