// Device code of the phases (see sg_phase.cuh) and the FP64 operators they
// share with the transposed launches.
#pragma once

#include <type_traits>

#include "sg_phase.cuh"

namespace sg
{
    // One warp per listed word, lane b on bit b.  The list holds the
    // non-empty words of a superset (reference or leaf cells) in
    // ascending order; word_of(w) narrows it to the subset a kernel acts
    // on.  Consecutive cells of a word are consecutive doubles, so every
    // field access of a warp is one 256-byte segment.
    template <class WordF, class CellF>
    __device__ __forceinline__ void warp_list(const int* list, long long begin, long long end, long long warp0, long long nwarps, WordF word_of,
                                              CellF cell)
    {
        const int lane = threadIdx.x & 31;
        for (long long i = begin + warp0; i < end; i += nwarps)
        {
            const long long w = list[i];
            const uint32_t v  = word_of(w);
            if ((v >> lane) & 1u)
            {
                cell(w, lane);
            }
        }
    }

    constexpr unsigned FULL_MASK = 0xffffffffu;

    __device__ __forceinline__ long long warp_id()
    {
        return (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
    }

    __device__ __forceinline__ long long warp_count()
    {
        return (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
    }


    // The prediction coefficients interp_coeffs<3> (numeric/prediction.hpp:32-36)
    // of tap t in {0,1,2} for a child of parity q are 1 at t = 1 and
    // +-1/8 at t = 0, 2 (negative at t = 0 for odd children, at t = 2 for
    // even ones); products over the axes are +-8^-k, k = off-centre taps.

    // Element of a cell that the reference algorithm guarantees to be in
    // the stored box.  A position outside it (a bug or an invalid mesh)
    // is recorded in the device error word and redirected to element 0,
    // so that no access leaves the allocation.
    __device__ __forceinline__ long long elem_at(const Geom& g, int l, int x, int y, int z)
    {
        const Pos p = pos_of(g, l, x, y, z);
        if (p.w < 0)
        {
            atomicOr(g.err, 1);
            return 0;
        }
        return elem(p);
    }

    // x * 2^-s (0 < s < 64), exactly, without the FP64 pipe when it can: for
    // a normal x whose product stays normal the product is x with its
    // exponent lowered by s (what the multiplication rounds to, since it is
    // exact); zeros keep their bits; other values take the multiplication.
    __device__ __forceinline__ double scale_down(double x, int s)
    {
        const long long b = __double_as_longlong(x);
        const int e       = static_cast<int>((b >> 52) & 0x7FF);
        if (e > s && e < 0x7FF)
        {
            return __longlong_as_double(b - (static_cast<long long>(s) << 52));
        }
        if ((static_cast<unsigned long long>(b) << 1) == 0)
        {
            return x;
        }
        return x * __longlong_as_double(static_cast<long long>(1023 - s) << 52);
    }

    // x * 8^-k: the prediction coefficients' magnitudes
    __device__ __forceinline__ double scale8(double x, int k)
    {
        return scale_down(x, 3 * k);
    }

    template <int CAP>
    __device__ __forceinline__ LinForm<CAP> scale_down(const LinForm<CAP>& x, int s)
    {
        return x * (1.0 / static_cast<double>(1LL << s));
    }

    // -x when neg, by the sign bit (exact, no FP64 operation)
    __device__ __forceinline__ double negate_if(bool neg, double x)
    {
        return __longlong_as_double(__double_as_longlong(x) ^ (static_cast<long long>(neg) << 63));
    }

    template <int CAP>
    __device__ __forceinline__ LinForm<CAP> scale8(const LinForm<CAP>& x, int k)
    {
        return x * (k == 1 ? 0.125 : (k == 2 ? 0.015625 : 0.001953125));
    }

    template <int CAP>
    __device__ __forceinline__ LinForm<CAP> negate_if(bool neg, const LinForm<CAP>& x)
    {
        return neg ? -x : x;
    }

    // A box of cells [x0, x0+n) x [y0, y0+n) x [z0, z0+n) at level l as a base
    // element and strides: both corners are checked against the stored
    // box (a violation is recorded and every access goes to element 0)
    struct Box3
    {
        long long base, sy, sz;
    };

    template <int DIM>
    __device__ __forceinline__ Box3 box_at(const Geom& g, int l, int x0, int y0, int z0, int n)
    {
        const Pos lo = pos_of(g, l, x0, y0, DIM == 3 ? z0 : 0);
        const Pos hi = pos_of(g, l, x0 + n - 1, y0 + n - 1, DIM == 3 ? z0 + n - 1 : 0);
        if (lo.w < 0 || hi.w < 0)
        {
            atomicOr(g.err, 1);
            return {0, 0, 0};
        }
        const LevelGeom& L = g.lv[l];
        return {elem(lo), 32LL * L.W, 32LL * L.W * L.R};
    }

    // prediction_op<order,false> for one fine cell (numeric/prediction.hpp:286-361)
    template <int DIM, class A>
    __device__ __forceinline__ typename A::V predict_one(const Geom& g, const A& u, int l, int x, int y, int z, int order)
    {
        const int px = x >> 1, py = y >> 1, pz = z >> 1;
        if (order == 0)
        {
            return u.get(elem_at(g, l - 1, px, py, pz));
        }
        // acc + u * coeff with coeff = ((1 * cx) * cy) * cz = +-8^-k (k = axes
        // with an off-centre tap): u * coeff is +-(u * 8^-k) bit for bit
        // (power-of-two scaling is exact) and acc + (-m) is acc - m
        typename A::V acc = A::konst(0.);
        const int qx = x & 1, qy = y & 1, qz = z & 1;
        const Box3 bx     = box_at<DIM>(g, l - 1, px - 1, py - 1, pz - 1, 3);
#pragma unroll
        for (int sz = 0; sz < (DIM == 3 ? 3 : 1); ++sz)
        {
#pragma unroll
            for (int sy = 0; sy < 3; ++sy)
            {
                const long long base = bx.base + sy * bx.sy + sz * bx.sz;
#pragma unroll
                for (int sx = 0; sx < 3; ++sx)
                {
                    const int k      = (sx != 1) + (sy != 1) + (DIM == 3 && sz != 1);
                    const bool neg   = ((sx == 0 && qx) || (sx == 2 && !qx)) ^ ((sy == 0 && qy) || (sy == 2 && !qy))
                                     ^ (DIM == 3 && ((sz == 0 && qz) || (sz == 2 && !qz)));
                    const typename A::V v = u.get(base + sx);
                    // acc + u * coeff == acc + (+-m): one FP64 addition per tap
                    const typename A::V m = k == 0 ? v : scale8(v, k);
                    acc                   = acc + negate_if(neg, m);
                }
            }
        }
        return acc;
    }

    // projection_op_ (numeric/projection.hpp:15-65)
    template <int DIM, class A>
    __device__ __forceinline__ typename A::V project_one(const Geom& g, const A& u, int lf, int x, int y, int z)
    {
        typename A::V sum = A::konst(0.);
        const Box3 bx     = box_at<DIM>(g, lf, 2 * x, 2 * y, 2 * z, 2);
#pragma unroll
        for (int sz = 0; sz < (DIM == 3 ? 2 : 1); ++sz)
        {
#pragma unroll
            for (int sy = 0; sy < 2; ++sy)
            {
                const long long e = bx.base + sy * bx.sy + sz * bx.sz;
                sum               = sum + (u.get(e) + u.get(e + 1));
            }
        }
        // sum * (1 / 2^dim)
        return scale_down(sum, DIM);
    }

    // PolynomialExtrapolation of the second ghost layer (bc/polynomial_extrapolation.hpp:22-92, stencil of 4
    // cells along d from c - d): u(c + 2d) = u(c - d) - 3 u(c) + 3 u(c + d), in the reference's operation order
    template <class A>
    __device__ __forceinline__ void extrapolate_layer2(const Geom& g, int l, const int* c, const int* d, const A& u)
    {
        const int z = g.dim == 3;
        const long long em = elem_at(g, l, c[0] - d[0], c[1] - d[1], z ? c[2] - d[2] : 0);
        const long long e0 = elem_at(g, l, c[0], c[1], z ? c[2] : 0);
        const long long e1 = elem_at(g, l, c[0] + d[0], c[1] + d[1], z ? c[2] + d[2] : 0);
        const long long e2 = elem_at(g, l, c[0] + 2 * d[0], c[1] + 2 * d[1], z ? c[2] + 2 * d[2] : 0);
        u.put(e2, (u.get(em) - u.get(e0) * 3.0) + u.get(e1) * 3.0);
    }

    // ------------------------------------------------------------ threads
    // the threads a phase runs on: the whole grid of its own launch, or the
    // cluster of a chain
    struct Team
    {
        int tid, nthr;      // thread
        int block, nblocks; // block

        __device__ __forceinline__ int warp0() const
        {
            return tid >> 5;
        }

        __device__ __forceinline__ int nwarps() const
        {
            return nthr >> 5;
        }
    };

    // the blocks from `first` on
    __device__ __forceinline__ Team grid_team(int first = 0)
    {
        const int b = static_cast<int>(blockIdx.x) - first, n = static_cast<int>(gridDim.x) - first;
        return {b * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x), n * static_cast<int>(blockDim.x), b, n};
    }

    // ------------------------------------------------------------ items
    // The cells of a set, spread evenly over the threads of each block: a block
    // takes a chunk of words (at most one per thread, loaded together), ranks
    // their set bits with a block prefix sum and hands the items out in order, one
    // per thread and round; with several fields the rounds run over (field, item)
    // pairs.  The bands of cells the path works on fill a few words of a row and
    // leave the next ones empty; a warp per word (or per few words) waits for its
    // fullest word.  item(valid, w, b, field) is called by every thread of a
    // block (it may shuffle), consecutive threads on consecutive items.
    constexpr int ITEM_THREADS = 1024; // largest block
    constexpr int ITEM_BLOCK   = 512;  // largest block of the phases and kernels that need more than 64 registers

    struct ItemShared
    {
        int pre[ITEM_THREADS];
        int w[ITEM_THREADS];
        uint32_t m[ITEM_THREADS];
        int part[32];
    };

    __device__ __forceinline__ ItemShared& item_shared()
    {
        __shared__ ItemShared s;
        return s;
    }

    // Everything the launch this one depends on has written is visible after it (nothing to wait for in a launch
    // without the programmatic attribute).  PDL: the code runs in such a launch.
    template <bool PDL>
    __device__ __forceinline__ void dependency_wait()
    {
        if constexpr (PDL)
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
        }
    }

    // position of set bit number r (from 0) of m
    __device__ __forceinline__ int nth_bit(uint32_t m, int r)
    {
        int pos = 0;
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1)
        {
            const int cnt = __popc(m & ((1u << sh) - 1u));
            if (r >= cnt)
            {
                r -= cnt;
                m >>= sh;
                pos += sh;
            }
        }
        return pos;
    }

    // list: word indices, entries [begin, end); null: the words [begin, end) themselves
    template <class WordF, class ItemF>
    __device__ __forceinline__ void block_items(const int* list, int begin, int end, const Team& T, int nf, WordF word_of, ItemF item)
    {
        ItemShared& S  = item_shared();
        const int B    = static_cast<int>(blockDim.x), t = static_cast<int>(threadIdx.x);
        const int lane = t & 31, warp = t >> 5, nwarp = B >> 5;
        const int n    = end - begin;
        // words per block and round: an even share, between 16 and one per thread
        const int chunk = min(B, max(16, (n + T.nblocks - 1) / T.nblocks));
        for (int c0 = T.block * chunk; c0 < n; c0 += T.nblocks * chunk)
        {
            int w      = 0;
            uint32_t m = 0u;
            if (t < chunk && c0 + t < n)
            {
                w = list ? list[begin + c0 + t] : begin + c0 + t;
                m = word_of(w);
            }
            int incl = __popc(m);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int x = __shfl_up_sync(FULL_MASK, incl, o);
                incl += lane >= o ? x : 0;
            }
            __syncthreads(); // the previous round's readers are done
            if (lane == 31)
            {
                S.part[warp] = incl;
            }
            __syncthreads();
            int before = 0, total = 0;
            if (lane < nwarp)
            {
                total = S.part[lane];
            }
            before = lane < warp ? total : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                before += __shfl_xor_sync(FULL_MASK, before, o);
                total += __shfl_xor_sync(FULL_MASK, total, o);
            }
            if (total == 0)
            {
                continue; // the same on every thread
            }
            S.pre[t] = before + incl - __popc(m);
            S.w[t]   = w;
            S.m[t]   = m;
            __syncthreads();
            const int all = total * nf;
            for (int base = 0; base < all; base += B)
            {
                int j = base + t, f = 0;
                const bool valid = j < all;
                if (!valid)
                {
                    j = 0;
                }
                while (j >= total)
                {
                    j -= total;
                    ++f;
                }
                // the word of item j: the last one whose prefix does not exceed j
                int lo = 0;
                for (int step = 1 << (31 - __clz(B - 1)); step > 0; step >>= 1)
                {
                    if (lo + step < B && S.pre[lo + step] <= j)
                    {
                        lo += step;
                    }
                }
                item(valid, S.w[lo], nth_bit(S.m[lo], j - S.pre[lo]), f);
            }
        }
    }

    // ------------------------------------------------------------ words
    // A bitmap word in its level: row (ry, rz) of the padded box, word wi of the row
    struct Word
    {
        int l, w, ry, rz, wi;
    };

    template <int DIM>
    __device__ __forceinline__ Word word_at(const Geom& g, int l, int w)
    {
        const LevelGeom& L = g.lv[l];
        const unsigned loc = static_cast<unsigned>(w - static_cast<int>(L.woff));
        const unsigned row = fastdiv(loc, L.mW, L.sW);
        Word p;
        p.l  = l;
        p.w  = w;
        p.wi = static_cast<int>(loc - row * static_cast<unsigned>(L.W));
        if (DIM == 2)
        {
            p.ry = static_cast<int>(row);
            p.rz = PY;
        }
        else
        {
            const unsigned z = fastdiv(row, L.mR, L.sR);
            p.rz             = static_cast<int>(z);
            p.ry             = static_cast<int>(row - z * static_cast<unsigned>(L.R));
        }
        return p;
    }

    // the level of word w in [l0, l1]; the finest levels hold most words
    __device__ __forceinline__ int level_down(const Geom& g, int w, int l0, int l1)
    {
        int l = l1;
        while (l > l0 && w < static_cast<int>(g.lv[l].woff))
        {
            --l;
        }
        return l;
    }

    template <int DIM, class F>
    __device__ __forceinline__ void team_words(const Geom& g, const Team& T, int l0, int l1, F f)
    {
        const int begin = static_cast<int>(g.lv[l0].woff);
        const int end   = static_cast<int>(g.lv[l1].woff + g.lv[l1].nwords);
        for (int w = begin + T.tid; w < end; w += T.nthr)
        {
            f(word_at<DIM>(g, level_down(g, w, l0, l1), w));
        }
    }

    // first word of row (ry, rz) of level l
    template <int DIM>
    __device__ __forceinline__ int row_base(const LevelGeom& L, int ry, int rz)
    {
        return static_cast<int>(L.woff) + (DIM == 2 ? ry : rz * L.R + ry) * L.W;
    }

    // Rows further than 4 cells from the box hold no cell of any set of the
    // path (the sets reach at most 4 cells outside it), so a dilation is empty
    // there; inside, its source rows lie in the stored box, and a word's
    // neighbours in the flat array stand for its neighbours in the row (beyond
    // a row's ends the flat neighbour's bits next to the word are never set).
    template <int DIM>
    __device__ __forceinline__ bool live_row(const Geom& g, const Word& p)
    {
        const int n = g.lv[p.l].n;
        return p.ry >= PY - 4 && p.ry < n + PY + 4 && (DIM == 2 || (p.rz >= PY - 4 && p.rz < n + PY + 4));
    }

    template <int DIM>
    __device__ __forceinline__ uint32_t dilate_xy(const Geom& g, const uint32_t* src, const Word& p, int r)
    {
        const int W  = g.lv[p.l].W;
        uint32_t out = 0u;
        for (int dy = -r; dy <= r; ++dy)
        {
            const uint32_t* s  = src + p.w + dy * W;
            const uint32_t mid = s[0], left = s[-1], right = s[1];
            if (mid | left | right)
            {
                out |= dilate_x(left, mid, right, r);
            }
        }
        return out;
    }

    __device__ __forceinline__ uint32_t dilate_z(const Geom& g, const uint32_t* src, const Word& p, int r)
    {
        const int plane = g.lv[p.l].W * g.lv[p.l].R;
        uint32_t out    = 0u;
        for (int dz = -r; dz <= r; ++dz)
        {
            out |= src[p.w + dz * plane];
        }
        return out;
    }

    // The child words of word p (level l): in each of the 2^(DIM-1) child rows
    // the words base + k and base + k + 1, k = 2 wi - 1, hold the children of
    // its low and high 16 cells.  f(row number, low index or -1, high index or -1)
    template <int DIM, class F>
    __device__ __forceinline__ void child_words(const Geom& g, const Word& p, F f)
    {
        const LevelGeom& F_ = g.lv[p.l + 1];
        const int k         = 2 * p.wi - 1;
#pragma unroll
        for (int s = 0; s < (DIM == 3 ? 4 : 2); ++s)
        {
            const int fy = 2 * p.ry - PY + (s & 1);
            const int fz = 2 * p.rz - PY + (s >> 1);
            if (fy < 0 || fy >= F_.R || (DIM == 3 && (fz < 0 || fz >= F_.R)))
            {
                continue;
            }
            const int base = row_base<DIM>(F_, fy, fz);
            f(s, (k >= 0 && k < F_.W) ? base + k : -1, (k + 1 < F_.W) ? base + k + 1 : -1);
        }
    }

    // parents of any member: word p of the set one level coarser than `fine`
    template <int DIM>
    __device__ __forceinline__ uint32_t coarsen(const Geom& g, const uint32_t* fine, const Word& p)
    {
        uint32_t lo = 0u, hi = 0u;
        child_words<DIM>(g, p,
                         [&](int, int a, int b)
                         {
                             lo |= a >= 0 ? fine[a] : 0u;
                             hi |= b >= 0 ? fine[b] : 0u;
                         });
        return (lo | hi) ? compress_pairs(lo, hi) : 0u;
    }

    // the word that holds the parents of word p's cells, and which half of it
    struct Parent
    {
        int w; // -1: outside the coarse box
        int shift;
        int ry, rz, wi;
    };

    template <int DIM>
    __device__ __forceinline__ Parent parent_of(const Geom& g, const Word& p)
    {
        const LevelGeom& C = g.lv[p.l - 1];
        Parent q;
        q.ry    = ((p.ry - PY) >> 1) + PY;
        q.rz    = DIM == 3 ? ((p.rz - PY) >> 1) + PY : PY;
        q.wi    = (p.wi + 1) >> 1;
        q.shift = ((p.wi + 1) & 1) ? 16 : 0;
        q.w     = (q.ry >= 0 && q.ry < C.R && (DIM == 2 || (q.rz >= 0 && q.rz < C.R)) && q.wi < C.W) ? row_base<DIM>(C, q.ry, q.rz) + q.wi : -1;
        return q;
    }

    template <int DIM>
    __device__ __forceinline__ WordLoc loc_of(const Geom& g, const Word& p)
    {
        return {DIM == 2 ? p.ry : static_cast<long long>(p.rz) * g.lv[p.l].R + p.ry, p.wi};
    }

    template <int DIM>
    __device__ __forceinline__ uint32_t box_bits(const Geom& g, const Word& p, int lo, int hi)
    {
        const WordLoc q = loc_of<DIM>(g, p);
        return box_mask(g, p.l, q.row, q.wi, lo, hi);
    }

    // ------------------------------------------------------- ghost update
    // The 2^DIM (M = 2) or 4^DIM (M = 4) cells under cell (x, y, z) of level l
    // at level l + log2 M: the members of ref, row by row (M consecutive cells,
    // aligned to M: one word)
    template <int DIM, int M>
    struct Children
    {
        static constexpr int ROWS = DIM == 3 ? M * M : M;
        uint32_t bits[ROWS];
        long long el[ROWS];

        __device__ __forceinline__ void load(const Geom& g, int lc, int x, int y, int z, const uint32_t* ref)
        {
#pragma unroll
            for (int s = 0; s < ROWS; ++s)
            {
                const Pos p = pos_of(g, lc, M * x, M * y + s % M, DIM == 3 ? M * z + s / M : 0);
                bits[s]     = p.w >= 0 ? (ref[p.w] >> p.b) & ((1u << M) - 1u) : 0u;
                el[s]       = elem(p);
            }
        }

        __device__ __forceinline__ int count() const
        {
            int n = 0;
#pragma unroll
            for (int s = 0; s < ROWS; ++s)
            {
                n += __popc(bits[s]);
            }
            return n;
        }

        // f on the members in the reference's order (z, y, x ascending)
        template <class F>
        __device__ __forceinline__ void each(F f) const
        {
#pragma unroll
            for (int s = 0; s < ROWS; ++s)
            {
#pragma unroll
                for (int k = 0; k < M; ++k)
                {
                    if ((bits[s] >> k) & 1u)
                    {
                        f(el[s] + k);
                    }
                }
            }
        }
    };

    // the sum of the members' values, in order from 0: loaded together, then added one by one
    template <int DIM, int M, class A>
    __device__ __forceinline__ typename A::V sum_children(const Children<DIM, M>& ch, const A& u)
    {
        typename A::V sum = A::konst(0.);
        if constexpr (std::is_same<A, ValAcc>::value && (DIM == 2 || M == 2))
        {
            double v[Children<DIM, M>::ROWS * M];
#pragma unroll
            for (int s = 0; s < Children<DIM, M>::ROWS * M; ++s)
            {
                v[s] = ((ch.bits[s / M] >> (s % M)) & 1u) ? u.get(ch.el[s / M] + s % M) : 0.;
            }
#pragma unroll
            for (int s = 0; s < Children<DIM, M>::ROWS * M; ++s)
            {
                if ((ch.bits[s / M] >> (s % M)) & 1u)
                {
                    sum = sum + v[s];
                }
            }
        }
        else
        {
            ch.each([&](long long e) { sum = sum + u.get(e); });
        }
        return sum;
    }

    // v / n for a member count n: a power of two only moves the exponent
    template <class A>
    __device__ __forceinline__ typename A::V mean_of(const typename A::V& v, int n)
    {
        if constexpr (std::is_same<A, ValAcc>::value)
        {
            if ((n & (n - 1)) == 0)
            {
                return n == 1 ? v : scale_down(v, 31 - __clz(n));
            }
        }
        return v / static_cast<double>(n);
    }

    struct FaceArgs
    {
        int l;
        int do_project;   // project_bc: level < max_level
        int do_dirichlet; // apply_field_bc: level >= min_level and a BC is attached
        int do_predict;   // predict_bc: min_level <= level < max_level
    };

    // One face position of level l: the Dirichlet ghost 2v - u
    // (bc/dirichlet.hpp:22-29) of a leaf and predict_bc to level l+1
    // (update_outer_ghost.hpp:195-266), or project_bc
    // (update_outer_ghost.hpp:20-155) next to a union cell.
    template <int DIM, bool PDL, class A>
    __device__ __forceinline__ void face_item(const Geom& g, const FaceArgs& a, long long t, const uint32_t* cells, const uint32_t* uni,
                                              const uint32_t* ref, const A& u, double value)
    {
        const int l = a.l;
        // n = 2^l: the direction and the position on the face are bit fields of t
        const int n = g.lv[l].n, k = static_cast<int>(t >> (l * (DIM - 1)));
        const int axis = k >> 1, sgn = (k & 1) ? -1 : 1; // (+e0, -e0, +e1, -e1, ...) (stencil.hpp:301-317)
        const int f0 = static_cast<int>(t) & (n - 1), f1 = DIM == 3 ? static_cast<int>(t >> l) & (n - 1) : 0;
        if ((g.periodic >> axis) & 1)
        {
            return; // a periodic axis has no boundary
        }
        const int at = sgn > 0 ? n - 1 : 0;
        // the free coordinates fill the other axes in order
        const int in[3]  = {axis == 0 ? at : f0, axis == 1 ? at : (axis == 0 ? f0 : f1), DIM == 3 ? (axis == 2 ? at : f1) : 0};
        const int dir[3] = {axis == 0 ? sgn : 0, axis == 1 ? sgn : 0, axis == 2 ? sgn : 0};
        const int gx = in[0] + dir[0], gy = in[1] + dir[1], gz = in[2] + dir[2];
        // most positions of a fine level have neither a leaf nor a finer leaf behind them; for the others
        // everything the roles ask first is loaded together
        const Pos pi      = pos_of(g, l, in[0], in[1], in[2]);
        const uint32_t wc = cells[pi.w], wu = uni[pi.w];
        if (!(((wc | wu) >> pi.b) & 1u))
        {
            return;
        }
        const Pos pg       = pos_of(g, l, gx, gy, gz);
        const uint32_t wg  = ref[pg.w];
        const long long eg = elem(pg);
        Children<DIM, 2> c2;
        if (l + 1 < g.nlev)
        {
            c2.load(g, l + 1, gx, gy, gz, ref);
        }
        dependency_wait<PDL>();
        const typename A::V ui = u.get(elem(pi));
        if ((a.do_dirichlet || a.do_predict) && ((wc >> pi.b) & 1u))
        {
            typename A::V v;
            if (a.do_dirichlet)
            {
                v = A::konst(2 * value) - ui;
                u.put(eg, v);
                // update_further_ghosts_by_polynomial_extrapolation (bc/apply_field_bc.hpp:531-593), ghost
                // width 2: the second layer beyond a boundary leaf, where it is a reference cell
                if (g.ghost_width >= 2 && test(ref, g, l, gx + dir[0], gy + dir[1], gz + dir[2]))
                {
                    extrapolate_layer2(g, l, in, dir, u);
                }
            }
            else
            {
                v = u.get(eg);
            }
            if (a.do_predict)
            {
                c2.each([&](long long e) { u.put(e, v); });
            }
        }
        else if (a.do_project && ((wu >> pi.b) & 1u))
        {
            if (!((wg >> pg.b) & 1u))
            {
                return;
            }
            typename A::V v = A::konst(0.);
            int nch         = c2.count();
            if (nch)
            {
                v = mean_of<A>(sum_children<DIM, 2>(c2, u), nch);
            }
            else if (l + 2 < g.nlev)
            {
                Children<DIM, 4> c4;
                c4.load(g, l + 2, gx, gy, gz, ref);
                nch = c4.count();
                if (nch)
                {
                    v = mean_of<A>(sum_children<DIM, 4>(c4, u), nch);
                }
            }
            u.put(eg, v);
            // the second ghost layer beyond a boundary cell that is not a leaf but has finer leaves
            // (apply_extrapolation_bc_ghosts, bc/apply_field_bc.hpp:196-214), ghost width 2
            if (g.ghost_width >= 2 && a.do_dirichlet && test(ref, g, l, gx + dir[0], gy + dir[1], gz + dir[2]))
            {
                extrapolate_layer2(g, l, in, dir, u);
            }
        }
    }

    // corner positions of level l: the 2^DIM corners and, in 3D, the 12 edges' n positions
    template <int DIM>
    __host__ __device__ __forceinline__ long long corner_count(const Geom& g, int l)
    {
        return DIM == 2 ? 4 : 8 + 12LL * g.lv[l].n;
    }

    // One corner position: update_outer_corners_by_polynomial_extrapolation
    // (bc/apply_field_bc.hpp:371-505), then project_corner_below
    // (algorithm/update_outer_ghost.hpp:268-337).  Layer 1 copies the corner leaf, layer 2 (ghost width 2)
    // extrapolates along the diagonal d, then the other ghosts of the corner block copy the diagonal ones (the
    // off-diagonal copies).  The coarse corner ghost one or two levels below takes the value of the fine one at
    // the first of its positions along the edge, the position of the thread that owns the fine one.
    // parts: 1 the corners, 2 their projection below, 3 both.
    template <int DIM, bool PDL, class A>
    __device__ __forceinline__ void corner_item(const Geom& g, int l, long long t, const uint32_t* cells, const uint32_t* ref, const A& u, int parts)
    {
        const int n = g.lv[l].n;
        int d[3]    = {0, 0, 0};
        int pos     = 0, free_axis = -1;
        if (t < (1 << DIM))
        {
            for (int k = 0; k < DIM; ++k)
            {
                d[k] = ((t >> k) & 1) ? 1 : -1;
            }
        }
        else
        {
            const int e = static_cast<int>((t - 8) >> l); // n = 2^l positions per edge
            pos         = static_cast<int>(t - 8) & (n - 1);
            free_axis   = e >> 2;
            d[free_axis == 0 ? 1 : 0] = (e & 1) ? 1 : -1;
            d[free_axis == 2 ? 1 : 2] = (e & 2) ? 1 : -1;
        }
        if (crosses_periodic(g, d))
        {
            return; // no corner across a periodic axis
        }
        int c[3] = {0, 0, 0};
        for (int k = 0; k < DIM; ++k)
        {
            c[k] = d[k] > 0 ? n - 1 : (d[k] < 0 ? 0 : pos);
        }
        // the fine position of a projection below is the ghost eg of this thread; all it reads is loaded together
        const Pos pc = pos_of(g, l, c[0], c[1], c[2]);
        const Pos pe = pos_of(g, l, c[0] + d[0], c[1] + d[1], DIM == 3 ? c[2] + d[2] : 0);
        const long long eg = elem(pe);
        Pos below[2];
        bool project[2];
        const bool in_ref = test(ref, pe);
#pragma unroll
        for (int k = 0; k < 2; ++k)
        {
            const int dl = k + 1, pl = l - dl;
            below[k]   = Pos{-1, 0};
            project[k] = (parts & 2) && pl >= 0 && (free_axis < 0 || (pos & ((1 << dl) - 1)) == 0);
            if (project[k])
            {
                const int np = g.lv[pl].n;
                below[k]     = pos_of(g, pl, d[0] > 0 ? np : (d[0] < 0 ? -1 : pos >> dl), d[1] > 0 ? np : (d[1] < 0 ? -1 : pos >> dl),
                                  DIM == 3 ? (d[2] > 0 ? np : (d[2] < 0 ? -1 : pos >> dl)) : 0);
                project[k]   = test(ref, below[k]);
            }
        }
        const bool leaf       = (parts & 1) && test(cells, pc);
        dependency_wait<PDL>();
        const typename A::V v = leaf ? u.get(elem(pc)) : u.get(eg);
        if (leaf)
        {
            {
                u.put(eg, v);
                if (g.ghost_width >= 2)
                {
                    if (test(ref, g, l, c[0] + 2 * d[0], c[1] + 2 * d[1], DIM == 3 ? c[2] + 2 * d[2] : 0))
                    {
                        extrapolate_layer2(g, l, c, d, u);
                    }
                    // off-diagonal copies: from c + k d (k = 1, 2) to c + k d + delta, delta moving the
                    // non-zero components after the first by g - (k - 1), g in [0, 2), not all zero
                    int nz[3], nnz = 0;
                    for (int k = 0; k < DIM; ++k)
                    {
                        if (d[k] != 0)
                        {
                            nz[nnz++] = k;
                        }
                    }
                    const int combos = nnz == 3 ? 4 : 2;
                    for (int k = 1; k <= 2; ++k)
                    {
                        const int sx = c[0] + k * d[0], sy = c[1] + k * d[1], sz = DIM == 3 ? c[2] + k * d[2] : 0;
                        const long long es = elem_at(g, l, sx, sy, sz);
                        for (int combo = 0; combo < combos; ++combo)
                        {
                            int delta[3] = {0, 0, 0};
                            bool source  = true;
                            int tmp      = combo;
                            for (int p = 1; p < nnz; ++p)
                            {
                                const int dp = (tmp % 2) - (k - 1);
                                tmp /= 2;
                                delta[nz[p]] += dp * d[nz[p]];
                                source = source && dp == 0;
                            }
                            if (!source)
                            {
                                u.put(elem_at(g, l, sx + delta[0], sy + delta[1], sz + delta[2]), u.get(es));
                            }
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
        {
            if (project[k] && in_ref)
            {
                u.put(elem(below[k]), v);
            }
        }
    }

    // The items of the set bm on level l.  Every word of the level is looked at
    // when the team has a thread for it (one load to the bits); larger levels go
    // through the list of reference words.
    template <bool PDL, class ItemF>
    __device__ __forceinline__ void level_items(const Geom& g, int l, const MeshPtrs& m, const uint32_t* bm, const Team& T, int nf, ItemF item)
    {
        const LevelGeom& L = g.lv[l];
        const int first    = static_cast<int>(L.woff);
        const bool dense   = L.nwords <= T.nthr;
        block_items(dense ? nullptr : m.wl_ref, dense ? first : static_cast<int>(m.lo[LO_REF + l]),
                    dense ? first + static_cast<int>(L.nwords) : static_cast<int>(m.lo[LO_REF + l + 1]), T, nf, [&](int w) { return bm[w]; },
                    [&](bool valid, int w, int b, int f)
                    {
                        dependency_wait<PDL>(); // up to here nothing but the mesh's bitmaps was read
                        if (valid)
                        {
                            item(static_cast<long long>(w), b, cell_of(g, l, w, b), f);
                        }
                    });
    }

    // projection of the reference cells of level l onto proj_cells[l-1]
    // (numeric/projection.hpp:15-65); the children of a projection cell are
    // reference cells by construction.  item(word, bit, cell, field)
    template <bool PDL, class ItemF>
    __device__ __forceinline__ void project_items(const Geom& g, int l, const MeshPtrs& m, const Team& T, int nf, ItemF item)
    {
        level_items<PDL>(g, l - 1, m, m.proj, T, nf, item);
    }

    // prediction of the ghosts of level l from level l-1
    // (algorithm/update_ghost_mr.hpp:224-233)
    template <bool PDL, class ItemF>
    __device__ __forceinline__ void predict_items(const Geom& g, int l, const MeshPtrs& m, const Team& T, int nf, ItemF item)
    {
        level_items<PDL>(g, l, m, m.pred, T, nf, item);
    }

    // Boundary positions of level l: corners first, padded to whole warps (corner
    // and face items take different branches), then the faces.
    template <int DIM>
    __host__ __device__ __forceinline__ long long corner_slots(const Geom& g, int l)
    {
        return l >= g.min_level ? (corner_count<DIM>(g, l) + 31) / 32 * 32 : 0;
    }

    template <int DIM>
    __host__ __device__ __forceinline__ long long boundary_count(const Geom& g, int l)
    {
        const int n = g.lv[l].n;
        return corner_slots<DIM>(g, l) + 2LL * DIM * (DIM == 2 ? n : static_cast<long long>(n) * n);
    }

    // boundary position t of level l on accessor u
    template <int DIM, bool PDL, class A>
    __device__ __forceinline__ void boundary_item(const Geom& g, int l, long long t, const MeshPtrs& m, const A& u, bool has_bc, double value, int corner_parts)
    {
        const long long nc = corner_slots<DIM>(g, l);
        if (t < nc)
        {
            if (t < corner_count<DIM>(g, l))
            {
                corner_item<DIM, PDL>(g, l, t, m.cells, m.ref, u, corner_parts);
            }
        }
        else
        {
            const FaceArgs a{l, l < g.max_level, l >= g.min_level && has_bc, l >= g.min_level && l < g.max_level};
            face_item<DIM, PDL>(g, a, t - nc, m.cells, m.uni, m.ref, u, value);
        }
    }
} // namespace sg
