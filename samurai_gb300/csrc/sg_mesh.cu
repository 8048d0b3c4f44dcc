#include <algorithm>
// Mesh construction on the device: the MRMesh ids from a leaf-cell bitmap,
// and the integer kernels of the adaptation (tags -> new cells, graduation).
//
// Set algebra follows samurai's subset semantics: operators act on cells of
// one level, coarser operands are refined, .on(l) coarsens to the parent of
// any member (subset/projection.hpp:68-177).  On bitmaps these are word-wise
// AND/OR/ANDNOT, bit-pair compression (coarsen) and bit spreading (refine).
#include <nvtx3/nvToolsExt.h>

#include "sg_phase.cuh"

namespace sg
{
    cudaEvent_t take_event(Ctx& c)
    {
        if (!c.timers.pool.empty())
        {
            cudaEvent_t e = c.timers.pool.back();
            c.timers.pool.pop_back();
            return e;
        }
        cudaEvent_t e = nullptr;
        cudaEventCreate(&e);
        return e;
    }

    void give_event(Ctx& c, cudaEvent_t e)
    {
        if (e)
        {
            c.timers.pool.push_back(e);
        }
    }

    void clear_graphs(Ctx& c)
    {
        for (auto& ge : c.graphs)
        {
            cudaGraphExecDestroy(ge.exec);
            for (const auto& mk : ge.marks)
            {
                bool in_window = false;
                for (const auto& tm : c.trace.marks)
                {
                    in_window = in_window || tm.second == mk.second;
                }
                if (!in_window)
                {
                    give_event(c, mk.second);
                }
            }
        }
        c.graphs.clear();
    }

    void launched(Ctx& c, const char* name, int count)
    {
        c.n_launches += count;
        if (c.trace.enabled)
        {
            trace_mark(c, name);
        }
    }

    // a trace event after the work queued so far; name null for the head of a launch sequence (the time before
    // it, a host round trip included, is charged to no kernel)
    void trace_mark(Ctx& c, const char* name)
    {
        // inside a stream capture an external record becomes an event-record node of the graph (a plain
        // record would only order the capture); outside a capture it is a plain record
        cudaEvent_t e              = take_event(c);
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(c.stream, &cs);
        if (cs == cudaStreamCaptureStatusActive)
        {
            cudaEventRecordWithFlags(e, c.stream, cudaEventRecordExternal);
        }
        else
        {
            cudaEventRecord(e, c.stream);
        }
        c.trace.marks.push_back({name, e});
    }

    namespace
    {
        // samurai's timer names (timers.hpp:111-1036) as NVTX ranges, so that a
        // profiler's timeline shows the phases under the reference's names
        const char* const TIMER_NAMES[T_COUNT] = {"mesh adaptation",  "ghost update",    "detail computation", "tag cells",     "tag finalization",
                                                  "mesh update",      "make_graduation", "mesh construction",  "fields update", "field expressions"};
    } // namespace

    void timer_start(Ctx& c, int id)
    {
        nvtxRangePushA(TIMER_NAMES[id]);
        if (!c.timers.enabled)
        {
            return;
        }
        cudaEvent_t e = take_event(c);
        cudaEventRecord(e, c.stream);
        c.timers.pending[id] = e;
    }

    void timer_stop(Ctx& c, int id)
    {
        nvtxRangePop();
        if (!c.timers.enabled || !c.timers.pending[id])
        {
            return;
        }
        cudaEvent_t e = take_event(c);
        cudaEventRecord(e, c.stream);
        c.timers.open[id].push_back({c.timers.pending[id], e});
        c.timers.pending[id] = nullptr;
        ++c.timers.calls[id];
    }

    void timers_flush(Ctx& c)
    {
        cudaStreamSynchronize(c.stream);
        for (int id = 0; id < T_COUNT; ++id)
        {
            for (auto& pr : c.timers.open[id])
            {
                float ms = 0.f;
                if (cudaEventElapsedTime(&ms, pr.first, pr.second) == cudaSuccess)
                {
                    c.timers.ms[id] += ms;
                }
                c.timers.pool.push_back(pr.first);
                c.timers.pool.push_back(pr.second);
            }
            c.timers.open[id].clear();
        }
        cudaGetLastError();
    }

    int host_counts(Ctx& c, DeviceMesh& m)
    {
        if (m.host_valid)
        {
            return SG_OK;
        }
        if (cudaStreamSynchronize(c.stream) != cudaSuccess)
        {
            return check(c, "host_counts");
        }
        return counts_arrived(c, m);
    }

    int counts_arrived(Ctx& c, DeviceMesh& m)
    {
        m.nb_ref     = m.h_lo[0];
        m.nb_cells   = m.h_lo[2];
        m.host_valid = true;
        if (m.nb_ref >= (1LL << 31))
        {
            c.err = "reference mesh exceeds 2^31 cells";
            return SG_ERR_CAPACITY;
        }
        return SG_OK;
    }

    // Mesh_base::finalize_mesh for the serial unit-box case:
    // construct_union (mesh.hpp:1231-1262), MRMesh::update_sub_mesh_impl
    // (mr/mesh.hpp:222-455) and renumbering (mesh.hpp:894-911), on mesh n of
    // the sequence from its cells.
    //
    // Leaf cells lie in levels min_level .. max_level, so each set can be
    // non-empty only on a known range of levels; it is computed on that range,
    // and its other levels keep the zeros they were created with (no phase ever
    // writes them).  Operations that read the same inputs share a phase.
    void build_mesh_phases(Sequence& s, bool clear)
    {
        const Geom& g    = s.c.g;
        const int minl   = g.min_level, maxl = g.max_level;
        const bool multi = maxl != minl;
        const int lmin   = minl >= 2 ? minl - 2 : 0; // lowest level of the reference
        const int h2lo = std::max(minl - 2, 0), h2hi = maxl - 2;
        const int t1lo = std::max(minl - 1, 0), t1hi = maxl - 1;
        if (clear)
        {
            s.add(OP_CLEAR_UNION);
        }
        s.add(OP_HC_CAG, std::min(std::max(minl - 1, 0), minl), maxl);
        if (g.dim == 2)
        {
            const int lo2 = multi ? std::min(h2lo, t1lo) : h2lo;
            const int hi2 = multi ? std::max(h2hi, t1hi) : h2hi;
            if (lo2 <= hi2)
            {
                s.add(OP_HC2_CAG, lo2, hi2);
            }
        }
        else
        {
            s.add(OP_HC2_CAG, std::min(h2lo, minl), maxl);
            if (multi)
            {
                s.add(OP_CAG_ON, t1lo, t1hi);
            }
        }
        if (!multi)
        {
            s.add(OP_SINGLE_LEVEL);
            if (g.periodic)
            {
                // the translated cells expanded by the stencil radius, within the
                // expanded domain (mr/mesh.hpp:294-317)
                s.add(OP_REF_PERIODIC, minl, maxl);
            }
        }
        else
        {
            if (g.dim == 2)
            {
                s.add(OP_REF0, lmin, maxl);
            }
            else
            {
                s.add(OP_REF0_XY, lmin, maxl);
                s.add(OP_REF0_Z, lmin, maxl);
            }
            if (g.periodic)
            {
                s.add(OP_REF_PERIODIC_SRC, lmin, maxl);
                s.add(OP_REF_PERIODIC, lmin, maxl);
            }
            // children of the projection cells, bottom-up; the reference starts at
            // min_level - 2, so the first level with a source is above it
            const int ref_lo = std::max(1, lmin + 1);
            if (!g.periodic)
            {
                s.add(OP_REF_CHILDREN, ref_lo - 1, maxl);
            }
            else
            {
                for (int l = ref_lo; l <= maxl; ++l)
                {
                    s.add(OP_REF_CHILDREN_LEVEL, l, l);
                }
            }
        }
        if (!multi || g.periodic)
        {
            s.add(OP_SCAN_SUMS); // otherwise added up by the children's pass
        }
        s.add(OP_SCAN_WRITE);
    }

    int build_mesh(Ctx& c, DeviceMesh& m)
    {
        ScopedTimer timer(c, T_CONSTRUCTION);
        Sequence s(c, m, m);
        build_mesh_phases(s, true);
        if (int st = s.done("build_mesh"))
        {
            return st;
        }
        m.host_valid = false;
        return SG_OK;
    }

    // One pass of make_graduation (algorithm/graduation.hpp:573-726, 245-330)
    // on mesh n's cells: the flag `slot` is raised when the pass refined
    // something; guard: the slot of the flag the whole pass hangs on, or -1.
    // The contiguous-boundary pass (graduation.hpp:121-249) is a no-op for a
    // max_stencil_radius of 1.
    void grad_pass_phases(Sequence& s, int slot, int guard)
    {
        const Geom& g = s.c.g;
        // A cell of level l must be refined when a cell of level l+2 or finer
        // lies within 2 gw cells of it at that finer level: levels min_level ..
        // max_level-2 can hold such cells.
        const int dtop = g.max_level - 2;
        const int dlo  = g.min_level;
        // radius 2: the contiguous-boundary cells refine leaves of levels min_level .. max_level-1 too
        const bool contiguous = s.c.cfg.max_stencil_radius == 2;
        const int rtop        = contiguous ? g.max_level - 1 : dtop;
        const int aux         = grad_aux(slot, guard);
        if (dtop >= dlo)
        {
            s.add(OP_GRAD_COARSEN, dlo, dtop + 1, aux);
            if (g.dim == 2)
            {
                s.add(OP_GRAD_EXPAND, dlo + 1, dtop + 1, aux);
            }
            else
            {
                s.add(OP_GRAD_EXPAND_XY, dlo + 1, dtop + 1, aux);
                s.add(OP_GRAD_EXPAND_Z, dlo + 1, dtop + 1, aux);
            }
            if (g.periodic)
            {
                s.add(OP_GRAD_PERIODIC, dlo + 1, dtop + 1, aux);
                for (int l = dtop; l >= dlo; --l)
                {
                    s.add(OP_GRAD_DOWN, l, l, aux);
                }
            }
        }
        else if (!contiguous || g.max_level <= dlo)
        {
            return;
        }
        if (!g.periodic || contiguous)
        {
            s.add(OP_GRAD_REFINE, dlo, rtop, aux);
        }
        s.add(OP_GRAD_APPLY, dlo, rtop + 1, grad_aux(slot, slot)); // nothing to apply unless the pass raised its flag
    }

    // make_graduation to the fixed point, with a host test after each pass
    int graduate(Ctx& c, DeviceMesh& m, DeviceMesh& nm, int* iterations)
    {
        ScopedTimer timer(c, T_GRADUATION);
        int nit = 0;
        for (;;)
        {
            ++nit;
            cudaMemsetAsync(c.d_flags + F_GRADX, 0, sizeof(int), c.stream);
            Sequence s(c, m, nm);
            grad_pass_phases(s, F_GRADX, -1);
            if (int st = s.done("graduation"))
            {
                return st;
            }
            cudaMemcpyAsync(c.h_flags + F_GRADX, c.d_flags + F_GRADX, sizeof(int), cudaMemcpyDeviceToHost, c.stream);
            if (cudaStreamSynchronize(c.stream) != cudaSuccess)
            {
                return check(c, "graduate sync");
            }
            if (!c.h_flags[F_GRADX])
            {
                break;
            }
            if (nit > 64)
            {
                c.err = "graduation did not converge";
                return SG_ERR_STATE;
            }
        }
        if (iterations)
        {
            *iterations = nit - 1;
        }
        return SG_OK;
    }
} // namespace sg
