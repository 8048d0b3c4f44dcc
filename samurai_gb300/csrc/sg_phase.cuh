// The step as a sequence of phases.
//
// A phase is one data-parallel operation on the mesh or its fields (a level of
// the ghost update, the details, a level of the tag finalisation, a pass of the
// mesh construction, ...) whose items are independent; each phase reads what
// the ones before it wrote.  The device code of a phase is written once,
// against a Team of threads, and runs in one of two ways (sg_phase.cu):
//  - as a kernel of its own over the whole chip (large levels), or
//  - as one link of a chain: consecutive small phases in a single launch of one
//    thread-block cluster that separates them by hardware cluster barriers.
// Data written by one phase and read by the next may cross SMs inside a chain:
// phases load with plain (coherent) loads, never through the read-only path.
#pragma once

#include <vector>

#include "sg_access.cuh"
#include "sg_ctx.cuh"

namespace sg
{
    constexpr int PHASE_FIELDS = 8;    // fields one phase works on together
    constexpr int SCAN_WORDS   = 2048; // words per chunk of the scan

    enum Op : int
    {
        OP_PASS_BEGIN,      // threshold bitmaps and flags cleared
        OP_GHOST,           // top-down pass of update_ghost_mr, level l0
        OP_PREDICT,         // bottom-up pass, level l0
        OP_ABSMAX_INIT,     // relative details: max |u| over the leaves
        OP_ABSMAX,
        OP_DETAIL,          // details and their threshold bits, levels l0..l1
        OP_CRITERIA,        // tags from the threshold bits
        OP_MAXIMUM,         // tag finalisation, children at level l0
        OP_NEW_CELLS,       // leaf cells of mesh n from the tags
        OP_GRAD_COARSEN,    // graduation of mesh n's cells (the first to the last of these may hang on a flag)
        OP_GRAD_EXPAND,
        OP_GRAD_EXPAND_XY,
        OP_GRAD_EXPAND_Z,
        OP_GRAD_PERIODIC,
        OP_GRAD_DOWN,       // level l0
        OP_GRAD_REFINE,     // levels l0..l1
        OP_GRAD_APPLY,      // levels l0..l1
        OP_COMPARE,         // do the leaf cells of m and n differ
        OP_CLEAR_UNION,     // construction of mesh n from its cells
        OP_HC_CAG,
        OP_HC2_CAG,         // levels l0..l1
        OP_CAG_ON,          // levels l0..l1
        OP_REF0,
        OP_REF0_XY,
        OP_REF0_Z,
        OP_REF_PERIODIC_SRC,
        OP_REF_PERIODIC,
        OP_REF_CHILDREN,    // levels l0..l1
        OP_REF_CHILDREN_LEVEL, // level l0
        OP_SINGLE_LEVEL,
        OP_SCAN_SUMS,
        OP_SCAN_WRITE,
        OP_UPDATE_FIELDS,   // from mesh m to mesh n
        OP_PERIODIC_COPY,   // level l0, axis aux
        OP_PERIODIC_TAG,    // level l0, axis aux >> 2, sides aux & 3 (1: upper, 2: lower, 3: both)
        OP_COUNT
    };

    // aux of a graduation phase: the slot of the flag it raises, and the slot of the flag it hangs on
    inline int grad_aux(int slot, int guard = -1)
    {
        return slot | ((guard + 1) << 3);
    }

    struct Phase
    {
        short op, l0, l1, aux;
    };

    // device pointers of one mesh
    struct MeshPtrs
    {
        uint32_t *cells, *cag, *proj, *uni, *ref, *hc, *hc2, *pred;
        int *rank, *wl_ref, *wl_cells;
        long long* lo;
        long long* host_lo; // pinned: the scan leaves the counters [0..3] here too
    };

    struct FieldSlot
    {
        double* u;      // values on mesh m
        double* un;     // update_fields: values on mesh n
        double bcv;     // Dirichlet value
        int has_bc;
    };

    // what the phases of one sequence work on: mesh m (the current one), mesh n
    // (the one being built), scratch, up to PHASE_FIELDS fields
    struct Env
    {
        Geom g;
        MeshPtrs m, n;
        uint32_t *t0, *t1, *t2, *t3, *rf;
        uint32_t *tk, *tc, *tr;    // tags: keep, coarsen, refine
        uint32_t *above, *ref_above, *par_above; // |detail| over the coarsen, refine and parent thresholds
        uint32_t* exam;            // cells with a detail
        double* det;
        long long capacity;
        PassSetup* setup;
        const PassSetup* setup_host; // pinned: copied into setup when a pass begins (null: setup is in place)
        int* report;                 // pinned: where OP_COMPARE leaves the flags, with the mesh's error word at F_ERR (or null)
        const int* guard;            // when not null, the phases run only if this flag is set
        unsigned long long* absmax;
        int* flags;
        long long* block_sums;
        int order;          // prediction stencil radius
        int radius;         // max_stencil_radius
        int grad_width;
        int refine_boundary;
        int relative;
        int nf;
        FieldSlot f[PHASE_FIELDS];
    };

    constexpr int CHAIN_MAX     = 96;  // phases of one chain
    constexpr int CHAIN_THREADS = 512; // threads per block of a chain

    constexpr short PHASE_SOLO  = 0x100; // bit of op: the phase runs in the chain's first block alone
    // Levels whose phases do: a word per thread in 2D (levels up to 6: a few hundred cells, nine additions of 66
    // cycles each for a predicted ghost); 3D levels up to 2, whose padded rows are mostly empty.
    constexpr long long SOLO_WORDS_2D = 512;
    constexpr long long SOLO_WORDS_3D = 1300;

    struct PhaseList
    {
        int n;
        Phase p[CHAIN_MAX];
    };

    constexpr short FOLLOWS = 1; // aux of a ghost-update level: launched right behind another one

    // Launches phases in order: small consecutive ones as one chain, the others
    // one by one.
    struct Sequence
    {
        Ctx& c;
        Env env;
        int status = SG_OK;
        std::vector<Phase> chain; // pending
        int last_alone = -1;      // the phase launched last, if it was on its own

        Sequence(Ctx& ctx, const DeviceMesh& m, const DeviceMesh& n);
        void fields(const FieldSlot* fs, int first, int nf); // the fields of the following phases: fs[first .. first + nf)
        void add(int op, int l0 = 0, int l1 = 0, int aux = 0);
        void report(int* host);      // where OP_COMPARE reports
        void guard(const int* flag); // the following phases hang on a device flag
        void flush();                // before anything else is queued on the stream
        void timer_start(int id);
        void timer_stop(int id);
        int done(const char* what);
    };

    void build_mesh_phases(Sequence& s, bool clear);           // mesh construction of mesh n from its cells; clear: its union may hold marks
    void grad_pass_phases(Sequence& s, int slot, int guard);   // one graduation pass on mesh n's cells
    MeshPtrs mesh_ptrs(const DeviceMesh& m);
    int launch_phase_alone(Ctx& c, const Env& e, const Phase& p);
    int chain_blocks(const Geom& g);
    long long phase_words(const Geom& g, const Phase& p);
    const char* phase_name(int op);
} // namespace sg
