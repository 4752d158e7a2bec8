// EU3D B200 hot path: handle, memory, launches and the C ABI declared in
// include/eu3d_gpu.h.  One translation unit so that the mechanism lives in a
// single __constant__ object shared by every kernel.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "../../include/eu3d_gpu.h"
#include "bc.cuh"
#include "cell.cuh"
#include "common.cuh"
#include "flux.cuh"
#include "mlp.cuh"
#include "surrogate.cuh"
#include "train.cuh"
#include "tecplot.cuh"
#include "dlb.cuh"

using namespace eu3d;

namespace {

thread_local std::string g_err;
MechConst g_mech_loaded[1];
int g_mech_refs = 0;

int fail(int code, const std::string &msg)
{
    g_err = msg;
    return code;
}

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return fail(EU3D_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

struct StepKey {
    int react, type, timeadv, diff, bc_kind;
    double cfl, final_time;
    bool operator<(const StepKey &o) const
    {
        return std::tie(react, type, timeadv, diff, bc_kind, cfl, final_time) <
               std::tie(o.react, o.type, o.timeadv, o.diff, o.bc_kind, o.cfl, o.final_time);
    }
};

}  // namespace

// node spacings the reference's CFLcondition uses: node(1) - node(0) of each
// axis (src/Flowfield.cpp:244-246)
struct Spacing {
    double dx, dy, dz;
};

struct eu3d_handle {
    int dev = 0;
    cudaStream_t st = nullptr;
    Layout L{};
    int flux_bits = 64;
    unsigned quirks = 0;
    double *cs = nullptr, *cs0 = nullptr, *T = nullptr, *E = nullptr;
    void *rhs = nullptr;  // flux residual, NV fields in the primitives' precision
    void *prim = nullptr;
    int *nchem = nullptr;
    double *xn = nullptr, *yn = nullptr, *zn = nullptr;
    Spacing sp{};  // taken from the nodes at creation (read back, it cost each eu3d_cfl three blocking copies)
    double *scal = nullptr;  // [0] dt, [1] time
    double *partial = nullptr;
    int nparts = 0;     // persistent-queue blocks (fallback queue)
    int cfl_parts = 0;  // CFL reduction blocks (one partial triple each)
    Status *status = nullptr;
    double *inflow = nullptr;
    double *stage = nullptr;
    size_t stage_bytes = 0;
    double wedge[3] = {0, 0, 0};
    int wedge_on = 0;
    int4 *wedge_band = nullptr;  // solid cells the stencils reach, with their mirror sources
    int wedge_nband = 0;
    bool spec = false;  // mechanism equals the compiled-in H2_JA919 tables
    int flux_kz = 16;   // z planes walked by one flux block (set per grid at creation)
    int flux_stage = 2; // FP32 flux: 2 TMA ring (k_flux_ring), 1 staged by loads (k_flux_stage), 0 through L1
    CUtensorMap tq{};   // TMA map of the FP32 primitive array (k_flux_ring)
    bool tq_ok = false;
    int chem_queue = 1; // adaptive trapezoid on the persistent work queue (0: one thread per cell)
    int queue_blocks = 3;  // resident queue blocks per SM
    int sur_fused = 0;     // surrogate: network and apply in one kernel (1) or two kernels (0, faster)
    unsigned wait_tries = 1u << 19;  // bound of the flux ring's copy waits (eu3d_set_wait_limit)
    int adapt_queue = 0;   // FP64 adaptive chemistry on the persistent queue (1) or one thread per cell (0)
    int cell_blocks = 3;   // accepted (3 or 4) and reported; the stage updates run at CellShape's occupancy
    int gate_fused = 1;    // surrogate with its gate: the gate runs inside SSP-RK2's stage 2 (1) or on its own (0)
    bool sur_gated = false;  // the last stage 2 listed the active cells; the next surrogate step uses that list
    AdaptCfg acfg{0.02, 0.5, 1024};  // adaptive chemistry (EU3D_REACT_ADAPTIVE, surrogate fallback)
    double proj_eps = 1e-4;
    bool elements = false;  // element matrix loaded (eu3d_set_elements)
    bool rhs_applied = false;  // the next M_ADAPT launch finds the flux update decoded already
    int *qlist = nullptr, *qbins = nullptr;
    std::map<StepKey, cudaGraphExec_t> graphs;
    // per-kernel CUDA-event timing (eu3d_profile_enable)
    bool profile = false;
    struct ProfRec {
        const char *name;
        cudaEvent_t a, b;
    };
    std::vector<ProfRec> prof_pending;
    std::vector<cudaEvent_t> prof_pool;
    std::map<std::string, std::pair<double, long long>> prof_acc;
    // learned chemistry (eu3d_set_surrogate): network outputs, fallback list
    eu3d_surrogate *sur = nullptr;
    float *sur_out = nullptr;
    int *sur_list = nullptr, *sur_count = nullptr;
    double *sur_audit = nullptr;
    double *sur_res = nullptr;  // fallback results per list slot ((NS + 1) x sur_cap)
    int *sur_info = nullptr;    // fallback substep counts and flags per list slot
    long long sur_cap = 0;
    int sur_audit_stride = 0;
    int *sur_active = nullptr;  // cells the frozen-chemistry gate passes to the network
    double gate_T = 0.0, gate_y = 0.0;  // eu3d_set_surrogate_gate (gate_T = 0: off)
    unsigned gate_mask = 0;
    int gate_audit = 0;
    // result files (eu3d_write_tecplot): gathered columns on the device and in
    // pinned host memory, and the background writer
    double *tp_dev = nullptr, *tp_host = nullptr;
    int *tp_ldev = nullptr, *tp_lhost = nullptr;
    std::vector<double> tp_nodes;  // ghosted x, y, z node coordinates
    std::thread writer;
    std::string writer_err;
    // dynamic load balancing of the adaptive trapezoid (eu3d_chem_load, eu3d_dlb_*)
    long long *dlb_rowload = nullptr;  // per interior row, device
    std::vector<long long> dlb_rows;   // host copy of the last eu3d_chem_load
    DlbSegs dlb_segs{};                // the transfers this rank sends (rows, offsets in DLB_OUT fields)
    long long away_lo = 0, away_hi = 0;  // rows the next queue pass leaves to other ranks
    // guest store: cells received from other ranks, field stride g_cap
    long long g_cap = 0;
    double *g_cs = nullptr, *g_T = nullptr, *g_E = nullptr;
    int *g_nchem = nullptr, *g_list = nullptr, *g_bins = nullptr;
    void *g_prim = nullptr;
    // ... and its learned-chemistry fallback queue: audit temperatures,
    // per-slot results, list counts
    double *g_audit = nullptr, *g_res = nullptr;
    int *g_info = nullptr, *g_count = nullptr;
    // fallback load balancing: the list length of the last eu3d_sur_load, the
    // slots kept, the transfers this rank sends (segments of list slots)
    long long sdlb_total = -1, sdlb_keep = 0;  // -1: no eu3d_sur_load since the last SUR_PREDICT
    DlbGuestSegs sdlb_segs{};
};

namespace {

int prim_bytes(const eu3d_handle *h) { return h->flux_bits == 64 ? 8 : 4; }

cudaEvent_t prof_event(eu3d_handle *h)
{
    if (!h->prof_pool.empty()) {
        cudaEvent_t e = h->prof_pool.back();
        h->prof_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

// Brackets one kernel launch with CUDA events on the handle's stream while
// profiling is enabled (eu3d_step then runs without its graph).
struct ProfScope {
    eu3d_handle *h;
    const char *name;
    cudaEvent_t a = nullptr;
    ProfScope(eu3d_handle *hh, const char *n) : h(hh), name(n)
    {
        if (h->profile) {
            a = prof_event(h);
            cudaEventRecord(a, h->st);
        }
    }
    ~ProfScope()
    {
        if (h->profile && a) {
            cudaEvent_t b = prof_event(h);
            cudaEventRecord(b, h->st);
            h->prof_pending.push_back({name, a, b});
        }
    }
};

CellArgs cell_args(eu3d_handle *h)
{
    CellArgs a;
    a.L = h->L;
    a.quirks = h->quirks;
    a.cs = h->cs;
    a.rhs = h->rhs;
    a.T = h->T;
    a.E = h->E;
    a.cs0 = h->cs0;
    a.nchem = h->nchem;
    a.scal = h->scal;
    a.st = h->status;
    a.xn = h->xn;
    a.yn = h->yn;
    a.wedge[0] = h->wedge[0];
    a.wedge[1] = h->wedge[1];
    a.wedge[2] = h->wedge[2];
    a.wedge_on = h->wedge_on;
    a.qbins = h->qbins;
    a.acfg = h->acfg;
    a.proj_eps = h->proj_eps;
    a.rhs_applied = h->rhs_applied ? 1 : 0;
    return a;
}

// blocks of bx threads for kernels that take their cell from cell_of_thread
unsigned cell_blocks_of(const Layout &L, int bx)
{
    const long long segs = (long long)L.nj * L.nk * ((L.ni + 31) / 32);
    return (unsigned)((segs + bx / 32 - 1) / (bx / 32));
}

dim3 cell_grid(const Layout &L, int bx) { return dim3((L.ni + bx - 1) / bx, L.nj, L.nk); }

template <class P, int MODE, bool SPEC>
void launch_cell_mode(eu3d_handle *h, const CellArgs &a, P *q)
{
    constexpr int threads = CellShape<MODE>::THREADS;
    k_cell<P, MODE, SPEC><<<cell_blocks_of(h->L, threads), threads, 0, h->st>>>(a, q);
}

template <class P, bool SPEC>
void launch_cell_t(eu3d_handle *h, int mode)
{
    CellArgs a = cell_args(h);
    P *q = (P *)h->prim;
    static const char *names[] = {"cell_decode", "cell_adv",   "cell_imex",          "cell_trap0", "cell_trap1",
                                  "cell_rk1",    "cell_rk2",   "cell_nochem",        "cell_trap1_predict",
                                  "cell_adapt",  "cell_rk3_2", "cell_rk3_3"};
    ProfScope ps(h, names[mode]);
    switch (mode) {
    case M_DECODE: launch_cell_mode<P, M_DECODE, SPEC>(h, a, q); break;
    case M_ADV: launch_cell_mode<P, M_ADV, SPEC>(h, a, q); break;
    case M_IMEX: launch_cell_mode<P, M_IMEX, SPEC>(h, a, q); break;
    case M_TRAP0: launch_cell_mode<P, M_TRAP0, SPEC>(h, a, q); break;
    case M_TRAP1: launch_cell_mode<P, M_TRAP1, SPEC>(h, a, q); break;
    case M_RK_STAGE1: launch_cell_mode<P, M_RK_STAGE1, SPEC>(h, a, q); break;
    case M_RK_STAGE2: launch_cell_mode<P, M_RK_STAGE2, SPEC>(h, a, q); break;
    case M_NOCHEM: launch_cell_mode<P, M_NOCHEM, SPEC>(h, a, q); break;
    case M_ADAPT: launch_cell_mode<P, M_ADAPT, SPEC>(h, a, q); break;
    case M_RK3_STAGE2: launch_cell_mode<P, M_RK3_STAGE2, SPEC>(h, a, q); break;
    case M_RK3_STAGE3: launch_cell_mode<P, M_RK3_STAGE3, SPEC>(h, a, q); break;
    }
}

int queue_grid(const eu3d_handle *h)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->dev);
    return sms * h->queue_blocks;
}

// Adaptive trapezoid on the work queue: predict + bin, then offsets, list,
// workers.  Between the two a multi-rank driver may hand rows to other ranks
// (eu3d_dlb_pack), which the list then leaves out.
template <class P, bool SPEC>
void trap1_predict(eu3d_handle *h)
{
    CellArgs a = cell_args(h);
    cudaMemsetAsync(h->qbins, 0, QBINS * sizeof(int), h->st);
    h->away_lo = h->away_hi = 0;
    h->dlb_segs.n = 0;  // a new prediction: no rows selected yet
    ProfScope ps(h, "trap1_predict");
    launch_cell_mode<P, M_TRAP1_PREDICT, SPEC>(h, a, (P *)h->prim);
}

template <class P, bool SPEC>
void trap1_work(eu3d_handle *h)
{
    CellArgs a = cell_args(h);
    ChemQueue qu{h->qlist, h->qbins, h->away_lo, h->away_hi};
    {
        ProfScope ps(h, "trap1_list");
        k_queue_scan<<<1, 32, 0, h->st>>>(qu);
        k_queue_scatter<<<cell_grid(h->L, 128), 128, 0, h->st>>>(a, qu);
    }
    {
        ProfScope ps(h, "trap1_work");
        k_trap1_work<P, SPEC><<<queue_grid(h), 128, 0, h->st>>>(a, (P *)h->prim, qu);
    }
}

template <class P, bool SPEC>
void launch_trap1_queue(eu3d_handle *h)
{
    trap1_predict<P, SPEC>(h);
    trap1_work<P, SPEC>(h);
}

// one half of the queued adaptive trapezoid: 0 predict, 1 work
int trap1_part(eu3d_handle *h, int half)
{
    if (h->flux_bits == 64) {
        if (h->spec)
            half ? trap1_work<double, true>(h) : trap1_predict<double, true>(h);
        else
            half ? trap1_work<double, false>(h) : trap1_predict<double, false>(h);
    } else {
        if (h->spec)
            half ? trap1_work<float, true>(h) : trap1_predict<float, true>(h);
        else
            half ? trap1_work<float, false>(h) : trap1_predict<float, false>(h);
    }
    CK(cudaGetLastError());
    return EU3D_OK;
}

template <class P>
void launch_cell(eu3d_handle *h, int mode)
{
    if (mode == M_TRAP1 && h->chem_queue && h->qlist) {
        if (h->spec)
            launch_trap1_queue<P, true>(h);
        else
            launch_trap1_queue<P, false>(h);
        return;
    }
    if (h->spec)
        launch_cell_t<P, true>(h, mode);
    else
        launch_cell_t<P, false>(h, mode);
}

int ensure_queue(eu3d_handle *h)
{
    if (h->qlist) return EU3D_OK;
    CK(cudaMalloc(&h->qlist, (size_t)h->L.interior_cells() * sizeof(int)));
    CK(cudaMalloc(&h->qbins, (3 * QBINS + 2) * sizeof(int)));
    CK(cudaMemset(h->qbins, 0, (3 * QBINS + 2) * sizeof(int)));
    return EU3D_OK;
}

int cell_op(eu3d_handle *h, int mode)
{
    if (h->flux_bits == 64)
        launch_cell<double>(h, mode);
    else
        launch_cell<float>(h, mode);
    CK(cudaGetLastError());
    return EU3D_OK;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda)
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled()
{
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *f = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)f;
        else
            cudaGetLastError();
    }
    return fn;
}

// TMA map of the FP32 primitives as a 4-D tensor {x: px, y: NJ, z: NK,
// field: NPRIM}, box {36, 12, 1, 16}: one tile plane with its halo.
bool make_prim_map(eu3d_handle *h)
{
    EncodeTiledFn enc = encode_tiled();
    if (!enc || h->flux_bits != 32 || h->L.bc != 2) return false;
    const Layout &L = h->L;
    const cuuint64_t dims[4] = {(cuuint64_t)L.px, (cuuint64_t)L.NJ, (cuuint64_t)L.NK, (cuuint64_t)NPRIM};
    const cuuint64_t strides[3] = {(cuuint64_t)L.px * 4, (cuuint64_t)L.px * L.NJ * 4, (cuuint64_t)L.fs * 4};
    const cuuint32_t box[4] = {FluxRing::BOX[0], FluxRing::BOX[1], FluxRing::BOX[2], FluxRing::BOX[3]};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return enc(&h->tq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, h->prim, dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// blocks of the FP64 flux with 32 x 7 tiles and walks of kz planes
long long flux64_blocks(const Layout &L, int kz)
{
    return (long long)((L.ni + FT_X - 1) / FT_X) * ((L.nj + 6) / 7) * ((L.nk + kz - 1) / kz);
}

// z planes a block of the FP64 flux walks: the setting flux_kz, halved while the
// tiles leave fewer than two waves of two blocks an SM, down to one plane.  A
// walk of 16 already hides its extra z face (240 x 256 x 200: 2.32 ms, 2.43 with
// 4 planes, 2.90 with 1); on smaller grids the blocks count for more (160^3: 0.75
// ms with 4, 0.77 with 16; 121 x 81 x 61: 137 us with 2 or 4, 154 with 1, 178 with
// 16; 241 x 81 x 2: 15.4 us with 1, 19.7 with 2; 4000 x 2 x 2: 12.6, 16.7).  Taken
// at the launch, so that no setting, the autotuner's candidates among them, leaves
// a small grid to a few long walks.
int flux64_walk(const Layout &L, int kz)
{
    while (kz > 1 && flux64_blocks(L, kz) < 2LL * 2 * 148) kz /= 2;
    return kz;
}

// FP64 flux launch: tiles of 32 x 7 columns, two blocks of 8 warps per SM (128
// registers a thread) where the grid fills the GPU; where it leaves less than a
// wave of them, 32 x 3 tiles, whose shorter blocks spread over more SMs.  7 and 3
// rows, us a launch: 4000 x 2 x 2 16.7, 12.6; 241 x 81 x 2 18.6, 15.7; 64 x 64 x 40
// 44.4, 43.2 (above the line); 121 x 81 x 61 138, 141; 512 x 256 x 2 64.5, 80.2;
// 160^3 777, 860.  (78, 87 us and 5.0 to 6.4 ms before the division-free faces, first
// two and last.)
template <int DIFF, bool SQ, int TY, int NB>
void launch_flux64(eu3d_handle *h, const FluxSolid &wedge, int kz)
{
    const Layout &L = h->L;
    FieldBase qf;
    for (int f = 0; f < NPRIM; f++) qf.p[f] = (const char *)((const double *)h->prim + f * L.fs);
    const dim3 g((L.ni + FT_X - 1) / FT_X, (L.nj + TY - 1) / TY, (L.nk + kz - 1) / kz);
    k_flux64<DIFF, SQ, TY, NB><<<g, dim3(FT_X, TY + 1), Flux64<TY>::SMEM, h->st>>>(L, qf, h->xn, h->yn, h->zn, h->scal,
                                                                                  (double *)h->rhs, kz, wedge);
}

template <class P, int DIFF>
void launch_adv_t(eu3d_handle *h)
{
    const int sq = (h->quirks & EU3D_Q_SPECIES_FACES) ? 1 : 0;
    const Layout &L = h->L;
    const int kz = h->flux_kz;
    const FluxSolid wedge{h->wedge[0], h->wedge[1], h->wedge[2], h->wedge_on};
    ProfScope ps(h, "advection");
    if constexpr (sizeof(P) == 8) {
        const int kw = flux64_walk(L, kz);
        if (flux64_blocks(L, kw) < 2 * 148)
            sq ? launch_flux64<DIFF, true, 3, 4>(h, wedge, kw) : launch_flux64<DIFF, false, 3, 4>(h, wedge, kw);
        else
            sq ? launch_flux64<DIFF, true, 7, 2>(h, wedge, kw) : launch_flux64<DIFF, false, 7, 2>(h, wedge, kw);
    } else {
        const float *qf = (const float *)h->prim;
        if (h->flux_stage == 2 && h->tq_ok) {
            dim3 gs((L.ni + FT_X - 1) / FT_X, (L.nj + FR_TY - 1) / FR_TY, (L.nk + kz - 1) / kz);
            dim3 bs(FT_X, FR_TY + 2);
            if (sq)
                k_flux_ring<DIFF, true><<<gs, bs, FluxRing::SMEM, h->st>>>(
                    h->tq, L, qf, h->xn, h->yn, h->zn, h->scal, (float *)h->rhs, kz, h->status, wedge, h->wait_tries);
            else
                k_flux_ring<DIFF, false><<<gs, bs, FluxRing::SMEM, h->st>>>(
                    h->tq, L, qf, h->xn, h->yn, h->zn, h->scal, (float *)h->rhs, kz, h->status, wedge, h->wait_tries);
            return;
        }
        if (h->flux_stage) {
            dim3 gs((L.ni + FT_X - 1) / FT_X, (L.nj + FS_TY - 1) / FS_TY, (L.nk + kz - 1) / kz);
            dim3 bs(FT_X, FS_TY + 2);
            k_flux_stage<DIFF><<<gs, bs, FluxStage::SMEM, h->st>>>(L, qf, h->xn, h->yn, h->zn, h->scal, (float *)h->rhs, sq,
                                                                   kz, wedge);
            return;
        }
        dim3 g((L.ni + FT_X - 1) / FT_X, (L.nj + FluxTile::TY - 1) / FluxTile::TY, (L.nk + kz - 1) / kz);
        k_flux_tile<DIFF><<<g, dim3(FT_X, FluxTile::TY + 2), FluxTile::SMEM, h->st>>>(L, qf, h->xn, h->yn, h->zn, h->scal,
                                                                                  (float *)h->rhs, sq, kz, wedge);
    }
}

template <class P>
void launch_adv(eu3d_handle *h, int diff)
{
    if (diff == EU3D_DIFF_MUSCL1)
        launch_adv_t<P, EU3D_DIFF_MUSCL1>(h);
    else if (diff == EU3D_DIFF_MUSCL2)
        launch_adv_t<P, EU3D_DIFF_MUSCL2>(h);
    else
        launch_adv_t<P, EU3D_DIFF_WENO>(h);
}

// dynamic shared memory of the tiled flux kernels (above the 48 KB default);
// the TMA ring kernel runs two blocks per SM
template <int DIFF>
void flux_attributes()
{
    for (auto k : {k_flux_ring<DIFF, false>, k_flux_ring<DIFF, true>}) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FluxRing::SMEM);
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    }
    cudaFuncSetAttribute(k_flux_stage<DIFF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FluxStage::SMEM);
    cudaFuncSetAttribute(k_flux_tile<DIFF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FluxTile::SMEM);
    for (auto k : {k_flux64<DIFF, false, 7, 2>, k_flux64<DIFF, true, 7, 2>})
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Flux64<7>::SMEM);
    static_assert(Flux64<3>::SMEM <= 48 * 1024, "the small tile fits the default shared memory");
}

int adv_op(eu3d_handle *h, int timeadv, int diff)
{
    if (timeadv == EU3D_ADV_TVD_RK3) return EU3D_OK;  // TimeAdv::TVD_RK3 leaves RHS as it is
    if (h->flux_bits == 64)
        launch_adv<double>(h, diff);
    else
        launch_adv<float>(h, diff);
    CK(cudaGetLastError());
    return EU3D_OK;
}

template <class P>
void launch_ghost(eu3d_handle *h, int kind)
{
    GhostArgs a;
    a.L = h->L;
    a.quirks = h->quirks;
    a.T = h->T;
    a.E = h->E;
    a.inflow = h->inflow;
    a.kind = kind;
    P *q = (P *)h->prim;
    const Layout &L = h->L;
    const int g = 2 * L.bc;
    if (kind != EU3D_BC_NONE && std::min({L.ni, L.nj, L.nk}) < L.bc) {
        // an extent of one cell: mirror images are ghost cells, filled in order
        auto blocks = [](long long lines) { return (unsigned)((lines + 127) / 128); };
        ProfScope ps(h, "ghost");
        k_ghost_line<P, 0><<<blocks((long long)L.nj * L.nk), 128, 0, h->st>>>(a, q);
        k_ghost_line<P, 1><<<blocks((long long)L.NI * L.nk), 128, 0, h->st>>>(a, q);
        k_ghost_line<P, 2><<<blocks((long long)L.NI * L.NJ), 128, 0, h->st>>>(a, q);
    } else if (kind != EU3D_BC_NONE) {
        const long long n = (long long)g * (L.NI * L.NJ + L.NI * L.nk + L.nj * L.nk);
        ProfScope ps(h, "ghost");
        k_ghost<P><<<(unsigned)((n + 127) / 128), 128, 0, h->st>>>(a, q);
    }
    if (h->wedge_on && h->wedge_nband > 0) {
        const double tn = h->wedge[2];
        const double cs = 1.0 / sqrt(1.0 + tn * tn), sn = tn * cs;
        dim3 gw((h->wedge_nband + 127) / 128, L.NK);
        ProfScope ps(h, "wedge");
        k_wedge_band<P><<<gw, 128, 0, h->st>>>(a, q, h->wedge_band, h->wedge_nband, -sn, cs);
    }
}

int ghost_op(eu3d_handle *h, int kind)
{
    if (kind < EU3D_BC_RSBI || kind > EU3D_BC_NONE) return fail(EU3D_ERR_ARG, "unknown boundary kind");
    if (kind == EU3D_BC_ODM && !h->inflow) return fail(EU3D_ERR_STATE, "ODM boundary needs eu3d_set_inflow first");
    if (h->flux_bits == 64)
        launch_ghost<double>(h, kind);
    else
        launch_ghost<float>(h, kind);
    CK(cudaGetLastError());
    return EU3D_OK;
}

template <class P>
void launch_cfl(eu3d_handle *h, const Spacing &sp, double cfl, double final_time, int advance)
{
    const int use_z = (h->quirks & EU3D_Q_CFL_NO_Z) ? 0 : 1;
    // one 128-cell segment a warp while the grid has fewer than cfl_parts blocks of them
    const Layout &L = h->L;
    const long long units = (long long)L.nj * L.nk * ((L.ni + CFL_SEG - 1) / CFL_SEG);
    const int blocks = (int)std::min<long long>(h->cfl_parts, (units + CFL_WARPS - 1) / CFL_WARPS);
    ProfScope ps(h, "cfl");
    k_cfl<P><<<blocks, 32 * CFL_WARPS, 0, h->st>>>(L, (const P *)h->prim, use_z, h->xn, h->yn, h->wedge[0], h->wedge[1],
                                                  h->wedge[2], h->wedge_on, h->partial, h->cfl_parts, sp.dx, sp.dy, sp.dz,
                                                  cfl, final_time, h->scal, advance);
}

int cfl_op(eu3d_handle *h, double cfl, double final_time, const Spacing &sp, int advance = 1)
{
    if (h->flux_bits == 64)
        launch_cfl<double>(h, sp, cfl, final_time, advance);
    else
        launch_cfl<float>(h, sp, cfl, final_time, advance);
    CK(cudaGetLastError());
    return EU3D_OK;
}

// host reference layout <-> device SoA layout
// Host arrays are the reference's (i, j, k[, field]) order -- field fastest,
// then k -- and the device fields are x-fastest planes, so an upload or a
// download is a transpose.  One block moves a tile of 32 cells in x by 8
// planes in z of one row j, every field, through shared memory: the host
// side is read (written) in runs of 8 n contiguous values per x cell, the
// device side in 32-cell rows.
constexpr int XFER_XT = 32, XFER_KT = 8;

template <class D>
__global__ void __launch_bounds__(256) k_h2d(Layout L, const double *__restrict__ stage, int n, D *__restrict__ dst,
                                             long long dfs)
{
    __shared__ double tile[NV][XFER_KT][XFER_XT + 1];
    const int i0 = blockIdx.x * XFER_XT, j = blockIdx.y, k0 = blockIdx.z * XFER_KT;
    const int ni = min(XFER_XT, L.NI - i0), nk = min(XFER_KT, L.NK - k0), run = nk * n;
    for (int e = threadIdx.x; e < ni * run; e += blockDim.x) {
        const int il = e / run, r = e - il * run, kl = r / n, s = r - kl * n;
        tile[s][kl][il] = stage[(((long long)(i0 + il) * L.NJ + j) * L.NK + k0) * n + r];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < XFER_XT * XFER_KT * n; e += blockDim.x) {
        const int il = e % XFER_XT, r = e / XFER_XT, kl = r % XFER_KT, s = r / XFER_KT;
        if (il < ni && kl < nk) dst[s * dfs + L.at(i0 + il, j, k0 + kl)] = (D)tile[s][kl][il];
    }
}

template <class S>
__global__ void __launch_bounds__(256) k_d2h(Layout L, const S *__restrict__ src, long long sfs, int n,
                                             double *__restrict__ stage)
{
    __shared__ double tile[NV][XFER_KT][XFER_XT + 1];
    const int i0 = blockIdx.x * XFER_XT, j = blockIdx.y, k0 = blockIdx.z * XFER_KT;
    const int ni = min(XFER_XT, L.NI - i0), nk = min(XFER_KT, L.NK - k0), run = nk * n;
    for (int e = threadIdx.x; e < XFER_XT * XFER_KT * n; e += blockDim.x) {
        const int il = e % XFER_XT, r = e / XFER_XT, kl = r % XFER_KT, s = r / XFER_KT;
        if (il < ni && kl < nk) tile[s][kl][il] = (double)src[s * sfs + L.at(i0 + il, j, k0 + kl)];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < ni * run; e += blockDim.x) {
        const int il = e / run, r = e - il * run, kl = r / n, s = r - kl * n;
        stage[(((long long)(i0 + il) * L.NJ + j) * L.NK + k0) * n + r] = tile[s][kl][il];
    }
}

dim3 xfer_grid(const Layout &L)
{
    return dim3((L.NI + XFER_XT - 1) / XFER_XT, L.NJ, (L.NK + XFER_KT - 1) / XFER_KT);
}

// derived download fields: C = sqrt(G P / D); Mc = CS_s / Mw * 1000; Di = CS_s
template <class P>
__global__ void k_derive(Layout L, const P *__restrict__ q, const double *__restrict__ cs, int what, double *stage, int n)
{
    const long long cells = (long long)L.NI * L.NJ * L.NK;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < cells * n;
         t += (long long)gridDim.x * blockDim.x) {
        const long long hc = t / n;
        const int s = (int)(t % n);
        const int k = (int)(hc % L.NK), j = (int)((hc / L.NK) % L.NJ), i = (int)(hc / ((long long)L.NK * L.NJ));
        const long long c = L.at(i, j, k);
        double v;
        if (what == EU3D_FIELD_C)
            v = sqrt((double)q[PG * L.fs + c] * (double)q[PP * L.fs + c] / (double)q[PD * L.fs + c]);
        else if (what == EU3D_FIELD_MC)
            v = cs[s * L.fs + c] / cM.mw[s] * 1000;
        else
            v = cs[s * L.fs + c];
        stage[t] = v;
    }
}

// FieldInitial's completion of a primitive state (src/Flowfield.cpp:193-229)
struct Uniform {
    double P, T, U, V, W, Y[NS];
};

template <class P>
__global__ void k_init_uniform(Layout L, Uniform u, unsigned quirks, P *q, double *cs, double *T, double *E)
{
    const long long cells = (long long)L.NK * L.NJ * L.px;
    const TPow p = tpow(u.T, quirks);
    double sdiv = 0.0, cp = 0.0, h = 0.0, e = 0.0;
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const double cpi = cM.ri[s] * cp_r(s, p), hi = cM.ri[s] * h_r(s, p);
        sdiv += u.Y[s] / cM.mw[s];
        cp += cpi * u.Y[s];
        h += u.Y[s] * hi;
        e += u.Y[s] * (hi - cM.ri[s] * u.T);
    }
    const double Rgas = R_GAS * 1000 / (1.0 / sdiv);
    const double D = u.P / (Rgas * u.T);
    const double Cp = cp * 1000, H = h * 1000, En = e * 1000;
    const double G = Cp / (Cp - R_GAS * sdiv * 1000);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < cells; c += (long long)gridDim.x * blockDim.x) {
        q[PD * L.fs + c] = (P)D;
        q[PU * L.fs + c] = (P)u.U;
        q[PV * L.fs + c] = (P)u.V;
        q[PW * L.fs + c] = (P)u.W;
        q[PP * L.fs + c] = (P)u.P;
        q[PH * L.fs + c] = (P)H;
        q[PG * L.fs + c] = (P)G;
#pragma unroll
        for (int s = 0; s < NS; s++) {
            q[(PY + s) * L.fs + c] = (P)u.Y[s];
            cs[s * L.fs + c] = D * u.Y[s];
        }
        cs[NS * L.fs + c] = D * u.U;
        cs[(NS + 1) * L.fs + c] = D * u.V;
        cs[(NS + 2) * L.fs + c] = D * u.W;
        cs[(NS + 3) * L.fs + c] = D * En + 0.5 * (u.U * u.U + u.V * u.V + u.W * u.W) * D;
        T[c] = u.T;
        E[c] = En;
    }
}

int field_shape(int field, int *n)
{
    switch (field) {
    case EU3D_FIELD_YI:
    case EU3D_FIELD_MC:
    case EU3D_FIELD_DI: *n = NS; return 0;
    case EU3D_FIELD_CS:
    case EU3D_FIELD_RHS: *n = NV; return 0;
    default:
        if (field < 0 || field >= EU3D_FIELD_COUNT) return -1;
        *n = 1;
        return 0;
    }
}

int prim_index(int field)
{
    switch (field) {
    case EU3D_FIELD_U: return PU;
    case EU3D_FIELD_V: return PV;
    case EU3D_FIELD_W: return PW;
    case EU3D_FIELD_P: return PP;
    case EU3D_FIELD_D: return PD;
    case EU3D_FIELD_H: return PH;
    case EU3D_FIELD_GAMMA: return PG;
    case EU3D_FIELD_YI: return PY;
    default: return -1;
    }
}

int grid_blocks(long long n) { return (int)std::min<long long>((n + 255) / 256, 148LL * 32); }

int validate_mech(const eu3d_desc *d, MechConst &m)
{
    memset(&m, 0, sizeof(m));
    for (int r = 0; r < 2; r++)
        for (int k = 0; k < 9; k++)
            for (int s = 0; s < NS; s++) m.c[r][k][s] = (r ? d->coeff1 : d->coeff0)[k * NS + s];
    for (int s = 0; s < NS; s++) {
        if (!(d->mw[s] > 0)) return fail(EU3D_ERR_ARG, "molar masses must be positive");
        m.mw[s] = d->mw[s];
        m.ri[s] = R_GAS / d->mw[s];
        m.imw[s] = 1.0 / d->mw[s];
    }
    for (int r = 0; r < NR; r++) {
        m.af[r] = d->af[r];
        m.bf[r] = d->bf[r];
        m.eaf[r] = d->eaf[r];
        double xr = 0.0;
        int tb = 0;
        for (int s = 0; s < NS; s++) {
            const double f = d->stoi_f[s * NR + r], b = d->stoi_b[s * NR + r];
            if (!(f == 0 || f == 1 || f == 2) || !(b == 0 || b == 1 || b == 2))
                return fail(EU3D_ERR_ARG, "stoichiometric coefficients must be 0, 1 or 2");
            m.sf[s][r] = f;
            m.sb[s][r] = b;
            m.tb[s][r] = d->react_tb[s * NR + r];
            m.nu[s][r] = b - f;
            xr += (b - f);
            tb |= d->react_tb[s * NR + r] != 0;
        }
        m.xr[r] = xr;
        m.p0xr[r] = pow((P0 * 1e-6), xr);
        m.has_tb[r] = tb;
        if (!(xr == 0 || xr == 1 || xr == -1)) return fail(EU3D_ERR_ARG, "net molecularity change must be -1, 0 or 1");
    }
    return EU3D_OK;
}

void free_handle(eu3d_handle *h)
{
    for (auto &r : h->prof_pending) {
        cudaEventDestroy(r.a);
        cudaEventDestroy(r.b);
    }
    for (auto e : h->prof_pool) cudaEventDestroy(e);
    for (auto &g : h->graphs) cudaGraphExecDestroy(g.second);
    h->graphs.clear();
    void *ptrs[] = {h->cs,      h->rhs,    h->cs0,    h->T,       h->E,         h->prim,
                    h->nchem,   h->xn,     h->yn,     h->zn,      h->scal,      h->partial,
                    h->status,  h->inflow, h->stage,  h->sur_out, h->sur_list,  h->sur_count,
                    h->sur_audit, h->qlist,   h->qbins,  h->wedge_band, h->dlb_rowload, h->g_cs,
                    h->g_T,     h->g_E,    h->g_nchem, h->g_list, h->g_bins,  h->g_prim, h->sur_active,
                    h->sur_res, h->sur_info, h->g_audit, h->g_res, h->g_info, h->g_count};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (h->writer.joinable()) h->writer.join();
    if (h->tp_dev) cudaFree(h->tp_dev);
    if (h->tp_ldev) cudaFree(h->tp_ldev);
    if (h->tp_host) cudaFreeHost(h->tp_host);
    if (h->tp_lhost) cudaFreeHost(h->tp_lhost);
    if (h->st) cudaStreamDestroy(h->st);
    delete h;
}

int ensure_stage(eu3d_handle *h, size_t bytes)
{
    if (h->stage_bytes >= bytes) return EU3D_OK;
    if (h->stage) cudaFree(h->stage);
    h->stage = nullptr;
    h->stage_bytes = 0;
    CK(cudaMalloc(&h->stage, bytes));
    h->stage_bytes = bytes;
    return EU3D_OK;
}

// learned chemistry step (sur_host.cuh), whole or one half: SUR_HALF_PREDICT
// runs everything up to the fallback list (the flux update, gate, network and
// apply), SUR_HALF_WORK the fallback queue on the list slots kept (all of
// them unless eu3d_sdlb_pack sent some away)
constexpr int SUR_HALF_PREDICT = 1, SUR_HALF_WORK = 2, SUR_HALF_BOTH = 3;
int sur_chem_op(eu3d_handle *h, bool decoded, int half = SUR_HALF_BOTH);
// SSP-RK2 stage 2 with the surrogate's frozen-chemistry gate fused in (sur_host.cuh)
int rk2_gate_op(eu3d_handle *h);

bool is_rk(int timeadv) { return timeadv == EU3D_ADV_SSPRK2 || timeadv == EU3D_ADV_SSPRK3; }
int rk_stages(int timeadv) { return timeadv == EU3D_ADV_SSPRK2 ? 2 : timeadv == EU3D_ADV_SSPRK3 ? 3 : 1; }

// The step after the CFL and the first ghost fill, in parts so that a
// multi-rank driver can exchange x-slab halos between them (eu3d_step_part):
// the advection stage (SSP-RK: stage 1), each further SSP-RK stage after its
// own ghost fill, and the chemistry.
int stage1_op(eu3d_handle *h, const eu3d_step_desc *s)
{
    int rc;
    h->sur_gated = false;
    if (is_rk(s->timeadv)) {
        if ((rc = adv_op(h, EU3D_ADV_EE, s->diff))) return rc;
        return cell_op(h, M_RK_STAGE1);
    }
    return adv_op(h, s->timeadv, s->diff);
}

// stage 2 or 3 of an SSP-RK step; the last stage leaves RHS zero for the chemistry
int stage_op(eu3d_handle *h, const eu3d_step_desc *s, int stage)
{
    int rc;
    if ((rc = adv_op(h, EU3D_ADV_EE, s->diff))) return rc;
    const int mode = s->timeadv == EU3D_ADV_SSPRK2 ? M_RK_STAGE2 : stage == 2 ? M_RK3_STAGE2 : M_RK3_STAGE3;
    // a surrogate step with its gate on lists its active cells in stage 2
    if (mode == M_RK_STAGE2 && s->react == EU3D_REACT_SURROGATE && h->sur && h->gate_T > 0.0 && h->gate_fused)
        rc = rk2_gate_op(h);
    else
        rc = cell_op(h, mode);
    if (rc) return rc;
    if (stage == rk_stages(s->timeadv))
        CK(cudaMemsetAsync(h->rhs, 0, (size_t)NV * h->L.fs * prim_bytes(h), h->st));
    return EU3D_OK;
}

// Cell list and queue buffers shared by the surrogate's fallback and the
// queued adaptive chemistry (allocated outside any stream capture).
int ensure_cell_list(eu3d_handle *h)
{
    const long long n = h->L.interior_cells();
    if (h->L.fs > (long long)SUR_CELL_MASK) return fail(EU3D_ERR_ARG, "grid too large for the cell list");
    if (h->sur_cap < n) {
        CK(cudaStreamSynchronize(h->st));
        void *ptrs[] = {h->sur_out, h->sur_list, h->sur_audit, h->sur_active, h->sur_res, h->sur_info};
        for (void *q : ptrs)
            if (q) cudaFree(q);
        h->sur_out = nullptr;
        h->sur_list = nullptr;
        h->sur_audit = nullptr;
        h->sur_active = nullptr;
        h->sur_res = nullptr;
        h->sur_info = nullptr;
        h->sur_cap = 0;
        CK(cudaMalloc(&h->sur_out, (size_t)n * SUR_NOUT * sizeof(float)));
        CK(cudaMalloc(&h->sur_list, (size_t)n * sizeof(int)));
        CK(cudaMalloc(&h->sur_audit, (size_t)n * sizeof(double)));
        CK(cudaMalloc(&h->sur_active, (size_t)n * sizeof(int)));
        CK(cudaMalloc(&h->sur_res, (size_t)n * (NS + 1) * sizeof(double)));
        CK(cudaMalloc(&h->sur_info, (size_t)n * sizeof(int)));
        h->sur_cap = n;
    }
    if (!h->sur_count) CK(cudaMalloc(&h->sur_count, 4 * sizeof(int)));
    return EU3D_OK;
}

// FP64 adaptive chemistry on the persistent queue (tuning adapt_queue): every
// fluid cell is listed and the surrogate's fallback workers integrate them,
// one cell per lane with refill, so a warp never waits for the slowest cell
// of a fixed batch.  Same split step and arithmetic as k_cell<M_ADAPT>.
template <class P, bool SPEC>
void adapt_queue_t(eu3d_handle *h, bool decoded)
{
    const Layout &L = h->L;
    P *q = (P *)h->prim;
    cudaMemsetAsync(h->sur_count, 0, 4 * sizeof(int), h->st);
    if (!decoded) launch_cell_t<P, SPEC>(h, M_ADV);
    SurQueue qu{h->sur_list, h->sur_count, h->sur_audit, L.interior_cells(), h->sur_res, h->sur_info};
    {
        ProfScope ps(h, "adapt_list");
        k_list_fluid<<<cell_grid(L, 256), 256, 0, h->st>>>(cell_args(h), qu);
    }
    {
        ProfScope ps(h, "adapt_queue");
        k_sur_fallback<P, SPEC><<<h->nparts, 128, 0, h->st>>>(cell_args(h), q, qu);
    }
    ProfScope ps(h, "adapt_finish");
    k_sur_fallback_finish<P, SPEC><<<FALLBACK_FINISH_BLOCKS, 128, 0, h->st>>>(cell_args(h), q, qu);
}

int adapt_queue_op(eu3d_handle *h, bool decoded)
{
    if (!h->sur_count) return fail(EU3D_ERR_STATE, "adaptive queue buffers missing");
    if (h->flux_bits == 64) {
        if (h->spec) adapt_queue_t<double, true>(h, decoded);
        else adapt_queue_t<double, false>(h, decoded);
    } else {
        if (h->spec) adapt_queue_t<float, true>(h, decoded);
        else adapt_queue_t<float, false>(h, decoded);
    }
    CK(cudaGetLastError());
    return EU3D_OK;
}

int react_op(eu3d_handle *h, const eu3d_step_desc *s)
{
    switch (s->react) {
    case EU3D_REACT_IMEX: return cell_op(h, M_IMEX);
    case EU3D_REACT_TRAPEZOID: return cell_op(h, s->type == 0 ? M_TRAP0 : M_TRAP1);
    case EU3D_REACT_NONE:
        // Euler::DNN (src/Euler.cpp:773-780): Update_after_Adv, then Explicit()
        return cell_op(h, M_NOCHEM);
    // after SSP-RK the state is decoded and RHS holds zeros already
    case EU3D_REACT_SURROGATE: return sur_chem_op(h, is_rk(s->timeadv));
    case EU3D_REACT_ADAPTIVE: {
        if (h->adapt_queue) return adapt_queue_op(h, is_rk(s->timeadv));
        h->rhs_applied = is_rk(s->timeadv);
        const int rc = cell_op(h, M_ADAPT);
        h->rhs_applied = false;
        return rc;
    }
    default: return fail(EU3D_ERR_ARG, "unsupported reaction scheme for eu3d_step");
    }
}

int enqueue_step(eu3d_handle *h, const eu3d_step_desc *s, const Spacing &sp)
{
    int rc;
    if (s->cfl != 0 && (rc = cfl_op(h, s->cfl, s->final_time, sp))) return rc;
    if ((rc = ghost_op(h, s->bc_kind))) return rc;
    if ((rc = stage1_op(h, s))) return rc;
    for (int stage = 2; stage <= rk_stages(s->timeadv); stage++) {
        if ((rc = ghost_op(h, s->bc_kind))) return rc;
        if ((rc = stage_op(h, s, stage))) return rc;
    }
    return react_op(h, s);
}

}  // namespace

// ---------------------------------------------------------------------------
// Allocation-free CFL time step (eu3d_cfl_noalloc).
//
// Some callers cannot allocate device memory: code that runs while another
// framework owns the device memory pool and forbids allocations, or code that
// must not call cudaMalloc/cudaFree because those calls synchronise the device
// and would stall work in flight.  For them this entry point computes the CFL
// step from device fields the caller already holds, writing dt and time into
// caller-owned device memory, and allocates nothing: its one piece of scratch
// memory -- the per-block partial minima of the reduction -- is the
// file-scope device array below.  Every GPU that loads the library keeps this
// array (8 KB) until the process exits.
namespace {

constexpr int NOALLOC_CFL_MAX_BLOCKS = 1024;
constexpr int NOALLOC_CFL_DEFAULT_BLOCKS = 148 * 4;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) double g_cfl_scratch[NOALLOC_CFL_MAX_BLOCKS];

// Device address of g_cfl_scratch per device.  In host code the symbol
// g_cfl_scratch names a host-side stand-in, not device memory, so kernels are
// given this address, obtained once per device with that device current.
// Atomic: host threads making their first call on one device at the same time
// may both look it up (the same value); neither reads a torn pointer.
std::atomic<double *> g_cfl_scratch_dev[NOALLOC_MAX_DEVICES] = {};

struct CflFields {
    const double *D, *U, *V, *W, *P, *G;
    int ni, nj, nk, bc;
    long long pitch, plane;
};

__global__ void k_cfl_fields_partial(CflFields f, double dx, double dy, double dz, int use_z, double *partial)
{
    const long long n = (long long)f.ni * f.nj * f.nk;
    double m = 1e10;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int i = f.bc + (int)(t % f.ni);
        const int j = f.bc + (int)((t / f.ni) % f.nj);
        const int k = f.bc + (int)(t / ((long long)f.ni * f.nj));
        const long long c = k * f.plane + j * f.pitch + i;
        const double C = sqrt(f.G[c] * f.P[c] / f.D[c]);
        const double a = dx / (fabs(f.U[c]) + C), b = dy / (fabs(f.V[c]) + C);
        double tmp = (b < a) ? b : a;
        if (use_z) {
            const double z = dz / (fabs(f.W[c]) + C);
            tmp = (z < tmp) ? z : tmp;
        }
        if (tmp < m) m = tmp;
    }
    __shared__ double sm[32];
    for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 1e10;
        for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_down_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) partial[blockIdx.x] = m;
    }
}

__global__ void k_cfl_fields_final(const double *partial, int nparts, double cfl, double final_time, double *dt_out,
                                   double *time_inout)
{
    double m = 1e10;
    for (int t = threadIdx.x; t < nparts; t += blockDim.x) m = fmin(m, partial[t]);
    __shared__ double sm[32];
    for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 1e10;
        for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_down_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) {
            double dt = cfl * m;
            if (*time_inout + dt > final_time) dt = final_time - *time_inout;
            *dt_out = dt;
            *time_inout += dt;
        }
    }
}

}  // namespace

extern "C" {

const char *eu3d_last_error(void) { return g_err.c_str(); }

int eu3d_create(const eu3d_desc *d, eu3d_handle **out)
{
    if (!d || !out) return fail(EU3D_ERR_ARG, "null argument");
    *out = nullptr;
    if (d->NS != NS || d->NR != NR) return fail(EU3D_ERR_ARG, "this build supports NS=9, NR=19");
    if (d->bc != 2) return fail(EU3D_ERR_ARG, "ghost width bc must be 2");
    if (d->ni < 1 || d->nj < 1 || d->nk < 1) return fail(EU3D_ERR_ARG, "grid extents must be positive");
    if (d->flux_bits != 64 && d->flux_bits != 32) return fail(EU3D_ERR_ARG, "flux_bits must be 64 or 32");
    if (!d->xnode || !d->ynode || !d->znode || !d->stoi_f || !d->stoi_b || !d->react_tb || !d->af || !d->bf ||
        !d->eaf || !d->coeff0 || !d->coeff1 || !d->mw)
        return fail(EU3D_ERR_ARG, "null table pointer");
    MechConst m;
    int rc = validate_mech(d, m);
    if (rc) return rc;
    CK(cudaSetDevice(d->device));
    if (g_mech_refs > 0 && memcmp(&m, &g_mech_loaded[0], sizeof(m)) != 0)
        return fail(EU3D_ERR_MECH, "a handle with different mechanism tables is alive");

    eu3d_handle *h = new eu3d_handle();
    h->dev = d->device;
    {
        using namespace h2ja919;
        bool same = true;
        for (int q = 0; q < NS * NR; q++)
            same = same && d->stoi_f[q] == K_STOI_F[q] && d->stoi_b[q] == K_STOI_B[q] && d->react_tb[q] == K_TB[q];
        for (int r = 0; r < NR; r++) same = same && d->af[r] == K_AF[r] && d->bf[r] == K_BF[r] && d->eaf[r] == K_EAF[r];
        for (int q = 0; q < 9 * NS; q++) same = same && d->coeff0[q] == K_C0[q] && d->coeff1[q] == K_C1[q];
        for (int q = 0; q < NS; q++) same = same && d->mw[q] == K_MW[q];
        const char *env = getenv("EU3D_GENERIC_CHEM");
        h->spec = same && !(env && env[0] == '1');
    }
    h->flux_bits = d->flux_bits;
    h->quirks = d->quirks;
    Layout &L = h->L;
    L.ni = d->ni;
    L.nj = d->nj;
    L.nk = d->nk;
    L.bc = d->bc;
    L.NI = d->ni + 2 * d->bc;
    L.NJ = d->nj + 2 * d->bc;
    L.NK = d->nk + 2 * d->bc;
    L.px = (L.NI + 31) / 32 * 32;
    L.fs = (long long)L.px * L.NJ * L.NK;
    // z planes per flux block: deep walks load fewer extra planes per cell
    // (one per block), but the grid should keep at least four waves of two
    // blocks per SM; 64 on the 512 x 256 x 256 ODW
    {
        const long long cols = (long long)((L.ni + 31) / 32) * ((L.nj + 7) / 8);
        int kz = 64;
        while (kz > 4 && cols * ((L.nk + kz - 1) / kz) < 4LL * 2 * 148) kz /= 2;
        if (d->flux_bits == 64) kz = 16;  // at most (flux64_walk)
        h->flux_kz = kz;
    }
    if ((long long)NPRIM * L.fs >= (1LL << 31)) {
        delete h;
        return fail(EU3D_ERR_ARG, "grid too large for one handle (primitive fields exceed 2^31 elements)");
    }
    const size_t f8 = (size_t)L.fs * sizeof(double);
#define ALLOC(p, bytes)                                                                    \
    do {                                                                                   \
        if (cudaMalloc((void **)&(p), (bytes)) != cudaSuccess) {                           \
            free_handle(h);                                                                \
            cudaGetLastError();                                                            \
            return fail(EU3D_ERR_NOMEM, "device allocation of " + std::to_string(bytes) + " bytes failed"); \
        }                                                                                  \
    } while (0)
    if (cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking) != cudaSuccess) {
        delete h;
        return fail(EU3D_ERR_CUDA, "stream creation failed");
    }
    ALLOC(h->cs, NV * f8);
    ALLOC(h->rhs, (size_t)NV * L.fs * prim_bytes(h));
    ALLOC(h->T, f8);
    ALLOC(h->E, f8);
    ALLOC(h->prim, (size_t)NPRIM * L.fs * prim_bytes(h));
    ALLOC(h->nchem, (size_t)L.fs * sizeof(int));
    ALLOC(h->xn, L.NI * sizeof(double));
    ALLOC(h->yn, L.NJ * sizeof(double));
    ALLOC(h->zn, L.NK * sizeof(double));
    ALLOC(h->scal, 8 * sizeof(double));
    h->nparts = 148 * 4;
    // CFL: 16 blocks of 8 warps per SM, each warp walking a few rows, keep
    // enough loads in flight to stream the six primitive fields
    h->cfl_parts = 148 * 16;
    ALLOC(h->partial, (3 * h->cfl_parts + 1) * sizeof(double));  // per block: largest |U|+C, |V|+C, |W|+C; a count
    ALLOC(h->status, sizeof(Status));
#undef ALLOC
    cudaMemsetAsync(h->cs, 0, NV * f8, h->st);
    cudaMemsetAsync(h->rhs, 0, (size_t)NV * L.fs * prim_bytes(h), h->st);
    cudaMemsetAsync(h->T, 0, f8, h->st);
    cudaMemsetAsync(h->E, 0, f8, h->st);
    cudaMemsetAsync(h->prim, 0, (size_t)NPRIM * L.fs * prim_bytes(h), h->st);
    cudaMemsetAsync(h->nchem, 0, (size_t)L.fs * sizeof(int), h->st);
    cudaMemsetAsync(h->scal, 0, 8 * sizeof(double), h->st);
    cudaMemsetAsync(h->partial, 0, (3 * h->cfl_parts + 1) * sizeof(double), h->st);
    cudaMemsetAsync(h->status, 0, sizeof(Status), h->st);
    h->sp = Spacing{d->xnode[1] - d->xnode[0], d->ynode[1] - d->ynode[0], d->znode[1] - d->znode[0]};
    cudaMemcpyAsync(h->xn, d->xnode, L.NI * sizeof(double), cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->yn, d->ynode, L.NJ * sizeof(double), cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->zn, d->znode, L.NK * sizeof(double), cudaMemcpyHostToDevice, h->st);
    {
        flux_attributes<EU3D_DIFF_MUSCL1>();
        flux_attributes<EU3D_DIFF_MUSCL2>();
        flux_attributes<EU3D_DIFF_WENO>();
        h->tq_ok = make_prim_map(h);
        if (!h->tq_ok) h->flux_stage = 1;
    }
    if (g_mech_refs == 0) {
        cudaError_t e = cudaMemcpyToSymbol(cM, &m, sizeof(m));
        if (e != cudaSuccess) {
            free_handle(h);
            return fail(EU3D_ERR_CUDA, std::string("mechanism upload: ") + cudaGetErrorString(e));
        }
        g_mech_loaded[0] = m;
    }
    g_mech_refs++;
    cudaError_t e = cudaStreamSynchronize(h->st);
    if (e != cudaSuccess) {
        g_mech_refs--;
        free_handle(h);
        return fail(EU3D_ERR_CUDA, std::string("create: ") + cudaGetErrorString(e));
    }
    *out = h;
    return EU3D_OK;
}

int eu3d_destroy(eu3d_handle *h)
{
    if (!h) return EU3D_OK;
    cudaSetDevice(h->dev);
    cudaStreamSynchronize(h->st);
    free_handle(h);
    if (g_mech_refs > 0) g_mech_refs--;
    return EU3D_OK;
}

void *eu3d_stream(eu3d_handle *h) { return h ? (void *)h->st : nullptr; }

// ------------------------------------------------------------ result files
int eu3d_write_wait(eu3d_handle *h)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    if (h->writer.joinable()) h->writer.join();
    if (!h->writer_err.empty()) {
        const std::string e = h->writer_err;
        h->writer_err.clear();
        return fail(EU3D_ERR_IO, e);
    }
    return EU3D_OK;
}

int eu3d_write_tecplot(eu3d_handle *h, const char *path, double wait_time, int background)
{
    if (!h || !path) return fail(EU3D_ERR_ARG, "null argument");
    int rc = eu3d_write_wait(h);  // one file at a time per handle
    if (rc) return rc;
    CK(cudaSetDevice(h->dev));
    const Layout &L = h->L;
    const long long n = L.interior_cells();
    if (!h->tp_dev) {
        CK(cudaMalloc(&h->tp_dev, (size_t)TP_COLS * n * sizeof(double)));
        CK(cudaMalloc(&h->tp_ldev, (size_t)n * sizeof(int)));
        CK(cudaHostAlloc(&h->tp_host, (size_t)TP_COLS * n * sizeof(double), cudaHostAllocDefault));
        CK(cudaHostAlloc(&h->tp_lhost, (size_t)n * sizeof(int), cudaHostAllocDefault));
    }
    const int blocks = (int)std::min<long long>((n + 255) / 256, 148 * 16);
    if (h->flux_bits == 64)
        k_tecplot_gather<double><<<blocks, 256, 0, h->st>>>(L, (const double *)h->prim, h->T, h->nchem, h->tp_dev,
                                                            h->tp_ldev);
    else
        k_tecplot_gather<float><<<blocks, 256, 0, h->st>>>(L, (const float *)h->prim, h->T, h->nchem, h->tp_dev,
                                                           h->tp_ldev);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(h->tp_host, h->tp_dev, (size_t)TP_COLS * n * sizeof(double), cudaMemcpyDeviceToHost, h->st));
    CK(cudaMemcpyAsync(h->tp_lhost, h->tp_ldev, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost, h->st));
    h->tp_nodes.resize((size_t)L.NI + L.NJ + L.NK);
    CK(cudaMemcpyAsync(h->tp_nodes.data(), h->xn, L.NI * sizeof(double), cudaMemcpyDeviceToHost, h->st));
    CK(cudaMemcpyAsync(h->tp_nodes.data() + L.NI, h->yn, L.NJ * sizeof(double), cudaMemcpyDeviceToHost, h->st));
    CK(cudaMemcpyAsync(h->tp_nodes.data() + L.NI + L.NJ, h->zn, L.NK * sizeof(double), cudaMemcpyDeviceToHost,
                       h->st));
    CK(cudaStreamSynchronize(h->st));  // the snapshot is on the host: the device may step on
    const std::string p(path);
    auto job = [h, p, wait_time, L]() {
        const double *nodes = h->tp_nodes.data();
        h->writer_err = tecplot::write(p.c_str(), L.ni, L.nj, L.nk, L.bc, nodes, nodes + L.NI, nodes + L.NI + L.NJ,
                                       h->tp_host, h->tp_lhost, wait_time);
    };
    if (background) {
        h->writer = std::thread(job);
        return EU3D_OK;
    }
    job();
    return eu3d_write_wait(h);
}

int eu3d_tecplot_write_host(const char *path, int ni, int nj, int nk, int bc, const double *xnode, const double *ynode,
                            const double *znode, const double *cols, const int *lcol, double wait_time)
{
    if (!path || !xnode || !ynode || !znode || !cols || !lcol) return fail(EU3D_ERR_ARG, "null argument");
    if (ni < 1 || nj < 1 || nk < 1 || bc < 0) return fail(EU3D_ERR_ARG, "bad extents");
    const std::string e = tecplot::write(path, ni, nj, nk, bc, xnode, ynode, znode, cols, lcol, wait_time);
    return e.empty() ? EU3D_OK : fail(EU3D_ERR_IO, e);
}



int eu3d_upload_field(eu3d_handle *h, int field, const double *host)
{
    if (!h || !host) return fail(EU3D_ERR_ARG, "null argument");
    int n;
    if (field_shape(field, &n) || field > EU3D_FIELD_RHS) return fail(EU3D_ERR_ARG, "field cannot be uploaded");
    const Layout &L = h->L;
    const long long cells = (long long)L.NI * L.NJ * L.NK;
    const size_t bytes = (size_t)cells * n * sizeof(double);
    int rc = ensure_stage(h, bytes);
    if (rc) return rc;
    CK(cudaMemcpyAsync(h->stage, host, bytes, cudaMemcpyHostToDevice, h->st));
    const dim3 xg = xfer_grid(L);
    const int pi = prim_index(field);
    if (pi >= 0) {
        if (h->flux_bits == 64)
            k_h2d<double><<<xg, 256, 0, h->st>>>(L, h->stage, n, (double *)h->prim + pi * L.fs, L.fs);
        else
            k_h2d<float><<<xg, 256, 0, h->st>>>(L, h->stage, n, (float *)h->prim + pi * L.fs, L.fs);
    } else if (field == EU3D_FIELD_RHS) {
        if (h->flux_bits == 64)
            k_h2d<double><<<xg, 256, 0, h->st>>>(L, h->stage, n, (double *)h->rhs, L.fs);
        else
            k_h2d<float><<<xg, 256, 0, h->st>>>(L, h->stage, n, (float *)h->rhs, L.fs);
    } else {
        double *dst = field == EU3D_FIELD_T ? h->T : field == EU3D_FIELD_E ? h->E : h->cs;
        k_h2d<double><<<xg, 256, 0, h->st>>>(L, h->stage, n, dst, L.fs);
    }
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

int eu3d_download_field(eu3d_handle *h, int field, double *host)
{
    if (!h || !host) return fail(EU3D_ERR_ARG, "null argument");
    int n;
    if (field_shape(field, &n)) return fail(EU3D_ERR_ARG, "unknown field");
    const Layout &L = h->L;
    const long long cells = (long long)L.NI * L.NJ * L.NK;
    const size_t bytes = (size_t)cells * n * sizeof(double);
    int rc = ensure_stage(h, bytes);
    if (rc) return rc;
    const int gb = grid_blocks(cells * n);
    const dim3 xg = xfer_grid(L);
    const int pi = prim_index(field);
    if (pi >= 0) {
        if (h->flux_bits == 64)
            k_d2h<double><<<xg, 256, 0, h->st>>>(L, (const double *)h->prim + pi * L.fs, L.fs, n, h->stage);
        else
            k_d2h<float><<<xg, 256, 0, h->st>>>(L, (const float *)h->prim + pi * L.fs, L.fs, n, h->stage);
    } else if (field == EU3D_FIELD_C || field == EU3D_FIELD_MC || field == EU3D_FIELD_DI) {
        if (h->flux_bits == 64)
            k_derive<double><<<gb, 256, 0, h->st>>>(L, (const double *)h->prim, h->cs, field, h->stage, n);
        else
            k_derive<float><<<gb, 256, 0, h->st>>>(L, (const float *)h->prim, h->cs, field, h->stage, n);
    } else if (field == EU3D_FIELD_NCHEM) {
        k_d2h<int><<<xg, 256, 0, h->st>>>(L, h->nchem, L.fs, 1, h->stage);
    } else if (field == EU3D_FIELD_RHS) {
        if (h->flux_bits == 64)
            k_d2h<double><<<xg, 256, 0, h->st>>>(L, (const double *)h->rhs, L.fs, n, h->stage);
        else
            k_d2h<float><<<xg, 256, 0, h->st>>>(L, (const float *)h->rhs, L.fs, n, h->stage);
    } else {
        const double *src = field == EU3D_FIELD_T ? h->T : field == EU3D_FIELD_E ? h->E : h->cs;
        k_d2h<double><<<xg, 256, 0, h->st>>>(L, src, L.fs, n, h->stage);
    }
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(host, h->stage, bytes, cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

int eu3d_set_inflow(eu3d_handle *h, const double *U, const double *V, const double *W, const double *Pp,
                    const double *D, const double *T, const double *H, const double *E, const double *G,
                    const double *Y)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    const size_t pl = (size_t)h->L.nj * h->L.nk;
    if (!h->inflow) {
        CK(cudaMalloc(&h->inflow, (9 + NS) * pl * sizeof(double)));
        CK(cudaMemsetAsync(h->inflow, 0, (9 + NS) * pl * sizeof(double), h->st));
    }
    // host planes are (nj, nk) with k fastest (Yint (nj, nk, NS)); the device
    // planes are field-major with j fastest, the order the x-face ghost fill
    // reads them in
    const int nj = h->L.nj, nk = h->L.nk;
    std::vector<double> tmp((9 + NS) * pl);
    const double *src[9] = {U, V, W, Pp, D, T, H, E, G};
    CK(cudaStreamSynchronize(h->st));
    for (int f = 0; f < 9 + NS; f++) {
        if (f < 9 ? !src[f] : !Y) continue;
        double *dst = tmp.data() + f * pl;
        for (int j = 0; j < nj; j++)
            for (int k = 0; k < nk; k++) {
                const size_t p = (size_t)j * nk + k;
                dst[(size_t)k * nj + j] = f < 9 ? src[f][p] : Y[p * NS + (f - 9)];
            }
        CK(cudaMemcpy(h->inflow + f * pl, dst, pl * sizeof(double), cudaMemcpyHostToDevice));
    }
    return EU3D_OK;
}

int eu3d_init_uniform(eu3d_handle *h, double P, double T, double U, double V, double W, const double *Y)
{
    if (!h || !Y) return fail(EU3D_ERR_ARG, "null argument");
    if (!(P > 0) || !(T > 0)) return fail(EU3D_ERR_ARG, "pressure and temperature must be positive");
    Uniform u;
    u.P = P;
    u.T = T;
    u.U = U;
    u.V = V;
    u.W = W;
    for (int s = 0; s < NS; s++) u.Y[s] = Y[s];
    const int gb = grid_blocks((long long)h->L.fs);
    if (h->flux_bits == 64)
        k_init_uniform<double><<<gb, 256, 0, h->st>>>(h->L, u, h->quirks, (double *)h->prim, h->cs, h->T, h->E);
    else
        k_init_uniform<float><<<gb, 256, 0, h->st>>>(h->L, u, h->quirks, (float *)h->prim, h->cs, h->T, h->E);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

int eu3d_set_wedge(eu3d_handle *h, double x0, double y0, double tan_angle, int enabled)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    h->wedge[0] = x0;
    h->wedge[1] = y0;
    h->wedge[2] = tan_angle;
    h->wedge_on = enabled ? 1 : 0;
    if (h->wedge_band) cudaFree(h->wedge_band);
    h->wedge_band = nullptr;
    h->wedge_nband = 0;
    if (h->wedge_on) {
        // the band of solid cells within two cells (along x or y) of the
        // fluid and the mirror source of each, on the host in the order of
        // operations of the wedge fill
        const Layout &L = h->L;
        std::vector<double> xn(L.NI), yn(L.NJ);
        CK(cudaMemcpy(xn.data(), h->xn, L.NI * sizeof(double), cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(yn.data(), h->yn, L.NJ * sizeof(double), cudaMemcpyDeviceToHost));
        auto solid = [&](double x, double y) { return x > x0 && (y - y0) < (x - x0) * tan_angle; };
        const double cs = 1.0 / sqrt(1.0 + tan_angle * tan_angle), sn = tan_angle * cs;
        const double nx = -sn, ny = cs;
        const double dx = xn[L.bc + 1] - xn[L.bc], dy = yn[L.bc + 1] - yn[L.bc];
        std::vector<int4> band;
        for (int i = 0; i < L.NI; i++)
            for (int j = 0; j < L.NJ; j++) {
                const double x = xn[i], y = yn[j];
                if (!solid(x, y)) continue;
                bool near = false;
                for (int o = -2; o <= 2 && !near; o++) {
                    if (o == 0) continue;
                    if (i + o >= 0 && i + o < L.NI && !solid(xn[i + o], y)) near = true;
                    if (j + o >= 0 && j + o < L.NJ && !solid(x, yn[j + o])) near = true;
                }
                if (!near) continue;
                const double dist = (x - x0) * sn - (y - y0) * cs;
                const double xi = x + 2.0 * dist * nx, yi = y + 2.0 * dist * ny;
                int si = (int)floor((xi - xn[0]) / dx + 0.5);
                int sj = (int)floor((yi - yn[0]) / dy + 0.5);
                si = si < 0 ? 0 : (si > L.NI - 1 ? L.NI - 1 : si);
                sj = sj < 0 ? 0 : (sj > L.NJ - 1 ? L.NJ - 1 : sj);
                while (sj < L.NJ - 1 && solid(xn[si], yn[sj])) sj++;
                band.push_back(make_int4(i, j, si, sj));
            }
        if (!band.empty()) {
            CK(cudaMalloc(&h->wedge_band, band.size() * sizeof(int4)));
            CK(cudaMemcpy(h->wedge_band, band.data(), band.size() * sizeof(int4), cudaMemcpyHostToDevice));
        }
        h->wedge_nband = (int)band.size();
    }
    for (auto &g : h->graphs) cudaGraphExecDestroy(g.second);
    h->graphs.clear();
    return EU3D_OK;
}

int eu3d_set_dt(eu3d_handle *h, double dt)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    CK(cudaMemcpyAsync(h->scal, &dt, sizeof(double), cudaMemcpyHostToDevice, h->st));
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

int eu3d_set_time(eu3d_handle *h, double t)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    CK(cudaMemcpyAsync(h->scal + 1, &t, sizeof(double), cudaMemcpyHostToDevice, h->st));
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

int eu3d_get_dt(eu3d_handle *h, double *dt)
{
    if (!h || !dt) return fail(EU3D_ERR_ARG, "null argument");
    CK(cudaMemcpyAsync(dt, h->scal, sizeof(double), cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

int eu3d_cfl(eu3d_handle *h, double cfl, double final_time, double *dt_out)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    int rc = cfl_op(h, cfl, final_time, h->sp);
    if (rc) return rc;
    return dt_out ? eu3d_get_dt(h, dt_out) : EU3D_OK;
}

// ------------------------------------------------------- x-slab decomposition
// A multi-rank run splits the x extent into slabs, one handle per rank, and
// replaces Flowfield::Mpi_Boundary (src/Flowfield.cpp:775-1083) and the
// MPI_Reduce/Bcast of CFLcondition (:242-272) with these calls around a
// collective library of the caller's choice (NCCL over NVLink).

int eu3d_halo_bytes(eu3d_handle *h, long long *bytes)
{
    if (!h || !bytes) return fail(EU3D_ERR_ARG, "null argument");
    const long long n = 2LL * h->L.NJ * h->L.NK;
    *bytes = n * (NPRIM * (long long)prim_bytes(h) + 2 * (long long)sizeof(double));
    return EU3D_OK;
}

namespace {
int halo_op(eu3d_handle *h, int side, int overlap, void *buf, int pack)
{
    if (!h || !buf) return fail(EU3D_ERR_ARG, "null argument");
    if (side != 0 && side != 1) return fail(EU3D_ERR_ARG, "side must be 0 (low x) or 1 (high x)");
    if (overlap != 0 && overlap != 1) return fail(EU3D_ERR_ARG, "overlap must be 0 or 1");
    if (h->L.ni < 2 + overlap) return fail(EU3D_ERR_ARG, "slab narrower than the planes it sends");
    if ((uintptr_t)buf % 16) return fail(EU3D_ERR_ARG, "halo buffer must be 16-byte aligned");
    const Layout &L = h->L;
    // packed: the two interior planes next to the face (past the shared
    // node when overlap = 1); unpacked: the face's two ghost planes
    const int i0 = pack ? (side == 0 ? L.bc + overlap : L.ni + L.bc - 2 - overlap) : (side == 0 ? 0 : L.ni + L.bc);
    const long long n = 2LL * L.NJ * L.NK;
    const int blocks = (int)std::min<long long>((n + 255) / 256, 148 * 8);
    ProfScope ps(h, pack ? "halo_pack" : "halo_unpack");
    if (h->flux_bits == 64)
        k_halo<double><<<blocks, 256, 0, h->st>>>(L, (double *)h->prim, h->T, h->E, (unsigned char *)buf, i0, pack);
    else
        k_halo<float><<<blocks, 256, 0, h->st>>>(L, (float *)h->prim, h->T, h->E, (unsigned char *)buf, i0, pack);
    CK(cudaGetLastError());
    return EU3D_OK;
}
}  // namespace

int eu3d_halo_pack(eu3d_handle *h, int side, int overlap, void *dst) { return halo_op(h, side, overlap, dst, 1); }
int eu3d_halo_unpack(eu3d_handle *h, int side, const void *src)
{
    return halo_op(h, side, 0, const_cast<void *>(src), 0);
}

int eu3d_cfl_local(eu3d_handle *h, double cfl, double final_time)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    return cfl_op(h, cfl, final_time, h->sp, 0);
}

double *eu3d_dt_device(eu3d_handle *h) { return h ? h->scal : nullptr; }

int eu3d_advance_time(eu3d_handle *h)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    k_advance_time<<<1, 1, 0, h->st>>>(h->scal);
    CK(cudaGetLastError());
    return EU3D_OK;
}

int eu3d_wedge_fill(eu3d_handle *h)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    return ghost_op(h, EU3D_BC_NONE);
}

namespace {
int prepare_step(eu3d_handle *h, const eu3d_step_desc *s);
}

int eu3d_step_part(eu3d_handle *h, const eu3d_step_desc *s, int part)
{
    int rc = prepare_step(h, s);
    if (rc) return rc;
    switch (part) {
    case EU3D_PART_STAGE1: return stage1_op(h, s);
    case EU3D_PART_STAGE2:
        if (!is_rk(s->timeadv)) return fail(EU3D_ERR_ARG, "stage 2 exists for SSP-RK2/RK3 only");
        return stage_op(h, s, 2);
    case EU3D_PART_STAGE3:
        if (s->timeadv != EU3D_ADV_SSPRK3) return fail(EU3D_ERR_ARG, "stage 3 exists for SSP-RK3 only");
        return stage_op(h, s, 3);
    case EU3D_PART_REACT: return react_op(h, s);
    case EU3D_PART_CHEM_PREDICT:
    case EU3D_PART_CHEM_WORK:
        if (s->react != EU3D_REACT_TRAPEZOID || s->type != 1)
            return fail(EU3D_ERR_ARG, "the chemistry halves exist for the adaptive trapezoid (type 1) only");
        if (!h->chem_queue || !h->qlist) return fail(EU3D_ERR_STATE, "the chemistry halves need the work queue");
        return trap1_part(h, part == EU3D_PART_CHEM_WORK ? 1 : 0);
    case EU3D_PART_SUR_PREDICT:
    case EU3D_PART_SUR_WORK:
        if (s->react != EU3D_REACT_SURROGATE) return fail(EU3D_ERR_ARG, "the surrogate halves need react SURROGATE");
        return sur_chem_op(h, is_rk(s->timeadv), part == EU3D_PART_SUR_WORK ? SUR_HALF_WORK : SUR_HALF_PREDICT);
    default: return fail(EU3D_ERR_ARG, "unknown step part");
    }
}

// ---------------------------------------------------------------------------
// Dynamic load balancing of the adaptive trapezoid across ranks
// (DynamicLoadBalancer, src/LoadBalance.cpp; Euler::Trapezoid type 1,
// src/Euler.cpp:380-700).

static_assert(EU3D_DLB_OUT_FIELDS == DLB_OUT && EU3D_DLB_BACK_FIELDS == DLB_BACK &&
                  EU3D_DLB_MAX_TRANSFERS == DLB_MAXSEG,
              "packet constants of the C ABI");

int eu3d_dlb_plan(const long long *loads, int nranks, int cap, int *sender, int *receiver, long long *amount,
                  int *ntransfers)
{
    if (!loads || !ntransfers || nranks < 1) return fail(EU3D_ERR_ARG, "bad arguments");
    std::vector<int> s, r;
    std::vector<long long> a;
    dlb::plan(loads, nranks, s, r, a);
    *ntransfers = (int)s.size();
    if ((int)s.size() > cap || ((!sender || !receiver || !amount) && !s.empty()))
        return fail(EU3D_ERR_ARG, "transfer arrays too small");
    for (size_t t = 0; t < s.size(); t++) {
        sender[t] = s[t];
        receiver[t] = r[t];
        amount[t] = a[t];
    }
    return EU3D_OK;
}

int eu3d_dlb_select_rows(const long long *rowload, long long nrows, int npacks, const long long *amount,
                         long long *bounds, long long *moved)
{
    if (!rowload || nrows < 0 || npacks < 0 || (npacks && (!amount || !moved)) || !bounds)
        return fail(EU3D_ERR_ARG, "bad arguments");
    dlb::select_rows(rowload, nrows, npacks, amount, bounds, moved);
    return EU3D_OK;
}

int eu3d_chem_load(eu3d_handle *h, long long *load)
{
    if (!h || !load) return fail(EU3D_ERR_ARG, "null argument");
    if (!h->qlist) return fail(EU3D_ERR_STATE, "no queued chemistry prediction on this handle");
    CK(cudaSetDevice(h->dev));
    const Layout &L = h->L;
    const long long nrows = (long long)L.nj * L.nk;
    if (!h->dlb_rowload) CK(cudaMalloc(&h->dlb_rowload, (size_t)nrows * sizeof(long long)));
    const int blocks = (int)std::min<long long>((nrows * 32 + 255) / 256, 148 * 16);
    k_dlb_rowload<<<blocks, 256, 0, h->st>>>(cell_args(h), h->dlb_rowload);
    CK(cudaGetLastError());
    h->dlb_rows.resize((size_t)nrows);
    CK(cudaMemcpyAsync(h->dlb_rows.data(), h->dlb_rowload, (size_t)nrows * sizeof(long long), cudaMemcpyDeviceToHost,
                       h->st));
    CK(cudaStreamSynchronize(h->st));
    long long s = 0;
    for (long long v : h->dlb_rows) s += v;
    *load = s;
    return EU3D_OK;
}

int eu3d_dlb_select(eu3d_handle *h, int ntransfers, const long long *amount, long long *cells, long long *moved)
{
    if (!h || ntransfers < 0 || ntransfers > DLB_MAXSEG || (ntransfers && (!amount || !cells || !moved)))
        return fail(EU3D_ERR_ARG, "bad arguments");
    const Layout &L = h->L;
    const long long nrows = (long long)L.nj * L.nk;
    if ((long long)h->dlb_rows.size() != nrows) return fail(EU3D_ERR_STATE, "eu3d_chem_load first");
    long long bounds[DLB_MAXSEG + 1];
    long long mv[DLB_MAXSEG];
    dlb::select_rows(h->dlb_rows.data(), nrows, ntransfers, amount, bounds, mv);
    DlbSegs &sg = h->dlb_segs;
    sg.n = ntransfers;
    long long off = 0;
    for (int p = 0; p <= ntransfers; p++) sg.row[p] = bounds[p];
    for (int p = 0; p < ntransfers; p++) {
        cells[p] = (bounds[p + 1] - bounds[p]) * L.ni;
        moved[p] = mv[p];
        sg.off[p] = off;
        off += DLB_OUT * cells[p];
    }
    return EU3D_OK;
}

int eu3d_dlb_pack(eu3d_handle *h, double *buf)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    const DlbSegs &sg = h->dlb_segs;
    if (sg.n == 0 || sg.row[sg.n] == sg.row[0]) return EU3D_OK;
    if (!buf) return fail(EU3D_ERR_ARG, "null buffer");
    CK(cudaSetDevice(h->dev));
    const long long total = (sg.row[sg.n] - sg.row[0]) * h->L.ni;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    {
        ProfScope ps(h, "dlb_pack");
        k_dlb_pack<<<blocks, 256, 0, h->st>>>(cell_args(h), sg, buf, h->qbins);
    }
    CK(cudaGetLastError());
    h->away_lo = sg.row[0];
    h->away_hi = sg.row[sg.n];
    return EU3D_OK;
}

extern "C++" {
namespace {
int ensure_guest(eu3d_handle *h, long long cells)
{
    if (cells <= h->g_cap) return EU3D_OK;
    const long long cap = std::max<long long>(cells, 2 * h->g_cap);
    // earlier guest work queued on the handle's stream may still read the old store
    CK(cudaStreamSynchronize(h->st));
    void *old[] = {h->g_cs, h->g_T, h->g_E, h->g_nchem, h->g_list, h->g_prim, h->g_audit, h->g_res, h->g_info};
    for (void *p : old)
        if (p) cudaFree(p);
    h->g_cs = h->g_T = h->g_E = h->g_audit = h->g_res = nullptr;
    h->g_nchem = h->g_list = h->g_info = nullptr;
    h->g_prim = nullptr;
    h->g_cap = 0;
    CK(cudaMalloc(&h->g_cs, (size_t)NV * cap * sizeof(double)));
    CK(cudaMalloc(&h->g_T, (size_t)cap * sizeof(double)));
    CK(cudaMalloc(&h->g_E, (size_t)cap * sizeof(double)));
    CK(cudaMalloc(&h->g_nchem, (size_t)cap * sizeof(int)));
    CK(cudaMalloc(&h->g_list, (size_t)cap * sizeof(int)));
    CK(cudaMalloc(&h->g_prim, (size_t)NPRIM * cap * prim_bytes(h)));
    CK(cudaMalloc(&h->g_audit, (size_t)cap * sizeof(double)));
    CK(cudaMalloc(&h->g_res, (size_t)(NS + 1) * cap * sizeof(double)));
    CK(cudaMalloc(&h->g_info, (size_t)cap * sizeof(int)));
    if (!h->g_bins) CK(cudaMalloc(&h->g_bins, (3 * QBINS + 2) * sizeof(int)));
    if (!h->g_count) CK(cudaMalloc(&h->g_count, 4 * sizeof(int)));
    h->g_cap = cap;
    return EU3D_OK;
}

template <class P, bool SPEC>
void guest_work(eu3d_handle *h, const DlbGuestSegs &sg, const double *in, double *out)
{
    const long long total = sg.first[sg.n];
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    ChemQueue qu{h->g_list, h->g_bins};
    cudaMemsetAsync(h->g_bins, 0, (3 * QBINS + 2) * sizeof(int), h->st);
    k_dlb_guest_in<<<blocks, 256, 0, h->st>>>(sg, in, h->g_cap, h->g_cs, h->g_T, h->g_nchem, h->g_bins);
    k_queue_scan<<<1, 32, 0, h->st>>>(qu);
    k_dlb_guest_list<<<blocks, 256, 0, h->st>>>(h->g_nchem, total, qu);
    // the store as a field of g_cap cells: trap1_cell reads only the field
    // stride of the layout
    CellArgs a = cell_args(h);
    a.L.fs = h->g_cap;
    a.cs = h->g_cs;
    a.T = h->g_T;
    a.E = h->g_E;
    a.nchem = h->g_nchem;
    a.rhs = nullptr;
    a.cs0 = nullptr;
    a.wedge_on = 0;
    {
        ProfScope ps(h, "dlb_guest_work");
        k_trap1_work<P, SPEC><<<queue_grid(h), 128, 0, h->st>>>(a, (P *)h->g_prim, qu);
    }
    k_dlb_guest_out<P><<<blocks, 256, 0, h->st>>>(sg, h->g_cap, h->g_cs, h->g_T, h->g_E, (const P *)h->g_prim,
                                                  h->g_nchem, out);
}
}  // namespace
}  // extern "C++"

int eu3d_dlb_guest(eu3d_handle *h, int nseg, const long long *seg_cells, const double *in, double *out)
{
    if (!h || nseg < 0 || nseg > DLB_MAXSEG || (nseg && !seg_cells)) return fail(EU3D_ERR_ARG, "bad arguments");
    DlbGuestSegs sg{};
    sg.n = nseg;
    sg.first[0] = 0;
    for (int s = 0; s < nseg; s++) {
        if (seg_cells[s] < 0) return fail(EU3D_ERR_ARG, "negative segment size");
        sg.off_in[s] = DLB_OUT * sg.first[s];
        sg.off_out[s] = DLB_BACK * sg.first[s];
        sg.first[s + 1] = sg.first[s] + seg_cells[s];
    }
    const long long total = sg.first[nseg];
    if (total == 0) return EU3D_OK;
    if (!in || !out) return fail(EU3D_ERR_ARG, "null buffer");
    CK(cudaSetDevice(h->dev));
    int rc = ensure_guest(h, total);
    if (rc) return rc;
    if (h->flux_bits == 64) {
        if (h->spec)
            guest_work<double, true>(h, sg, in, out);
        else
            guest_work<double, false>(h, sg, in, out);
    } else {
        if (h->spec)
            guest_work<float, true>(h, sg, in, out);
        else
            guest_work<float, false>(h, sg, in, out);
    }
    CK(cudaGetLastError());
    return EU3D_OK;
}

int eu3d_dlb_unpack(eu3d_handle *h, const double *back)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    DlbSegs sg = h->dlb_segs;
    if (sg.n == 0 || sg.row[sg.n] == sg.row[0]) return EU3D_OK;
    if (!back) return fail(EU3D_ERR_ARG, "null buffer");
    CK(cudaSetDevice(h->dev));
    long long off = 0;
    for (int p = 0; p < sg.n; p++) {
        sg.off[p] = off;
        off += DLB_BACK * (sg.row[p + 1] - sg.row[p]) * h->L.ni;
    }
    const long long total = (sg.row[sg.n] - sg.row[0]) * h->L.ni;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    {
        ProfScope ps(h, "dlb_unpack");
        if (h->flux_bits == 64)
            k_dlb_unpack<double><<<blocks, 256, 0, h->st>>>(cell_args(h), sg, back, (double *)h->prim);
        else
            k_dlb_unpack<float><<<blocks, 256, 0, h->st>>>(cell_args(h), sg, back, (float *)h->prim);
    }
    CK(cudaGetLastError());
    return EU3D_OK;
}

// ---------------------------------------------------------------------------
// Load balancing of the learned chemistry's FP64 fallback across ranks
int eu3d_sur_load(eu3d_handle *h, long long *load)
{
    if (!h || !load) return fail(EU3D_ERR_ARG, "null argument");
    if (!h->sur_count) return fail(EU3D_ERR_STATE, "no fallback list on this handle");
    CK(cudaSetDevice(h->dev));
    int cnt = 0;
    CK(cudaMemcpyAsync(&cnt, h->sur_count, sizeof(int), cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    h->sdlb_total = std::min<long long>(cnt, h->L.interior_cells());
    h->sdlb_keep = h->sdlb_total;
    h->sdlb_segs = DlbGuestSegs{};
    *load = h->sdlb_total;
    return EU3D_OK;
}

int eu3d_sdlb_select(eu3d_handle *h, int ntransfers, const long long *amount, long long *cells)
{
    if (!h || ntransfers < 0 || ntransfers > DLB_MAXSEG || (ntransfers && (!amount || !cells)))
        return fail(EU3D_ERR_ARG, "bad arguments");
    if (h->sdlb_total < 0) return fail(EU3D_ERR_STATE, "eu3d_sur_load after the step's SUR_PREDICT first");
    DlbGuestSegs &sg = h->sdlb_segs;
    sg = DlbGuestSegs{};
    sg.n = ntransfers;
    long long left = h->sdlb_total;
    for (int p = 0; p < ntransfers; p++) {
        if (amount[p] < 0) return fail(EU3D_ERR_ARG, "negative amount");
        cells[p] = std::min(amount[p], left);
        left -= cells[p];
    }
    // the transfers take the last slots, segment p after segment p - 1
    h->sdlb_keep = left;
    for (int p = 0; p < ntransfers; p++) {
        sg.off_in[p] = SDLB_OUT * sg.first[p];
        sg.off_out[p] = SDLB_BACK * sg.first[p];
        sg.first[p + 1] = sg.first[p] + cells[p];
    }
    return EU3D_OK;
}

int eu3d_sdlb_pack(eu3d_handle *h, double *buf)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    const DlbGuestSegs &sg = h->sdlb_segs;
    const long long total = sg.first[sg.n];
    if (total == 0) return EU3D_OK;
    if (!buf) return fail(EU3D_ERR_ARG, "null buffer");
    CK(cudaSetDevice(h->dev));
    const SurQueue qu{h->sur_list, h->sur_count, h->sur_audit, h->L.interior_cells(), h->sur_res, h->sur_info};
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    {
        ProfScope ps(h, "sdlb_pack");
        k_sdlb_pack<<<blocks, 256, 0, h->st>>>(cell_args(h), qu, sg, h->sdlb_keep, buf);
        k_sdlb_keep<<<1, 1, 0, h->st>>>(h->sur_count, (int)h->sdlb_keep);
    }
    CK(cudaGetLastError());
    return EU3D_OK;
}

extern "C++" {
namespace {
template <class P, bool SPEC>
void sdlb_guest_work(eu3d_handle *h, const DlbGuestSegs &sg, const double *in, double *out)
{
    const long long total = sg.first[sg.n];
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    k_sdlb_guest_in<<<blocks, 256, 0, h->st>>>(sg, in, h->g_cap, h->g_cs, h->g_T, h->g_audit, h->g_list);
    k_sdlb_keep<<<1, 1, 0, h->st>>>(h->g_count, (int)total);
    // the store as a field of g_cap cells: the fallback kernels read only the
    // field stride of the layout and the cell of each list entry
    CellArgs a = cell_args(h);
    a.L.fs = h->g_cap;
    a.cs = h->g_cs;
    a.T = h->g_T;
    a.E = h->g_E;
    a.rhs = nullptr;
    a.cs0 = nullptr;
    a.wedge_on = 0;
    const SurQueue qu{h->g_list, h->g_count, h->g_audit, h->g_cap, h->g_res, h->g_info};
    {
        ProfScope ps(h, "sdlb_guest_work");
        k_sur_fallback<P, SPEC><<<h->nparts, 128, 0, h->st>>>(a, (P *)h->g_prim, qu);
    }
    {
        ProfScope ps(h, "sdlb_guest_finish");
        k_sur_fallback_finish<P, SPEC><<<FALLBACK_FINISH_BLOCKS, 128, 0, h->st>>>(a, (P *)h->g_prim, qu);
    }
    k_sdlb_guest_out<P><<<blocks, 256, 0, h->st>>>(sg, h->g_cap, h->g_cs, h->g_T, h->g_E, (const P *)h->g_prim, out);
}
}  // namespace
}  // extern "C++"

int eu3d_sdlb_guest(eu3d_handle *h, int nseg, const long long *seg_cells, const double *in, double *out)
{
    if (!h || nseg < 0 || nseg > DLB_MAXSEG || (nseg && !seg_cells)) return fail(EU3D_ERR_ARG, "bad arguments");
    if (!h->sur) return fail(EU3D_ERR_STATE, "no surrogate attached (eu3d_set_surrogate)");
    DlbGuestSegs sg{};
    sg.n = nseg;
    for (int p = 0; p < nseg; p++) {
        if (seg_cells[p] < 0) return fail(EU3D_ERR_ARG, "negative segment size");
        sg.off_in[p] = SDLB_OUT * sg.first[p];
        sg.off_out[p] = SDLB_BACK * sg.first[p];
        sg.first[p + 1] = sg.first[p] + seg_cells[p];
    }
    const long long total = sg.first[nseg];
    if (total == 0) return EU3D_OK;
    if (!in || !out) return fail(EU3D_ERR_ARG, "null buffer");
    if (total > (long long)SUR_CELL_MASK) return fail(EU3D_ERR_ARG, "too many received cells");
    CK(cudaSetDevice(h->dev));
    int rc = ensure_guest(h, total);
    if (rc) return rc;
    if (h->flux_bits == 64) {
        if (h->spec)
            sdlb_guest_work<double, true>(h, sg, in, out);
        else
            sdlb_guest_work<double, false>(h, sg, in, out);
    } else {
        if (h->spec)
            sdlb_guest_work<float, true>(h, sg, in, out);
        else
            sdlb_guest_work<float, false>(h, sg, in, out);
    }
    CK(cudaGetLastError());
    return EU3D_OK;
}

int eu3d_sdlb_unpack(eu3d_handle *h, const double *back)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    const DlbGuestSegs &sg = h->sdlb_segs;
    const long long total = sg.first[sg.n];
    if (total == 0) return EU3D_OK;
    if (!back) return fail(EU3D_ERR_ARG, "null buffer");
    CK(cudaSetDevice(h->dev));
    const SurQueue qu{h->sur_list, h->sur_count, h->sur_audit, h->L.interior_cells(), h->sur_res, h->sur_info};
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    {
        ProfScope ps(h, "sdlb_unpack");
        if (h->flux_bits == 64)
            k_sdlb_unpack<double><<<blocks, 256, 0, h->st>>>(cell_args(h), qu, sg, h->sdlb_keep, back, (double *)h->prim);
        else
            k_sdlb_unpack<float><<<blocks, 256, 0, h->st>>>(cell_args(h), qu, sg, h->sdlb_keep, back, (float *)h->prim);
    }
    CK(cudaGetLastError());
    return EU3D_OK;
}

int eu3d_boundary(eu3d_handle *h, int kind)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    return ghost_op(h, kind);
}

int eu3d_advection(eu3d_handle *h, int timeadv, int diff)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    if (timeadv != EU3D_ADV_EE && timeadv != EU3D_ADV_TVD_RK3) return fail(EU3D_ERR_ARG, "timeadv must be EE or TVD_RK3");
    if (diff < EU3D_DIFF_MUSCL1 || diff > EU3D_DIFF_WENO) return fail(EU3D_ERR_ARG, "unknown difference scheme");
    return adv_op(h, timeadv, diff);
}

int eu3d_update_after_adv(eu3d_handle *h) { return h ? cell_op(h, M_ADV) : fail(EU3D_ERR_ARG, "null handle"); }
int eu3d_update_after_cs(eu3d_handle *h) { return h ? cell_op(h, M_DECODE) : fail(EU3D_ERR_ARG, "null handle"); }
int eu3d_react_imex(eu3d_handle *h) { return h ? cell_op(h, M_IMEX) : fail(EU3D_ERR_ARG, "null handle"); }
int eu3d_react_trapezoid(eu3d_handle *h, int type)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    if (type != 0 && type != 1) return fail(EU3D_ERR_ARG, "trapezoid type must be 0 or 1");
    int rc;
    if (type == 1 && h->chem_queue && (rc = ensure_queue(h))) return rc;
    return cell_op(h, type == 0 ? M_TRAP0 : M_TRAP1);
}

namespace {
// argument and state checks of a step, and the buffers it needs (the SSP-RK
// stage state, the trapezoid work queue), for eu3d_step and eu3d_step_part
int prepare_step(eu3d_handle *h, const eu3d_step_desc *s)
{
    if (!h || !s) return fail(EU3D_ERR_ARG, "null argument");
    if (s->timeadv < EU3D_ADV_EE || s->timeadv > EU3D_ADV_SSPRK3) return fail(EU3D_ERR_ARG, "unknown time scheme");
    if (s->diff < EU3D_DIFF_MUSCL1 || s->diff > EU3D_DIFF_WENO) return fail(EU3D_ERR_ARG, "unknown difference scheme");
    if (s->react != EU3D_REACT_IMEX && s->react != EU3D_REACT_TRAPEZOID && s->react != EU3D_REACT_NONE &&
        s->react != EU3D_REACT_SURROGATE && s->react != EU3D_REACT_ADAPTIVE)
        return fail(EU3D_ERR_ARG, "unsupported reaction scheme");
    if (s->react == EU3D_REACT_ADAPTIVE && !h->elements)
        return fail(EU3D_ERR_STATE, "element composition not set (eu3d_set_elements)");
    if (s->react == EU3D_REACT_SURROGATE && !h->sur) return fail(EU3D_ERR_STATE, "no surrogate attached");
    if (s->bc_kind == EU3D_BC_ODM && !h->inflow) return fail(EU3D_ERR_STATE, "ODM boundary needs eu3d_set_inflow first");
    CK(cudaSetDevice(h->dev));
    if (is_rk(s->timeadv) && !h->cs0) CK(cudaMalloc(&h->cs0, (size_t)NV * h->L.fs * sizeof(double)));
    if (s->react == EU3D_REACT_TRAPEZOID && s->type == 1 && h->chem_queue) {
        int rc = ensure_queue(h);
        if (rc) return rc;
    }
    return EU3D_OK;
}
}  // namespace

int eu3d_step(eu3d_handle *h, const eu3d_step_desc *s)
{
    int prc = prepare_step(h, s);
    if (prc) return prc;
    if (h->profile) return enqueue_step(h, s, h->sp);
    StepKey key{s->react, s->type, s->timeadv, s->diff, s->bc_kind, s->cfl, s->final_time};
    auto it = h->graphs.find(key);
    if (it == h->graphs.end()) {
        const Spacing sp = h->sp;
        cudaGraph_t g;
        CK(cudaStreamBeginCapture(h->st, cudaStreamCaptureModeThreadLocal));
        int rc = enqueue_step(h, s, sp);
        cudaError_t e = cudaStreamEndCapture(h->st, &g);
        if (rc) {
            if (e == cudaSuccess) cudaGraphDestroy(g);
            return rc;
        }
        CK(e);
        cudaGraphExec_t ex;
        e = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        CK(e);
        it = h->graphs.emplace(key, ex).first;
    }
    CK(cudaGraphLaunch(it->second, h->st));
    return EU3D_OK;
}

int eu3d_run(eu3d_handle *h, const eu3d_step_desc *s, int nsteps, int check_time)
{
    for (int n = 0; n < nsteps; n++) {
        int rc = eu3d_step(h, s);
        if (rc) return rc;
        if (check_time) {
            double sc[2];
            CK(cudaMemcpyAsync(sc, h->scal, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->st));
            CK(cudaStreamSynchronize(h->st));
            if (!(sc[1] < s->final_time)) break;
        }
    }
    return EU3D_OK;
}

int eu3d_profile_enable(eu3d_handle *h, int on)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    h->profile = on != 0;
    return EU3D_OK;
}

int eu3d_profile_read(eu3d_handle *h, char *names, size_t names_cap, double *ms, long long *counts, int max_kernels,
                      int *n_out)
{
    if (!h || !n_out) return fail(EU3D_ERR_ARG, "null argument");
    CK(cudaStreamSynchronize(h->st));
    for (auto &r : h->prof_pending) {
        float t = 0.f;
        CK(cudaEventElapsedTime(&t, r.a, r.b));
        auto &acc = h->prof_acc[r.name];
        acc.first += t;
        acc.second += 1;
        h->prof_pool.push_back(r.a);
        h->prof_pool.push_back(r.b);
    }
    h->prof_pending.clear();
    int n = 0;
    size_t used = 0;
    for (auto &kv : h->prof_acc) {
        if (n >= max_kernels) break;
        const size_t len = kv.first.size() + 1;
        if (names) {
            if (used + len > names_cap) break;
            memcpy(names + used, kv.first.c_str(), len - 1);
            names[used + len - 1] = '\n';
        }
        used += len;
        if (ms) ms[n] = kv.second.first;
        if (counts) counts[n] = kv.second.second;
        n++;
    }
    if (names && used < names_cap) names[used] = 0;
    *n_out = n;
    h->prof_acc.clear();
    return EU3D_OK;
}

int eu3d_cfl_noalloc(const double *D, const double *U, const double *V, const double *W, const double *Pp,
                     const double *Gamma, int ni, int nj, int nk, int bc, long long pitch, long long plane, double dx,
                     double dy, double dz, int use_z, double cfl, double final_time, double *time_inout,
                     double *dt_out, int nblocks, void *stream)
{
    if (!D || !U || !V || !W || !Pp || !Gamma || !time_inout || !dt_out) return fail(EU3D_ERR_ARG, "null argument");
    if (ni < 1 || nj < 1 || nk < 1 || bc < 0) return fail(EU3D_ERR_ARG, "grid extents must be positive");
    if (pitch < ni + 2LL * bc || plane < pitch * (nj + 2LL * bc))
        return fail(EU3D_ERR_ARG, "pitch/plane stride smaller than the ghosted extents");
    if (nblocks <= 0) nblocks = NOALLOC_CFL_DEFAULT_BLOCKS;
    if (nblocks > NOALLOC_CFL_MAX_BLOCKS)
        return fail(EU3D_ERR_ARG, "nblocks exceeds the 1024-entry scratch array of eu3d_cfl_noalloc");
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return fail(EU3D_ERR_ARG, "device ordinal beyond 63");
    double *scratch = g_cfl_scratch_dev[dev].load(std::memory_order_acquire);
    if (!scratch) {
        void *p = nullptr;
        CK(cudaGetSymbolAddress(&p, g_cfl_scratch));
        scratch = (double *)p;
        g_cfl_scratch_dev[dev].store(scratch, std::memory_order_release);
    }
    CflFields f{D, U, V, W, Pp, Gamma, ni, nj, nk, bc, pitch, plane};
    cudaStream_t st = (cudaStream_t)stream;
    k_cfl_fields_partial<<<nblocks, 256, 0, st>>>(f, dx, dy, dz, use_z, scratch);
    k_cfl_fields_final<<<1, 1024, 0, st>>>(scratch, nblocks, cfl, final_time, dt_out, time_inout);
    CK(cudaGetLastError());
    return EU3D_OK;
}

int eu3d_gemm_bf16(const void *A, const void *B, float *C, int M, int N, int K, int accumulate, int *err,
                   void *stream)
{
    if (!A || !B || !C) return fail(EU3D_ERR_ARG, "null argument");
    if (M <= 0 || M % 128 || N < 16 || N > 256 || N % 16 || K <= 0 || K % 16)
        return fail(EU3D_ERR_ARG, "gemm shape: M % 128 == 0, N in [16, 256] with N % 16 == 0, K % 16 == 0");
    if (((uintptr_t)A | (uintptr_t)B) & 15) return fail(EU3D_ERR_ARG, "gemm operands must be 16-byte aligned");
    static bool attr = false;
    if (!attr) {
        CK(cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem_bytes()));
        attr = true;
    }
    k_gemm_tc<<<M / 128, 128, gemm_smem_bytes(), (cudaStream_t)stream>>>(
        (const __nv_bfloat16 *)A, (const __nv_bfloat16 *)B, C, M, N, K, accumulate, err);
    CK(cudaGetLastError());
    return EU3D_OK;
}

int eu3d_set_elements(eu3d_handle *h, const double *atoms)
{
    if (!h || !atoms) return fail(EU3D_ERR_ARG, "null argument");
    CK(cudaSetDevice(h->dev));
    double A[SUR_NELEM][NS];
    for (int e = 0; e < SUR_NELEM; e++)
        for (int k = 0; k < NS; k++) {
            if (!(atoms[e * NS + k] >= 0)) return fail(EU3D_ERR_ARG, "atom counts must be >= 0");
            A[e][k] = atoms[e * NS + k] / g_mech_loaded[0].mw[k];
        }
    CK(cudaMemcpyToSymbol(c_sur_elem, A, sizeof(A)));
    h->elements = true;
    return EU3D_OK;
}

int eu3d_set_adaptive(eu3d_handle *h, double rel, double amp, int nmax)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    if (!(rel > 0 && rel <= 1) || !(amp > 0 && amp < 1) || nmax < 1 || nmax > NCHEM_CAP)
        return fail(EU3D_ERR_ARG, "adaptive chemistry: 0 < rel <= 1, 0 < amp < 1, 1 <= nmax <= 2^20");
    h->acfg = AdaptCfg{rel, amp, nmax};
    for (auto &g : h->graphs) cudaGraphExecDestroy(g.second);
    h->graphs.clear();
    return EU3D_OK;
}

int eu3d_react_adaptive(eu3d_handle *h)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    if (!h->elements) return fail(EU3D_ERR_STATE, "element composition not set (eu3d_set_elements)");
    return h->adapt_queue ? adapt_queue_op(h, false) : cell_op(h, M_ADAPT);
}

int eu3d_set_tuning(eu3d_handle *h, const eu3d_tuning *t)
{
    if (!h || !t) return fail(EU3D_ERR_ARG, "null argument");
    if (t->flux_kz < 1 || t->flux_kz > 256) return fail(EU3D_ERR_ARG, "flux_kz must be in [1, 256]");
    if (t->queue_blocks < 1 || t->queue_blocks > 16) return fail(EU3D_ERR_ARG, "queue_blocks must be in [1, 16]");
    h->flux_kz = t->flux_kz;
    h->chem_queue = t->chem_queue ? 1 : 0;
    h->queue_blocks = t->queue_blocks;
    if (t->flux_stage < 0 || t->flux_stage > 2) return fail(EU3D_ERR_ARG, "flux_stage must be 0, 1 or 2");
    // the TMA ring needs the tensor map; without it the staged kernel runs (and is reported)
    h->flux_stage = (t->flux_stage == 2 && !h->tq_ok) ? 1 : t->flux_stage;
    h->sur_fused = t->sur_fused ? 1 : 0;
    // (builds for 5 and 6 blocks, at 96 and 85 registers, scheduled the
    // decode's arithmetic differently and changed results in the last bits:
    // left out)
    if (t->cell_blocks != 3 && t->cell_blocks != 4) return fail(EU3D_ERR_ARG, "cell_blocks must be 3 or 4");
    h->cell_blocks = t->cell_blocks;
    h->gate_fused = t->gate_fused ? 1 : 0;
    h->adapt_queue = t->adapt_queue ? 1 : 0;
    if (h->adapt_queue) {
        int rc = ensure_cell_list(h);
        if (rc) return rc;
    }
    for (auto &g : h->graphs) cudaGraphExecDestroy(g.second);
    h->graphs.clear();
    return EU3D_OK;
}

int eu3d_set_wait_limit(eu3d_handle *h, long long tries)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    if (tries < 0 || tries > (1LL << 24)) return fail(EU3D_ERR_ARG, "wait limit must be in [0, 2^24]");
    h->wait_tries = (unsigned)tries;
    for (auto &g : h->graphs) cudaGraphExecDestroy(g.second);
    h->graphs.clear();
    return EU3D_OK;
}

int eu3d_get_tuning(eu3d_handle *h, eu3d_tuning *t)
{
    if (!h || !t) return fail(EU3D_ERR_ARG, "null argument");
    t->flux_kz = h->flux_kz;
    t->chem_queue = h->chem_queue;
    t->queue_blocks = h->queue_blocks;
    t->flux_stage = h->flux_stage;
    t->sur_fused = h->sur_fused;
    t->adapt_queue = h->adapt_queue;
    t->cell_blocks = h->cell_blocks;
    t->gate_fused = h->gate_fused;
    return EU3D_OK;
}

int eu3d_autotune(eu3d_handle *h, const eu3d_step_desc *s, int steps, eu3d_tuning *best, double *best_ms)
{
    if (!h || !s) return fail(EU3D_ERR_ARG, "null argument");
    if (steps < 1) return fail(EU3D_ERR_ARG, "steps must be >= 1");
    CK(cudaSetDevice(h->dev));
    const eu3d_tuning start{h->flux_kz,   h->chem_queue,  h->queue_blocks, h->flux_stage,
                            h->sur_fused, h->adapt_queue, h->cell_blocks, h->gate_fused};
    // the trials advance the state: keep a copy and put it back after each
    const size_t fs = (size_t)h->L.fs;
    const size_t nprim = (size_t)NPRIM * fs * prim_bytes(h);
    const size_t bytes = (NV + 2) * fs * sizeof(double) + nprim + 2 * sizeof(double) + sizeof(Status);
    char *bk = nullptr;
    CK(cudaMalloc(&bk, bytes));
    struct Piece {
        void *p;
        size_t n;
    } pieces[] = {{h->cs, NV * fs * sizeof(double)}, {h->T, fs * sizeof(double)}, {h->E, fs * sizeof(double)},
                  {h->prim, nprim},
                  {h->scal, 2 * sizeof(double)},
                  {h->status, sizeof(Status)}};
    auto copy = [&](bool save) {
        size_t off = 0;
        for (auto &pc : pieces) {
            if (save) cudaMemcpyAsync(bk + off, pc.p, pc.n, cudaMemcpyDeviceToDevice, h->st);
            else cudaMemcpyAsync(pc.p, bk + off, pc.n, cudaMemcpyDeviceToDevice, h->st);
            off += pc.n;
        }
    };
    copy(true);
    // the setting the handle has comes first: the best is never a slower one
    std::vector<eu3d_tuning> cands{start};
    const bool q = s->react == EU3D_REACT_TRAPEZOID && s->type == 1;
    const bool aq = s->react == EU3D_REACT_ADAPTIVE;
    for (int fst : {0, 1, 2})
        for (int kz : {4, 8, 16, 32, 64})
            for (int cq : {0, 1})
                for (int qb : {2, 3, 4})
                    for (int ad : {0, 1}) {
                        if (h->flux_bits == 64 && fst != start.flux_stage) continue;
                        if (!q && (cq != start.chem_queue || qb != start.queue_blocks)) continue;
                        if (q && cq == 0 && qb != start.queue_blocks) continue;
                        if (!aq && ad != start.adapt_queue) continue;
                        cands.push_back({kz, cq, qb, fst, start.sur_fused, ad, start.cell_blocks, start.gate_fused});
                    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best_t = 1e300;
    eu3d_tuning bt = start;
    int rc = EU3D_OK;
    for (const auto &c : cands) {
        if ((rc = eu3d_set_tuning(h, &c))) break;
        if ((rc = eu3d_step(h, s))) break;  // records the graph, warms up
        cudaEventRecord(e0, h->st);
        for (int n = 0; n < steps && !rc; n++) rc = eu3d_step(h, s);
        cudaEventRecord(e1, h->st);
        if (rc) break;
        if (cudaStreamSynchronize(h->st) != cudaSuccess) {
            rc = fail(EU3D_ERR_CUDA, "autotune trial failed");
            break;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms / steps < best_t) {
            best_t = ms / steps;
            bt = c;
        }
        copy(false);
    }
    copy(false);
    cudaStreamSynchronize(h->st);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(bk);
    if (rc) {
        eu3d_set_tuning(h, &start);
        return rc;
    }
    eu3d_set_tuning(h, &bt);
    if (best) *best = bt;
    if (best_ms) *best_ms = best_t;
    return EU3D_OK;
}

int eu3d_synchronize(eu3d_handle *h)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

int eu3d_get_status(eu3d_handle *h, eu3d_status *o)
{
    if (!h || !o) return fail(EU3D_ERR_ARG, "null argument");
    Status s;
    double sc[2];
    CK(cudaMemcpyAsync(&s, h->status, sizeof(Status), cudaMemcpyDeviceToHost, h->st));
    CK(cudaMemcpyAsync(sc, h->scal, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    o->nonfinite_cells = (long long)s.nonfinite;
    o->newton_capped = (long long)s.newton_capped;
    o->substeps = (long long)s.substeps;
    o->nchem_max = s.nchem_max;
    o->substep_capped = s.substep_capped;
    o->surrogate_cells = (long long)s.sur_cells;
    o->surrogate_fallback = (long long)s.sur_fallback;
    o->surrogate_audited = (long long)s.audit_cells;
    double mx;
    memcpy(&mx, &s.audit_max_dT_bits, sizeof(double));
    o->surrogate_audit_max_dT = mx;
    for (int r = 0; r < 4; r++) o->surrogate_rejects[r] = (long long)s.sur_reject[r];
    o->wait_timeouts = (long long)s.wait_timeouts;
    o->surrogate_frozen = (long long)s.sur_frozen;
    o->frozen_audited = (long long)s.frozen_audit_cells;
    memcpy(&mx, &s.frozen_audit_max_dT_bits, sizeof(double));
    o->frozen_audit_max_dT = mx;
    o->drain_timeouts = (long long)s.drain_timeouts;
    o->dt = sc[0];
    o->time = sc[1];
    return EU3D_OK;
}

int eu3d_reset_status(eu3d_handle *h)
{
    if (!h) return fail(EU3D_ERR_ARG, "null handle");
    CK(cudaMemsetAsync(h->status, 0, sizeof(Status), h->st));
    CK(cudaStreamSynchronize(h->st));
    return EU3D_OK;
}

}  // extern "C"

#include "sur_host.cuh"
