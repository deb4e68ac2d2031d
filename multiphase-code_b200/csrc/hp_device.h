// hp_device.h -- device-side layout of one case (mesh + state) and the
// per-variant kernel entry table.  Shared by the host code (hp_host.cu) and
// every precision variant (hp_variant_*.cu).
//
// Layout in HBM: structure of arrays, one column per variable (primitives and
// gradients: tiles of 32 cells, see prim_off), leading
// dimension `ld` (= ntot rounded up to 64 cells) so each column starts on a
// 512-byte boundary.  Cell ids are 0-based internally: elements [0, neles),
// boundary ghosts [neles, neles + nghosts) -- the reference's 1-based ids
// minus one (src/main.F90:103).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/hydraphase.h"   // HP_IBLANK_HALO*, HP_X_*

namespace hp {

enum { NEQ = 10, NPR = 14, NGR = 33, NLSQ = 16, NLSQB = 12 };

// primitive columns (the reference's ug,vg,wg,tg,pg,pp,phig,phip,up,vp,wp,
// tp,rog,rop of src/mod_GlobalVariables.F90:13)
enum { P_UG = 0, P_VG, P_WG, P_TG, P_PG, P_PP, P_PHIG, P_PHIP, P_UP, P_VP,
       P_WP, P_TP, P_ROG, P_ROP };
// Primitives are stored in tiles of 32 cells, a tile's 14 columns together:
// column k of cell c stands at pr[PR_TILE * k + prim_off(c)].  Consecutive
// cells share sectors as in plain columns, and the columns of a cell lie at
// fixed distances from one address.
enum { PR_TILE = 32 };
#if defined(__CUDACC__)
__host__ __device__
#endif
inline size_t prim_off(int c) {
    return (size_t)((unsigned)c / PR_TILE) * (NPR * PR_TILE) + ((unsigned)c % PR_TILE);
}
// stored gradient columns (x,y,z per field), src/sr_derivative.F90:259-309
enum { G_UG = 0, G_VG = 3, G_WG = 6, G_TG = 9, G_UP = 12, G_VP = 15,
       G_WP = 18, G_TP = 21, G_PG = 24, G_PP = 27, G_PHIG = 30 };

// face kind bits per cell, 4 bits per face: bit 0 = wall (ghost type 5),
// bit 1 = MUSCL-reconstruct across the face (interior or partition ghost).
enum { FK_WALL = 1, FK_RECON = 2 };
// cell bits of the same word, set at set-up where a least-squares weight,
// determinant or centroid difference of the cell (LSQA, LSQB tables), or the
// area or area vector of a face, lies outside the range in which the kernels'
// shared-reciprocal division is exact
enum { FK_LSQA_RANGE = 1 << 16, FK_LSQB_RANGE = 1 << 17, FK_AREA_RANGE = 1 << 18 };

struct DevParams {
    double gamag, gamap, pinf, cpp, cpg, prg, rrg, prp;
    double emin, emax, phipzero;
    double ugmin, vgmin, wgmin, upmin, vpmin, wpmin, tgmin, tpmin, pmin;
    double as, ts, c23, co2, co4, fsd;   // fsd = 4 sigma / d
    double cfl, venkat_k, twall, amup;
    // correctly rounded reciprocals of constant divisors
    double r_emm, r_gm1, r_gamap, r_prg, r_prp;
    int rk_scheme, inviscid, myorder, nstage;
    int myflux;   // 1 HLLC-Zien, 2 HLLC-Batten (src/mod_Fluxmodule.F90:8-11)
    // five-phase model: dispersed phases q, r, s (conserved columns 10-21)
    int five_phase;
    double rhod[3], radd[3], vold[3];   // densities, radii, particle volumes
};

// A handle holds one case or a batch of cases whose meshes are concatenated:
// the elements of case c occupy [elem_base_c, elem_base_c + neles_c) and its
// ghosts a range of [neles, neles + nghosts); neighbour ids point into the
// same case only, so every kernel sweeps all cases in one launch.  `cid`
// maps an element to its case (null for a single case: case 0).
struct DevMesh {
    int neles, nghosts, ntot, aliased;
    long long ld;
    int ncase;
    const int* cid;         // [neles] case of each element, or null
    const int* nc;          // [4][ld] face neighbours
    const int* snb;         // [4][ld] neighbours as smoothing sees them
    const unsigned* fk;     // [ld] face kind nibbles
    const int* iblank;      // [ld]
    const double *xc, *yc, *zc, *vol, *dl, *dd;   // [ld]
    // limiter epsilon^2 = (K dl)^3 per cell (src/sr_VK.F90:34), evaluated
    // once at set-up with the host's pow, as the reference evaluates it
    const double* eps2;     // [ld]
    // Geometry tables, of leading dimension ldt.  FP64 handles, and FP32 ones
    // without a face list, have a row for every cell.  Where only the FP64
    // kernels of the wall layers read them, a row for each cell of gcells in
    // list order (trows = 1): gcells starts with wcells, so row k is that of
    // wcells[k] too, and with wprefix that of cell k.  Else no rows (null).
    long long ldt;
    int trows, trows_n;     // rows by list position; number of rows
    const double* sc;       // [12][ldt] face area vectors sc1x..sc4z
    const double* scq;      // [12][ld] the same for every cell (five-phase model, else null)
    const double* fch;      // [12][ldt] face centroids, 0.3333 factor (HLLC, VK): x of faces 1-4, then y, z
    const double* fxo;      // [12][ldt] the same minus the cell's centroid (k_grad4, else null)
    // face areas or, for the Jameson flux, unit normal (x, y, z) and area of
    // face 1, then 2, 3, 4; formed on the device by the variant that reads them
    // (Variant::setup), null when the handle runs no FP64 flux kernel
    const double* area;     // [4][ldt]
    const double* nrm;      // [16][ldt]
    const double* fcv;      // [12][ldt] face centroids, /3 (viscous; null in inviscid handles)
    // geometry-only least-squares terms, evaluated once at set-up with the
    // reference's expressions: [0..3] weights, [4..9] a1 a2 a3 b1 b2 b3,
    // [10] the determinant; LSQA for the 1/r^2 cell gradients
    // (src/sr_derivative.F90:163-176,255), then the correctly rounded
    // reciprocals of the weights ([11..14]) and of the determinant ([15]);
    // LSQB for the 1/r gradient of alpha_g in the sources
    // (src/sr_source.F90:100-117), then that of the determinant ([11]) and,
    // with the Jameson flux, those of the weights ([12..15])
    const double* dxn;      // [12][ldt] centroid of neighbour f minus the
                            // cell's (x, y, z of face 1, then 2, 3, 4; k_grad4
                            // and the sources beside the Jameson flux, else null)
    // (null where nothing reads them: no FP64 kernels, no gradients)
    const double* lsqa;     // [NLSQ][ldt]
    const double* lsqb;     // [NLSQB or NLSQB + 4][ldt]
    const int *g_par, *g_id, *g_type;   // [nghosts] ghost list (reference order)
    // overset fringe (nfringe = 0: none): cells, 4 donor cells each and
    // barycentric weights, [4][nfringe] column-major
    // unique faces (FP32-arithmetic variants; nface = 0: cell-centric
    // fluxes): owner cell and local face of each, and per cell and local
    // face the signed face id + 1 (negative when the cell is not the owner).
    // Faces between two cells of the FP64 wall layers, or of one and a ghost,
    // feed only FP64 kernels and are not in the list (0 in cface)
    int nface;
    long long fld;          // leading dimension of the face-flux columns
    const int* f_i;
    const int* f_code;      // local face of the owner (bits 0-1)
    // what the face kernels read of a face, in face order: the cell on its
    // other side, the owner's area vector and the face centroid minus the
    // centroids of owner and neighbour in the arithmetic of the fluxes, and
    // the viscous face centroid; filled at set-up
    const int* f_j;
    const float* fgeo;      // [9][fld] area vector, offset from owner, from neighbour
    const double* fgcv;     // [3][fld]
    // centroid differences and face centroid offsets in float for the FP32
    // gradients (FP32-arithmetic variants without aliased ghosts and without
    // the FP64 tables of every cell; else null)
    const float *dxnf, *fxof;   // [12][ld] as dxn, fxo
    const int* cface;       // [4][ld]
    // face modes 2 (colouring) and 3 (atomics): the face fluxes are added
    // to a per-cell accumulator instead of stored as records.  Mode 2 takes
    // the faces colour by colour (no two faces of a colour share a cell, so
    // each colour adds without atomics, in a fixed order); fcolor lists the
    // face ids colour by colour, colour c at [fcoff[c], fcoff[c + 1]).
    int face_mode;
    int ncolor;
    const int* fcolor;      // [nface]
    int fcoff[33];
    int nfringe;
    const int* fr;
    const int* fdon;
    const double* fw;
    // partition halo (nhalo = 0: none): after every RK stage cell hdst[t]
    // takes the conserved state of cell hsrc[t] (the parts of one mesh as
    // the cases of a batch); the cases then share one dt
    int nhalo;
    const int* hdst;
    const int* hsrc;
    // FP64 wall layers of the FP32-arithmetic variants (nwall = 0: none):
    // the cells within a few layers of a wall ghost (wcells, ascending) take
    // their viscous terms, fluxes, sources and RK update from the FP64
    // kernels over these lists; gcells adds their interior neighbours, whose
    // FP64 gradients those fluxes reconstruct from; wclass[i] != 0 marks the
    // cells of wcells, which the FP32 kernels leave alone (2: no neighbour
    // outside the layers, so not even their FP32 gradients are read)
    int nwall, ngwall;
    int wprefix;            // 1: wcells and gcells are 0, 1, ... (the layer
                            // cells first in the cell order, see hp_host.cu)
    const int* wcells;
    const int* gcells;
    const unsigned char* wclass;   // [ld]
};

// Per-case scalars (one entry per case of the handle).
struct DevScalars {
    unsigned long long dtmin_bits;    // running min of dl/(a+|u|), skips NaN
    unsigned long long diff_bits[4];  // running max |cn - cu|, skips NaN
    unsigned long long nan_count;
    double dt, time, velmag;
    int total;                        // step counter (src/main.F90:522)
    int step_in_call;
    double fcarry[10];                // stale-flux carry (aliased meshes)
    int err_flags;
    int cell1;                        // internal id of the case's cell 1
    unsigned blocks_done;             // case 0: finished blocks of the step's closing pass
};

// R values per face record of the face-based variants: 48 bytes in FP32, read
// as three 16-byte loads
constexpr int FACE_REC = 12;

template <class R>
struct DevState {
    double *cn, *cu, *cn1;   // [10][ld]
    double* pr;              // [ld / 32][14][32], see prim_off
    R* prr;                  // as pr: primitives in R: pr itself when R is
                             // double, a float copy otherwise
    R* gr;                   // [ld / 32][33][32], see GRD in hp_kernels.cuh
    double* phi;             // [ld]
    R* agrad;                // [3][ld] 1/r-weighted gradient of alpha_g (the
                             // sources'), formed beside the others by the
                             // FP32 gradient kernel; null where that does not run
    // switches and Laplacian of the smoothing passes, dead once d24 stands:
    // they share the memory of vis (written by the viscous pass after them;
    // inviscid handles, whose vis is zero, keep two columns for anu) and of
    // cn1 (written by the first stage)
    double *anu, *d2q;       // [2][ld], [10][ld]
    double *d24, *vis;       // [10][ld], [8][ld]
    double* egt;             // [2][ld] ghost egtotal/eptotal (aliased meshes, else null)
    // five-phase model only (null otherwise): cn, cu, cn1, d2q and d24 then
    // hold 22 columns
    double* qpr;             // [12][ld] phi, u, v, w of q, r, s
    double* anuq;            // [3][ld] their JST switches
    double* qdrag;           // [9][ld] drag of q, r, s on the liquid (x, y, z)
    double* racc;            // [10][ld] face modes 2, 3: the cells' face sums
    R* ff;                   // [nface][FACE_REC] face records (face-based
                             // variants): 10 flux components, the wall flag
                             // (1: pressure terms only), one pad
    DevScalars* s;
    double* diag;            // [max_steps][8]
    int max_diag;
    double* gr64;            // as gr: FP64 gradients of the wall layers
                             // (FP32 variants with nwall > 0; else null)
};

// The FP64 view of an FP32-arithmetic state for the wall-layer kernels: the
// FP64 primitives as their primitives and gr64 as their gradients; every
// other array is shared.
template <class R>
inline DevState<double> fp64_view(const DevState<R>& s) {
    DevState<double> v;
    v.cn = s.cn; v.cu = s.cu; v.cn1 = s.cn1; v.pr = s.pr; v.prr = s.pr; v.gr = s.gr64; v.phi = s.phi;
    v.agrad = nullptr;
    v.anu = s.anu; v.d2q = s.d2q; v.d24 = s.d24; v.vis = s.vis; v.egt = s.egt;
    v.qpr = s.qpr; v.anuq = s.anuq; v.qdrag = s.qdrag; v.racc = s.racc; v.ff = nullptr;
    v.s = s.s; v.diag = s.diag; v.max_diag = s.max_diag; v.gr64 = s.gr64;
    return v;
}

// FP64 kernels over the wall-layer lists, provided by the FP64 variant and
// called by the FP32-arithmetic variants' step.
struct WallFp64 {
    void (*setup)(const DevMesh&, cudaStream_t);
    void (*visc)(const DevMesh&, const DevState<double>&, const DevParams&, cudaStream_t);
    void (*grad)(const DevMesh&, const DevState<double>&, const DevParams&, cudaStream_t);
    void (*flux)(const DevMesh&, const DevState<double>&, const DevParams&, cudaStream_t, int stage);
};
extern const WallFp64 wall_fp64;

// Grid-wide barrier of the fused step kernel (zeroed at set-up): arrivals,
// generation, and a flag set when a wait gave up (its spin is bounded).
struct GridSync {
    unsigned count;
    unsigned gen;
    int err;
    int pad;
};

// Kernel kinds, for per-kernel timing (hp_profile_steps).
enum KernelKind {
    KK_PRIM_START = 0, KK_STEP_BEGIN, KK_SMOOTH1, KK_SMOOTH2, KK_BC_VISC, KK_VISC,
    KK_PRIM_STAGE, KK_BC, KK_GRAD, KK_FLUX, KK_PRIM_END, KK_STEP_END, KK_SERIAL,
    KK_OVERSET, KK_HALO, KK_QRS, KK_COUNT
};

// Optional hook called before every launch (and with KK_COUNT after the
// last one) so the host can bracket each kernel with CUDA events.
struct StepHook {
    void (*mark)(void* ctx, int kind);      // before each kernel (may be null)
    void* ctx;
    // exchange points of a part run on several GPUs (may be null):
    // HP_X_DT before the step's dt is formed, HP_X_HALO after each RK stage
    void (*exchange)(void* ctx, int point);
    void* xctx;
};

// What one precision variant provides to the host.
struct Variant {
    const char* name;
    size_t grad_bytes;  // sizeof(R) of the gradient columns
    // enqueue the start-of-step primitive recovery + dt contributions
    void (*enqueue_start)(const DevMesh&, const void* st, const DevParams&,
                          cudaStream_t, int block, const StepHook* hook);
    // enqueue one full step (after enqueue_start of the same step)
    void (*enqueue_step)(const DevMesh&, const void* st, const DevParams&,
                         cudaStream_t, int block, const StepHook* hook);
    // 1 when the viscous fluxes are evaluated once per face on meshes with a
    // face list (k_facevisc + k_vis_gather instead of one kernel)
    int face_visc;
    // 1 when the flux kernel of meshes with a face list recovers the next
    // stage's primitives (see recover_in_flux in hp_kernels.cuh)
    int flux_recovers;
    // fills the tables that the flux kernels read (m.area, m.nrm), once per handle
    void (*setup)(const DevMesh&, cudaStream_t);
    // fused step (one cooperative launch per step): the grid it runs with on
    // this device (blocks of 128 threads), and the launch of one step
    int (*fused_grid)(const DevMesh&, const DevParams&);
    cudaError_t (*enqueue_fused)(const DevMesh&, const void* st, const DevParams&, cudaStream_t,
                                 GridSync* sync, int grid);
};

extern const Variant variant_fp64_parity;
extern const Variant variant_fp64;
extern const Variant variant_mixed;
extern const Variant variant_fp32;

}  // namespace hp
