// common.cuh -- device data layout shared by the kernels of the MCM step.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/mcm_gpu.h"

namespace mcm {

constexpr int kMaxMat = MCM_GPU_MAX_MATERIALS;
constexpr int kWarp = 32;
constexpr int kNoCell = -1;

// Material constants on the device (mirrors mcm_gpu_material).
struct DevMaterial {
    int model, eos, visc_type, pad;
    double rho, g, av_l, av_q, mass, h, rho_min, rho_max;
    double strinput[48];
    double eosinput[24];
    double k_cont, n_cont;   // repulsive contact (contacttype > 0)
};

// Scalars of the time loop kept on the device so that whole steps can be
// enqueued (and captured) without host round trips.
struct DevTime {
    double dt, dtold, ptime, endtime;
    double critts;
    int ended;        // MCM/mcm_solution.f90:101 fired
    int steps_done;   // completed loop iterations in the current mcm_gpu_run
};

// First error raised on the device; later kernels of the step return early.
struct DevStatus {
    int code;
    int req_stride;   // neighbour-list entries needed (real part); -1: a row is too long
    int req_gstride;  // neighbour-table width needed (ghost part)
    int req_ngp;      // ghost storage needed
    int req_sstride;  // skin-list entries needed
    int req_cstride;  // contact-list entries needed (real contacts)
    int req_gcstride; // contact-list entries needed (ghost contacts)
    long long req_cells;
    int bad_index;
    int max_nbr, max_gnbr;
    unsigned long long sum_nbr;  // for the mean neighbour count
};

// Linked-list grid of MCM/mcm_setuplist.f90, recomputed every step.
struct DevGrid {
    double gridmin[3];
    double gridsize[3];
    int gridlim[3];
    int pad;
    long long ncells;
    double hcut;      // largest h of the particles in cells (bounds the search reach)
    double hmin;      // smallest h of the particles in cells
    double cell[3];   // cell size 1 / gridsize
};

// Boundary planes (MCM/mcm_init_boundary.f90:28-116).
struct DevPlanes {
    int code[2][3];
    double bx[2][3];
    int type[3];
    double mult[6][3];
    double add[6][3];
};

// Run options used inside kernels.
struct DevParams {
    int ndim, disctype, tcrit_opt, boundary, baseaccel, drelax, nmat, diag;
    int asym;         // a material of the cap model is present: the momentum sum reads both triangles of sigma
    int h_opt;        // variable smoothing length (MCM/mcm_update_h.f90): 0 fixed, 1 strain rate, 2 density
    int veloc_opt;    // 1: XSPH velocity smoothing (MCM/mcm_update_velocity.f90:61-87)
    int contacttype;  // 0: particles of other materials are neighbours (kernel contact); > 0: contacts
    int contact;      // contacttype > 0 with more than one material: contact lists and repulsion are built
    int kahan;        // mixed precision: pair sums compensated per lane (Kahan) before the lane combination
    double drelax_scale, tssf, hmax;
    double skin;      // > 0: neighbour lists filtered from skin lists kept within h_i + h_j + skin * hmax
    double base_a[3];
    DevPlanes planes;
};

// Per-particle field identifiers of the FP64 state (one array of npad
// doubles each).  Symmetric tensors keep 6 components: 11 22 33 12 13 23.
enum Field {
    FX = 0, FY, FZ, FVX, FVY, FVZ, FH, FMASS, FRHO, FE, FP, FC, FEFPS, FPCUT, FPCUT2, FFAIL, FVABS, FHOLD,
    FS11, FS22, FS33, FS12, FS13, FS23,      // sigma
    FQ,                                      // isotropic artificial viscosity
    FD11, FD22, FD33, FD12, FD13, FD23,      // deviator s
    FA11, FA22, FA33, FA12, FA13, FA23,      // back stress alfa (model 3)
    FCAPA,
    // diagnostics refreshed by the split path (and on request)
    FR11, FR22, FR33, FR12, FR13, FR23,      // rod
    FW12, FW13, FW23,                        // spin
    FTR, FETRY, FEINC, FRHOOLD, FMINDIST, FCRITTS, FAX, FAY, FAZ,
    // lower triangle of sigma (21, 31, 32): equal to the upper one except for
    // the cap model, whose return map writes the upper triangle only
    FL21, FL31, FL32,
    FH0,                                     // initial smoothing length (h_opt 2)
    FXS0, FXS1, FXS2,                        // XSPH velocity sums of the step
    FRPX, FRPY, FRPZ,                        // repulsive contact acceleration (contacttype > 0)
    NFIELD
};

struct Fields {
    double *f[NFIELD];
    int *mat, *dispbc, *orig, *ptype;
};

__host__ __device__ inline long long cell_key(int bx, int by, int bz, const int *gl) {
    return (long long)(bx - 1) + (long long)gl[0] * ((long long)(by - 1) + (long long)gl[1] * (long long)(bz - 1));
}

// The grid check lets up to 2^31 - 1 cells through, and their planes' layers
// hold up to twice as many (an axis with a plane has at least two cells, one
// with two planes three): counts of either are unsigned, so that no index or
// loop counter that steps past them wraps.
constexpr unsigned kScanChunk = 4096;   // cells or layer cells per block of their scans
__host__ __device__ inline unsigned scan_chunks(unsigned n) { return n / kScanChunk + (n % kScanChunk ? 1u : 0u); }
// The layer cells of the planes in `active` (bit 2 * axis + side), plane after
// plane: first[p] is where plane p's begin, first[6] their number.
__host__ __device__ inline void layer_starts(const int *gl, unsigned active, unsigned *first) {
    first[0] = 0;
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        const int d = p >> 1;
        const unsigned area = (unsigned)gl[d == 0 ? 1 : 0] * (unsigned)gl[d == 2 ? 1 : 2];
        first[p + 1] = first[p] + ((active >> p & 1u) ? area : 0u);
    }
}

// Lower corner of cell b (1-based) along axis d of the grid.
__host__ __device__ inline double cell_origin(const DevGrid &g, int d, int b) {
    return g.gridmin[d] + (double)(b - 1) * g.cell[d];
}

// Half-width of the band around the cutoff within which the search's FP32
// distances do not decide.  With u = 2^-24 and N cells of size cell along x,
// whose coordinates are relative to the grid's origin, two of them differ from
// the true difference by e = 2 N u cell at most: the squared distance is off by
// less than (2 e / cell + (e / cell)^2 + 30 u) cell^2, and the cutoff by 5 u of
// itself.  The band is 4 times the terms in e (16 in e^2, which counts from
// some 10^7 cells on) and 8 times the rest.
__host__ __device__ inline float search_band(int n, float cell) {
    const float e4 = (float)n * 4.76837158203125e-7f;   // 4 e / cell
    return (1.52587890625e-5f + 2.0f * e4 + e4 * e4) * cell * cell;
}

// First statement of every kernel of the step's chain (launch_chained): waits
// until the launch before it in the stream has completed and its memory is
// visible.  Every path through such a kernel passes here, so the kernels still
// follow one another; and none reads memory through the non-coherent path,
// which assumes that nothing is written while the kernel is in place.
// chain_start, of the short kernels, then lets the launch behind it begin, so
// that its blocks are in place when this kernel ends.  The searches, gathers
// and the constitutive update only wait (chain_wait): blocks that wait beside
// them cost more than the launch (685 824 particles: 100.6 ms against 96.7).
__device__ __forceinline__ void chain_start() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void raise_status(DevStatus *st, int code, int idx = -1) {
    if (atomicCAS(&st->code, 0, code) == 0) st->bad_index = idx;
}

}  // namespace mcm
