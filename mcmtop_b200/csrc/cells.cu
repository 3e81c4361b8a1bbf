// cells.cu -- device cell list, boundary ghosts and the neighbour search of
// the MCM explicit step.
//
// Replaces MCM/mcm_setuplist.f90 (linked-list grid), MCM/mcm_ghost_setup.f90
// (ghost particles) and MCM/mcm_ll_neighbours.f90 (27-cell search).  The cell
// list is a counting sort by cell key (one radix digit of width = number of
// cells) followed by a per-cell sort into descending reference index, which is
// the order in which the reference walks a head-inserted linked list.  Rows of
// three x-adjacent cells are contiguous in that order, so the search visits
// candidates exactly in the reference's z/y/x cell order and the neighbour
// lists come out as the same sequences, not only the same sets.
//
// Compiled without fused multiply-add: the cell index int(gridsize*(x-gridmin))
// and the predicate d^2 < (h_i+h_j)^2 are evaluated exactly as the reference
// does in FP64, so borderline pairs resolve identically.
#include "nbr_iter.cuh"
#include "time_step.cuh"

namespace mcm {

// ------------------------------------------------------------- grid set-up
// MCM/mcm_setuplist.f90:30-81; true when a span has no finite cell count (no
// particle with a finite position leaves the box at 1e20 to -1e20).  A box that
// lies wholly beyond a plane gives an axis less than one cell: such a grid has
// none.
__device__ __forceinline__ bool make_grid(const StepArgs &a, DevGrid &g) {
    const DevParams &P = a.prm;
    const double factor = 2.0;
    const double hmax = a.hmax[0];   // fixed, or the last mcm_update_h's maximum
    for (int i = 0; i < 3; ++i) {
        g.gridmin[i] = 0.0;
        g.gridlim[i] = 1;
        g.gridsize[i] = 1.0 / (factor * hmax);
    }
    bool bad = false;
    for (int i = 0; i < P.ndim; ++i) {
        double span = 0.0;
        switch (P.planes.type[i]) {
            case 1:
                g.gridmin[i] = a.bbox[i] - 0.01 * hmax;
                span = g.gridsize[i] * (a.bbox[3 + i] - g.gridmin[i]);
                if (!(fabs(span) < 1.0e9)) { bad = true; span = 0; }
                g.gridlim[i] = (int)span + 1;
                break;
            case 2:
                g.gridmin[i] = P.planes.bx[0][i];
                span = g.gridsize[i] * (a.bbox[3 + i] - g.gridmin[i]);
                if (!(fabs(span) < 1.0e9)) { bad = true; span = 0; }
                g.gridlim[i] = (int)span + 1;
                break;
            case 3:
                span = g.gridsize[i] * (P.planes.bx[1][i] - a.bbox[i]);
                if (!(fabs(span) < 1.0e9)) { bad = true; span = 0; }
                g.gridlim[i] = (int)span + 1;
                g.gridmin[i] = P.planes.bx[1][i] - g.gridlim[i] * factor * hmax;
                break;
            case 4:
                g.gridmin[i] = P.planes.bx[0][i];
                span = g.gridsize[i] * (P.planes.bx[1][i] - P.planes.bx[0][i]);
                if (!(fabs(span) < 1.0e9)) { bad = true; span = 0; }
                g.gridlim[i] = (int)span;
                g.gridlim[i] = g.gridlim[i] > 1 ? g.gridlim[i] : 1;
                g.gridsize[i] = (double)(float)g.gridlim[i] / (P.planes.bx[1][i] - P.planes.bx[0][i]);
                break;
        }
    }
    for (int i = 0; i < P.ndim; ++i) {
        int c0 = P.planes.code[0][i];
        if (c0 == 1 || c0 == 2) {
            g.gridlim[i] = g.gridlim[i] + 1;
            g.gridmin[i] = g.gridmin[i] - (1.0 / g.gridsize[i]);
        }
        int c1 = P.planes.code[1][i];
        if (c1 == 1 || c1 == 2) g.gridlim[i] = g.gridlim[i] + 1;
    }
    g.pad = 0;
    for (int i = 0; i < 3; ++i) g.cell[i] = 1.0 / g.gridsize[i];
    g.ncells = 1;   // held at 2^31, which is too many: three axes of 10^9 would wrap
    for (int i = 0; i < 3; ++i) {
        g.ncells = g.gridlim[i] < 1 ? 0 : g.ncells * g.gridlim[i];
        if (g.ncells > (1LL << 31)) g.ncells = 1LL << 31;
    }
    g.hcut = 0.0;                                          // raised by k_cell_order
    g.hmin = __longlong_as_double(0x7fffffffffffffffll);   // lowered by k_cell_order
    return bad;
}

// --------------------------------------------------------------- cell keys
// The grid (every block forms it for itself, block 0 writes it down), the
// particles' cells (MCM/mcm_setuplist.f90:110-135: particles outside the grid
// get none) and the cells' counts.  cell_count is zero on entry: the scatter
// takes every count down to zero again.
__global__ void __launch_bounds__(256) k_cell_keys(StepArgs a) {
    chain_start();
    __shared__ DevGrid g;
    __shared__ int stop;
    // block 0 raises the status in this launch, so only thread 0 reads it: the
    // block stops or goes on as a whole
    if (threadIdx.x == 0) stop = a.status->code;
    if (threadIdx.x == 0 && !stop) {
        const bool bad = make_grid(a, g);
        stop = (bad || g.ncells >= (1LL << 31)) ? MCM_EGRID_TOO_LARGE : g.ncells > a.cell_cap ? MCM_EGRID_OVERFLOW : 0;
        if (blockIdx.x == 0) {
            if (stop == MCM_EGRID_OVERFLOW) a.status->req_cells = g.ncells;
            if (stop) raise_status(a.status, stop);
            *a.grid = g;
            *a.ngp = 0;
            *a.n_inside = 0;
            *a.scan_ticket = 0;
            *a.ghost_ticket = 0;
            *a.crit_ticket = 0;
            *a.crit_bits = order_bits((unsigned long long)__double_as_longlong(1.0e20));
        }
    }
    __syncthreads();
    if (stop) return;
    if (a.prm.boundary)
        for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < (unsigned)g.ncells; c += gridDim.x * blockDim.x)
            a.gcell[c] = make_int2(0, 0);
    const int ndim = a.prm.ndim;
    const double *X[3] = {a.F.f[FX], a.F.f[FY], a.F.f[FZ]};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        int box[3] = {1, 1, 1};
        bool in = true;
        for (int j = 0; j < ndim; ++j) {
            double t = g.gridsize[j] * (X[j][i] - g.gridmin[j]);
            // int() of the reference truncates toward zero; out-of-range values are outside anyway
            if (!(t > -2.0e9 && t < 2.0e9)) { in = false; continue; }
            box[j] = (int)t + 1;
            if (box[j] < 1 || box[j] > g.gridlim[j]) in = false;
        }
        int key = in ? (int)cell_key(box[0], box[1], box[2], g.gridlim) : kNoCell;
        a.key[i] = key;
        // lanes of one cell add their count once (the particles are mostly in
        // cell order, so a warp holds few distinct cells)
        const unsigned act = __activemask();
        const unsigned grp = __match_any_sync(act, key);
        if (key >= 0 && (threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&a.cell_count[key], __popc(grp));
    }
}

// ------------------------------------------------------------------- scan
// Exclusive prefix of cell_count: within a chunk of cells in cell_local, over
// the chunks in scan_sums (by the block that ends last; the total behind
// them).  A grid larger than the cell arrays has raised the status in
// k_cell_keys: nothing is read or written then (the step is run again once the
// arrays have grown).
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
static_assert(kScanChunk == kScanThreads * kScanItems, "a chunk per block");

__device__ __forceinline__ int block_exclusive_scan(int v, int *smem, int &total) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem[w] = x;
    __syncthreads();
    if (w == 0) {
        int s = (lane < (int)(blockDim.x >> 5)) ? smem[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        smem[lane] = s;
    }
    __syncthreads();
    int prefix = (w > 0 ? smem[w - 1] : 0) + x - v;
    total = smem[(blockDim.x >> 5) - 1];
    __syncthreads();
    return prefix;
}


__global__ void __launch_bounds__(kScanThreads) k_cell_scan(StepArgs a) {
    chain_start();
    __shared__ int smem[32];
    __shared__ int last;
    if (a.status->code) return;
    const unsigned n = (unsigned)a.grid->ncells;
    const int nblocks = scan_chunks(n);
    if (n == 0 && blockIdx.x == 0 && threadIdx.x == 0) a.scan_sums[0] = 0;
    if ((int)blockIdx.x >= nblocks) return;
    const unsigned base = blockIdx.x * kScanChunk + threadIdx.x * kScanItems;
    int v[kScanItems];
    int local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? a.cell_count[base + k] : 0;
        local += v[k];
    }
    int total;
    int pre = block_exclusive_scan(local, smem, total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) a.cell_local[base + k] = pre;
        pre += v[k];
    }
    if (threadIdx.x == 0) {
        a.scan_sums[blockIdx.x] = total;
        __threadfence();
        last = atomicAdd(a.scan_ticket, 1) == nblocks - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int carry = 0;
    for (int b = 0; b < nblocks; b += kScanThreads) {
        const int q = b + threadIdx.x;
        const int w = q < nblocks ? *(volatile int *)(a.scan_sums + q) : 0;
        const int p = block_exclusive_scan(w, smem, total);
        if (q < nblocks) a.scan_sums[q] = p + carry;
        carry += total;
    }
    if (threadIdx.x == 0) a.scan_sums[nblocks] = carry;
}

// --------------------------------------------------------------- scatter
// The cells' first positions, and the particles into their cells.  Particles
// outside the grid (llpointer = -1 in the reference) take the positions after
// the last cell; they have no neighbours and are never one.
__global__ void __launch_bounds__(256) k_cell_scatter(StepArgs a) {
    chain_start();
    if (a.status->code) return;
    const unsigned ncells = (unsigned)a.grid->ncells;
    const int base_out = a.scan_sums[scan_chunks(ncells)];
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c <= ncells; c += gridDim.x * blockDim.x)
        a.cell_start[c] = c < ncells ? a.cell_local[c] + a.scan_sums[c / kScanChunk] : base_out;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        int key = a.key[i];
        const unsigned act = __activemask();
        const unsigned grp = __match_any_sync(act, key);
        if (key < 0) {
            a.cell_list[base_out + atomicAdd(a.n_inside, 1)] = i;
            continue;
        }
        // one atomic per cell and warp: the group's slots are the n below the
        // returned count, one per lane in lane order
        const int lane = threadIdx.x & 31, lead = __ffs(grp) - 1;
        int top = 0;
        if (lane == lead) top = atomicSub(&a.cell_count[key], __popc(grp));
        top = __shfl_sync(grp, top, lead);
        int slot = top - 1 - __popc(grp & ((1u << lane) - 1u));
        a.cell_list[a.cell_local[key] + a.scan_sums[key / kScanChunk] + slot] = i;
    }
}

// ------------------------------------------------------- order and records
// Per-cell order: descending reference index (head insertion in
// MCM/mcm_setuplist.f90:126-130 over i = 1..np ascending), the order of the
// reference's lists.  (Ascending x, which lets a search window its rows,
// measured slower for every later kernel of the FP64-fast and mixed steps:
// 1.25 against 1.23 ms per mixed step of the 685 824-particle bar.)
// One warp per cell: each lane takes one of the cell's particles (cells of up
// to 32, the common case) or up to kSortPer of them, and counts how many of
// the cell's particles come before each (a rank sort: the order is total, so
// the ranks are a permutation); all ranks are known before any entry is
// written back.  Cells of more than 32 * kSortPer particles are sorted by
// insertion in one lane.
//
// The lane that has placed a particle writes its records: FP64 position and h,
// the FP32 coordinates by which the search decides all but the near-tie
// candidates (negated, one array each, x relative to the grid origin, so that
// the candidates of a row's two or three cells share one frame in x, y and z
// relative to the origin of the particle's own cell; cposf, all three relative
// to the cell, for the searches that read it), and the strain gather's record
// of the step's arithmetic REC: positions shifted back half a step
// (MCM/mcm_strain.f90:27-31), velocities and V = m/rho
// (MCM/mcm_oldstrain.f90:44).
template <int REC>
__device__ __forceinline__ void write_records(const StepArgs &a, const DevGrid &g, int p, int i, int key, double dt,
                                              bool with_cposf, unsigned long long &hbits, unsigned long long &lbits) {
    const double *const *f = a.F.f;
    const double x = f[FX][i], y = f[FY][i], z = f[FZ][i], h = f[FH][i];
    const double vx = f[FVX][i], vy = f[FVY][i], vz = f[FVZ][i];
    a.cpos[p] = make_double4(x, y, z, h);
    a.pos_of[i] = p;
    if (a.prm.boundary) a.ghost_of[i] = -1;
    a.cmat[p] = a.F.mat[i];
    a.ckey[p] = key;
    double o[3] = {0.0, 0.0, 0.0};
    float4 r = make_float4(0.f, 0.f, 0.f, (float)h);
    if (key >= 0) {
        int b[3];
        cell_coords(key, g.gridlim, b[0], b[1], b[2]);
        for (int d = 0; d < 3; ++d) o[d] = cell_origin(g, d, b[d]);
        r.x = (float)(x - o[0]);
        r.y = (float)(y - o[1]);
        r.z = (float)(z - o[2]);
        const unsigned long long hb = (unsigned long long)__double_as_longlong(h);   // h > 0: bits order like values
        hbits = hb > hbits ? hb : hbits;
        lbits = hb < lbits ? hb : lbits;
    }
    if (with_cposf) a.cposf[p] = r;
    a.snx[p] = -(float)(x - g.gridmin[0]);
    a.sny[p] = -r.y;
    a.snz[p] = -r.z;
    a.snh[p] = r.w;
    const double xs = x - 0.5 * vx * dt, ys = y - 0.5 * vy * dt, zs = z - 0.5 * vz * dt;
    const double vol = f[FMASS][i] / f[FRHO][i];
    if (REC == kRecMixed) {
        a.frec0[2 * (size_t)p] = make_float4((float)(xs - o[0]), (float)(ys - o[1]), (float)(zs - o[2]), (float)h);
        a.frec0[2 * (size_t)p + 1] = make_float4((float)vx, (float)vy, (float)vz, (float)vol);
    } else {
        a.rec0[p] = make_double4(xs, ys, zs, h);
        a.rec1[p] = make_double4(vx, vy, vz, vol);
    }
}

constexpr int kSortPer = 4;
template <int REC>
__device__ __forceinline__ void order_cell(const StepArgs &a, const DevGrid &g, int c, int s, int e, double dt,
                                           bool with_cposf, unsigned long long &hbits, unsigned long long &lbits) {
    const int lane = threadIdx.x & 31, n = e - s;
    if (n <= 32) {
        // one particle per lane (the common case)
        const bool on = lane < n;
        const int v = on ? a.cell_list[s + lane] : 0;
        const int o = on ? a.F.orig[v] : 0;
        int rank = 0;
        for (int k = 0; k < n; ++k) rank += __shfl_sync(0xffffffffu, o, k) > o ? 1 : 0;
        __syncwarp();
        if (on) {
            a.cell_list[s + rank] = v;
            write_records<REC>(a, g, s + rank, v, c, dt, with_cposf, hbits, lbits);
        }
        __syncwarp();
        return;
    }
    if (n <= 32 * kSortPer) {
        int v[kSortPer], o[kSortPer], rank[kSortPer];
#pragma unroll
        for (int u = 0; u < kSortPer; ++u) {
            const int j = lane + 32 * u;
            v[u] = j < n ? a.cell_list[s + j] : 0;
            o[u] = j < n ? a.F.orig[v[u]] : 0;
            rank[u] = 0;
        }
        for (int k0 = 0; k0 < n; k0 += 32) {
            // the chunk's keys, one per lane, broadcast by shuffles
            const int uk = k0 >> 5;
            int ok = 0;
#pragma unroll
            for (int u = 0; u < kSortPer; ++u)
                if (u == uk) ok = o[u];
            const int m = n - k0 < 32 ? n - k0 : 32;
            for (int k = 0; k < m; ++k) {
                const int ob = __shfl_sync(0xffffffffu, ok, k);
#pragma unroll
                for (int u = 0; u < kSortPer; ++u)
                    if (lane + 32 * u < n && ob > o[u]) ++rank[u];
            }
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kSortPer; ++u)
            if (lane + 32 * u < n) a.cell_list[s + rank[u]] = v[u];
    } else if (lane == 0) {
        for (int k = s + 1; k < e; ++k) {
            const int v = a.cell_list[k];
            const int ov = a.F.orig[v];
            int m = k - 1;
            while (m >= s && a.F.orig[a.cell_list[m]] < ov) {
                a.cell_list[m + 1] = a.cell_list[m];
                --m;
            }
            a.cell_list[m + 1] = v;
        }
    }
    __syncwarp();
    for (int p = s + lane; p < e; p += 32)
        write_records<REC>(a, g, p, a.cell_list[p], c, dt, with_cposf, hbits, lbits);
    __syncwarp();
}

template <int REC>
__global__ void __launch_bounds__(256) k_cell_order(StepArgs a, int with_cposf) {
    chain_start();
    __shared__ DevGrid g;
    __shared__ unsigned long long smax[8], smin[8];
    if (a.status->code) return;
    if (threadIdx.x == 0) g = *a.grid;
    __syncthreads();
    const unsigned ncells = (unsigned)g.ncells;
    const double dt = a.time->dt;
    const int lane = threadIdx.x & 31;
    const unsigned nw = gridDim.x * (blockDim.x >> 5);
    unsigned long long hbits = 0ull, lbits = ~0ull;
    // a warp takes every nw-th cell and reads the ends of 32 of them at once: of a
    // sparse grid only the cells that hold particles are walked
    for (unsigned c0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c0 < ncells; c0 += 32u * nw) {
        const unsigned c = c0 + lane * nw;
        const int s = c < ncells ? a.cell_start[c] : 0, e = c < ncells ? a.cell_start[c + 1] : 0;
        for (unsigned todo = __ballot_sync(0xffffffffu, e > s); todo; todo &= todo - 1u) {
            const int at = __ffs(todo) - 1;
            order_cell<REC>(a, g, (int)(c0 + at * nw), __shfl_sync(0xffffffffu, s, at), __shfl_sync(0xffffffffu, e, at), dt,
                            with_cposf != 0, hbits, lbits);
        }
    }
    // particles outside the grid
    for (int p = a.cell_start[ncells] + blockIdx.x * blockDim.x + threadIdx.x; p < a.n; p += gridDim.x * blockDim.x)
        write_records<REC>(a, g, p, a.cell_list[p], kNoCell, dt, with_cposf != 0, hbits, lbits);
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, hbits, o);
        const unsigned long long u = __shfl_xor_sync(0xffffffffu, lbits, o);
        hbits = v > hbits ? v : hbits;
        lbits = u < lbits ? u : lbits;
    }
    if (lane == 0) { smax[threadIdx.x >> 5] = hbits; smin[threadIdx.x >> 5] = lbits; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            hbits = smax[w] > hbits ? smax[w] : hbits;
            lbits = smin[w] < lbits ? smin[w] : lbits;
        }
        atomicMax(reinterpret_cast<unsigned long long *>(&a.grid->hcut), hbits);
        atomicMin(reinterpret_cast<unsigned long long *>(&a.grid->hmin), lbits);
    }
}

static int grid_blocks(long long work, int threads) {
    long long b = (work + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148LL * 32) b = 148LL * 32;
    return (int)b;
}

// Four launches: keys and counts, their scan, the scatter, the order within
// the cells with everything that is written per particle in cell order.  All
// but the scan loop over the cells as well as over the particles, and a few
// particles may lie in a large grid: their blocks follow both, the cells by
// the arrays' length (the host does not know the grid).  At the most 4 cells to
// a thread of the short kernels and 16 to a warp that orders them, up to the
// full chip, which the bodies that run at the same time share (24 bars on 16
// lanes: 72.1 ms without, 71.2 with, 71.2 by the particles alone).  (us a cell list, with blocks by the particles alone and a cell at
// a time, and now: 2 080 particles in 153 cells 23 and 20, in 54 972 264 and 24,
// in 4 million 18 700 and 122; 16 848 in 1 152 25 and 21, in 55 440 54 and 26;
// 685 824 in 53 240 71 and 72; 450 604 in 117 120 61 and 55.)
static int blocks_for(long long particles, long long cells) {
    const long long b = grid_blocks(particles, 256) > cells ? grid_blocks(particles, 256) : cells;
    return (int)(b < 148 * 8 ? b : 148 * 8);
}
void launch_cell_build(const StepArgs &a, cudaStream_t s) {
    const int wide = blocks_for(a.n, a.cell_cap / (4 * 256 * a.share));
    launch_chained(k_cell_keys, wide, 256, 0, s, a);
    launch_chained(k_cell_scan, (unsigned)((a.cell_cap + kScanChunk - 1) / kScanChunk), kScanThreads, 0, s, a);
    launch_chained(k_cell_scatter, wide, 256, 0, s, a);
    // about 16 particles to a warp, a cell of a full body
    const int ob = blocks_for((long long)a.n * 2, a.cell_cap / (16 * 8 * a.share));
    const int with_cposf = a.search_kind == 3 || a.prm.skin > 0.0 ? 1 : 0;
    if (a.frec0) launch_chained(k_cell_order<kRecMixed>, ob, 256, 0, s, a, with_cposf);
    else launch_chained(k_cell_order<kRecFP64>, ob, 256, 0, s, a, with_cposf);
}

// ------------------------------------------------------------- re-sorting
// Permutes the particle state into the cell order of the last step's list,
// so that the gathers of later steps walk memory nearly in order.  Results do
// not depend on it: every order used by the step is defined by cell keys and
// reference indices, not by storage positions.
__global__ void k_permute_int(const int *src, int *dst, const int *perm, int n) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) dst[p] = src[perm[p]];
}
__global__ void k_copy_back_int(const int *src, int *dst, int n) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) dst[p] = src[p];
}

// A group of nf consecutive fields (field k of the group at base + k np),
// permuted into tmp (padding copied as it is) in one pass over the positions.
__global__ void k_permute_group(const double *base, size_t np, int nf, double *tmp, const int *perm, int n) {
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < np; p += (size_t)gridDim.x * blockDim.x) {
        const size_t j = p < (size_t)n ? (size_t)perm[p] : p;
        for (int k = 0; k < nf; ++k) tmp[k * np + p] = base[k * np + j];
    }
}

void launch_reorder(const StepArgs &a, cudaStream_t s) {
    const int b = grid_blocks(a.n, 256);
    // the fields lie at F.f[0] + f npad: each group is one contiguous range
    const size_t np = (size_t)a.npad;
    for (int f0 = 0; f0 < NFIELD; f0 += kReorderGroup) {
        const int nf = NFIELD - f0 < kReorderGroup ? NFIELD - f0 : kReorderGroup;
        k_permute_group<<<b, 256, 0, s>>>(a.F.f[f0], np, nf, a.reorder_grp, a.cell_list, a.n);
        cudaMemcpyAsync(a.F.f[f0], a.reorder_grp, sizeof(double) * nf * np, cudaMemcpyDeviceToDevice, s);
    }
    int *ints[4] = {a.F.mat, a.F.dispbc, a.F.orig, a.F.ptype};
    for (int *p : ints) {
        k_permute_int<<<b, 256, 0, s>>>(p, (int *)a.reorder_tmp, a.cell_list, a.n);
        k_copy_back_int<<<b, 256, 0, s>>>((const int *)a.reorder_tmp, p, a.n);
    }
}

// ------------------------------------------------------------------ ghosts
// MCM/mcm_ghost_setup.f90:29-284.  The reference makes the planes' ghosts one
// plane after the other (xmin xmax ymin ymax zmin zmax): each walks the 2-D
// layer of cells inside the plane and emits, per source cell, its members in
// chain order into the cell outside.  A later plane's source cell may itself lie
// in the layer of an earlier plane and then holds ghosts, newest first.  Where
// a cell's content comes from follows from its coordinates alone, so all planes
// are made at once: the layer cells of all planes, in the reference's order,
// are one sequence; each looks up the cell whose real particles it mirrors and
// through which planes, one scan over the counts gives the ghosts' numbers, and
// then every cell writes its ghosts.  Two launches and no waiting of one plane
// for another (one plane took 20 us and five 84 however few particles).

// The layer cells of the active planes, plane after plane.
struct Layers {
    unsigned first[7];   // of each plane's cells in the sequence
    unsigned active;     // bit 2 * axis + side
    int gl[3];
};
__device__ __forceinline__ Layers make_layers(const StepArgs &a) {
    Layers l;
    for (int d = 0; d < 3; ++d) l.gl[d] = a.grid->gridlim[d];
    l.active = 0u;
    // an axis of one cell has no layer to mirror; a grid without cells has none
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        const int code = a.prm.planes.code[p & 1][p >> 1];
        if ((code == 1 || code == 2) && (p >> 1) < a.prm.ndim && l.gl[p >> 1] > 1 && a.grid->ncells > 0) l.active |= 1u << p;
    }
    layer_starts(l.gl, l.active, l.first);
    return l;
}
__device__ __forceinline__ int layer_key(const Layers &l, const int *c) {
    return (c[0] - 1) + l.gl[0] * ((c[1] - 1) + l.gl[1] * (c[2] - 1));   // below 2^31
}
// Coordinate of the layer that plane (d, side) mirrors.
__device__ __forceinline__ int source_layer(const StepArgs &a, const Layers &l, int d, int side) {
    const bool sym = a.prm.planes.code[side][d] == 1;
    return (side == 0) == sym ? 2 : l.gl[d] - 1;
}

// Where layer cell t's ghosts come from: the real particles of cell `from`,
// mirrored through planes[depth - 1], ..., planes[0] in turn; `to` receives
// them.
//
// The source cell may lie in the layers of earlier axes; it then holds the
// ghosts of the last of them whose own source held anything, and so on down.
// With one hop per such axis, from the layer to the cell it mirrors, what the
// cell holds are the reals of the one cell of {no hop, first axis, second axis,
// both} that has any.  Two that have some mean that a cell holds both reals and
// ghosts, or the ghosts of two planes, and so does one of the four around `to`
// when it receives any: MCM_EGHOST_LAYER.
struct Origin {
    int from, to, count, depth, planes[3];
};
__device__ __forceinline__ Origin origin_of(const StepArgs &a, const Layers &l, unsigned t) {
    int plane = 0;
#pragma unroll
    for (int p = 1; p < 6; ++p)
        if (t >= l.first[p]) plane = p;
    const int d = plane >> 1, side = plane & 1;
    const int ad = d == 2 ? 1 : 2, bd = d == 0 ? 1 : 0;   // the layer's outer and inner axis
    const int r = (int)(t - l.first[plane]);   // a layer has less than 2^31 cells
    const int nb = l.gl[bd];
    int c[3];
    c[ad] = r / nb + 1;
    c[bd] = r - (c[ad] - 1) * nb + 1;
    Origin o;
    c[d] = side == 0 ? 1 : l.gl[d];
    o.to = layer_key(l, c);
    c[d] = source_layer(a, l, d, side);
    const int source = layer_key(l, c);
    unsigned in = 0u;          // earlier axes along which the cell lies in a layer
    int hop[2] = {0, 0}, via[2] = {0, 0};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        if (e >= d) continue;
        const int es = c[e] == 1 && (l.active >> (2 * e) & 1u) ? 0 : (c[e] == l.gl[e] && (l.active >> (2 * e + 1) & 1u) ? 1 : -1);
        if (es < 0) continue;
        in |= 1u << e;
        via[e] = 2 * e + es;
        hop[e] = (source_layer(a, l, e, es) - c[e]) * (e == 0 ? 1 : l.gl[0]);
    }
    o.from = source;
    o.count = 0;
    unsigned taken = 0u;
    bool clash = false;
#pragma unroll
    for (unsigned m = 0u; m < 4u; ++m) {
        if (m & ~in) continue;
        const int k = source + (m & 1u ? hop[0] : 0) + (m & 2u ? hop[1] : 0);
        const int n = a.cell_start[k + 1] - a.cell_start[k];
        if (n == 0) continue;
        clash = clash || o.count > 0;
        o.from = k;
        o.count = n;
        taken = m;
    }
    if (o.count > 0) {
#pragma unroll
        for (unsigned m = 0u; m < 4u; ++m) {
            if (m & ~in) continue;
            const int k = o.to + (m & 1u ? hop[0] : 0) + (m & 2u ? hop[1] : 0);
            clash = clash || a.cell_start[k + 1] > a.cell_start[k];
        }
        if (clash) raise_status(a.status, MCM_EGHOST_LAYER, o.to);
    }
    o.depth = 1 + __popc(taken);
    o.planes[0] = plane;
    o.planes[1] = taken & 2u ? via[1] : via[0];
    o.planes[2] = via[0];
    return o;
}

// Counts of the layer cells and their prefix sums: within a chunk in
// layer_off, over the chunks in layer_sums (by the block that ends last).
__global__ void __launch_bounds__(kScanThreads) k_ghost_count(StepArgs a) {
    chain_start();
    __shared__ int smem[32];
    __shared__ int last;
    // EGHOST_LAYER may be this launch's own
    if (__syncthreads_or(a.status->code && a.status->code != MCM_EGHOST_LAYER)) return;
    const Layers l = make_layers(a);
    const unsigned T = l.first[6];
    if (T > a.layer_cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(a.status, MCM_EGRID_OVERFLOW);
        return;
    }
    const unsigned base = blockIdx.x * kScanChunk;
    const int nblocks = scan_chunks(T);   // blocks that hold layer cells
    if ((int)blockIdx.x >= nblocks) return;
    int v[kScanItems];
    int local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const unsigned t = base + threadIdx.x * kScanItems + k;
        v[k] = t < T ? origin_of(a, l, t).count : 0;
        local += v[k];
    }
    int total;
    int pre = block_exclusive_scan(local, smem, total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const unsigned t = base + threadIdx.x * kScanItems + k;
        if (t < T) {
            a.layer_count[t] = v[k];
            a.layer_off[t] = pre;
        }
        pre += v[k];
    }
    int carry = 0;
    if (nblocks == 1) {
        if (threadIdx.x == 0) a.layer_sums[0] = 0;
        carry = total;
    } else {
        if (threadIdx.x == 0) {
            a.layer_sums[blockIdx.x] = total;
            __threadfence();
            last = atomicAdd(a.ghost_ticket, 1) == nblocks - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
    }
    for (int b = 0; nblocks > 1 && b < nblocks; b += kScanThreads) {
        const int q = b + threadIdx.x;
        const int n = q < nblocks ? *(volatile int *)(a.layer_sums + q) : 0;
        const int p = block_exclusive_scan(n, smem, total);
        if (q < nblocks) a.layer_sums[q] = p + carry;
        carry += total;
    }
    if (threadIdx.x == 0) {
        if (carry > a.ghost_cap) {
            if (carry > a.status->req_ngp) a.status->req_ngp = carry;
            raise_status(a.status, MCM_EGHOST_OVERFLOW);
        }
        *a.ngp = carry;
    }
}

// One warp per layer cell, its lanes over the cell's ghosts.
__global__ void k_ghost_emit(StepArgs a) {
    chain_start();
    if (a.status->code) return;
    const Layers l = make_layers(a);
    const unsigned T = l.first[6];
    const int lane = threadIdx.x & 31;
    const unsigned nw = gridDim.x * (blockDim.x >> 5);
    for (unsigned t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < T; t += nw) {
        const int cnt = a.layer_count[t];
        if (cnt == 0) continue;
        const Origin o = origin_of(a, l, t);
        const int g0 = a.layer_sums[t / kScanChunk] + a.layer_off[t];
        if (lane == 0) a.gcell[o.to] = make_int2(g0, cnt);
        const int rs = a.cell_start[o.from];
        for (int r = lane; r < cnt; r += 32) {
            const int g = g0 + r;
            // MCM/mcm_ghost_setup.f90:324-355 (create_ghost_from_real), :392-423
            // (create_ghost_from_ghost: the chain's order turns round each time)
            const int j = a.cell_list[rs + ((o.depth & 1) ? r : cnt - 1 - r)];
            double x[3] = {a.F.f[FX][j], a.F.f[FY][j], a.F.f[FZ][j]};
            double v[3] = {a.F.f[FVX][j], a.F.f[FVY][j], a.F.f[FVZ][j]};
            int flips = 0;
#pragma unroll
            for (int q = 2; q >= 0; --q) {
                if (q >= o.depth) continue;
                const int plane = o.planes[q];
                const double *mult = a.prm.planes.mult[plane];
                const double *add = a.prm.planes.add[plane];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    x[d] = x[d] * mult[d] + add[d];
                    v[d] = v[d] * mult[d];
                    // axes mirrored (bit d: x_d -> -x_d + add_d), composed along the chain
                    if (mult[d] < 0.0) flips ^= 1 << d;
                }
            }
            a.gpar[g] = j;
            a.gnext[g] = atomicExch(&a.ghost_of[j], g);
            a.gflip[g] = flips;
            a.gmat[g] = a.F.mat[j];
            a.gmass[g] = a.F.f[FMASS][j];
            a.gh[g] = a.F.f[FH][j];
            a.ghold[g] = a.F.f[FHOLD][j];
            a.grho[g] = a.F.f[FRHO][j];
            a.gx[g] = x[0];
            a.gy[g] = x[1];
            a.gz[g] = x[2];
            a.gvx[g] = v[0];
            a.gvy[g] = v[1];
            a.gvz[g] = v[2];
            // the strain gather's records: ghosts keep their unshifted positions
            const double vol = a.F.f[FMASS][j] / a.F.f[FRHO][j];
            a.grec0[g] = make_double4(x[0], x[1], x[2], a.F.f[FH][j]);
            if (a.frec0) a.gfrec1[g] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)vol);
            else a.grec1[g] = make_double4(v[0], v[1], v[2], vol);
        }
    }
}

void launch_ghosts(const StepArgs &a, cudaStream_t s) {
    launch_chained(k_ghost_count, scan_chunks(a.layer_cap), kScanThreads, 0, s, a);
    long long eb = ((long long)a.layer_cap + 7) / 8;   // 8 warps (layer cells) per block
    if (eb > 148LL * 4) eb = 148LL * 4;
    launch_chained(k_ghost_emit, (unsigned)(eb < 1 ? 1 : eb), 256, 0, s, a);
}

// ------------------------------------------------------------------ search
// MCM/mcm_ll_neighbours.f90:96-299.  The candidates of the particle at
// cell-order position t are the cells of its 27-cell neighbourhood in z, y, x
// order, each a contiguous range of positions in the reference's order, so
// appending the accepted ones in position order gives the reference's lists.
//
// Two phases.  First every candidate is reduced to one bit: groups of four
// aligned positions are read as three 16-byte loads (negated x, y and z lie in
// arrays of their own), the distances of two candidates are formed by one
// packed FP32 instruction each, with the cutoff as the chain's starting value,
// so the sign of the result is the decision and a funnel shift moves it into
// the mask: about 6 instructions a candidate, without divergence or stores.
// Then the set bits (one candidate in six) are walked in position order and
// written.  The FP32 decision is final outside a narrow band around the
// cutoff, wider than the FP32 rounding; a mask with a candidate inside the
// band (a signed integer minimum over the results finds it: of the negative
// floats those nearest zero are the smallest integers) is walked through the
// reference's FP64 expression before it is written, as all are when the FP64
// minimum distance is wanted.  Cells whose box lies beyond h_i + max h cannot
// hold a neighbour and are left out.

__device__ __forceinline__ double exact_d2(double4 a, double4 b) {
    double d = __dsub_rn(b.x, a.x);
    double s = __dmul_rn(d, d);
    d = __dsub_rn(b.y, a.y);
    s = __dadd_rn(s, __dmul_rn(d, d));
    d = __dsub_rn(b.z, a.z);
    s = __dadd_rn(s, __dmul_rn(d, d));
    return s;
}

// Variants of the search, fixed at compile time so that the common case (one
// material, no repulsive contact, no minimum distance) tests none of them.
enum { kSrchContact = 1, kSrchTwoPass = 2, kSrchMind = 4 };

// What the search of one particle needs of it and of the grid.
struct Seeker {
    double4 xi;
    float qx, ux, uy, uz;     // x relative to the grid origin; x, y, z to the own cell's
    float cs[3];              // cell size
    float hi, reach2, kb;     // own h; squared box reach; decision band
    bool uni;                 // one smoothing length for all
    float thr;                // then: minus the upper cutoff
    int tie_at;               // results below this as signed integers lie in the band
    int key, gl0, gl1;        // own cell, the grid's extent in x and y
    int bx, by, bz, lo1, hi1, lo2, hi2;
    bool has_l, has_r;
    // key of the own cell's neighbour in row (my, nz)
    __device__ __forceinline__ int row_key(int my, int nz) const { return key + gl0 * ((my - by) + gl1 * (nz - bz)); }
};
constexpr float kRelBand = 3.814697265625e-6f;   // 2^-18

__device__ __forceinline__ Seeker make_seeker(const StepArgs &a, const DevGrid &g, int t, int key) {
    Seeker k;
    k.key = key;
    k.gl0 = g.gridlim[0];
    k.gl1 = g.gridlim[1];
    cell_coords(key, g.gridlim, k.bx, k.by, k.bz);
    k.lo1 = k.by > 1 ? k.by - 1 : 1;
    k.hi1 = k.by < g.gridlim[1] ? k.by + 1 : g.gridlim[1];
    k.lo2 = k.bz > 1 ? k.bz - 1 : 1;
    k.hi2 = k.bz < g.gridlim[2] ? k.bz + 1 : g.gridlim[2];
    k.has_l = k.bx > 1;
    k.has_r = k.bx < g.gridlim[0];
    k.xi = a.cpos[t];
    for (int d = 0; d < 3; ++d) k.cs[d] = (float)g.cell[d];
    const float csm = fmaxf(k.cs[0], fmaxf(k.cs[1], k.cs[2]));
    k.hi = (float)k.xi.w;
    k.qx = -a.snx[t];
    k.uy = -a.sny[t];
    k.uz = -a.snz[t];
    k.ux = (float)(k.xi.x - cell_origin(g, 0, k.bx));
    k.kb = search_band(g.gridlim[0], csm);
    const float reach = k.hi + (float)g.hcut;
    k.reach2 = reach * reach * 1.0009765625f + 9.765625e-4f * csm * csm;
    k.uni = g.hmin == g.hcut;
    const float r = k.hi + k.hi;
    k.thr = -(r * r * (1.0f + kRelBand) + k.kb);
    k.tie_at = __float_as_int(-(reach * reach * (2.0f * kRelBand) * 1.0009765625f + 2.0f * k.kb));
    return k;
}
// squared y-z distance of the row (my, nz)'s boxes
__device__ __forceinline__ float row_gap2(const Seeker &k, int my, int nz) {
    const float gz = fmaxf(nz < k.bz ? k.uz : (nz > k.bz ? k.cs[2] - k.uz : 0.0f), 0.0f);
    const float gy = fmaxf(my < k.by ? k.uy : (my > k.by ? k.cs[1] - k.uy : 0.0f), 0.0f);
    return gy * gy + gz * gz;
}

// The decision bits of groups g0 .. g0 + m - 1 (1 <= m <= 8), candidate c at
// bit 31 - c; least: the signed minimum over the results.  Groups are taken
// two at a time, so one group past the range may be read (the arrays are
// padded) and positions outside the caller's range have to be masked off.
// UNI: one smoothing length; otherwise the candidate's own h enters the cutoff.
template <bool UNI>
__device__ __forceinline__ unsigned group_bits(const StepArgs &a, int g0, int m, float qx, float qy, float qz,
                                               const Seeker &k, int &least) {
    const float4 *X = reinterpret_cast<const float4 *>(a.snx) + g0;
    const float4 *Y = reinterpret_cast<const float4 *>(a.sny) + g0;
    const float4 *Z = reinterpret_cast<const float4 *>(a.snz) + g0;
    const float4 *H = reinterpret_cast<const float4 *>(a.snh) + g0;
    const float2 qx2 = make_float2(qx, qx), qy2 = make_float2(qy, qy), qz2 = make_float2(qz, qz);
    const float2 thr = make_float2(k.thr, k.thr), hi2 = make_float2(k.hi, k.hi);
    const float2 rel = make_float2(-(1.0f + kRelBand), -(1.0f + kRelBand)), band = make_float2(-k.kb, -k.kb);
    unsigned bits = 0u;
    const int turns = (m + 1) >> 1;
#pragma unroll 1
    for (int j = 0; j < turns; ++j) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float4 x = X[2 * j + u], y = Y[2 * j + u], z = Z[2 * j + u];
            float2 t0 = thr, t1 = thr;
            if (!UNI) {
                const float4 h = H[2 * j + u];
                const float2 h0 = __fadd2_rn(hi2, make_float2(h.x, h.y)), h1 = __fadd2_rn(hi2, make_float2(h.z, h.w));
                t0 = __ffma2_rn(__fmul2_rn(h0, rel), h0, band);
                t1 = __ffma2_rn(__fmul2_rn(h1, rel), h1, band);
            }
            const float2 dx0 = __fadd2_rn(qx2, make_float2(x.x, x.y)), dx1 = __fadd2_rn(qx2, make_float2(x.z, x.w));
            const float2 dy0 = __fadd2_rn(qy2, make_float2(y.x, y.y)), dy1 = __fadd2_rn(qy2, make_float2(y.z, y.w));
            const float2 dz0 = __fadd2_rn(qz2, make_float2(z.x, z.y)), dz1 = __fadd2_rn(qz2, make_float2(z.z, z.w));
            t0 = __ffma2_rn(dz0, dz0, t0);
            t1 = __ffma2_rn(dz1, dz1, t1);
            t0 = __ffma2_rn(dy0, dy0, t0);
            t1 = __ffma2_rn(dy1, dy1, t1);
            t0 = __ffma2_rn(dx0, dx0, t0);
            t1 = __ffma2_rn(dx1, dx1, t1);
            const int i0 = __float_as_int(t0.x), i1 = __float_as_int(t0.y);
            const int i2 = __float_as_int(t1.x), i3 = __float_as_int(t1.y);
            bits = __funnelshift_l((unsigned)i0, bits, 1);
            bits = __funnelshift_l((unsigned)i1, bits, 1);
            bits = __funnelshift_l((unsigned)i2, bits, 1);
            bits = __funnelshift_l((unsigned)i3, bits, 1);
            least = min(least, min(min(i0, i1), min(i2, i3)));
        }
    }
    return bits << (32 - 8 * turns);
}

// The bits of the positions of [pb, pe) in the 32 from p0 = 4 g0 on, without t
// itself; those in the decision band settled by the reference's FP64
// expression, which also gives the minimum distance (of the own material's
// particles with repulsive contact).
template <int V>
__device__ __forceinline__ unsigned accept_bits(const StepArgs &a, const Seeker &k, int t, int mati, int g0, int m,
                                                int pb, int pe, float qy, float qz, double &mind) {
    constexpr bool want_mind = (V & kSrchMind) != 0;
    const int p0 = 4 * g0;
    int least = 0x7fffffff;
    unsigned bits = k.uni ? group_bits<true>(a, g0, m, k.qx, qy, qz, k, least)
                          : group_bits<false>(a, g0, m, k.qx, qy, qz, k, least);
    if (p0 < pb) bits &= 0xffffffffu >> (pb - p0);
    if (pe - p0 < 32) bits &= ~(0xffffffffu >> (pe - p0));
    if ((unsigned)(t - p0) < 32u) bits &= ~(0x80000000u >> (t - p0));
    if (want_mind || least < k.tie_at) {
        unsigned left = bits;
        while (left) {
            const int c = __clz(left);
            left &= ~(0x80000000u >> c);
            const double4 cd = a.cpos[p0 + c];
            const double d2 = exact_d2(k.xi, cd);
            const double hs = __dadd_rn(cd.w, k.xi.w);
            if (!(d2 < __dmul_rn(hs, hs))) bits &= ~(0x80000000u >> c);
            else if (want_mind && (!(V & kSrchContact) || a.cmat[p0 + c] == mati)) mind = fmin(mind, d2);
        }
    }
    return bits;
}

// The set bits that belong to particles of other materials.
__device__ __forceinline__ unsigned other_bits(const StepArgs &a, unsigned bits, int p0, int mati) {
    unsigned oth = 0u, left = bits;
    while (left) {
        const int c = __clz(left);
        left &= ~(0x80000000u >> c);
        if (a.cmat[p0 + c] != mati) oth |= 0x80000000u >> c;
    }
    return oth;
}

// Ghost neighbours (and contacts) of t, found by the G lanes of grp together:
// only neighbourhoods that reach a ghost layer have any; a cell's ghosts are
// visited newest first (the reference's chain order).
template <int V, int G>
__device__ __forceinline__ void search_ghosts(const StepArgs &a, const Seeker &k, int t, int i,
                                              int mati, int sub, unsigned grp, int &gn, int &gcn, double &mind) {
    constexpr bool contact = (V & kSrchContact) != 0;
    constexpr bool two_pass = (V & kSrchTwoPass) != 0;
    const int lo0 = k.has_l ? k.bx - 1 : k.bx, hi0 = k.has_r ? k.bx + 1 : k.bx;
    const DevPlanes &pl = a.prm.planes;
    const bool near = (lo0 == 1 && pl.code[0][0]) || (hi0 == k.gl0 && pl.code[1][0]) ||
                      (k.lo1 == 1 && pl.code[0][1]) || (k.hi1 == k.gl1 && pl.code[1][1]) ||
                      (k.lo2 == 1 && pl.code[0][2]) || (k.hi2 == a.grid->gridlim[2] && pl.code[1][2]);
    if (!near) return;
    const int np = a.npad;
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll 1
    for (int pass = 0; pass < (two_pass ? 2 : 1); ++pass) {
        for (int nz = k.lo2; nz <= k.hi2; ++nz)
            for (int my = k.lo1; my <= k.hi1; ++my)
                for (int lx = lo0; lx <= hi0; ++lx) {
                    const int2 gc = a.gcell[k.row_key(my, nz) + lx - k.bx];
                    for (int r0 = 0; r0 < gc.y; r0 += G) {
                        const int r = r0 + sub;
                        const int q = gc.x + gc.y - 1 - r;
                        bool in = false, inc = false;
                        if (r < gc.y) {
                            const double4 c = make_double4(a.gx[q], a.gy[q], a.gz[q], a.gh[q]);
                            const double d2 = exact_d2(k.xi, c);
                            const double hs = __dadd_rn(c.w, k.xi.w);
                            in = d2 < __dmul_rn(hs, hs);
                            if (contact && in && a.gmat[q] != mati) { inc = true; in = false; }
                            if (two_pass && in) in = (a.gmat[q] == mati) == (pass == 0);
                            if (in) mind = fmin(mind, d2);
                        }
                        if (G == 1) {
                            if (in) {
                                if (gn < a.gstride) a.gnbr[(size_t)gn * np + t] = q;
                                ++gn;
                            }
                            if (contact && inc) {
                                if (gcn < a.gcstride) a.gcont[(size_t)gcn * np + t] = q;
                                ++gcn;
                            }
                        } else {
                            const unsigned bal = __ballot_sync(grp, in) & grp;
                            const int at = gn + __popc(bal & below);
                            if (in && at < a.gstride) a.gnbr[(size_t)at * np + t] = q;
                            gn += __popc(bal);
                            if (contact) {
                                const unsigned cb = __ballot_sync(grp, inc) & grp;
                                const int ac = gcn + __popc(cb & below);
                                if (inc && ac < a.gcstride) a.gcont[(size_t)ac * np + t] = q;
                                gcn += __popc(cb);
                            }
                        }
                    }
                }
    }
    if (sub == 0 && gn > a.gstride) {
        atomicMax(&a.status->req_gstride, gn);
        raise_status(a.status, MCM_ENBR_OVERFLOW, i);
    }
    if (contact && sub == 0 && gcn > a.gcstride) {
        atomicMax(&a.status->req_gcstride, gcn);
        raise_status(a.status, MCM_ENBR_OVERFLOW, i);
    }
}

// Counts of t, and the largest of a warp's for the status.
template <int V>
__device__ __forceinline__ void search_counts(const StepArgs &a, int t, int i, int nn, int gn, int nc, int gcn, double mind) {
    a.nnbr[t] = nn;
    a.gnnbr[t] = gn;
    if (V & kSrchContact) { a.ncont[t] = nc; a.gncont[t] = gcn; }
    if (V & kSrchMind) a.F.f[FMINDIST][i] = mind;
}
__device__ __forceinline__ void search_max(const StepArgs &a, int nn, int gn) {
    const int mn = __reduce_max_sync(0xffffffffu, nn), mg = __reduce_max_sync(0xffffffffu, gn);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&a.status->max_nbr, mn);
        atomicMax(&a.status->max_gnbr, mg);
    }
}
__device__ __forceinline__ void list_overflow(const StepArgs &a, int i, int nn, int nc, bool contact) {
    if (nn > a.nstride) {
        atomicMax(&a.status->req_stride, nn);
        raise_status(a.status, MCM_ENBR_OVERFLOW, i);
    }
    if (contact && nc > a.cstride) {
        atomicMax(&a.status->req_cstride, nc);
        raise_status(a.status, MCM_ENBR_OVERFLOW, i);
    }
}

// One thread per particle (bodies that fill the chip; 64 registers for 32 warps
// per SM, with 52 to 72 bytes spilled).  The lanes of a warp walk
// the nine rows together (they lie in one or two cells, so their rows mostly
// are the same ones), 32 candidates to a mask, and collect their entries in
// shared memory, entry k of lane l at word 33 k + l.  When a lane has no room
// for the next mask the whole warp moves the collected entries on, eight lanes
// to a particle, each with one 16-byte store per four entries (rows start at
// multiples of 4); up to three stay behind.
constexpr int kSearchThreads = 256;   // the most a block of a search may have (128 unless the caller asks)
constexpr int kSrchKeep = 36;   // entries a lane can hold
template <int V>
__global__ void __launch_bounds__(kSearchThreads, 4) k_search(StepArgs a) {
    chain_wait();
    constexpr bool contact = (V & kSrchContact) != 0;   // contacttype > 0: other materials -> contact list
    constexpr bool two_pass = (V & kSrchTwoPass) != 0;  // kernel contact between materials: own material first
    constexpr unsigned kAll = 0xffffffffu;
    extern __shared__ unsigned stage_all[];             // 33 kSrchKeep words per warp
    if (a.status->code) return;
    const int lane = threadIdx.x & 31;
    unsigned *keep = stage_all + (threadIdx.x >> 5) * (33 * kSrchKeep) + lane;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int cap = a.nstride;
    const int key = t < a.n ? a.ckey[t] : kNoCell;
    const bool live = key >= 0;
    Seeker k;
    if (live) k = make_seeker(a, *a.grid, t, key);
    const int mati = (live && (contact || two_pass)) ? a.cmat[t] : 0;
    int nn = 0, held = 0;   // entries in the list (a multiple of 4) and in keep
    int nc = 0, gn = 0, gcn = 0;
    double mind = 1.0e20;
    unsigned *row0 = a.nidx + (size_t)(t - lane) * cap;   // list of the warp's first particle
    auto move_on = [&]() {
        __syncwarp();
        const int quads = held >> 2;
#pragma unroll 1
        for (int p0 = 0; p0 < 32; p0 += 4) {
            const int p = p0 + (lane >> 3), q = lane & 7;
            const int nq = __shfl_sync(kAll, quads, p), at = __shfl_sync(kAll, nn, p);
            const unsigned *src = keep - lane + p;
            unsigned *dst = row0 + (size_t)p * cap + at;
            for (int i = q; i < nq; i += 8) {
                const uint4 v = make_uint4(src[33 * (4 * i)], src[33 * (4 * i + 1)], src[33 * (4 * i + 2)], src[33 * (4 * i + 3)]);
                if (at + 4 * i + 4 <= cap) *reinterpret_cast<uint4 *>(dst + 4 * i) = v;
            }
        }
        __syncwarp();
        const int left = held & 3;
        for (int i = 0; i < left; ++i) keep[33 * i] = keep[33 * (4 * quads + i)];
        nn += 4 * quads;
        held = left;
    };
    const float gxl = fmaxf(k.ux, 0.0f), gxr = fmaxf(k.cs[0] - k.ux, 0.0f);
    int others = 0;   // two_pass: neighbours of other materials, appended by a second walk
#pragma unroll 1
    for (int pass = 0; pass < (two_pass ? 2 : 1); ++pass) {
        if (two_pass && pass == 1 && !__any_sync(kAll, others > 0)) break;
#pragma unroll 1
        for (int row = 0; row < 9; ++row) {
            const int dy = row % 3 - 1, dz = row / 3 - 1;
            int pb = 0, pe = 0, s1 = 0, s2 = 0;
            float qy = 0.0f, qz = 0.0f;
            if (live && !(two_pass && pass == 1 && others == 0)) {
                const int my = k.by + dy, nz = k.bz + dz;
                const float gyz = row_gap2(k, my, nz);
                if (my >= k.lo1 && my <= k.hi1 && nz >= k.lo2 && nz <= k.hi2 && !(gyz > k.reach2)) {
                    const int kc = k.row_key(my, nz);
                    s1 = a.cell_start[kc];
                    s2 = a.cell_start[kc + 1];
                    pb = (k.has_l && !(gyz + gxl * gxl > k.reach2)) ? a.cell_start[kc - 1] : s1;
                    pe = (k.has_r && !(gyz + gxr * gxr > k.reach2)) ? a.cell_start[kc + 2] : s2;
                    qy = k.uy - (float)dy * k.cs[1];
                    qz = k.uz - (float)dz * k.cs[2];
                }
            }
            const unsigned code = (unsigned)(3 * row) << 26;
            const int ge = pb < pe ? (pe + 3) >> 2 : 0;
#pragma unroll 1
            for (int g0 = pb >> 2; __any_sync(kAll, g0 < ge); g0 += 8) {
                unsigned bits = 0u;
                if (g0 < ge) bits = accept_bits<V>(a, k, t, mati, g0, min(8, ge - g0), pb, pe, qy, qz, mind);
                if (contact || two_pass) {
                    unsigned oth = other_bits(a, bits, 4 * g0, mati);
                    bits &= ~oth;
                    if (two_pass && pass == 0) others += __popc(oth);
                    if (two_pass && pass == 1) bits = oth;
                    if (contact) {
                        while (oth) {
                            const int b = __clz(oth);
                            oth &= ~(0x80000000u >> b);
                            const int p = 4 * g0 + b;
                            unsigned e = (unsigned)p + code;
                            if (p >= s1) e += 1u << 26;
                            if (p >= s2) e += 1u << 26;
                            if (nc < a.cstride) a.cidx[(size_t)t * a.cstride + nc] = e;
                            ++nc;
                        }
                    }
                }
                if (__any_sync(kAll, held + __popc(bits) > kSrchKeep)) move_on();
                unsigned *to = keep + 33 * held;
                held += __popc(bits);
                while (bits) {
                    const int b = __clz(bits);
                    bits ^= 0x80000000u >> b;
                    const int p = 4 * g0 + b;
                    unsigned e = (unsigned)p + code;
                    if (p >= s1) e += 1u << 26;
                    if (p >= s2) e += 1u << 26;
                    *to = e;
                    to += 33;
                }
            }
        }
    }
    move_on();
    for (int i = 0; i < held; ++i)
        if (nn + i < cap) a.nidx[(size_t)t * cap + nn + i] = keep[33 * i];
    nn += held;
    if (t < a.n) {
        const int i = a.cell_list[t];
        if (live) {
            list_overflow(a, i, nn, nc, contact);
            if (a.prm.boundary) search_ghosts<V, 1>(a, k, t, i, mati, 0, 0u, gn, gcn, mind);
            mind = sqrt(mind);
        }
        if (a.prm.disctype == 1) nn += 1;   // MCM/mcm_ll_neighbours.f90:288-299 (for every particle)
        search_counts<V>(a, t, i, nn, gn, nc, gcn, mind);
    }
    search_max(a, nn, gn);
}

// G lanes per particle (bodies too small to fill the chip with one thread per
// particle; 80 registers, 72 to 132 bytes spilled).  A row's three cells are one contiguous range; each lane takes a
// run of its groups, and the lanes' counts give each where its entries begin.
// The three rows of a plane are decided before any is written, so that their
// loads overlap.
template <int V, int G>
__global__ void __launch_bounds__(kSearchThreads, 3) k_search_lanes(StepArgs a) {
    chain_wait();
    constexpr bool contact = (V & kSrchContact) != 0;
    constexpr bool two_pass = (V & kSrchTwoPass) != 0;
    constexpr bool want_mind = (V & kSrchMind) != 0;
    if (a.status->code) return;
    const int t = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) / G);
    const int sub = threadIdx.x % G;
    // the G lanes of a particle take every branch below together
    const unsigned grp = ((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
    const int cap = a.nstride;
    int nn = 0, gn = 0;
    if (t < a.n) {
        const int key = a.ckey[t];
        const int i = a.cell_list[t];
        int nc = 0, gcn = 0;
        double mind = 1.0e20;
        if (key >= 0) {
            const Seeker k = make_seeker(a, *a.grid, t, key);
            const int mati = (contact || two_pass) ? a.cmat[t] : 0;
            unsigned *out = a.nidx + (size_t)t * cap;
            unsigned *cout = contact ? a.cidx + (size_t)t * a.cstride : nullptr;
            const float gxl = fmaxf(k.ux, 0.0f), gxr = fmaxf(k.cs[0] - k.ux, 0.0f);
            // exclusive sums over the lanes; total gets the sum
            auto scan = [&](int v, int &total) {
                int x = v;
#pragma unroll
                for (int o = 1; o < G; o <<= 1) {
                    const int y = __shfl_up_sync(grp, x, o, G);
                    if (sub >= o) x += y;
                }
                total = __shfl_sync(grp, x, G - 1, G);
                return x - v;
            };
            auto write = [&](unsigned set, int at, unsigned *list, int room, int p0, int s1, int s2, unsigned code) {
                while (set) {
                    const int b = __clz(set);
                    set &= ~(0x80000000u >> b);
                    const int p = p0 + b;
                    unsigned e = (unsigned)p + (code << 26);
                    if (p >= s1) e += 1u << 26;
                    if (p >= s2) e += 1u << 26;
                    if (at < room) list[at] = e;
                    ++at;
                }
            };
            int others = 0;
#pragma unroll 1
            for (int pass = 0; pass < (two_pass ? 2 : 1); ++pass) {
                if (two_pass && pass == 1 && others == 0) break;
#pragma unroll 1
                for (int nz = k.lo2; nz <= k.hi2; ++nz) {
                    const float qz = k.uz + (float)(k.bz - nz) * k.cs[2];
                    int rb[3], re[3], s1[3], s2[3], most = 0;
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        const int my = k.by - 1 + r;
                        rb[r] = re[r] = s1[r] = s2[r] = 0;
                        const float gyz = row_gap2(k, my, nz);
                        if (my < k.lo1 || my > k.hi1 || gyz > k.reach2) continue;
                        const int kc = k.row_key(my, nz);
                        s1[r] = a.cell_start[kc];
                        s2[r] = a.cell_start[kc + 1];
                        rb[r] = (k.has_l && !(gyz + gxl * gxl > k.reach2)) ? a.cell_start[kc - 1] : s1[r];
                        re[r] = (k.has_r && !(gyz + gxr * gxr > k.reach2)) ? a.cell_start[kc + 2] : s2[r];
                        if (rb[r] < re[r]) most = max(most, ((re[r] + 3) >> 2) - (rb[r] >> 2));
                    }
                    if (most == 0) continue;
                    if (most <= 8 * G) {
                        unsigned bits[3], oth[3];
                        int p0[3];
#pragma unroll
                        for (int r = 0; r < 3; ++r) {
                            const int gb = rb[r] >> 2, ge = (re[r] + 3) >> 2;
                            const int per = (ge - gb + G - 1) / G;
                            const int g0 = gb + sub * per, m = rb[r] < re[r] ? min(per, ge - g0) : 0;
                            p0[r] = 4 * g0;
                            bits[r] = oth[r] = 0u;
                            if (m > 0)
                                bits[r] = accept_bits<V>(a, k, t, mati, g0, m, rb[r], min(re[r], 4 * (g0 + m)),
                                                         k.uy + (float)(1 - r) * k.cs[1], qz, mind);
                        }
                        if (contact || two_pass) {
#pragma unroll
                            for (int r = 0; r < 3; ++r) {
                                oth[r] = other_bits(a, bits[r], p0[r], mati);
                                bits[r] &= ~oth[r];
                                if (two_pass && pass == 0) others += __popc(oth[r]);
                                if (two_pass && pass == 1) bits[r] = oth[r];
                            }
                        }
                        // three counts of at most 32 G <= 256 in one word
                        int tot;
                        const int ex = scan(__popc(bits[0]) | __popc(bits[1]) << 10 | __popc(bits[2]) << 20, tot);
                        int at = nn;
#pragma unroll
                        for (int r = 0; r < 3; ++r) {
                            write(bits[r], at + ((ex >> (10 * r)) & 1023), out, cap, p0[r], s1[r], s2[r],
                                  (unsigned)(3 * r + 9 * (nz - k.bz + 1)));
                            at += (tot >> (10 * r)) & 1023;
                        }
                        nn = at;
                        if (contact) {
                            const int cx = scan(__popc(oth[0]) | __popc(oth[1]) << 10 | __popc(oth[2]) << 20, tot);
                            at = nc;
#pragma unroll
                            for (int r = 0; r < 3; ++r) {
                                write(oth[r], at + ((cx >> (10 * r)) & 1023), cout, a.cstride, p0[r], s1[r], s2[r],
                                      (unsigned)(3 * r + 9 * (nz - k.bz + 1)));
                                at += (tot >> (10 * r)) & 1023;
                            }
                            nc = at;
                        }
                    } else {
                        // rows of more than 32 G candidates: sub-runs of 8 groups per lane, row by row
                        for (int r = 0; r < 3; ++r) {
                            const unsigned code = (unsigned)(3 * r + 9 * (nz - k.bz + 1));
                            const float qy = k.uy + (float)(1 - r) * k.cs[1];
                            // (dynamic r: the row's values by selection)
                            const int b = r == 0 ? rb[0] : (r == 1 ? rb[1] : rb[2]);
                            const int e = r == 0 ? re[0] : (r == 1 ? re[1] : re[2]);
                            const int f1 = r == 0 ? s1[0] : (r == 1 ? s1[1] : s1[2]);
                            const int f2 = r == 0 ? s2[0] : (r == 1 ? s2[1] : s2[2]);
                            const int ge = (e + 3) >> 2;
                            if (b >= e) continue;
                            for (int gw = b >> 2; gw < ge; gw += 8 * G) {
                                const int g0 = gw + 8 * sub, m = min(8, ge - g0);
                                unsigned bits = 0u, oth = 0u;
                                if (m > 0) bits = accept_bits<V>(a, k, t, mati, g0, m, b, e, qy, qz, mind);
                                if (contact || two_pass) {
                                    oth = other_bits(a, bits, 4 * g0, mati);
                                    bits &= ~oth;
                                    if (two_pass && pass == 0) others += __popc(oth);
                                    if (two_pass && pass == 1) bits = oth;
                                }
                                int tot;
                                int ex = scan(__popc(bits), tot);
                                write(bits, nn + ex, out, cap, 4 * g0, f1, f2, code);
                                nn += tot;
                                if (contact) {
                                    ex = scan(__popc(oth), tot);
                                    write(oth, nc + ex, cout, a.cstride, 4 * g0, f1, f2, code);
                                    nc += tot;
                                }
                            }
                        }
                    }
                }
                if (two_pass) others = __reduce_add_sync(grp, others);
            }
            if (sub == 0) list_overflow(a, i, nn, nc, contact);
            if (a.prm.boundary) search_ghosts<V, G>(a, k, t, i, mati, sub, grp, gn, gcn, mind);
            if (want_mind)
                for (int o = G / 2; o > 0; o >>= 1) mind = fmin(mind, __shfl_xor_sync(grp, mind, o, G));
            mind = sqrt(mind);
        }
        if (a.prm.disctype == 1) nn += 1;   // MCM/mcm_ll_neighbours.f90:288-299 (for every particle)
        if (sub == 0) search_counts<V>(a, t, i, nn, gn, nc, gcn, mind);
    }
    search_max(a, nn, gn);
}

// The same search with one warp per cell (search_kind 3): the lanes are the
// particles of one cell (32 at a time), so every lane walks the same rows of
// the same 27-cell neighbourhood and the loop control is warp-uniform.  Each
// row's contiguous candidate range is staged 32 records at a time in shared
// memory by one coalesced load per lane and then read by every lane as a
// broadcast, so the inner loop has no global load.  Candidates are visited in
// k_search's order.  The FP32 decision is its own: coordinates relative to the
// cells (cposf) and a band of 2^-12 of the cutoff and of the cell's square; the
// band is left to the same FP64 expression, so the lists are k_search's, entry
// for entry.
constexpr int kCellWarps = 8;
__global__ void __launch_bounds__(kCellWarps * 32, 3) k_search_cell(StepArgs a) {
    chain_wait();
    __shared__ float4 stage[kCellWarps][32];
    __shared__ int stage_mat[kCellWarps][32];
    if (a.status->code) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long ncells = a.grid->ncells;
    const int gl0 = a.grid->gridlim[0], gl1 = a.grid->gridlim[1], gl2 = a.grid->gridlim[2];
    // cell keys from scalars (an array passed by pointer would live in local memory)
    auto key_of = [gl0, gl1](int x, int y, int z) { return (x - 1) + gl0 * ((y - 1) + gl1 * (z - 1)); };
    const float hcut = (float)a.grid->hcut;
    const int np = a.npad;
    const int cap = a.nstride;
    const bool with_self = (a.prm.disctype == 1);
    const bool want_mind = (a.prm.tcrit_opt == 2 || a.prm.diag);
    const bool contact = a.prm.contact != 0;
    const bool multi = a.nmat > 1;
    const float cs[3] = {(float)(1.0 / a.grid->gridsize[0]), (float)(1.0 / a.grid->gridsize[1]),
                         (float)(1.0 / a.grid->gridsize[2])};
    const float csm = fmaxf(cs[0], fmaxf(cs[1], cs[2]));
    const float kb = 2.44140625e-4f * csm * csm;
    const float khi = 1.0f + 2.44140625e-4f, klo = 1.0f - 2.44140625e-4f;
    float4 *st = stage[w];
    int *stm = stage_mat[w];
    const long long nwarps = (long long)gridDim.x * kCellWarps;
    for (long long c = (long long)blockIdx.x * kCellWarps + w; c < ncells; c += nwarps) {
        const int c0 = a.cell_start[c], c1 = a.cell_start[c + 1];
        if (c0 == c1) continue;   // warp-uniform
        const int bx = (int)(c % gl0) + 1;
        const int by = (int)((c / gl0) % gl1) + 1;
        const int bz = (int)(c / ((long long)gl0 * gl1)) + 1;
        const int lo0 = bx > 1 ? bx - 1 : 1, hi0 = bx < gl0 ? bx + 1 : gl0;
        const int lo1 = by > 1 ? by - 1 : 1, hi1 = by < gl1 ? by + 1 : gl1;
        const int lo2 = bz > 1 ? bz - 1 : 1, hi2 = bz < gl2 ? bz + 1 : gl2;
        for (int base = c0; base < c1; base += 32) {
            const int t = base + lane;
            const bool live = t < c1;
            double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
            float4 ui = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            int mati = 0, i = 0;
            if (live) {
                xi = a.cpos[t];
                ui = a.cposf[t];
                mati = a.cmat[t];
                i = a.cell_list[t];
            }
            const float reach = ui.w + hcut;
            const float reach2 = reach * reach * 1.0009765625f + 9.765625e-4f * csm * csm;
            unsigned *out = a.nidx + (size_t)(live ? t : 0) * cap;
            unsigned *cout = contact ? a.cidx + (size_t)(live ? t : 0) * a.cstride : nullptr;
            int nn = 0, gn = 0, nc = 0, gcn = 0;
            double mind = 1.0e20;
            // x extent of the own cell's neighbours: distance to the side columns
            const float gxl = fmaxf(ui.x, 0.0f), gxr = fmaxf(cs[0] - ui.x, 0.0f);
            const int passes = (multi && a.prm.contacttype == 0) ? 2 : 1;
            for (int pass = 0; pass < passes; ++pass) {
                for (int nz = lo2; nz <= hi2; ++nz) {
                    const float qz = ui.z + (float)(bz - nz) * cs[2];
                    const float gz = fmaxf(nz < bz ? ui.z : (nz > bz ? cs[2] - ui.z : 0.0f), 0.0f);
                    for (int my = lo1; my <= hi1; ++my) {
                        const float qy = ui.y + (float)(by - my) * cs[1];
                        const float gy = fmaxf(my < by ? ui.y : (my > by ? cs[1] - ui.y : 0.0f), 0.0f);
                        const float gyz = gy * gy + gz * gz;
                        const bool rowok = live && !(gyz > reach2);
                        if (!__any_sync(0xffffffffu, rowok)) continue;
                        // per lane: which of the row's cells can hold a neighbour
                        const bool okl = rowok && !(gyz + gxl * gxl > reach2);
                        const bool okr = rowok && !(gyz + gxr * gxr > reach2);
                        const int k0 = key_of(lo0, my, nz);
                        const int rb = a.cell_start[k0];
                        const int re = a.cell_start[k0 + (hi0 - lo0) + 1];
                        const int s1 = a.cell_start[k0 + 1];
                        const int s2 = (hi0 - lo0 >= 2) ? a.cell_start[k0 + 2] : re;
                        const unsigned code_yz = (unsigned)(3 * (my - by + 1) + 9 * (nz - bz + 1));
                        for (int chunk = rb; chunk < re; chunk += 32) {
                            const int pc = chunk + lane;
                            if (pc < re) {
                                st[lane] = a.cposf[pc];
                                if (multi) stm[lane] = a.cmat[pc];
                            }
                            __syncwarp();
                            const int m = (re - chunk) < 32 ? (re - chunk) : 32;
                            if (rowok) {
                                for (int k = 0; k < m; ++k) {
                                    const int p = chunk + k;
                                    const int lx = lo0 + (p >= s1 ? 1 : 0) + (p >= s2 ? 1 : 0);
                                    if (lx < bx ? !okl : (lx > bx ? !okr : false)) continue;
                                    const float4 cd4 = st[k];
                                    const float qx = ui.x + (float)(bx - lx) * cs[0];
                                    const float dx = qx - cd4.x, dy = qy - cd4.y, dz = qz - cd4.z;
                                    const float d2f = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                                    const float hsf = ui.w + cd4.w;
                                    const float r2f = hsf * hsf;
                                    if (d2f >= fmaf(r2f, khi, kb)) continue;
                                    if (p == t) continue;
                                    double d2 = 0.0;
                                    if (d2f > fmaf(r2f, klo, -kb) || want_mind) {
                                        const double4 cd = a.cpos[p];
                                        d2 = exact_d2(xi, cd);
                                        const double hs = __dadd_rn(cd.w, xi.w);
                                        if (!(d2 < __dmul_rn(hs, hs))) continue;
                                    }
                                    const unsigned code = (code_yz + (unsigned)(lx - bx + 1)) << 26;
                                    if (contact) {
                                        if (stm[k] != mati) {
                                            if (nc < a.cstride) cout[nc] = (unsigned)p | code;
                                            ++nc;
                                            continue;
                                        }
                                    } else if (multi && (stm[k] == mati) != (pass == 0)) {
                                        continue;
                                    }
                                    if (want_mind) mind = fmin(mind, d2);
                                    if (nn < cap) out[nn] = (unsigned)p | code;
                                    ++nn;
                                }
                            }
                            __syncwarp();
                        }
                    }
                }
            }
            // ghosts: only neighbourhoods that reach a ghost layer (warp-uniform test)
            if (a.prm.boundary && live) {
                const DevPlanes &pl = a.prm.planes;
                const bool near = (lo0 == 1 && pl.code[0][0]) || (hi0 == gl0 && pl.code[1][0]) ||
                                  (lo1 == 1 && pl.code[0][1]) || (hi1 == gl1 && pl.code[1][1]) ||
                                  (lo2 == 1 && pl.code[0][2]) || (hi2 == gl2 && pl.code[1][2]);
                if (near) {
                    const int gpasses = (multi && a.prm.contacttype == 0) ? 2 : 1;
                    for (int pass = 0; pass < gpasses; ++pass) {
                        for (int nz = lo2; nz <= hi2; ++nz)
                            for (int my = lo1; my <= hi1; ++my)
                                for (int lx = lo0; lx <= hi0; ++lx) {
                                    const int2 gcl = a.gcell[key_of(lx, my, nz)];
                                    for (int r = 0; r < gcl.y; ++r) {
                                        const int q = gcl.x + gcl.y - 1 - r;   // chain order: newest first
                                        const double4 gq = make_double4(a.gx[q], a.gy[q], a.gz[q], a.gh[q]);
                                        const double d2 = exact_d2(xi, gq);
                                        const double hs = __dadd_rn(gq.w, xi.w);
                                        if (d2 < __dmul_rn(hs, hs)) {
                                            if (contact) {
                                                if (a.gmat[q] != mati) {
                                                    if (gcn < a.gcstride) a.gcont[(size_t)gcn * np + t] = q;
                                                    ++gcn;
                                                    continue;
                                                }
                                            } else if (multi && (a.gmat[q] == mati) != (pass == 0)) {
                                                continue;
                                            }
                                            mind = fmin(mind, d2);
                                            if (gn < a.gstride) a.gnbr[(size_t)gn * np + t] = q;
                                            ++gn;
                                        }
                                    }
                                }
                    }
                }
            }
            if (!live) continue;
            if (nn > cap) {
                atomicMax(&a.status->req_stride, nn);
                raise_status(a.status, MCM_ENBR_OVERFLOW, i);
            }
            if (gn > a.gstride) {
                atomicMax(&a.status->req_gstride, gn);
                raise_status(a.status, MCM_ENBR_OVERFLOW, i);
            }
            if (contact && nc > a.cstride) {
                atomicMax(&a.status->req_cstride, nc);
                raise_status(a.status, MCM_ENBR_OVERFLOW, i);
            }
            if (contact && gcn > a.gcstride) {
                atomicMax(&a.status->req_gcstride, gcn);
                raise_status(a.status, MCM_ENBR_OVERFLOW, i);
            }
            mind = sqrt(mind);
            if (with_self) nn += 1;   // MCM/mcm_ll_neighbours.f90:288-299 (for every particle)
            a.nnbr[t] = nn;
            a.gnnbr[t] = gn;
            if (contact) { a.ncont[t] = nc; a.gncont[t] = gcn; }
            if (want_mind) a.F.f[FMINDIST][i] = mind;
            atomicMax(&a.status->max_nbr, nn);
            atomicMax(&a.status->max_gnbr, gn);
        }
    }
    // particles outside the grid (the last positions) have no neighbours
    const int first_out = a.cell_start[ncells];
    for (int t = first_out + blockIdx.x * blockDim.x + threadIdx.x; t < a.n; t += gridDim.x * blockDim.x) {
        const int nn = with_self ? 1 : 0;
        a.nnbr[t] = nn;
        a.gnnbr[t] = 0;
        if (contact) { a.ncont[t] = 0; a.gncont[t] = 0; }
        if (want_mind) a.F.f[FMINDIST][a.cell_list[t]] = 1.0e20;
        atomicMax(&a.status->max_nbr, nn);
    }
}

// ------------------------------------------------------------- skin lists
// For the FP64-fast and mixed steps, whose sums do not follow the reference's
// neighbour order: the neighbour lists of a step are filtered from a skin
// list, a superset of each particle's neighbours kept from the last build.
// A pair (i, j) missing from the skin list was at least h_i + h_j + skin apart
// at the build; while every particle has moved less than skin/2 since then,
// it is still at least h_i + h_j apart, so it cannot be a neighbour.  The
// step rebuilds the skin lists when the largest displacement reaches skin/2
// (or on request), and filters them every step with k_search_cell's FP32
// decision and the FP64 tie test, among the candidates in the 27 cells around the
// particle's cell of the current grid (the only ones the reference examines),
// so the neighbour sets are the reference's; their order is the skin list's.

// Largest squared displacement since the last build (state order).
__global__ void __launch_bounds__(256) k_skin_disp(StepArgs a) {
    __shared__ unsigned long long sm[8];
    if (a.status->code) return;
    unsigned long long best = 0ull;
    const double *X = a.F.f[FX], *Y = a.F.f[FY], *Z = a.F.f[FZ];
    const size_t np = a.npad;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const double dx = X[i] - a.xref[i], dy = Y[i] - a.xref[np + i], dz = Z[i] - a.xref[2 * np + i];
        const double d2 = dx * dx + dy * dy + dz * dz;   // >= 0: the bit pattern orders like the value
        const unsigned long long b = (unsigned long long)__double_as_longlong(d2);
        best = b > best ? b : best;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, best, o);
        best = v > best ? v : best;
    }
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) best = sm[w] > best ? sm[w] : best;
        atomicMax(a.skin_d2, best);
    }
}

// One thread: build when asked to, or when 2 * max displacement >= skin.
__global__ void k_skin_decide(StepArgs a) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (a.status->code) return;
    const double dmax = sqrt(__longlong_as_double((long long)*a.skin_d2));
    const double skin = a.prm.skin * a.hmax[0];
    const int need = (a.skin_flags[0] != 0 || !(2.0 * dmax < skin)) ? 1 : 0;
    a.skin_flags[1] = need;
    a.skin_flags[0] = 0;
    if (need) a.skin_flags[2] += 1;
    *a.skin_d2 = 0ull;
}

// The skin lists: one thread per cell-order position, candidates in the
// cells within reach (up to two cells away), accepted when their FP32
// distance lies below h_i + h_j + skin with a margin (a superset needs no
// exact test).  Positions outside the grid keep an empty list.
__global__ void __launch_bounds__(256) k_skin_build(StepArgs a) {
    if (a.status->code || !a.skin_flags[1]) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.n) return;
    const int i = a.cell_list[t];
    const size_t np = a.npad;
    const double4 xi = a.cpos[t];
    a.xref[i] = xi.x;
    a.xref[np + i] = xi.y;
    a.xref[2 * np + i] = xi.z;
    const int key = a.ckey[t];
    int nn = 0;
    if (key >= 0) {
        const int gl0 = a.grid->gridlim[0], gl1 = a.grid->gridlim[1], gl2 = a.grid->gridlim[2];
        const int bx = key % gl0 + 1, by = (key / gl0) % gl1 + 1, bz = key / (gl0 * gl1) + 1;
        const float cs[3] = {(float)(1.0 / a.grid->gridsize[0]), (float)(1.0 / a.grid->gridsize[1]),
                             (float)(1.0 / a.grid->gridsize[2])};
        const float skin = (float)(a.prm.skin * a.hmax[0]);
        const float4 ui = a.cposf[t];
        const float reach = ui.w + (float)a.grid->hcut + skin;
        const float reach2 = reach * reach * 1.001f + 1.0e-3f * cs[0] * cs[0];
        int *out = a.sup + (size_t)i * a.sstride;
        for (int nz = max(bz - 2, 1); nz <= min(bz + 2, gl2); ++nz) {
            const float qz = ui.z + (float)(bz - nz) * cs[2];
            const float gz = nz < bz ? ui.z + (float)(bz - nz - 1) * cs[2] : (nz > bz ? (float)(nz - bz) * cs[2] - ui.z : 0.0f);
            for (int my = max(by - 2, 1); my <= min(by + 2, gl1); ++my) {
                const float qy = ui.y + (float)(by - my) * cs[1];
                const float gy = my < by ? ui.y + (float)(by - my - 1) * cs[1] : (my > by ? (float)(my - by) * cs[1] - ui.y : 0.0f);
                const float gyz = fmaxf(gy, 0.0f) * fmaxf(gy, 0.0f) + fmaxf(gz, 0.0f) * fmaxf(gz, 0.0f);
                if (gyz > reach2) continue;
                for (int lx = max(bx - 2, 1); lx <= min(bx + 2, gl0); ++lx) {
                    const float gx = lx < bx ? ui.x + (float)(bx - lx - 1) * cs[0] : (lx > bx ? (float)(lx - bx) * cs[0] - ui.x : 0.0f);
                    if (gyz + fmaxf(gx, 0.0f) * fmaxf(gx, 0.0f) > reach2) continue;
                    const int k = (lx - 1) + gl0 * ((my - 1) + gl1 * (nz - 1));
                    const int cb = a.cell_start[k], ce = a.cell_start[k + 1];
                    const float qx = ui.x + (float)(bx - lx) * cs[0];
                    for (int p = cb; p < ce; ++p) {
                        if (p == t) continue;
                        const float4 c = a.cposf[p];
                        const float dx = qx - c.x, dy = qy - c.y, dz = qz - c.z;
                        const float d2f = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                        const float r = ui.w + c.w + skin;
                        if (d2f >= r * r * 1.001f + 1.0e-3f * cs[0] * cs[0]) continue;
                        if (nn < a.sstride) out[nn] = a.cell_list[p];
                        ++nn;
                    }
                }
            }
        }
    }
    a.supn[i] = nn;
    if (nn > a.sstride) {
        atomicMax(&a.status->req_sstride, nn);
        raise_status(a.status, MCM_ENBR_OVERFLOW, i);
    }
}

// The step's neighbour lists from the skin lists: k_search_cell's decisions on
// the candidates that lie in the 27 cells around the particle's cell, in
// skin-list order; ghosts, contacts, minimum distances and counts as k_search.
__global__ void __launch_bounds__(256, 4) k_skin_filter(StepArgs a) {
    if (a.status->code) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.n) return;
    const int np = a.npad;
    const int cap = a.nstride;
    const int key = a.ckey[t];
    const int i = a.cell_list[t];
    const bool with_self = (a.prm.disctype == 1);
    const bool want_mind = (a.prm.tcrit_opt == 2 || a.prm.diag);
    const bool contact = a.prm.contact != 0;
    int nn = 0, gn = 0, nc = 0, gcn = 0;
    double mind = 1.0e20;
    if (key >= 0) {
        const int gl0 = a.grid->gridlim[0], gl1 = a.grid->gridlim[1], gl2 = a.grid->gridlim[2];
        const int bx = key % gl0 + 1, by = (key / gl0) % gl1 + 1, bz = key / (gl0 * gl1) + 1;
        const double4 xi = a.cpos[t];
        const float4 ui = a.cposf[t];
        const float cs[3] = {(float)(1.0 / a.grid->gridsize[0]), (float)(1.0 / a.grid->gridsize[1]),
                             (float)(1.0 / a.grid->gridsize[2])};
        const float csm = fmaxf(cs[0], fmaxf(cs[1], cs[2]));
        const float kb = 2.44140625e-4f * csm * csm;
        const float khi = 1.0f + 2.44140625e-4f, klo = 1.0f - 2.44140625e-4f;
        const int mati = a.cmat[t];
        unsigned *out = a.nidx + (size_t)t * cap;
        unsigned *cout = contact ? a.cidx + (size_t)t * a.cstride : nullptr;
        const int *cand = a.sup + (size_t)i * a.sstride;
        const int ns = a.supn[i];
        // with kernel contact the other materials follow the own material's neighbours
        const int passes = (a.nmat > 1 && a.prm.contacttype == 0) ? 2 : 1;
        for (int pass = 0; pass < passes; ++pass) {
            for (int k = 0; k < ns; ++k) {
                const int p = a.pos_of[cand[k]];
                const int kp = a.ckey[p];
                if (kp < 0) continue;
                const int ex = kp % gl0 + 1 - bx, ey = (kp / gl0) % gl1 + 1 - by, ez = kp / (gl0 * gl1) + 1 - bz;
                if (ex < -1 || ex > 1 || ey < -1 || ey > 1 || ez < -1 || ez > 1) continue;
                const float4 c = a.cposf[p];
                const float dx = (ui.x - (float)ex * cs[0]) - c.x;
                const float dy = (ui.y - (float)ey * cs[1]) - c.y;
                const float dz = (ui.z - (float)ez * cs[2]) - c.z;
                const float d2f = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                const float hsf = ui.w + c.w;
                const float r2f = hsf * hsf;
                if (d2f >= fmaf(r2f, khi, kb)) continue;
                double d2 = 0.0;
                if (d2f > fmaf(r2f, klo, -kb) || want_mind) {
                    const double4 cd = a.cpos[p];
                    d2 = exact_d2(xi, cd);
                    const double hs = __dadd_rn(cd.w, xi.w);
                    if (!(d2 < __dmul_rn(hs, hs))) continue;
                }
                const unsigned code = (unsigned)((ex + 1) + 3 * (ey + 1) + 9 * (ez + 1)) << 26;
                if (contact) {
                    if (a.cmat[p] != mati) {
                        if (nc < a.cstride) cout[nc] = (unsigned)p | code;
                        ++nc;
                        continue;
                    }
                } else if (a.nmat > 1 && (a.cmat[p] == mati) != (pass == 0)) {
                    continue;
                }
                if (want_mind) mind = fmin(mind, d2);
                if (nn < cap) out[nn] = (unsigned)p | code;
                ++nn;
            }
        }
        if (nn > cap) {
            atomicMax(&a.status->req_stride, nn);
            raise_status(a.status, MCM_ENBR_OVERFLOW, i);
        }
        if (contact && nc > a.cstride) {
            atomicMax(&a.status->req_cstride, nc);
            raise_status(a.status, MCM_ENBR_OVERFLOW, i);
        }
        // ghosts: as k_search, from the current grid's ghost cells
        if (a.prm.boundary) {
            const int lo0 = bx > 1 ? bx - 1 : 1, hi0 = bx < gl0 ? bx + 1 : gl0;
            const int lo1 = by > 1 ? by - 1 : 1, hi1 = by < gl1 ? by + 1 : gl1;
            const int lo2 = bz > 1 ? bz - 1 : 1, hi2 = bz < gl2 ? bz + 1 : gl2;
            const DevPlanes &pl = a.prm.planes;
            const bool near = (lo0 == 1 && pl.code[0][0]) || (hi0 == gl0 && pl.code[1][0]) ||
                              (lo1 == 1 && pl.code[0][1]) || (hi1 == gl1 && pl.code[1][1]) ||
                              (lo2 == 1 && pl.code[0][2]) || (hi2 == gl2 && pl.code[1][2]);
            if (near) {
                const int gpasses = (a.nmat > 1 && a.prm.contacttype == 0) ? 2 : 1;
                for (int pass = 0; pass < gpasses; ++pass) {
                    for (int nz = lo2; nz <= hi2; ++nz)
                        for (int my = lo1; my <= hi1; ++my)
                            for (int lx = lo0; lx <= hi0; ++lx) {
                                const int2 gcl = a.gcell[(lx - 1) + gl0 * ((my - 1) + gl1 * (nz - 1))];
                                for (int r = 0; r < gcl.y; ++r) {
                                    const int q = gcl.x + gcl.y - 1 - r;
                                    const double4 gq = make_double4(a.gx[q], a.gy[q], a.gz[q], a.gh[q]);
                                    const double d2 = exact_d2(xi, gq);
                                    const double hs = __dadd_rn(gq.w, xi.w);
                                    if (d2 < __dmul_rn(hs, hs)) {
                                        if (contact) {
                                            if (a.gmat[q] != mati) {
                                                if (gcn < a.gcstride) a.gcont[(size_t)gcn * np + t] = q;
                                                ++gcn;
                                                continue;
                                            }
                                        } else if (a.nmat > 1 && (a.gmat[q] == mati) != (pass == 0)) {
                                            continue;
                                        }
                                        mind = fmin(mind, d2);
                                        if (gn < a.gstride) a.gnbr[(size_t)gn * np + t] = q;
                                        ++gn;
                                    }
                                }
                            }
                }
                if (gn > a.gstride) {
                    atomicMax(&a.status->req_gstride, gn);
                    raise_status(a.status, MCM_ENBR_OVERFLOW, i);
                }
                if (gcn > a.gcstride) {
                    atomicMax(&a.status->req_gcstride, gcn);
                    raise_status(a.status, MCM_ENBR_OVERFLOW, i);
                }
            }
        }
        mind = sqrt(mind);
    }
    if (with_self) nn += 1;   // MCM/mcm_ll_neighbours.f90:288-299 (for every particle)
    a.nnbr[t] = nn;
    a.gnnbr[t] = gn;
    if (contact) { a.ncont[t] = nc; a.gncont[t] = gcn; }
    if (want_mind) a.F.f[FMINDIST][i] = mind;
    atomicMax(&a.status->max_nbr, nn);
    atomicMax(&a.status->max_gnbr, gn);
}

__global__ void k_skin_force(StepArgs a) {
    if (threadIdx.x == 0 && blockIdx.x == 0) a.skin_flags[0] = 1;
}

void launch_skin_force(const StepArgs &a, cudaStream_t s) { k_skin_force<<<1, 32, 0, s>>>(a); }

void launch_skin_search(const StepArgs &a, cudaStream_t s) {
    const int nb = (a.n + 255) / 256;
    k_skin_disp<<<nb < 148 * 8 ? nb : 148 * 8, 256, 0, s>>>(a);
    k_skin_decide<<<1, 32, 0, s>>>(a);
    k_skin_build<<<nb, 256, 0, s>>>(a);
    k_skin_filter<<<nb, 256, 0, s>>>(a);
}

// Lanes per particle of the search: one thread per particle is the cheapest
// walk where it fills the chip, but its chain of nine rows takes 62 us however
// few particles there are.  Measured (us a search, 1 / 4 / 8 lanes, taylor
// bars, mixed): 16 848 particles 62 / 48 / 34, 38 880: 70 / 53 / 55, 685 824:
// 340 / 546 / 766.  Around the line between four lanes and one (1 / 4): 62 484:
// 72 / 62, 68 120: 72 / 65, 80 592: 76 / 72, 91 008: 77 / 80, 131 544: 86 / 108.
// The two meet near 85 000: the line is on the safe side of that, and bodies
// between the two pay up to 8 us.  Bodies of a batch fill the chip together, so
// the particles of all that run at the same time count.
constexpr int kSearch8Below = 24000, kSearch4Below = 64000;
template <int V, int G>
static void launch_lanes(const StepArgs &a, int threads, cudaStream_t s) {
    launch_chained(k_search_lanes<V, G>, (unsigned)(((long long)a.n * G + threads - 1) / threads), threads, 0, s, a);
}
template <int V>
static void launch_search_v(const StepArgs &a, cudaStream_t s) {
    const int threads = search_threads_of(a);
    const long long n = (long long)a.n * a.share;
    if (a.search_kind == 2 || n < kSearch8Below) launch_lanes<V, 8>(a, threads, s);
    else if (n < kSearch4Below) launch_lanes<V, 4>(a, threads, s);
    else launch_chained(k_search<V>, (a.n + threads - 1) / threads, threads, (threads / 32) * 33 * kSrchKeep * sizeof(unsigned), s, a);
}

void launch_search(const StepArgs &a, cudaStream_t s) {
    if (a.search_kind == 3) {
        // grid-stride over the cells (ncells is on the device): up to 16 blocks per SM
        long long b = (a.cell_cap + kCellWarps - 1) / kCellWarps;
        if (b > 148LL * 16) b = 148LL * 16;
        launch_chained(k_search_cell, (unsigned)(b < 1 ? 1 : b), kCellWarps * 32, 0, s, a);
        return;
    }
    const bool mind = a.prm.tcrit_opt == 2 || a.prm.diag;
    switch ((a.prm.contact ? kSrchContact : 0) | ((a.nmat > 1 && a.prm.contacttype == 0) ? kSrchTwoPass : 0) |
            (mind ? kSrchMind : 0)) {
        case 0: launch_search_v<0>(a, s); break;
        case kSrchContact: launch_search_v<kSrchContact>(a, s); break;
        case kSrchTwoPass: launch_search_v<kSrchTwoPass>(a, s); break;
        case kSrchMind: launch_search_v<kSrchMind>(a, s); break;
        case kSrchContact | kSrchMind: launch_search_v<kSrchContact | kSrchMind>(a, s); break;
        default: launch_search_v<kSrchTwoPass | kSrchMind>(a, s); break;
    }
}

}  // namespace mcm
