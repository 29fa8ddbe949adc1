// force_tile.cuh — fused velocity + position phase of the Particle Life step:
// the force kernels and their launchers, instantiated per dimension by
// k_force.cu (2D) and k_force3.cu (3D), which compile in parallel.
//
// One thread per particle of the cell-sorted order B.  It replaces
//   Physics.updateVelocity  (backend/Physics.java:397-441),
//   the default Accelerator (app/Main.java:275-280),
//   Physics.updatePosition  (backend/Physics.java:443-450) with
//   Range.wrap / Range.clamp (backend/Range.java:40-96),
// and, in its epilogue, the counting pass of the next makeContainers
// (Physics.java:328-332) on the new position.
//
// Tiling.  A block takes 128 (3D variant 1: 64) consecutive targets of the
// sorted order, one thread each; their cells come from the sort.  The cells are
// nondecreasing, so the targets fall into a few "segments" (targets of one
// grid row: one y in 2D, one (y, z) in 3D).  A target in column cx needs the
// window of columns cx-1..cx+1 over its R stencil rows (3 in 2D, 9 in 3D);
// the block stages the sorted union of its targets' windows into shared
// memory column by column, each column's R cells in turn, so that every
// target's neighbourhood is one contiguous run.  When the whole block's
// windows fit, one staging serves every target; otherwise the block's
// cells are staged in parts, as many at a time as fit (of a cell that does not
// fit by itself, a slice), and each part serves every target whose window
// meets it.  The candidates come in the same order and give the same bits
// throughout.  The 2D
// candidate loop is branch-free FP32; a 3D window is tested by distance
// first, and terms are formed for what that keeps.  A target that meets a
// candidate needing the FP64 decision is deferred: its warp recomputes it from global
// memory at the end (fixup_target).
//
// Pair test.  The reference keeps a pair when d2 != 0 && d2 <= rmax*rmax in
// FP64, with d = wrapConnection(q - p) (Physics.java:428-432).  Here d2 is
// first formed in FP32 from differences that are exact or rounded once: a
// periodic image is taken by cell, as (q - 1) - p or q - (p - 1), where the
// shifted operand lies in [0.5, 1] and the shift is exact.  The FP32 d2 is
// within 5 ulp of the FP64 one, so a pair with d2 <= lo is inside, a pair
// with d2 >= hi is outside, and only pairs in the band (lo, hi) or below
// `tiny` are re-decided with the reference's exact FP64 operation sequence
// (fp64_keeps).  The interacting-pair set is therefore bit-identical to the
// FP64 reference run on the same FP32 positions.  Only the decision is FP64:
// the term of a kept band pair is FP32 like every other term (the force
// vanishes at rmax, so it is tiny); only a pair whose FP32 d2 underflowed
// (d2 < tiny, distinct particles closer than about 1e-15) takes the FP64 term.
//
// Stencil.  The reference scans the 9 (27) cells around floor(x/cs) without
// clamping (Physics.java:404-409).  For a particle in the last partial cell
// [nx*cs, 1) that base is nx, not the binning cell nx-1.  This kernel uses
// the binning cell; the two stencils differ only by column nx-2 (scanned
// here, not there) and column 1 (scanned there, never within rmax).  A pair
// of column nx-2 within rmax lies within 1e-15 relative of rmax^2, so it
// reaches fp64_keeps, which rejects it like the reference.  Grids with fewer
// than 3 cells per axis, where the reference visits a cell more than once,
// take the literal path (general_scan).
#pragma once

#include "force_common.cuh"

namespace plg {

namespace {

__device__ __forceinline__ int wrap_container(int c, int n) {
    // wrapContainerX / wrapContainerY, Physics.java:377-395.
    return c < 0 ? c + n : (c >= n ? c - n : c);
}

// Literal stencil of Physics.java:404-421 for grids with nx < 3: unclamped
// base cell, every offset visited (a cell may repeat), each candidate decided
// and evaluated in FP64.
template <int D, bool DBG>
__device__ void general_scan(const ForceArgs<D>& A, const float* Mrow, int s, float px, float py, float pz,
                             Acc& acc) {
    const ForceParams& P = A.p;
    const int nx = P.g.nx;
    const int cx0 = axis_cell_unclamped(px, P.g), cy0 = axis_cell_unclamped(py, P.g);
    const int cz0 = D == 3 ? axis_cell_unclamped(pz, P.g) : 0;
    for (int oz = (D == 3 ? -1 : 0); oz <= (D == 3 ? 1 : 0); ++oz) {
        for (int oy = -1; oy <= 1; ++oy) {
            for (int ox = -1; ox <= 1; ++ox) {
                int cx = wrap_container(cx0 + ox, nx), cy = wrap_container(cy0 + oy, nx);
                int cz = D == 3 ? wrap_container(cz0 + oz, nx) : 0;
                if (P.wrap) {
                    cx = wrap_container(cx, nx);
                    cy = wrap_container(cy, nx);
                    if (D == 3) cz = wrap_container(cz, nx);
                } else if (cx < 0 || cx >= nx || cy < 0 || cy >= nx || (D == 3 && (cz < 0 || cz >= nx))) {
                    continue;
                }
                const int ci = cx + (cy + cz * nx) * nx;
                const int j0 = __ldg(A.cstart + ci), j1 = __ldg(A.cstart + ci + 1);
                for (int j = j0; j < j1; ++j) {
                    if (j == s) continue;
                    if (DBG) acc.cand++;
                    const float4 q = __ldg(A.bpt + j);
                    const float4 c = rare_pair<D>(P, px, py, pz, q, Mrow[Layout<D>::type(q)], 0);
                    if (c.w != 0.f) add_pair<D, DBG>(acc, c, DBG ? id_of<D>(A, j) : 0ull);
                }
            }
        }
    }
}

// ---- literal-path kernel (nx < 3) ----

template <int D, bool DBG, bool SMEM_M>
__global__ void __launch_bounds__(kThreads) k_force_general(const __grid_constant__ ForceArgs<D> A) {
    pdl_wait();  // the sort before it
    const ForceParams& P = A.p;
    extern __shared__ float smat[];
    const float* M = P.matrix;
    const int nt = P.ntypes, ms = SMEM_M ? smem_matrix_stride<D>(nt) : nt;
    if (SMEM_M) {
        for (int k = threadIdx.x; k < nt * nt; k += kThreads)
            smat[D == 3 ? (k / nt) * ms + k % nt : k] = P.matrix[k];
        __syncthreads();
        M = smat;
    }
    const int s = blockIdx.x * kThreads + threadIdx.x;
    const bool valid = s < P.n;
    uint32_t newcell = 0;
    if (valid) {
        const float4 me = A.bpt[s];
        Acc acc = {0.f, 0.f, 0.f, 0, 0ull, 0ull, 0ull};
        general_scan<D, DBG>(A, M + Layout<D>::type(me) * ms, s, me.x, me.y, D == 3 ? me.z : 0.f, acc);
        newcell = integrate<D, DBG>(A, A.p, s, me, A.bvel[s], acc);
    }
    const unsigned mask = __ballot_sync(kFull, valid);
    if (valid) {
        bin_add(A.counts, newcell, mask);
        A.cell[s] = newcell;
    }
}

// ---- tiled kernel (nx >= 3) ----

// Tile variants (the autotuner's choice, PLG_TILE_*):
//   kTargets    targets per block, one thread each
//   kMinBlocks  resident blocks per SM asked for (caps the registers: more
//               blocks with spilled registers measured slower)
//   kCap        staged candidates per staging
//   kCells      stencil cells per staging (R x columns)
// 2D: tiles of 128 targets throughout (256 at 4 blocks per SM lose 2% at 6
// particles per cell and 30% at 3 and below, where their windows need more
// than the 256 stencil cells).  Variant 0: 8 blocks at 64 registers.  Variant
// 1: 2048 candidates at 6 blocks for crowded cells (400k particles, 123 per
// cell: 336 us against 367, 250 per cell: 765 against 794, 61 per cell: 169
// against 167).  Variant 2: 7
// blocks with more registers and candidates, for worlds of about one wave.
// 3D: 71 staged columns of 9 cells in variants 0 and 2, so that the sparse
// tails of a blob world stage in one or two rounds.  Variant 0: 4 blocks of
// 128 targets with 2176 candidates, for dense cells and for worlds of about
// one wave.  Variant 1: the smaller tile for small sparse worlds, 9 blocks of
// 64 targets with the candidates their shared memory holds (asking for 10,
// which did not fit beside 832 candidates, 9 ran with too few registers: 250k
// uniform 95 us, now 90; 10 blocks of 808 candidates 96).  Variant 2:
// 5 blocks of 128 targets with 1776 candidates, as much shared memory as five
// blocks have, for large worlds (4M in blobs 1045 us against variant 0's 1135;
// 1M at 2.4 per cell 127 us against 141.  With 448 cells 4% longer in blobs and
// 21% at 2.4 per cell, with 832 cells and 1600 candidates 5% in blobs, with six
// blocks of 1216 candidates 22% at 2.4 per cell).
template <int D, int V>
struct TileCfg;
template <>
struct TileCfg<2, 0> {
    static constexpr int kTargets = 128, kMinBlocks = 8, kCap = 1152, kCells = 256;
};
template <>
struct TileCfg<2, 1> {
    static constexpr int kTargets = 128, kMinBlocks = 6, kCap = 2048, kCells = 128;
};
template <>
struct TileCfg<2, 2> {
    static constexpr int kTargets = 128, kMinBlocks = 7, kCap = 1280, kCells = 256;
};
template <>
struct TileCfg<3, 0> {
    static constexpr int kTargets = 128, kMinBlocks = 4, kCap = 2176, kCells = 640;
};
template <>
struct TileCfg<3, 1> {
    static constexpr int kTargets = 64, kMinBlocks = 9, kCap = 944, kCells = 320;
};
template <>
struct TileCfg<3, 2> {
    static constexpr int kTargets = 128, kMinBlocks = 5, kCap = 1776, kCells = 640;
};

// Words of 32 candidates a 3D target tests before it forms the kept terms.
constexpr int kCullWords = 8;

// Lives in dynamic shared memory (22 KB in 2D variant 0; 51 KB in 3D
// variant 0, 44 KB in variant 2).
// Listed columns: the sorted union of the windows cx-1..cx+1 of the staged
// targets, as "virtual" columns -1..nx (-1 and nx being the periodic images
// of columns nx-1 and 0), each with the grid row of its segment.
template <int D, int V>
struct TileSmem {
    static constexpr int kCols = TileCfg<D, V>::kCells / TileRows<D>::R;
    // Staged candidates, column-major by stencil cell, from index kLead on.
    // The 3D distance test also reads the kLead entries before them and up to
    // a group after them, and keeps none of those.
    static constexpr int kLead = D == 3 ? 8 : 0;
    float4 slots[kLead + TileCfg<D, V>::kCap + (D == 3 ? kCullGroup : 0)];
    int coff[TileCfg<D, V>::kCells + 1];   // staged start of stencil cell e = column * R + row
    int cglob[TileCfg<D, V>::kCells];      // sorted-order start of stencil cell e
    int colv[kCols];                       // virtual column of staged column ci
    int colrow[kCols];                     // grid row of staged column ci: y, or y | z << 16
    int wsum[TileCfg<D, V>::kTargets / 32];
    int wcol[TileCfg<D, V>::kTargets / 32];
    // 3D: the words of 32 candidates that keep some, thread t's k-th at
    // [k * kTargets + t] (bits, staged index of bit 31)
    uint2 kept[D == 3 ? (kCullWords + 1) * TileCfg<D, V>::kTargets : 1];
    float mat[kSmemMatrixMax * smem_matrix_stride<D>(kSmemMatrixMax)];
    uint8_t image[TileCfg<D, V>::kCells];  // image shifts of stencil cell e (kUp*, kDown*)
};

// The blocks per SM that a variant asks for fit into an SM's shared memory:
// 228 KB, in units of 128 bytes, and 1 KB more per block.
template <int D, int V>
constexpr bool blocks_fit() {
    return TileCfg<D, V>::kMinBlocks * ((sizeof(TileSmem<D, V>) + 127) / 128 * 128 + 1024) <= 228 * 1024;
}
static_assert(blocks_fit<2, 0>() && blocks_fit<2, 1>() && blocks_fit<2, 2>(), "2D tile");
static_assert(blocks_fit<3, 0>() && blocks_fit<3, 1>() && blocks_fit<3, 2>(), "3D tile");

// Stages ncell cells of the listed columns (sm.colv, sm.colrow), from cell
// `off` of the first one on, column-major: for each column the cells of its R
// stencil rows in turn, so that the neighbourhood of a target whose window
// starts at column k is the single contiguous range of columns k .. k+2;
// without the first `skip` members of the first cell.  Images below the box are
// shifted down by 1 here (exact: their coordinates are >= 0.5); images above
// it are flagged for a target shift instead.  Thread t places cells
// t*per .. t*per+per-1: it reads their extents, and the block scans the
// per-thread sums.  Then groups of lanes copy a cell each with asynchronous
// copies, all in flight at once: one memory latency for the whole block.
// (One thread copying its own cells, a few members at a time, held the block
// behind the longest chain of dependent round trips, about 10 in 3D.  The
// staging and the target rows without integer divisions, together: force
// kernel of 1M particles in 2D 95.9 -> 88.3 us, of 4M in 3D blobs 1383 ->
// 1187 us.)
// Returns the number of cells staged to their end (the same in every thread):
// as many of the first ones as fit; 0 when not even one does, with its first
// kCap members (after the skipped ones) staged.  ncell <= kCells is the
// caller's.
template <int D, int V>
__device__ __forceinline__ int stage_cells(const ForceArgs<D>& A, const ForceParams& P,
                                           const uint32_t* __restrict__ cs, TileSmem<D, V>& sm, int off, int ncell,
                                           int skip) {
    constexpr int R = TileRows<D>::R;
    constexpr int kT = TileCfg<D, V>::kTargets;
    constexpr int kPer = (TileCfg<D, V>::kCells + kT - 1) / kT;
    const int nx = P.g.nx;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = (ncell + kT - 1) / kT;
    int g0[kPer], len[kPer];
    int sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int e = tid * per + i;
        g0[i] = 0;
        len[i] = 0;
        if (i < per && e < ncell) {
            const int ci = (e + off) / R, r = e + off - ci * R;
            const int v = sm.colv[ci], row = sm.colrow[ci];
            int image = v < 0 ? kDownX : (v >= nx ? kUpX : 0);
            const int col = v < 0 ? v + nx : (v >= nx ? v - nx : v);
            int ry = (D == 3 ? row & 0xffff : row) + r % 3 - 1, rz = D == 3 ? (row >> 16) + r / 3 - 1 : 0;
            if (ry < 0) ry += nx, image |= kDownY;
            if (ry >= nx) ry -= nx, image |= kUpY;
            if (D == 3) {
                if (rz < 0) rz += nx, image |= kDownZ;
                if (rz >= nx) rz -= nx, image |= kUpZ;
            }
            const int c = (rz * nx + ry) * nx + col;
            g0[i] = (int)__ldg(cs + c);
            len[i] = (int)__ldg(cs + c + 1) - g0[i];
            if (e == 0) {
                g0[i] += skip;
                len[i] -= skip;
            }
            sm.image[e] = P.wrap ? image : 0;
        }
        sum += len[i];
    }
    int inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(kFull, inc, d);
        if (lane >= d) inc += t;
    }
    if (lane == 31) sm.wsum[warp] = inc;
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kT / 32; ++w) {
        const int x = sm.wsum[w];
        before += w < warp ? x : 0;
        total += x;
    }
    bool slice = false;
    if (total > TileCfg<D, V>::kCap) {  // block-uniform
        int fit = 0, end = before + inc - sum;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int e = tid * per + i;
            end += len[i];
            if (i < per && e < ncell && end <= TileCfg<D, V>::kCap) ++fit;
        }
        fit = __reduce_add_sync(kFull, fit);
        if (lane == 0) sm.wcol[warp] = fit;
        __syncthreads();
        ncell = 0;
#pragma unroll
        for (int w = 0; w < kT / 32; ++w) ncell += sm.wcol[w];
        if (ncell == 0) {
            slice = true;
            ncell = 1;
            if (tid == 0) len[0] = TileCfg<D, V>::kCap;
        }
    }
    int run = before + inc - sum;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int e = tid * per + i;
        if (i < per && e < ncell) {
            sm.cglob[e] = g0[i];
            sm.coff[e] = run;
            if (e == ncell - 1) sm.coff[ncell] = run + len[i];
        }
        run += len[i];
    }
    __syncthreads();
    // Lanes per cell: by the cells' mean size (block-uniform).
    const int lg = total >= kDenseCell * ncell ? 5 : (total >= kSparseCell * ncell ? 3 : 2);
    for (int e = tid >> lg; e < ncell; e += kT >> lg) {
        const int d = sm.coff[e], m = sm.coff[e + 1] - d, image = sm.image[e];
        const float4* __restrict__ src = A.bpt + sm.cglob[e];
        float4* dst = sm.slots + TileSmem<D, V>::kLead + d;
        int k = tid & ((1 << lg) - 1);
        if (image) {
            for (; k < m; k += 1 << lg) dst[k] = shift_candidate<D>(__ldg(src + k), image);
        } else {
            for (; k < m; k += 1 << lg) copy16_async(dst + k, src + k);
        }
    }
    copy_wait();
    __syncthreads();
    return slice ? 0 : ncell;
}

// Main force kernel (nx >= 3): one thread per target; a block takes
// kTargets consecutive targets and stages their windows
// so that each target reads one contiguous run (or one per part).  Neighbouring threads mostly share a cell, hence a
// window, so their candidate loads are broadcasts.  FP32 only: a target
// whose neighbourhood holds a candidate that needs the FP64 decision is
// deferred to its warp's closing pass (fixup_target), which recomputes it
// completely.
// BATCH: the sorted order holds many worlds one after another (their cells
// are disjoint ranges of one global cell index).  Tiles are laid out per
// world: block b works on tile b - tile_off[k] of the world k that owns it,
// so a block never mixes worlds and every world is cut into exactly the
// tiles a single-world launch uses: each world computes bit for bit what
// plg_step computes for it, whatever else is in the batch.
//
// SNAP (single world, not instrumented): each warp also writes its slots'
// new state to the snapshot arrays A.snap once its deferred targets are done.
template <int D, bool DBG, bool SMEM_M, bool BATCH, int V, bool SNAP = false>
__global__ void __launch_bounds__(TileCfg<D, V>::kTargets, TileCfg<D, V>::kMinBlocks)
    k_force_tile(const __grid_constant__ ForceArgs<D> A) {
    static_assert(!SNAP || (!DBG && !BATCH), "the snapshot form is the plain single-world kernel");
    constexpr int kT = TileCfg<D, V>::kTargets;
    constexpr int R = TileRows<D>::R;
    extern __shared__ __align__(16) unsigned char smraw[];
    TileSmem<D, V>& sm = *reinterpret_cast<TileSmem<D, V>*>(smraw);
    const int tid = threadIdx.x;
    pdl_wait();  // the sort before it: B, slot_cell, cstart, the drained counts
    pdl_release();  // the next step's scan may be scheduled once every block runs
    int wk = 0, s0 = blockIdx.x * kT, nw = A.p.n;
    if (BATCH) {
        const int q = world_of(A.tile_off, A.nworlds, blockIdx.x);
        wk = __ldg(A.tile_off + A.nworlds + 1 + q);
        const int t = blockIdx.x - __ldg(A.tile_off + q);
        s0 = __ldg(A.wp_off + wk) + t * kT;
        nw = __ldg(A.wp_off + wk + 1) - s0;  // targets of this world from s0 on
    } else {
        nw -= s0;
    }
    const int nvalid = min(kT, nw);
    const bool valid = tid < nvalid;
    const int s = s0 + tid;
    const ForceParams& P = BATCH ? A.worlds[wk] : A.p;
    if (BATCH && A.steps_left && __ldg(A.steps_left + wk) < 0) {
        // A world that has used up its steps is left exactly as its last
        // step left it: A (its state, in that step's order) is not touched,
        // and the cells that step computed for it are counted again for the
        // next sort (the scan consumed the counts).  A world's slots are the
        // same range in A and B, so this tile's slots are its A slots.
        uint32_t c = 0;
        if (valid) c = A.cell[s];
        const unsigned m = __ballot_sync(kFull, valid);
        if (valid) bin_add(A.counts, c, m);
        return;
    }
    // Autotuner: the block's duration in SM cycles, summed per world.
    const long long t_start = BATCH && A.wcycles ? clock64() : 0;
    const int nt = P.ntypes, ms = SMEM_M ? smem_matrix_stride<D>(nt) : nt;
    const float* M = SMEM_M ? sm.mat : P.matrix;
    float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
    typename Layout<D>::Vel vme{};
    const int lane = tid & 31, warp = tid >> 5;
    int cx = 0, row = INT_MAX, prow = INT_MAX, pcx = 0, cy = 0, cz = 0;
    // The matrix rows, two per warp at a time: loaded beside the targets'
    // cells, stored once those are on their way.
    constexpr int kMatLoads = (kSmemMatrixMax + kT / 16 - 1) / (kT / 16);
    float mrow[kMatLoads];
    if (SMEM_M) {
#pragma unroll
        for (int r = 0; r < kMatLoads; ++r) {
            const int i = (tid >> 4) + r * (kT / 16), j = tid & 15;
            mrow[r] = i < nt && j < nt ? __ldg(P.matrix + i * nt + j) : 0.f;
        }
    }
    if (valid) {
        // The target's cell is the one the sort binned it by (computed from
        // these same coordinates by the previous epilogue or the upload).
        // The first lane of a warp also reads the cell of the target before
        // it (the other lanes take their neighbour's by a shuffle).
        const uint32_t c = __ldg(A.slot_cell + s) - P.cell_base;
        const uint32_t cp = lane == 0 && tid > 0 ? __ldg(A.slot_cell + s - 1) - P.cell_base : 0u;
        me = A.bpt[s];
        vme = A.bvel[s];  // needed only by the epilogue: loaded early, off its critical path
        const int nx = P.g.nx;
        row = grid_row(c, P);
        cx = (int)c - row * nx;
        prow = grid_row(cp, P);
        pcx = (int)cp - prow * nx;
        cz = D == 3 ? grid_row((uint32_t)row, P) : 0;
        cy = row - cz * nx;
    }
    if (SMEM_M) {
#pragma unroll
        for (int r = 0; r < kMatLoads; ++r) {
            const int i = (tid >> 4) + r * (kT / 16), j = tid & 15;
            if (i < nt && j < nt) sm.mat[i * ms + j] = mrow[r];
        }
    }
    // Segments: maximal runs of targets in one grid row (rows are
    // nondecreasing, and so are the columns within a segment).  Window
    // columns: each first target of a column adds the columns of its window
    // cx-1..cx+1 that the previous column's window has not added (3 at a
    // segment start); a block-wide scan numbers them, so the target's window
    // starts at staged column kwin = incl - 3.
    {
        const int r_up = __shfl_up_sync(kFull, row, 1), c_up = __shfl_up_sync(kFull, cx, 1);
        if (lane > 0) {
            prow = r_up;
            pcx = c_up;
        }
    }
    const int pcol = tid > 0 ? pcx : 0;
    const bool start = valid && (tid == 0 || prow != row);
    const bool lead = valid && (start || pcol != cx);
    const unsigned leads = __ballot_sync(kFull, lead);
    const int newc = !lead ? 0 : (start ? 3 : min(3, cx - pcol));
    int incl = newc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) sm.wcol[warp] = incl;
    __syncthreads();
    int cbefore = 0, ncol = 0;
#pragma unroll
    for (int w = 0; w < kT / 32; ++w) {
        const int y = sm.wcol[w];
        cbefore += w < warp ? y : 0;
        ncol += y;
    }
    incl += cbefore;
    const int kwin = incl - 3;
    // Staged columns [cb, ce) of the block numbering, as 0 .. ce-cb-1.
    auto fill_columns = [&](int cb, int ce) {
        for (int i = 0; i < newc; ++i) {
            const int ci = incl - newc + i;
            if (ci >= cb && ci < ce) {
                sm.colv[ci - cb] = cx + 2 - newc + i;
                sm.colrow[ci - cb] = D == 3 ? cy | (cz << 16) : row;
            }
        }
    };
    const int nx = P.g.nx;
    const float px = me.x, py = me.y, pz = D == 3 ? me.z : 0.f;
    const float4* const cand = sm.slots + TileSmem<D, V>::kLead;
    const float* Mrow = M + (valid ? Layout<D>::type(me) : 0) * ms;
    Acc acc = {0.f, 0.f, 0.f, 0, 0ull, 0ull, 0ull};
    bool defer = false;
    // 2D, the whole warp together (a lane without `mine` takes no part): the
    // target's staged cells lo .. up-1, its own cell being `own` (which may not
    // be among them, or not with the target's slice of it).  Only a target in the last column or row of a
    // periodic box meets candidates flagged for a target shift; its whole warp
    // then heeds the flags.
    auto evaluate2 = [&](bool mine, int lo, int up, int own, int ncell) {
        const bool any_shift = __any_sync(kFull, mine && P.wrap && (cx == nx - 1 || cy == nx - 1));
        if (!mine) return;
        const int j0 = sm.coff[lo], j1 = sm.coff[up];
        int o0 = j1, o1 = j1, self_j = -1;
        if ((unsigned)(own - lo) < (unsigned)(up - lo)) {
            o0 = sm.coff[own];
            o1 = sm.coff[own + 1];
            self_j = o0 + (s - sm.cglob[own]);
        }
        defer |= any_shift ? cand_window<D, DBG, true>(A, P, cand, sm.coff, sm.cglob, Mrow, ncell, j0, o0, o1, j1,
                                                       self_j, px, py, pz, acc)
                           : cand_window<D, DBG, false>(A, P, cand, sm.coff, sm.cglob, Mrow, ncell, j0, o0, o1, j1,
                                                        self_j, px, py, pz, acc);
    };
    // 3D, the whole warp together (a lane without `mine` takes no part):
    // kCullWords words at a time, the distance test, then the kept
    // candidates' terms.
    auto evaluate3 = [&](bool mine, int lo, int up, int own, int ncell) {
        int j0 = 0, j1 = 0, self = -1;
        if (mine) {
            j0 = sm.coff[lo];
            j1 = sm.coff[up];
            if ((unsigned)(own - lo) < (unsigned)(up - lo)) self = sm.coff[own] + (s - sm.cglob[own]);
            if (DBG) acc.cand += j1 - j0 - (self >= j0 && self < j1 ? 1 : 0);
        }
        // The lanes of a cell read the same candidates; the r-th cell of the
        // warp starts up to 7 before its window, at a staged index of r mod 8,
        // so that the cells' 16-byte loads fall into different banks
        // (250k uniform particles 87.1 -> 85.6 us, 4M blobs 1157 -> 1148 us).
        const int js = j0 - ((j0 - __popc(leads & (kFull >> (31 - lane)))) & 7);
        const LoopK K(P);
        const float neg_thr = -(float)P.rmax2 * (1.f + kCullRel);
        float umin = INFINITY;
        uint2* kept = sm.kept + tid;
        auto walk = [&](auto shifted) {
            constexpr bool kShifted = decltype(shifted)::value;
            const float px1 = px - 1.f, py1 = py - 1.f, pz1 = pz - 1.f;
            for (int j = js; j < j1; j += 32 * kCullWords) {
                const int nw = min(kCullWords, (j1 - j + 31) >> 5);
                // The words that keep something, with the staged index of
                // their bit 31, and how many candidates they keep.
                uint2* put = kept;
                int n = 0;
                for (int i = 0; i < nw; ++i) {
                    const int base = j + 32 * i;
                    uint32_t m = cull_word<kShifted>(cand + base, min(32, j1 - base), px, py, pz, neg_thr);
                    if (base < j0) m &= kFull >> (j0 - base);
                    if ((unsigned)(self - base) < 32u) m &= ~(0x80000000u >> (self - base));
                    if (m) {
                        *put = make_uint2(m, (uint32_t)base + 31);
                        put += kT;
                        n += __popc(m);
                    }
                }
                uint2 next = kept[0];  // the word after the current one
                const uint2* get = kept;
                uint32_t m = 0, top = 0;
                for (; n > 0; --n) {
                    if (m == 0u) {
                        m = next.x;
                        top = next.y;
                        get += kT;
                        next = *get;
                    }
                    const int b = top_bit(m);
                    m &= (1u << b) - 1u;
                    const float4 q = cand[(int)top - b];
                    int tb = __float_as_int(q.w);
                    float pxe = px, pye = py, pze = pz;
                    if (kShifted) {
                        pxe = (tb & kShiftX) ? px1 : px;
                        pye = (tb & kShiftY) ? py1 : py;
                        pze = (tb & kShiftZ) ? pz1 : pz;
                        tb &= 0xffff;
                    }
                    const Term<D> t = cand_term<D>(K, q.x, q.y, q.z, pxe, pye, pze, Mrow[tb], umin);
                    add_term<D>(acc, t);
                    if (DBG && (t.d2 <= K.lo) && t.d2 > 0.f)
                        add_pair<D, true>(acc, make_float4(0.f, 0.f, 0.f, 0.f),
                                          id_of<D>(A, staged_global(sm.coff, sm.cglob, ncell,
                                                                    (int)(top - b))));
                }
            }
        };
        // Only a target in the last column, row or layer of a periodic box
        // meets candidates flagged for a target shift.
        if (__any_sync(kFull, mine && P.wrap && (cx == nx - 1 || cy == nx - 1 || cz == nx - 1)))
            walk(std::true_type{});
        else
            walk(std::false_type{});
        if (mine) defer |= needs_fp64(K, umin);
    };
    auto evaluate = [&](bool mine, int lo, int up, int own, int ncell) {
        if constexpr (D == 3)
            evaluate3(mine, lo, up, own, ncell);
        else
            evaluate2(mine, lo, up, own, ncell);
    };
    const uint32_t* cs = A.cstart + P.cell_base;
    // Stagings of the block's stencil cells (R a column) one after another:
    // [a, a + m) serves every target for the part of its window that lies in
    // it, so a cell is staged once and all lanes of a crowded cell stay at
    // work however few cells fit.  One staging serves them all when every
    // window fits.  The parts follow in the window's order, hence the same
    // bits.  A staging may span segments: its columns are staged one by one
    // with their own rows, and a window never leaves its segment.  A cell that
    // does not fit by itself comes in slices, the last of them with the cells
    // after it.
    // (Whole windows per staging, a window that did not fit read from global
    // memory: 400k particles, 2D at 198 per cell, tile 1, 717 us a step, at
    // 250 992; 3D at 50 per cell, tile 0, 825, tile 2 890; 16 and 128 worlds
    // clustered for 620 steps 1018 and 9237.  In parts 602, 784, 560, 570, 892
    // and 8345; whole columns per part 621, 820, 608 and 620.)
    constexpr int kCols = TileSmem<D, V>::kCols;
    for (int a = 0, skip = 0; a < R * ncol;) {
        const int c = a / R, off = a - c * R, hi = min(c + kCols, ncol);
        fill_columns(c, hi);  // the previous staging no longer reads the columns
        __syncthreads();
        const int m = stage_cells<D, V>(A, P, cs, sm, off, R * (hi - c) - off, skip);
        const int w = R * kwin - a;  // the window's first cell in this staging
        const int staged = max(m, 1), lo = max(w, 0), up = min(w + 3 * R, staged);
        evaluate(valid && lo < up, lo, up, w + R + R / 2, staged);
        a += m;
        skip = m > 0 ? 0 : skip + TileCfg<D, V>::kCap;
    }
    const bool done = valid && !defer;
    uint32_t newcell = 0;
    if (done) newcell = integrate<D, DBG>(A, P, s, me, vme, acc);
    const unsigned mask = __ballot_sync(kFull, done);
    if (done) {
        bin_add(A.counts, newcell, mask);
        A.cell[s] = newcell;
    }
    // Deferred targets (FP64 band pairs): each warp recomputes its own, one
    // at a time, from global memory.  Most warps have none.
    unsigned dm = __ballot_sync(kFull, valid && defer);
    if (dm && lane == 0) atomicAdd(A.defer_count, (uint32_t)__popc(dm));
    while (dm) {
        const int src = __ffs(dm) - 1;
        dm &= dm - 1;
        fixup_target<D, DBG>(A, P, cs, M, __shfl_sync(kFull, s, src), lane);
    }
    if constexpr (SNAP) write_snapshot_warp<D>(A, s0 + 32 * warp, min(32, nvalid - 32 * warp), lane);
    if (BATCH && A.wcycles) {  // block-uniform
        __syncthreads();
        if (tid == 0) atomicAdd(A.wcycles + wk, (unsigned long long)(clock64() - t_start));
    }
}

template <int D, bool DBG, bool BATCH, int V>
void launch_tile(cudaStream_t st, const ForceArgs<D>& A, bool smem_matrix, int batch_tiles) {
    constexpr int kT = TileCfg<D, V>::kTargets;
    const int grid = BATCH ? batch_tiles : (A.n_total + kT - 1) / kT;
    if (grid <= 0) return;
    const size_t sb = sizeof(TileSmem<D, V>);
    if constexpr (!DBG && !BATCH) {
        if (A.snap.any()) {
            if (smem_matrix)
                launch_after(k_force_tile<D, false, true, false, V, true>, dim3(grid), dim3(kT), sb, st, A);
            else
                launch_after(k_force_tile<D, false, false, false, V, true>, dim3(grid), dim3(kT), sb, st, A);
            return;
        }
    }
    if (smem_matrix)
        launch_after(k_force_tile<D, DBG, true, BATCH, V>, dim3(grid), dim3(kT), sb, st, A);
    else
        launch_after(k_force_tile<D, DBG, false, BATCH, V>, dim3(grid), dim3(kT), sb, st, A);
}

template <int D, bool DBG, bool BATCH>
void launch_tile_variant(cudaStream_t st, const ForceArgs<D>& A, bool smem_matrix, int variant, int batch_tiles) {
    if (variant == 1)
        launch_tile<D, DBG, BATCH, 1>(st, A, smem_matrix, batch_tiles);
    else if (variant == 2)
        launch_tile<D, DBG, BATCH, 2>(st, A, smem_matrix, batch_tiles);
    else
        launch_tile<D, DBG, BATCH, 0>(st, A, smem_matrix, batch_tiles);
}

template <int D, bool DBG>
void launch_variant(cudaStream_t st, const ForceArgs<D>& A, bool general, int variant) {
    const int n = A.p.n;
    const bool smem = A.p.ntypes <= kSmemMatrixMax;
    if (general) {
        const int grid = (n + kThreads - 1) / kThreads;
        const size_t sb = smem ? sizeof(float) * A.p.ntypes * smem_matrix_stride<D>(A.p.ntypes) : 0;
        if (smem)
            launch_after(k_force_general<D, DBG, true>, dim3(grid), dim3(kThreads), sb, st, A);
        else
            launch_after(k_force_general<D, DBG, false>, dim3(grid), dim3(kThreads), 0, st, A);
    } else {
        launch_tile_variant<D, DBG, false>(st, A, smem, variant, 0);
    }
}

}  // namespace

template <int D>
void launch_force(cudaStream_t st, const ForceParams& p, bool general, StateBuf<D> b, const uint32_t* cstart,
                  const uint32_t* slot_cell, StateBuf<D> a, uint32_t* cell, uint32_t* counts, uint32_t* defer,
                  const DebugOut* dbg, int variant, const HostSnap* snap) {
    if (p.n <= 0) return;
    ForceArgs<D> A = make_args<D>(p, b, cstart, slot_cell, a, cell, counts, defer, dbg);
    if (snap && !dbg && !general) A.snap = *snap;
    if (dbg)
        launch_variant<D, true>(st, A, general, variant);
    else
        launch_variant<D, false>(st, A, general, variant);
}

template <int D>
void launch_force_batch(cudaStream_t st, const ForceParams* worlds, const int* wp_off, const int* tile_off,
                        const int* steps_left, int tiles, int nworlds, int n_total, bool smem_matrix, StateBuf<D> b,
                        const uint32_t* cstart, const uint32_t* slot_cell, StateBuf<D> a, uint32_t* cell,
                        uint32_t* counts, uint32_t* defer, const DebugOut* dbg, int variant,
                        unsigned long long* wcycles) {
    if (n_total <= 0 || nworlds <= 0 || tiles <= 0) return;
    ForceParams none{};
    ForceArgs<D> A = make_args<D>(none, b, cstart, slot_cell, a, cell, counts, defer, dbg);
    A.worlds = worlds;
    A.wp_off = wp_off;
    A.tile_off = tile_off;
    A.steps_left = steps_left;
    A.wcycles = wcycles;
    A.nworlds = nworlds;
    A.n_total = n_total;
    if (dbg)
        launch_tile_variant<D, true, true>(st, A, smem_matrix, variant, tiles);
    else
        launch_tile_variant<D, false, true>(st, A, smem_matrix, variant, tiles);
}

// Resident blocks per SM of the batched force kernel of one variant (the
// autotuner turns block cycles into SM time with it).
template <int D, int V>
int batch_blocks_per_sm(bool smem_matrix) {
    int nb = 0;
    const cudaError_t e =
        smem_matrix ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_force_tile<D, false, true, true, V>,
                                                                   TileCfg<D, V>::kTargets, sizeof(TileSmem<D, V>))
                    : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_force_tile<D, false, false, true, V>,
                                                                   TileCfg<D, V>::kTargets, sizeof(TileSmem<D, V>));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return nb > 0 ? nb : 1;
}

namespace {

// Every tiled kernel of one dimension and variant may use its TileSmem.
template <int D, bool DBG, bool SMEM_M, bool BATCH, int V, bool SNAP = false>
cudaError_t allow_one() {
    return cudaFuncSetAttribute(k_force_tile<D, DBG, SMEM_M, BATCH, V, SNAP>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem<D, V>));
}

template <int D, int V>
cudaError_t allow_tile_smem() {
    const cudaError_t es[] = {allow_one<D, false, true, false, V>(), allow_one<D, false, false, false, V>(),
                              allow_one<D, true, true, false, V>(),  allow_one<D, true, false, false, V>(),
                              allow_one<D, false, true, true, V>(),  allow_one<D, false, false, true, V>(),
                              allow_one<D, true, true, true, V>(),   allow_one<D, true, false, true, V>(),
                              allow_one<D, false, true, false, V, true>(), allow_one<D, false, false, false, V, true>()};
    for (cudaError_t e : es)
        if (e != cudaSuccess) return e;
    return cudaSuccess;
}

}  // namespace

}  // namespace plg
