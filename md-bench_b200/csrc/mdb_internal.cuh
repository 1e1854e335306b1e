// Internal declarations shared by the libmdb translation units.
// Device data layout (HBM), per context:
//   x        double4[nall_cap + 1]  positions of locals then ghosts; .w holds the type
//                               id as raw int bits (never used arithmetically); last
//                               the dummy atom (MDB_FAR), which pads rows of the list
//   xr       float4[nall_cap + 1]  mixed path: position relative to the centre of the
//                               atom's cell (cells of edge G, a power of two, fixed at
//                               each rebuild), .w type bits
//   qcell    int[nall_cap]      mixed path: the cell of each atom, 10 bits per axis
//   vx,vy,vz / fx,fy,fz         SoA doubles over locals
//   neighbors int32 [ceil(maxneighs / 8)][ld][8]  tiles of 8 consecutive entries of
//                               a row: entry k of atom i at list_at(k, ld, i). A warp
//                               of consecutive atoms reads a tile as 1 KB, and a row
//                               is written in whole 32-byte sectors. Entries of a
//                               row's last tile past numneigh[i] name the dummy atom
//                               nall_cap, which is out of every atom's reach.
//                               Mixed path: the atom index above MDB_CODE_BITS bits
//                               of the pair's cell-offset code
//   numneigh  int32 [nlocal]    entries of atom i
//   bins: CSR (bin_start[mbins+1]) with atoms of a bin in ascending index order,
//         so lists come out in the reference order; their FP32 positions as three
//         arrays (binf, [3][bin_stride(nall_cap)]) and {index, cell} (bin_jq)
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mdb.h"

#define MDB_MAX_TYPES   8
#define MDB_MAX_STENCIL 1331 /* (2*5+1)^3 */
#define MDB_CODE_BITS   6    /* mixed-path list entries: cell-offset code below the index */
#define MDB_IDX_MASK    ((1 << (32 - MDB_CODE_BITS)) - 1)
#define MDB_CODE_SAME   0x15 /* the code of two atoms in one cell */
#define MDB_FAR         1.0e18 /* coordinates of the dummy atom */

#define MDB_TILE        8 /* list entries of one row in one 32-byte sector */

// device counters (int slots)
enum {
    CNT_NGHOST       = 0, // ghosts in use (clamped to capacity)
    CNT_NGHOST_TOTAL = 1, // ghosts requested by the last setupPbc
    CNT_MAXNEED      = 2, // largest numneigh seen when a row overflowed
    CNT_BADBIN       = 3, // atoms found outside the bin grid
    CNT_BADCELL      = 4, // mixed path: neighbour farther than two cells
    CNT_TYPES        = 5, // and 6: the type check's two ints (zero between checks)
    CNT_SLOTS        = 8
};

struct BinGeom {
    int nbinx, nbiny, nbinz;
    int mbinx, mbiny, mbinz;
    int pad_x, pad_y, pad_z;
    int nstencil, mbins;
    double binsizex, binsizey, binsizez;
    double bininvx, bininvy, bininvz;
    double xlo, ylo, zlo; // fabs(0 - pad*binsize) + 1e-9, verletlist/neighbor.c:361-366
};

struct LJTable {
    int ntypes;
    int uniform; // every type pair has the same epsilon and sigma6
    double eps[MDB_MAX_TYPES * MDB_MAX_TYPES];
    double sig6[MDB_MAX_TYPES * MDB_MAX_TYPES];
};

struct LJTableF {
    int ntypes;
    int uniform;
    float eps[MDB_MAX_TYPES * MDB_MAX_TYPES];
    float sig6[MDB_MAX_TYPES * MDB_MAX_TYPES];
};

// Mixed-path cells: edge G, the smallest power of two >= cutneigh, so the
// cells of a listed pair differ by -1, 0 or +1 per axis and offset * G is
// exact in FP32. A list entry stores the three offsets + 1 as 2-bit fields
// below the index bits.
struct CellFrame {
    double g;
    double ginv;
};

struct CellShift {
    float g;
};

// atom index of a mixed-path entry
__device__ __forceinline__ int entry_index(int e) { return (int)((unsigned)e >> MDB_CODE_BITS); }

// Field a of an entry's cell-offset code as an exact float, 4^a (offset + 1)
// above 1.5 * 2^23, without a shift or an int->float conversion: the field
// stays where it is in the mantissa. Less CELL_BIAS(a) that is 4^a * offset,
// which times G / 4^a (exact, powers of two) is offset * G.
__device__ __forceinline__ float cell_field(int e, int a)
{
    return __int_as_float(0x4B400000 | (e & (3 << (2 * a))));
}
#define CELL_BIAS(a) (12582912.0f + (float)(1 << (2 * (a))))

// pair difference p_i - p_j - offset * G on the mixed path; a fused multiply-add
// with the exact product offset * G rounds once
__device__ __forceinline__ void cell_delta(const float4& pi, const float4& pj, int e, float g,
    float& dx, float& dy, float& dz)
{
    dx = __fmaf_rn(CELL_BIAS(0) - cell_field(e, 0), g, pi.x - pj.x);
    dy = __fmaf_rn(CELL_BIAS(1) - cell_field(e, 1), 0.25f * g, pi.y - pj.y);
    dz = __fmaf_rn(CELL_BIAS(2) - cell_field(e, 2), 0.0625f * g, pi.z - pj.z);
}

struct EamDev {
    int nrho, nr;
    double rdr, rdrho;
    // two double4 per grid point: coefficients 3..6 (the value's cubic), then
    // 0..2 (its derivative's quadratic)
    const double4* frho;
    const double4* rhor;
    const double4* z2r;
    // mixed path, FP32 rows: dens32[m] = rho coefficients 3..6 (the density
    // pass); pair32[2m], pair32[2m + 1] = z2r coefficients 3..6, then rho
    // coefficients 0..2 and z2r coefficient 0 (the force pass: z2r 1 and 2
    // are 2 c4 / dr and c5 / dr of the spline, formed in the kernel)
    const float4* dens32;
    const float4* pair32;
};

namespace mdb {

// ---- small device helpers ---------------------------------------------------
__device__ __forceinline__ int type_of(const double4& p) { return (int)__double_as_longlong(p.w); }

// a double4 in one 256-bit read-only load (sm_100; p 32-byte aligned, as
// every double4 array from cudaMalloc is)
__device__ __forceinline__ double4 ldg4(const double4* p)
{
    double4 r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w)
        : "l"(p));
    return r;
}

__device__ __forceinline__ int pack_cell(int cx, int cy, int cz)
{
    return (cx + 512) | ((cy + 512) << 10) | ((cz + 512) << 20);
}

__device__ __forceinline__ int cell_axis(int q, int a) { return ((q >> (10 * a)) & 1023) - 512; }

// position relative to the centre of cell q, FP32
__device__ __forceinline__ float4 rel_position(const double4& p, int q, const CellFrame& cf)
{
    float4 r;
    r.x = (float)(p.x - ((double)cell_axis(q, 0) + 0.5) * cf.g);
    r.y = (float)(p.y - ((double)cell_axis(q, 1) + 0.5) * cf.g);
    r.z = (float)(p.z - ((double)cell_axis(q, 2) + 0.5) * cf.g);
    r.w = __int_as_float(type_of(p));
    return r;
}

// entry k of row i of a tiled list
__host__ __device__ __forceinline__ size_t list_at(int k, int ld, int i)
{
    return ((size_t)(k / MDB_TILE) * ld + i) * MDB_TILE + k % MDB_TILE;
}

// floats of one coordinate of the bin-ordered positions: 16-byte aligned
// loads, which may reach 7 entries past the binned atoms
__host__ __device__ __forceinline__ int bin_stride(int nall_cap) { return (nall_cap + 11) & ~3; }

// ints of a tiled list of rows of up to maxneighs entries
__host__ __device__ __forceinline__ size_t list_ints(int maxneighs, int ld)
{
    return (size_t)((maxneighs + MDB_TILE - 1) / MDB_TILE) * ld * MDB_TILE;
}

// one tile (32-byte aligned) in one 256-bit load that leaves L1 to the
// gathered positions
__device__ __forceinline__ void ld_tile(const int* p, int (&e)[MDB_TILE])
{
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(e[0]), "=r"(e[1]), "=r"(e[2]), "=r"(e[3]), "=r"(e[4]), "=r"(e[5]),
                   "=r"(e[6]), "=r"(e[7])
                 : "l"(p));
}

// block-wide sum; the result is valid in thread 0 (all threads must call)
__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double ws[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) ws[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (warp == 0) {
        t = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1)
            t += __shfl_down_sync(0xffffffffu, t, o);
    }
    __syncthreads();
    return t;
}

// ---- launch helpers (implemented in the .cu files) --------------------------

// scan: out[0..n] exclusive prefix sums of in[0..n-1]; out[n] = total.
// scratch must hold scan_scratch_ints(n) ints.
int scan_scratch_ints(int n);
void scan_exclusive(const int* in, int* out, int n, int* scratch, cudaStream_t s);
void scan_exclusive_steps(const int* in, int* out, int n, int* scratch, cudaStream_t s);

// integrator / pbc / thermo (mdb_vl.cu). xr/qcell are null on the FP64 path.
// (final_: finalIntegrate of the step before in the same pass)
struct VlImages { // what an initial integration does besides, see initial_step
    const int* off      = nullptr; // ghosts of each atom (null: no ghost update)
    const int* code     = nullptr;
    const int* counters = nullptr;
    int nlocal = 0, zero = 0;
    double xprd = 0, yprd = 0, zprd = 0;
};
// half-list systems of at most this many atoms clear their forces there (their
// arrays and the integrator's streams then stay in L2 together)
#define VL_ZERO_ATOMS (1 << 18)
void launch_initial_integrate(cudaStream_t s, bool final_, int n, double dtf, double dt,
    double4* x, double* vx, double* vy, double* vz, double* fx, double* fy, double* fz,
    float4* xr, const int* qcell, CellFrame cf, const VlImages& img);
void launch_final_integrate(cudaStream_t s, int n, double dtf, double* vx, double* vy,
    double* vz, const double* fx, const double* fy, const double* fz);
// out (two zeroed ints): {1 + the largest type, > 0 if one is negative}
void launch_type_range(cudaStream_t s, int n, const int* type, int* out);
void launch_pack_atoms(cudaStream_t s, int n, const double* xa, const double* va,
    const int* ta, double4* x, double* vx, double* vy, double* vz);
void launch_unpack_atoms(cudaStream_t s, int n, const double4* x, const double* vx,
    const double* vy, const double* vz, const double* fx, const double* fy, const double* fz,
    double* xa, double* va, double* fa, int* ta);
void launch_wrap(cudaStream_t s, int n, double4* x, double xprd, double yprd, double zprd);
// gathers of sortAtom: out[k] = in[order[k]] (three SoA arrays into out[0..3n))
void launch_permute4(cudaStream_t s, int n, const int* order, const double4* in, double4* out);
void launch_permute3(cudaStream_t s, int n, const int* order, const double* a, const double* b,
    const double* c, double* out);
void launch_ghost_count(cudaStream_t s, int n, const double4* x, double cut, double xprd,
    double yprd, double zprd, int px, int py, int pz, int* cnt);
void launch_ghost_write(cudaStream_t s, int n, int ghost_cap, double4* x, double cut,
    double xprd, double yprd, double zprd, int px, int py, int pz, const int* off,
    int* border_map, int* pbc_code, int* counters);
// ghost positions from their owners; with xr/qcell also the mixed-path copies
// (then x of the ghosts is not written: only the rebuild needs it)
void launch_ghost_update(cudaStream_t s, int nlocal, int ghost_cap, double4* x,
    const int* border_map, const int* pbc_code, double xprd, double yprd, double zprd,
    const int* counters, float4* xr, const int* qcell, CellFrame cf);
// cells and relative positions of atoms [first, first + count) (count may be
// read from counters: pass count < 0 to use nlocal + counters[CNT_NGHOST])
void launch_cells(cudaStream_t s, int nlocal, int nall_cap, const double4* x, float4* xr,
    int* qcell, CellFrame cf, const int* counters, int locals_only);
void launch_bin_count(cudaStream_t s, int nlocal, int nall_cap, const double4* x, BinGeom g,
    int* atom_bin, int* atom_slot, int* bin_count, int* bin_lcount, int* counters);
void launch_bin_scatter(cudaStream_t s, int nlocal, int nall_cap, const int* atom_bin,
    const int* atom_slot, const int* bin_start, int* bin_atoms, const int* counters);
// the atoms of each bin in index order: {index, cell} and FP32 positions in bin
// order (binf: x, then y, then z, bin_stride(nall_cap) each), and the locals
// bin by bin (local_order); qcell null: cells 0
void launch_bin_order(cudaStream_t s, int nlocal, int nall_cap, int mbins, const double4* x,
    const int* atom_bin, const int* bin_start, const int* bin_atoms, const int* loc_start,
    const int* qcell, int2* bin_jq, float* binf, int* local_order);
// the Verlet list from the bin-ordered positions; rows: the stencil's runs of
// bins along x, {flat offset of the middle bin, dy, dz, bins to either side};
// margin bounds the FP32 prefilter's rsq error (only candidates within it take
// the exact FP64 test)
void launch_build_list(cudaStream_t s, int nlocal, int nall_cap, const int* local_order,
    const int* loc_start, const double4* x, BinGeom g, int nrows, const int4* rows, const int* atom_bin,
    const int* bin_start, const int2* bin_jq, const float* binf, double cutneighsq,
    float margin, int half, int maxneighs, int ld, int* neighbors, int* numneigh, int* counters,
    const int* qcell);
int ke_partial_blocks(int n);
void launch_ke_partial(cudaStream_t s, int n, const double* vx, const double* vy,
    const double* vz, double mass, double* partials);
void launch_reduce_partials(cudaStream_t s, int nparts, const double* partials, double* out);

// forces (mdb_force_lj.cu, mdb_force_eam.cu)
// blocks (= energy partials) of the mixed and the FP64 LJ kernels
int force_partial_blocks(int n);
int lj_fp64_blocks(int half, int n);
void launch_lj_fp64(cudaStream_t s, int half, int energy, int nlocal,
    const double4* x, const int* numneigh, const int* neighbors, int ld, double cutforcesq,
    const LJTable& tab, double* fx, double* fy, double* fz, double* epart);
void launch_lj_mixed(cudaStream_t s, int comp, int half, int energy, int nlocal,
    const float4* xr, const CellShift& sh, const int* numneigh,
    const int* neighbors, int ld, float cutforcesq, const LJTableF& tab, double* fx,
    double* fy, double* fz, double* epart);
void launch_eam_fp64(cudaStream_t s, int energy, int nlocal,
    const double4* x, const int* numneigh, const int* neighbors, int ld, double cutforcesq,
    EamDev eam, const int* ghost_off, const int* counters, double* fp, double* fx,
    double* fy, double* fz, double* epart_rho, double* epart_pair);
// mixed EAM: a thread per atom (rho_lanes 2: two in the density pass); xe
// (nlocal + ghost_cap) receives
// (position, F'(rho)) of every atom for the force pass; comp: two-sum
// compensated force sums; returns the energy partials written per pass
int launch_eam_mixed(cudaStream_t s, int energy, int comp, int rho_lanes, int nlocal,
    const float4* xr, const CellShift& sh, const int* numneigh, const int* neighbors, int ld,
    float cutforcesq, EamDev eam, const int* ghost_off, const int* counters, int* cut,
    int* ncut, double* fp, float4* xe, double* fx, double* fy, double* fz, double* epart_rho,
    double* epart_pair);
// blocks (= energy partials per pass) of the EAM kernels
int eam_mixed_blocks(int nlocal);
int eam_fp64_blocks(int nlocal);

// domain-decomposed runs: positions of atoms idx[0..n) plus a shift, AoS
// triples (the halo another domain receives); and the positions of halo
// atoms [first, first + n) from AoS triples (mixed: relative copies too)
void launch_gather_positions(cudaStream_t s, int n, const int* idx, const double4* x, double sx,
    double sy, double sz, double* out);
void launch_set_halo(cudaStream_t s, int first, int n, const double* in, double4* x, float4* xr,
    const int* qcell, const CellFrame& cf);

// launches issued through these helpers by the calling host thread (per
// thread, so that contexts driven from different threads count their own:
// a context is used by one thread at a time)
extern thread_local long long g_launches;

} // namespace mdb

#define MDB_NTHREADS 256
static inline int mdb_blocks(long long n, int t) { return (int)((n + t - 1) / t); }
