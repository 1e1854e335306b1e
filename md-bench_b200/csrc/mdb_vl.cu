// Verlet-list scheme kernels other than the forces: integrator, periodic
// images (ghost map and update), binning, list build and the thermo sums.
// Compiled with -fmad=false: every FP64 expression rounds exactly as the
// reference's strict build evaluates it, which keeps the FP64 path
// bit-identical to the reference (see the parity tests).
#include <algorithm>

#include "mdb_cp_f2.cuh"
#include "mdb_internal.cuh"

namespace mdb {

thread_local long long g_launches = 0;

// ---- integrator: verletlist/integrate.c:21-42 -------------------------------
// The periodic images of an atom follow its new position at once (updatePbcCPU,
// verletlist/pbc.c:42-58): the ghosts of atom i are off[i] .. off[i + 1], as
// setupPbc numbered them. img.off null: no ghost update. img.zero: the force is
// cleared after its use (half lists accumulate into it). The separate ghost
// kernel and the three clearings cost as much as the integrator itself in small
// systems (1.8 + 3 x 1.2 us beside 2.1 us, and the time between kernels).
__device__ __forceinline__ void initial_step(int i, double dtf, double dt, double4* x,
    double& a, double& b, double& c, double* fx, double* fy, double* fz, float4* xr,
    const int* qcell, const CellFrame& cf, const VlImages& img, int g, int gend, double4 p)
{
    a = a + dtf * fx[i];
    b = b + dtf * fy[i];
    c = c + dtf * fz[i];
    if (img.zero) fx[i] = fy[i] = fz[i] = 0.0;
    p.x  = p.x + dt * a;
    p.y  = p.y + dt * b;
    p.z  = p.z + dt * c;
    x[i] = p;
    if (xr) xr[i] = rel_position(p, qcell[i], cf);
    for (; g < gend; g++) {
        const int code = img.code[g];
        const int sx = (code & 3) - 1, sy = ((code >> 2) & 3) - 1, sz = ((code >> 4) & 3) - 1;
        double4 q;
        q.x = p.x + sx * img.xprd;
        q.y = p.y + sy * img.yprd;
        q.z = p.z + sz * img.zprd;
        q.w = p.w;
        if (xr) xr[img.nlocal + g] = rel_position(q, qcell[img.nlocal + g], cf);
        else x[img.nlocal + g] = q;
    }
}

// finalIntegrate(n) (FINAL) then initialIntegrate(n+1): two separately rounded
// velocity updates, exactly as the two reference calls, in one pass
template <bool FINAL>
__global__ void k_initial_integrate(int n, double dtf, double dt, double4* x,
    double* __restrict__ vx, double* __restrict__ vy, double* __restrict__ vz, double* fx,
    double* fy, double* fz, float4* xr, const int* __restrict__ qcell, CellFrame cf, VlImages img)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int g = 0, gend = 0;
    if (img.off) {
        g    = __ldg(&img.off[i]);
        gend = min(__ldg(&img.off[i + 1]), img.counters[CNT_NGHOST]);
    }
    const double4 p = x[i];
    double a = vx[i], b = vy[i], c = vz[i];
    if (FINAL) {
        a = a + dtf * fx[i];
        b = b + dtf * fy[i];
        c = c + dtf * fz[i];
    }
    initial_step(i, dtf, dt, x, a, b, c, fx, fy, fz, xr, qcell, cf, img, g, gend, p);
    vx[i] = a;
    vy[i] = b;
    vz[i] = c;
}

__global__ void k_final_integrate(int n, double dtf, double* __restrict__ vx,
    double* __restrict__ vy, double* __restrict__ vz, const double* __restrict__ fx,
    const double* __restrict__ fy, const double* __restrict__ fz)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vx[i] = vx[i] + dtf * fx[i];
    vy[i] = vy[i] + dtf * fy[i];
    vz[i] = vz[i] + dtf * fz[i];
}

void launch_initial_integrate(cudaStream_t s, bool final_, int n, double dtf, double dt,
    double4* x, double* vx, double* vy, double* vz, double* fx, double* fy, double* fz,
    float4* xr, const int* qcell, CellFrame cf, const VlImages& img)
{
    if (n <= 0) return;
    const int nb = mdb_blocks(n, MDB_NTHREADS);
    if (final_)
        k_initial_integrate<true><<<nb, MDB_NTHREADS, 0, s>>>(n, dtf, dt, x, vx, vy, vz, fx, fy,
            fz, xr, qcell, cf, img);
    else
        k_initial_integrate<false><<<nb, MDB_NTHREADS, 0, s>>>(n, dtf, dt, x, vx, vy, vz, fx, fy,
            fz, xr, qcell, cf, img);
    g_launches++;
}

void launch_final_integrate(cudaStream_t s, int n, double dtf, double* vx, double* vy,
    double* vz, const double* fx, const double* fy, const double* fz)
{
    if (n <= 0) return;
    k_final_integrate<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, dtf, vx, vy, vz,
        fx, fy, fz);
    g_launches++;
}

// ---- host-layout transfer: AoS triples <-> device layout ---------------------
__global__ void k_pack_atoms(int n, const double* __restrict__ xa, const double* __restrict__ va,
    const int* __restrict__ ta, double4* __restrict__ x, double* __restrict__ vx,
    double* __restrict__ vy, double* __restrict__ vz)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    x[i]  = make_double4(xa[3 * i], xa[3 * i + 1], xa[3 * i + 2],
         __longlong_as_double((long long)ta[i]));
    vx[i] = va[3 * i];
    vy[i] = va[3 * i + 1];
    vz[i] = va[3 * i + 2];
}

__global__ void k_unpack_atoms(int n, const double4* __restrict__ x,
    const double* __restrict__ vx, const double* __restrict__ vy,
    const double* __restrict__ vz, const double* __restrict__ fx,
    const double* __restrict__ fy, const double* __restrict__ fz, double* __restrict__ xa,
    double* __restrict__ va, double* __restrict__ fa, int* __restrict__ ta)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 p     = x[i];
    xa[3 * i]     = p.x;
    xa[3 * i + 1] = p.y;
    xa[3 * i + 2] = p.z;
    ta[i]         = type_of(p);
    va[3 * i]     = vx[i];
    va[3 * i + 1] = vy[i];
    va[3 * i + 2] = vz[i];
    fa[3 * i]     = fx[i];
    fa[3 * i + 1] = fy[i];
    fa[3 * i + 2] = fz[i];
}

// out[0] = 1 + the largest type, out[1] > 0 if one is negative (out starts 0)
__global__ void k_type_range(int n, const int* __restrict__ type, int* out)
{
    int hi = 0, neg = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int t = type[i];
        hi          = max(hi, t < 0x7fffffff ? t + 1 : t);
        neg |= t < 0;
    }
    hi  = __reduce_max_sync(0xffffffffu, hi);
    neg = __any_sync(0xffffffffu, neg);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&out[0], hi);
        if (neg) out[1] = 1;
    }
}

void launch_type_range(cudaStream_t s, int n, const int* type, int* out)
{
    if (n <= 0) return;
    k_type_range<<<std::min(mdb_blocks(n, MDB_NTHREADS), 296), MDB_NTHREADS, 0, s>>>(n, type,
        out);
    g_launches++;
}

void launch_pack_atoms(cudaStream_t s, int n, const double* xa, const double* va,
    const int* ta, double4* x, double* vx, double* vy, double* vz)
{
    if (n <= 0) return;
    k_pack_atoms<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, xa, va, ta, x, vx, vy,
        vz);
    g_launches++;
}

void launch_unpack_atoms(cudaStream_t s, int n, const double4* x, const double* vx,
    const double* vy, const double* vz, const double* fx, const double* fy, const double* fz,
    double* xa, double* va, double* fa, int* ta)
{
    if (n <= 0) return;
    k_unpack_atoms<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, x, vx, vy, vz, fx,
        fy, fz, xa, va, fa, ta);
    g_launches++;
}

// ---- wrap: updateAtomsPbcCPU, verletlist/pbc.c:62-87 ------------------------
__global__ void k_wrap(int n, double4* __restrict__ x, double xprd, double yprd, double zprd)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 p = x[i];
    if (p.x < 0.0) p.x += xprd;
    else if (p.x >= xprd) p.x -= xprd;
    if (p.y < 0.0) p.y += yprd;
    else if (p.y >= yprd) p.y -= yprd;
    if (p.z < 0.0) p.z += zprd;
    else if (p.z >= zprd) p.z -= zprd;
    x[i] = p;
}

void launch_wrap(cudaStream_t s, int n, double4* x, double xprd, double yprd, double zprd)
{
    if (n <= 0) return;
    k_wrap<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, x, xprd, yprd, zprd);
    g_launches++;
}

// ---- sortAtom, verletlist/neighbor.c:466-536 ----------------------------------
// New atom k is old atom order[k] (the locals bin by bin, each bin's atoms in
// index order); positions carry the type bits, so types move with them.
__global__ void k_permute4(int n, const int* __restrict__ order, const double4* __restrict__ in,
    double4* __restrict__ out)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[k] = in[order[k]];
}

// three SoA arrays a, b, c into out[0..n), out[n..2n), out[2n..3n)
__global__ void k_permute3(int n, const int* __restrict__ order, const double* __restrict__ a,
    const double* __restrict__ b, const double* __restrict__ c, double* __restrict__ out)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int o = order[k];
    out[k]         = a[o];
    out[n + k]     = b[o];
    out[2 * n + k] = c[o];
}

void launch_permute4(cudaStream_t s, int n, const int* order, const double4* in, double4* out)
{
    if (n <= 0) return;
    k_permute4<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, order, in, out);
    g_launches++;
}

void launch_permute3(cudaStream_t s, int n, const int* order, const double* a, const double* b,
    const double* c, double* out)
{
    if (n <= 0) return;
    k_permute3<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, order, a, b, c, out);
    g_launches++;
}

// ---- ghost map: setupPbc, verletlist/pbc.c:103-232 ---------------------------
// The 26 image candidates of one atom, enumerated in the reference's order
// (6 faces, 8 corners, 12 edges). For each candidate `visit(sx, sy, sz)` is
// called when the atom lies within cutneigh of the faces it crosses.
template <typename F>
__device__ __forceinline__ void for_each_image(double x, double y, double z, double c,
    double xp, double yp, double zp, int px, int py, int pz, F visit)
{
    const bool xl = x < c, xh = x >= (xp - c);
    const bool yl = y < c, yh = y >= (yp - c);
    const bool zl = z < c, zh = z >= (zp - c);
    if (px) {
        if (xl) visit(+1, 0, 0);
        if (xh) visit(-1, 0, 0);
    }
    if (py) {
        if (yl) visit(0, +1, 0);
        if (yh) visit(0, -1, 0);
    }
    if (pz) {
        if (zl) visit(0, 0, +1);
        if (zh) visit(0, 0, -1);
    }
    if (px && py && pz) {
        if (xl && yl && zl) visit(+1, +1, +1);
        if (xl && yh && zl) visit(+1, -1, +1);
        if (xl && yl && zh) visit(+1, +1, -1);
        if (xl && yh && zh) visit(+1, -1, -1);
        if (xh && yl && zl) visit(-1, +1, +1);
        if (xh && yh && zl) visit(-1, -1, +1);
        if (xh && yl && zh) visit(-1, +1, -1);
        if (xh && yh && zh) visit(-1, -1, -1);
    }
    if (px && pz) {
        if (xl && zl) visit(+1, 0, +1);
        if (xl && zh) visit(+1, 0, -1);
        if (xh && zl) visit(-1, 0, +1);
        if (xh && zh) visit(-1, 0, -1);
    }
    if (py && pz) {
        if (yl && zl) visit(0, +1, +1);
        if (yl && zh) visit(0, +1, -1);
        if (yh && zl) visit(0, -1, +1);
        if (yh && zh) visit(0, -1, -1);
    }
    if (px && py) {
        if (yl && xl) visit(+1, +1, 0);
        if (yl && xh) visit(-1, +1, 0);
        if (yh && xl) visit(+1, -1, 0);
        if (yh && xh) visit(-1, -1, 0);
    }
}

__global__ void k_ghost_count(int n, const double4* __restrict__ x, double c, double xp,
    double yp, double zp, int px, int py, int pz, int* __restrict__ cnt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 p = x[i];
    int k     = 0;
    for_each_image(p.x, p.y, p.z, c, xp, yp, zp, px, py, pz, [&](int, int, int) { k++; });
    cnt[i] = k;
}

__device__ __forceinline__ int pack_shift(int sx, int sy, int sz)
{
    return (sx + 1) | ((sy + 1) << 2) | ((sz + 1) << 4);
}

__global__ void k_ghost_write(int n, int ghost_cap, double4* __restrict__ x, double c,
    double xp, double yp, double zp, int px, int py, int pz, const int* __restrict__ off,
    int* __restrict__ border_map, int* __restrict__ pbc_code)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 p = x[i];
    int g     = off[i];
    for_each_image(p.x, p.y, p.z, c, xp, yp, zp, px, py, pz, [&](int sx, int sy, int sz) {
        if (g < ghost_cap) {
            border_map[g] = i;
            pbc_code[g]   = pack_shift(sx, sy, sz);
            double4 gp;
            gp.x     = p.x + sx * xp;
            gp.y     = p.y + sy * yp;
            gp.z     = p.z + sz * zp;
            gp.w     = p.w;
            x[n + g] = gp;
        }
        g++;
    });
}

__global__ void k_ghost_finalize(int n, int ghost_cap, const int* __restrict__ off,
    int* __restrict__ counters)
{
    int total                  = off[n];
    counters[CNT_NGHOST_TOTAL] = total;
    counters[CNT_NGHOST]       = total < ghost_cap ? total : ghost_cap;
}

void launch_ghost_count(cudaStream_t s, int n, const double4* x, double cut, double xprd,
    double yprd, double zprd, int px, int py, int pz, int* cnt)
{
    if (n <= 0) return;
    k_ghost_count<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, x, cut, xprd, yprd,
        zprd, px, py, pz, cnt);
    g_launches++;
}

void launch_ghost_write(cudaStream_t s, int n, int ghost_cap, double4* x, double cut,
    double xprd, double yprd, double zprd, int px, int py, int pz, const int* off,
    int* border_map, int* pbc_code, int* counters)
{
    k_ghost_finalize<<<1, 1, 0, s>>>(n, ghost_cap, off, counters);
    g_launches++;
    if (n <= 0) return;
    k_ghost_write<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, ghost_cap, x, cut,
        xprd, yprd, zprd, px, py, pz, off, border_map, pbc_code);
    g_launches++;
}

// ---- ghost update: updatePbcCPU, verletlist/pbc.c:42-58 ----------------------
__global__ void k_ghost_update(int nlocal, double4* __restrict__ x,
    const int* __restrict__ border_map, const int* __restrict__ pbc_code, double xp,
    double yp, double zp, const int* __restrict__ counters, float4* __restrict__ xr,
    const int* __restrict__ qcell, CellFrame cf)
{
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= counters[CNT_NGHOST]) return;
    int b     = border_map[g];
    int code  = pbc_code[g];
    int sx    = (code & 3) - 1, sy = ((code >> 2) & 3) - 1, sz = ((code >> 4) & 3) - 1;
    double4 p = x[b];
    double4 q;
    q.x = p.x + sx * xp;
    q.y = p.y + sy * yp;
    q.z = p.z + sz * zp;
    q.w = p.w;
    if (xr) xr[nlocal + g] = rel_position(q, qcell[nlocal + g], cf);
    else x[nlocal + g] = q;
}

void launch_ghost_update(cudaStream_t s, int nlocal, int ghost_cap, double4* x,
    const int* border_map, const int* pbc_code, double xprd, double yprd, double zprd,
    const int* counters, float4* xr, const int* qcell, CellFrame cf)
{
    if (ghost_cap <= 0) return;
    k_ghost_update<<<mdb_blocks(ghost_cap, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(nlocal, x,
        border_map, pbc_code, xprd, yprd, zprd, counters, xr, qcell, cf);
    g_launches++;
}

// ---- mixed-path cells: qcell = floor(x / G) per axis, xr relative to its centre
__global__ void k_cells(int nlocal, const double4* __restrict__ x, float4* __restrict__ xr,
    int* __restrict__ qcell, CellFrame cf, const int* __restrict__ counters, int locals_only)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = locals_only ? nlocal : nlocal + counters[CNT_NGHOST];
    if (i >= n) return;
    double4 p = x[i];
    int q     = pack_cell((int)floor(p.x * cf.ginv), (int)floor(p.y * cf.ginv),
            (int)floor(p.z * cf.ginv));
    qcell[i]  = q;
    xr[i]     = rel_position(p, q, cf);
}

void launch_cells(cudaStream_t s, int nlocal, int nall_cap, const double4* x, float4* xr,
    int* qcell, CellFrame cf, const int* counters, int locals_only)
{
    int n = locals_only ? nlocal : nall_cap;
    if (n <= 0) return;
    k_cells<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(nlocal, x, xr, qcell, cf,
        counters, locals_only);
    g_launches++;
}

// ---- binning: coord2bin + binatoms, verletlist/neighbor.c:355-464 ------------
__device__ __forceinline__ int coord2bin(const double4& p, const BinGeom& g)
{
    int ix = (int)((p.x + g.xlo) * g.bininvx);
    int iy = (int)((p.y + g.ylo) * g.bininvy);
    int iz = (int)((p.z + g.zlo) * g.bininvz);
    if (ix < 0 || iy < 0 || iz < 0 || ix >= g.mbinx || iy >= g.mbiny || iz >= g.mbinz)
        return -1;
    return iz * g.mbiny * g.mbinx + iy * g.mbinx + ix;
}

// bin_count[b]: atoms in bin b; bin_lcount[b]: local atoms in bin b
__global__ void k_bin_count(int nlocal, const double4* __restrict__ x, BinGeom g,
    int* __restrict__ atom_bin, int* __restrict__ atom_slot, int* __restrict__ bin_count,
    int* __restrict__ bin_lcount, int* __restrict__ counters)
{
    int i    = blockIdx.x * blockDim.x + threadIdx.x;
    int nall = nlocal + counters[CNT_NGHOST];
    if (i >= nall) return;
    int b = coord2bin(x[i], g);
    if (b < 0) {
        atomicAdd(&counters[CNT_BADBIN], 1);
        atom_bin[i] = -1;
        return;
    }
    atom_bin[i]  = b;
    atom_slot[i] = atomicAdd(&bin_count[b], 1);
    if (i < nlocal) atomicAdd(&bin_lcount[b], 1);
}

__global__ void k_bin_scatter(int nlocal, const int* __restrict__ atom_bin,
    const int* __restrict__ atom_slot, const int* __restrict__ bin_start,
    int* __restrict__ bin_atoms, const int* __restrict__ counters)
{
    int i    = blockIdx.x * blockDim.x + threadIdx.x;
    int nall = nlocal + counters[CNT_NGHOST];
    if (i >= nall) return;
    int b = atom_bin[i];
    if (b < 0) return;
    bin_atoms[bin_start[b] + atom_slot[i]] = i;
}

// Atoms of a bin in ascending index order: the order binatoms produces when it
// fills bins in one serial pass (verletlist/neighbor.c:443-454). One thread per
// binned atom counts the smaller indices of its bin. Locals have the smaller
// indices, so they form the head of each bin; the heads of all bins,
// concatenated in bin order, give local_order (the order in which sortAtom
// places the local atoms).
__global__ void k_bin_order(int nlocal, int mbins, int stride, const double4* __restrict__ x,
    const int* __restrict__ atom_bin, const int* __restrict__ bin_start,
    const int* __restrict__ bin_atoms, const int* __restrict__ loc_start,
    const int* __restrict__ qcell, int2* __restrict__ bin_jq, float* __restrict__ binf,
    int* __restrict__ local_order)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= bin_start[mbins]) return;
    const int j = bin_atoms[m], b = atom_bin[j];
    const int s = bin_start[b], e = bin_start[b + 1];
    int r = 0;
    for (int k = s; k < e; k++)
        r += bin_atoms[k] < j;
    if (j < nlocal) local_order[loc_start[b] + r] = j;
    const double4 p      = x[j];
    bin_jq[s + r]        = make_int2(j, qcell ? qcell[j] : 0);
    binf[s + r]          = (float)p.x;
    binf[stride + s + r] = (float)p.y;
    binf[2 * (size_t)stride + s + r] = (float)p.z;
}

void launch_bin_count(cudaStream_t s, int nlocal, int nall_cap, const double4* x, BinGeom g,
    int* atom_bin, int* atom_slot, int* bin_count, int* bin_lcount, int* counters)
{
    k_bin_count<<<mdb_blocks(nall_cap, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(nlocal, x, g,
        atom_bin, atom_slot, bin_count, bin_lcount, counters);
    g_launches++;
}

void launch_bin_scatter(cudaStream_t s, int nlocal, int nall_cap, const int* atom_bin,
    const int* atom_slot, const int* bin_start, int* bin_atoms, const int* counters)
{
    k_bin_scatter<<<mdb_blocks(nall_cap, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(nlocal, atom_bin,
        atom_slot, bin_start, bin_atoms, counters);
    g_launches++;
}

void launch_bin_order(cudaStream_t s, int nlocal, int nall_cap, int mbins, const double4* x,
    const int* atom_bin, const int* bin_start, const int* bin_atoms, const int* loc_start,
    const int* qcell, int2* bin_jq, float* binf, int* local_order)
{
    if (nall_cap <= 0) return;
    k_bin_order<<<mdb_blocks(nall_cap, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(nlocal, mbins,
        bin_stride(nall_cap), x, atom_bin, bin_start, bin_atoms, loc_start, qcell, bin_jq, binf,
        local_order);
    g_launches++;
}

// ---- list build: buildNeighborCPU, verletlist/neighbor.c:260-352 -------------
// One thread per local atom, taken in bin order so that a warp's threads walk
// the same candidates. The stencil is walked in the reference order as runs of
// consecutive bins along x, whose atoms are one contiguous range of the
// bin-ordered copies, and each bin's atoms stand in index order, so row i holds
// exactly the reference's neighbours of i in the reference's order. A run is
// cut to the bins whose box can lie within cutneigh of the atom (a lower bound
// on every distance to its atoms, with a relative margin: only candidates that
// would fail the test are left out). Candidates are tested eight at a time, two
// per packed instruction and without a branch: the signs of rsq - hi collect in
// a bit mask of up to 32 candidates. hi lies above cutneigh^2 by the FP32 rounding
// error `margin`; a mask with a candidate within twice that below hi goes through
// the reference's exact FP64 test. The accepted ones' places go, in order, to a ring in shared memory;
// its full tiles are turned into list entries together (the threads of a warp
// stay converged there) and leave as whole 32-byte sectors, wherever the row
// lies. On the mixed path each entry also carries the cell offset of the pair
// (2 bits per axis below the index). Bound by instructions: threads of a warp
// differ in their runs and accepted candidates (15 of 32 threads active). 1M LJ
// atoms 1,330 -> 913 us, 47,840 137 -> 111 us (half lists), Cu 131,072 227 -> 127
// us, 3,960 130 -> 62 us against one branching test per candidate. The bound of 64
// registers serves the large systems: the form before it took 974 us at 1M atoms, but
// 99 at 47,840, which have few blocks.
static constexpr int BL_THREADS = 128;
static constexpr int BL_KEEP    = 15; // entries that wait before tiles are written
static constexpr int BL_RING    = 48; // > BL_KEEP + 32 accepted of a mask

__global__ void __launch_bounds__(BL_THREADS, 8) k_build_list(int nlocal,
    const int* __restrict__ local_order, const int* __restrict__ loc_start,
    const double4* __restrict__ x, BinGeom g, int nrows, const int4* __restrict__ rows,
    const int* __restrict__ atom_bin, const int* __restrict__ bin_start,
    const int2* __restrict__ bin_jq, const float* __restrict__ binf, int stride,
    double cutneighsq, float margin, int half, int maxneighs, int ld, int dummy,
    int* __restrict__ neighbors, int* __restrict__ numneigh, int* __restrict__ counters,
    const int* __restrict__ qcell)
{
    using namespace cp;
    __shared__ int s_ring[BL_RING][BL_THREADS];
    extern __shared__ int4 s_rows[];
    for (int k = threadIdx.x; k < nrows; k += blockDim.x)
        s_rows[k] = rows[k];
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t < nlocal ? local_order[t] : -1;
    if (i < 0) return; // past the binned locals (an atom outside the grid is an error)
    const double4 xi = x[i];
    const int ibin   = atom_bin[i];
    // i's own place: the locals lead their bin, in local_order's order
    const int self   = bin_start[ibin] + t - loc_start[ibin];
    const double ux  = (xi.x + g.xlo) * g.bininvx;
    const double uy  = (xi.y + g.ylo) * g.bininvy;
    const double uz  = (xi.z + g.zlo) * g.bininvz;
    const float fx   = (float)(ux - (double)(int)ux);
    const float fy   = (float)(uy - (double)(int)uy);
    const float fz   = (float)(uz - (double)(int)uz);
    const float by = (float)g.binsizey, bz = (float)g.binsizez;
    const float bxinv = 1.0f / (float)g.binsizex;
    const float skip2 = (float)cutneighsq * 1.0001f + 1e-4f;
    const float hi = (float)cutneighsq + margin;
    const float near = 2.0f * margin + 1e-6f * hi; // hi - rsq of a candidate left to FP64
    const f2 XI = f2_pack((float)xi.x, (float)xi.x), YI = f2_pack((float)xi.y, (float)xi.y),
             ZI = f2_pack((float)xi.z, (float)xi.z);
    const f2 HI = f2_pack(hi, hi);
    // 1 + the difference of two packed cells, field by field
    const int q1 = qcell ? 0x00100401 - qcell[i] : 0;
    int* ring    = &s_ring[0][threadIdx.x];
    int n = 0, nf = 0; // accepted, written to the list
    int bad = 0;

    // |distance to the run in y and z|^2 at the least
    auto gap2 = [&](const int4& r) {
        float gy = r.y > 0 ? (r.y - fy) : (r.y < 0 ? (fy - (r.y + 1)) : 0.f);
        float gz = r.z > 0 ? (r.z - fz) : (r.z < 0 ? (fz - (r.z + 1)) : 0.f);
        gy *= by;
        gz *= bz;
        return gy * gy + gz * gz;
    };
    // the ring's entries nf .. nf + 7 as a tile of the list; those past n: the
    // dummy atom
    auto flush = [&]() {
        if (nf < maxneighs) {
            int v[MDB_TILE];
#pragma unroll
            for (int u = 0; u < MDB_TILE; u++) {
                const bool real = nf + u < n;
                const int2 jq   = __ldg(&bin_jq[real ? ring[((nf + u) % BL_RING) * BL_THREADS]
                                                     : self]);
                v[u]            = real ? jq.x : dummy;
                if (qcell) {
                    // each field 0, 1 or 2; another value sets a bit outside
                    // the fields or both bits of one
                    const int d = jq.y + q1;
                    bad |= (d & ~0x00300c03) | (d & (d >> 1) & 0x00100401);
                    v[u] = (v[u] << MDB_CODE_BITS) | ((d | (d >> 8) | (d >> 16)) & 0x3f);
                }
            }
            int4* p = reinterpret_cast<int4*>(neighbors + list_at(nf, ld, i));
            p[0]    = make_int4(v[0], v[1], v[2], v[3]);
            p[1]    = make_int4(v[4], v[5], v[6], v[7]);
        }
        nf += MDB_TILE;
    };

    for (int r0 = 0; r0 < nrows; r0 += 32) {
        // the runs within reach first, so that the threads of a warp stay together
        const int nr = min(32, nrows - r0);
        unsigned rm  = 0;
        for (int r = 0; r < nr; r++)
            if (gap2(s_rows[r0 + r]) <= skip2) rm |= 1u << r;
        while (rm) {
            const int4 run = s_rows[r0 + __ffs(rm) - 1];
            rm &= rm - 1;
            const float ext = sqrtf(skip2 - gap2(run)) * bxinv * 1.00001f + 1e-5f;
            const int imax  = min(run.w, (int)floorf(fx + ext));
            const int imin  = max(-run.w, (int)ceilf(fx - ext - 1.0f));
            const int b0 = max(ibin + run.x + imin, 0), b1 = min(ibin + run.x + imax + 1, g.mbins);
            const int beg = b0 < b1 ? __ldg(&bin_start[b0]) : 0;
            const int end = b0 < b1 ? __ldg(&bin_start[b1]) : 0;
            for (int mb = beg & ~3; mb < end; mb += 32) {
                const int ng    = min(4, (end - mb + 7) >> 3);
                const float4* p = reinterpret_cast<const float4*>(binf + mb);
                const int s4    = stride >> 2;
                unsigned in = 0;     // first candidate in the highest bit
                float mn    = 1e30f; // smallest |rsq - hi|
                for (int q = 0; q < ng; q++, p += 2) {
                    float4 X[2], Y[2], Z[2];
#pragma unroll
                    for (int w = 0; w < 2; w++) {
                        X[w] = __ldg(p + w);
                        Y[w] = __ldg(p + s4 + w);
                        Z[w] = __ldg(p + 2 * (size_t)s4 + w);
                    }
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        const float4 &a = X[w / 2], &b = Y[w / 2], &c = Z[w / 2];
                        const f2 dx = f2_sub(XI, w & 1 ? f2_pack(a.z, a.w) : f2_pack(a.x, a.y));
                        const f2 dy = f2_sub(YI, w & 1 ? f2_pack(b.z, b.w) : f2_pack(b.x, b.y));
                        const f2 dz = f2_sub(ZI, w & 1 ? f2_pack(c.z, c.w) : f2_pack(c.x, c.y));
                        const f2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
                        float a0, a1;
                        f2_unpack(f2_sub(r2, HI), a0, a1);
                        in = __funnelshift_l(__float_as_uint(a0), in, 1);
                        in = __funnelshift_l(__float_as_uint(a1), in, 1);
                        mn = fminf(fminf(fabsf(a0), fabsf(a1)), mn);
                    }
                }
                in <<= 32 - 8 * ng;
                if (beg > mb) in &= 0xffffffffu >> (beg - mb);
                if (end - mb < 32) in &= ~(0xffffffffu >> (end - mb));
                if ((unsigned)(self - mb) < 32u) in &= ~(0x80000000u >> (self - mb));
                // near the cutoff (3 atoms in 100 have such a candidate):
                // the reference's test, verletlist/neighbor.c:320-330
                for (unsigned un = mn <= near ? in : 0; un;) {
                    const unsigned bit = 0x80000000u >> __clz(un);
                    un ^= bit;
                    const double4 xj = ldg4(&x[bin_jq[mb + __clz(bit)].x]);
                    double delx      = xi.x - xj.x;
                    double dely      = xi.y - xj.y;
                    double delz      = xi.z - xj.z;
                    double rsq       = delx * delx + dely * dely + delz * delz;
                    if (!(rsq <= cutneighsq)) in ^= bit;
                }
                while (in) {
                    const int u = __clz(in);
                    in ^= 0x80000000u >> u;
                    if (half && __ldg(&bin_jq[mb + u].x) < i) continue;
                    ring[(n % BL_RING) * BL_THREADS] = mb + u;
                    n++;
                }
                // the threads that are here together write together
                if (__any_sync(__activemask(), n - nf > BL_KEEP))
                    while (n - nf >= MDB_TILE)
                        flush();
            }
        }
    }
    while (nf < n)
        flush();
    // the stored count never exceeds the row capacity, so no consumer can read
    // past the list; the true count of an overflowing row goes to the host,
    // which grows the list and rebuilds before any force is computed
    numneigh[i] = n < maxneighs ? n : maxneighs;
    if (n > maxneighs) atomicMax(&counters[CNT_MAXNEED], n);
    if (bad) atomicAdd(&counters[CNT_BADCELL], 1);
}

void launch_build_list(cudaStream_t s, int nlocal, int nall_cap, const int* local_order,
    const int* loc_start, const double4* x, BinGeom g, int nrows, const int4* rows,
    const int* atom_bin, const int* bin_start, const int2* bin_jq, const float* binf,
    double cutneighsq, float margin, int half, int maxneighs, int ld, int* neighbors,
    int* numneigh, int* counters, const int* qcell)
{
    if (nlocal <= 0) return;
    const size_t smem = sizeof(int4) * nrows;
    k_build_list<<<mdb_blocks(nlocal, BL_THREADS), BL_THREADS, smem, s>>>(nlocal, local_order,
        loc_start, x, g, nrows, rows, atom_bin, bin_start, bin_jq, binf, bin_stride(nall_cap),
        cutneighsq, margin, half, maxneighs, ld, nall_cap, neighbors, numneigh, counters, qcell);
    g_launches++;
}

// ---- thermo: sum of m v.v per block, then one fixed-order reduction ----------
static constexpr int KE_THREADS    = 256;
static constexpr int KE_MAX_BLOCKS = 1184; // 8 x 148 SMs

int ke_partial_blocks(int n)
{
    int b = mdb_blocks(n, KE_THREADS);
    return b < KE_MAX_BLOCKS ? (b > 0 ? b : 1) : KE_MAX_BLOCKS;
}

__global__ void k_ke_partial(int n, const double* __restrict__ vx,
    const double* __restrict__ vy, const double* __restrict__ vz, double mass,
    double* __restrict__ part)
{
    // sum of (vx^2 + vy^2 + vz^2) * mass, common/thermo.c:74-77
    double t = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double a = vx[i], b = vy[i], c = vz[i];
        t += (a * a + b * b + c * c) * mass;
    }
    t = block_sum(t);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

__global__ void k_reduce_partials(int nparts, const double* __restrict__ part,
    double* __restrict__ out)
{
    double t = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x)
        t += part[i];
    t = block_sum(t);
    if (threadIdx.x == 0) *out = t;
}

void launch_ke_partial(cudaStream_t s, int n, const double* vx, const double* vy,
    const double* vz, double mass, double* partials)
{
    k_ke_partial<<<ke_partial_blocks(n), KE_THREADS, 0, s>>>(n, vx, vy, vz, mass, partials);
    g_launches++;
}

void launch_reduce_partials(cudaStream_t s, int nparts, const double* partials, double* out)
{
    k_reduce_partials<<<1, 1024, 0, s>>>(nparts, partials, out);
    g_launches++;
}

// ---- halo atoms of a domain-decomposed run ------------------------------------
// out[3k..3k+2] = position of atom idx[k] plus shift (the periodic image a
// neighbouring domain sees across the global box boundary; one FP64 addition
// per coordinate, as a ghost image is made)
__global__ void k_gather_positions(int n, const int* __restrict__ idx,
    const double4* __restrict__ x, double sx, double sy, double sz, double* __restrict__ out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double4 p = x[idx[k]];
    out[3 * k]      = p.x + sx;
    out[3 * k + 1]  = p.y + sy;
    out[3 * k + 2]  = p.z + sz;
}

void launch_gather_positions(cudaStream_t s, int n, const int* idx, const double4* x, double sx,
    double sy, double sz, double* out)
{
    if (n <= 0) return;
    k_gather_positions<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(n, idx, x, sx, sy,
        sz, out);
    g_launches++;
}

// halo atoms [first, first + n) take positions from in (AoS triples); their
// type bits stay; the mixed path's relative copy follows (cells fixed at the
// last build, as for the atoms the integrator moves)
__global__ void k_set_halo(int first, int n, const double* __restrict__ in, double4* x,
    float4* xr, const int* __restrict__ qcell, CellFrame cf)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = first + k;
    double4 p   = x[i];
    p.x = in[3 * k], p.y = in[3 * k + 1], p.z = in[3 * k + 2];
    x[i] = p;
    if (xr) xr[i] = rel_position(p, qcell[i], cf);
}

void launch_set_halo(cudaStream_t s, int first, int n, const double* in, double4* x, float4* xr,
    const int* qcell, const CellFrame& cf)
{
    if (n <= 0) return;
    k_set_halo<<<mdb_blocks(n, MDB_NTHREADS), MDB_NTHREADS, 0, s>>>(first, n, in, x, xr, qcell,
        cf);
    g_launches++;
}

} // namespace mdb
