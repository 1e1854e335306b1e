// Lennard-Jones forces over Verlet lists (computeForceLJFullNeigh /
// computeForceLJHalfNeigh, verletlist/force_lj.c:17-206).
//
// Thread t handles atom t and its row of the list, a tile of 8 entries at a
// time (one 256-bit load, 1 KB coalesced per warp); neighbour positions are
// 32-byte (FP64) or 16-byte (mixed) gathers that mostly hit L1/L2. All gathers
// of a tile are issued before any arithmetic, which keeps enough bytes in
// flight. Pairs are summed in list order.
//
// FP64 path: -fmad=false keeps every product and sum rounded as the
// reference's strict build rounds them, so full-list forces are bit-identical.
// Mixed path: FP32 positions relative to the centre of each atom's cell (edge
// G, a power of two) plus the cell offset of the pair (-1, 0, +1 per axis,
// 2-bit fields of the list entry): dx = (p_i - p_j) - offset * G, the offset
// decoded into an exact float with one integer bit operation. No int->float
// conversions, no shared-memory table, one approximate reciprocal per pair;
// FP32 force sums (or two-sum compensated sums), FP64 energy sums.
#include "mdb_cp_f2.cuh"
#include "mdb_internal.cuh"

namespace mdb {

static constexpr int LJ_THREADS = 128;

int force_partial_blocks(int n) { return mdb_blocks(n > 0 ? n : 1, LJ_THREADS); }

// Whether an FP64 system of n atoms shares an atom among 8 threads
// (k_lj_fp64_shared): half lists at every size (29.5 -> 19.7 us per launch at
// 47,840 atoms, 311 -> 235 at 702,464: more of their atomics are in flight), full
// lists while a thread per atom leaves the chip idle. us per launch, a thread per atom
// / 8 threads: 15.5 / 5.6 at 4,000 atoms, 15.5 / 11.5 at 16,384, 16.6 / 15.3 at
// 23,328, 16.8 / 20.2 at 32,000, 39.0 / 65.6 at 119,164. They cross at about 25,000;
// the line lies at 16,384, where the gain is still a quarter.
static bool lj_fp64_shared(int half, int n) { return half || n <= 16384; }

int lj_fp64_blocks(int half, int n)
{
    return lj_fp64_shared(half, n) ? mdb_blocks(n > 0 ? n : 1, LJ_THREADS / MDB_TILE)
                                   : force_partial_blocks(n);
}

template <bool UNIFORM, bool ENERGY>
__global__ void __launch_bounds__(LJ_THREADS) k_lj_fp64(int nlocal, const double4* __restrict__ x,
    const int* __restrict__ numneigh, const int* __restrict__ neighbors, int ld,
    double cutforcesq, LJTable tab, double* __restrict__ fx, double* __restrict__ fy,
    double* __restrict__ fz, double* __restrict__ epart)
{
    __shared__ double s_eps[MDB_MAX_TYPES * MDB_MAX_TYPES];
    __shared__ double s_sig6[MDB_MAX_TYPES * MDB_MAX_TYPES];
    const int nt = tab.ntypes;
    if (!UNIFORM) {
        for (int k = threadIdx.x; k < nt * nt; k += blockDim.x) {
            s_eps[k]  = tab.eps[k];
            s_sig6[k] = tab.sig6[k];
        }
        __syncthreads();
    }
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double epot = 0.0;
    if (t < nlocal) {
        const int i      = t;
        const double4 xi = x[i];
        const int ti     = type_of(xi);
        const int n      = numneigh[i];
        const int* nb    = neighbors + list_at(0, ld, i);
        double fix = 0.0, fiy = 0.0, fiz = 0.0;
        const double eps0 = tab.eps[0], sig0 = tab.sig6[0];

        auto pair = [&](const double4& xj) {
            double delx = xi.x - xj.x;
            double dely = xi.y - xj.y;
            double delz = xi.z - xj.z;
            double rsq  = delx * delx + dely * dely + delz * delz;
            double sigma6 = sig0, epsilon = eps0;
            if (!UNIFORM) {
                int tij = ti * nt + type_of(xj);
                sigma6  = s_sig6[tij];
                epsilon = s_eps[tij];
            }
            if (rsq < cutforcesq) {
                double sr2   = 1.0 / rsq;
                double sr6   = sr2 * sr2 * sr2 * sigma6;
                double force = 48.0 * sr6 * (sr6 - 0.5) * sr2 * epsilon;
                fix += delx * force;
                fiy += dely * force;
                fiz += delz * force;
                if (ENERGY) epot += 0.5 * (4.0 * epsilon * sr6 * (sr6 - 1.0));
            }
        };

        // the next tile is in flight while one is worked on
        int jn[MDB_TILE];
        if (n > 0) ld_tile(nb, jn);
        for (int k = 0; k < n; k += MDB_TILE) {
            int j[MDB_TILE];
            double4 xj[MDB_TILE];
#pragma unroll
            for (int u = 0; u < MDB_TILE; u++)
                j[u] = jn[u];
            nb += (size_t)ld * MDB_TILE;
            if (k + MDB_TILE < n) ld_tile(nb, jn);
#pragma unroll
            for (int u = 0; u < MDB_TILE; u++)
                xj[u] = ldg4(x + j[u]);
#pragma unroll
            for (int u = 0; u < MDB_TILE; u++)
                pair(xj[u]);
        }
        fx[i] = fix;
        fy[i] = fiy;
        fz[i] = fiz;
    }
    if (ENERGY) {
        double e = block_sum(epot);
        if (threadIdx.x == 0) epart[blockIdx.x] = e;
    }
}

// The same with 8 threads per atom, one entry of a tile each: a thread per atom
// leaves small systems with a few warps per scheduler, each on a chain of gathers
// and divisions. Full lists leave their terms in shared memory, where one thread
// per component adds them in list order (a pair outside the cutoff adds an exact
// zero), so forces stay bit-identical; half lists sum per thread and then across
// the 8.
template <bool HALF, bool UNIFORM, bool ENERGY>
__global__ void __launch_bounds__(LJ_THREADS) k_lj_fp64_shared(int nlocal,
    const double4* __restrict__ x, const int* __restrict__ numneigh,
    const int* __restrict__ neighbors, int ld, double cutforcesq, LJTable tab,
    double* __restrict__ fx, double* __restrict__ fy, double* __restrict__ fz,
    double* __restrict__ epart)
{
    constexpr int ATOMS = LJ_THREADS / MDB_TILE;
    __shared__ double s_eps[MDB_MAX_TYPES * MDB_MAX_TYPES];
    __shared__ double s_sig6[MDB_MAX_TYPES * MDB_MAX_TYPES];
    __shared__ double s_term[HALF ? 1 : ATOMS][3][MDB_TILE + 1];
    const int nt = tab.ntypes;
    if (!UNIFORM) {
        for (int k = threadIdx.x; k < nt * nt; k += blockDim.x) {
            s_eps[k]  = tab.eps[k];
            s_sig6[k] = tab.sig6[k];
        }
        __syncthreads();
    }
    const int g = threadIdx.x / MDB_TILE, u = threadIdx.x % MDB_TILE;
    const int i = blockIdx.x * ATOMS + g;
    const int ia     = i < nlocal ? i : 0;
    const double4 xi = x[ia];
    const int ti     = type_of(xi);
    const int n      = i < nlocal ? numneigh[ia] : 0;
    const int* nb    = neighbors + list_at(0, ld, ia) + u;
    const int nmax   = __reduce_max_sync(0xffffffffu, n);
    double epot      = 0.0;
    double sx = 0.0, sy = 0.0, sz = 0.0; // full lists: sx of threads 0, 1, 2 = x, y, z
    // positions of the next tile and entries of the one after it are in flight
    auto entry = [&](int k) {
        return k < n ? __ldcs(nb + (size_t)(k / MDB_TILE) * ld * MDB_TILE) : -1;
    };
    int j      = entry(0), j1 = entry(MDB_TILE);
    double4 xn = ldg4(x + max(j, 0));
    for (int k = 0; k < nmax; k += MDB_TILE) {
        double tx = 0.0, ty = 0.0, tz = 0.0;
        const double4 xj = xn;
        xn               = ldg4(x + max(j1, 0));
        const int j2     = entry(k + 2 * MDB_TILE);
        if (j >= 0) {
            double delx = xi.x - xj.x;
            double dely = xi.y - xj.y;
            double delz = xi.z - xj.z;
            double rsq  = delx * delx + dely * dely + delz * delz;
            if (rsq < cutforcesq) {
                const int tij        = UNIFORM ? 0 : ti * nt + type_of(xj);
                const double sigma6  = UNIFORM ? tab.sig6[0] : s_sig6[tij];
                const double epsilon = UNIFORM ? tab.eps[0] : s_eps[tij];
                double sr2   = 1.0 / rsq;
                double sr6   = sr2 * sr2 * sr2 * sigma6;
                double force = 48.0 * sr6 * (sr6 - 0.5) * sr2 * epsilon;
                tx = delx * force;
                ty = dely * force;
                tz = delz * force;
                if (HALF && j < nlocal) {
                    atomicAdd(&fx[j], -tx);
                    atomicAdd(&fy[j], -ty);
                    atomicAdd(&fz[j], -tz);
                }
                if (ENERGY) {
                    double e = 4.0 * epsilon * sr6 * (sr6 - 1.0);
                    epot += (HALF && j < nlocal) ? e : 0.5 * e;
                }
            }
        }
        if (HALF) {
            sx += tx;
            sy += ty;
            sz += tz;
        } else {
            s_term[g][0][u] = tx;
            s_term[g][1][u] = ty;
            s_term[g][2][u] = tz;
            __syncwarp();
            if (u < 3) {
#pragma unroll
                for (int q = 0; q < MDB_TILE; q++)
                    sx += s_term[g][u][q];
            }
            __syncwarp();
        }
        j  = j1;
        j1 = j2;
    }
    if (HALF) {
#pragma unroll
        for (int o = MDB_TILE / 2; o > 0; o >>= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sy += __shfl_xor_sync(0xffffffffu, sy, o);
            sz += __shfl_xor_sync(0xffffffffu, sz, o);
        }
        if (i < nlocal && u < 3)
            atomicAdd(u == 0 ? &fx[i] : u == 1 ? &fy[i] : &fz[i], u == 0 ? sx : u == 1 ? sy : sz);
    } else if (i < nlocal && u < 3) {
        (u == 0 ? fx : u == 1 ? fy : fz)[i] = sx;
    }
    if (ENERGY) {
        double e = block_sum(epot);
        if (threadIdx.x == 0) epart[blockIdx.x] = e;
    }
}

template <bool HALF, bool UNIFORM, bool ENERGY, bool COMP>
__global__ void __launch_bounds__(LJ_THREADS) k_lj_mixed(int nlocal, const float4* __restrict__ xr, CellShift sh,
    const int* __restrict__ numneigh, const int* __restrict__ neighbors, int ld,
    float cutforcesq, LJTableF tab, double* __restrict__ fx, double* __restrict__ fy,
    double* __restrict__ fz, double* __restrict__ epart)
{
    __shared__ float s_eps[MDB_MAX_TYPES * MDB_MAX_TYPES];
    __shared__ float s_sig6[MDB_MAX_TYPES * MDB_MAX_TYPES];
    const int nt = tab.ntypes;
    if (!UNIFORM) {
        for (int k = threadIdx.x; k < nt * nt; k += blockDim.x) {
            s_eps[k]  = tab.eps[k];
            s_sig6[k] = tab.sig6[k];
        }
        __syncthreads();
    }
    const float cg = sh.g;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double epot = 0.0;
    if (t < nlocal) {
        const int i     = t;
        const float4 pi = xr[i];
        const int ti    = __float_as_int(pi.w);
        const int n     = numneigh[i];
        const int* nb   = neighbors + list_at(0, ld, i);
        float fix = 0.f, fiy = 0.f, fiz = 0.f;
        float cx = 0.f, cy = 0.f, cz = 0.f; // compensation terms
        const float eps0 = tab.eps[0], sig0 = tab.sig6[0];
        // one type: force / r = sr2 s (A s - B), s = 1 / r^6, A = 48 eps sigma^12,
        // B = 24 eps sigma^6
        const float cA = 48.0f * eps0 * sig0 * sig0, cB = 24.0f * eps0 * sig0;

        auto acc = [&](float& s, float& c, float d, float f) {
            if (COMP) { // Knuth two-sum: s + c carries the running sum exactly
                float v  = d * f;
                float u  = s + v;
                float bp = u - s;
                float e  = (s - (u - bp)) + (v - bp);
                s        = u;
                c += e;
            } else {
                s = __fmaf_rn(d, f, s);
            }
        };

        auto pair = [&](int e, const float4& pj) {
            const int j = entry_index(e);
            float delx, dely, delz;
            cell_delta(pi, pj, e, cg, delx, dely, delz);
            float rsq = __fmaf_rn(delx, delx, __fmaf_rn(dely, dely, delz * delz));
            float sigma6 = sig0, epsilon = eps0;
            if (!UNIFORM) {
                int tij = ti * nt + __float_as_int(pj.w);
                sigma6  = s_sig6[tij];
                epsilon = s_eps[tij];
            }
            if (rsq < cutforcesq) {
                float sr2 = __fdividef(1.0f, rsq);
                float sr6, force;
                if (UNIFORM) {
                    const float s3 = sr2 * sr2 * sr2;
                    sr6            = s3 * sigma6;
                    force          = sr2 * s3 * __fmaf_rn(cA, s3, -cB);
                } else {
                    sr6   = sr2 * sr2 * sr2 * sigma6;
                    force = 48.0f * sr6 * (sr6 - 0.5f) * sr2 * epsilon;
                }
                acc(fix, cx, delx, force);
                acc(fiy, cy, dely, force);
                acc(fiz, cz, delz, force);
                if (HALF && j < nlocal) {
                    atomicAdd(&fx[j], -(double)(delx * force));
                    atomicAdd(&fy[j], -(double)(dely * force));
                    atomicAdd(&fz[j], -(double)(delz * force));
                }
                if (ENERGY) {
                    double en = (double)(4.0f * epsilon * sr6 * (sr6 - 1.0f));
                    epot += (HALF && j < nlocal) ? en : 0.5 * en;
                }
            }
        };

        double rx = 0.0, ry = 0.0, rz = 0.0;
        int en[MDB_TILE]; // the next tile is in flight while one is worked on
        if (n > 0) ld_tile(nb, en);
        if (UNIFORM && !HALF && !COMP) {
            // One type, full lists: two entries per packed instruction and no
            // branch; a pair outside the cutoff adds an exact zero (the same
            // forces with and without the energy). Even and odd
            // entries of a tile sum apart in FP32, the tiles in FP64 (6 instructions
            // in 8 pairs; a row's sum then rounds less than pair by pair in FP32).
            // 168 -> 126 us per launch at 1M atoms (155 with tiles alone, 132 with
            // the next tile not loaded ahead): half the instructions per pair,
            // the gathers' latency and L1 bound it.
            using namespace cp;
            const f2 G0 = f2_pack(-cg, -cg), G1 = f2_pack(-0.25f * cg, -0.25f * cg),
                     G2 = f2_pack(-0.0625f * cg, -0.0625f * cg);
            const f2 B0 = f2_pack(CELL_BIAS(0), CELL_BIAS(0)),
                     B1 = f2_pack(CELL_BIAS(1), CELL_BIAS(1)),
                     B2 = f2_pack(CELL_BIAS(2), CELL_BIAS(2));
            const f2 A2 = f2_pack(cA, cA), mB2 = f2_pack(-cB, -cB);
            for (int k = 0; k < n; k += MDB_TILE) {
                int e[MDB_TILE];
                float4 pj[MDB_TILE];
#pragma unroll
                for (int u = 0; u < MDB_TILE; u++)
                    e[u] = en[u];
                nb += (size_t)ld * MDB_TILE;
                if (k + MDB_TILE < n) ld_tile(nb, en);
#pragma unroll
                for (int u = 0; u < MDB_TILE; u++)
                    pj[u] = __ldg(xr + entry_index(e[u]));
                f2 tx = 0, ty = 0, tz = 0;
#pragma unroll
                for (int u = 0; u < MDB_TILE; u += 2) {
                    const float4 &a = pj[u], &b = pj[u + 1];
                    const f2 dx = f2_fma(
                        f2_sub(f2_pack(cell_field(e[u], 0), cell_field(e[u + 1], 0)), B0), G0,
                        f2_pack(pi.x - a.x, pi.x - b.x));
                    const f2 dy = f2_fma(
                        f2_sub(f2_pack(cell_field(e[u], 1), cell_field(e[u + 1], 1)), B1), G1,
                        f2_pack(pi.y - a.y, pi.y - b.y));
                    const f2 dz = f2_fma(
                        f2_sub(f2_pack(cell_field(e[u], 2), cell_field(e[u + 1], 2)), B2), G2,
                        f2_pack(pi.z - a.z, pi.z - b.z));
                    const f2 rsq = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
                    float r0, r1;
                    f2_unpack(rsq, r0, r1);
                    const float u0 = rcp_approx(r0), u1 = rcp_approx(r1);
                    const f2 U  = f2_pack(r0 < cutforcesq ? u0 : 0.0f, r1 < cutforcesq ? u1 : 0.0f);
                    const f2 U2 = f2_mul(U, U);
                    const f2 U3 = f2_mul(U2, U);
                    const f2 F  = f2_mul(f2_mul(U2, U2), f2_fma(A2, U3, mB2));
                    if (ENERGY) {
                        float s0, s1;
                        f2_unpack(f2_mul(U3, f2_pack(sig0, sig0)), s0, s1);
                        epot += 0.5 * (double)(4.0f * eps0 * s0 * (s0 - 1.0f));
                        epot += 0.5 * (double)(4.0f * eps0 * s1 * (s1 - 1.0f));
                    }
                    tx = u ? f2_fma(dx, F, tx) : f2_mul(dx, F);
                    ty = u ? f2_fma(dy, F, ty) : f2_mul(dy, F);
                    tz = u ? f2_fma(dz, F, tz) : f2_mul(dz, F);
                }
                float t0, t1;
                f2_unpack(tx, t0, t1);
                rx += (double)(t0 + t1);
                f2_unpack(ty, t0, t1);
                ry += (double)(t0 + t1);
                f2_unpack(tz, t0, t1);
                rz += (double)(t0 + t1);
            }
        } else {
            for (int k = 0; k < n; k += MDB_TILE) {
                int e[MDB_TILE];
                float4 pj[MDB_TILE];
#pragma unroll
                for (int u = 0; u < MDB_TILE; u++)
                    e[u] = en[u];
                nb += (size_t)ld * MDB_TILE;
                if (k + MDB_TILE < n) ld_tile(nb, en);
#pragma unroll
                for (int u = 0; u < MDB_TILE; u++)
                    pj[u] = __ldg(xr + entry_index(e[u]));
#pragma unroll
                for (int u = 0; u < MDB_TILE; u++)
                    pair(e[u], pj[u]);
            }
        }
        rx += (double)fix + (double)cx;
        ry += (double)fiy + (double)cy;
        rz += (double)fiz + (double)cz;
        if (HALF) {
            atomicAdd(&fx[i], rx);
            atomicAdd(&fy[i], ry);
            atomicAdd(&fz[i], rz);
        } else {
            fx[i] = rx;
            fy[i] = ry;
            fz[i] = rz;
        }
    }
    if (ENERGY) {
        double e = block_sum(epot);
        if (threadIdx.x == 0) epart[blockIdx.x] = e;
    }
}

template <bool HALF, bool UNIFORM, bool ENERGY>
static void lj64(cudaStream_t s, int nlocal, const double4* x, const int* numneigh,
    const int* neighbors, int ld, double cut, const LJTable& tab, double* fx, double* fy,
    double* fz, double* epart)
{
    const int nb = lj_fp64_blocks(HALF, nlocal);
    if (lj_fp64_shared(HALF, nlocal))
        k_lj_fp64_shared<HALF, UNIFORM, ENERGY><<<nb, LJ_THREADS, 0, s>>>(nlocal, x, numneigh,
            neighbors, ld, cut, tab, fx, fy, fz, epart);
    else
        k_lj_fp64<UNIFORM, ENERGY><<<nb, LJ_THREADS, 0, s>>>(nlocal, x, numneigh, neighbors, ld,
            cut, tab, fx, fy, fz, epart);
}

template <bool HALF, bool UNIFORM>
static void lj64_e(cudaStream_t s, int energy, int nlocal, const double4* x, const int* numneigh,
    const int* neighbors, int ld, double cut, const LJTable& tab, double* fx, double* fy,
    double* fz, double* epart)
{
    if (energy)
        lj64<HALF, UNIFORM, true>(s, nlocal, x, numneigh, neighbors, ld, cut, tab, fx, fy, fz,
            epart);
    else
        lj64<HALF, UNIFORM, false>(s, nlocal, x, numneigh, neighbors, ld, cut, tab, fx, fy, fz,
            epart);
}

void launch_lj_fp64(cudaStream_t s, int half, int energy, int nlocal,
    const double4* x, const int* numneigh, const int* neighbors, int ld, double cutforcesq,
    const LJTable& tab, double* fx, double* fy, double* fz, double* epart)
{
    if (nlocal <= 0) return;
#define LJ64(H, U)                                                                       \
    lj64_e<H, U>(s, energy, nlocal, x, numneigh, neighbors, ld, cutforcesq, tab, fx, fy, fz, epart)
    if (half) tab.uniform ? LJ64(true, true) : LJ64(true, false);
    else tab.uniform ? LJ64(false, true) : LJ64(false, false);
#undef LJ64
    g_launches++;
}

template <bool HALF, bool UNIFORM, bool COMP>
static void ljmx(cudaStream_t s, int energy, int nb, int nlocal,
    const float4* xr, const CellShift& sh, const int* numneigh, const int* neighbors, int ld,
    float cut, const LJTableF& tab, double* fx, double* fy, double* fz, double* epart)
{
    if (energy)
        k_lj_mixed<HALF, UNIFORM, true, COMP><<<nb, LJ_THREADS, 0, s>>>(nlocal, xr, sh,
            numneigh, neighbors, ld, cut, tab, fx, fy, fz, epart);
    else
        k_lj_mixed<HALF, UNIFORM, false, COMP><<<nb, LJ_THREADS, 0, s>>>(nlocal, xr, sh,
            numneigh, neighbors, ld, cut, tab, fx, fy, fz, epart);
}

template <bool HALF, bool COMP>
static void ljmx_u(cudaStream_t s, int energy, int nb, int nlocal,
    const float4* xr, const CellShift& sh, const int* numneigh, const int* neighbors, int ld,
    float cut, const LJTableF& tab, double* fx, double* fy, double* fz, double* epart)
{
    if (tab.uniform)
        ljmx<HALF, true, COMP>(s, energy, nb, nlocal, xr, sh, numneigh, neighbors, ld,
            cut, tab, fx, fy, fz, epart);
    else
        ljmx<HALF, false, COMP>(s, energy, nb, nlocal, xr, sh, numneigh, neighbors, ld,
            cut, tab, fx, fy, fz, epart);
}

void launch_lj_mixed(cudaStream_t s, int comp, int half, int energy, int nlocal,
    const float4* xr, const CellShift& sh, const int* numneigh,
    const int* neighbors, int ld, float cutforcesq, const LJTableF& tab, double* fx,
    double* fy, double* fz, double* epart)
{
    if (nlocal <= 0) return;
    int nb = force_partial_blocks(nlocal);
    if (half) {
        if (comp)
            ljmx_u<true, true>(s, energy, nb, nlocal, xr, sh, numneigh, neighbors, ld,
                cutforcesq, tab, fx, fy, fz, epart);
        else
            ljmx_u<true, false>(s, energy, nb, nlocal, xr, sh, numneigh, neighbors, ld,
                cutforcesq, tab, fx, fy, fz, epart);
    } else {
        if (comp)
            ljmx_u<false, true>(s, energy, nb, nlocal, xr, sh, numneigh, neighbors, ld,
                cutforcesq, tab, fx, fy, fz, epart);
        else
            ljmx_u<false, false>(s, energy, nb, nlocal, xr, sh, numneigh, neighbors, ld,
                cutforcesq, tab, fx, fy, fz, epart);
    }
    g_launches++;
}

} // namespace mdb
