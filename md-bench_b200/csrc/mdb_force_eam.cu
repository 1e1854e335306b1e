// EAM forces over Verlet lists (computeForceEam, verletlist/force_eam.c:19-228)
// as two kernels: (1) density rho_i and fp_i = F'(rho_i) per local atom, written
// for its ghosts too (the mid-step halo, verletlist/force_eam.c:120-130: atom i's
// ghosts are ghost_off[i] .. ghost_off[i + 1]; a kernel of its own took 1.7 us
// and the time around it, of 28 us per step at 3,960 atoms), (2) pair forces from
// rho', phi' and fp_i + fp_j.
//
// Thread t handles atom t. Spline tables are re-laid out as rows of 8
// coefficients, 3..6 (the value) then 0..2 (the derivative), so each half is one
// aligned sector in one 256-bit load.
// FP64 path: -fmad=false, bit-identical to the reference's strict build.
// Mixed path: pair terms and spline rows in FP32 on cell-relative FP32
// positions (see mdb_force_lj.cu); the density (embedding) sum, F'(rho) and
// all energy sums in FP64.
#include "mdb_internal.cuh"

namespace mdb {

static constexpr int EAM_THREADS = 128;

// one 32-byte row (two float4) in one 256-bit load (sm_100); p 32-byte aligned
__device__ __forceinline__ void ldg_row32(const float4* p, float4& a, float4& b)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z),
          "=f"(b.w)
        : "l"(p));
}
static constexpr int EUNROLL     = 4;

// FP64 passes: a row's sums must add its pairs one after the other, in list
// order, for bit-identical results, but everything else of a pair is
// independent. So 8 threads share an atom, one entry of a tile each, and leave
// their terms in shared memory, where one thread per sum adds them up in order.
// (One thread per atom spent its time waiting on its own chain of dependent
// square roots, divisions and table rows, at 31 blocks for 4,000 atoms.)
// A pair outside the cutoff adds an exact zero. Both passes: 85 -> 16 us at 3,960
// atoms, 302 -> 211 us at 131,072, where the scattered table rows bound them (one
// 32-byte load per half row; 307 us with eight-byte loads of the coefficients).
static constexpr int EAM64_ATOMS = EAM_THREADS / MDB_TILE; // atoms per block

int eam_fp64_blocks(int nlocal) { return mdb_blocks(nlocal, EAM64_ATOMS); }

template <bool ENERGY>
__global__ void __launch_bounds__(EAM_THREADS) k_eam_rho_fp64(int nlocal,
    const double4* __restrict__ x, const int* __restrict__ numneigh,
    const int* __restrict__ neighbors, int ld, double cutforcesq, EamDev e,
    const int* __restrict__ ghost_off, const int* __restrict__ counters,
    double* __restrict__ fp, double* __restrict__ epart)
{
    __shared__ double s_term[EAM64_ATOMS][MDB_TILE + 1];
    const int g = threadIdx.x / MDB_TILE, u = threadIdx.x % MDB_TILE;
    const int i = blockIdx.x * EAM64_ATOMS + g;
    double eng  = 0.0;
    const int ia     = i < nlocal ? i : 0;
    const double4 xi = x[ia];
    const int n      = i < nlocal ? numneigh[ia] : 0;
    const int* nb    = neighbors + list_at(0, ld, ia) + u;
    const int nmax   = __reduce_max_sync(0xffffffffu, n);
    double rhoi      = 0.0;
    // the next tile's positions and the entries of the one after it are in flight
    // while a tile is worked on
    auto entry = [&](int k) {
        return k < n ? __ldcs(nb + (size_t)(k / MDB_TILE) * ld * MDB_TILE) : -1;
    };
    int j      = entry(0), j1 = entry(MDB_TILE);
    double4 xn = ldg4(x + max(j, 0));
    for (int k = 0; k < nmax; k += MDB_TILE) {
        double term      = 0.0;
        const double4 xj = xn;
        xn               = ldg4(x + max(j1, 0));
        const int j2     = entry(k + 2 * MDB_TILE);
        if (j >= 0) {
            double delx = xi.x - xj.x;
            double dely = xi.y - xj.y;
            double delz = xi.z - xj.z;
            double rsq  = delx * delx + dely * dely + delz * delz;
            if (rsq < cutforcesq) {
                double p = sqrt(rsq) * e.rdr + 1.0;
                int m    = (int)(p);
                m        = m < e.nr - 1 ? m : e.nr - 1;
                p -= m;
                p               = p < 1.0 ? p : 1.0;
                const double4 c = ldg4(e.rhor + 2 * m);
                term            = ((c.x * p + c.y) * p + c.z) * p + c.w;
            }
        }
        s_term[g][u] = term;
        __syncwarp();
        if (u == 0) {
#pragma unroll
            for (int q = 0; q < MDB_TILE; q++)
                rhoi += s_term[g][q];
        }
        __syncwarp();
        j  = j1;
        j1 = j2;
    }
    double fpi = 0.0;
    if (u == 0 && i < nlocal) {
        double p = 1.0 * rhoi * e.rdrho + 1.0;
        int m    = (int)(p);
        m        = m < e.nrho - 1 ? m : e.nrho - 1;
        m        = m > 1 ? m : 1;
        p -= m;
        p               = p < 1.0 ? p : 1.0;
        const double4 c = ldg4(e.frho + 2 * m), d = ldg4(e.frho + 2 * m + 1);
        fpi             = (d.x * p + d.y) * p + d.z;
        fp[i]           = fpi;
        if (ENERGY) eng = ((c.x * p + c.y) * p + c.z) * p + c.w;
    }
    fpi = __shfl_sync(0xffffffffu, fpi, 0, MDB_TILE);
    if (i < nlocal) {
        const int gend = min(ghost_off[i + 1], counters[CNT_NGHOST]);
        for (int g = ghost_off[i] + u; g < gend; g += MDB_TILE)
            fp[nlocal + g] = fpi;
    }
    if (ENERGY) {
        double s = block_sum(eng);
        if (threadIdx.x == 0) epart[blockIdx.x] = s;
    }
}

template <bool ENERGY>
__global__ void __launch_bounds__(EAM_THREADS) k_eam_force_fp64(int nlocal,
    const double4* __restrict__ x, const int* __restrict__ numneigh,
    const int* __restrict__ neighbors, int ld, double cutforcesq, EamDev e,
    const double* __restrict__ fp, double* __restrict__ fx, double* __restrict__ fy,
    double* __restrict__ fz, double* __restrict__ epart)
{
    __shared__ double s_term[EAM64_ATOMS][3][MDB_TILE + 1];
    const int g = threadIdx.x / MDB_TILE, u = threadIdx.x % MDB_TILE;
    const int i = blockIdx.x * EAM64_ATOMS + g;
    double eng  = 0.0;
    const int ia     = i < nlocal ? i : 0;
    const double4 xi = x[ia];
    const int n      = i < nlocal ? numneigh[ia] : 0;
    const int* nb    = neighbors + list_at(0, ld, ia) + u;
    const int nmax   = __reduce_max_sync(0xffffffffu, n);
    const double fpi = fp[ia];
    double sum       = 0.0; // threads 0, 1, 2: the x, y, z force
    auto entry       = [&](int k) {
        return k < n ? __ldcs(nb + (size_t)(k / MDB_TILE) * ld * MDB_TILE) : -1;
    };
    int j      = entry(0), j1 = entry(MDB_TILE);
    double4 xn = ldg4(x + max(j, 0));
    double fpn = __ldg(fp + max(j, 0));
    for (int k = 0; k < nmax; k += MDB_TILE) {
        double tx = 0.0, ty = 0.0, tz = 0.0;
        const double4 xj = xn;
        const double fpj = fpn;
        xn               = ldg4(x + max(j1, 0));
        fpn              = __ldg(fp + max(j1, 0));
        const int j2     = entry(k + 2 * MDB_TILE);
        if (j >= 0) {
            double delx = xi.x - xj.x;
            double dely = xi.y - xj.y;
            double delz = xi.z - xj.z;
            double rsq  = delx * delx + dely * dely + delz * delz;
            if (rsq < cutforcesq) {
                double r = sqrt(rsq);
                double p = r * e.rdr + 1.0;
                int m    = (int)(p);
                m        = m < e.nr - 1 ? m : e.nr - 1;
                p -= m;
                p                = p < 1.0 ? p : 1.0;
                const double4 cr = ldg4(e.rhor + 2 * m + 1);
                const double4 cz = ldg4(e.z2r + 2 * m), cd = ldg4(e.z2r + 2 * m + 1);
                double rhoip     = (cr.x * p + cr.y) * p + cr.z;
                double z2p       = (cd.x * p + cd.y) * p + cd.z;
                double z2        = ((cz.x * p + cz.y) * p + cz.z) * p + cz.w;
                double recip = 1.0 / r;
                double phi   = z2 * recip;
                double phip  = z2p * recip - phi * recip;
                double psip  = fpi * rhoip + fpj * rhoip + phip;
                double fpair = -psip * recip;
                tx = delx * fpair;
                ty = dely * fpair;
                tz = delz * fpair;
                if (ENERGY) eng += 0.5 * phi;
            }
        }
        s_term[g][0][u] = tx;
        s_term[g][1][u] = ty;
        s_term[g][2][u] = tz;
        __syncwarp();
        if (u < 3) {
#pragma unroll
            for (int q = 0; q < MDB_TILE; q++)
                sum += s_term[g][u][q];
        }
        __syncwarp();
        j  = j1;
        j1 = j2;
    }
    if (i < nlocal && u < 3) (u == 0 ? fx : u == 1 ? fy : fz)[i] = sum;
    if (ENERGY) {
        double s = block_sum(eng);
        if (threadIdx.x == 0) epart[blockIdx.x] = s;
    }
}

// ---- mixed ------------------------------------------------------------------
// Thread t handles atom t. The density pass also writes, per atom, the list
// entries inside the cutoff in list order (cut, laid out like the list, and
// their count ncut), and xe = (position, F'(rho)) of the atom and its ghosts. The
// force pass then runs over the in-cutoff
// entries only and gathers a neighbour's position and F'(rho_j) in one
// 16-byte load: the same pairs in the same order as a pass over the whole list
// that skips the rest, without the skin entries (about 40 % of a list at
// r_c + 1 A) and without a cutoff branch that diverges inside a warp. The two
// passes compute rsq from the same FP32 values with the same operations, so
// every entry of cut is inside the cutoff in the force pass too.
// F'(rho_i) and position for atom i (p: its position) and its ghosts
__device__ __forceinline__ void put_fp(int i, int nlocal, double fpi, const float4& p,
    const float4* __restrict__ xr, const int* __restrict__ ghost_off,
    const int* __restrict__ counters, double* __restrict__ fp, float4* __restrict__ xe)
{
    fp[i]          = fpi;
    xe[i]          = make_float4(p.x, p.y, p.z, (float)fpi);
    const int gend = min(ghost_off[i + 1], counters[CNT_NGHOST]);
    for (int g = ghost_off[i]; g < gend; g++) {
        const float4 q = xr[nlocal + g];
        fp[nlocal + g] = fpi;
        xe[nlocal + g] = make_float4(q.x, q.y, q.z, (float)fpi);
    }
}

int eam_mixed_blocks(int nlocal) { return mdb_blocks(nlocal, EAM_THREADS); }

template <bool ENERGY>
__global__ void __launch_bounds__(EAM_THREADS) k_eam_rho_mixed(int nlocal,
    const float4* __restrict__ xr, CellShift sh, const int* __restrict__ numneigh,
    const int* __restrict__ neighbors, int ld, float cutforcesq, EamDev e,
    const int* __restrict__ ghost_off, const int* __restrict__ counters,
    int* __restrict__ cut, int* __restrict__ ncut, double* __restrict__ fp,
    float4* __restrict__ xe, double* __restrict__ epart)
{
    const float cg = sh.g;
    const int i    = blockIdx.x * blockDim.x + threadIdx.x;
    double eng     = 0.0;
    if (i < nlocal) {
        const float4 pi = xr[i];
        const int n     = numneigh[i];
        const int* nb   = neighbors + list_at(0, ld, i);
        int* out        = cut + i;
        int c           = 0;
        double rhoi     = 0.0; // FP64 embedding (density) sum
        const float rdr = (float)e.rdr;
        auto pair       = [&](int en, const float4& pj) {
            float dx, dy, dz;
            cell_delta(pi, pj, en, cg, dx, dy, dz);
            float rsq = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
            if (rsq < cutforcesq) {
                float p = __fmaf_rn(sqrtf(rsq), rdr, 1.0f);
                int m   = (int)p;
                m       = m < e.nr - 1 ? m : e.nr - 1;
                p -= (float)m;
                p              = p < 1.0f ? p : 1.0f;
                const float4 a = __ldg(e.dens32 + m); // coefficients 3..6
                rhoi += (double)__fmaf_rn(__fmaf_rn(__fmaf_rn(a.x, p, a.y), p, a.z), p, a.w);
                __stcg(out + (size_t)c * ld, en);
                c++;
            }
        };
        int nx[MDB_TILE]; // the next tile is in flight while one is worked on
        if (n > 0) ld_tile(nb, nx);
        for (int k = 0; k < n; k += MDB_TILE) {
            int en[MDB_TILE];
            float4 pj[MDB_TILE];
#pragma unroll
            for (int v = 0; v < MDB_TILE; v++)
                en[v] = nx[v];
            nb += (size_t)ld * MDB_TILE;
            if (k + MDB_TILE < n) ld_tile(nb, nx);
#pragma unroll
            for (int v = 0; v < MDB_TILE; v++)
                pj[v] = __ldg(xr + entry_index(en[v]));
#pragma unroll
            for (int v = 0; v < MDB_TILE; v++)
                pair(en[v], pj[v]);
        }
        ncut[i]   = c;
        double p = 1.0 * rhoi * e.rdrho + 1.0;
        int m    = (int)(p);
        m        = m < e.nrho - 1 ? m : e.nrho - 1;
        m        = m > 1 ? m : 1;
        p -= m;
        p                = p < 1.0 ? p : 1.0;
        const double4 cf = ldg4(e.frho + 2 * m), df = ldg4(e.frho + 2 * m + 1);
        const double fpi = (df.x * p + df.y) * p + df.z;
        put_fp(i, nlocal, fpi, pi, xr, ghost_off, counters, fp, xe);
        if (ENERGY) eng = ((cf.x * p + cf.y) * p + cf.z) * p + cf.w;
    }
    if (ENERGY) {
        double s = block_sum(eng);
        if (threadIdx.x == 0) epart[blockIdx.x] = s;
    }
}

// The density pass with two lanes per atom (lanes 2q and 2q + 1 of a warp on
// atom 16 w + q): the lanes take list entries k and k + 1 of each pair and
// append the in-cutoff ones to cut in list order (the lower lane's first), so
// the force pass reads the same rows as after the one-lane pass; the two FP64
// partial densities are added at the end. Twice the warps of the one-lane pass
// keep more gathers in flight on a 131k-atom system. Blocks of 2 x EAM_THREADS
// threads cover the same EAM_THREADS atoms as a block of the one-lane pass, so
// both write the same energy partials.
template <bool ENERGY>
__global__ void __launch_bounds__(2 * EAM_THREADS) k_eam_rho_mixed2(int nlocal,
    const float4* __restrict__ xr, CellShift sh, const int* __restrict__ numneigh,
    const int* __restrict__ neighbors, int ld, float cutforcesq, EamDev e,
    const int* __restrict__ ghost_off, const int* __restrict__ counters,
    int* __restrict__ cut, int* __restrict__ ncut, double* __restrict__ fp,
    float4* __restrict__ xe, double* __restrict__ epart)
{
    const float cg  = sh.g;
    const int lane  = threadIdx.x & 31;
    const int u     = lane & 1;
    const int i     = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 16 + (lane >> 1);
    const bool act  = i < nlocal;
    const int ia    = act ? i : 0;
    const float4 pi = act ? xr[ia] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int n     = act ? numneigh[ia] : 0;
    int* out        = cut + ia;
    int c           = 0;     // entries appended so far (both lanes)
    double rhoi     = 0.0;   // this lane's FP64 partial density
    double eng      = 0.0;
    const float rdr = (float)e.rdr;
    const unsigned pairmask = 3u << (lane & ~1);
    auto pair = [&](int en, const float4& pj, bool valid) {
        bool in = false;
        if (valid) {
            float dx, dy, dz;
            cell_delta(pi, pj, en, cg, dx, dy, dz);
            const float rsq = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
            in              = rsq < cutforcesq;
            if (in) {
                float p = __fmaf_rn(sqrtf(rsq), rdr, 1.0f);
                int m   = (int)p;
                m       = m < e.nr - 1 ? m : e.nr - 1;
                p -= (float)m;
                p              = p < 1.0f ? p : 1.0f;
                const float4 a = __ldg(e.dens32 + m); // coefficients 3..6
                rhoi += (double)__fmaf_rn(__fmaf_rn(__fmaf_rn(a.x, p, a.y), p, a.z), p, a.w);
            }
        }
        const unsigned bal = __ballot_sync(0xffffffffu, in) & pairmask;
        if (in) __stcg(out + (size_t)(c + (u ? __popc(bal) - 1 : 0)) * ld, en);
        c += __popc(bal);
    };
    // a warp runs as many pair steps as its longest row
    int nmax = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nmax = max(nmax, __shfl_xor_sync(0xffffffffu, nmax, o));
    int k = 0;
    for (; k + 2 * EUNROLL <= nmax; k += 2 * EUNROLL) {
        int en[EUNROLL];
        float4 pj[EUNROLL];
#pragma unroll
        for (int v = 0; v < EUNROLL; v++) {
            const int kk = k + 2 * v + u;
            en[v]        = kk < n ? __ldcs(neighbors + list_at(kk, ld, ia)) : 0;
        }
#pragma unroll
        for (int v = 0; v < EUNROLL; v++)
            pj[v] = k + 2 * v + u < n ? __ldg(xr + entry_index(en[v])) : pi;
#pragma unroll
        for (int v = 0; v < EUNROLL; v++)
            pair(en[v], pj[v], k + 2 * v + u < n);
    }
    for (; k < nmax; k += 2) {
        const bool valid = k + u < n;
        const int en     = valid ? __ldcs(neighbors + list_at(k + u, ld, ia)) : 0;
        pair(en, valid ? __ldg(xr + entry_index(en)) : pi, valid);
    }
    rhoi += __shfl_xor_sync(0xffffffffu, rhoi, 1);
    if (act && u == 0) {
        ncut[i]  = c;
        double p = 1.0 * rhoi * e.rdrho + 1.0;
        int m    = (int)(p);
        m        = m < e.nrho - 1 ? m : e.nrho - 1;
        m        = m > 1 ? m : 1;
        p -= m;
        p                = p < 1.0 ? p : 1.0;
        const double4 cf = ldg4(e.frho + 2 * m), df = ldg4(e.frho + 2 * m + 1);
        const double fpi = (df.x * p + df.y) * p + df.z;
        put_fp(i, nlocal, fpi, pi, xr, ghost_off, counters, fp, xe);
        if (ENERGY) eng = ((cf.x * p + cf.y) * p + cf.z) * p + cf.w;
    }
    if (ENERGY) {
        double s = block_sum(eng);
        if (threadIdx.x == 0) epart[blockIdx.x] = s;
    }
}

// COMP: Knuth two-sum compensated force sums (MDB_PREC_MIXED_COMP)
template <bool ENERGY, bool COMP>
__global__ void __launch_bounds__(EAM_THREADS) k_eam_force_mixed(int nlocal,
    const float4* __restrict__ xe, CellShift sh, const int* __restrict__ ncut,
    const int* __restrict__ cut, int ld, EamDev e, double* __restrict__ fx,
    double* __restrict__ fy, double* __restrict__ fz, double* __restrict__ epart)
{
    const float cg = sh.g;
    const int i    = blockIdx.x * blockDim.x + threadIdx.x;
    double eng     = 0.0;
    if (i < nlocal) {
        const float4 pi = xe[i];
        const int n     = ncut[i];
        const int* nb   = cut + i;
        const float fpi = pi.w;
        const float rdr = (float)e.rdr;
        const float rdr2 = 2.0f * rdr;
        float fix = 0.f, fiy = 0.f, fiz = 0.f;
        float cx = 0.f, cy = 0.f, cz = 0.f; // compensation terms
        auto acc = [&](float& s, float& c, float d, float f) {
            if (COMP) { // s + c carries the running sum exactly
                float v  = d * f;
                float w  = s + v;
                float bp = w - s;
                float r  = (s - (w - bp)) + (v - bp);
                s        = w;
                c += r;
            } else {
                s = __fmaf_rn(d, f, s);
            }
        };
        auto pair = [&](int en, const float4& pj) {
            float dx, dy, dz;
            cell_delta(pi, pj, en, cg, dx, dy, dz);
            const float rsq = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
            const float r   = sqrtf(rsq);
            float p         = __fmaf_rn(r, rdr, 1.0f);
            int m           = (int)p;
            m               = m < e.nr - 1 ? m : e.nr - 1;
            p -= (float)m;
            p               = p < 1.0f ? p : 1.0f;
            // z2r coefficients 3..6, then rho 0..2 and z2r 0; z2r 1 and 2 are
            // 2 c4 / dr and c5 / dr (spline7's derivative rows)
            float4 za, rb;
            ldg_row32(e.pair32 + 2 * m, za, rb);
            float rhoip = __fmaf_rn(__fmaf_rn(rb.x, p, rb.y), p, rb.z);
            float z2p   = __fmaf_rn(__fmaf_rn(rb.w, p, za.y * rdr2), p, za.z * rdr);
            float z2    = __fmaf_rn(__fmaf_rn(__fmaf_rn(za.x, p, za.y), p, za.z), p, za.w);
            float recip = __fdividef(1.0f, r);
            float phi   = z2 * recip;
            float phip  = __fmaf_rn(z2p, recip, -phi * recip);
            float psip  = __fmaf_rn(fpi + pj.w, rhoip, phip);
            float fpair = -psip * recip;
            acc(fix, cx, dx, fpair);
            acc(fiy, cy, dy, fpair);
            acc(fiz, cz, dz, fpair);
            if (ENERGY) eng += 0.5 * (double)phi;
        };
        int k = 0;
        int nx[EUNROLL]; // the next entries are in flight while four are worked on
#pragma unroll
        for (int v = 0; v < EUNROLL; v++)
            nx[v] = v < n ? __ldcs(nb + (size_t)v * ld) : 0;
        for (; k + EUNROLL <= n; k += EUNROLL) {
            int en[EUNROLL];
            float4 pj[EUNROLL];
#pragma unroll
            for (int v = 0; v < EUNROLL; v++) {
                en[v]      = nx[v];
                const int q = k + EUNROLL + v;
                if (q < n) nx[v] = __ldcs(nb + (size_t)q * ld);
            }
#pragma unroll
            for (int v = 0; v < EUNROLL; v++)
                pj[v] = __ldg(xe + entry_index(en[v]));
#pragma unroll
            for (int v = 0; v < EUNROLL; v++)
                pair(en[v], pj[v]);
        }
#pragma unroll
        for (int v = 0; v < EUNROLL; v++)
            if (k + v < n) pair(nx[v], __ldg(xe + entry_index(nx[v])));
        fx[i] = (double)fix + (double)cx;
        fy[i] = (double)fiy + (double)cy;
        fz[i] = (double)fiz + (double)cz;
    }
    if (ENERGY) {
        double s = block_sum(eng);
        if (threadIdx.x == 0) epart[blockIdx.x] = s;
    }
}

void launch_eam_fp64(cudaStream_t s, int energy, int nlocal,
    const double4* x, const int* numneigh, const int* neighbors, int ld, double cutforcesq,
    EamDev eam, const int* ghost_off, const int* counters, double* fp, double* fx,
    double* fy, double* fz, double* epart_rho, double* epart_pair)
{
    if (nlocal <= 0) return;
    const int nb = eam_fp64_blocks(nlocal);
    if (energy)
        k_eam_rho_fp64<true><<<nb, EAM_THREADS, 0, s>>>(nlocal, x, numneigh, neighbors,
            ld, cutforcesq, eam, ghost_off, counters, fp, epart_rho);
    else
        k_eam_rho_fp64<false><<<nb, EAM_THREADS, 0, s>>>(nlocal, x, numneigh, neighbors,
            ld, cutforcesq, eam, ghost_off, counters, fp, epart_rho);
    g_launches++;
    if (energy)
        k_eam_force_fp64<true><<<nb, EAM_THREADS, 0, s>>>(nlocal, x, numneigh,
            neighbors, ld, cutforcesq, eam, fp, fx, fy, fz, epart_pair);
    else
        k_eam_force_fp64<false><<<nb, EAM_THREADS, 0, s>>>(nlocal, x, numneigh,
            neighbors, ld, cutforcesq, eam, fp, fx, fy, fz, epart_pair);
    g_launches++;
}

int launch_eam_mixed(cudaStream_t s, int energy, int comp, int rho_lanes, int nlocal,
    const float4* xr, const CellShift& sh, const int* numneigh, const int* neighbors, int ld,
    float cutforcesq, EamDev eam, const int* ghost_off, const int* counters, int* cut,
    int* ncut, double* fp, float4* xe, double* fx, double* fy, double* fz, double* epart_rho,
    double* epart_pair)
{
    if (nlocal <= 0) return 0;
    const int nb = eam_mixed_blocks(nlocal);
    if (rho_lanes == 2) {
        if (energy)
            k_eam_rho_mixed2<true><<<nb, 2 * EAM_THREADS, 0, s>>>(nlocal, xr, sh, numneigh,
                neighbors, ld, cutforcesq, eam, ghost_off, counters, cut, ncut, fp, xe, epart_rho);
        else
            k_eam_rho_mixed2<false><<<nb, 2 * EAM_THREADS, 0, s>>>(nlocal, xr, sh, numneigh,
                neighbors, ld, cutforcesq, eam, ghost_off, counters, cut, ncut, fp, xe, epart_rho);
    } else if (energy)
        k_eam_rho_mixed<true><<<nb, EAM_THREADS, 0, s>>>(nlocal, xr, sh, numneigh, neighbors,
            ld, cutforcesq, eam, ghost_off, counters, cut, ncut, fp, xe, epart_rho);
    else
        k_eam_rho_mixed<false><<<nb, EAM_THREADS, 0, s>>>(nlocal, xr, sh, numneigh, neighbors,
            ld, cutforcesq, eam, ghost_off, counters, cut, ncut, fp, xe, epart_rho);
    g_launches++;
#define EAM_FM(E, C)                                                                     \
    k_eam_force_mixed<E, C><<<nb, EAM_THREADS, 0, s>>>(nlocal, xe, sh, ncut, cut, ld, eam, fx, \
        fy, fz, epart_pair)
    if (energy) {
        if (comp) EAM_FM(true, true);
        else EAM_FM(true, false);
    } else {
        if (comp) EAM_FM(false, true);
        else EAM_FM(false, false);
    }
#undef EAM_FM
    g_launches++;
    return nb;
}

} // namespace mdb
