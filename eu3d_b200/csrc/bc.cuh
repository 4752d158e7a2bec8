// Ghost-cell fills and the CFL time step.
//
// Reference: Flowfield::FieldBoundary_3dRSBI (src/Flowfield.cpp:559-773),
// FieldBoundary_3dODM (:378-558), Flowfield::CFLcondition (:242-272).
#pragma once

#include "common.cuh"

namespace eu3d {

struct GhostArgs {
    Layout L;
    unsigned quirks;
    double *T, *E;
    const double *inflow;  // ODM planes: U V W P D T H E G, then NS species planes, each nj*nk
    int kind;
};

// Every fill loads all the values it copies before its first store.  The
// destination of a fill is never a source of another thread of the same launch
// (ghost cells take interior cells; the wedge band's solid cells take fluid
// ones), so the order changes nothing but the timing: the compiler, which cannot prove
// that the stores miss the later loads, would otherwise issue each load only
// after the store before it, one memory round trip per field.
template <class P>
__device__ __forceinline__ void ghost_load(const GhostArgs &a, const P *q, long long s, P v[NPRIM], double &T,
                                           double &E)
{
    const long long fs = a.L.fs;
#pragma unroll
    for (int f = 0; f < NPRIM; f++) v[f] = q[f * fs + s];
    T = a.T[s];
    E = a.E[s];
}

template <class P>
__device__ __forceinline__ void ghost_store(const GhostArgs &a, P *q, long long d, const P v[NPRIM], double T,
                                            double E)
{
    const long long fs = a.L.fs;
#pragma unroll
    for (int f = 0; f < NPRIM; f++) q[f * fs + d] = v[f];
    a.T[d] = T;
    a.E[d] = E;
}

// the ODM inflow state of row j, k (interior indices from 0)
template <class P>
__device__ __forceinline__ void ghost_inflow(const GhostArgs &a, int j, int k, P v[NPRIM], double &T, double &E)
{
    const long long p = (long long)k * a.L.nj + j, pl = (long long)a.L.nj * a.L.nk;
    double in[9 + NS];
#pragma unroll
    for (int f = 0; f < 9 + NS; f++) in[f] = a.inflow[f * pl + p];
    v[PU] = (P)in[0];
    v[PV] = (P)in[1];
    v[PW] = (P)in[2];
    v[PP] = (P)in[3];
    v[PD] = (P)in[4];
    T = in[5];
    v[PH] = (P)in[6];
    E = in[7];
    v[PG] = (P)in[8];
#pragma unroll
    for (int s = 0; s < NS; s++) v[PY + s] = (P)in[9 + s];
}

// wall-side thermodynamic recompute of the reflective faces
// (src/Flowfield.cpp:409-436 pattern): D from P/(T Rgas), H, E, Gamma from T
template <class P>
__device__ __forceinline__ void ghost_wall(const GhostArgs &a, P v[NPRIM], double T, double &E)
{
    const TPow p = tpow(T, a.quirks);
    double rg = 0.0, cp = 0.0, h = 0.0, e = 0.0;
#pragma unroll
    for (int sp = 0; sp < NS; sp++) {
        const double Y = (double)v[PY + sp];
        const double cpi = cM.ri[sp] * cp_r(sp, p);
        const double hi = cM.ri[sp] * h_r(sp, p);
        const double ei = hi - cM.ri[sp] * T;
        rg += Y * cM.ri[sp];
        cp += cpi * Y;
        h += Y * hi;
        e += Y * ei;
    }
    const double Rgas = rg * 1000;
    const double Cp = cp * 1000;
    v[PD] = (P)((double)v[PP] / (T * Rgas));
    v[PH] = (P)(h * 1000);
    E = e * 1000;
    v[PG] = (P)(Cp / (Cp - Rgas));
}

// All ghost cells in one launch, for extents of at least bc (so that a mirror
// image is an interior cell; launch_ghost).  The reference fills x, then y over every i,
// then z over every i, j, each direction from the cells the one before has
// finished; a cell of an edge or a corner is therefore its z image's y image's
// x image.  Each thread follows that chain to the interior cell (or inflow
// plane) at its end and applies what the chain does to it: copies, velocity
// flips, and the wall-side recompute, which depends on T, P and Y alone and so
// need be done once however often the chain asks for it.  As three launches a small grid paid two more launches
// and their drain per fill (4000 x 2 x 2: 12 us of a 75 us step).
template <class P>
__global__ void __launch_bounds__(128) k_ghost(GhostArgs a, P *q)
{
    const Layout &L = a.L;
    const int bc = L.bc, g = 2 * bc;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nz = L.NI * L.NJ * g, ny = L.NI * g * L.nk, nx = g * L.nj * L.nk;
    int i, j, k;
    if (t < nz) {
        // z faces: every i, j
        i = t % L.NI;
        j = (t / L.NI) % L.NJ;
        const int gk = t / (L.NI * L.NJ);
        k = gk < bc ? gk : L.nk + gk;
    } else if ((t -= nz) < ny) {
        // y faces: every i, k interior
        i = t % L.NI;
        const int gj = (t / L.NI) % g;
        j = gj < bc ? gj : L.nj + gj;
        k = bc + t / (L.NI * g);
    } else if ((t -= ny) < nx) {
        // x faces: j, k interior; a warp covers the bc ghost cells of
        // consecutive rows j on one face, so neighbouring lanes write
        // neighbouring cells and read the inflow planes (j fastest) in order
        const int gi = t % bc;
        j = bc + (t / bc) % L.nj;
        i = (t / (bc * L.nj)) % 2 == 0 ? gi : L.ni + bc + gi;
        k = bc + t / (g * L.nj);
    } else {
        return;
    }
    const long long d = L.at(i, j, k);
    bool wall = false, flipv = false, flipw = false, inflow = false;
    if (k < bc || k >= L.nk + bc) {
        k = k < bc ? 2 * bc - 1 - k : 2 * (L.nk + bc) - 1 - k;
        if (a.kind == EU3D_BC_ODM) wall = flipw = true;
    }
    if (j < bc || j >= L.nj + bc) {
        const bool lower = j < bc;
        j = lower ? 2 * bc - 1 - j : 2 * (L.nj + bc) - 1 - j;
        if (lower && a.kind != EU3D_BC_TRANSMISSIVE) wall = true;
        if (lower && a.kind == EU3D_BC_ODM) flipv = true;
    }
    if (i < bc || i >= L.ni + bc) {
        const bool lower = i < bc;
        if (a.kind == EU3D_BC_TRANSMISSIVE) {
            i = lower ? bc : L.ni + bc - 1;
        } else if (a.kind == EU3D_BC_ODM && lower) {
            inflow = true;
        } else {
            i = lower ? 2 * bc - 1 - i : 2 * (L.ni + bc) - 1 - i;
            if (a.kind == EU3D_BC_ODM) wall = true;
        }
    }
    P v[NPRIM];
    double T, E;
    if (inflow)
        ghost_inflow(a, j - bc, k - bc, v, T, E);
    else
        ghost_load(a, q, L.at(i, j, k), v, T, E);
    if (flipv) v[PV] = -v[PV];
    if (flipw) v[PW] = -v[PW];
    if (wall) ghost_wall(a, v, T, E);
    ghost_store(a, q, d, v, T, E);
}

// The ghost cells of one axis (0: x, 1: y, 2: z), one thread per grid line, in the
// reference's order: the lower end from the outside in, then the upper from the
// inside out.  With an extent below bc the mirror image of an outer ghost cell
// is a ghost cell of the other end -- the lower end takes what the last fill left
// there, the upper what this one has just stored -- so a line is one thread's.
template <class P, int AXIS>
__global__ void __launch_bounds__(128) k_ghost_line(GhostArgs a, P *q)
{
    const Layout &L = a.L;
    const int bc = L.bc, t = blockIdx.x * blockDim.x + threadIdx.x;
    // lines: x over interior j, k; y over all i, interior k; z over all i, j
    const int n1 = AXIS == 0 ? L.nj : L.NI, n2 = AXIS == 2 ? L.NJ : L.nk;
    if (t >= n1 * n2) return;
    const int c1 = t % n1 + (AXIS == 0 ? bc : 0), c2 = t / n1 + (AXIS == 2 ? 0 : bc);
    const int n = AXIS == 0 ? L.ni : AXIS == 1 ? L.nj : L.nk;
    const bool odm = a.kind == EU3D_BC_ODM, transm = a.kind == EU3D_BC_TRANSMISSIVE;
    auto cell = [&](int p) { return AXIS == 0 ? L.at(p, c1, c2) : AXIS == 1 ? L.at(c1, p, c2) : L.at(c1, c2, p); };
    for (int g = 0; g < 2 * bc; g++) {
        const bool lower = g < bc;
        const int p = lower ? g : n + g;
        P v[NPRIM];
        double T, E;
        if (AXIS == 0 && odm && lower) {
            ghost_inflow(a, c1 - bc, c2 - bc, v, T, E);
        } else {
            const int mirror = lower ? 2 * bc - 1 - p : 2 * (n + bc) - 1 - p;
            ghost_load(a, q, cell(AXIS == 0 && transm ? (lower ? bc : n + bc - 1) : mirror), v, T, E);
            if (AXIS == 1 && odm && lower) v[PV] = -v[PV];
            if (AXIS == 2 && odm) v[PW] = -v[PW];
            if (AXIS == 0 ? odm : AXIS == 1 ? lower && !transm : odm) ghost_wall(a, v, T, E);
        }
        ghost_store(a, q, cell(p), v, T, E);
    }
}

// Wedge immersed boundary (new): solid cells take the state of the fluid
// cell nearest to their mirror image across the wedge surface, with the
// velocity reflected about the surface.  Only the band of solid cells that
// flux stencils reach is filled (fluid within two cells along x or y);
// band[n] = (i, j, si, sj): the solid column and its mirror source, the same
// for every k, listed on the host when the wedge is set.
template <class P>
__global__ void k_wedge_band(GhostArgs a, P *q, const int4 *__restrict__ band, int nband, double nx, double ny)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (n >= nband) return;
    const int4 b = band[n];
    const Layout &L = a.L;
    const long long d = L.at(b.x, b.y, k), s = L.at(b.z, b.w, k);
    P w[NPRIM];
    double T, E;
    ghost_load(a, q, s, w, T, E);
    const double u = (double)w[PU], v = (double)w[PV];
    const double un = u * nx + v * ny;
    w[PU] = (P)(u - 2.0 * un * nx);
    w[PV] = (P)(v - 2.0 * un * ny);
    ghost_store(a, q, d, w, T, E);
}

// CFL: block minima of min(dx/(|U|+C), dy/(|V|+C)[, dz/(|W|+C)]) over the
// interior (solid wedge cells excluded), C = sqrt(Gamma P / D) as the decode
// defines it.
// CFLcondition (src/Flowfield.cpp:242-272) as block maxima: because IEEE
// division is monotone in the divisor, the smallest dx / (|U| + C) over the
// cells is dx over the largest |U| + C, bit for bit; so each block keeps the
// largest |U| + C, |V| + C, |W| + C of its cells and the last block to
// finish divides once.  A cell whose x time is NaN is skipped, as the reference's
// comparisons skip it; NaN y or z times drop out of fmax as they drop out of
// the reference's min.  One warp takes 128-cell segments of the (j, k) rows of
// interior cells: a whole row per warp left a 4000 x 2 x 2 grid to four warps (41 us;
// 5 with segments and the division in the same launch).
// FP64 primitives: the reference's FP64 arithmetic (C = sqrt(gamma p / rho),
// src/Flowfield.cpp:1281).  FP32 primitives: the same speeds in FP32 (the
// inputs carry FP32 precision already), widened exactly for the maxima.
__device__ __forceinline__ void cfl_speeds(double D, double Pp, double G, double U, double V, double W, double &ax,
                                           double &ay, double &az)
{
    const double x = G * Pp;
    // straight-line quotient and root (the same bits) where they round as IEEE's
    const bool normal = D >= 1e-290 && D <= 1e290 && fabs(x) <= 1e290;
    const double C = normal ? sqrt_rn(div_rn(x, D)) : sqrt(x / D);
    ax = fabs(U) + C;
    ay = fabs(V) + C;
    az = fabs(W) + C;
}

__device__ __forceinline__ void cfl_speeds(float D, float Pp, float G, float U, float V, float W, double &ax,
                                           double &ay, double &az)
{
    const float C = sqrtf(__fdividef(__fmul_rn(G, Pp), D));
    ax = (double)__fadd_rn(fabsf(U), C);
    ay = (double)__fadd_rn(fabsf(V), C);
    az = (double)__fadd_rn(fabsf(W), C);
}

constexpr int CFL_U = 4;  // cells a lane has in flight
constexpr int CFL_WARPS = 8, CFL_SEG = 32 * CFL_U;

// largest of each speed over the block, in thread 0
__device__ __forceinline__ void cfl_block_max(double &sx, double &sy, double &sz)
{
    __shared__ double sm[3][CFL_WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        sx = fmax(sx, __shfl_down_sync(0xffffffffu, sx, o));
        sy = fmax(sy, __shfl_down_sync(0xffffffffu, sy, o));
        sz = fmax(sz, __shfl_down_sync(0xffffffffu, sz, o));
    }
    __syncthreads();
    if (lane == 0) {
        sm[0][wid] = sx;
        sm[1][wid] = sy;
        sm[2][wid] = sz;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < CFL_WARPS; w++) {
            sx = fmax(sx, sm[0][w]);
            sy = fmax(sy, sm[1][w]);
            sz = fmax(sz, sm[2][w]);
        }
}

// partial: one triple per block, then (at 3 max_parts) the count of finished
// blocks, zero between launches.  advance: time += dt as well (one rank); 0
// leaves time for after the all-ranks minimum of dt (k_advance_time).  dt_conv
// starts at 1e10 as in the reference, so a domain without fluid cells gets
// cfl * 1e10.
template <class P>
__global__ void __launch_bounds__(32 * CFL_WARPS) k_cfl(Layout L, const P *__restrict__ q, int use_z,
                                                        const double *__restrict__ xn, const double *__restrict__ yn,
                                                        double x0, double y0, double tn, int wedge_on,
                                                        double *partial, int max_parts, double dx, double dy, double dz,
                                                        double cfl, double final_time, double *scal, int advance)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long fs = L.fs;
    const int nseg = (L.ni + CFL_SEG - 1) / CFL_SEG;
    const int units = L.nj * L.nk * nseg;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int t = blockIdx.x * CFL_WARPS + wid; t < units; t += gridDim.x * CFL_WARPS) {
        const int r = t / nseg, i0 = L.bc + (t - r * nseg) * CFL_SEG + lane;
        const int j = L.bc + r % L.nj, k = L.bc + r / L.nj;
        const double y = yn[j];
        const long long base = L.at(0, j, k);
        // all loads of the segment are issued before the first speed is formed
        // (the maxima do not depend on the order)
        bool ok[CFL_U];
        P vd[CFL_U], vp[CFL_U], vg[CFL_U], vu[CFL_U], vv[CFL_U], vw[CFL_U];
#pragma unroll
        for (int u = 0; u < CFL_U; u++) {
            const int i = i0 + 32 * u;
            ok[u] = i < L.ni + L.bc;
            if (ok[u] && wedge_on) {
                const double x = xn[i];
                ok[u] = !(x > x0 && (y - y0) < (x - x0) * tn);
            }
            if (ok[u]) {
                const long long c = base + i;
                vd[u] = q[PD * fs + c];
                vp[u] = q[PP * fs + c];
                vg[u] = q[PG * fs + c];
                vu[u] = q[PU * fs + c];
                vv[u] = q[PV * fs + c];
                vw[u] = q[PW * fs + c];
            }
        }
#pragma unroll
        for (int u = 0; u < CFL_U; u++) {
            if (!ok[u]) continue;
            double ax, ay, az;
            cfl_speeds(vd[u], vp[u], vg[u], vu[u], vv[u], vw[u], ax, ay, az);
            if (isnan(ax)) continue;
            sx = fmax(sx, ax);
            sy = fmax(sy, ay);
            if (use_z) sz = fmax(sz, az);
        }
    }
    cfl_block_max(sx, sy, sz);
    __shared__ bool last;
    unsigned *done = reinterpret_cast<unsigned *>(partial + 3 * (size_t)max_parts);
    if (threadIdx.x == 0) {
        partial[3 * blockIdx.x + 0] = sx;
        partial[3 * blockIdx.x + 1] = sy;
        partial[3 * blockIdx.x + 2] = sz;
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // the last block: every other block's triple is visible
    __threadfence();
    sx = sy = sz = 0.0;
    for (int t = threadIdx.x; t < (int)gridDim.x; t += blockDim.x) {
        sx = fmax(sx, __ldcg(partial + 3 * t + 0));
        sy = fmax(sy, __ldcg(partial + 3 * t + 1));
        sz = fmax(sz, __ldcg(partial + 3 * t + 2));
    }
    cfl_block_max(sx, sy, sz);
    if (threadIdx.x == 0) {
        *done = 0;
        // the smallest of dx/sx, dy/sy (and dz/sz); a zero speed gives an
        // infinite time, which the reference's 1e10 start caps
        double m = 1e10;
        const double a = dx / sx, b = dy / sy;
        if (a < m) m = a;
        if (b < m) m = b;
        if (use_z) {
            const double z = dz / sz;
            if (z < m) m = z;
        }
        double dt = cfl * m;
        if (scal[1] + dt > final_time) dt = final_time - scal[1];
        scal[0] = dt;
        if (advance) scal[1] += dt;
    }
}

__global__ void k_advance_time(double *scal) { scal[1] += scal[0]; }

// x-slab halo: two x planes of every field the ghost fills write (NPRIM
// primitives, T, E) over the whole y-z extent, ghost rows included, to or
// from a contiguous buffer laid out [field][plane][k][j].  The primitives
// come first in P, then T and E in FP64.  src/Flowfield.cpp:775-1083
// (Mpi_Boundary) exchanges the same planes field by field.
template <class P>
__global__ void k_halo(Layout L, P *__restrict__ q, double *__restrict__ T, double *__restrict__ E,
                       unsigned char *__restrict__ buf, int i0, int pack)
{
    const long long plane = (long long)L.NJ * L.NK;
    const long long n = 2 * plane;
    P *bp = reinterpret_cast<P *>(buf);
    double *bd = reinterpret_cast<double *>(buf + (size_t)NPRIM * n * sizeof(P));
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(t / plane);
        const long long r = t - p * plane;
        const int j = (int)(r % L.NJ), k = (int)(r / L.NJ);
        const long long c = L.at(i0 + p, j, k);
        if (pack) {
#pragma unroll
            for (int f = 0; f < NPRIM; f++) bp[f * n + t] = q[f * L.fs + c];
            bd[t] = T[c];
            bd[n + t] = E[c];
        } else {
#pragma unroll
            for (int f = 0; f < NPRIM; f++) q[f * L.fs + c] = bp[f * n + t];
            T[c] = bd[t];
            E[c] = bd[n + t];
        }
    }
}

}  // namespace eu3d
