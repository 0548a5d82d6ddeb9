// Hexahedral edge-element FEM (orders 1-3) of the fem_v2 family on one GPU:
// leapfrog (fem_v2/fem_simulation.cpp:560-655), 2nd-order symplectic
// (symplectic_2/fem_simulation.cpp:557-672) and its 4th-order triple jump
// (symplectic_4/fem_simulation.cpp:1280-1281,1347-1350).
//
// The reference applies the dense element matrix per element and scatters
// with atomics (fem_v2/fem_kernels.hpp:13-175).  Here every edge DOF gathers
// the contributions of the (at most four) elements that contain it, so there
// are no atomics and results are deterministic.  In FP64 the contributions
// are summed in the reference's element-visiting order (outer elements of
// fem_simulation.cpp:424-455 first, then inner elements) with unfused
// operations, and the source enters between the outer and inner sweeps as in
// the reference; the result is bit-identical to the serial reference.
// Orders 1 and 2 run in two passes: the element values K u of every element,
// then the DOFs, which sum theirs and take the whole update of the substep.
// Order 3 forms the rows DOF by DOF (144 values per element do not fit the
// registers of the element pass), and so do grids of 2^31 DOFs and more per
// component, small FP64 grids of order 2, and grids that leave no memory for
// the element values.
#include <cuda_runtime.h>

#include <cmath>
#include <fstream>
#include <iomanip>
#include <utility>

#include "ems_internal.hpp"

namespace ems {

__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double xsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float xsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float xmul(float a, float b) { return __fmul_rn(a, b); }

constexpr int kMaxSrc = 8;

// Division of a value below 2^31 by a divisor known to the host, as a product
// and a shift: m = floor(2^s / d) + 1 with s = 31 + ceil(log2 d).
struct HexDiv {
    unsigned m;
    int s;
    __device__ __forceinline__ unsigned operator()(unsigned t) const { return (unsigned)((unsigned long long)t * m >> s); }
};
constexpr size_t kHexDivLimit = (size_t)1 << 31;
static HexDiv hex_div(int d)
{
    int l = 0;
    while ((1ll << l) < d) ++l;
    return l ? HexDiv{(unsigned)((1ull << (31 + l)) / (unsigned)d + 1), 31 + l} : HexDiv{1u, 0};
}

struct HexGeom {
    int o, gx, gy, gz, EX, EY, EZ, nouter, dof, total;
    size_t nc[3];
    HexDiv row[2], col[2];   // by gx, gx + 1 and gy, gy + 1
};

// Rank of element (i,j,k) in the reference's visiting order.
__device__ __forceinline__ int elem_rank(const HexGeom &g, int i, int j, int k)
{
    const int EX = g.EX, EY = g.EY, EZ = g.EZ;
    if (k == 0) return i + j * EX;
    if (k == EZ - 1) return EX * EY + i + j * EX;
    int b = 2 * EX * EY;
    if (i == 0) return b + j + (k - 1) * EY;
    if (i == EX - 1) return b + EY * (EZ - 2) + j + (k - 1) * EY;
    b += 2 * EY * (EZ - 2);
    if (j == 0) return b + (k - 1) + (i - 1) * (EZ - 2);
    if (j == EY - 1) return b + (EZ - 2) * (EX - 2) + (k - 1) + (i - 1) * (EZ - 2);
    return g.nouter + (i - 1) + (j - 1) * (EX - 2) + (k - 1) * (EX - 2) * (EY - 2);
}

__device__ __forceinline__ bool on_pec(const HexGeom &g, int c, int ix, int iy, int iz)
{
    if (c == 0) return iy == 0 || iy == g.gy || iz == 0 || iz == g.gz;
    if (c == 1) return ix == 0 || ix == g.gx || iz == 0 || iz == g.gz;
    return ix == 0 || ix == g.gx || iy == 0 || iy == g.gy;
}

// Source values of the run: entry (step, substep) of vals for every source.
struct SrcTab {
    int n, nsub, q;
    int comp[kMaxSrc];
    int idx[kMaxSrc];
    const double *vals;
    // steps done, counted twice: step[0] is read by the sampling and moved on
    // by a step's last launch, step[1] by its first element pass and read by
    // the DOF passes, so no launch reads what it writes
    int *step;
    bool last;
};

struct SrcList {
    int n;
    int comp[kMaxSrc];
    int idx[kMaxSrc];
    double val[kMaxSrc];
};

// Force on one DOF: sum over the containing elements of row r of K times the
// element's gathered local vector.  sign -1: fem_v2 (-=), +1: symplectic (+=).
// EXACT: reference order and unfused FP ops; otherwise FMA accumulation.
template <class T, int O, bool EXACT>
__device__ T dof_force(const HexGeom &g, const T *__restrict__ K, const T *const lv[3], int c, int ix, int iy, int iz,
                       T sign, bool has_src, T srcval)
{
    constexpr int D = O * (O + 1) * (O + 1);
    constexpr int TT = 3 * D;
    // candidate element coordinates and local offsets per axis
    int ec[3][2], lc[3][2], nc_[3];
    const int pos[3] = {ix, iy, iz};
    const int ne[3] = {g.EX, g.EY, g.EZ};
    for (int d = 0; d < 3; ++d) {
        int p = pos[d];
        int e0 = p / O;
        nc_[d] = 0;
        if (d == c) {  // along the edge direction: exactly one element
            if (e0 < ne[d]) { ec[d][0] = e0; lc[d][0] = p - O * e0; nc_[d] = 1; }
        } else {
            if (e0 < ne[d]) { ec[d][nc_[d]] = e0; lc[d][nc_[d]] = p - O * e0; ++nc_[d]; }
            if (p % O == 0 && e0 - 1 >= 0 && e0 - 1 < ne[d]) { ec[d][nc_[d]] = e0 - 1; lc[d][nc_[d]] = O; ++nc_[d]; }
        }
    }
    int cnt = 0, rk[4], ex_[4], ey_[4], ez_[4], row[4];
    for (int a = 0; a < nc_[0]; ++a)
        for (int b = 0; b < nc_[1]; ++b)
            for (int q = 0; q < nc_[2]; ++q) {
                int l = lc[0][a], m = lc[1][b], n = lc[2][q], r;
                if (c == 0) r = l + m * O + n * O * (O + 1);
                else if (c == 1) r = D + l + m * (O + 1) + n * O * (O + 1);
                else r = 2 * D + l + m * (O + 1) + n * (O + 1) * (O + 1);
                ex_[cnt] = ec[0][a]; ey_[cnt] = ec[1][b]; ez_[cnt] = ec[2][q]; row[cnt] = r;
                rk[cnt] = EXACT ? elem_rank(g, ec[0][a], ec[1][b], ec[2][q]) : cnt;
                ++cnt;
            }
    if (EXACT)  // insertion sort by visiting rank
        for (int a = 1; a < cnt; ++a)
            for (int b = a; b > 0 && rk[b - 1] > rk[b]; --b) {
                int t;
                t = rk[b]; rk[b] = rk[b - 1]; rk[b - 1] = t;
                t = ex_[b]; ex_[b] = ex_[b - 1]; ex_[b - 1] = t;
                t = ey_[b]; ey_[b] = ey_[b - 1]; ey_[b - 1] = t;
                t = ez_[b]; ez_[b] = ez_[b - 1]; ez_[b - 1] = t;
                t = row[b]; row[b] = row[b - 1]; row[b - 1] = t;
            }
    T acc = 0;
    bool src_done = !has_src;
    const int gx = g.gx, gy = g.gy;
    for (int e = 0; e < cnt; ++e) {
        if (!src_done && rk[e] >= g.nouter) { acc = xadd(acc, srcval); src_done = true; }
        const T *Kr = K + (size_t)row[e] * TT;
        const int fx = O * ex_[e], fy = O * ey_[e], fz = O * ez_[e];
        T temp = 0;
        int mm = 0;
        for (int n = 0; n < O + 1; ++n)
            for (int m = 0; m < O + 1; ++m)
                for (int l = 0; l < O; ++l, ++mm) {
                    T v = lv[0][(size_t)(fx + l) + (size_t)(fy + m) * gx + (size_t)(fz + n) * gx * (gy + 1)];
                    temp = EXACT ? xadd(temp, xmul(Kr[mm], v)) : fma(Kr[mm], v, temp);
                }
        for (int n = 0; n < O + 1; ++n)
            for (int m = 0; m < O; ++m)
                for (int l = 0; l < O + 1; ++l, ++mm) {
                    T v = lv[1][(size_t)(fx + l) + (size_t)(fy + m) * (gx + 1) + (size_t)(fz + n) * (gx + 1) * gy];
                    temp = EXACT ? xadd(temp, xmul(Kr[mm], v)) : fma(Kr[mm], v, temp);
                }
        for (int n = 0; n < O; ++n)
            for (int m = 0; m < O + 1; ++m)
                for (int l = 0; l < O + 1; ++l, ++mm) {
                    T v = lv[2][(size_t)(fx + l) + (size_t)(fy + m) * (gx + 1) + (size_t)(fz + n) * (gx + 1) * (gy + 1)];
                    temp = EXACT ? xadd(temp, xmul(Kr[mm], v)) : fma(Kr[mm], v, temp);
                }
        acc = sign < 0 ? xsub(acc, temp) : xadd(acc, temp);
    }
    if (!src_done) acc = xadd(acc, srcval);
    return acc;
}

// Coordinates of DOF t of component c, for fewer than 2^31 of them (see HexDiv).
__device__ __forceinline__ void dof_coords32(const HexGeom &g, int c, unsigned u, int &ix, int &iy, int &iz)
{
    const int nxc = c == 0 ? g.gx : g.gx + 1, nyc = c == 1 ? g.gy : g.gy + 1;
    const unsigned r = c == 0 ? g.row[0](u) : g.row[1](u);
    ix = (int)(u - r * nxc);
    iz = (int)(c == 1 ? g.col[0](r) : g.col[1](r));
    iy = (int)(r - (unsigned)iz * nyc);
}
__device__ __forceinline__ void dof_coords(const HexGeom &g, int c, size_t t, int &ix, int &iy, int &iz)
{
    if (g.nc[c] < kHexDivLimit) return dof_coords32(g, c, (unsigned)t, ix, iy, iz);
    const int nxc = c == 0 ? g.gx : g.gx + 1, nyc = c == 1 ? g.gy : g.gy + 1;
    const size_t r = t / nxc;
    ix = (int)(t % nxc);
    iy = (int)(r % nyc);
    iz = (int)(r / nyc);
}

// Leapfrog step, one thread per DOF: E2 = (-K E1, boundary zeroed) + 2 E1 - E0,
// then the point source, then PEC (fem_v2/fem_simulation.cpp:576-654, 1115).
template <class T, int O, bool EXACT>
__global__ void __launch_bounds__(128) hex_leapfrog_kernel(HexGeom g, const T *__restrict__ K, const T *E1x, const T *E1y,
                                                           const T *E1z, const T *E0x, const T *E0y, const T *E0z,
                                                           T *E2x, T *E2y, T *E2z, SrcList src)
{
    const int c = blockIdx.y;
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.nc[c]) return;
    int ix, iy, iz;
    dof_coords(g, c, t, ix, iy, iz);
    const T *lv[3] = {E1x, E1y, E1z};
    T f = 0;
    bool pec = on_pec(g, c, ix, iy, iz);
    if (!pec) f = dof_force<T, O, EXACT>(g, K, lv, c, ix, iy, iz, T(-1), false, T(0));
    const T *e1 = c == 0 ? E1x : c == 1 ? E1y : E1z;
    const T *e0 = c == 0 ? E0x : c == 1 ? E0y : E0z;
    T v = xadd(f, xsub(xmul(T(2), e1[t]), e0[t]));
    for (int s = 0; s < src.n; ++s)
        if (src.comp[s] == c && (size_t)src.idx[s] == t) v = xsub(v, (T)src.val[s]);
    if (pec) v = 0;
    T *e2 = c == 0 ? E2x : c == 1 ? E2y : E2z;
    e2[t] = v;
}

// Symplectic kick: F = K U (+ source between outer and inner elements),
// boundary F zeroed, P -= dt F (symplectic_2/fem_simulation.cpp:603-653).
// F is also stored (the reference keeps it in level 2).
template <class T, int O, bool EXACT>
__global__ void __launch_bounds__(128) hex_kick_kernel(HexGeom g, const T *__restrict__ K, const T *Ux, const T *Uy, const T *Uz,
                                                       T *Px, T *Py, T *Pz, T *Fx, T *Fy, T *Fz, T dt, SrcList src)
{
    const int c = blockIdx.y;
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.nc[c]) return;
    int ix, iy, iz;
    dof_coords(g, c, t, ix, iy, iz);
    const T *lv[3] = {Ux, Uy, Uz};
    bool has = false;
    T sv = 0;
    for (int s = 0; s < src.n; ++s)
        if (src.comp[s] == c && (size_t)src.idx[s] == t) { has = true; sv = (T)src.val[s]; }
    T f = 0;
    if (!on_pec(g, c, ix, iy, iz)) f = dof_force<T, O, EXACT>(g, K, lv, c, ix, iy, iz, T(1), has, sv);
    T *F = c == 0 ? Fx : c == 1 ? Fy : Fz;
    T *P = c == 0 ? Px : c == 1 ? Py : Pz;
    F[t] = f;
    P[t] = EXACT ? xsub(P[t], xmul(dt, f)) : fma(-dt, f, P[t]);
}

// Drift U += coef * P / m (symplectic_2/fem_simulation.cpp:583-601, 647-668);
// coef = 0.5*deltat, inv_m = 8/o^3 as in the reference's operand order; with
// `pec` set, U and P are zeroed on the boundary afterwards (1132-1276).  MUL:
// m is a power of two and comes as 1 / m, the same value without the division.
template <class T, bool EXACT, bool MUL>
__global__ void hex_drift_kernel(const __grid_constant__ HexGeom g, T *Ux, T *Uy, T *Uz, T *Px, T *Py, T *Pz, T coef, T m, int pec)
{
    wait_for_last();
    const int c = blockIdx.y;
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.nc[c]) return;
    T *U = c == 0 ? Ux : c == 1 ? Uy : Uz;
    T *P = c == 0 ? Px : c == 1 ? Py : Pz;
    const T v = MUL ? xmul(xmul(coef, P[t]), m) : (T)(xmul(coef, P[t]) / m);
    T u = xadd(U[t], v);
    if (pec) {
        int ix, iy, iz;
        dof_coords(g, c, t, ix, iy, iz);
        if (on_pec(g, c, ix, iy, iz)) { u = 0; P[t] = 0; }
    }
    U[t] = u;
}

// Receivers: fem_v2/fem_simulation.cpp:1273-1312 (one thread per receiver),
// row s of the table.
template <class T>
__device__ __forceinline__ void hex_sample(const HexGeom &g, const T *Lx, const T *Ly, const T *Lz, int o, const int *obs, double *tr,
                                           int nsamp, int s)
{
    const int gx = g.gx, gy = g.gy;
    int ox = obs[3 * o], oy = obs[3 * o + 1], oz = obs[3 * o + 2];
    double *out = tr + ((size_t)o * nsamp + s) * 4;
    double a = __dadd_rn(__dadd_rn(__dadd_rn((double)Lx[ox - 1], (double)Lx[ox]), (double)Lx[ox + gx * (gy + 1) - 1]), (double)Lx[ox + gx * (gy + 1)]);
    double b = __dadd_rn(__dadd_rn(__dadd_rn((double)Ly[oy - (gx + 1)], (double)Ly[oy]), (double)Ly[oy + (gx + 1) * (gy - 1)]), (double)Ly[oy + (gx + 1) * gy]);
    out[1] = a / 4.0;
    out[2] = b / 4.0;
    out[3] = (double)Lz[oz];
}

template <class T>
__global__ void hex_sample_kernel(HexGeom g, const T *Lx, const T *Ly, const T *Lz, int nobs, const int *obs, double *tr, int nsamp, int s,
                                  const int *step, int tf)
{
    wait_for_last();
    if (step) {   // a replayed step: the row from the step counter
        if (*step % tf) return;
        s = *step / tf;
    }
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o < nobs) hex_sample<T>(g, Lx, Ly, Lz, o, obs, tr, nsamp, s);
}
// Sampling by the blocks behind the elements' of a leapfrog step's element
// pass (it reads the level that is sampled).
struct HexRec {
    int n, nsamp, tf;
    const int *obs;
    double *tr;
};

// The step counter and the sampling blocks of an element pass; true for a
// block without elements.
template <class T>
__device__ __forceinline__ bool hex_elem_head(const HexGeom &g, const T *Ux, const T *Uy, const T *Uz, int ne, int nt, int *step, const HexRec &rec)
{
    if (step && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) step[1] += 1;
    const int first = (ne + nt - 1) / nt, b = (int)blockIdx.x - first;
    if (b < 0) return false;
    const int o = b * nt + threadIdx.x;
    if (blockIdx.y == 0 && o < rec.n && step[0] % rec.tf == 0) hex_sample<T>(g, Ux, Uy, Uz, o, rec.obs, rec.tr, rec.nsamp, step[0] / rec.tf);
    return true;
}

// Element pass: rows c D .. c D + D - 1 of K u of one element per thread
// (component c = blockIdx.y), fe[row][element].  Each sum runs in column order
// as dof_force's.  K is laid out column by column, each padded to 16 bytes.
// In FP32 it is a kernel argument, so a multiply-add takes its value from the
// constant bank; from shared memory, one vector for four rows of a column, the
// load pipe was the bound (14.8 us a pass against 12.9, order 2 on 72^3 grid
// cells, each launch alone).  FP64 keeps shared memory: its pass is bound by
// the FP64 pipe.  A symp4 step there: FP32 278 us in one pass DOF by DOF,
// 65 in two; FP64 2402 and 1857.  step: given to a step's first pass (see SrcTab).
template <class T, int O> struct HexRows {
    static constexpr int D = O * (O + 1) * (O + 1), TT = 3 * D, W = 16 / (int)sizeof(T), RP = (D + W - 1) / W * W;
};
template <class T, int O> struct HexK { const T *k; };   // K of the element pass, [3][TT][RP]
template <int O> struct HexK<float, O> { float k[3 * HexRows<float, O>::TT * HexRows<float, O>::RP]; };
template <class T, int O, bool EXACT>
__global__ void __launch_bounds__(128) hex_elem_kernel(const __grid_constant__ HexGeom g, const __grid_constant__ HexK<T, O> K,
                                                       const T *Ux, const T *Uy, const T *Uz, T *fe, int *step, HexRec rec)
{
    constexpr int D = HexRows<T, O>::D, TT = HexRows<T, O>::TT, W = HexRows<T, O>::W, RP = HexRows<T, O>::RP;
    constexpr bool ARG = sizeof(T) == 4;
    __shared__ __align__(16) T sK[ARG ? 1 : TT * RP];
    const int c = blockIdx.y;
    const int ne = g.EX * g.EY * g.EZ, e = blockIdx.x * 128 + threadIdx.x;
    if constexpr (!ARG) {
        const int4 *k4 = reinterpret_cast<const int4 *>(K.k + (size_t)c * TT * RP);   // does not change: ahead of the wait
        for (int q = threadIdx.x; q < TT * RP / W; q += 128) reinterpret_cast<int4 *>(sK)[q] = k4[q];
        __syncthreads();
    }
    wait_for_last();
    if (hex_elem_head<T>(g, Ux, Uy, Uz, ne, 128, step, rec)) return;
    if (e >= ne) return;
    const int r0 = e / g.EX, ei = e - r0 * g.EX, ek = r0 / g.EY, ej = r0 - ek * g.EY;
    const int gx = g.gx, gy = g.gy;
    const T *px = Ux + (O * ei + O * ej * gx + (size_t)(O * ek) * gx * (gy + 1));
    const T *py = Uy + (O * ei + O * ej * (gx + 1) + (size_t)(O * ek) * (gx + 1) * gy);
    const T *pz = Uz + (O * ei + O * ej * (gx + 1) + (size_t)(O * ek) * (gx + 1) * (gy + 1));
    T u[TT];
    int at = 0;
#pragma unroll
    for (int n = 0; n < O + 1; ++n)
#pragma unroll
        for (int m = 0; m < O + 1; ++m)
#pragma unroll
            for (int l = 0; l < O; ++l) u[at++] = px[l + m * gx + n * gx * (gy + 1)];
#pragma unroll
    for (int n = 0; n < O + 1; ++n)
#pragma unroll
        for (int m = 0; m < O; ++m)
#pragma unroll
            for (int l = 0; l < O + 1; ++l) u[at++] = py[l + m * (gx + 1) + n * (gx + 1) * gy];
#pragma unroll
    for (int n = 0; n < O; ++n)
#pragma unroll
        for (int m = 0; m < O + 1; ++m)
#pragma unroll
            for (int l = 0; l < O + 1; ++l) u[at++] = pz[l + m * (gx + 1) + n * (gx + 1) * (gy + 1)];
    T f[RP];
#pragma unroll
    for (int r = 0; r < RP; ++r) f[r] = T(0);
#pragma unroll
    for (int mm = 0; mm < TT; ++mm) {
        T k[RP];
#pragma unroll
        for (int r = 0; r < RP; r += W) {
            if constexpr (ARG) {
#pragma unroll
                for (int w = 0; w < W; ++w) k[r + w] = K.k[(c * TT + mm) * RP + r + w];
            } else *reinterpret_cast<int4 *>(&k[r]) = *reinterpret_cast<const int4 *>(&sK[mm * RP + r]);
        }
#pragma unroll
        for (int r = 0; r < D; ++r) f[r] = EXACT ? xadd(f[r], xmul(k[r], u[mm])) : fma(k[r], u[mm], f[r]);
    }
#pragma unroll
    for (int r = 0; r < D; ++r) fe[(size_t)(c * D + r) * ne + e] = f[r];
}

// Order-1 element pass in FP64.  The entries of K have one size per class:
// edges of one direction by how many of their two offsets differ, edges of
// two directions by whether their offset along the third axis differs.  So a
// column needs 5 products, not 12, and a product enters the rows with their
// signs (exact): 204 FP64 operations per element instead of 288.  The host
// checks the classes on the K it loaded and takes hex_elem_kernel otherwise.
struct HexClasses {
    double k[5];
    unsigned sign[12];   // bit j: entry (row, j) is negative
};
__host__ __device__ constexpr int hex1_pos(int e, int axis)   // offset of local edge e along an axis
{
    const int c = e / 4, q = e % 4, lo = q & 1, hi = q >> 1;
    return axis == c ? 0 : c == 0 ? (axis == 1 ? lo : hi) : c == 1 ? (axis == 0 ? lo : hi) : (axis == 0 ? lo : hi);
}
__host__ __device__ constexpr int hex1_class(int i, int j)
{
    const int c = i / 4, d = j / 4;
    if (c != d) return 3 + (hex1_pos(i, 3 - c - d) != hex1_pos(j, 3 - c - d) ? 1 : 0);
    int n = 0;
    for (int a = 0; a < 3; ++a) n += hex1_pos(i, a) != hex1_pos(j, a) ? 1 : 0;
    return n;
}
template <int J, int... I>
__device__ __forceinline__ void hex1_column(std::integer_sequence<int, I...>, const double (&p)[5], const HexClasses &k, double (&f)[12])
{
    ((f[I] = __dadd_rn(f[I], __hiloint2double(__double2hiint(p[hex1_class(I, J)]) ^ (int)((k.sign[I] >> J & 1u) << 31),
                                              __double2loint(p[hex1_class(I, J)])))), ...);
}
template <int... J>
__device__ __forceinline__ void hex1_columns(std::integer_sequence<int, J...>, const double (&u)[12], const HexClasses &k, double (&f)[12])
{
    auto col = [&](auto j) {
        constexpr int C = decltype(j)::value;
        double p[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) p[q] = __dmul_rn(k.k[q], u[C]);
        hex1_column<C>(std::make_integer_sequence<int, 12>{}, p, k, f);
    };
    (col(std::integral_constant<int, J>{}), ...);
}
__global__ void __launch_bounds__(32) hex1_elem_kernel(HexGeom g, const __grid_constant__ HexClasses k, const double *Ux,
                                                       const double *Uy, const double *Uz, double *fe,
                                                       int *step, HexRec rec)
{
    wait_for_last();
    const int ne = g.EX * g.EY * g.EZ, e = blockIdx.x * 32 + threadIdx.x;
    if (hex_elem_head<double>(g, Ux, Uy, Uz, ne, 32, step, rec) || e >= ne) return;
    const int r0 = e / g.EX, ei = e - r0 * g.EX, ek = r0 / g.EY, ej = r0 - ek * g.EY, gx = g.gx, gy = g.gy;
    const double *px = Ux + (ei + ej * gx + (size_t)ek * gx * (gy + 1));
    const double *py = Uy + (ei + ej * (gx + 1) + (size_t)ek * (gx + 1) * gy);
    const double *pz = Uz + (ei + ej * (gx + 1) + (size_t)ek * (gx + 1) * (gy + 1));
    double u[12], f[12];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        u[q] = px[(q & 1) * gx + (q >> 1) * gx * (gy + 1)];
        u[4 + q] = py[(q & 1) + (q >> 1) * (gx + 1) * gy];
        u[8 + q] = pz[(q & 1) + (q >> 1) * (gx + 1)];
    }
#pragma unroll
    for (int r = 0; r < 12; ++r) f[r] = 0.0;
    hex1_columns(std::make_integer_sequence<int, 12>{}, u, k, f);
#pragma unroll
    for (int r = 0; r < 12; ++r) fe[(size_t)r * ne + e] = f[r];
}

// Sum of an inner DOF's element values with the source, in dof_force's order.
// Its (at most four) elements are the one at its place and the ones below it
// along the two axes across the edge, a and b, present where it lies on their
// common face; the values of those are a fixed distance away in fe.
template <class T, int O, bool EXACT, int C>
__device__ __forceinline__ T dof_sum(const HexGeom &g, const T *__restrict__ fe, int ix, int iy, int iz, T sign, bool has_src, T srcval)
{
    constexpr int D = O * (O + 1) * (O + 1);
    constexpr int RX = 1, RY = C == 0 ? O : O + 1, RZ = C == 2 ? (O + 1) * (O + 1) : O * (O + 1);   // rows of K along the axes
    const int ex = ix / O, ey = iy / O, ez = iz / O, l = ix - O * ex, m = iy - O * ey, n = iz - O * ez;
    const long long ne = (long long)g.EX * g.EY * g.EZ;
    // a grid that is no whole number of elements has DOFs behind the last one
    const bool in = ex < g.EX + (C != 0) && ey < g.EY + (C != 1) && ez < g.EZ + (C != 2);
    const bool a0 = in && (C == 0 ? ey < g.EY : ex < g.EX), b0 = in && (C == 2 ? ey < g.EY : ez < g.EZ);
    const bool a1 = in && (C == 0 ? m : l) == 0, b1 = in && (C == 2 ? m : n) == 0;
    const bool p[4] = {a0 && b0, a0 && b1, a1 && b0, a1 && b1};
    const long long da = O * (C == 0 ? RY : RX) * ne - (C == 0 ? g.EX : 1), db = O * (C == 2 ? RY : RZ) * ne - (C == 2 ? g.EX : g.EX * g.EY);
    const T *f = fe + ((C * D + l * RX + m * RY + n * RZ) * ne + (ex + g.EX * (ey + (long long)g.EY * ez)));
    T v[4] = {};
#pragma unroll
    for (int s = 0; s < 4; ++s)
        if (p[s]) v[s] = f[(s >> 1) * da + (s & 1) * db];
    T acc = 0;
    auto add = [&](T x) { acc = sign < 0 ? xsub(acc, x) : xadd(acc, x); };
    if (!EXACT) {   // element by element, the source behind them
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (p[s]) add(v[s]);
        return has_src ? xadd(acc, srcval) : acc;
    }
    const int xl = ex - (C != 0 && a1), yl = ey - (C == 0 ? a1 : C == 2 && b1), zl = ez - (C != 2 && b1);   // lowest element
    if (xl > 0 && yl > 0 && zl > 0 && ex < g.EX - 1 && ey < g.EY - 1 && ez < g.EZ - 1) {
        // only inner elements: visited behind the source, in index order
        if (has_src) acc = xadd(acc, srcval);
        if (p[3]) add(v[3]);
        if (p[1]) add(v[1]);
        if (p[2]) add(v[2]);
        add(v[0]);
        return acc;
    }
    int rk[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int sa = s >> 1, sb = s & 1;
        rk[s] = !p[s] ? 0x7fffffff : elem_rank(g, ex - (C != 0 ? sa : 0), ey - (C == 0 ? sa : C == 2 ? sb : 0), ez - (C != 2 ? sb : 0));
    }
    auto order = [&](int x, int y) {
        if (rk[x] > rk[y]) {
            const int r = rk[x];
            rk[x] = rk[y];
            rk[y] = r;
            const T t = v[x];
            v[x] = v[y];
            v[y] = t;
        }
    };
    order(0, 1); order(2, 3); order(0, 2); order(1, 3); order(1, 2);
    bool src_done = !has_src;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        if (rk[s] == 0x7fffffff) continue;
        if (!src_done && rk[s] >= g.nouter) { acc = xadd(acc, srcval); src_done = true; }
        add(v[s]);
    }
    if (!src_done) acc = xadd(acc, srcval);
    return acc;
}

template <class T> struct HexDofs {
    T *a[3], *b[3], *c[3];   // leapfrog: E1, E0, E2; symplectic: U, P, F
};

// Sources on a DOF.
__device__ __forceinline__ int sources_at(const SrcTab &src, int c, unsigned t)
{
    int n = 0;
    for (int s = 0; s < src.n; ++s) n += src.comp[s] == c && (unsigned)src.idx[s] == t;
    return n;
}

// DOF pass of a leapfrog step (see hex_leapfrog_kernel), component C.
template <class T, int O, bool EXACT, int C>
__device__ __forceinline__ void leap_dof(const HexGeom &g, const T *__restrict__ fe, const HexDofs<T> &d, const SrcTab &src)
{
    const unsigned t = blockIdx.x * 128 + threadIdx.x;
    if (C == 0 && t == 0) src.step[0] += 1;
    if (t >= g.nc[C]) return;
    int ix, iy, iz;
    dof_coords32(g, C, t, ix, iy, iz);
    const bool pec = on_pec(g, C, ix, iy, iz);
    const T a = d.a[C][t], b = d.b[C][t];
    T f = 0;
    if (!pec) f = dof_sum<T, O, EXACT, C>(g, fe, ix, iy, iz, T(-1), false, T(0));
    T v = xadd(f, xsub(xmul(T(2), a), b));
    for (int n = sources_at(src, C, t); n > 0; --n) v = xsub(v, (T)src.vals[src.step[1] - 1]);
    if (pec) v = 0;
    d.c[C][t] = v;
}
// The two DOF passes are bound by instructions, not by their L2 traffic: code
// of its own per component and divisions by products took the kick of order 2
// on 72^3 grid cells from 17.7 to 10.4 us (each launch alone).
template <class T, int O, bool EXACT>
__global__ void __launch_bounds__(128) hex_leap_dof_kernel(const __grid_constant__ HexGeom g, const T *fe, const __grid_constant__ HexDofs<T> d,
                                                           const __grid_constant__ SrcTab src)
{
    wait_for_last();
    if (blockIdx.y == 0) leap_dof<T, O, EXACT, 0>(g, fe, d, src);
    else if (blockIdx.y == 1) leap_dof<T, O, EXACT, 1>(g, fe, d, src);
    else leap_dof<T, O, EXACT, 2>(g, fe, d, src);
}

// DOF pass of a symplectic substep: the force (stored, as the reference keeps
// it), the kick, the closing half drift with the PEC planes zeroed, and the
// opening half drift of the next substep (h2 != 0; FP32 runs take both half
// drifts as one, h1).  Drifts add (h P) / m; 1 / m is a power of two.
template <class T, int O, bool EXACT, int C>
__device__ __forceinline__ void kick_dof(const HexGeom &g, const T *__restrict__ fe, const HexDofs<T> &d, const SrcTab &src, T dt, T h1, T h2, T rm)
{
    const unsigned t = blockIdx.x * 128 + threadIdx.x;
    if (src.last && C == 0 && t == 0) src.step[0] += 1;
    if (t >= g.nc[C]) return;
    int ix, iy, iz;
    dof_coords32(g, C, t, ix, iy, iz);
    const bool pec = on_pec(g, C, ix, iy, iz), has = sources_at(src, C, t) > 0;
    T p = d.b[C][t], u = d.a[C][t], sv = 0, f = 0;
    if (has) sv = (T)src.vals[(size_t)(src.step[1] - 1) * src.nsub + src.q];
    if (!pec) f = dof_sum<T, O, EXACT, C>(g, fe, ix, iy, iz, T(1), has, sv);
    if (src.last) d.c[C][t] = f;   // the step's force is its last substep's
    p = EXACT ? xsub(p, xmul(dt, f)) : fma(-dt, f, p);
    u = xadd(u, xmul(xmul(h1, p), rm));
    if (pec) { u = 0; p = 0; }
    if (h2 != T(0)) u = xadd(u, xmul(xmul(h2, p), rm));
    d.b[C][t] = p;
    d.a[C][t] = u;
}
template <class T, int O, bool EXACT>
__global__ void __launch_bounds__(128) hex_kick_dof_kernel(const __grid_constant__ HexGeom g, const T *fe, const __grid_constant__ HexDofs<T> d,
                                                           const __grid_constant__ SrcTab src, T dt, T h1, T h2, T rm)
{
    wait_for_last();
    if (blockIdx.y == 0) kick_dof<T, O, EXACT, 0>(g, fe, d, src, dt, h1, h2, rm);
    else if (blockIdx.y == 1) kick_dof<T, O, EXACT, 1>(g, fe, d, src, dt, h1, h2, rm);
    else kick_dof<T, O, EXACT, 2>(g, fe, d, src, dt, h1, h2, rm);
}

__global__ void hex_widen_kernel(const float *x, double *y, size_t n)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) y[t] = (double)x[t];
}

static double femv2_source(double t)
{
    const double freq = 1.0e9;
    const double chi = 1.0 / freq;
    double delay = t - chi;
    double zeta = 2.0 * M_PI * M_PI * freq * freq;
    return 2.0 * zeta * (2.0 * zeta * delay * delay - 1.0) * std::exp(0.0 - zeta * delay * delay) * 0.001;
}

struct HexFemSim : Sim {
    ems_hexfem_params P;
    std::string kdir;
    HexGeom g{};
    bool fp64, exact;
    DevBuf lev[3];         // per component: 3 levels
    DevBuf dK, dKr;        // K as the element pass takes it, and row by row
    bool one_pass = false; // the force DOF by DOF (see below)
    std::vector<double> Kh;
    std::vector<std::array<int, 4>> srcs;   // comp, flat index
    std::vector<std::array<int, 3>> obs_idx; // x, y, z flat indices
    std::vector<std::array<int, 3>> obs_ijk;
    int l0 = 0, l1 = 1, l2 = 2;              // leapfrog ring
    HexClasses cls{};                        // order 1 in FP64: the sizes and signs of K's entries
    bool classes = false;
    std::vector<float> k32;                  // orders 1 and 2 in FP32: K as the element pass takes it
    double cur_time = 0.0;
    DevBuf d_obs, d_tr, d_fe, d_vals, d_step;
    cudaGraphExec_t graph = nullptr;         // kGraphSteps steps, kept while the buffers stay the same
    std::vector<unsigned long long> graph_key, last_key;   // of the graph, of the last run
    static constexpr int kGraphSteps = 9;    // a multiple of the three levels' ring
    // Capturing and instantiating a graph takes 60 to 170 us.  A run of this many
    // launches earns it (leapfrog of 512 elements, a fresh handle: 16 steps 211 us
    // with a graph and 170 before there was one, 100 steps 455 and 690), and so
    // does a run that repeats the last one.
    static constexpr int kGraphMinLaunches = 160;
    ~HexFemSim() override
    {
        if (graph) cudaGraphExecDestroy(graph);
    }

    explicit HexFemSim(const ems_hexfem_params *p) : Sim(Kind::HEXFEM), P(*p)
    {
        kdir = P.kmat_dir ? P.kmat_dir : "kmat";
        P.kmat_dir = nullptr;
        EMS_CHECK_ARG(P.order >= 1 && P.order <= 3, "order must be 1, 2 or 3");
        EMS_CHECK_ARG(P.integrator == EMS_LEAPFROG || P.integrator == EMS_SYMP2 || P.integrator == EMS_SYMP4,
                      "hexahedral integrator must be EMS_LEAPFROG, EMS_SYMP2 or EMS_SYMP4");
        EMS_CHECK_ARG(P.precision == EMS_FP64 || P.precision == EMS_FP32, "precision must be EMS_FP64 or EMS_FP32");
        EMS_CHECK_ARG(P.h > 0 && P.dt > 0 && P.permittivity > 0 && P.permeability > 0, "h, dt, eps, mu must be positive");
        EMS_CHECK_ARG(P.time_frequency > 0, "time_frequency must be positive");
        int o = P.order;
        g.o = o; g.gx = P.grid[0]; g.gy = P.grid[1]; g.gz = P.grid[2];
        g.EX = g.gx / o; g.EY = g.gy / o; g.EZ = g.gz / o;
        // with fewer than two elements per direction the reference's outer
        // list visits boundary elements twice; such grids are rejected
        EMS_CHECK_ARG(g.EX >= 2 && g.EY >= 2 && g.EZ >= 2, "need at least two elements per direction");
        double c = 1.0 / std::sqrt(P.permittivity * P.permeability);
        EMS_CHECK_ARG(c * P.dt < P.h, "time step violates c*dt < h (reference check_params)");
        g.dof = o * (o + 1) * (o + 1);
        g.total = 3 * g.dof;
        g.nouter = 2 * g.EX * g.EY + 2 * g.EY * (g.EZ - 2) + 2 * (g.EZ - 2) * (g.EX - 2);
        g.nc[0] = (size_t)g.gx * (g.gy + 1) * (g.gz + 1);
        g.nc[1] = (size_t)(g.gx + 1) * g.gy * (g.gz + 1);
        g.nc[2] = (size_t)(g.gx + 1) * (g.gy + 1) * g.gz;
        for (int q = 0; q < 2; ++q) { g.row[q] = hex_div(g.gx + q); g.col[q] = hex_div(g.gy + q); }
        fp64 = P.precision == EMS_FP64;
        exact = fp64;
        // Order 3, grids beyond the two passes' 32-bit indices, and small FP64 grids of order 2
        one_pass = o == 3 || std::max(g.nc[0], std::max(g.nc[1], g.nc[2])) >= kHexDivLimit ||
                   (o == 2 && fp64 && (long long)g.EX * g.EY * g.EZ < kHex2MinElements);
        // element matrix (fem_v2/fem_simulation.cpp:458-490, symplectic_2 473)
        std::string fn = kdir + "/" + (P.use_ofem ? std::to_string(o) : "lamped" + std::to_string(o)) + ".csv";
        auto M = load_matrix_csv(fn);
        int T = g.total;
        if ((int)M.size() != T) throw Error{EMS_ERR_IO, fn + ": expected " + std::to_string(T) + " rows"};
        for (auto &r : M)
            if ((int)r.size() != T) throw Error{EMS_ERR_IO, fn + ": expected " + std::to_string(T) + " columns"};
        double scale;
        if (P.integrator == EMS_LEAPFROG)
            scale = 4.0 * P.dt * P.dt / (P.h * o) / (P.h * o) / P.permeability / P.permittivity / (8.0 / o / o / o);
        else
            scale = 4.0 / (P.h * o) / (P.h * o) / P.permeability / P.permittivity;
        Kh.resize((size_t)T * T);
        for (int i = 0; i < T; ++i)
            for (int j = 0; j < T; ++j) Kh[(size_t)i * T + j] = scale * M[i][j];
        if (o == 1 && fp64) {
            classes = true;
            for (int i = 0; i < 12; ++i)
                for (int j = 0; j < 12; ++j) {
                    const double k = Kh[12 * i + j];
                    double &size = cls.k[hex1_class(i, j)];
                    if (size == 0.0) size = std::fabs(k);
                    classes = classes && k != 0.0 && std::fabs(k) == size;
                    if (k < 0.0) cls.sign[i] |= 1u << j;
                }
        }
        init_stream();
        size_t w = fp64 ? 8 : 4;
        for (int q = 0; q < 3; ++q) { lev[q].alloc(3 * g.nc[q] * w); lev[q].zero(stream); }
        if (one_pass) {
            if (fp64) matrix_rows<double>(); else matrix_rows<float>();
        } else {
            if (fp64) upload_matrix<double>(); else upload_matrix<float>();
        }
        EMS_CUDA(cudaStreamSynchronize(stream));
    }

    template <class T> void upload(DevBuf &d, const std::vector<T> &k)
    {
        d.alloc(k.size() * sizeof(T));
        copy_in(d.p, k.data(), k.size() * sizeof(T));
    }
    // K as hex_elem_kernel takes it (orders 1 and 2)
    template <class T> void upload_matrix()
    {
        const int D = g.dof, TT = g.total, W = 16 / (int)sizeof(T), RP = (D + W - 1) / W * W;
        std::vector<T> k((size_t)3 * TT * RP, T(0));
        for (int r = 0; r < TT; ++r)
            for (int m = 0; m < TT; ++m) k[((size_t)(r / D) * TT + m) * RP + r % D] = (T)Kh[(size_t)r * TT + m];
        if constexpr (sizeof(T) == 4) k32 = std::move(k);
        else upload(dK, k);
    }
    // K row by row, for the one-pass kernels
    template <class T> const T *matrix_rows()
    {
        if (!dKr.p) upload(dKr, std::vector<T>(Kh.begin(), Kh.end()));
        return dKr.as<T>();
    }

    int flat(int c, const int *q) const
    {
        if (c == 0) return q[0] + q[1] * g.gx + q[2] * g.gx * (g.gy + 1);
        if (c == 1) return q[0] + q[1] * (g.gx + 1) + q[2] * (g.gx + 1) * g.gy;
        return q[0] + q[1] * (g.gx + 1) + q[2] * (g.gx + 1) * (g.gy + 1);
    }

    template <class T> T *L(int c, int level) const { return lev[c].as<T>() + (size_t)level * g.nc[c]; }

    template <class T, int O> void launch_leapfrog(const SrcList &s)
    {
        size_t mx = std::max(g.nc[0], std::max(g.nc[1], g.nc[2]));
        dim3 grid((unsigned)((mx + 127) / 128), 3);
        auto k = hex_leapfrog_kernel<T, O, sizeof(T) == 8>;
        k<<<grid, 128, 0, stream>>>(g, matrix_rows<T>(), L<T>(0, l1), L<T>(1, l1), L<T>(2, l1), L<T>(0, l0), L<T>(1, l0), L<T>(2, l0),
                                    L<T>(0, l2), L<T>(1, l2), L<T>(2, l2), s);
    }
    template <class T, int O> void launch_kick(T dt, const SrcList &s)
    {
        size_t mx = std::max(g.nc[0], std::max(g.nc[1], g.nc[2]));
        dim3 grid((unsigned)((mx + 127) / 128), 3);
        auto k = hex_kick_kernel<T, O, sizeof(T) == 8>;
        k<<<grid, 128, 0, stream>>>(g, matrix_rows<T>(), L<T>(0, 0), L<T>(1, 0), L<T>(2, 0), L<T>(0, 1), L<T>(1, 1), L<T>(2, 1),
                                    L<T>(0, 2), L<T>(1, 2), L<T>(2, 2), dt, s);
    }
    template <class T> void launch_drift(T coef, int pec)
    {
        size_t mx = std::max(g.nc[0], std::max(g.nc[1], g.nc[2]));
        dim3 grid((unsigned)((mx + 255) / 256), 3);
        const bool mul = g.o < 3;
        const T m = mul ? (T)(g.o * g.o * g.o / 8.0) : (T)(8.0 / g.o / g.o / g.o);
        auto k = mul ? hex_drift_kernel<T, sizeof(T) == 8, true> : hex_drift_kernel<T, sizeof(T) == 8, false>;
        launch_after(k, grid, dim3(256), 0, stream, g, L<T>(0, 0), L<T>(1, 0), L<T>(2, 0), L<T>(0, 1), L<T>(1, 1), L<T>(2, 1),
                     coef, m, pec);
    }

    SrcList sources(double val) const
    {
        SrcList s{};
        s.n = (int)srcs.size();
        for (int q = 0; q < s.n; ++q) { s.comp[q] = srcs[q][0]; s.idx[q] = srcs[q][1]; s.val[q] = val; }
        return s;
    }

    dim3 dof_grid() const
    {
        const size_t mx = std::max(g.nc[0], std::max(g.nc[1], g.nc[2]));
        return dim3((unsigned)((mx + 127) / 128), 3);
    }
    // The element values of the two passes (12 or 54 per element); a grid whose
    // fields leave no room for them takes the one-pass kernels.
    void make_fe()
    {
        if (one_pass) return;
        try {
            d_fe.ensure((size_t)g.total * g.EX * g.EY * g.EZ * (fp64 ? 8 : 4));
        } catch (const Error &e) {
            if (e.code != EMS_ERR_OUT_OF_MEMORY) throw;
            one_pass = true;
        }
    }
    int nsub() const { return P.integrator == EMS_SYMP4 ? 3 : 1; }
    void substeps(double sub[3], double off[3]) const
    {
        const double x1 = 1.0 / (2.0 - std::pow(2.0, 1.0 / 3.0)), x2 = 1.0 - 2.0 * x1;
        sub[0] = P.dt; off[0] = 0.0;
        if (P.integrator == EMS_SYMP4) { sub[0] = x1 * P.dt; sub[1] = x2 * P.dt; off[1] = x1 * P.dt; sub[2] = x1 * P.dt; off[2] = (x1 + x2) * P.dt; }
    }
    // The order-1 FP64 pass with one thread per element pays where the FP64 pipes
    // are full.  A leapfrog step of 4096 elements 12.4 us with it and 8.1 without,
    // 8000 12.9 and 12.0, 13824 13.6 and 15.6, 21952 15.5 and 19.8, 50061 28.0 and 35.9.
    static constexpr int kHex1MinElements = 10000;
    // In FP64 a warp of the order-2 element pass takes 65 us for its 1944
    // operations a thread (its quarter of the SM does one in 64 clocks), however few
    // warps there are.  DOF by DOF a small grid has more of them: leapfrog step of
    // 512 elements 24.6 us against 77, 2197 55 against 78, 2744 72 against 78,
    // 3375 87 against 78.
    static constexpr int kHex2MinElements = 3000;
    // Element pass of orders 1 and 2 over the level u; samp: with the sampling blocks
    template <class T, int O> void elements(T *const (&u)[3], bool first, bool samp)
    {
        constexpr bool X = sizeof(T) == 8;
        const int ne = g.EX * g.EY * g.EZ;
        const HexRec rec{samp ? nobs : 0, nsamp, P.time_frequency, d_obs.as<int>(), d_tr.as<double>()};
        int *step = first ? d_step.as<int>() : nullptr;
        if constexpr (X && O == 1)
            if (classes && ne >= kHex1MinElements) {
                launch_after(hex1_elem_kernel, dim3((ne + 31) / 32 + (rec.n + 31) / 32), dim3(32), 0, stream, g, cls, u[0],
                             u[1], u[2], d_fe.as<T>(), step, rec);
                return;
            }
        HexK<T, O> kk{};
        if constexpr (sizeof(T) == 4) std::copy(k32.begin(), k32.end(), kk.k);
        else kk.k = dK.as<T>();
        launch_after(hex_elem_kernel<T, O, X>, dim3((ne + 127) / 128 + (rec.n + 127) / 128, 3), dim3(128), 0, stream, g, kk,
                     u[0], u[1], u[2], d_fe.as<T>(), step, rec);
    }
    // One step of orders 1 and 2 in two passes per force; launches made.
    template <class T, int O> int enqueue_step()
    {
        int n = 0;
        const bool leap = P.integrator == EMS_LEAPFROG;
        if (nobs > 0 && !leap) {   // the symplectic steps sample U before the step
            launch_after(hex_sample_kernel<T>, dim3((nobs + 63) / 64), dim3(64), 0, stream, g, L<T>(0, 0), L<T>(1, 0),
                         L<T>(2, 0), nobs, d_obs.as<int>(), d_tr.as<double>(), nsamp, 0, d_step.as<int>(), P.time_frequency);
            ++n;
        }
        SrcTab src{};
        src.n = (int)srcs.size();
        src.nsub = nsub();
        for (int q = 0; q < src.n; ++q) { src.comp[q] = srcs[q][0]; src.idx[q] = srcs[q][1]; }
        src.vals = d_vals.as<double>();
        src.step = d_step.as<int>();
        constexpr bool X = sizeof(T) == 8;
        HexDofs<T> d;
        for (int c = 0; c < 3; ++c) {
            d.a[c] = L<T>(c, leap ? l1 : 0);
            d.b[c] = L<T>(c, leap ? l0 : 1);
            d.c[c] = L<T>(c, leap ? l2 : 2);
        }
        if (leap) {   // fem_v2 samples E^n, which the step leaves alone
            elements<T, O>(d.a, true, nobs > 0);
            launch_after(hex_leap_dof_kernel<T, O, X>, dof_grid(), dim3(128), 0, stream, g, d_fe.as<T>(), d, src);
            l0 = (l0 + 1) % 3; l1 = (l1 + 1) % 3; l2 = (l2 + 1) % 3;
            return n + 2;
        }
        double sub[3], off[3];
        substeps(sub, off);
        const int ns = nsub();
        launch_drift<T>((T)(0.5 * sub[0]), 0);
        for (int q = 0; q < ns; ++q) {
            elements<T, O>(d.a, q == 0, false);
            const bool last = q + 1 == ns;
            src.q = q;
            src.last = last;
            const T h1 = X || last ? (T)(0.5 * sub[q]) : (T)(0.5 * sub[q] + 0.5 * sub[q + 1]), h2 = X && !last ? (T)(0.5 * sub[q + 1]) : T(0);
            launch_after(hex_kick_dof_kernel<T, O, X>, dof_grid(), dim3(128), 0, stream, g, d_fe.as<T>(), d, src, (T)sub[q], h1,
                         h2, (T)(g.o * g.o * g.o / 8.0));
        }
        return n + 1 + 2 * ns;
    }
    template <class T, int O> long long run_two_pass(int nsteps, std::vector<double> &times)
    {
        const int ns = nsub();
        double sub[3], off[3];
        substeps(sub, off);
        std::vector<double> vals((size_t)std::max(nsteps, 1) * ns);
        double t = cur_time;
        for (int st = 0; st < nsteps; ++st) {
            if (st % P.time_frequency == 0) times[st / P.time_frequency] = t;
            for (int q = 0; q < ns; ++q)
                vals[(size_t)st * ns + q] = P.integrator == EMS_LEAPFROG
                    ? femv2_source(t) * P.dt * P.dt / P.permittivity / P.h / P.h / P.h
                    : femv2_source(t + off[q] + 0.5 * sub[q]) * 8.0 / P.permittivity / (P.h * g.o) / (P.h * g.o) / (P.h * g.o);
            t += P.dt;
        }
        d_vals.ensure(vals.size() * 8);
        d_step.ensure(2 * sizeof(int));
        EMS_CUDA(cudaMemcpyAsync(d_vals.p, vals.data(), vals.size() * 8, cudaMemcpyHostToDevice, stream));
        EMS_CUDA(cudaMemsetAsync(d_step.p, 0, 2 * sizeof(int), stream));
        EMS_CUDA(cudaStreamSynchronize(stream));   // vals ends here; the run's clock starts behind the copies
        EMS_CUDA(cudaEventRecord(ev0, stream));
        long long launches = 0;
        int step = 0;
        std::vector<unsigned long long> key = {(unsigned long long)nobs, (unsigned long long)nsamp, srcs.size()};
        for (const auto &q : srcs) { key.push_back((unsigned long long)q[0]); key.push_back((unsigned long long)q[1]); }
        for (const void *q : {d_fe.p, d_vals.p, d_step.p, d_obs.p, d_tr.p}) key.push_back((unsigned long long)reinterpret_cast<uintptr_t>(q));
        const bool kept = graph && key == graph_key;
        const int per = P.integrator == EMS_LEAPFROG ? 2 : 1 + 2 * ns + (nobs > 0);
        if (kept || key == last_key || nsteps * per >= kGraphMinLaunches) {
            for (; l0 != 0 && step < nsteps; ++step) launches += enqueue_step<T, O>();   // the graph's ring begins at level 0
            if (nsteps - step >= kGraphSteps) {
                if (!kept) {
                    if (graph) {
                        cudaGraphExecDestroy(graph);
                        graph = nullptr;
                    }
                    const cudaGraph_t gr = capture([&] {   // the ring ends where it began
                        for (int r = 0; r < kGraphSteps; ++r) graph_launches = enqueue_step<T, O>();
                    });
                    const cudaError_t e = cudaGraphInstantiate(&graph, gr, 0);
                    cudaGraphDestroy(gr);
                    EMS_CUDA(e);
                    graph_key = key;
                }
                for (; step + kGraphSteps <= nsteps; step += kGraphSteps) {
                    EMS_CUDA(cudaGraphLaunch(graph, stream));
                    launches += (long long)kGraphSteps * graph_launches;
                }
            }
        }
        last_key = std::move(key);
        for (; step < nsteps; ++step) launches += enqueue_step<T, O>();
        cur_time = t;
        return launches;
    }
    int graph_launches = 0;

    // Receivers from `level` into row s of the table.
    template <class T> void sample_level(int level, int s)
    {
        launch_after(hex_sample_kernel<T>, dim3((nobs + 63) / 64), dim3(64), 0, stream, g, L<T>(0, level), L<T>(1, level),
                     L<T>(2, level), nobs, d_obs.as<int>(), d_tr.as<double>(), nsamp, s, nullptr, 1);
    }
    // The run with the force DOF by DOF, launch by launch.
    template <class T, int O> long long run_one_pass(int nsteps, std::vector<double> &times)
    {
        const int tf = P.time_frequency, o = g.o;
        long long launches = 0;
        for (int step = 0; step < nsteps; ++step) {
            bool samp = nobs > 0 && step % tf == 0;
            if (P.integrator == EMS_LEAPFROG) {
                // fem_v2 samples level 1 (E^n) after computing E^{n+1}; E^n is untouched by the step
                if (samp) {
                    sample_level<T>(l1, step / tf);
                    times[step / tf] = cur_time;
                    ++launches;
                }
                double sv = femv2_source(cur_time) * P.dt * P.dt / P.permittivity / P.h / P.h / P.h;
                launch_leapfrog<T, O>(sources(sv));
                ++launches;
                l0 = (l0 + 1) % 3; l1 = (l1 + 1) % 3; l2 = (l2 + 1) % 3;
            } else {
                if (samp) {
                    sample_level<T>(0, step / tf);
                    times[step / tf] = cur_time;
                    ++launches;
                }
                double sub[3], off[3];
                substeps(sub, off);
                const int ns = nsub();
                for (int q = 0; q < ns; ++q) {
                    double deltat = sub[q];
                    double sv = femv2_source(cur_time + off[q] + 0.5 * deltat) * 8.0 / P.permittivity / (P.h * o) / (P.h * o) / (P.h * o);
                    if (exact || q == 0) launch_drift<T>((T)(0.5 * deltat), 0), ++launches;
                    launch_kick<T, O>((T)deltat, sources(sv));
                    ++launches;
                    if (exact || q == ns - 1) launch_drift<T>((T)(0.5 * deltat), 1);
                    else launch_drift<T>((T)(0.5 * deltat + 0.5 * sub[q + 1]), 1);
                    ++launches;
                }
            }
            cur_time += P.dt;
        }
        return launches;
    }

    template <class T, int O> void run_o(int nsteps)
    {
        const int tf = P.time_frequency;
        nobs = (int)obs_idx.size();
        nsamp = nsteps > 0 ? (nsteps - 1) / tf + 1 : 0;
        ncols = 4;
        std::vector<int> oi;
        for (auto &q : obs_idx) { oi.push_back(q[0]); oi.push_back(q[1]); oi.push_back(q[2]); }
        if (oi.empty()) oi.assign(3, 0);
        d_obs.ensure(oi.size() * 4);
        EMS_CUDA(cudaMemcpyAsync(d_obs.p, oi.data(), oi.size() * 4, cudaMemcpyHostToDevice, stream));
        size_t ntr = (size_t)std::max(nobs, 1) * std::max(nsamp, 1) * 4;
        d_tr.ensure(ntr * 8);
        d_tr.zero(stream);
        std::vector<double> times(std::max(nsamp, 1), 0.0);
        long long launches = 0;
        make_fe();
        EMS_CUDA(cudaEventRecord(ev0, stream));
        if constexpr (O <= 2) launches = one_pass ? run_one_pass<T, O>(nsteps, times) : run_two_pass<T, O>(nsteps, times);
        else launches = run_one_pass<T, O>(nsteps, times);
        EMS_CUDA(cudaGetLastError());
        EMS_CUDA(cudaEventRecord(ev1, stream));
        EMS_CUDA(cudaStreamSynchronize(stream));
        float ms = 0;
        EMS_CUDA(cudaEventElapsedTime(&ms, ev0, ev1));
        last_ms = ms;
        last_launches = launches;
        traces.assign(ntr, 0.0);
        EMS_CUDA(cudaMemcpy(traces.data(), d_tr.p, ntr * 8, cudaMemcpyDeviceToHost));
        traces.resize((size_t)nobs * nsamp * 4);
        for (int ob = 0; ob < nobs; ++ob)
            for (int s = 0; s < nsamp; ++s) traces[((size_t)ob * nsamp + s) * 4] = times[s];
    }

    template <class T> void run_t(int nsteps)
    {
        if (g.o == 1) run_o<T, 1>(nsteps);
        else if (g.o == 2) run_o<T, 2>(nsteps);
        else run_o<T, 3>(nsteps);
    }

    void run(int nsteps) override
    {
        EMS_CHECK_ARG(nsteps >= 0, "num_steps must be >= 0");
        EMS_CHECK_ARG(srcs.size() <= (size_t)kMaxSrc, "at most 8 point sources");
        if (fp64) run_t<double>(nsteps); else run_t<float>(nsteps);
        const size_t w = fp64 ? 8 : 4;
        check_finite({{lev[0].p, lev[0].bytes / w}, {lev[1].p, lev[1].bytes / w}, {lev[2].p, lev[2].bytes / w}}, fp64);
    }

    size_t field_size(int which) const override
    {
        if (which < 0 || which > 2) throw Error{EMS_ERR_INVALID_ARGUMENT, "field index must be 0..2 (x, y, z components)"};
        return 3 * g.nc[which];
    }
    // levels returned in the reference's storage order (ring index 0,1,2)
    void get_field(int which, double *out) const override
    {
        const size_t cnt = field_size(which);
        if (fp64) download(out, lev[which].as<double>(), cnt);
        else
            download(out, cnt, [&](size_t at, size_t n, double *dst) {
                hex_widen_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(lev[which].as<float>() + at, dst, n);
            });
    }
    void set_field(int which, const double *in) override
    {
        size_t cnt = field_size(which);
        if (fp64) {
            copy_in(lev[which].p, in, cnt * 8);
        } else {
            std::vector<float> tmp(in, in + cnt);
            copy_in(lev[which].p, tmp.data(), cnt * 4);
        }
    }

    // fem_v2/fem_simulation.cpp:1322-1344: setprecision(15) scientific,
    // header time,Ex,Ey,Ez.  The reference writes every receiver to the same
    // name; here receiver i > 0 gets the suffix _<i> before the extension.
    void save(const char *path) const override
    {
        EMS_CHECK_ARG(path && *path, "file name required");
        for (int o = 0; o < nobs; ++o) {
            std::string fn = path;
            if (o > 0) {
                size_t dot = fn.rfind('.');
                std::string suf = "_" + std::to_string(o);
                if (dot == std::string::npos) fn += suf; else fn.insert(dot, suf);
            }
            std::ofstream f(fn);
            if (!f.is_open()) throw Error{EMS_ERR_IO, "cannot open " + fn};
            f << std::setprecision(15) << std::scientific;
            f << "time,Ex,Ey,Ez" << std::endl;
            for (int s = 0; s < nsamp; ++s) {
                const double *r = &traces[((size_t)o * nsamp + s) * 4];
                f << r[0] << "," << r[1] << "," << r[2] << "," << r[3] << std::endl;
            }
        }
    }

    void reset() override
    {
        for (int q = 0; q < 3; ++q) lev[q].zero(stream);
        l0 = 0; l1 = 1; l2 = 2;
        cur_time = 0.0;
        EMS_CUDA(cudaStreamSynchronize(stream));
    }

    void time_dominant(int launches, double *ms, double *bytes, std::string *name) override
    {
        size_t w = fp64 ? 8 : 4;
        size_t ndof = g.nc[0] + g.nc[1] + g.nc[2];
        std::vector<DevBuf> save(3);
        for (int q = 0; q < 3; ++q) {
            save[q].alloc(lev[q].bytes);
            EMS_CUDA(cudaMemcpyAsync(save[q].p, lev[q].p, lev[q].bytes, cudaMemcpyDeviceToDevice, stream));
        }
        make_fe();
        auto body = [&](auto tag) {
            using T = decltype(tag);
            SrcList s = sources(0.0);
            for (int r = 0; r <= launches; ++r) {
                if (r == 1) EMS_CUDA(cudaEventRecord(ev0, stream));
                auto go = [&](auto oc) {
                    constexpr int O = decltype(oc)::value;
                    if constexpr (O <= 2)
                        if (!one_pass) {
                            T *u[3];
                            for (int c = 0; c < 3; ++c) u[c] = L<T>(c, P.integrator == EMS_LEAPFROG ? l1 : 0);
                            elements<T, O>(u, false, false);
                            return;
                        }
                    if (P.integrator == EMS_LEAPFROG) launch_leapfrog<T, O>(s); else launch_kick<T, O>((T)P.dt, s);
                };
                if (g.o == 1) go(std::integral_constant<int, 1>());
                else if (g.o == 2) go(std::integral_constant<int, 2>());
                else go(std::integral_constant<int, 3>());
            }
        };
        if (fp64) body(double()); else body(float());
        EMS_CUDA(cudaEventRecord(ev1, stream));
        EMS_CUDA(cudaStreamSynchronize(stream));
        float t = 0;
        EMS_CUDA(cudaEventElapsedTime(&t, ev0, ev1));
        for (int q = 0; q < 3; ++q)
            EMS_CUDA(cudaMemcpyAsync(lev[q].p, save[q].p, lev[q].bytes, cudaMemcpyDeviceToDevice, stream));
        EMS_CUDA(cudaStreamSynchronize(stream));
        *ms = t / launches;
        // element pass: read U, write the element values; one-pass leapfrog: read E^n, E^{n-1}, write
        // E^{n+1}; kick: read U, read/write P, write F
        *bytes = one_pass ? (double)ndof * w * (P.integrator == EMS_LEAPFROG ? 3.0 : 4.0)
                          : w * ((double)ndof + (double)g.total * g.EX * g.EY * g.EZ);
        *name = std::string(one_pass ? (P.integrator == EMS_LEAPFROG ? "hex_leapfrog_kernel" : "hex_kick_kernel")
                                     : classes && g.EX * g.EY * g.EZ >= kHex1MinElements ? "hex1_elem_kernel" : "hex_elem_kernel") +
                "<o=" + std::to_string(g.o) + ">";
    }
};

Sim *make_hexfem(const ems_hexfem_params *p) { return new HexFemSim(p); }

void hexfem_set_source(Sim *s, int comp, const int ijk[3])
{
    auto *f = static_cast<HexFemSim *>(s);
    EMS_CHECK_ARG(comp >= 0 && comp < 3 && ijk, "component must be 0, 1 or 2");
    int lim[3] = {f->g.gx - (comp == 0), f->g.gy - (comp == 1), f->g.gz - (comp == 2)};
    for (int d = 0; d < 3; ++d) EMS_CHECK_ARG(ijk[d] >= 0 && ijk[d] <= lim[d], "source edge outside the grid");
    EMS_CHECK_ARG(f->srcs.size() < (size_t)kMaxSrc, "at most 8 point sources");
    f->srcs.push_back({comp, f->flat(comp, ijk), 0, 0});
}

void hexfem_add_observation(Sim *s, const int ijk[3])
{
    auto *f = static_cast<HexFemSim *>(s);
    EMS_CHECK_ARG(ijk != nullptr, "position required");
    // the sample reads x-edges (i-1..i, j, k..k+1), y-edges (i, j-1..j, k..k+1), z-edge (i,j,k)
    EMS_CHECK_ARG(ijk[0] >= 1 && ijk[0] < f->g.gx && ijk[1] >= 1 && ijk[1] < f->g.gy && ijk[2] >= 0 && ijk[2] < f->g.gz,
                  "observation point must be an interior node");
    f->obs_idx.push_back({f->flat(0, ijk), f->flat(1, ijk), f->flat(2, ijk)});
    f->obs_ijk.push_back({ijk[0], ijk[1], ijk[2]});
}

}  // namespace ems
