// Yee FDTD on one GPU: the reference time loop of fdtd/fdtd_simulation.cpp
// (H from curl E 119-169, E from curl H 170-220, sources 222-239, receivers
// 261-303), extended with per-cell materials and a convolutional PML.
//
// The API shows the reference's padded field layout (55-88).  On the device
// all fields share one pitched layout, so one offset addresses them all and a
// thread moves 16 bytes (4 FP32 or 2 FP64 cells along x) per access: rows of
// `pitch` values, planes of ny + 2 rows, and the components that the
// reference pads in x (Ey, Ez) stored one column to the left, next to the H
// cell that reads them.
//
// Arithmetic is written with explicitly rounded operations (no contraction
// into fused multiply-adds) in the reference's operand order, so the FP64
// path reproduces the reference bit for bit; the FP32 path runs the same
// operations in single precision.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <sstream>
#include <iomanip>

#include "ems_internal.hpp"

namespace ems {

__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }

// CPML coefficient profile along one axis, sampled at the derivative
// positions; the layer is off for lo <= s < hi.  (The x profile of the E-type
// derivatives starts at s = 1, as the columns of Ey and Ez do.)
template <class T> struct Prof {
    const T *b, *a, *kinv;
    int lo, hi;
    __device__ __forceinline__ bool on(int s) const { return s < lo || s >= hi; }
};

// (ca, cb) of one material, loaded as one vector.
template <class T> struct alignas(2 * sizeof(T)) CaCb {
    T ca, cb;
};

template <class T> struct FdtdArgs {
    T *Ex, *Ey, *Ez, *Hx, *Hy, *Hz;   // the first column of row 0, plane 0
    int nx, ny, nz;
    // threads per row (V cells each): [g0, g1) touch no x layer and run in the
    // first blocks of a launch, the gr others in the blocks behind them
    int g0, g1, gr;
    unsigned magic[2], shift[2];   // t / (g1 - g0) and t / gr as (t * magic) >> shift (see divider)
    unsigned pitch;                // values per row
    size_t plane;                  // values per plane
    T ch, ce;                      // uniform update coefficients dt/mu/h, dt/eps/h
    const uint16_t *mat;           // per-cell material id (MAT), rows of mpitch, the last column repeated
    unsigned mpitch;
    const CaCb<T> *cab;            // per-material E coefficients (MAT)
    Prof<T> pe[3], ph[3];          // CPML profiles for E- and H-type derivatives (PML)
    T *psiE[3][2], *psiH[3][2];    // CPML auxiliary fields in the fields' layout (PML)
};

// 16 bytes of consecutive cells.
template <class T> struct Vec {
    static constexpr int V = 16 / sizeof(T);
    T v[V];
};
__device__ __forceinline__ void vload(Vec<float> &r, const float *p)
{
    const float4 t = *reinterpret_cast<const float4 *>(p);
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
}
__device__ __forceinline__ void vload(Vec<double> &r, const double *p)
{
    const double2 t = *reinterpret_cast<const double2 *>(p);
    r.v[0] = t.x; r.v[1] = t.y;
}
// the n first values (all of them in one store)
__device__ __forceinline__ void vstore(float *p, const Vec<float> &r, int n)
{
    if (n >= 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
        return;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (q < n) p[q] = r.v[q];
}
__device__ __forceinline__ void vstore(double *p, const Vec<double> &r, int n)
{
    if (n >= 2) *reinterpret_cast<double2 *>(p) = make_double2(r.v[0], r.v[1]);
    else if (n == 1) p[0] = r.v[0];
}
__device__ __forceinline__ void mload(unsigned (&m)[4], const uint16_t *p)
{
    const ushort4 t = *reinterpret_cast<const ushort4 *>(p);
    m[0] = t.x; m[1] = t.y; m[2] = t.z; m[3] = t.w;
}
__device__ __forceinline__ void mload(unsigned (&m)[2], const uint16_t *p)
{
    const ushort2 t = *reinterpret_cast<const ushort2 *>(p);
    m[0] = t.x; m[1] = t.y;
}

// Sources and receiver samples that the E kernel serves itself: the entries
// of plane k are list[plane[k]] .. list[plane[k + 1] - 1] in order of their
// offset, those of one place as they were added, sources before samples.  A
// launch belongs to step *base + step.
struct FdtdPoint {
    long long off;  // offset in the component's array
    int comp;       // component, + 4 for a receiver sample
    int idx;        // source number, or place of the sample in a row of samp
};
struct FdtdPoints {
    const int *plane;        // null: no points
    const FdtdPoint *list;
    const double *vals;      // [step - 1][ns] source values
    double *samp;            // [row][nsm] sampled values
    const int *base;
    int step, ns, nsm, tf;
};

// d = ((p - q) - r) + s, the reference's evaluation order of a curl difference.
template <class T> __device__ __forceinline__ T curl4(T p, T q, T r, T s) { return radd(rsub(rsub(p, q), r), s); }

// The CPML along one axis on the cells of a thread: t = kinv d and the new
// psi = b psi + a d; without a layer (kind 0) t = d and nothing moves.  kind 1:
// all cells at position s; kind 2: the cells run along the axis from s.
template <class T>
__device__ __forceinline__ void layer(int kind, const Vec<T> &d, const Prof<T> &p, int s, T *psi, Vec<T> &t, Vec<T> &q)
{
    constexpr int V = Vec<T>::V;
    if (kind == 0) {
#pragma unroll
        for (int v = 0; v < V; ++v) { t.v[v] = d.v[v]; q.v[v] = T(0); }
        return;
    }
    Vec<T> b, a, k;
    vload(q, psi);
    if (kind == 2) {
        vload(b, p.b + s);
        vload(a, p.a + s);
        vload(k, p.kinv + s);
    } else {
        b.v[0] = p.b[s]; a.v[0] = p.a[s]; k.v[0] = p.kinv[s];
#pragma unroll
        for (int v = 1; v < V; ++v) { b.v[v] = b.v[0]; a.v[v] = a.v[0]; k.v[v] = k.v[0]; }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
        q.v[v] = radd(rmul(b.v[v], q.v[v]), rmul(a.v[v], d.v[v]));
        t.v[v] = rmul(k.v[v], d.v[v]);
    }
    vstore(psi, q, V);
}

// Curl differences of the cells of a thread: ((p - q) - r) + s, or in a layer
// of either axis kinv1 d1 - kinv2 d2 + psi1 - psi2 with d1 = p - q, d2 = r - s
// (oracle/orc_fdtd.c order; the auxiliary value of an axis without a layer
// is zero and is not touched).  xm: the cells inside the x layer.
template <class T, bool PML>
__device__ __forceinline__ Vec<T> curl_vec(const Vec<T> &p, const Vec<T> &q, const Vec<T> &r, const Vec<T> &s, int k1, const Prof<T> &p1, int s1,
                                           T *psi1, int k2, const Prof<T> &p2, int s2, T *psi2, unsigned xm)
{
    constexpr int V = Vec<T>::V;
    Vec<T> c;
#pragma unroll
    for (int v = 0; v < V; ++v) c.v[v] = curl4(p.v[v], q.v[v], r.v[v], s.v[v]);
    if (PML && (k1 | k2)) {
        Vec<T> d1, d2, t1, t2, q1, q2;
#pragma unroll
        for (int v = 0; v < V; ++v) { d1.v[v] = rsub(p.v[v], q.v[v]); d2.v[v] = rsub(r.v[v], s.v[v]); }
        layer(k1, d1, p1, s1, psi1, t1, q1);
        layer(k2, d2, p2, s2, psi2, t2, q2);
        const bool all = k1 == 1 || k2 == 1;
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (all || ((xm >> v) & 1)) c.v[v] = rsub(radd(rsub(t1.v[v], t2.v[v]), q1.v[v]), q2.v[v]);
    }
    return c;
}

// Bits of the cells i .. i + V - 1 inside the x layer.
template <class T> __device__ __forceinline__ unsigned x_bits(const Prof<T> &p, int i)
{
    unsigned m = 0;
#pragma unroll
    for (int v = 0; v < Vec<T>::V; ++v)
        if (p.on(i + v)) m |= 1u << v;
    return m;
}
// The cells of a thread: V columns from i of row j, plane k (false: none).
// Threads run through the rows of a plane without a break, so short rows fill
// the warps too.  The columns near an x layer (xl) have blocks of their own:
// in one warp with the others they made nearly every warp of a row of 400
// cells run the layer's code (400 x 384 x 368 FP32: 72.0 ms for 60 steps).
template <class T>
__device__ __forceinline__ bool fdtd_cells(const FdtdArgs<T> &a, int kz, unsigned mblocks, int &i, int &j, int &k, size_t &o, bool &xl)
{
    xl = blockIdx.x >= mblocks;
    const unsigned t = (blockIdx.x - (xl ? mblocks : 0)) * (blockDim.x * blockDim.y) + threadIdx.y * blockDim.x + threadIdx.x;
    const unsigned row = (unsigned)(((unsigned long long)t * a.magic[xl]) >> a.shift[xl]);
    int g = (int)(t - row * (xl ? a.gr : a.g1 - a.g0));
    if (!xl) g += a.g0;
    else if (g >= a.g0) g += a.g1 - a.g0;
    j = (int)row;
    i = g * Vec<T>::V;
    k = kz + blockIdx.z;
    o = (size_t)k * a.plane + (size_t)row * a.pitch + i;
    return j <= a.ny;
}

// H from curl E: fdtd_simulation.cpp:119-169.  Every load of the thread is
// issued before its first store.  Bound by DRAM on large grids: per cell and
// step 18 values of E and H move, 9 of them here.
template <class T, bool PML>
__global__ void __launch_bounds__(256) fdtd_h_kernel(FdtdArgs<T> a, int kz, unsigned mblocks, int *ctr, int inc)
{
    constexpr int V = Vec<T>::V;
    wait_for_last();
    // the step counter of a replayed graph, moved on by its first launch (the H kernels do not read it)
    if (ctr && blockIdx.x == 0 && blockIdx.z == 0 && threadIdx.x == 0 && threadIdx.y == 0) *ctr += inc;
    int i, j, k;
    size_t o;
    bool xl;
    if (!fdtd_cells(a, kz, mblocks, i, j, k, o, xl)) return;
    const size_t oy = o + a.pitch, oz = o + a.plane;
    const bool hy = j < a.ny, hz = k < a.nz;
    const int nx = min(V, a.nx - i), n = min(V, a.nx + 1 - i);   // valid cells of Hx, and of Hy and Hz
    Vec<T> z11, z1, y1k, y1, x1k, x1, x0, h0, h1, h2, z0, y0;
    vload(z11, a.Ez + oy);                 // Ez(i+1, j+1, k)
    vload(z1, a.Ez + o);                   // Ez(i+1, j, k)
    vload(y1k, a.Ey + oz);                 // Ey(i+1, j, k+1)
    vload(y1, a.Ey + o);                   // Ey(i+1, j, k)
    vload(x1k, a.Ex + oz + a.pitch);       // Ex(i, j+1, k+1)
    vload(x1, a.Ex + oy);                  // Ex(i, j+1, k)
    vload(x0, a.Ex + oz);                  // Ex(i, j, k+1)
    z0.v[0] = a.Ez[(ptrdiff_t)oy - 1];     // Ez(i, j+1, k)
    y0.v[0] = a.Ey[(ptrdiff_t)oz - 1];     // Ey(i, j, k+1)
    vload(h0, a.Hx + o);
    vload(h1, a.Hy + o);
    vload(h2, a.Hz + o);
#pragma unroll
    for (int v = 1; v < V; ++v) {
        z0.v[v] = z11.v[v - 1];
        y0.v[v] = y1k.v[v - 1];
    }
    const unsigned xm = PML && xl ? x_bits(a.ph[0], i) : 0;
    const int kx = xm ? 2 : 0, ky = PML && a.ph[1].on(j) ? 1 : 0, kk = PML && a.ph[2].on(k) ? 1 : 0;
    if (nx > 0) {
        const Vec<T> c = curl_vec<T, PML>(z11, z1, y1k, y1, ky, a.ph[1], j, a.psiH[0][0] + o, kk, a.ph[2], k, a.psiH[0][1] + o, 0);
#pragma unroll
        for (int v = 0; v < V; ++v) h0.v[v] = rsub(h0.v[v], rmul(a.ch, c.v[v]));
        vstore(a.Hx + o, h0, nx);
    }
    if (hy) {
        const Vec<T> c = curl_vec<T, PML>(x1k, x1, z11, z0, kk, a.ph[2], k, a.psiH[1][0] + o, kx, a.ph[0], i, a.psiH[1][1] + o, xm);
#pragma unroll
        for (int v = 0; v < V; ++v) h1.v[v] = rsub(h1.v[v], rmul(a.ch, c.v[v]));
        vstore(a.Hy + o, h1, n);
    }
    if (hz) {
        const Vec<T> c = curl_vec<T, PML>(y1k, y0, x1k, x0, kx, a.ph[0], i, a.psiH[2][0] + o, ky, a.ph[1], j, a.psiH[2][1] + o, xm);
#pragma unroll
        for (int v = 0; v < V; ++v) h2.v[v] = rsub(h2.v[v], rmul(a.ch, c.v[v]));
        vstore(a.Hz + o, h2, n);
    }
}

// (ca, cb) of one material through the read-only path.
__device__ __forceinline__ CaCb<float> load_cab(const CaCb<float> *p)
{
    const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ CaCb<double> load_cab(const CaCb<double> *p)
{
    const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
    return {v.x, v.y};
}

// ca E + cb c with the cells' materials, or E + ce c without (ca = 1 multiplies exactly)
template <class T, bool MAT>
__device__ __forceinline__ void e_update(const FdtdArgs<T> &a, Vec<T> &e, const Vec<T> &c, const CaCb<T> (&m)[Vec<T>::V])
{
#pragma unroll
    for (int v = 0; v < Vec<T>::V; ++v)
        e.v[v] = MAT ? radd(rmul(m[v].ca, e.v[v]), rmul(m[v].cb, c.v[v])) : radd(e.v[v], rmul(a.ce, c.v[v]));
}
// The coefficients of the cells with ids at p; mostly one material, loaded once.
template <class T> __device__ __forceinline__ void e_material(const FdtdArgs<T> &a, const uint16_t *p, CaCb<T> (&m)[Vec<T>::V])
{
    unsigned id[Vec<T>::V];
    mload(id, p);
#pragma unroll
    for (int v = 0; v < Vec<T>::V; ++v) m[v] = load_cab(a.cab + id[v]);
}

// E from curl H: fdtd_simulation.cpp:170-220.  As in the H update, all loads
// of the thread are issued before the first store.  The plane's points then
// act on the updated values before they are stored: a launch for the sources
// and one for the receivers would cost more than a small grid's updates
// (64^3 FP64: 44.1 us a step with them, 30.5 without).
template <class T, bool MAT, bool PML>
__global__ void __launch_bounds__(256) fdtd_e_kernel(FdtdArgs<T> a, FdtdPoints pt, int kz, unsigned mblocks)
{
    constexpr int V = Vec<T>::V;
    int i, j, k;
    size_t o;
    bool xl;
    if (!fdtd_cells(a, kz, mblocks, i, j, k, o, xl)) return;
    const bool jn = j >= 1, kn = k >= 1;
    const size_t py = a.pitch, pz = a.plane;
    const int n = min(V, a.nx + 1 - i), nyz = min(V, a.nx - i);   // valid cells of Ex, and of Ey and Ez
    const bool ex = jn && kn, ey = kn && nyz > 0, ez = jn && nyz > 0;
    Vec<T> e0{}, e1{}, e2{}, zk{}, zjk{}, yj{}, yjk{}, xi{}, xik{}, xij{}, zk1{}, yj1{};
    CaCb<T> c0[V], c1[V], c2[V];
    wait_for_last();
    if (kn) {
        vload(zk, a.Hz + o - pz);                       // Hz(i, j, k-1)
        vload(xik, a.Hx + o - pz);                      // Hx(i, j, k-1)
        zk1.v[V - 1] = a.Hz[o - pz + V];
    }
    if (jn) {
        vload(yj, a.Hy + o - py);                       // Hy(i, j-1, k)
        vload(xij, a.Hx + o - py);                      // Hx(i, j-1, k)
        yj1.v[V - 1] = a.Hy[o - py + V];
    }
    vload(xi, a.Hx + o);                                // Hx(i, j, k)
    if (ex) {
        vload(zjk, a.Hz + o - py - pz);
        vload(yjk, a.Hy + o - py - pz);
        vload(e0, a.Ex + o);
    }
    if (ey) vload(e1, a.Ey + o);
    if (ez) vload(e2, a.Ez + o);
    if (MAT) {   // Ex(i,j,k) -> cell (min(i,nx-1), j-1, k-1), Ey -> (i-1, min(j,ny-1), k-1), Ez -> (i-1, j-1, min(k,nz-1))
        const size_t mrow = a.mpitch, mpl = mrow * a.ny;
        if (ex) e_material(a, a.mat + (j - 1) * mrow + (k - 1) * mpl + i, c0);
        if (ey) e_material(a, a.mat + min(j, a.ny - 1) * mrow + (k - 1) * mpl + i, c1);
        if (ez) e_material(a, a.mat + (j - 1) * mrow + min(k, a.nz - 1) * mpl + i, c2);
    }
#pragma unroll
    for (int v = 0; v < V - 1; ++v) {
        zk1.v[v] = zk.v[v + 1];                         // Hz(i+1, j, k-1)
        yj1.v[v] = yj.v[v + 1];                         // Hy(i+1, j-1, k)
    }
    const unsigned xm = PML && xl ? x_bits(a.pe[0], i) : 0;
    const int kx = xm ? 2 : 0, ky = PML && a.pe[1].on(j) ? 1 : 0, kk = PML && a.pe[2].on(k) ? 1 : 0;
    if (ex) {
        const Vec<T> c = curl_vec<T, PML>(zk, zjk, yj, yjk, ky, a.pe[1], j, a.psiE[0][0] + o, kk, a.pe[2], k, a.psiE[0][1] + o, 0);
        e_update<T, MAT>(a, e0, c, c0);
    }
    if (ey) {
        const Vec<T> c = curl_vec<T, PML>(xi, xik, zk1, zk, kk, a.pe[2], k, a.psiE[1][0] + o, kx, a.pe[0], i, a.psiE[1][1] + o, xm);
        e_update<T, MAT>(a, e1, c, c1);
    }
    if (ez) {
        const Vec<T> c = curl_vec<T, PML>(yj1, yj, xi, xij, kx, a.pe[0], i, a.psiE[2][0] + o, ky, a.pe[1], j, a.psiE[2][1] + o, xm);
        e_update<T, MAT>(a, e2, c, c2);
    }
    if (pt.plane) {
        const int q1 = __ldg(pt.plane + k + 1);
        int q = __ldg(pt.plane + k);
        for (int end = q1; end - q > 4;) {   // close to the first point at the thread's cells or behind them
            const int mid = (q + end) >> 1;
            if (pt.list[mid].off < (long long)o) q = mid + 1; else end = mid;
        }
        for (; q < q1; ++q) {
            const FdtdPoint r = pt.list[q];
            const long long at = r.off - (long long)o;
            if (at >= V) break;
            const int comp = r.comp & 3;
            if (at < 0 || !(comp == 0 ? ex : comp == 1 ? ey : ez)) continue;
            const int step = pt.step + (pt.base ? *pt.base : 0);
            const bool sample = r.comp >= 4, keep = sample && step % pt.tf == 0;
            const T src = sample ? T(0) : (T)pt.vals[(size_t)(step - 1) * pt.ns + r.idx];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if (v != at) continue;
                const T e = comp == 0 ? e0.v[v] : comp == 1 ? e1.v[v] : e2.v[v];
                if (keep) pt.samp[(size_t)(step / pt.tf) * pt.nsm + r.idx] = (double)e;
                if (sample) continue;
                if (comp == 0) e0.v[v] = rsub(e, src);
                else if (comp == 1) e1.v[v] = rsub(e, src);
                else e2.v[v] = rsub(e, src);
            }
        }
    }
    if (ex) vstore(a.Ex + o, e0, n);
    if (ey) vstore(a.Ey + o, e1, nyz);
    if (ez) vstore(a.Ez + o, e2, nyz);
}

// n values of one component from `at` on between the device layout and the
// API's array (rows of w values, ah rows per plane).
template <class T, bool GET>
__global__ void fdtd_field_kernel(T *f, double *api, size_t at, size_t n, int w, int ah, size_t pitch, size_t plane, int shift)
{
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x, t = at + q;
    if (q >= n) return;
    const size_t r = t / w;
    const ptrdiff_t o = (ptrdiff_t)((r / ah) * plane + (r % ah) * pitch + t % w) - shift;
    if (GET) api[q] = (double)f[o];
    else f[o] = (T)api[q];
}
// Material ids into rows of mpitch, the last column repeated, zero behind it.
__global__ void fdtd_mat_kernel(const uint16_t *id, uint16_t *mat, size_t cnt, unsigned mpitch, int nx)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= cnt) return;
    const size_t r = t / mpitch;
    const int i = (int)(t - r * mpitch);
    mat[t] = i <= nx ? id[r * nx + min(i, nx - 1)] : (uint16_t)0;
}

// Point sources in insertion order: E[src] -= v (fdtd_simulation.cpp:222-239).
template <class T>
__global__ void fdtd_source_kernel(T *Ex, T *Ey, T *Ez, const int *comp, const long long *off, const double *vals, int nsrc)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (int s = 0; s < nsrc; ++s) {
        T *f = comp[s] == 0 ? Ex : comp[s] == 1 ? Ey : Ez;
        f[off[s]] = rsub(f[off[s]], (T)vals[s]);
    }
}

// Receiver averages (fdtd_simulation.cpp:261-303): one thread per receiver,
// summing its listed samples in order, then dividing by the count.
template <class T>
__global__ void fdtd_receiver_kernel(const T *Ex, const T *Ey, const T *Ez, int nobs, const int *cnt,
                                     const int *start, const long long *off, double *trace_row, int nsamp)
{
    int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= nobs) return;
    double *out = trace_row + (size_t)o * nsamp * 3;
    int q = start[o];
    for (int c = 0; c < 3; ++c) {
        const T *f = c == 0 ? Ex : c == 1 ? Ey : Ez;
        int n = cnt[3 * o + c];
        double acc = out[c];
        for (int r = 0; r < n; ++r, ++q) acc = __dadd_rn(acc, (double)f[off[q]]);
        out[c] = acc / (double)n;
    }
}

// The same averages from the values that the E kernel sampled: one thread per
// receiver and sampled step (row 0, the start, stays zero).
__global__ void fdtd_trace_kernel(const double *samp, int nsm, int nobs, const int *cnt, const int *start, double *traces, int nsamp)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int row = (int)(t % nsamp), o = (int)(t / nsamp);
    if (o >= nobs || row == 0) return;
    const double *v = samp + (size_t)row * nsm + start[o];
    double *out = traces + ((size_t)o * nsamp + row) * 3;
    for (int c = 0; c < 3; ++c) {
        const int n = cnt[3 * o + c];
        double acc = 0.0;
        for (int r = 0; r < n; ++r) acc = __dadd_rn(acc, *v++);
        out[c] = acc / (double)n;
    }
}

double fdtd_source_value(int kind, double f0, double t, double h)
{
    if (kind == EMS_WAVE_REFERENCE)
        return -4.0 * M_PI * M_PI * f0 * f0 * (t - 1.0 / f0) *
               std::exp(-2.0 * M_PI * M_PI * f0 * f0 * (t - 1.0 / f0) * (t - 1.0 / f0)) / h / h / h * 0.001;
    double tau = t - std::sqrt(2.0) / f0;
    return (1.0 - 2.0 * M_PI * M_PI * f0 * f0 * tau * tau) * std::exp(-M_PI * M_PI * f0 * f0 * tau * tau) / h / h / h * 0.001;
}

struct FdtdSource {
    int comp;
    int ijk[3];
    int kind;
    double f0, amp;
    long long off;
};

struct FdtdSim : Sim {
    ems_fdtd_params P;
    int nx, ny, nz;
    bool fp64;
    size_t n[6];
    // device layout (see the head of the file): each array `lead` values in
    int V, lead;
    size_t pitch, plane, total, mpitch;
    int g0, g1;                 // threads of a row [g0, g1) that touch no x layer
    DevBuf F[6];
    // materials
    std::vector<uint16_t> mat_host;
    std::vector<double> mat_eps, mat_sigma;
    DevBuf d_mat, d_cab;
    // CPML
    DevBuf d_prof[2][3][3];   // [E/H][axis][b,a,kinv]
    std::vector<unsigned char> pml_on[2][3];   // host copies of the "on" flags
    int off_lo[2][3], off_hi[2][3];            // the index range between the layers
    DevBuf d_psiE[3][2], d_psiH[3][2];
    // sources, receivers
    std::vector<FdtdSource> srcs;
    std::vector<std::vector<std::array<int, 3>>> obs_lists;   // 3 per receiver
    std::vector<int> obs_n;
    DevBuf d_src_comp, d_src_off, d_src_vals, d_obs_cnt, d_obs_start, d_obs_off, d_traces;
    DevBuf d_pt_plane, d_pt_list, d_samp, d_step;
    bool dirty = true;

    explicit FdtdSim(const ems_fdtd_params *p) : Sim(Kind::FDTD), P(*p)
    {
        nx = P.grid[0]; ny = P.grid[1]; nz = P.grid[2];
        EMS_CHECK_ARG(nx > 0 && ny > 0 && nz > 0, "grid sizes must be positive");
        EMS_CHECK_ARG((double)(nx + 2) * (ny + 2) * (nz + 2) < 4294967296.0, "grid too large for 32-bit array offsets");
        EMS_CHECK_ARG(P.h > 0 && P.dt > 0 && P.permittivity > 0 && P.permeability > 0, "h, dt, eps, mu must be positive");
        EMS_CHECK_ARG(P.time_frequency > 0, "time_frequency must be positive");
        EMS_CHECK_ARG(P.precision == EMS_FP64 || P.precision == EMS_FP32, "precision must be EMS_FP64 or EMS_FP32");
        // the reference's check_params condition (fdtd_simulation.cpp:358): c*dt < h
        double c = 1.0 / std::sqrt(P.permittivity * P.permeability);
        EMS_CHECK_ARG(c * P.dt < P.h, "time step violates c*dt < h (reference check_params)");
        EMS_CHECK_ARG(P.pml_cells >= 0 && 2 * P.pml_cells < std::min(nx, std::min(ny, nz)), "pml_cells too large for the grid");
        if (P.pml_order == 0) P.pml_order = 3.0;
        if (P.pml_kappa_max == 0) P.pml_kappa_max = 1.0;
        if (P.pml_reflection == 0) P.pml_reflection = 1e-6;
        fp64 = P.precision == EMS_FP64;
        n[0] = (size_t)(nx + 1) * (ny + 2) * (nz + 2);
        n[1] = (size_t)(nx + 2) * (ny + 1) * (nz + 2);
        n[2] = (size_t)(nx + 2) * (ny + 2) * (nz + 1);
        n[3] = (size_t)nx * (ny + 1) * (nz + 1);
        n[4] = (size_t)(nx + 1) * ny * (nz + 1);
        n[5] = (size_t)(nx + 1) * (ny + 1) * nz;
        init_stream();
        const size_t w = fp64 ? 8 : 4;
        V = (int)(16 / w);
        lead = V;
        auto up = [](size_t x, size_t m) { return (x + m - 1) / m * m; };
        // columns -1 .. nx, the first one at the end of the row before; whole
        // 32-byte sectors, so that a thread's vectors never leave its row
        pitch = up(nx + 2, 32 / w);
        plane = pitch * (ny + 2);
        total = plane * (nz + 2) + lead + V;   // one more vector behind the last row is read
        mpitch = up(nx + 1 + V, 4);
        for (int q = 0; q < 6; ++q) { F[q].alloc(total * w); F[q].zero(stream); }
        g0 = 0;
        g1 = (nx + V) / V;
        if (P.pml_cells > 0) {
            setup_pml();
            const int lo = std::max(off_lo[0][0] - 1, off_lo[1][0]), hi = std::min(off_hi[0][0] - 1, off_hi[1][0]);
            g0 = std::min((lo + V - 1) / V, g1);
            g1 = std::max(std::min(hi / V, g1), g0);
        }
        EMS_CUDA(cudaStreamSynchronize(stream));
    }

    void setup_pml()
    {
        const int nn[3] = {nx, ny, nz};
        const int L = P.pml_cells;
        double eta = std::sqrt(P.permeability / P.permittivity);
        double smax = -(P.pml_order + 1.0) * std::log(P.pml_reflection) / (2.0 * eta * L * P.h);
        for (int eh = 0; eh < 2; ++eh)
            for (int d = 0; d < 3; ++d) {
                int cnt = nn[d] + 2;
                std::vector<double> b(cnt, 0.0), av(cnt, 0.0), kinv(cnt, 1.0);
                std::vector<unsigned char> on(cnt, 0);
                double shift = eh == 0 ? -0.5 : 0.0;
                for (int s = 0; s < cnt; ++s) {
                    double x = s + shift, lo = L - x, hi = x - (nn[d] - L);
                    double dd = lo > hi ? lo : hi;
                    dd = dd < 0.0 ? 0.0 : (dd > L ? 1.0 : dd / L);
                    if (dd <= 0.0) continue;
                    double g = std::pow(dd, P.pml_order);
                    double sig = smax * g, kap = 1.0 + (P.pml_kappa_max - 1.0) * g, alp = P.pml_alpha_max * (1.0 - dd);
                    double bb = std::exp(-(sig / kap + alp) * P.dt / P.permittivity);
                    b[s] = bb;
                    av[s] = sig > 0.0 ? sig / (sig * kap + kap * kap * alp) * (bb - 1.0) : 0.0;
                    kinv[s] = 1.0 / kap;
                    on[s] = 1;
                }
                // (whole vectors of the x profile are read)
                for (std::vector<double> *v : {&b, &av, &kinv}) {
                    if (eh == 0 && d == 0) v->erase(v->begin());   // from s = 1, the first column of Ey and Ez
                    v->resize(cnt + V, v == &kinv ? 1.0 : 0.0);
                }
                upload_real(d_prof[eh][d][0], b);
                upload_real(d_prof[eh][d][1], av);
                upload_real(d_prof[eh][d][2], kinv);
                pml_on[eh][d] = on;
                // the index range between the two layers
                int lo = 0, hi = cnt;
                while (lo < hi && on[lo]) ++lo;
                while (hi > lo && on[hi - 1]) --hi;
                for (int q = lo; q < hi; ++q)
                    if (on[q]) throw Error{EMS_ERR_STATE, "CPML profile is not two slabs"};
                off_lo[eh][d] = lo;
                off_hi[eh][d] = hi;
            }
        size_t w = fp64 ? 8 : 4;
        for (int c = 0; c < 3; ++c)
            for (int r = 0; r < 2; ++r) {
                d_psiE[c][r].alloc(total * w); d_psiE[c][r].zero(stream);
                d_psiH[c][r].alloc(total * w); d_psiH[c][r].zero(stream);
            }
        EMS_CUDA(cudaStreamSynchronize(stream));
    }

    void upload_real(DevBuf &d, const std::vector<double> &v)
    {
        if (fp64) {
            d.alloc(v.size() * 8);
            EMS_CUDA(cudaMemcpyAsync(d.p, v.data(), v.size() * 8, cudaMemcpyHostToDevice, stream));
        } else {
            std::vector<float> f(v.begin(), v.end());
            d.alloc(f.size() * 4);
            EMS_CUDA(cudaMemcpyAsync(d.p, f.data(), f.size() * 4, cudaMemcpyHostToDevice, stream));
        }
        EMS_CUDA(cudaStreamSynchronize(stream));
    }

    // offset of a padded index in the device layout (Ey, Ez: one column to the left)
    long long ex_index(int c, const int *q) const
    {
        return (long long)q[0] - (c > 0 ? 1 : 0) + (long long)q[1] * (long long)pitch + (long long)q[2] * (long long)plane;
    }
    bool in_e(int c, const int *q) const
    {
        int lim[3][3] = {{nx, ny + 1, nz + 1}, {nx + 1, ny, nz + 1}, {nx + 1, ny + 1, nz}};
        for (int d = 0; d < 3; ++d)
            if (q[d] < 0 || q[d] > lim[c][d]) return false;
        return true;
    }

    void set_material(const double *eps, const double *sigma)
    {
        EMS_CHECK_ARG(eps != nullptr, "eps array required");
        size_t nc = (size_t)nx * ny * nz;
        std::map<std::pair<double, double>, int> ids;
        mat_host.assign(nc, 0);
        mat_eps.clear(); mat_sigma.clear();
        double last_e = -1.0, last_s = -1.0;
        int last_id = -1;
        for (size_t q = 0; q < nc; ++q) {
            double e = eps[q], s = sigma ? sigma[q] : 0.0;
            if (e == last_e && s == last_s) {   // runs of equal material along x
                mat_host[q] = (uint16_t)last_id;
                continue;
            }
            EMS_CHECK_ARG(std::isfinite(e) && e > 0 && std::isfinite(s) && s >= 0, "eps must be > 0 and sigma >= 0");
            auto key = std::make_pair(e, s);
            auto it = ids.find(key);
            int id;
            if (it == ids.end()) {
                EMS_CHECK_ARG(ids.size() < 65535, "more than 65535 distinct (eps, sigma) pairs");
                id = (int)ids.size();
                ids.emplace(key, id);
                mat_eps.push_back(e); mat_sigma.push_back(s);
            } else {
                id = it->second;
            }
            mat_host[q] = (uint16_t)id;
            last_e = e; last_s = s; last_id = id;
        }
        std::vector<double> ca(mat_eps.size()), cb(mat_eps.size());
        for (size_t m = 0; m < mat_eps.size(); ++m) {
            double s = mat_sigma[m] * P.dt / (2.0 * mat_eps[m]);
            ca[m] = (1.0 - s) / (1.0 + s);
            cb[m] = P.dt / mat_eps[m] / P.h / (1.0 + s);
        }
        d_mat.ensure((size_t)ny * nz * mpitch * 2 + 16);
        const size_t rows = (size_t)ny * nz, piece = std::min(rows, std::max<size_t>(kStage / nx, 1));
        d_stage.grow(piece * nx * 2);
        for (size_t r = 0; r < rows; r += piece) {
            const size_t m = std::min(piece, rows - r), cnt = m * mpitch;
            copy_in(d_stage.p, mat_host.data() + r * nx, m * nx * 2);
            fdtd_mat_kernel<<<(unsigned)((cnt + 255) / 256), 256, 0, stream>>>(d_stage.as<uint16_t>(), d_mat.as<uint16_t>() + r * mpitch,
                                                                               cnt, (unsigned)mpitch, nx);
        }
        std::vector<double> cab(2 * ca.size());
        for (size_t m = 0; m < ca.size(); ++m) { cab[2 * m] = ca[m]; cab[2 * m + 1] = cb[m]; }
        upload_real(d_cab, cab);
    }

    // x / d = (x * magic) >> shift for x < 2^31: magic = ceil(2^shift / d) with
    // 2^shift >= 2^31 d, so the error x (magic d - 2^shift) / 2^shift stays
    // below 1; magic < 2^32
    static void divider(unsigned d, unsigned &magic, unsigned &shift)
    {
        unsigned l = 0;
        while ((1ull << l) < d) ++l;
        shift = 31 + l;
        magic = (unsigned)(((1ull << shift) + d - 1) / d);
    }

    template <class T> FdtdArgs<T> args() const
    {
        FdtdArgs<T> a{};
        T **f[6] = {&a.Ex, &a.Ey, &a.Ez, &a.Hx, &a.Hy, &a.Hz};
        for (int q = 0; q < 6; ++q) *f[q] = F[q].as<T>() + lead;
        a.nx = nx; a.ny = ny; a.nz = nz;
        a.g0 = g0; a.g1 = g1; a.gr = (nx + V) / V - (g1 - g0);
        divider(std::max(g1 - g0, 1), a.magic[0], a.shift[0]);
        divider(std::max(a.gr, 1), a.magic[1], a.shift[1]);
        a.pitch = (unsigned)pitch;
        a.plane = plane;
        a.mpitch = (unsigned)mpitch;
        a.ch = (T)(P.dt / P.permeability / P.h);
        a.ce = (T)(P.dt / P.permittivity / P.h);
        a.mat = d_mat.as<uint16_t>();
        a.cab = d_cab.as<CaCb<T>>();
        if (P.pml_cells > 0)
            for (int d = 0; d < 3; ++d) {
                const int s0 = d == 0 ? 1 : 0;   // the E-type x profile starts at s = 1
                a.pe[d] = Prof<T>{d_prof[0][d][0].as<T>(), d_prof[0][d][1].as<T>(), d_prof[0][d][2].as<T>(), off_lo[0][d] - s0,
                                  off_hi[0][d] - s0};
                a.ph[d] = Prof<T>{d_prof[1][d][0].as<T>(), d_prof[1][d][1].as<T>(), d_prof[1][d][2].as<T>(), off_lo[1][d], off_hi[1][d]};
                for (int r = 0; r < 2; ++r) {
                    a.psiE[d][r] = d_psiE[d][r].as<T>() + lead;
                    a.psiH[d][r] = d_psiH[d][r].as<T>() + lead;
                }
            }
        return a;
    }

    // Launch shape of the H and E kernels (x times y threads, each V cells
    // along x; one z plane per block row), chosen on the handle's first run
    // of at least kTuneMinSteps steps.  Every cell belongs to one thread
    // whatever the shape, so the shape changes no result.
    dim3 blk{32, 8, 1};
    bool tuned = false;
    dim3 block() const { return blk; }
    void launch_shape(int b[3]) override { b[0] = (int)blk.x; b[1] = (int)blk.y; b[2] = 1; }
    unsigned blocks_of(int groups) const   // blocks that cover `groups` threads of every row
    {
        const size_t t = (size_t)groups * (ny + 1), b = (size_t)blk.x * blk.y;
        return (unsigned)((t + b - 1) / b);
    }
    unsigned main_blocks() const { return blocks_of(g1 - g0); }
    dim3 grid(int planes) const { return dim3(main_blocks() + blocks_of((nx + V) / V - (g1 - g0)), 1, planes); }

    static constexpr int kShapes = 6, kTuneSteps = 3, kTuneMinSteps = 24;
    static constexpr unsigned kShape[kShapes][2] = {{32, 8}, {32, 4}, {64, 4}, {128, 2}, {256, 1}, {64, 2}};

    // Steps of this run spent tuning: the environment variable
    // EMS_FDTD_BLOCK="XxY" forces one of the shapes; otherwise the first run
    // of at least kTuneMinSteps steps advances kTuneSteps steps with each
    // shape (one warm-up, two timed) and keeps the fastest.
    int tune_steps(int nsteps)
    {
        if (tuned) return 0;
        if (const char *env = std::getenv("EMS_FDTD_BLOCK")) {
            unsigned x = 0, y = 0;
            if (std::sscanf(env, "%ux%u", &x, &y) == 2)
                for (auto &sh : kShape)
                    if (sh[0] == x && sh[1] == y) { blk = dim3(x, y, 1); tuned = true; return 0; }
            throw Error{EMS_ERR_INVALID_ARGUMENT, "EMS_FDTD_BLOCK must be one of 32x8 32x4 64x4 128x2 256x1 64x2"};
        }
        return nsteps >= kTuneMinSteps ? kShapes * kTuneSteps : 0;
    }

    // The H and E launches are set up ahead (launch_after: 24x20x16 FP64 7.9 -> 6.8 us a
    // step, 64^3 FP64 25.0 -> 24.2, 141x117x93 FP32 with CPML 29.2 -> 28.3, large
    // grids unchanged).  An early trigger in the kernels gave less, and so did
    // material loads ahead of the wait (400x384x368: 54.4 ms for 60 steps, 52.5
    // with the field loads first).
    // H update of planes [k0, k1)
    template <class T> void launch_h(const FdtdArgs<T> &a, int k0, int k1, int *ctr = nullptr, int inc = 0)
    {
        auto k = P.pml_cells > 0 ? fdtd_h_kernel<T, true> : fdtd_h_kernel<T, false>;
        launch_after(k, grid(k1 - k0), blk, 0, stream, a, k0, main_blocks(), ctr, inc);
    }
    // E update of planes [k0, k1) with the planes' points
    template <class T> void launch_e(const FdtdArgs<T> &a, int k0, int k1, const FdtdPoints &pt)
    {
        const bool mat = !mat_host.empty(), pml = P.pml_cells > 0;
        auto k = mat ? (pml ? fdtd_e_kernel<T, true, true> : fdtd_e_kernel<T, true, false>)
                     : (pml ? fdtd_e_kernel<T, false, true> : fdtd_e_kernel<T, false, false>);
        launch_after(k, grid(k1 - k0), blk, 0, stream, a, pt, k0, main_blocks());
    }

    // The sources and receiver samples as the E kernel's point lists; false
    // where the kernels after the E update have to serve them: a point in the
    // padding that no thread of the E kernel updates, more samples than 256 MB
    // or the free memory hold, or in FP32 so many points in so many planes that the threads'
    // search (each probe of a plane's list by each of its cells) takes longer
    // than the two launches.  192^3 FP32, us a step, served by the E kernel and
    // by the other two: 63 points in each plane (43 million probes) 94 and 93,
    // 180 (55 million) 104 and 93, 180 in one plane 79 and 92.  In FP64, bound by
    // the FP64 pipe, 180 in each plane 421 and 433.
    static constexpr double kMaxProbes = 4e7;
    bool fold_points(int nsamp_run, FdtdPoints &pt)
    {
        struct Item {
            int k;
            FdtdPoint p;
        };
        std::vector<Item> items;
        auto add = [&](int comp, const int *q, int tag, int idx) {
            const int lo[3] = {comp == 0 ? 0 : 1, comp == 1 ? 0 : 1, comp == 2 ? 0 : 1};
            if (q[0] < lo[0] || q[1] < lo[1] || q[2] < lo[2] || q[0] > nx || q[1] > ny || q[2] > nz) return false;
            items.push_back({q[2], {ex_index(comp, q), comp + tag, idx}});
            return true;
        };
        for (size_t s = 0; s < srcs.size(); ++s)
            if (!add(srcs[s].comp, srcs[s].ijk, 0, (int)s)) return false;
        int nsm = 0;
        for (size_t l = 0; l < obs_lists.size(); ++l)
            for (auto &q : obs_lists[l])
                if (!add((int)(l % 3), q.data(), 4, nsm++)) return false;
        if ((double)nsm * nsamp_run * 8.0 > 256e6) return false;
        std::stable_sort(items.begin(), items.end(), [](const Item &x, const Item &y) { return x.k != y.k ? x.k < y.k : x.p.off < y.p.off; });
        std::vector<int> plane(nz + 2, 0);
        std::vector<FdtdPoint> list(std::max<size_t>(items.size(), 1));
        for (size_t q = 0; q < items.size(); ++q) {
            list[q] = items[q].p;
            ++plane[items[q].k + 1];
        }
        double probes = 0.0;
        for (int k = 0; k <= nz; ++k) {
            probes += std::log2(1.0 + plane[k + 1]) * (nx + 1.0) * (ny + 1.0);
            plane[k + 1] += plane[k];
        }
        if (!fp64 && probes > kMaxProbes) return false;
        d_pt_plane.ensure(plane.size() * sizeof(int));
        d_pt_list.ensure(list.size() * sizeof(FdtdPoint));
        try {
            d_samp.ensure((size_t)std::max(nsm, 1) * nsamp_run * 8);
        } catch (const Error &e) {   // a grid that leaves no memory for them
            if (e.code != EMS_ERR_OUT_OF_MEMORY) throw;
            return false;
        }
        EMS_CUDA(cudaMemcpyAsync(d_pt_plane.p, plane.data(), plane.size() * sizeof(int), cudaMemcpyHostToDevice, stream));
        EMS_CUDA(cudaMemcpyAsync(d_pt_list.p, list.data(), list.size() * sizeof(FdtdPoint), cudaMemcpyHostToDevice, stream));
        EMS_CUDA(cudaStreamSynchronize(stream));   // the host vectors end here
        pt = FdtdPoints{items.empty() ? nullptr : d_pt_plane.as<int>(), d_pt_list.as<FdtdPoint>(), d_src_vals.as<double>(),
                        d_samp.as<double>(), nullptr, 0, (int)srcs.size(), nsm, P.time_frequency};
        return true;
    }

    // A graph of kGraphSteps steps, kept in the handle while the buffers and
    // the launch shape stay the same.
    static constexpr int kGraphSteps = 16;
    cudaGraphExec_t graph = nullptr;
    std::vector<unsigned long long> graph_key;
    ~FdtdSim() override
    {
        if (graph) cudaGraphExecDestroy(graph);
    }
    template <class T> void make_graph(const FdtdArgs<T> &a, FdtdPoints pt)
    {
        std::vector<unsigned long long> key = {blk.x, blk.y, (unsigned long long)pt.ns, (unsigned long long)pt.nsm,
                                               (unsigned long long)(pt.plane != nullptr), mat_host.empty()};
        for (const void *q : {F[0].p, F[1].p, F[2].p, F[3].p, F[4].p, F[5].p, d_mat.p, d_cab.p, d_pt_plane.p, d_pt_list.p, d_src_vals.p,
                              d_samp.p})
            key.push_back((unsigned long long)reinterpret_cast<uintptr_t>(q));
        if (graph && key == graph_key) return;
        if (graph) {
            cudaGraphExecDestroy(graph);
            graph = nullptr;
        }
        pt.base = d_step.as<int>();
        const cudaGraph_t g = capture([&] {
            for (int r = 0; r < kGraphSteps; ++r) {
                launch_h<T>(a, 0, nz + 1, r == 0 ? d_step.as<int>() : nullptr, kGraphSteps);
                pt.step = r + 1;
                launch_e<T>(a, 0, nz + 1, pt);
            }
        });
        const cudaError_t e = cudaGraphInstantiate(&graph, g, 0);
        cudaGraphDestroy(g);
        EMS_CUDA(e);
        graph_key = key;
    }

    template <class T> void run_t(int nsteps)
    {
        const int tf = P.time_frequency;
        nsamp = nsteps / tf + 1;
        nobs = (int)obs_n.size() / 3;
        ncols = 3;
        // source values per step, computed on the host in FP64 exactly as the
        // reference does (time accumulated by repeated addition of dt)
        int ns = (int)srcs.size();
        std::vector<double> vals((size_t)std::max(ns, 1) * nsteps, 0.0);
        double t = 0.0;
        for (int st = 0; st < nsteps; ++st) {
            for (int s = 0; s < ns; ++s) {
                const FdtdSource &q = srcs[s];
                double eps = P.permittivity, div = 1.0;
                if (!mat_host.empty()) {
                    // the cell whose material the E kernel takes at this point; the nearest one in the padding
                    int cell[3];
                    const int n3[3] = {nx, ny, nz};
                    for (int d = 0; d < 3; ++d) cell[d] = std::min(std::max(q.ijk[d] - (d == q.comp ? 0 : 1), 0), n3[d] - 1);
                    const int m = mat_host[(size_t)cell[0] + (size_t)cell[1] * nx + (size_t)cell[2] * nx * ny];
                    eps = mat_eps[m];
                    div = 1.0 + mat_sigma[m] * P.dt / (2.0 * mat_eps[m]);
                }
                double v = fdtd_source_value(q.kind, q.f0, t, P.h) * q.amp * P.dt / eps;
                if (div != 1.0) v /= div;
                vals[(size_t)st * ns + s] = v;
            }
            t += P.dt;
        }
        std::vector<int> comp(std::max(ns, 1));
        std::vector<long long> off(std::max(ns, 1));
        for (int s = 0; s < ns; ++s) { comp[s] = srcs[s].comp; off[s] = srcs[s].off; }
        d_src_comp.ensure(comp.size() * 4); d_src_off.ensure(off.size() * 8); d_src_vals.ensure(vals.size() * 8);
        EMS_CUDA(cudaMemcpyAsync(d_src_comp.p, comp.data(), comp.size() * 4, cudaMemcpyHostToDevice, stream));
        EMS_CUDA(cudaMemcpyAsync(d_src_off.p, off.data(), off.size() * 8, cudaMemcpyHostToDevice, stream));
        EMS_CUDA(cudaMemcpyAsync(d_src_vals.p, vals.data(), vals.size() * 8, cudaMemcpyHostToDevice, stream));
        // receivers
        std::vector<int> start(std::max(nobs, 1), 0);
        std::vector<long long> roff;
        for (int o = 0; o < nobs; ++o) {
            start[o] = (int)roff.size();
            for (int c = 0; c < 3; ++c)
                for (auto &q : obs_lists[3 * o + c]) roff.push_back(ex_index(c, q.data()));
        }
        if (roff.empty()) roff.push_back(0);
        d_obs_cnt.ensure(std::max<size_t>(obs_n.size(), 1) * 4);
        d_obs_start.ensure(start.size() * 4);
        d_obs_off.ensure(roff.size() * 8);
        if (!obs_n.empty()) EMS_CUDA(cudaMemcpyAsync(d_obs_cnt.p, obs_n.data(), obs_n.size() * 4, cudaMemcpyHostToDevice, stream));
        EMS_CUDA(cudaMemcpyAsync(d_obs_start.p, start.data(), start.size() * 4, cudaMemcpyHostToDevice, stream));
        EMS_CUDA(cudaMemcpyAsync(d_obs_off.p, roff.data(), roff.size() * 8, cudaMemcpyHostToDevice, stream));
        size_t ntr = (size_t)std::max(nobs, 1) * nsamp * 3;
        d_traces.ensure(ntr * 8);
        d_step.ensure(sizeof(int));
        d_traces.zero(stream);

        FdtdArgs<T> a = args<T>();
        long long launches = 0;
        const int tune = tune_steps(nsteps);
        FdtdPoints pt{};
        const bool folded = fold_points(nsamp, pt);
        const FdtdPoints none{};
        struct TuneEvents {   // destroyed on every exit path
            cudaEvent_t e[2 * kShapes] = {};
            ~TuneEvents()
            {
                for (cudaEvent_t x : e)
                    if (x) cudaEventDestroy(x);
            }
        } tev;
        if (tune)
            for (cudaEvent_t &x : tev.e) EMS_CUDA(cudaEventCreate(&x));
        EMS_CUDA(cudaEventRecord(ev0, stream));
        int step = 1;
        const auto direct = [&](int last) {   // steps up to `last`, launch by launch
            for (; step <= last; ++step) {
                const int ts = step - 1, c = ts / kTuneSteps, r = ts % kTuneSteps;
                if (ts < tune) {
                    blk = dim3(kShape[c][0], kShape[c][1], 1);
                    if (r == 1) EMS_CUDA(cudaEventRecord(tev.e[2 * c], stream));
                }
                launch_h<T>(a, 0, nz + 1);
                pt.step = step;
                launch_e<T>(a, 0, nz + 1, folded ? pt : none);
                launches += 2;
                if (ns > 0 && !folded) {
                    fdtd_source_kernel<T><<<1, 32, 0, stream>>>(a.Ex, a.Ey, a.Ez, d_src_comp.as<int>(), d_src_off.as<long long>(),
                                                               d_src_vals.as<double>() + (size_t)(step - 1) * ns, ns);
                    ++launches;
                }
                if (nobs > 0 && !folded && step % tf == 0) {
                    fdtd_receiver_kernel<T><<<(nobs + 127) / 128, 128, 0, stream>>>(
                        a.Ex, a.Ey, a.Ez, nobs, d_obs_cnt.as<int>(), d_obs_start.as<int>(), d_obs_off.as<long long>(),
                        d_traces.as<double>() + (size_t)(step / tf) * 3, nsamp);
                    ++launches;
                }
                if (ts < tune && r == kTuneSteps - 1) EMS_CUDA(cudaEventRecord(tev.e[2 * c + 1], stream));
                if (tune && step == tune) {   // all shapes timed: keep the fastest
                    EMS_CUDA(cudaEventSynchronize(tev.e[2 * kShapes - 1]));
                    float best = 0.0f;
                    int pick = 0;
                    for (int k = 0; k < kShapes; ++k) {
                        float ms = 0.0f;
                        EMS_CUDA(cudaEventElapsedTime(&ms, tev.e[2 * k], tev.e[2 * k + 1]));
                        if (k == 0 || ms < best) { best = ms; pick = k; }
                    }
                    blk = dim3(kShape[pick][0], kShape[pick][1], 1);
                    tuned = true;
                }
            }
        };
        if (!folded) {
            direct(nsteps);
        } else {
            direct(std::min(tune, nsteps));
            if (nsteps - step + 1 >= kGraphSteps) {
                make_graph<T>(a, pt);
                const int base = step - 1 - kGraphSteps;   // the graph's first launch moves it on
                EMS_CUDA(cudaMemcpyAsync(d_step.p, &base, sizeof(int), cudaMemcpyHostToDevice, stream));
                for (; step + kGraphSteps - 1 <= nsteps; step += kGraphSteps) {
                    EMS_CUDA(cudaGraphLaunch(graph, stream));
                    launches += 2 * kGraphSteps;
                }
            }
            direct(nsteps);
            if (nobs > 0 && nsamp > 1) {
                const size_t nt = (size_t)nobs * nsamp;
                fdtd_trace_kernel<<<(unsigned)((nt + 127) / 128), 128, 0, stream>>>(d_samp.as<double>(), pt.nsm, nobs, d_obs_cnt.as<int>(),
                                                                                    d_obs_start.as<int>(), d_traces.as<double>(), nsamp);
                ++launches;
            }
        }
        EMS_CUDA(cudaGetLastError());
        EMS_CUDA(cudaEventRecord(ev1, stream));
        EMS_CUDA(cudaStreamSynchronize(stream));
        float ms = 0;
        EMS_CUDA(cudaEventElapsedTime(&ms, ev0, ev1));
        last_ms = ms;
        last_launches = launches;
        traces.assign(ntr, 0.0);
        EMS_CUDA(cudaMemcpy(traces.data(), d_traces.p, ntr * 8, cudaMemcpyDeviceToHost));
        traces.resize((size_t)nobs * nsamp * 3);
    }

    void run(int nsteps) override
    {
        EMS_CHECK_ARG(nsteps >= 0, "num_steps must be >= 0");
        if (fp64) run_t<double>(nsteps); else run_t<float>(nsteps);
        check_finite({{F[0].p, total}, {F[1].p, total}, {F[2].p, total}, {F[3].p, total}, {F[4].p, total}, {F[5].p, total}}, fp64);
    }

    size_t field_size(int which) const override
    {
        if (which < 0 || which > 5) throw Error{EMS_ERR_INVALID_ARGUMENT, "field index must be 0..5 (Ex,Ey,Ez,Hx,Hy,Hz)"};
        return n[which];
    }
    // n values of a component from `at` on between the device layout and the API's
    template <class T, bool GET> void move_field(int which, size_t at, size_t n, double *api) const
    {
        const int w[6] = {nx + 1, nx + 2, nx + 2, nx, nx + 1, nx + 1}, h[6] = {ny + 2, ny + 1, ny + 2, ny + 1, ny, ny + 1};
        fdtd_field_kernel<T, GET><<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(
            F[which].as<T>() + lead, api, at, n, w[which], h[which], pitch, plane, which == 1 || which == 2 ? 1 : 0);
        EMS_CUDA(cudaGetLastError());
    }
    void get_field(int which, double *out) const override
    {
        download(out, field_size(which), [&](size_t at, size_t n, double *dst) {
            if (fp64) move_field<double, true>(which, at, n, dst); else move_field<float, true>(which, at, n, dst);
        });
    }
    void set_field(int which, const double *in) override
    {
        const size_t cnt = field_size(which), piece = std::min(cnt, kStage);
        d_stage.grow(piece * sizeof(double));
        for (size_t at = 0; at < cnt; at += piece) {
            const size_t n = std::min(piece, cnt - at);
            copy_in(d_stage.p, in + at, n * sizeof(double));
            if (fp64) move_field<double, false>(which, at, n, d_stage.as<double>());
            else move_field<float, false>(which, at, n, d_stage.as<double>());
        }
        EMS_CUDA(cudaStreamSynchronize(stream));
    }

    // fdtd_simulation.cpp:308-331: results_<i>_<dt>_<h>_<N>.csv in `path`
    // (a directory; "." if empty), default stream precision, columns
    // time,Ex,Ey,Ez with time = j*tf*dt.
    void save(const char *path) const override
    {
        std::string dir = (path && *path) ? path : ".";
        int nsteps_run = (nsamp - 1) * P.time_frequency;
        for (int o = 0; o < nobs; ++o) {
            std::string fn = dir + "/results_" + std::to_string(o) + "_" + std::to_string(P.dt) + "_" +
                             std::to_string(P.h) + "_" + std::to_string(nsteps_run) + ".csv";
            std::ofstream f(fn);
            if (!f.is_open()) throw Error{EMS_ERR_IO, "cannot open " + fn};
            f << "time,Ex,Ey,Ez" << std::endl;
            for (int j = 0; j < nsamp; ++j) {
                const double *r = &traces[((size_t)o * nsamp + j) * 3];
                f << j * P.time_frequency * P.dt << "," << r[0] << "," << r[1] << "," << r[2] << std::endl;
            }
        }
    }

    double sample_time(int j) const override { return j * P.time_frequency * P.dt; }

    void reset() override
    {
        for (int q = 0; q < 6; ++q) F[q].zero(stream);
        if (P.pml_cells > 0)
            for (int c = 0; c < 3; ++c)
                for (int r = 0; r < 2; ++r) {
                    d_psiE[c][r].zero(stream); d_psiH[c][r].zero(stream);
                }
        EMS_CUDA(cudaStreamSynchronize(stream));
    }

    // E points whose update runs the CPML recursion (two psi values each).
    double pml_e_points() const
    {
        if (P.pml_cells <= 0) return 0.0;
        auto pairs = [&](int d1, int n1, int d2, int n2) {
            double c = 0.0;
            for (int a = 1; a <= n1; ++a)
                for (int b = 1; b <= n2; ++b) c += (pml_on[0][d1][a] | pml_on[0][d2][b]) ? 1.0 : 0.0;
            return c;
        };
        return (nx + 1.0) * pairs(1, ny, 2, nz) + (ny + 1.0) * pairs(2, nz, 0, nx) + (nz + 1.0) * pairs(0, nx, 1, ny);
    }

    void time_dominant(int launches, double *ms, double *bytes, std::string *name) override
    {
        size_t w = fp64 ? 8 : 4;
        size_t cells = (size_t)nx * ny * nz;
        const double matb = mat_host.empty() ? 0.0 : 2.0 * cells;
        // E update: reads H (3), reads and writes E (3), the material id, and
        // reads and writes two psi values per point inside the CPML
        double b = (double)cells * 9.0 * w + matb + pml_e_points() * 4.0 * w;
        // what the E kernel writes: E and, in a CPML, its auxiliary fields
        std::vector<const DevBuf *> written = {&F[0], &F[1], &F[2]};
        if (P.pml_cells > 0)
            for (int c = 0; c < 3; ++c)
                for (int r = 0; r < 2; ++r) written.push_back(&d_psiE[c][r]);
        std::vector<DevBuf> save(written.size());
        for (size_t q = 0; q < written.size(); ++q) {
            save[q].alloc(written[q]->bytes);
            EMS_CUDA(cudaMemcpyAsync(save[q].p, written[q]->p, written[q]->bytes, cudaMemcpyDeviceToDevice, stream));
        }
        float t = 0;
        auto body = [&](auto tag) {
            using T = decltype(tag);
            const auto a = args<T>();
            for (int r = 0; r <= launches; ++r) {   // the first one untimed
                if (r == 1) EMS_CUDA(cudaEventRecord(ev0, stream));
                launch_e<T>(a, 0, nz + 1, {});
            }
        };
        if (fp64) body(double()); else body(float());
        EMS_CUDA(cudaEventRecord(ev1, stream));
        EMS_CUDA(cudaStreamSynchronize(stream));
        EMS_CUDA(cudaEventElapsedTime(&t, ev0, ev1));
        for (size_t q = 0; q < written.size(); ++q)
            EMS_CUDA(cudaMemcpyAsync(written[q]->p, save[q].p, written[q]->bytes, cudaMemcpyDeviceToDevice, stream));
        EMS_CUDA(cudaStreamSynchronize(stream));
        *ms = t / launches;
        *bytes = b;
        *name = fp64 ? "fdtd_e_kernel<double>" : "fdtd_e_kernel<float>";
    }
};

Sim *make_fdtd(const ems_fdtd_params *p) { return new FdtdSim(p); }

void fdtd_set_source(Sim *s, int comp, const int ijk[3], int waveform, double f0, double amp)
{
    auto *f = static_cast<FdtdSim *>(s);
    EMS_CHECK_ARG(comp >= 0 && comp < 3, "component must be 0, 1 or 2");
    EMS_CHECK_ARG(ijk != nullptr && f->in_e(comp, ijk), "source index outside the field array");
    EMS_CHECK_ARG(waveform == EMS_WAVE_REFERENCE || waveform == EMS_WAVE_RICKER, "unknown waveform");
    EMS_CHECK_ARG(f0 > 0 && std::isfinite(amp), "f0 must be positive");
    FdtdSource q{comp, {ijk[0], ijk[1], ijk[2]}, waveform, f0, amp, f->ex_index(comp, ijk)};
    f->srcs.push_back(q);
}

void fdtd_add_observation(Sim *s, const int *x, int nx_, const int *y, int ny_, const int *z, int nz_)
{
    auto *f = static_cast<FdtdSim *>(s);
    const int *lists[3] = {x, y, z};
    int cnt[3] = {nx_, ny_, nz_};
    for (int c = 0; c < 3; ++c) {
        EMS_CHECK_ARG(cnt[c] >= 0 && (cnt[c] == 0 || lists[c] != nullptr), "observation list missing");
        std::vector<std::array<int, 3>> v;
        for (int r = 0; r < cnt[c]; ++r) {
            EMS_CHECK_ARG(f->in_e(c, lists[c] + 3 * r), "observation index outside the field array");
            v.push_back({lists[c][3 * r], lists[c][3 * r + 1], lists[c][3 * r + 2]});
        }
        f->obs_lists.push_back(v);
        f->obs_n.push_back(cnt[c]);
    }
}

void fdtd_set_material(Sim *s, const double *eps, const double *sigma) { static_cast<FdtdSim *>(s)->set_material(eps, sigma); }

}  // namespace ems
