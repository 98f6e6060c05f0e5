// df.cu -- stage (c): frequency shift, dissipation and the df loss seed.
//
// Replaces the host NumPy/SciPy post-processing of SPAMMM:
//   compute_df_amp_dir  spammm/SPM/AFM.py:3203-3236 (9-point Gauss-Chebyshev,
//                       scipy.ndimage.map_coordinates(order=1, mode='nearest'),
//                       numpy.gradient with edge_order=1)
//   compute_df_dir      spammm/SPM/AFM.py:3105-3123
//   compute_dissipation spammm/SPM/AFM.py:3238-3277
//   df_loss_seed        spammm/SPM/AFM.py:3125-3200
// All arithmetic is FP64, as on the reference host.  The FEs volume is
// (nx,ny,nz,4) float32 with z fastest.  The amplitude df is FP64-arithmetic
// bound, so the nine quadrature nodes are folded into one filter per direction
// and the finite differences multiply by 1/dr and 1/(2 dr) instead of dividing (within an
// FP64 ulp of numpy.gradient's division; the float32 results are unchanged at
// the reference fixtures' tolerance).  Compiled with -fmad=false so the FP64
// expression order otherwise matches NumPy's.
#include "spm_internal.cuh"
#include "spm_diss.cuh"
#include "spm_batch.cuh"
#include <algorithm>
#include <cmath>

namespace spm {
namespace {

constexpr int DF_THREADS = 256;
constexpr int NQ = 9;  // Gauss-Chebyshev nodes

struct DfGeom {
    int nx, ny, nz;
    double n[3];       // oscillation direction (unit)
    double dr[3];      // spacing
    double shift[3];   // amp * n / dr
    double idr[3];     // 1 / dr and 1 / (2 dr): the one-sided and central differences multiply by them
    double idr2[3];
    double uk[NQ];     // cos((2k+1) pi / 18)
    double wk;         // 1/9
    int act[3];        // active axes (|n| > 1e-15)
    int nact;
};

// One (Fx,Fy,Fz,E) row of an FP32 or FP64 volume, widened to double.
struct Row {
    double x, y, z, w;
};
__device__ __forceinline__ Row load_row(const float* __restrict__ v, size_t i) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(v) + i);
    return Row{(double)f.x, (double)f.y, (double)f.z, (double)f.w};
}
__device__ __forceinline__ Row load_row(const double* __restrict__ v, size_t i) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(v) + 2 * i);
    const double2 b = __ldg(reinterpret_cast<const double2*>(v) + 2 * i + 1);
    return Row{a.x, a.y, b.x, b.y};
}

template <typename T>
__device__ __forceinline__ double fn_at(const T* __restrict__ FEs, const DfGeom& P, int ix, int iy, int iz) {
    const Row f = load_row(FEs, ((size_t)ix * P.ny + iy) * P.nz + iz);
    return (f.x * P.n[0] + f.y * P.n[1]) + f.z * P.n[2];
}

__device__ __forceinline__ int clampi(int i, int n) { return i < 0 ? 0 : (i >= n ? n - 1 : i); }

// map_coordinates(F_n, (ix,iy,iz) + u*shift, order=1, mode='nearest'):
// per-axis weights (1-t, t) at floor(c), clamped indices, corners summed with
// the last axis fastest and each term formed as ((f*w0)*w1)*w2.
template <typename T>
__device__ double shifted_fn(const T* __restrict__ FEs, const DfGeom& P, int ix, int iy, int iz, double u) {
    const int dims[3] = {P.nx, P.ny, P.nz};
    const int idx[3] = {ix, iy, iz};
    int i0[3];
    double w[3][2];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double c = (double)idx[d] + u * P.shift[d];
        const double fl = floor(c);
        const double t = c - fl;
        i0[d] = (int)fl;
        w[d][0] = 1.0 - t;
        w[d][1] = t;
    }
    double acc = 0.0;
#pragma unroll
    for (int a0 = 0; a0 < 2; a0++) {
        if (w[0][a0] == 0.0) continue;
#pragma unroll
        for (int a1 = 0; a1 < 2; a1++) {
            if (w[1][a1] == 0.0) continue;
#pragma unroll
            for (int a2 = 0; a2 < 2; a2++) {
                if (w[2][a2] == 0.0) continue;
                double coeff = fn_at(FEs, P, clampi(i0[0] + a0, dims[0]), clampi(i0[1] + a1, dims[1]),
                                     clampi(i0[2] + a2, dims[2]));
                coeff *= w[0][a0];
                coeff *= w[1][a1];
                coeff *= w[2][a2];
                acc += coeff;
            }
        }
    }
    return acc;
}

// numpy.gradient(S, dr, axis) at one point, uniform spacing, edge_order=1.
template <bool AMP, typename T>
__device__ double grad_at(const T* __restrict__ FEs, const DfGeom& P, int ax, int ix, int iy, int iz, double u) {
    const int dims[3] = {P.nx, P.ny, P.nz};
    int idx[3] = {ix, iy, iz};
    const int i = idx[ax], n = dims[ax];
    auto S = [&](int j) {
        int q[3] = {idx[0], idx[1], idx[2]};
        q[ax] = j;
        return AMP ? shifted_fn(FEs, P, q[0], q[1], q[2], u) : fn_at(FEs, P, q[0], q[1], q[2]);
    };
    if (i == 0) return (S(1) - S(0)) * P.idr[ax];
    if (i == n - 1) return (S(n - 1) - S(n - 2)) * P.idr[ax];
    return (S(i + 1) - S(i - 1)) * P.idr2[ax];
}

template <typename T>
__global__ void __launch_bounds__(DF_THREADS)
df_amp_dir_kernel(const T* __restrict__ FEs, DfGeom P, const int* __restrict__ out_iz, int n_out,
                  float* __restrict__ df) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)P.nx * P.ny * n_out;
    if (gid >= total) return;
    const int o = (int)(gid % n_out);
    const long long pix = gid / n_out;
    const int iy = (int)(pix % P.ny), ix = (int)(pix / P.ny);
    const int iz = out_iz ? out_iz[o] : o;
    if (iz < 0 || iz >= P.nz) {  // invalid selection: flag the element instead of reading out of bounds
        df[gid] = __int_as_float(0x7fc00000);
        return;
    }
    double acc = 0.0;
    for (int k = 0; k < NQ; k++) {
        for (int a = 0; a < P.nact; a++) {
            const int ax = P.act[a];
            const double g = grad_at<true>(FEs, P, ax, ix, iy, iz, P.uk[k]);
            acc -= (P.wk * P.n[ax]) * g;
        }
    }
    df[gid] = (float)acc;
}

// Oscillation along +-z only (the common case): one warp per pixel column.
//
// The nine shifted samples of a height are one fixed filter on the column: node
// k reads F_n at floor(u_k shift) and the next height with constant linear
// weights, so A[j] = sum_k wk S(j, u_k) is at most 18 taps (ZTaps, merged on the
// host), and the average of the nine central differences is the central
// difference of A.  Per output that is 18 FP64 FMAs and one difference where the
// node-by-node form took 9 x (floor, conversions, two products, a difference):
// the FP64 and conversion instructions bound it (0.32 ms on a 480 x 480 x 60
// volume against 0.04 ms for its bytes), this form is bound by the shared-memory
// reads of the taps.  Column ends clamp the tap's height (mode='nearest'): the
// staged column is padded with its end values so that the tap loop has no
// clamps, as far as pads and column fit the buffer; a longer one clamps.
constexpr int DFZ_WARPS = 8;
constexpr int DFZ_MAXNZ = 512;
constexpr int DFZ_TAB = 64;  // columns up to this height take A of each height once (a table row)
constexpr double TAP_SNAP = 1e-14;  // a linear weight this close to 0 or 1 is that (the rounding of j + u shift)

struct ZTaps {
    int n, padl, padr;
    int off[2 * NQ];
    double w[2 * NQ];
};

// floor and linear weight of a constant shift x in samples.
void split_shift(double x, long long& m, double& t) {
    const double f = floor(x);
    m = (long long)std::min(std::max(f, -1e15), 1e15);
    t = x - f;
    if (t < TAP_SNAP) t = 0.0;
    if (t > 1.0 - TAP_SNAP) { t = 0.0; m += 1; }
}

// The taps of a shift of `sh` samples.  Offsets beyond +-2^30 read the column's ends like any other
// beyond them; a shift that is not finite makes every value NaN.
ZTaps make_ztaps(const DfGeom& P, double sh) {
    ZTaps T = {};
    if (!std::isfinite(sh)) {
        T.n = 1;
        T.w[0] = std::nan("");
        return T;
    }
    auto add = [&](long long off, double w) {
        if (w == 0.0) return;  // never read: a non-finite neighbour does not count
        const int o = (int)std::min(std::max(off, -(1LL << 30)), 1LL << 30);
        for (int i = 0; i < T.n; i++)
            if (T.off[i] == o) { T.w[i] += w; return; }
        T.off[T.n] = o;
        T.w[T.n++] = w;
    };
    for (int k = 0; k < NQ; k++) {
        long long m;
        double t;
        split_shift(P.uk[k] * sh, m, t);
        add(m, P.wk * (1.0 - t));
        add(m + 1, P.wk * t);
    }
    for (int i = 0; i < T.n; i++) {
        if (-T.off[i] > T.padl) T.padl = -T.off[i];
        if (T.off[i] > T.padr) T.padr = T.off[i];
    }
    return T;
}

// Heights of a column and its pads fit the staging buffer.
__device__ __forceinline__ bool z_padded(const ZTaps& T, int nz) {
    return (long long)nz + T.padl + T.padr <= DFZ_MAXNZ;
}

// A[j] from the staged column (fn[j] = height j; PAD: heights -padl .. nz-1+padr hold the clamped
// values).  Two partial sums in a fixed order.
template <bool PAD>
__device__ __forceinline__ double tap_sum(const double* fn, int nz, int j, const ZTaps& T) {
    double a = 0.0, b = 0.0;
    auto at = [&](int i) { return fn[PAD ? j + T.off[i] : clampi(j + T.off[i], nz)]; };
    // unrolled over the most taps there can be: offsets and weights are then immediate constant-bank
    // operands (indexed constant loads per tap bound the rolled loop: 140 us on the 480 x 480 x 60 volume)
#pragma unroll
    for (int i = 0; i < 2 * NQ; i += 2) {
        if (i < T.n) a = __fma_rn(T.w[i], at(i), a);
        if (i + 1 < T.n) b = __fma_rn(T.w[i + 1], at(i + 1), b);
    }
    return a + b;
}

// df of one staged column by a warp: store(o, value) for every output o, whose height is iz_of(o)
// (outside [0, nz): NaN); c1, c2: -n_z^2 / dr and -n_z^2 / (2 dr).  nz >= 2.
template <bool PAD, class IzOf, class Store>
__device__ __forceinline__ void df_column(const double* fn, double* row, int nz, int l, const ZTaps& T, double c1,
                                          double c2, int n_out, const IzOf& iz_of, const Store& store) {
    const bool tab = nz <= DFZ_TAB;
    if (tab) {
        for (int j = l; j < nz; j += 32) row[j] = tap_sum<PAD>(fn, nz, j, T);
        __syncwarp();
    }
    auto A = [&](int j) { return tab ? row[j] : tap_sum<PAD>(fn, nz, j, T); };
    for (int o = l; o < n_out; o += 32) {
        const int iz = iz_of(o);
        if (iz < 0 || iz >= nz) {
            store(o, __int_as_float(0x7fc00000));
            continue;
        }
        const int jp = iz + 1 < nz ? iz + 1 : nz - 1, jm = iz > 0 ? iz - 1 : 0;
        store(o, (float)((A(jp) - A(jm)) * (jp - jm == 2 ? c2 : c1)));
    }
}

// Fz of row i of a z-only oscillation, NaN where Fx or Fy is not finite (the general sum F.n multiplies
// them by 0).  A float row takes no FP64 arithmetic beyond its one conversion; n_z is applied to the
// difference.
__device__ __forceinline__ double z_at(const float* __restrict__ v, size_t i) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(v) + i);
    return (double)((f.x * 0.f + f.y * 0.f) + f.z);
}
__device__ __forceinline__ double z_at(const double* __restrict__ v, size_t i) {
    const Row f = load_row(v, i);
    return (f.x * 0.0 + f.y * 0.0) + f.z;
}

// Stage a column (fn_at(z), z < nz) with its end values repeated over the pads.
template <class FnAt>
__device__ __forceinline__ void stage_column(double* buf, int nz, int l, int padl, int padr, const FnAt& fn_at_z) {
    for (int z = l; z < nz; z += 32) buf[padl + z] = fn_at_z(z);
    __syncwarp();
    for (int i = l; i < padl; i += 32) buf[i] = buf[padl];
    for (int i = l; i < padr; i += 32) buf[padl + nz + i] = buf[padl + nz - 1];
    __syncwarp();
}

template <typename T>
__global__ void __launch_bounds__(DFZ_WARPS * 32)
df_amp_z_kernel(const T* __restrict__ FEs, DfGeom P, ZTaps Z, const int* __restrict__ out_iz, int n_out,
                float* __restrict__ df) {
    __shared__ double s_fn[DFZ_WARPS][DFZ_MAXNZ];
    __shared__ double s_row[DFZ_WARPS][DFZ_TAB];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const long long pix = (long long)blockIdx.x * DFZ_WARPS + w;
    if (pix >= (long long)P.nx * P.ny) return;  // whole warp exits together: no CTA barrier below
    const int nz = P.nz;
    const bool pad = z_padded(Z, nz);
    double* fn = s_fn[w] + (pad ? Z.padl : 0);
    stage_column(s_fn[w], nz, l, pad ? Z.padl : 0, pad ? Z.padr : 0, [&](int z) { return z_at(FEs, (size_t)pix * nz + z); });
    const double n2 = -P.n[2] * P.n[2], c1 = n2 * P.idr[2], c2 = n2 * P.idr2[2];
    auto iz_of = [&](int o) { return out_iz ? out_iz[o] : o; };
    auto store = [&](int o, float v) { df[pix * n_out + o] = v; };
    if (pad) df_column<true>(fn, s_row[w], nz, l, Z, c1, c2, n_out, iz_of, store);
    else df_column<false>(fn, s_row[w], nz, l, Z, c1, c2, n_out, iz_of, store);
}

// Any other oscillation direction: the same filter in three dimensions.  Node k
// reads the eight corners of one cell at a constant offset with constant
// weights, so A = sum_k wk S(., u_k) is at most 72 taps (merged on the host) and
// df = -sum_a n_a dA/dr_a.  A CTA stages F_n of its tile, widened by the taps'
// reach and one sample for the differences, in shared memory (indices clamped to
// the volume, mode='nearest'), forms A once per point of the tile and takes the
// differences from it.  df_amp_dir_kernel evaluates 9 nodes x 3 axes x 2 samples
// x 8 corners per output from global memory, 432 rows against 72 shared doubles
// and 2 staged rows: 482 -> 41 us on a 101 x 97 x 41 float64 volume.
constexpr int DFT_THREADS = 256;
constexpr int DFT_MAX = 8 * NQ;

struct TileTaps {
    int n;
    int lo[3], hi[3];        // reach of the taps along each axis
    int t[3];                // outputs per tile
    int a[3], f[3];          // points of A and of F_n per tile
    int e[3];                // 1 along the axes that are differentiated
    int off[DFT_MAX];        // linear offsets in the staged F_n
    double w[DFT_MAX];
};

template <typename T>
__global__ void __launch_bounds__(DFT_THREADS)
df_amp_tile_kernel(const T* __restrict__ FEs, DfGeom P, TileTaps Q, int nty, int ntz, const int* __restrict__ out_iz,
                   int n_out, float* __restrict__ df) {
    extern __shared__ double s_tile[];
    double* s_f = s_tile;
    double* s_a = s_tile + Q.f[0] * Q.f[1] * Q.f[2];
    const int b = blockIdx.x;
    const int o0[3] = {b / (nty * ntz) * Q.t[0], b / ntz % nty * Q.t[1], b % ntz * Q.t[2]};
    const int nf = Q.f[0] * Q.f[1] * Q.f[2], na = Q.a[0] * Q.a[1] * Q.a[2];
    for (int i = threadIdx.x; i < nf; i += DFT_THREADS) {
        const int z = i % Q.f[2], y = i / Q.f[2] % Q.f[1], x = i / Q.f[2] / Q.f[1];
        s_f[i] = fn_at(FEs, P, clampi(o0[0] - Q.e[0] + Q.lo[0] + x, P.nx), clampi(o0[1] - Q.e[1] + Q.lo[1] + y, P.ny),
                       clampi(o0[2] - Q.e[2] + Q.lo[2] + z, P.nz));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < na; i += DFT_THREADS) {
        const int z = i % Q.a[2], y = i / Q.a[2] % Q.a[1], x = i / Q.a[2] / Q.a[1];
        const double* f = s_f + ((x - Q.lo[0]) * Q.f[1] + (y - Q.lo[1])) * Q.f[2] + (z - Q.lo[2]);
        double s0 = 0.0, s1 = 0.0;
        int k = 0;
#pragma unroll 4
        for (; k + 1 < Q.n; k += 2) {
            s0 = __fma_rn(Q.w[k], f[Q.off[k]], s0);
            s1 = __fma_rn(Q.w[k + 1], f[Q.off[k + 1]], s1);
        }
        if (k < Q.n) s0 = __fma_rn(Q.w[k], f[Q.off[k]], s0);
        s_a[i] = s0 + s1;
    }
    __syncthreads();
    // with a height list (out_iz) ntz is 1 and the tile holds every height
    const int zo = out_iz ? n_out : min(Q.t[2], P.nz - o0[2]);
    const int xo = min(Q.t[0], P.nx - o0[0]), yo = min(Q.t[1], P.ny - o0[1]);
    const int dims[3] = {P.nx, P.ny, P.nz}, st[3] = {Q.a[1] * Q.a[2], Q.a[2], 1};
    for (int i = threadIdx.x; i < xo * yo * zo; i += DFT_THREADS) {
        const int o = i % zo, y = i / zo % yo, x = i / zo / yo;
        const int iz = out_iz ? out_iz[o] : o0[2] + o;
        const size_t at = ((size_t)(o0[0] + x) * P.ny + (o0[1] + y)) * n_out + (out_iz ? o : iz);
        if (iz < 0 || iz >= P.nz) {
            df[at] = __int_as_float(0x7fc00000);
            continue;
        }
        const int g[3] = {o0[0] + x, o0[1] + y, iz};
        const double* A = s_a + ((x + Q.e[0]) * Q.a[1] + (y + Q.e[1])) * Q.a[2] + (iz - o0[2] + Q.e[2]);
        double acc = 0.0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            if (!Q.e[d]) continue;
            const int up = g[d] + 1 < dims[d] ? 1 : 0, dn = g[d] > 0 ? 1 : 0;
            acc -= P.n[d] * ((A[up * st[d]] - A[-dn * st[d]]) * (up + dn == 2 ? P.idr2[d] : P.idr[d]));
        }
        df[at] = (float)acc;
    }
}

// Taps and tile of a direction; false when the shift's reach leaves no tile that fits shared memory
// (the general kernel then).  The tile: 4 x 8 columns of up to 32 heights (all of them with a height
// list), halved along x, y while it does not fit 96 KB (two CTAs per SM).
bool make_tile(const DfGeom& P, bool list, TileTaps& Q) {
    const int dims[3] = {P.nx, P.ny, P.nz};
    Q = TileTaps{};
    struct Tap { int o[3]; double w; } tap[DFT_MAX];
    for (int d = 0; d < 3; d++)
        if (!(fabs(P.shift[d]) < 1e6)) return false;
    for (int a = 0; a < P.nact; a++) Q.e[P.act[a]] = 1;
    for (int k = 0; k < NQ; k++) {
        long long m[3];
        double t[3];
        for (int d = 0; d < 3; d++) split_shift(P.uk[k] * P.shift[d], m[d], t[d]);
        for (int c = 0; c < 8; c++) {
            double w = P.wk;
            int o[3];
            for (int d = 0; d < 3; d++) {
                const int hi = (c >> (2 - d)) & 1;
                w *= hi ? t[d] : 1.0 - t[d];
                o[d] = (int)m[d] + hi;
            }
            if (w == 0.0) continue;
            int i = 0;
            while (i < Q.n && !(tap[i].o[0] == o[0] && tap[i].o[1] == o[1] && tap[i].o[2] == o[2])) i++;
            if (i < Q.n) {
                tap[i].w += w;
                continue;
            }
            tap[Q.n].w = w;
            for (int d = 0; d < 3; d++) tap[Q.n].o[d] = o[d];
            Q.n++;
        }
    }
    for (int d = 0; d < 3; d++) {
        Q.lo[d] = Q.hi[d] = tap[0].o[d];
        for (int i = 1; i < Q.n; i++) {
            Q.lo[d] = Q.lo[d] < tap[i].o[d] ? Q.lo[d] : tap[i].o[d];
            Q.hi[d] = Q.hi[d] > tap[i].o[d] ? Q.hi[d] : tap[i].o[d];
        }
    }
    Q.t[0] = 4;
    Q.t[1] = 8;
    const int nzt = list ? 1 : (P.nz + 31) / 32;
    Q.t[2] = (P.nz + nzt - 1) / nzt;
    while (true) {
        long long nf = 1, na = 1;
        for (int d = 0; d < 3; d++) {
            if (Q.t[d] > dims[d]) Q.t[d] = dims[d];
            Q.a[d] = Q.t[d] + 2 * Q.e[d];
            Q.f[d] = Q.a[d] + Q.hi[d] - Q.lo[d];
            nf *= Q.f[d];
            na *= Q.a[d];
        }
        if ((nf + na) * 8 <= 96 * 1024) break;
        const int d = Q.t[0] >= Q.t[1] ? 0 : 1;
        if (Q.t[d] == 1) return false;
        Q.t[d] = (Q.t[d] + 1) / 2;
    }
    for (int i = 0; i < Q.n; i++) {
        Q.w[i] = tap[i].w;
        Q.off[i] = (tap[i].o[0] * Q.f[1] + tap[i].o[1]) * Q.f[2] + tap[i].o[2];
    }
    return true;
}

// Node by node (df_amp_dir_kernel) where the tiles would do more: they form A at every height of their columns,
// whatever the list, and a long reach across stages hundreds of points per output.  Times as fitted on volumes of 64^2
// to 480^2 pixels, in us: node by node 33 per axis (latency) + 1.8e-6 per row read (2.8e-6 for the scattered heights of
// a list); tiles 5.9e-6 per staged point + 3e-7 per tap.  Three axes, 480 x 480 x 60: 1 height 478 us and 1315 by
// tiles, 3 1033 and 1316, 4 1323 and 1317, all 12742 and 1230; along (1, 1, 0) with a reach of 9 samples, 64 x 64 x
// 100: 150 and 555.
bool by_nodes(const DfGeom& P, const TileTaps& Q, int n_out, bool list) {
    double tiles = 1.0;
    const int dims[3] = {P.nx, P.ny, P.nz};
    for (int d = 0; d < 3; d++) tiles *= (dims[d] + Q.t[d] - 1) / Q.t[d];
    const double staged = (double)Q.f[0] * Q.f[1] * Q.f[2], points = (double)Q.a[0] * Q.a[1] * Q.a[2];
    const double rows = (double)P.nx * P.ny * n_out * P.nact * (2.0 * DFT_MAX);
    return 33.0 * P.nact + rows * (list ? 2.8e-6 : 1.8e-6) < tiles * (staged * 5.9e-6 + points * Q.n * 3e-7);
}

template <typename T>
int launch_df_tile(const T* FEs, const DfGeom& P, const TileTaps& Q, const int* out_iz, int n_out, float* df,
                   cudaStream_t st) {
    const size_t smem = ((size_t)Q.f[0] * Q.f[1] * Q.f[2] + (size_t)Q.a[0] * Q.a[1] * Q.a[2]) * sizeof(double);
    if (smem > 48 * 1024 && cudaFuncSetAttribute(df_amp_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem) != cudaSuccess)
        return set_error(SPM_ERR_CUDA, "spm_df_amp_dir: cannot enable %zu B of shared memory", smem);
    const int ntx = (P.nx + Q.t[0] - 1) / Q.t[0], nty = (P.ny + Q.t[1] - 1) / Q.t[1];
    const int ntz = (P.nz + Q.t[2] - 1) / Q.t[2];
    df_amp_tile_kernel<<<(unsigned)((long long)ntx * nty * ntz), DFT_THREADS, smem, st>>>(FEs, P, Q, nty, ntz, out_iz,
                                                                                        n_out, df);
    return check_launch("spm_df_amp_dir");
}

template <typename T>
__global__ void __launch_bounds__(DF_THREADS)
df_dir_kernel(const T* __restrict__ FEs, DfGeom P, double* __restrict__ df) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)P.nx * P.ny * P.nz;
    if (gid >= total) return;
    const int iz = (int)(gid % P.nz);
    const long long pix = gid / P.nz;
    const int iy = (int)(pix % P.ny), ix = (int)(pix / P.ny);
    double acc = 0.0;
    for (int a = 0; a < P.nact; a++) {
        const int ax = P.act[a];
        acc -= P.n[ax] * grad_at<false>(FEs, P, ax, ix, iy, iz, 0.0);
    }
    df[gid] = acc;
}

struct DissGeom {
    int nx, ny, nz, n_out;
    double n[3];
};

// |sum_j (x[j+1]-x[j]) * (y[j] + y[j+1]) / 2| over the masked heights.  Float
// volumes use spm_diss.cuh's diss_value (shared with the fused epilogue of the
// paired relaxation in relax.cu): the same operations, as written below.
__global__ void __launch_bounds__(DF_THREADS)
dissipation_f32_kernel(const float4* __restrict__ Ff, const float4* __restrict__ Fb, DissGeom P,
                       const double* __restrict__ h, const int* __restrict__ off, const int* __restrict__ idx,
                       float* __restrict__ E) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)P.nx * P.ny * P.n_out;
    if (gid >= total) return;
    const int o = (int)(gid % P.n_out);
    const long long pix = gid / P.n_out;
    const double n[3] = {P.n[0], P.n[1], P.n[2]};
    E[gid] = diss_value(Ff, Fb, (size_t)pix * P.nz, P.nz, n, h, off, idx, o, LdgLoad{});
}

template <typename T>
__global__ void __launch_bounds__(DF_THREADS)
dissipation_kernel(const T* __restrict__ Ff, const T* __restrict__ Fb, DissGeom P,
                   const double* __restrict__ h, const int* __restrict__ off, const int* __restrict__ idx,
                   float* __restrict__ E) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)P.nx * P.ny * P.n_out;
    if (gid >= total) return;
    const int o = (int)(gid % P.n_out);
    const long long pix = gid / P.n_out;
    auto dF = [&](int j) {
        const Row a = load_row(Ff, (size_t)pix * P.nz + j), b = load_row(Fb, (size_t)pix * P.nz + j);
        const double fa = (a.x * P.n[0] + a.y * P.n[1]) + a.z * P.n[2];
        const double fbv = (b.x * P.n[0] + b.y * P.n[1]) + b.z * P.n[2];
        return fa - fbv;
    };
    double acc = 0.0;
    const int j0 = off[o], j1 = off[o + 1];
    for (int t = j0; t + 1 < j1; t++) {
        const int a = idx[t], b = idx[t + 1];
        if (a < 0 || a >= P.nz || b < 0 || b >= P.nz) {  // invalid index list: flag, never read out of bounds
            acc = __longlong_as_double(0x7ff8000000000000LL);
            break;
        }
        acc += (h[b] - h[a]) * (dF(a) + dF(b)) / 2.0;
    }
    E[gid] = (float)fabs(acc);
}

// ---- df loss seed: df, per-block partial sums of w and w*(df-t)^2 ----------
constexpr int LS_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(LS_THREADS)
loss_partials_kernel(const T* __restrict__ FEs, const double* __restrict__ tgt, const double* __restrict__ wts,
                     int nx, int ny, int nz, double idz2, double* __restrict__ df_out, double* __restrict__ partial) {
    __shared__ double s_w[LS_THREADS], s_l[LS_THREADS];
    const long long total = (long long)nx * ny * nz;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double w = 0.0, l = 0.0;
    if (gid < total) {
        const int iz = (int)(gid % nz);
        double d = 0.0;
        if (iz > 0 && iz < nz - 1) {
            const double fp = load_row(FEs, gid + 1).z, fm = load_row(FEs, gid - 1).z;
            d = -(fp - fm) * idz2;
        }
        df_out[gid] = d;
        w = wts ? wts[gid] : ((iz > 0 && iz < nz - 1) ? 1.0 : 0.0);
        const double diff = d - tgt[gid];
        l = w * (diff * diff);
    }
    s_w[threadIdx.x] = w;
    s_l[threadIdx.x] = l;
    __syncthreads();
    for (int s = LS_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            s_w[threadIdx.x] += s_w[threadIdx.x + s];
            s_l[threadIdx.x] += s_l[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        partial[2 * blockIdx.x] = s_w[0];
        partial[2 * blockIdx.x + 1] = s_l[0];
    }
}

// One CTA folds the per-block partials in a fixed order: (wsum, loss).
__global__ void __launch_bounds__(LS_THREADS)
loss_final_kernel(const double* __restrict__ partial, int nblk, double* __restrict__ sums, double* __restrict__ loss) {
    __shared__ double s_w[LS_THREADS], s_l[LS_THREADS];
    double w = 0.0, l = 0.0;
    for (int i = threadIdx.x; i < nblk; i += LS_THREADS) {
        w += partial[2 * i];
        l += partial[2 * i + 1];
    }
    s_w[threadIdx.x] = w;
    s_l[threadIdx.x] = l;
    __syncthreads();
    for (int s = LS_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            s_w[threadIdx.x] += s_w[threadIdx.x + s];
            s_l[threadIdx.x] += s_l[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        sums[0] = s_w[0];
        sums[1] = s_l[0];
        loss[0] = 0.5 * s_l[0] / s_w[0];
    }
}

// dL/dFz = transpose of the central-difference stencil applied to w*(df-t)/wsum (df and the
// gradient multiply by the reciprocals 1/(2 dz) and 1/wsum, computed once: within an ulp of the
// divisions, which cost the loss kernels a divergent FP64 division per state).
__global__ void __launch_bounds__(LS_THREADS)
loss_grad_kernel(const double* __restrict__ df, const double* __restrict__ tgt, const double* __restrict__ wts,
                 const double* __restrict__ sums, int nx, int ny, int nz, double coeff, float4* __restrict__ dL) {
    const long long total = (long long)nx * ny * nz;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= total) return;
    const int iz = (int)(gid % nz);
    const double iwsum = 1.0 / sums[0];  // one division per thread, the same for every thread
    auto g = [&](long long j) {
        const int jz = (int)(j % nz);
        const double w = wts ? wts[j] : ((jz > 0 && jz < nz - 1) ? 1.0 : 0.0);
        return w * (df[j] - tgt[j]) * iwsum;
    };
    double v;
    if (iz == 0) v = g(gid + 1) * coeff;
    else if (iz == nz - 1) v = -g(gid - 1) * coeff;
    else v = (g(gid + 1) - g(gid - 1)) * coeff;
    dL[gid] = make_float4(0.f, 0.f, (float)v, 0.f);
}

int fill_geom(DfGeom& P, int nx, int ny, int nz, const double* n, const double* dr, double amp) {
    P.nx = nx; P.ny = ny; P.nz = nz;
    P.nact = 0;
    for (int d = 0; d < 3; d++) {
        P.n[d] = n[d];
        P.dr[d] = dr[d];
        P.shift[d] = (amp * n[d]) / dr[d];
        P.idr[d] = 1.0 / dr[d];
        P.idr2[d] = 1.0 / (2.0 * dr[d]);
        if (fabs(n[d]) > 1e-15) P.act[P.nact++] = d;
    }
    for (int k = 0; k < NQ; k++) P.uk[k] = cos((double)(2 * k + 1) / (double)(2 * NQ) * M_PI);
    P.wk = 1.0 / NQ;
    const int dims[3] = {nx, ny, nz};
    for (int a = 0; a < P.nact; a++)
        if (dims[P.act[a]] < 2)
            return set_error(SPM_ERR_ARG, "df: FEs axis %d needs at least 2 samples for this oscillation direction",
                             P.act[a]);
    return SPM_OK;
}

}  // namespace
}  // namespace spm

extern "C" int spm_df_amp_dir(const void* FEs, int fes_dtype, int nx, int ny, int nz, const double* n,
                              const double* dr, double amp, const int* out_iz, int n_out, float* df, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(FEs && df && n && dr, "spm_df_amp_dir: null pointer");
    SPM_REQUIRE(fes_dtype == SPM_F32 || fes_dtype == SPM_F64, "spm_df_amp_dir: fes_dtype=%d", fes_dtype);
    SPM_REQUIRE(nx > 0 && ny > 0 && nz > 0, "spm_df_amp_dir: dims (%d,%d,%d) must be positive", nx, ny, nz);
    SPM_REQUIRE(aligned16(FEs), "spm_df_amp_dir: FEs not 16-byte aligned");
    for (int d = 0; d < 3; d++)
        SPM_REQUIRE(std::isfinite(n[d]) && std::isfinite(dr[d]) && dr[d] > 0.0,
                    "spm_df_amp_dir: n/dr must be finite with dr > 0");
    SPM_REQUIRE(std::isfinite(amp), "spm_df_amp_dir: amp must be finite");
    DfGeom P;
    int rc = fill_geom(P, nx, ny, nz, n, dr, amp);
    if (rc) return rc;
    if (out_iz == nullptr) n_out = nz;
    SPM_REQUIRE(n_out >= 0, "spm_df_amp_dir: n_out=%d < 0", n_out);
    const long long total = (long long)nx * ny * n_out;
    if (total == 0) return SPM_OK;
    if (n[0] == 0.0 && n[1] == 0.0 && nz <= DFZ_MAXNZ) {  // z-only oscillation: column kernel
        const long long npix = (long long)nx * ny;
        const unsigned nb = (unsigned)((npix + DFZ_WARPS - 1) / DFZ_WARPS);
        const ZTaps Z = make_ztaps(P, P.shift[2]);
        if (fes_dtype == SPM_F32)
            df_amp_z_kernel<<<nb, DFZ_WARPS * 32, 0, as_stream(stream)>>>(static_cast<const float*>(FEs), P, Z, out_iz,
                                                                           n_out, df);
        else
            df_amp_z_kernel<<<nb, DFZ_WARPS * 32, 0, as_stream(stream)>>>(static_cast<const double*>(FEs), P, Z, out_iz,
                                                                           n_out, df);
        return check_launch("spm_df_amp_dir");
    }
    TileTaps Q;
    if (make_tile(P, out_iz != nullptr, Q) && !by_nodes(P, Q, n_out, out_iz != nullptr)) {
        if (fes_dtype == SPM_F32)
            return launch_df_tile(static_cast<const float*>(FEs), P, Q, out_iz, n_out, df, as_stream(stream));
        return launch_df_tile(static_cast<const double*>(FEs), P, Q, out_iz, n_out, df, as_stream(stream));
    }
    const unsigned nb = (unsigned)((total + DF_THREADS - 1) / DF_THREADS);
    if (fes_dtype == SPM_F32)
        df_amp_dir_kernel<<<nb, DF_THREADS, 0, as_stream(stream)>>>(static_cast<const float*>(FEs), P, out_iz, n_out, df);
    else
        df_amp_dir_kernel<<<nb, DF_THREADS, 0, as_stream(stream)>>>(static_cast<const double*>(FEs), P, out_iz, n_out, df);
    return check_launch("spm_df_amp_dir");
}

extern "C" int spm_df_dir(const void* FEs, int fes_dtype, int nx, int ny, int nz, const double* n, const double* dr,
                          double* df, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(FEs && df && n && dr, "spm_df_dir: null pointer");
    SPM_REQUIRE(fes_dtype == SPM_F32 || fes_dtype == SPM_F64, "spm_df_dir: fes_dtype=%d", fes_dtype);
    SPM_REQUIRE(nx > 0 && ny > 0 && nz > 0, "spm_df_dir: dims (%d,%d,%d) must be positive", nx, ny, nz);
    SPM_REQUIRE(aligned16(FEs), "spm_df_dir: FEs not 16-byte aligned");
    for (int d = 0; d < 3; d++)
        SPM_REQUIRE(std::isfinite(n[d]) && std::isfinite(dr[d]) && dr[d] > 0.0, "spm_df_dir: n/dr must be finite, dr > 0");
    DfGeom P;
    int rc = fill_geom(P, nx, ny, nz, n, dr, 0.0);
    if (rc) return rc;
    const long long total = (long long)nx * ny * nz;
    const unsigned nb = (unsigned)((total + DF_THREADS - 1) / DF_THREADS);
    if (fes_dtype == SPM_F32)
        df_dir_kernel<<<nb, DF_THREADS, 0, as_stream(stream)>>>(static_cast<const float*>(FEs), P, df);
    else
        df_dir_kernel<<<nb, DF_THREADS, 0, as_stream(stream)>>>(static_cast<const double*>(FEs), P, df);
    return check_launch("spm_df_dir");
}

extern "C" int spm_dissipation(const void* FEs_fwd, const void* FEs_bwd, int fes_dtype, int nx, int ny, int nz,
                               const double* n, const double* h_scan, const int* off, const int* idx, int n_out,
                               float* E_diss, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(FEs_fwd && FEs_bwd && n && h_scan && off && idx && E_diss, "spm_dissipation: null pointer");
    SPM_REQUIRE(fes_dtype == SPM_F32 || fes_dtype == SPM_F64, "spm_dissipation: fes_dtype=%d", fes_dtype);
    SPM_REQUIRE(nx > 0 && ny > 0 && nz > 0 && n_out >= 0, "spm_dissipation: bad dims (%d,%d,%d) n_out=%d", nx, ny, nz,
                n_out);
    SPM_REQUIRE(aligned16(FEs_fwd) && aligned16(FEs_bwd), "spm_dissipation: FEs not 16-byte aligned");
    DissGeom P;
    P.nx = nx; P.ny = ny; P.nz = nz; P.n_out = n_out;
    for (int d = 0; d < 3; d++) P.n[d] = n[d];
    const long long total = (long long)nx * ny * n_out;
    if (total == 0) return SPM_OK;
    const unsigned nb = (unsigned)((total + DF_THREADS - 1) / DF_THREADS);
    if (fes_dtype == SPM_F32)
        dissipation_f32_kernel<<<nb, DF_THREADS, 0, as_stream(stream)>>>(
            static_cast<const float4*>(FEs_fwd), static_cast<const float4*>(FEs_bwd), P, h_scan, off, idx, E_diss);
    else
        dissipation_kernel<<<nb, DF_THREADS, 0, as_stream(stream)>>>(static_cast<const double*>(FEs_fwd),
                                                                     static_cast<const double*>(FEs_bwd), P, h_scan,
                                                                     off, idx, E_diss);
    return check_launch("spm_dissipation");
}

extern "C" long long spm_df_loss_scratch_bytes(int nx, int ny, int nz) {
    const long long total = (long long)nx * ny * nz;
    if (nx <= 0 || ny <= 0 || nz <= 0) return 0;
    const long long nblk = (total + spm::LS_THREADS - 1) / spm::LS_THREADS;
    return (2 * nblk + 2) * (long long)sizeof(double);
}

extern "C" int spm_df_loss_seed(const void* FEs, int fes_dtype, const double* target, const double* weights, int nx,
                                int ny, int nz, double dtip, double* df_out, float* dL_dFEs, double* loss_out,
                                void* scratch, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(FEs && target && df_out && dL_dFEs && loss_out && scratch, "spm_df_loss_seed: null pointer");
    SPM_REQUIRE(fes_dtype == SPM_F32 || fes_dtype == SPM_F64, "spm_df_loss_seed: fes_dtype=%d", fes_dtype);
    SPM_REQUIRE(nx > 0 && ny > 0, "spm_df_loss_seed: nx=%d ny=%d must be positive", nx, ny);
    SPM_REQUIRE(nz >= 3, "spm_df_loss_seed: need nz>=3 for central difference, got nz=%d", nz);
    SPM_REQUIRE(dtip < 0.0, "spm_df_loss_seed: dtip must be <0, got dtip=%g", dtip);
    SPM_REQUIRE(aligned16(FEs) && aligned16(dL_dFEs), "spm_df_loss_seed: FEs/dL_dFEs not 16-byte aligned");
    SPM_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 7u) == 0, "spm_df_loss_seed: scratch not 8-byte aligned");
    const long long total = (long long)nx * ny * nz;
    const long long nblk = (total + LS_THREADS - 1) / LS_THREADS;
    SPM_REQUIRE(nblk < (1LL << 31), "spm_df_loss_seed: volume too large");
    double* partial = reinterpret_cast<double*>(scratch);
    double* sums = partial + 2 * nblk;
    const double dz = fabs(dtip);
    cudaStream_t st = as_stream(stream);
    if (fes_dtype == SPM_F32)
        loss_partials_kernel<<<(unsigned)nblk, LS_THREADS, 0, st>>>(static_cast<const float*>(FEs), target, weights,
                                                                    nx, ny, nz, 1.0 / (2.0 * dz), df_out, partial);
    else
        loss_partials_kernel<<<(unsigned)nblk, LS_THREADS, 0, st>>>(static_cast<const double*>(FEs), target, weights,
                                                                    nx, ny, nz, 1.0 / (2.0 * dz), df_out, partial);
    loss_final_kernel<<<1, LS_THREADS, 0, st>>>(partial, (int)nblk, sums, loss_out);
    loss_grad_kernel<<<(unsigned)nblk, LS_THREADS, 0, st>>>(df_out, target, weights, sums, nx, ny, nz,
                                                            1.0 / (2.0 * dz), reinterpret_cast<float4*>(dL_dFEs));
    return check_launch("spm_df_loss_seed");
}

// ---------------------------------------------------------------------------
// Batched df and df loss: each molecule's states are its (n_scan,1,nz_steps)
// volume (z-step fastest, the first z-step highest).  Work items find their
// molecule through the descriptor prefixes (pix_off, chunk_off); every
// per-element expression and every reduction order is the single-volume
// kernel's, so each molecule's results are bit-identical to those calls.
// ---------------------------------------------------------------------------
namespace spm {
namespace {

// Warp per stroke.  The stroke is staged lowest z-step first, so the column
// is the ascending volume spm_df_amp_dir expects (dr = |dtip| > 0); results
// are written back in stroke order.
__global__ void __launch_bounds__(DFZ_WARPS * 32)
batch_df_amp_kernel(int n_mol, const spm_batch_mol* __restrict__ mols, long long n_pix,
                    const float* __restrict__ FEs, DfGeom P, ZTaps Z, float* __restrict__ df) {
    __shared__ double s_fn[DFZ_WARPS][DFZ_MAXNZ];
    __shared__ double s_row[DFZ_WARPS][DFZ_TAB];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const long long pix = (long long)blockIdx.x * DFZ_WARPS + w;
    if (pix >= n_pix) return;  // whole warp exits together: no CTA barrier below
    const spm_batch_mol* D = mols + SPM_MOL_BY(pix_off, mols, n_mol, pix);
    const int nz = D->nz_steps;
    const long long s0 = D->state_off + (pix - D->pix_off) * (long long)nz;
    if (nz < 2 || nz > DFZ_MAXNZ) {  // no central difference (or no room): flag the stroke
        for (int o = l; o < nz; o += 32) df[s0 + o] = __int_as_float(0x7fc00000);
        return;
    }
    const bool pad = z_padded(Z, nz);
    double* fn = s_fn[w] + (pad ? Z.padl : 0);
    stage_column(s_fn[w], nz, l, pad ? Z.padl : 0, pad ? Z.padr : 0, [&](int z) { return z_at(FEs, (size_t)(s0 + (nz - 1 - z))); });
    const double c1 = -P.idr[2], c2 = -P.idr2[2];  // n = z
    auto iz_of = [](int o) { return o; };
    auto store = [&](int o, float v) { df[s0 + (nz - 1 - o)] = v; };
    if (pad) df_column<true>(fn, s_row[w], nz, l, Z, c1, c2, nz, iz_of, store);
    else df_column<false>(fn, s_row[w], nz, l, Z, c1, c2, nz, iz_of, store);
}

// Loss chunks per CTA of the partials and gradient kernels.  The first
// chunk's molecule is found by binary search, the next ones by stepping
// forward from it, so the search's dependent descriptor loads are paid once
// per LS_CHUNKS chunks; every chunk is computed and reduced exactly as alone.
constexpr int LS_CHUNKS = 4;

// The chunk's single-volume tree (v[t] += v[t+s], s = 128 .. 1) of its threads' (w, l):
// levels >= 32 through shared memory, the last five in warp 0 by shuffles -- the same
// additions in the same order.  Ends with a barrier, so s_w / s_l can be reused.
__device__ __forceinline__ void chunk_partials(double w, double l, double* s_w, double* s_l, double* out) {
    s_w[threadIdx.x] = w;
    s_l[threadIdx.x] = l;
    __syncthreads();
    for (int s = LS_THREADS / 2; s >= 32; s >>= 1) {
        if (threadIdx.x < s) {
            s_w[threadIdx.x] += s_w[threadIdx.x + s];
            s_l[threadIdx.x] += s_l[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x < 32) {
        double vw = s_w[threadIdx.x], vl = s_l[threadIdx.x];
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            vw += __shfl_down_sync(0xffffffffu, vw, s);
            vl += __shfl_down_sync(0xffffffffu, vl, s);
        }
        if (threadIdx.x == 0) {
            out[0] = vw;
            out[1] = vl;
        }
    }
    __syncthreads();
}

// LS_CHUNKS consecutive 256-state chunks per CTA: df and each chunk's (w, w*diff^2) sums.
__global__ void __launch_bounds__(LS_THREADS)
batch_loss_partials_kernel(int n_mol, long long n_chunks, const spm_batch_mol* __restrict__ mols,
                           const float* __restrict__ FEs, const double* __restrict__ tgt,
                           const double* __restrict__ wts, double idz2, double* __restrict__ df_out,
                           double* __restrict__ partial) {
    __shared__ double s_w[LS_THREADS], s_l[LS_THREADS];
    const long long c0 = (long long)blockIdx.x * LS_CHUNKS;
    int m = SPM_MOL_BY(chunk_off, mols, n_mol, c0);
    // every state's terms first (independent loads of all chunks in flight), then the reductions
    double wv[LS_CHUNKS], lv[LS_CHUNKS];
#pragma unroll
    for (int k = 0; k < LS_CHUNKS; k++) {
        const long long ch = c0 + k;
        wv[k] = 0.0;
        lv[k] = 0.0;
        if (ch >= n_chunks) continue;
        m = SPM_MOL_STEP(chunk_off, mols, n_mol, m, ch);
        const spm_batch_mol* D = mols + m;
        const int nz = D->nz_steps;
        const long long nst = (long long)D->n_scan * nz;
        const long long ls = (ch - D->chunk_off) * LS_THREADS + threadIdx.x;
        if (ls < nst) {
            const long long gid = D->state_off + ls;
            const int iz = ls < (1LL << 32) ? (int)((unsigned)ls % (unsigned)nz) : (int)(ls % nz);  // 32-bit when it fits
            double d = 0.0;
            if (iz > 0 && iz < nz - 1) {
                const double fp = load_row(FEs, gid + 1).z, fm = load_row(FEs, gid - 1).z;
                d = -(fp - fm) * idz2;
            }
            df_out[gid] = d;
            wv[k] = wts ? wts[gid] : ((iz > 0 && iz < nz - 1) ? 1.0 : 0.0);
            const double diff = d - tgt[gid];
            lv[k] = wv[k] * (diff * diff);
        }
    }
#pragma unroll
    for (int k = 0; k < LS_CHUNKS; k++)
        if (c0 + k < n_chunks) chunk_partials(wv[k], lv[k], s_w, s_l, partial + 2 * (c0 + k));  // uniform over the CTA
}

// CTA per molecule: fold its chunk partials in the fixed single-volume order.
__global__ void __launch_bounds__(LS_THREADS)
batch_loss_final_kernel(const spm_batch_mol* __restrict__ mols, const double* __restrict__ partial,
                        double* __restrict__ sums, double* __restrict__ loss) {
    __shared__ double s_w[LS_THREADS], s_l[LS_THREADS];
    const int m = blockIdx.x;
    const spm_batch_mol* D = mols + m;
    const long long nst = (long long)D->n_scan * D->nz_steps;
    const long long nblk = (nst + LS_THREADS - 1) / LS_THREADS;
    const double* pm = partial + 2 * D->chunk_off;
    double w = 0.0, l = 0.0;
    for (long long i = threadIdx.x; i < nblk; i += LS_THREADS) {
        w += pm[2 * i];
        l += pm[2 * i + 1];
    }
    s_w[threadIdx.x] = w;
    s_l[threadIdx.x] = l;
    __syncthreads();
    for (int s = LS_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            s_w[threadIdx.x] += s_w[threadIdx.x + s];
            s_l[threadIdx.x] += s_l[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        sums[2 * m] = s_w[0];
        sums[2 * m + 1] = s_l[0];
        // zero total weight (no pixels, or every state masked): the molecule contributes nothing,
        // where the single-volume formula would give 0/0
        loss[m] = s_w[0] > 0.0 ? 0.5 * s_l[0] / s_w[0] : 0.0;
    }
}

__global__ void __launch_bounds__(LS_THREADS)
batch_loss_grad_kernel(int n_mol, long long n_chunks, const spm_batch_mol* __restrict__ mols,
                       const double* __restrict__ df, const double* __restrict__ tgt, const double* __restrict__ wts,
                       const double* __restrict__ sums, double coeff, float4* __restrict__ dL) {
    const long long c0 = (long long)blockIdx.x * LS_CHUNKS;
    int m = SPM_MOL_BY(chunk_off, mols, n_mol, c0);
#pragma unroll
    for (int k = 0; k < LS_CHUNKS; k++) {
        const long long ch = c0 + k;
        if (ch >= n_chunks) return;
        m = SPM_MOL_STEP(chunk_off, mols, n_mol, m, ch);
        const spm_batch_mol* D = mols + m;
        const int nz = D->nz_steps;
        const long long nst = (long long)D->n_scan * nz;
        const long long ls = (ch - D->chunk_off) * LS_THREADS + threadIdx.x;
        if (ls >= nst) continue;
        const long long gid = D->state_off + ls;
        const int iz = ls < (1LL << 32) ? (int)((unsigned)ls % (unsigned)nz) : (int)(ls % nz);  // 32-bit when it fits
        const double wsum = sums[2 * m];
        // no central difference (nz < 3: the stencil would leave the stroke) or zero total
        // weight (no loss): no gradient
        if (nz < 3 || !(wsum > 0.0)) {
            dL[gid] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const double iwsum = 1.0 / wsum;  // one division per thread, uniform over the molecule's chunk
        auto g = [&](long long j, int jz) {  // jz: the z-step of state j
            const double w = wts ? wts[j] : ((jz > 0 && jz < nz - 1) ? 1.0 : 0.0);
            return w * (df[j] - tgt[j]) * iwsum;
        };
        double v;
        if (iz == 0) v = g(gid + 1, 1) * coeff;
        else if (iz == nz - 1) v = -g(gid - 1, iz - 1) * coeff;
        else v = (g(gid + 1, iz + 1) - g(gid - 1, iz - 1)) * coeff;
        dL[gid] = make_float4(0.f, 0.f, (float)v, 0.f);
    }
}

}  // namespace
}  // namespace spm

extern "C" int spm_batch_df_amp(int n_mol, const spm_batch_mol* mols, long long n_pixels, const float* FEs,
                                double dtip, double amp, float* df, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(n_mol >= 0 && n_pixels >= 0, "spm_batch_df_amp: negative sizes");
    if (n_mol == 0 || n_pixels == 0) return SPM_OK;
    SPM_REQUIRE(mols && FEs && df, "spm_batch_df_amp: null pointer");
    SPM_REQUIRE(aligned16(FEs), "spm_batch_df_amp: FEs not 16-byte aligned");
    SPM_REQUIRE(std::isfinite(dtip) && dtip != 0.0 && std::isfinite(amp), "spm_batch_df_amp: dtip=%g amp=%g", dtip, amp);
    const double n[3] = {0.0, 0.0, 1.0}, dr[3] = {1.0, 1.0, fabs(dtip)};
    DfGeom P;
    int rc = fill_geom(P, 1, 1, 2, n, dr, amp);
    if (rc) return rc;
    const long long nb = (n_pixels + DFZ_WARPS - 1) / DFZ_WARPS;
    SPM_REQUIRE(nb < (1LL << 31), "spm_batch_df_amp: too many pixels");
    batch_df_amp_kernel<<<(unsigned)nb, DFZ_WARPS * 32, 0, as_stream(stream)>>>(n_mol, mols, n_pixels, FEs, P,
                                                                                make_ztaps(P, P.shift[2]), df);
    return check_launch("spm_batch_df_amp");
}

extern "C" long long spm_batch_loss_scratch_bytes(long long n_chunks, int n_mol) {
    if (n_chunks < 0 || n_mol < 0) return 0;
    return (2 * n_chunks + 2 * (long long)n_mol) * (long long)sizeof(double);
}

namespace spm {
namespace {
// weights[s] = w_base[s] * (status[s-1] == 0 && status[s] == 0 && status[s+1] == 0), neighbours
// taken cyclically over the whole state array, status = diag[.].w.
__global__ void __launch_bounds__(256)
failure_mask_kernel(long long n, const float4* __restrict__ diag, const double* __restrict__ w_base,
                    double* __restrict__ weights) {
    const long long s = (long long)blockIdx.x * 256 + threadIdx.x;
    if (s >= n) return;
    const long long sm = s > 0 ? s - 1 : n - 1, sp = s + 1 < n ? s + 1 : 0;
    const bool ok = diag[s].w == 0.f && diag[sm].w == 0.f && diag[sp].w == 0.f;
    weights[s] = w_base[s] * (ok ? 1.0 : 0.0);
}
}  // namespace
}  // namespace spm

extern "C" int spm_batch_failure_mask(long long n_states, const float* diag, const double* w_base, double* weights,
                                      void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(n_states >= 0, "spm_batch_failure_mask: n_states=%lld", n_states);
    if (n_states == 0) return SPM_OK;
    SPM_REQUIRE(diag && w_base && weights && aligned16(diag), "spm_batch_failure_mask: null or misaligned buffers");
    const long long nb = (n_states + 255) / 256;
    SPM_REQUIRE(nb < (1LL << 31), "spm_batch_failure_mask: too many states");
    failure_mask_kernel<<<(unsigned)nb, 256, 0, as_stream(stream)>>>(n_states, reinterpret_cast<const float4*>(diag),
                                                                     w_base, weights);
    return check_launch("spm_batch_failure_mask");
}

extern "C" int spm_batch_df_loss_seed(int n_mol, const spm_batch_mol* mols, long long n_chunks, const float* FEs,
                                      const double* target, const double* weights, double dtip, double* df_out,
                                      float* dL_dFEs, double* loss_out, void* scratch, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(n_mol >= 0 && n_chunks >= 0, "spm_batch_df_loss_seed: negative sizes");
    if (n_mol == 0) return SPM_OK;
    SPM_REQUIRE(mols && loss_out && scratch, "spm_batch_df_loss_seed: null pointer");
    SPM_REQUIRE(dtip < 0.0, "spm_batch_df_loss_seed: dtip must be <0, got dtip=%g", dtip);
    SPM_REQUIRE(n_chunks < (1LL << 31), "spm_batch_df_loss_seed: too many states");
    SPM_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 7u) == 0, "spm_batch_df_loss_seed: scratch not 8-byte aligned");
    if (n_chunks > 0)
        SPM_REQUIRE(FEs && target && df_out && dL_dFEs && aligned16(FEs) && aligned16(dL_dFEs),
                    "spm_batch_df_loss_seed: null or misaligned state buffers");
    double* partial = static_cast<double*>(scratch);
    double* sums = partial + 2 * n_chunks;
    const double dz = fabs(dtip);
    cudaStream_t st = as_stream(stream);
    const unsigned nblk = (unsigned)((n_chunks + LS_CHUNKS - 1) / LS_CHUNKS);
    if (n_chunks > 0)
        batch_loss_partials_kernel<<<nblk, LS_THREADS, 0, st>>>(n_mol, n_chunks, mols, FEs, target, weights,
                                                                1.0 / (2.0 * dz), df_out, partial);
    batch_loss_final_kernel<<<(unsigned)n_mol, LS_THREADS, 0, st>>>(mols, partial, sums, loss_out);
    if (n_chunks > 0)
        batch_loss_grad_kernel<<<nblk, LS_THREADS, 0, st>>>(n_mol, n_chunks, mols, df_out, target, weights, sums,
                                                            1.0 / (2.0 * dz), reinterpret_cast<float4*>(dL_dFEs));
    return check_launch("spm_batch_df_loss_seed");
}

// ---------------------------------------------------------------------------
// Allocation-free df loss seed.
//
// Some callers cannot allocate device memory around this call: code that runs
// inside a host framework whose allocator owns all device memory (and may not
// be re-entered from the loss callback), callers that must never trigger an
// implicit device synchronisation from cudaMalloc/cudaFree in a latency-bound
// fitting loop, or callers that hold device memory budgets fixed up front.
// For them spm_df_loss_seed_noalloc takes no scratch argument: its per-block
// partial sums live in a fixed file-scope device array of
// SPM_DF_LOSS_NOALLOC_MAX_ELEMS / 256 (w, w*diff^2) pairs (1 MiB) that every
// GPU loading this library holds until the process exits.
// ---------------------------------------------------------------------------
#include <mutex>

namespace spm {
namespace {

constexpr long long NOALLOC_MAX_BLOCKS = SPM_DF_LOSS_NOALLOC_MAX_ELEMS / LS_THREADS;
// Shared by every call on a device: partials of block b at [2b, 2b+1], the
// final (wsum, sum) pair after them.  Each call overwrites every slot it later
// reads, so nothing has to be cleared between calls.
static __device__ __align__(256) double g_loss_scratch[2 * NOALLOC_MAX_BLOCKS + 2];

constexpr int MAX_DEVICES = 64;
std::mutex g_scratch_mutex;
double* g_scratch_addr[MAX_DEVICES] = {nullptr};

// Device address of g_loss_scratch on the current device (resolved once per
// device with that device current; the host-side symbol is not a device address).
int loss_scratch_address(double** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(SPM_ERR_CUDA, "spm_df_loss_seed_noalloc: cudaGetDevice: %s",
                                           cudaGetErrorString(e));
    if (dev < 0 || dev >= MAX_DEVICES)
        return set_error(SPM_ERR_UNSUPPORTED, "spm_df_loss_seed_noalloc: device ordinal %d >= %d", dev, MAX_DEVICES);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_addr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_loss_scratch);
        if (e != cudaSuccess || p == nullptr)
            return set_error(SPM_ERR_CUDA, "spm_df_loss_seed_noalloc: cudaGetSymbolAddress: %s",
                             cudaGetErrorString(e));
        g_scratch_addr[dev] = static_cast<double*>(p);
    }
    *out = g_scratch_addr[dev];
    return SPM_OK;
}

}  // namespace
}  // namespace spm

extern "C" int spm_df_loss_seed_noalloc(const void* FEs, int fes_dtype, const double* target, const double* weights,
                                        int nx, int ny, int nz, double dtip, double* df_out, float* dL_dFEs,
                                        double* loss_out, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(FEs && target && df_out && dL_dFEs && loss_out, "spm_df_loss_seed_noalloc: null pointer");
    SPM_REQUIRE(fes_dtype == SPM_F32 || fes_dtype == SPM_F64, "spm_df_loss_seed_noalloc: fes_dtype=%d", fes_dtype);
    SPM_REQUIRE(nx > 0 && ny > 0, "spm_df_loss_seed_noalloc: nx=%d ny=%d must be positive", nx, ny);
    SPM_REQUIRE(nz >= 3, "spm_df_loss_seed_noalloc: need nz>=3 for central difference, got nz=%d", nz);
    SPM_REQUIRE(dtip < 0.0, "spm_df_loss_seed_noalloc: dtip must be <0, got dtip=%g", dtip);
    SPM_REQUIRE(aligned16(FEs) && aligned16(dL_dFEs), "spm_df_loss_seed_noalloc: FEs/dL_dFEs not 16-byte aligned");
    const long long total = (long long)nx * ny * nz;
    if (total > SPM_DF_LOSS_NOALLOC_MAX_ELEMS)
        return set_error(SPM_ERR_UNSUPPORTED,
                         "spm_df_loss_seed_noalloc: volume of %lld elements exceeds the fixed scratch limit of %lld "
                         "(use spm_df_loss_seed with caller scratch)", total, (long long)SPM_DF_LOSS_NOALLOC_MAX_ELEMS);
    double* partial = nullptr;
    int rc = loss_scratch_address(&partial);
    if (rc) return rc;
    const long long nblk = (total + LS_THREADS - 1) / LS_THREADS;
    double* sums = partial + 2 * nblk;
    const double dz = fabs(dtip);
    cudaStream_t st = as_stream(stream);
    if (fes_dtype == SPM_F32)
        loss_partials_kernel<<<(unsigned)nblk, LS_THREADS, 0, st>>>(static_cast<const float*>(FEs), target, weights,
                                                                    nx, ny, nz, 1.0 / (2.0 * dz), df_out, partial);
    else
        loss_partials_kernel<<<(unsigned)nblk, LS_THREADS, 0, st>>>(static_cast<const double*>(FEs), target, weights,
                                                                    nx, ny, nz, 1.0 / (2.0 * dz), df_out, partial);
    loss_final_kernel<<<1, LS_THREADS, 0, st>>>(partial, (int)nblk, sums, loss_out);
    loss_grad_kernel<<<(unsigned)nblk, LS_THREADS, 0, st>>>(df_out, target, weights, sums, nx, ny, nz,
                                                            1.0 / (2.0 * dz), reinterpret_cast<float4*>(dL_dFEs));
    return check_launch("spm_df_loss_seed_noalloc");
}
