// grid_build.cu -- stage (a): LJ/Morse + point-charge Coulomb force grid.
//
// Replaces evalLJC_QZs_toImg / evalMorseC_QZs_toImg (SPAMMM kernels/AFM.cl:
// 916-1056) behind AFMulator.make_forcefield (spammm/SPM/AFM.py:897-946).
//
// B200 shape.  One thread owns a z-column of GB_ZB (16) nodes at fixed (ia,ib); a
// CTA is 32 (x) x 4 (y) threads, so stores of the (nz,ny,nx,4) grid are
// 512-byte coalesced rows.  Atoms are staged GB_TILE at a time in shared
// memory already transformed for the inner loop, read back as warp-uniform
// broadcasts.  The work per (node, atom) pair is FP32 FMA + MUFU bound, so the
// inner loop is written to minimise issued instructions:
//   * every reference grid has dC = (0,0,dz): dx^2+dy^2+R2SAFE of a pair is
//     computed once per (thread, atom) and shared by the column's nodes;
//   * nodes are evaluated two at a time with Blackwell's packed FP32
//     instructions (fma/mul/add/sub .f32x2), halving the FP32 issue count;
//   * tip-charge sites with a zero z-offset sit on the node itself; their
//     charges are merged into one term that reuses the pair law's 1/r (one
//     MUFU rsqrt per pair in total for LJ + on-node Coulomb); sites with a
//     non-zero offset get their own rsqrt.
// Transcendentals use MUFU approximations (rsqrt.approx, ex2.approx).
//
// That direct sum is for molecules and for Morse.  The nodes of larger LJ systems
// (far_grid: slabs of 256 atoms or more) are built in blocks of 16^3, each atom at a
// block's nodes only when it is near the block; the smooth field of the distant atoms
// is evaluated at 8^3 Chebyshev points of the block and interpolated (build_cell below).
#include "spm_internal.cuh"
#include "spm_batch.cuh"
#include "spm_f32x2.cuh"
#include "spm_far.cuh"

namespace spm {
namespace {

constexpr int GB_TX = 32;     // threads along x
constexpr int GB_TY = 4;      // threads along y
constexpr int GB_ZB = 16;     // nodes along z per thread (8 packed pairs: the per-atom overhead
                              // of the tile loop amortised over 16 nodes; 7% faster than 8 on a
                              // 1200-atom 480x480x240 grid)
constexpr int GB_TILE = 256;  // atoms per shared-memory tile
constexpr float R2SAFE = 1e-4f;
constexpr float COULOMB_CONST = 14.3996448915f;
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float fast_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float fast_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ f2 rsqrt2(f2 x) {
    float a, b;
    upk(x, a, b);
    return pk(fast_rsqrt(a), fast_rsqrt(b));
}
__device__ __forceinline__ f2 ex2_2(f2 x) {
    float a, b;
    upk(x, a, b);
    return pk(fast_ex2(a), fast_ex2(b));
}
struct GridGeom {
    int nx, ny, nz;
    float4 p0, dA, dB, dC;
};

struct TipSites {
    float qs_on;   // sum of Qs[k]*COULOMB_CONST over sites with QZs[k] == 0
    float qs[4];   // Qs[k]*COULOMB_CONST of the non-zero sites with QZs[k] != 0
    float qz[4];   // their z-offsets
};

// Node coordinate along one axis: p0 + dA*ia + dB*ib (+ dC*ic), in this
// fixed operation order in every kernel, so a batched slab node gets the same
// bits as the same node of a full per-molecule grid.
__device__ __forceinline__ float node_xy(float p0, float da, float db, int ia, int ib) {
    return __fmaf_rn(db, (float)ib, __fmaf_rn(da, (float)ia, p0));
}

// The stored box of a build: columns [x_lo, x_lo + nxs), rows [y_lo, y_lo +
// nys) and layers [zst_lo, zst_hi) of the full grid.
struct StoreBox {
    int x_lo, nxs, y_lo, nys, zst_lo, zst_hi;
};

// One atom's pair law and tip-charge terms added to ZP node pairs of a z-column at (px, py): a =
// (x, y, z, Q*qs_on), c = the transformed pair parameters, q[k] = Q*Qs[k]*C of the off-node sites.
template <int KIND, bool ON, int NOFF, int ZP>
__device__ __forceinline__ void add_atom(const float4 a, const float4 c, const float* q, float px, float py,
                                         const f2 (&pz)[ZP], const TipSites& S, f2 (&fx)[ZP], f2 (&fy)[ZP],
                                         f2 (&fz)[ZP], f2 (&fe)[ZP]) {
    const f2 one = bc(1.f);
                    const float dxs = px - a.x;
                    const float dys = py - a.y;
                    const float dxy2s = fmaf(dxs, dxs, fmaf(dys, dys, R2SAFE));
                    const f2 dx = bc(dxs), dy = bc(dys), dxy2 = bc(dxy2s), az = bc(a.z);
                    const f2 c0 = bc(c.x), c1 = bc(c.y), c2 = bc(c.z), c3 = bc(c.w);
                    const f2 qon = bc(a.w);
    #pragma unroll
                    for (int p = 0; p < ZP; p++) {
                        const f2 dz = sub2(pz[p], az);
                        const f2 r2 = fma2(dz, dz, dxy2);
                        const f2 rs = rsqrt2(r2);
                        // s = |F|/r of the pair law plus the on-node charges; the charges' Q/r^3 is
                        // added before the last factor 1/r (Morse) or 1/r^2 (LJ) the two terms share
                        f2 s;
                        if (KIND == SPM_KIND_MORSE) {
                            // E = E0 e (e-2) = E0 (w - e), F = dp * (-2 K E0) w / r, w = e (e-1), e = exp(K (r-R0))
                            const f2 r = mul2(r2, rs);
                            const f2 e = ex2_2(fma2(c0, r, c1));
                            const f2 w = mul2(e, sub2(e, one));
                            fe[p] = fma2(c2, sub2(w, e), fe[p]);
                            const f2 m = mul2(c3, w);
                            if (ON) {
                                const f2 Ek = mul2(qon, rs);
                                fe[p] = add2(fe[p], Ek);
                                s = mul2(fma2(Ek, rs, m), rs);
                            } else {
                                s = mul2(m, rs);
                            }
                        } else {
                            // E = (c12 ir6 - c6) ir6, F = dp * (12 c12 ir6 - 6 c6) ir6 ir2
                            const f2 ir2 = mul2(rs, rs);
                            const f2 ir6 = mul2(mul2(ir2, ir2), ir2);
                            fe[p] = fma2(fma2(c1, ir6, c0), ir6, fe[p]);
                            if (ON) {
                                const f2 Ek = mul2(qon, rs);
                                fe[p] = add2(fe[p], Ek);
                                s = mul2(fma2(fma2(c3, ir6, c2), ir6, Ek), ir2);
                            } else {
                                s = mul2(mul2(fma2(c3, ir6, c2), ir6), ir2);
                            }
                        }
                        fx[p] = fma2(dx, s, fx[p]);
                        fy[p] = fma2(dy, s, fy[p]);
                        fz[p] = fma2(dz, s, fz[p]);
    #pragma unroll
                        for (int k = 0; k < NOFF; k++) {
                            // Coulomb at the tip-charge site node + zhat*QZs[k]
                            const f2 dzk = add2(dz, bc(S.qz[k]));
                            const f2 rsk = rsqrt2(fma2(dzk, dzk, dxy2));
                            const f2 Ek = mul2(bc(q[k]), rsk);
                            fe[p] = add2(fe[p], Ek);
                            const f2 sk = mul2(mul2(Ek, rsk), rsk);
                            fx[p] = fma2(dx, sk, fx[p]);
                            fy[p] = fma2(dy, sk, fy[p]);
                            fz[p] = fma2(dzk, sk, fz[p]);
                        }
                    }
}

// The staged form of an atom (pr: its parameter row).
template <int KIND>
__device__ __forceinline__ float4 atom_params(const float* __restrict__ pr) {
    if (KIND == SPM_KIND_MORSE) {
        const float R0 = __ldg(pr + 0), E0 = __ldg(pr + 1), K = __ldg(pr + 2);
        return make_float4(K * LOG2E, -K * R0 * LOG2E, E0, -2.f * K * E0);
    }
    const float c6 = __ldg(pr + 0), c12 = __ldg(pr + 1);
    return make_float4(-c6, c12, -6.f * c6, 12.f * c12);
}

// The ZP node pairs of column (xl, yl) (box indices) from layer ic0 on, capped, into the box's storage;
// layers above the box are left out, and with BELOW those below it (build_tile starts inside the box: the extra
// test there costs 2.6% of a batch's slabs).
template <int ZP, int LAYOUT, bool BELOW>
__device__ __forceinline__ void store_column(float4* __restrict__ out, const StoreBox& B, int xl, int yl, int ic0,
                                             const f2 (&fx)[ZP], const f2 (&fy)[ZP], const f2 (&fz)[ZP],
                                             const f2 (&fe)[ZP]) {
#pragma unroll
    for (int p = 0; p < ZP; p++) {
        float x[2], y[2], z[2], e[2];
        upk(fx[p], x[0], x[1]);
        upk(fy[p], y[0], y[1]);
        upk(fz[p], z[0], z[1]);
        upk(fe[p], e[0], e[1]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int ic = ic0 + 2 * p + h;
            if (ic >= B.zst_hi) break;
            if (BELOW && ic < B.zst_lo) continue;
            float4 o = make_float4(x[h], y[h], z[h], e[h]);
            // |E| > 100 cap of the reference builders (AFM.cl:1053-1054)
            // (the division only where it can scale: 100/|E| < 1 needs |E| > 100; NaN compares false)
            if (fabsf(o.w) > 100.f) {
                const float renorm = __fdiv_rn(100.f, fabsf(o.w));
                if (renorm < 1.f) { o.x *= renorm; o.y *= renorm; o.z *= renorm; o.w *= renorm; }
            }
            const int zl = ic - B.zst_lo;
            const size_t row = ((size_t)zl * B.nys + yl) * B.nxs;
            const int il = xl > 0 ? xl - 1 : B.nxs - 1;
            if (LAYOUT == 2) {
                out[2 * (row + xl)] = o;
                out[2 * (row + il) + 1] = o;
            } else if (LAYOUT == 4) {
                const int nzs = B.zst_hi - B.zst_lo;
                const size_t rowb = ((size_t)(zl > 0 ? zl - 1 : nzs - 1) * B.nys + yl) * B.nxs;
                out[4 * (row + xl) + 0] = o;
                out[4 * (row + il) + 1] = o;
                out[4 * (rowb + xl) + 2] = o;
                out[4 * (rowb + il) + 3] = o;
            } else {
                out[row + xl] = o;
            }
        }
    }
}

// One CTA tile: a (blockDim.x x blockDim.y) patch of z-columns (full-grid
// column ia, row ib), ZB nodes each starting at global layer ic0; nodes
// outside the box B are not stored, the rest go to out[idx], idx = (zl*nys +
// yl)*nxs + xl with (xl, yl, zl) = (ia - x_lo, ib - y_lo, ic - zst_lo)
// (LAYOUT 1).  LAYOUT 2, x-pairs: out[2*idx + dx] = value(x_lo + (xl + dx) mod
// nxs), so a node's value is also written to its x-1 neighbour's second slot.
// LAYOUT 4, xz-quads: out[4*idx + 2*dz + dx] = value(x_lo + (xl + dx) mod nxs,
// zst_lo + (zl + dz) mod (zst_hi - zst_lo)), written to the four nodes whose
// quads contain it.
// KIND: SPM_KIND_LJ / SPM_KIND_MORSE; ON: an on-node charge term exists;
// NOFF: number of off-node sites.
template <int KIND, bool ON, int NOFF, int ZB, int LAYOUT = 1>
__device__ __forceinline__ void build_tile(int na, const float4* __restrict__ atoms, const float* __restrict__ params,
                                           int pstride, float4* __restrict__ out, const GridGeom& G,
                                           const TipSites& S, const StoreBox& B, int ia, int ib, int ic0) {
    constexpr int ZP = ZB / 2;
    __shared__ float4 s_pos[GB_TILE];                   // (x, y, z, Q*qs_on)
    __shared__ float4 s_prm[GB_TILE];                   // transformed pair parameters
    __shared__ float s_q[NOFF > 0 ? NOFF : 1][GB_TILE];  // Q*Qs[k]*C per off-node site

    const int nthr = blockDim.x * blockDim.y;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int xl = ia - B.x_lo, yl = ib - B.y_lo;
    const bool active = (unsigned)xl < (unsigned)B.nxs && (unsigned)yl < (unsigned)B.nys;

    const float px = node_xy(G.p0.x, G.dA.x, G.dB.x, ia, ib);
    const float py = node_xy(G.p0.y, G.dA.y, G.dB.y, ia, ib);
    const float pzb = node_xy(G.p0.z, G.dA.z, G.dB.z, ia, ib);
    f2 pz[ZP];
#pragma unroll
    for (int p = 0; p < ZP; p++)
        pz[p] = pk(__fmaf_rn(G.dC.z, (float)(ic0 + 2 * p), pzb), __fmaf_rn(G.dC.z, (float)(ic0 + 2 * p + 1), pzb));

    const f2 zero = pk(0.f, 0.f);
    f2 fx[ZP], fy[ZP], fz[ZP], fe[ZP];
#pragma unroll
    for (int p = 0; p < ZP; p++) { fx[p] = zero; fy[p] = zero; fz[p] = zero; fe[p] = zero; }

    for (int t0 = 0; t0 < na; t0 += GB_TILE) {
        const int nt = min(GB_TILE, na - t0);
        for (int j = tid; j < nt; j += nthr) {
            float4 a = __ldg(atoms + t0 + j);
            const float* pr = params + (size_t)(t0 + j) * pstride;
            s_pos[j] = make_float4(a.x, a.y, a.z, a.w * S.qs_on);
            s_prm[j] = atom_params<KIND>(pr);
#pragma unroll
            for (int k = 0; k < NOFF; k++) s_q[k][j] = a.w * S.qs[k];
        }
        __syncthreads();
        if (active) {
#pragma unroll 1
            for (int j = 0; j < nt; j++) {
                float q[NOFF > 0 ? NOFF : 1];
#pragma unroll
                for (int k = 0; k < NOFF; k++) q[k] = s_q[k][j];
                add_atom<KIND, ON, NOFF, ZP>(s_pos[j], s_prm[j], q, px, py, pz, S, fx, fy, fz, fe);
            }
        }
        __syncthreads();
    }
    if (!active) return;
    store_column<ZP, LAYOUT, false>(out, B, xl, yl, ic0, fx, fy, fz, fe);
}

template <int KIND, bool ON, int NOFF>
__global__ void __launch_bounds__(GB_TX * GB_TY)
grid_build_kernel(int na, const float4* __restrict__ atoms, const float* __restrict__ params, int pstride,
                  float4* __restrict__ grid, GridGeom G, TipSites S) {
    const StoreBox B = {0, G.nx, 0, G.ny, 0, G.nz};
    build_tile<KIND, ON, NOFF, GB_ZB>(na, atoms, params, pstride, grid, G, S, B, blockIdx.x * GB_TX + threadIdx.x,
                                      blockIdx.y * GB_TY + threadIdx.y, blockIdx.z * GB_ZB);
}

// ---- blocks with a far field -------------------------------------------------
// The grid's nodes in blocks of FB^3 on the lattice of multiples of FB (so a batch
// slab and the full grid build a node from the same block: the same bits).  An
// atom FAR_RATIO half-edges or more from a block's centre is far: its four
// channels are smooth over the block and are summed at the block's FP^3 Chebyshev
// points (512 instead of 4096 evaluations), then interpolated to the nodes as a
// tensor product along x, y and z; near atoms are summed at the nodes as in
// build_tile, on top of the interpolated values.
//
// Interpolation error of one atom relative to its own force at the node (float64, worst corner and direction,
// at 9 half-edges): 1/r^2 3e-9, r^-7 1e-6, and much less over most of the block, falling as the eighth power of
// the distance -- the direct float32 sum rounds r^-7 by 8e-7 (rsqrt.approx), and the sums are 2-17 times
// shorter.  Measured against 64 bits over 256 to 1200 atoms on ionic slabs, spacings of 0.02 to 0.5 A and three sets of
// tip charges: the error of the forces at the nodes a probe reaches (|E| < 0.5 eV), relative to their norm, is 0.94 of
// the direct sum's (0.82 to 1.01 by spacing and size), over all nodes and relative to the terms' magnitudes 0.91; of
// the energies 0.94 and 0.85 (single systems where few atoms are far up to 1.2: alternating charges cancel less in
// another order).  1200 atoms at 0.1 A: 3.0e-6 -> 2.9e-6 over the
// whole grid.
//
// LJ only.  A Morse exponential varies with |K| times the half-edge, at any distance: at 0.1 A (|K| h = 1.35)
// its interpolation errs by 4e-6 of the local force, at |K| h = 1.5 by 1.7e-5, where the direct sum errs by up
// to 3e-6.  Morse grids are direct sums.
//
// The blocks come in groups of 2^3 whose common far atoms (FAR_RATIO group half-edges
// away) are summed once at the group's Chebyshev points; a block takes that field at
// its own points by interpolation and adds the atoms that are far for it alone.
//
// SPM_FAR_MIN_ATOMS: molecules keep the direct sum's order and bits.  Unpolished FIRE strokes stop where their
// force falls below the threshold, so a grid that differs in its last bits moves their images by 1e-4 (64
// molecules of 10 to 120 atoms), and with few atoms most are near most blocks: 38 atoms on 200^3 nodes take
// 187 us directly and 124 in blocks, 256 1223 against 461, 1200 on 480 x 480 x 240 32.0 ms against 2.37.  Of the
// latter's time the near sums take 0.67 ms, the far points 0.91, the interpolation along y and z 0.18, and
// classification, gathers, the interpolation along x and the stores the rest (each left out in turn).
constexpr int FAR_REF = 3 * 64 + 3 * 8 + 3;  // the point whose value is interpolated as a constant
constexpr int FAR_CHUNK = 256;       // atoms gathered at a time

template <int NOFF>
struct FarShared {
    float4 part[4][FN];  // far sums of the four atom subsets; later the interpolation's stages
    float4 group[FN];    // the group's far field at its points
    float4 pos[FAR_CHUNK], prm[FAR_CHUNK];
    float q[NOFF > 0 ? NOFF : 1][FAR_CHUNK];
    FarTab tab;
    float2 Lz[FB / 2][FP];  // L of node pairs
    int warp[8];
};

// Far of the cube: the pair law and every off-node charge (seen from the node moved by its offset).
// Alone, r^-13 varies too fast for the points at this ratio (9e-5 of the local force): the distance must also be
// at least 1.9 times that of the law's minimum, (2 c12 / c6)^(1/6), which holds by itself from about 0.1 A spacing
// on.  Worst error of the LJ force at both limits 2e-7; without the second one 2e-6 at 0.08 A, 4e-5 at 0.05, 9e-5 at
// 0.02.  Laws of another shape (c6 <= 0 or c12 < 0) and NaN positions or parameters are near.
template <int NOFF>
__device__ __forceinline__ bool is_far(const FarCube& C, const TipSites& S, float4 a, const float* __restrict__ pr) {
    const float dx = C.x - a.x, dy = C.y - a.y, dz = C.z - a.z;
    const float dxy2 = __fmaf_rn(dy, dy, __fmul_rn(dx, dx));
    const float r2 = __fmaf_rn(dz, dz, dxy2);
    const float c12 = __ldg(pr + 1);
    bool far = r2 >= C.lim2 && c12 >= 0.f && 94.f * c12 <= __ldg(pr) * r2 * r2 * r2;
#pragma unroll
    for (int k = 0; k < NOFF; k++) {
        const float dk = __fadd_rn(dz, S.qz[k]);
        far = far && __fmaf_rn(dk, dk, dxy2) >= C.lim2;
    }
    return far;
}

// Stages the atoms of [c0, c0 + FAR_CHUNK) that satisfy pick(atom, parameter row), in atom order; returns
// their number to every thread.
template <int NOFF, class Pick>
__device__ __forceinline__ int gather_atoms(FarShared<NOFF>& M, int tid, int nthr, int c0, int na,
                                            const float4* __restrict__ atoms, const float* __restrict__ params,
                                            int pstride, const TipSites& S, const Pick& pick) {
    const int lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
    const int c1 = min(c0 + FAR_CHUNK, na);
    int n = 0;
    for (int b = c0; b < c1; b += nthr) {
        const int j = b + tid;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        bool take = false;
        if (j < c1) {
            a = __ldg(atoms + j);
            take = pick(a, params + (size_t)j * pstride);
        }
        const unsigned m = __ballot_sync(0xffffffffu, take);
        __syncthreads();  // the previous round's warp counts and the previous chunk's atoms are read
        if (lane == 0) M.warp[warp] = __popc(m);
        __syncthreads();
        int at = n + __popc(m & ((1u << lane) - 1u));
        for (int w = 0; w < nw; w++) {
            const int c = M.warp[w];
            if (w < warp) at += c;
            n += c;
        }
        if (take) {
            M.pos[at] = make_float4(a.x, a.y, a.z, a.w * S.qs_on);
            M.prm[at] = atom_params<SPM_KIND_LJ>(params + (size_t)j * pstride);
#pragma unroll
            for (int k = 0; k < NOFF; k++) M.q[k][at] = a.w * S.qs[k];
        }
    }
    __syncthreads();
    return n;
}

template <class Pick>
__device__ __forceinline__ int count_atoms(int tid, int nthr, int na, const float4* __restrict__ atoms,
                                           const float* __restrict__ params, int pstride, const Pick& pick) {
    int n = 0;
    for (int b = 0; b < na; b += nthr) {
        const int j = b + tid;
        n += __syncthreads_count(j < na && pick(__ldg(atoms + j), params + (size_t)(j < na ? j : 0) * pstride));
    }
    return n;
}

// Sum of the picked atoms at the cube's Chebyshev points -> part[0] (point (kx, ky, kz) at kz*64 + kx*8 +
// ky).  Four runs of consecutive atoms go side by side and are added in a fixed order (consecutive: the
// charges of an ionic crystal listed in lattice order alternate, and every fourth of them would add up to a
// partial sum far above the total).
template <bool ON, int NOFF, class Pick>
__device__ __forceinline__ void far_points(FarShared<NOFF>& M, int tid, int nthr, int na,
                                           const float4* __restrict__ atoms, const float* __restrict__ params,
                                           int pstride, const GridGeom& G, const TipSites& S, const FarCube& C,
                                           const Pick& pick) {
    constexpr int ZP = FP / 2;
    for (int c0 = 0; c0 < na; c0 += FAR_CHUNK) {
        const int n = gather_atoms<NOFF>(M, tid, nthr, c0, na, atoms, params, pstride, S, pick);
        for (int i = tid; i < 4 * FP * FP; i += nthr) {
            const int g = i >> 6, col = i & 63;
            const float ux = C.half * M.tab.c[col >> 3], uy = C.half * M.tab.c[col & 7];
            const float px = __fmaf_rn(G.dB.x, uy, __fmaf_rn(G.dA.x, ux, C.x));
            const float py = __fmaf_rn(G.dB.y, uy, __fmaf_rn(G.dA.y, ux, C.y));
            const float pzb = __fmaf_rn(G.dB.z, uy, __fmaf_rn(G.dA.z, ux, C.z)), hz = __fmul_rn(G.dC.z, C.half);
            const f2 zero = bc(0.f);
            f2 pz[ZP], fx[ZP], fy[ZP], fz[ZP], fe[ZP];
#pragma unroll
            for (int p = 0; p < ZP; p++) {
                pz[p] = pk(__fmaf_rn(hz, M.tab.c[2 * p], pzb), __fmaf_rn(hz, M.tab.c[2 * p + 1], pzb));
                fx[p] = zero; fy[p] = zero; fz[p] = zero; fe[p] = zero;
            }
#pragma unroll 1
            for (int j = g * n / 4; j < (g + 1) * n / 4; j++) {
                float q[NOFF > 0 ? NOFF : 1];
#pragma unroll
                for (int k = 0; k < NOFF; k++) q[k] = M.q[k][j];
                add_atom<SPM_KIND_LJ, ON, NOFF, ZP>(M.pos[j], M.prm[j], q, px, py, pz, S, fx, fy, fz, fe);
            }
#pragma unroll
            for (int p = 0; p < ZP; p++) {
                float x[2], y[2], z[2], e[2];
                upk(fx[p], x[0], x[1]);
                upk(fy[p], y[0], y[1]);
                upk(fz[p], z[0], z[1]);
                upk(fe[p], e[0], e[1]);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float4& o = M.part[g][(2 * p + h) * 64 + col];
                    const float4 v = c0 == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : o;
                    o = make_float4(__fadd_rn(v.x, x[h]), __fadd_rn(v.y, y[h]), __fadd_rn(v.z, z[h]),
                                    __fadd_rn(v.w, e[h]));
                }
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < FN; i += nthr) {
        const float4 a = M.part[0][i], b = M.part[1][i], c = M.part[2][i], d = M.part[3][i];
        M.part[0][i] = make_float4(__fadd_rn(__fadd_rn(a.x, b.x), __fadd_rn(c.x, d.x)),
                                   __fadd_rn(__fadd_rn(a.y, b.y), __fadd_rn(c.y, d.y)),
                                   __fadd_rn(__fadd_rn(a.z, b.z), __fadd_rn(c.z, d.z)),
                                   __fadd_rn(__fadd_rn(a.w, b.w), __fadd_rn(c.w, d.w)));
    }
    __syncthreads();
}

__device__ __forceinline__ float4 fma4(float w, float4 v, float4 s) {
    return make_float4(__fmaf_rn(w, v.x, s.x), __fmaf_rn(w, v.y, s.y), __fmaf_rn(w, v.z, s.z), __fmaf_rn(w, v.w, s.w));
}

// out[i] = sum_k W[index of i along the axis][k] in[i with k there]; stride: of the axis in the point index.
__device__ __forceinline__ float4 far_axis(const float (*W)[FP], const float4* in, int i, int stride) {
    const int a = (i / stride) & (FP - 1), base = i - a * stride;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < FP; k++) s = fma4(W[a][k], in[base + k * stride], s);
    return s;
}

// Blocks [child0, child1) of the 2^3 of one lattice cell (x0, y0, z0: its first node), nodes inside the box B
// stored as build_tile does.  ZB: nodes along z per thread in the near sums, 8 or 16.
template <bool ON, int NOFF, int ZB, int LAYOUT>
__device__ __forceinline__ void build_cell(FarShared<NOFF>& M, int child0, int child1, int na,
                                           const float4* __restrict__ atoms, const float* __restrict__ params,
                                           int pstride, float4* __restrict__ out, const GridGeom& G, const TipSites& S,
                                           const StoreBox& B, int x0, int y0, int z0) {
    constexpr int ZP = ZB / 2;
    const int nthr = blockDim.x * blockDim.y, tid = threadIdx.y * blockDim.x + threadIdx.x;
    const FarCube C2 = far_cube(G, x0, y0, z0, SPM_FAR_CELL);
    auto far2 = [&](float4 a, const float* pr) { return is_far<NOFF>(C2, S, a, pr); };
    const bool use2 = count_atoms(tid, nthr, na, atoms, params, pstride, far2) >= FAR_FEWEST;
    if (use2) {
        far_points<ON, NOFF>(M, tid, nthr, na, atoms, params, pstride, G, S, C2, far2);
        for (int i = tid; i < FN; i += nthr) M.group[i] = M.part[0][i];
    }
    for (int child = child0; child < child1; child++) {
        const int sx = child & 1, sy = (child >> 1) & 1, sz = child >> 2;
        const int bx = x0 + sx * FB, by = y0 + sy * FB, bz = z0 + sz * FB;
        if (bx >= B.x_lo + B.nxs || bx + FB <= B.x_lo || by >= B.y_lo + B.nys || by + FB <= B.y_lo || bz >= B.zst_hi ||
            bz + FB <= B.zst_lo)
            continue;  // CTA-uniform: no node of this block is stored
        const FarCube C1 = far_cube(G, bx, by, bz, FB);
        // an atom of this block alone: not in the group's field
        auto own = [&](float4 a, const float* pr) { return !(use2 && is_far<NOFF>(C2, S, a, pr)); };
        auto far1 = [&](float4 a, const float* pr) { return own(a, pr) && is_far<NOFF>(C1, S, a, pr); };
        const int nfar = count_atoms(tid, nthr, na, atoms, params, pstride, far1);
        const bool use1 = nfar >= FAR_FEWEST, field = use1 || use2;
        auto near1 = [&](float4 a, const float* pr) {
            return own(a, pr) && !(use1 && is_far<NOFF>(C1, S, a, pr));
        };
        float4* stage = M.part[1];  // 1024 float4: parts 1 and 2
        __syncthreads();            // the group's copy, the previous block's stage
        if (use1) far_points<ON, NOFF>(M, tid, nthr, na, atoms, params, pstride, G, S, C1, far1);
        if (use2) {
            for (int i = tid; i < FN; i += nthr) M.part[1][i] = far_axis(M.tab.T[sx], M.group, i, 8);
            __syncthreads();
            for (int i = tid; i < FN; i += nthr) M.part[2][i] = far_axis(M.tab.T[sy], M.part[1], i, 1);
            __syncthreads();
            for (int i = tid; i < FN; i += nthr) {
                const float4 v = far_axis(M.tab.T[sz], M.part[2], i, 64);
                const float4 w = use1 ? M.part[0][i] : make_float4(0.f, 0.f, 0.f, 0.f);
                M.part[0][i] = make_float4(__fadd_rn(v.x, w.x), __fadd_rn(v.y, w.y), __fadd_rn(v.z, w.z),
                                           __fadd_rn(v.w, w.w));
            }
            __syncthreads();
        }
        // the interpolation acts on the differences from one point's value, which is added last: its rounding
        // is relative to the field's variation over the block, not to the field
        float4 ref = make_float4(0.f, 0.f, 0.f, 0.f);
        if (field) {  // along x: points (ky, kz) x 16 nodes
            ref = M.part[0][FAR_REF];
            for (int i = tid; i < FB * FP * FP; i += nthr) {
                const int x = i & (FB - 1), kk = i >> 4, ky = kk & 7, kz = kk >> 3;
                float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int k = 0; k < FP; k++) {
                    const float4 v = M.part[0][kz * 64 + k * 8 + ky];
                    s = fma4(M.tab.L[x][k], make_float4(__fsub_rn(v.x, ref.x), __fsub_rn(v.y, ref.y),
                                                        __fsub_rn(v.z, ref.z), __fsub_rn(v.w, ref.w)), s);
                }
                stage[i] = s;
            }
            __syncthreads();
        }
        for (int item = tid; item < FB * FB * (FB / ZB); item += nthr) {
            const int x = item & (FB - 1), y = (item >> 4) & (FB - 1), ic0 = bz + (item >> 8) * ZB;
            const int ia = bx + x, ib = by + y, xl = ia - B.x_lo, yl = ib - B.y_lo;
            const bool active = (unsigned)xl < (unsigned)B.nxs && (unsigned)yl < (unsigned)B.nys && ic0 < B.zst_hi &&
                                ic0 + ZB > B.zst_lo;
            const f2 zero = bc(0.f);
            f2 pz[ZP], fx[ZP], fy[ZP], fz[ZP], fe[ZP];
#pragma unroll
            for (int p = 0; p < ZP; p++) { fx[p] = zero; fy[p] = zero; fz[p] = zero; fe[p] = zero; }
            const float px = node_xy(G.p0.x, G.dA.x, G.dB.x, ia, ib);
            const float py = node_xy(G.p0.y, G.dA.y, G.dB.y, ia, ib);
            const float pzb = node_xy(G.p0.z, G.dA.z, G.dB.z, ia, ib);
#pragma unroll
            for (int p = 0; p < ZP; p++)
                pz[p] = pk(__fmaf_rn(G.dC.z, (float)(ic0 + 2 * p), pzb), __fmaf_rn(G.dC.z, (float)(ic0 + 2 * p + 1), pzb));
            if (field && active) {  // along y, then z
#pragma unroll 1
                for (int kz = 0; kz < FP; kz++) {
                    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int k = 0; k < FP; k++) s = fma4(M.tab.L[y][k], stage[(kz * 8 + k) * FB + x], s);
                    const f2 vx = bc(s.x), vy = bc(s.y), vz = bc(s.z), ve = bc(s.w);
#pragma unroll
                    for (int p = 0; p < ZP; p++) {
                        const float2 l = M.Lz[(item >> 8) * ZP + p][kz];
                        const f2 w = pk(l.x, l.y);
                        fx[p] = fma2(w, vx, fx[p]);
                        fy[p] = fma2(w, vy, fy[p]);
                        fz[p] = fma2(w, vz, fz[p]);
                        fe[p] = fma2(w, ve, fe[p]);
                    }
                }
                const f2 rx = bc(ref.x), ry = bc(ref.y), rz = bc(ref.z), re = bc(ref.w);
#pragma unroll
                for (int p = 0; p < ZP; p++) {
                    fx[p] = add2(fx[p], rx);
                    fy[p] = add2(fy[p], ry);
                    fz[p] = add2(fz[p], rz);
                    fe[p] = add2(fe[p], re);
                }
            }
            for (int c0 = 0; c0 < na; c0 += FAR_CHUNK) {
                const int nnear = gather_atoms<NOFF>(M, tid, nthr, c0, na, atoms, params, pstride, S, near1);
                if (active) {
#pragma unroll 1
                    for (int j = 0; j < nnear; j++) {
                        float q[NOFF > 0 ? NOFF : 1];
#pragma unroll
                        for (int k = 0; k < NOFF; k++) q[k] = M.q[k][j];
                        add_atom<SPM_KIND_LJ, ON, NOFF, ZP>(M.pos[j], M.prm[j], q, px, py, pz, S, fx, fy, fz, fe);
                    }
                }
            }
            if (active) store_column<ZP, LAYOUT, true>(out, B, xl, yl, ic0, fx, fy, fz, fe);
        }
    }
}

template <int NOFF>
__device__ __forceinline__ void load_far_tab(FarShared<NOFF>& M, const FarTab& tab) {
    const int nthr = blockDim.x * blockDim.y, tid = threadIdx.y * blockDim.x + threadIdx.x;
    const float* src = reinterpret_cast<const float*>(&tab);
    float* dst = reinterpret_cast<float*>(&M.tab);
    for (int i = tid; i < (int)(sizeof(FarTab) / sizeof(float)); i += nthr) dst[i] = src[i];
    for (int i = tid; i < FB / 2 * FP; i += nthr)
        M.Lz[i / FP][i % FP] = make_float2(tab.L[2 * (i / FP)][i % FP], tab.L[2 * (i / FP) + 1][i % FP]);
    __syncthreads();
}

// 256 threads, 16 nodes along z each, at 128 registers (two CTAs per SM, 60 to 150 bytes spilled): measured in turn on
// the 1200-atom 480 x 480 x 240 grid 2.24 ms, 128 threads 2.25, 8 nodes each (no spills) 2.36; on 527 atoms, 243 x
// 138 x 98, 0.47, 0.71 and 0.44.
constexpr int FAR_THREADS = 256;

// A whole grid: one CTA per lattice cell, or per 4, 2 or 1 blocks of a group while the groups alone would
// leave SMs idle (each CTA then sums the group's field itself: the same values).
template <bool ON, int NOFF>
__global__ void __launch_bounds__(FAR_THREADS, 2)
grid_block_kernel(int split, int na, const float4* __restrict__ atoms, const float* __restrict__ params, int pstride,
                  float4* __restrict__ grid, GridGeom G, TipSites S, const __grid_constant__ FarTab tab) {
    extern __shared__ __align__(16) unsigned char far_smem[];
    FarShared<NOFF>& M = *reinterpret_cast<FarShared<NOFF>*>(far_smem);
    load_far_tab(M, tab);
    const StoreBox B = {0, G.nx, 0, G.ny, 0, G.nz};
    const int e = SPM_FAR_CELL, nb = 8 / split, part = blockIdx.x % split;
    build_cell<ON, NOFF, GB_ZB, 1>(M, part * nb, (part + 1) * nb, na, atoms, params, pstride, grid, G, S, B,
                                         blockIdx.x / split * e, blockIdx.y * e, blockIdx.z * e);
}

template <bool ON, int NOFF>
int launch_blocks(int na, const float4* atoms, const float* params, int pstride, float4* out, const GridGeom& G,
                  const TipSites& S, cudaStream_t st) {
    static const FarTab tab = make_far_tab();
    const auto kern = grid_block_kernel<ON, NOFF>;
    const size_t smem = sizeof(FarShared<NOFF>);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return set_error(SPM_ERR_CUDA, "spm_grid_build: cannot enable %zu B of shared memory", smem);
    const int e = SPM_FAR_CELL;
    const long long cells = (long long)((G.nx + e - 1) / e) * ((G.ny + e - 1) / e) * ((G.nz + e - 1) / e);
    int dev = 0, sms = 0, split = 1;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return set_error(SPM_ERR_CUDA, "spm_grid_build: cannot query the device");
    while (split < 8 && cells * split < 3LL * sms / 2) split *= 2;
    kern<<<dim3((G.nx + e - 1) / e * split, (G.ny + e - 1) / e, (G.nz + e - 1) / e), FAR_THREADS, smem, st>>>(
        split, na, atoms, params, pstride, out, G, S, tab);
    return check_launch("spm_grid_build");
}

template <int KIND, bool ON>
int launch_noff(int noff, dim3 grd, dim3 block, cudaStream_t st, int na, const float4* atoms, const float* params,
                int pstride, float4* out, const GridGeom& G, const TipSites& S) {
    if (KIND == SPM_KIND_LJ && far_grid(na, G.nx, G.ny, &G.dA.x, &G.dB.x, &G.dC.x)) {
        switch (noff) {
            case 0: return launch_blocks<ON, 0>(na, atoms, params, pstride, out, G, S, st);
            case 1: return launch_blocks<ON, 1>(na, atoms, params, pstride, out, G, S, st);
            case 2: return launch_blocks<ON, 2>(na, atoms, params, pstride, out, G, S, st);
            case 3: return launch_blocks<ON, 3>(na, atoms, params, pstride, out, G, S, st);
            default: return launch_blocks<ON, 4>(na, atoms, params, pstride, out, G, S, st);
        }
    }
    switch (noff) {
        case 0: grid_build_kernel<KIND, ON, 0><<<grd, block, 0, st>>>(na, atoms, params, pstride, out, G, S); break;
        case 1: grid_build_kernel<KIND, ON, 1><<<grd, block, 0, st>>>(na, atoms, params, pstride, out, G, S); break;
        case 2: grid_build_kernel<KIND, ON, 2><<<grd, block, 0, st>>>(na, atoms, params, pstride, out, G, S); break;
        case 3: grid_build_kernel<KIND, ON, 3><<<grd, block, 0, st>>>(na, atoms, params, pstride, out, G, S); break;
        default: grid_build_kernel<KIND, ON, 4><<<grd, block, 0, st>>>(na, atoms, params, pstride, out, G, S); break;
    }
    return check_launch("spm_grid_build");
}

template <int KIND>
int launch_kind(bool on, int noff, dim3 grd, dim3 block, cudaStream_t st, int na, const float4* atoms,
                const float* params, int pstride, float4* out, const GridGeom& G, const TipSites& S) {
    if (on) return launch_noff<KIND, true>(noff, grd, block, st, na, atoms, params, pstride, out, G, S);
    return launch_noff<KIND, false>(noff, grd, block, st, na, atoms, params, pstride, out, G, S);
}

// Tip-charge sites: zero-offset charges merged into the on-node term.
TipSites make_sites(const float* Qs, const float* QZs, bool& on, int& noff) {
    TipSites S = {};
    noff = 0;
    on = false;
    for (int k = 0; k < 4; k++) {
        if (Qs[k] == 0.f) continue;  // a zero-charge site only adds zeros
        if (QZs[k] == 0.f) {
            S.qs_on += Qs[k] * COULOMB_CONST;
            on = true;
        } else {
            S.qs[noff] = Qs[k] * COULOMB_CONST;
            S.qz[noff] = QZs[k];
            noff++;
        }
    }
    return S;
}

// ---- batched slabs ----------------------------------------------------------
// One CTA per tile of the batch: 32*TY consecutive (x fastest) of the slab's
// nx_slab*ny_slab columns, ZB layers; tiles of a molecule are numbered columns
// first, then z, over ceil(nx_slab*ny_slab / (32*TY)) x ceil(nz_slab/ZB).
// (Column tiles need not fit the slab's rows: a 32 x TY box of rows would
// leave a quarter of the node-atom pairs idle on the batch distribution.)
template <int KIND, bool ON, int NOFF, int ZB, int LAYOUT>
__global__ void __launch_bounds__(256)
batch_grid_build_kernel(int n_mol, const spm_batch_mol* __restrict__ mols, const float4* __restrict__ atoms,
                        const float* __restrict__ params, int pstride, float4* __restrict__ grid, TipSites S) {
    const long long tile = blockIdx.x;
    const spm_batch_mol* D = mols + SPM_MOL_BY(tile_off, mols, n_mol, tile);
    if (KIND == SPM_KIND_LJ && far_grid(*D)) return;  // built by batch_grid_block_kernel
    const int ty = blockDim.y;
    const int z_lo = D->z_lo, nzs = D->nz_slab;
    const StoreBox B = {D->x_lo, D->nx_slab, D->y_lo, D->ny_slab, z_lo, z_lo + nzs};
    const long long lt = tile - D->tile_off;
    const long long ncol = (long long)B.nxs * B.nys;
    const int cpt = GB_TX * ty;  // columns per tile
    const long long ntc = (ncol + cpt - 1) / cpt;
    const long long bc = lt % ntc, bz = lt / ntc;
    if (bz * ZB >= nzs) return;  // whole CTA: outside the slab (prefix of another shape)
    const long long col = bc * cpt + threadIdx.y * GB_TX + threadIdx.x;
    // a column past the slab's last gets a row outside the box: computed by nobody, stored nowhere
    const int yl = col < ncol ? (int)(col / B.nxs) : B.nys, xl = col < ncol ? (int)(col - (long long)yl * B.nxs) : 0;
    GridGeom G;
    G.nx = D->nx; G.ny = D->ny; G.nz = D->nz;
    G.p0 = ld4f(D->p0);
    G.dA = ld4f(D->dA);
    G.dB = ld4f(D->dB);
    G.dC = ld4f(D->dC);
    const int ao = D->atom_off;
    build_tile<KIND, ON, NOFF, ZB, LAYOUT>(D->n_atoms, atoms + ao, params + (size_t)ao * pstride, pstride,
                                           grid + LAYOUT * D->grid_off, G, S, B, B.x_lo + xl, B.y_lo + yl,
                                           z_lo + (int)bz * ZB);
}

// The LJ molecules that take blocks (far_grid): persistent CTAs over their lattice cells (block_off:
// prefix of cells over the batch), each cell's nodes inside the molecule's box as grid_block_kernel builds
// them.
constexpr int BATCH_FAR_THREADS = 128;  // 16 molecules of 300 to 600 atoms: 7.2 ms, 256 threads 7.4, 64 12.0

template <bool ON, int NOFF, int LAYOUT>
__global__ void __launch_bounds__(BATCH_FAR_THREADS, 4)
batch_grid_block_kernel(int n_mol, const spm_batch_mol* __restrict__ mols, const float4* __restrict__ atoms,
                        const float* __restrict__ params, int pstride, float4* __restrict__ grid, TipSites S,
                        const __grid_constant__ FarTab tab) {
    extern __shared__ __align__(16) unsigned char far_smem[];
    FarShared<NOFF>& M = *reinterpret_cast<FarShared<NOFF>*>(far_smem);
    const long long total = (long long)mols[n_mol - 1].block_off + far_cells(mols[n_mol - 1]);
    if (blockIdx.x >= total) return;  // a batch of molecules only: 5 us for the launch
    load_far_tab(M, tab);
    for (long long c = blockIdx.x; c < total; c += gridDim.x) {
        const spm_batch_mol* D = mols + SPM_MOL_BY(block_off, mols, n_mol, c);
        const int e = SPM_FAR_CELL;
        const StoreBox B = {D->x_lo, D->nx_slab, D->y_lo, D->ny_slab, D->z_lo, D->z_lo + D->nz_slab};
        const int cx0 = B.x_lo / e, cy0 = B.y_lo / e, cz0 = B.zst_lo / e;
        const int ncx = (B.x_lo + B.nxs - 1) / e - cx0 + 1, ncy = (B.y_lo + B.nys - 1) / e - cy0 + 1;
        const int lc = (int)(c - D->block_off);
        GridGeom G;
        G.nx = D->nx; G.ny = D->ny; G.nz = D->nz;
        G.p0 = ld4f(D->p0);
        G.dA = ld4f(D->dA);
        G.dB = ld4f(D->dB);
        G.dC = ld4f(D->dC);
        const int ao = D->atom_off;
        build_cell<ON, NOFF, 8, LAYOUT>(M, 0, 8, D->n_atoms, atoms + ao, params + (size_t)ao * pstride, pstride,
                                              grid + LAYOUT * D->grid_off, G, S, B, (cx0 + lc % ncx) * e,
                                              (cy0 + lc / ncx % ncy) * e, (cz0 + lc / ncx / ncy) * e);
        __syncthreads();  // the next cell reuses the shared memory
    }
}

struct BatchLaunch {
    unsigned blocks;
    dim3 block;
    cudaStream_t st;
    int n_mol;
    const spm_batch_mol* mols;
    const float4* atoms;
    const float* params;
    int pstride;
    float4* grid;
    int layout;  // float4 per node: 2 (x-pairs) or 4 (xz-quads)
};

template <int KIND, bool ON, int NOFF, int ZB, int LAYOUT>
int launch_batch_z(const BatchLaunch& L, const TipSites& S) {
    batch_grid_build_kernel<KIND, ON, NOFF, ZB, LAYOUT><<<L.blocks, L.block, 0, L.st>>>(
        L.n_mol, L.mols, L.atoms, L.params, L.pstride, L.grid, S);
    if (KIND != SPM_KIND_LJ) return check_launch("spm_batch_grid_build");
    static const FarTab tab = make_far_tab();
    const auto kern = batch_grid_block_kernel<ON, NOFF, LAYOUT>;
    const size_t smem = sizeof(FarShared<NOFF>);
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BATCH_FAR_THREADS, smem) != cudaSuccess)
        return set_error(SPM_ERR_CUDA, "spm_batch_grid_build: cannot prepare the block kernel");
    kern<<<sms * (per_sm > 0 ? per_sm : 1), BATCH_FAR_THREADS, smem, L.st>>>(L.n_mol, L.mols, L.atoms, L.params,
                                                                             L.pstride, L.grid, S, tab);
    return check_launch("spm_batch_grid_build");
}

template <int KIND, bool ON, int NOFF>
int launch_batch_zb(int zb, const BatchLaunch& L, const TipSites& S) {
    if (L.layout == 4)
        return zb == 16 ? launch_batch_z<KIND, ON, NOFF, 16, 4>(L, S) : launch_batch_z<KIND, ON, NOFF, 8, 4>(L, S);
    return zb == 16 ? launch_batch_z<KIND, ON, NOFF, 16, 2>(L, S) : launch_batch_z<KIND, ON, NOFF, 8, 2>(L, S);
}

template <int KIND, bool ON>
int launch_batch_noff(int noff, int zb, const BatchLaunch& L, const TipSites& S) {
    switch (noff) {
        case 0: return launch_batch_zb<KIND, ON, 0>(zb, L, S);
        case 1: return launch_batch_zb<KIND, ON, 1>(zb, L, S);
        case 2: return launch_batch_zb<KIND, ON, 2>(zb, L, S);
        case 3: return launch_batch_zb<KIND, ON, 3>(zb, L, S);
        default: return launch_batch_zb<KIND, ON, 4>(zb, L, S);
    }
}

template <int KIND>
int launch_batch_kind(bool on, int noff, int zb, const BatchLaunch& L, const TipSites& S) {
    return on ? launch_batch_noff<KIND, true>(noff, zb, L, S) : launch_batch_noff<KIND, false>(noff, zb, L, S);
}

}  // namespace
}  // namespace spm

extern "C" int spm_batch_grid_build(int kind, int n_mol, const spm_batch_mol* mols, long long n_tiles,
                                    const spm_batch_shape* shape, const float* atoms, const float* params,
                                    const float* Qs, const float* QZs, float* grid, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(kind == SPM_KIND_LJ || kind == SPM_KIND_MORSE, "spm_batch_grid_build: kind=%d", kind);
    SPM_REQUIRE(shape && Qs && QZs, "spm_batch_grid_build: null shape or host vector");
    SPM_REQUIRE(n_mol >= 0 && n_tiles >= 0, "spm_batch_grid_build: negative sizes");
    if (n_mol == 0 || n_tiles == 0) return SPM_OK;
    SPM_REQUIRE(mols && grid && atoms && params, "spm_batch_grid_build: null device pointer");
    SPM_REQUIRE(aligned16(grid) && aligned16(atoms) && (reinterpret_cast<uintptr_t>(mols) & 7u) == 0,
                "spm_batch_grid_build: misaligned buffers");
    SPM_REQUIRE(shape->gb_ty == 2 || shape->gb_ty == 4 || shape->gb_ty == 8, "spm_batch_grid_build: gb_ty=%d",
                shape->gb_ty);
    SPM_REQUIRE(shape->gb_zb == 8 || shape->gb_zb == 16, "spm_batch_grid_build: gb_zb=%d", shape->gb_zb);
    SPM_REQUIRE(shape->grid_layout == 0 || shape->grid_layout == 1, "spm_batch_grid_build: grid_layout=%d",
                shape->grid_layout);
    SPM_REQUIRE(n_tiles <= 0x7fffffffLL, "spm_batch_grid_build: %lld tiles exceed one launch", n_tiles);
    int noff = 0;
    bool on = false;
    const TipSites S = make_sites(Qs, QZs, on, noff);
    BatchLaunch L;
    L.blocks = (unsigned)n_tiles;
    L.block = dim3(GB_TX, shape->gb_ty, 1);
    L.st = as_stream(stream);
    L.n_mol = n_mol;
    L.mols = mols;
    L.atoms = reinterpret_cast<const float4*>(atoms);
    L.params = params;
    L.pstride = (kind == SPM_KIND_MORSE) ? 4 : 2;
    L.grid = reinterpret_cast<float4*>(grid);
    L.layout = shape->grid_layout ? 4 : 2;
    if (kind == SPM_KIND_MORSE) return launch_batch_kind<SPM_KIND_MORSE>(on, noff, shape->gb_zb, L, S);
    return launch_batch_kind<SPM_KIND_LJ>(on, noff, shape->gb_zb, L, S);
}

extern "C" int spm_grid_build(int kind, int n_atoms, const float* atoms, const float* params, float* grid,
                              int nx, int ny, int nz, const float* p0, const float* dA, const float* dB,
                              const float* dC, const float* Qs, const float* QZs, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(kind == SPM_KIND_LJ || kind == SPM_KIND_MORSE, "spm_grid_build: kind=%d is not LJ(0)/Morse(1)", kind);
    SPM_REQUIRE(n_atoms >= 0, "spm_grid_build: n_atoms=%d < 0", n_atoms);
    SPM_REQUIRE(nx > 0 && ny > 0 && nz > 0, "spm_grid_build: grid dims (%d,%d,%d) must be positive", nx, ny, nz);
    SPM_REQUIRE(grid && p0 && dA && dB && dC && Qs && QZs, "spm_grid_build: null grid or host vector");
    SPM_REQUIRE(n_atoms == 0 || (atoms && params), "spm_grid_build: null atoms/params with n_atoms=%d", n_atoms);
    SPM_REQUIRE(aligned16(grid) && (n_atoms == 0 || aligned16(atoms)), "spm_grid_build: grid/atoms not 16-byte aligned");
    long long nab = 0, total = 0;
    SPM_REQUIRE(mul_ok(nx, ny, &nab) && mul_ok(nab, nz, &total), "spm_grid_build: node count overflows");
    if (dC[0] != 0.f || dC[1] != 0.f)
        return set_error(SPM_ERR_UNSUPPORTED, "spm_grid_build: dC=(%g,%g,%g) must be (0,0,dz)", dC[0], dC[1], dC[2]);
    if ((long long)ny > 65535LL * GB_TY || ((long long)nz + GB_ZB - 1) / GB_ZB > 65535LL)
        return set_error(SPM_ERR_UNSUPPORTED, "spm_grid_build: ny=%d or nz=%d exceeds the launch limits", ny, nz);
    GridGeom G;
    G.nx = nx; G.ny = ny; G.nz = nz;
    G.p0 = make_float4(p0[0], p0[1], p0[2], p0[3]);
    G.dA = make_float4(dA[0], dA[1], dA[2], dA[3]);
    G.dB = make_float4(dB[0], dB[1], dB[2], dB[3]);
    G.dC = make_float4(dC[0], dC[1], dC[2], dC[3]);
    int noff = 0;
    bool on = false;
    const TipSites S = make_sites(Qs, QZs, on, noff);
    dim3 block(GB_TX, GB_TY, 1);
    dim3 grd((nx + GB_TX - 1) / GB_TX, (ny + GB_TY - 1) / GB_TY, (nz + GB_ZB - 1) / GB_ZB);
    const int pstride = (kind == SPM_KIND_MORSE) ? 4 : 2;
    cudaStream_t st = as_stream(stream);
    const float4* a4 = reinterpret_cast<const float4*>(atoms);
    float4* g4 = reinterpret_cast<float4*>(grid);
    if (kind == SPM_KIND_MORSE) return launch_kind<SPM_KIND_MORSE>(on, noff, grd, block, st, n_atoms, a4, params, pstride, g4, G, S);
    return launch_kind<SPM_KIND_LJ>(on, noff, grd, block, st, n_atoms, a4, params, pstride, g4, G, S);
}

// ---- the uncapped pair sums at arbitrary points ----------------------------
// Replaces cs_brute_afm_morse_c_points (kernels/contact_surface.cl:1341-1390,
// called by AFMulator._brute_afm_morse_c_queries, spammm/SPM/AFM.py:1051-1067):
// per query point the LJ or Morse law plus the Coulomb law at the four
// tip-charge sites (point + zhat*QZs[k], weighted by Qs[k]*COULOMB_CONST) summed
// over all atoms, with no |E| > 100 cap.  One thread per point, atoms staged in
// shared memory; FP32 with IEEE division, sqrt and exp.
namespace spm {
namespace {
constexpr int PQ_THREADS = 128;

template <int KIND>
__global__ void __launch_bounds__(PQ_THREADS)
pair_points_kernel(int na, const float4* __restrict__ atoms, const float* __restrict__ params, int pstride,
                   const float* __restrict__ q, int nq, float4 qs, float4 qz, float4* __restrict__ out) {
    __shared__ float4 s_a[PQ_THREADS];
    __shared__ float4 s_p[PQ_THREADS];
    const int iq = blockIdx.x * PQ_THREADS + threadIdx.x;
    const bool act = iq < nq;
    const float px = act ? q[3 * (size_t)iq] : 0.f, py = act ? q[3 * (size_t)iq + 1] : 0.f,
                pz = act ? q[3 * (size_t)iq + 2] : 0.f;
    const float sq[4] = {qs.x, qs.y, qs.z, qs.w}, sz[4] = {qz.x, qz.y, qz.z, qz.w};
    float fx = 0.f, fy = 0.f, fz = 0.f, fe = 0.f;
    for (int t0 = 0; t0 < na; t0 += PQ_THREADS) {
        const int j = t0 + threadIdx.x;
        if (j < na) {
            s_a[threadIdx.x] = __ldg(atoms + j);
            const float* pr = params + (size_t)j * pstride;
            s_p[threadIdx.x] = make_float4(__ldg(pr), __ldg(pr + 1), KIND == SPM_KIND_MORSE ? __ldg(pr + 2) : 0.f, 0.f);
        }
        __syncthreads();
        const int nt = min(PQ_THREADS, na - t0);
        for (int jj = 0; jj < nt; jj++) {
            const float4 a = s_a[jj];
            const float4 c = s_p[jj];
            const float dx = px - a.x, dy = py - a.y, dz = pz - a.z;
            const float r2 = dx * dx + dy * dy + dz * dz + R2SAFE;
            float s;
            if (KIND == SPM_KIND_MORSE) {  // getMorse: E0 e (e - 2), F = dp * (-2 K E0 e (e-1)) / r
                const float r = sqrtf(r2);
                const float e = expf(c.z * (r - c.x));
                fe += c.y * e * (e - 2.f);
                s = __fdiv_rn(-c.y * e * (e - 1.f) * 2.f * c.z, r);
            } else {  // getLJ: (c12 ir6 - c6) ir6, F = dp * (12 c12 ir6 - 6 c6) ir6 ir2
                const float ir2 = __fdiv_rn(1.f, r2);
                const float ir6 = ir2 * ir2 * ir2;
                fe += (c.y * ir6 - c.x) * ir6;
                s = (12.f * c.y * ir6 - 6.f * c.x) * ir6 * ir2;
            }
            fx += dx * s;
            fy += dy * s;
            fz += dz * s;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (sq[k] == 0.f) continue;
                const float dzk = dz + sz[k];
                const float ir2 = __fdiv_rn(1.f, dx * dx + dy * dy + dzk * dzk + R2SAFE);
                const float E = a.w * sqrtf(ir2) * sq[k];
                fe += E;
                const float sk = E * ir2;
                fx += dx * sk;
                fy += dy * sk;
                fz += dzk * sk;
            }
        }
        __syncthreads();
    }
    if (act) out[iq] = make_float4(fx, fy, fz, fe);
}
}  // namespace
}  // namespace spm

extern "C" int spm_pair_fe_points(int kind, int n_atoms, const float* atoms, const float* params, const float* queries,
                                  int n_q, const float* Qs, const float* QZs, float* out, void* stream) {
    using namespace spm;
    clear_error();
    SPM_REQUIRE(kind == SPM_KIND_LJ || kind == SPM_KIND_MORSE, "spm_pair_fe_points: kind=%d", kind);
    SPM_REQUIRE(n_atoms >= 0 && n_q >= 0, "spm_pair_fe_points: negative sizes");
    SPM_REQUIRE(Qs && QZs, "spm_pair_fe_points: null host vectors");
    if (n_q == 0) return SPM_OK;
    SPM_REQUIRE(queries && out && (n_atoms == 0 || (atoms && params)), "spm_pair_fe_points: null device pointer");
    SPM_REQUIRE(aligned16(out) && (n_atoms == 0 || aligned16(atoms)), "spm_pair_fe_points: out/atoms not aligned");
    const float4 qs = make_float4(Qs[0] * COULOMB_CONST, Qs[1] * COULOMB_CONST, Qs[2] * COULOMB_CONST,
                                  Qs[3] * COULOMB_CONST);
    const float4 qz = make_float4(QZs[0], QZs[1], QZs[2], QZs[3]);
    const unsigned nb = (unsigned)((n_q + PQ_THREADS - 1) / PQ_THREADS);
    cudaStream_t st = as_stream(stream);
    const float4* a4 = reinterpret_cast<const float4*>(atoms);
    float4* o4 = reinterpret_cast<float4*>(out);
    if (kind == SPM_KIND_MORSE)
        pair_points_kernel<SPM_KIND_MORSE><<<nb, PQ_THREADS, 0, st>>>(n_atoms, a4, params, 4, queries, n_q, qs, qz, o4);
    else
        pair_points_kernel<SPM_KIND_LJ><<<nb, PQ_THREADS, 0, st>>>(n_atoms, a4, params, 2, queries, n_q, qs, qz, o4);
    return check_launch("spm_pair_fe_points");
}
