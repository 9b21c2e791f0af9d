// Brick-staged pair passes (sm_103a): the uniform-h summation density
// (+ Tait) and the PGrad + Monaghan AV (+ XSPH) rates of one simulation.
//
// Replaces, for the configurations it covers, the same reference routines
// as the list-streaming kernels of pairs.cu: SPHCalc.sph -> SPHFunction.eval
// -> eval_nbr over density_funcs.pyx:38-74 (SPHRho), eos_funcs.pyx:105-116
// (TaitEquation), pressure_funcs.pyx:40-91 (SPHPressureGradient),
// viscosity_funcs.pyx:41-124 (MonaghanArtificialVsicosity) and
// xsph_funcs.pyx:31-88 (XSPHCorrection), and the neighbour cache of
// base/nnps.pyx:566-620.
//
// One block owns one brick of bx * by * bz grid cells.  It copies the
// records of every source particle within the stencil half-width K of the
// brick -- the particles of the brick's rows of cells grown by K cells on
// every side -- once into shared memory, with positions relative to the
// brick's centre cell (FP32, |x| < ~12 cells, so |r_ab| keeps ~2e-7 of
// relative accuracy).  A destination's neighbour list then holds 16-bit
// indices into that staging, fixed between full builds (the sorted order and
// the cell table do not change), so a pair costs one list entry, shared-
// memory records and the pair arithmetic: no cell-offset decoding and no
// global gathers.  The entries of a destination are grouped by eight (one
// 16-byte load), groups of consecutive destinations adjacent, and the last
// group is padded with the index of a zero-mass record placed far away
// (index T, just past the staged records): the pair loop needs no bounds
// predicates.
//
// The tables of a block -- the slots and cells of its sources and of its
// destinations -- are written once per full build (k_brick_count,
// k_brick_fill), so a pass reads where its records are instead of deriving
// it: the passes are bound by instruction issue, and finding the records from
// the cell table in every block (a scan, a binary search and two divisions
// per record) was nearly half of their instructions.  At 1 M particles (3D
// lattice, 61 neighbours) density 151 -> 115 us, rates 255 -> 213 us.
//
// Small simulations do not fill the GPU with a thread per destination: there
// S = 2 or 4 neighbouring threads (lanes) share a destination, lane s takes
// the list's groups s, s + S, ..., and the groups' sums are folded in the
// list's order (shuffles), so the result is the same bit for bit; the bricks
// are divided into parts (blocks of their own, with the brick's origin).  (Whether a
// block reads two records per pair or three is its own matter: a part may hold
// one source mass where its brick holds two, or fit the shared memory where its
// brick does not.  The last bit of the viscosity's sound speed then differs.)
//
// The neighbour relation is the reference's: strict r^2 < (radius_scale
// h)^2, decided in FP32 outside a +-1e-5 relative band around the threshold
// and by the FP64 test of base/nnps.pyx:337-353 inside it.  Neighbours are
// visited in the order of the list-streaming kernels (stencil rows in (dz,
// dy) order, ascending sorted slot within a row), and every destination's
// sums are Neumaier-compensated FP32 over plain batch partials.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <utility>
#include <vector>

#include "sph_internal.cuh"

namespace sphgb {

namespace {

// destination threads per block are chosen per build (the largest brick
// population rounded to warps); the kernels are compiled for at most this
constexpr int kBrickMaxThreads = 512;

// an array as the sources of a pass
struct BrickSrcDev {
    const float4 *pm, *velh, *st;
    const float *scx;
    const int *cstart, *perm;
    const int4 *bsrc;
    const int2 *brow, *bstage;
    const double *x, *y, *z;
};

// an array as the destinations of a pass
struct BrickDstDev {
    const float4 *pm, *velh, *st;
    const int *perm;
    const int2 *bdst, *bdest;
    const int64_t *tag;
    const double *x, *y, *z, *u, *v, *w, *p, *cs;
};

// shared-memory layout of a block (byte offsets into the dynamic array)
// position records behind the padding record that a traversal may read (it
// takes eight at a time)
constexpr int kSlack = 6;

struct BrickSmem {
    int off_v, off_s;   // rates: velocity / state records
    int off_scell;      // list build: cell table
};

// The neighbour radius of a uniform h, computed on the host with the
// operations of the per-destination test: radius2 = (h rs)^2 in FP64, its
// FP32 band [r2lo, r2hi] and the list radius r2list (0 without a skin).
struct BrickRadius {
    double radius2;
    float r2lo, r2hi, r2list;
};

struct BrickDensityArgs {
    Grid g;
    BrickGeom bk;
    BrickDstDev d;
    BrickSrcDev s;
    BrickSmem sm;
    BrickRadius rad;
    uint16_t *nbr;      // list: 8-entry group g of destination d of brick b is
                        // the uint4 (bdst[b] * cap / 8 + g * D_b + d)
    int *cnt;           // neighbour count per destination, brick order
    int *maxcnt;
    int cap;
    int write_out;      // 0: list build only
    int dim, tait;
    float co, ro, gamma;
    double *rho_out, *p_out, *cs_out;
    float4 *st_out;
    const unsigned *gate;
};

struct BrickRatesArgs {
    Grid g;
    BrickGeom bk;
    BrickDstDev d;
    BrickSrcDev s;
    BrickSmem sm;
    BrickRadius rad;
    const uint16_t *nbr;
    const int *cnt;
    const int *maxcnt;
    int cap;
    int dim;
    float alpha, beta, eta2, eps;
    int add_velocity, add_gravity, accumulate;
    // the sources' cs follows Tait with gamma = 7 from their rho (alpha cs /
    // 2 = tait_kc (rho / 2)^3): blocks whose sources share one mass then
    // read two records per pair instead of three
    int tait_state;
    float tait_kc;
    double gx, gy, gz;
    double *acc[3];
    double *pos[3];
    const unsigned *gate;
};

// The block's cells: its part [x0, x1) x [y0, y1) x [z0, z1) of a brick, the
// staged region [xs0, xs1) x ... (the part grown by the stencil half-widths,
// clipped to the grid) and the origin cell of the staged positions (the
// centre of the whole brick).
struct BlockGeo {
    int x0, x1, y0, y1, z0, z1;
    int xs0, ys0, zs0, xs1, ys1, zs1;
    int lx, ry, nr;
    int cxc, cyc, czc;
};

// part i of the bricks of e cells (each in p parts) along an axis of n cells
__device__ __forceinline__ void axis_part(int n, int e, int p, int i, int k, int &lo, int &hi,
                                          int &slo, int &shi, int &centre) {
    const int brick = i / p, part = i - brick * p;
    const int b0 = brick * e;
    const int q = e / p, rem = e - q * p;
    lo = min(n, b0 + part * q + min(part, rem));
    hi = min(n, lo + q + (part < rem ? 1 : 0));
    slo = max(0, lo - k);
    shi = min(n, hi + k);
    centre = b0 + e / 2;
}

__device__ __forceinline__ BlockGeo block_geo(const Grid &g, const BrickGeom &bk, int b) {
    BlockGeo G;
    const int ibx = b % bk.nbx;
    const int rest = b / bk.nbx;
    const int iby = rest % bk.nby;
    const int ibz = rest / bk.nby;
    axis_part(g.nx, bk.bx, bk.px, ibx, g.kx, G.x0, G.x1, G.xs0, G.xs1, G.cxc);
    axis_part(g.ny, bk.by, bk.py, iby, g.ky, G.y0, G.y1, G.ys0, G.ys1, G.cyc);
    axis_part(g.nz, bk.bz, bk.pz, ibz, g.kz, G.z0, G.z1, G.zs0, G.zs1, G.czc);
    G.lx = G.xs1 - G.xs0;
    G.ry = G.ys1 - G.ys0;
    G.nr = G.ry * (G.zs1 - G.zs0);
    return G;
}

// A brow entry: first sorted slot of the row's staged cells, staging offset
// and length (both below 65 535 wherever the tables are used).
__device__ __forceinline__ int row_off(const int2 &e) { return (int)((unsigned)e.y & 0xffffu); }
__device__ __forceinline__ int row_len(const int2 &e) { return (int)((unsigned)e.y >> 16); }

// A bstage or bdest entry: sorted slot and cell relative to the origin cell,
// 128 added to each coordinate (a byte each; a brick spans at most 64 cells
// and three more on either side).
__device__ __forceinline__ int pack_cell(int cx, int cy, int cz) {
    return (cx + 128) | ((cy + 128) << 8) | ((cz + 128) << 16);
}
template <int C>
__device__ __forceinline__ int cell_int(int code) { return ((code >> (8 * C)) & 0xff) - 128; }
// the same as a float: the byte OR-ed into the bits of 2^23, less 2^23 + 128
template <int C>
__device__ __forceinline__ float cell_float(int code) {
    return __uint_as_float(__byte_perm((unsigned)code, 0x4B000000u, 0x7540u | C)) - 8388736.f;
}

// bstage entry t of the calling block, from its rows
__device__ __noinline__ int2 row_entry(const Grid &g, const BrickGeom &bk, const BrickSrcDev &S,
                                       int t) {
    const BlockGeo G = block_geo(g, bk, blockIdx.x);
    const int2 *rows = S.brow + (size_t)blockIdx.x * bk.nrmax;
    int r = 0;      // the last row that starts at or before t: the one that holds it
    for (int hi = G.nr - 1; r < hi;) {
        const int mid = (r + hi + 1) >> 1;
        if (row_off(rows[mid]) <= t) r = mid;
        else hi = mid - 1;
    }
    const int j = rows[r].x + (t - row_off(rows[r]));
    return make_int2(j, pack_cell((int)S.scx[j] - G.cxc, G.ys0 + r % G.ry - G.cyc,
                                  G.zs0 + r / G.ry - G.czc));
}

// The entries of the calling block's staged records: its part of bstage, or
// (TABLE = false: a build without that table, see brick_fill) found from the
// rows of cells that they come from.
template <bool TABLE>
struct StageTab;

template <>
struct StageTab<true> {
    const int2 *tab;
    __device__ __forceinline__ const int2 &operator[](int t) const { return tab[t]; }
};

template <>
struct StageTab<false> {
    const Grid *g;
    const BrickGeom *bk;
    const BrickSrcDev *S;
    __device__ __forceinline__ int2 operator[](int t) const { return row_entry(*g, *bk, *S, t); }
};

template <bool TABLE, class Args>
__device__ __forceinline__ StageTab<TABLE> stage_tab(const Args &A, const int4 &sh) {
    if constexpr (TABLE) return StageTab<true>{A.s.bstage + sh.y};
    else return StageTab<false>{&A.g, &A.bk, &A.s};
}

// Position record (brick-relative x, y, z and the mass) of record p in the
// cell of a table entry: the same FP32 operations for destinations and
// sources.
__device__ __forceinline__ float4 rel_pos(const float4 &p, int code, float csf) {
    return make_float4(fmaf(cell_float<0>(code), csf, p.x), fmaf(cell_float<1>(code), csf, p.y),
                       fmaf(cell_float<2>(code), csf, p.z), p.w);
}

// The dynamic shared memory of the brick kernels: the staged records from
// byte 0, then the cell table of a list build.
extern __shared__ __align__(16) unsigned char brick_smem[];

// The padding record (index T): far away, zero mass, at rest -- every pair
// term with it is exactly 0.
__device__ __forceinline__ float4 pad_pos() { return make_float4(1e15f, 1e15f, 1e15f, 0.f); }
__device__ __forceinline__ float4 pad_vel() { return make_float4(0.f, 0.f, 0.f, 0.f); }
// rates pass: the position record carries rho / 2, the state record (m,
// alpha cs / 2); the padding record has zero mass
__device__ __forceinline__ float4 pad_rpos() { return make_float4(1e15f, 1e15f, 1e15f, 0.5f); }
__device__ __forceinline__ float2 pad_rstate() { return make_float2(0.f, 0.f); }

// Source records: staged in shared memory, or (STAGED = false, a brick
// more populous than the shared memory holds) recomputed from the sorted
// arrays with the same operations.
template <bool STAGED, bool TABLE>
struct SrcRecords;

// Staged: the position record of source t at byte 16 t of the shared
// memory (x, y, z from the brick's centre cell, and m in the density pass,
// rho / 2 in the rates pass), in the rates pass the velocity record (u, v,
// w, p / rho^2) at voff + 16 t and the state record (m, alpha cs / 2) at
// soff + 8 t: 32-bit offsets into the shared array, so a record costs one
// address operation.  (Position and velocity interleaved in 32-byte
// records took 11 % longer: twice the bank conflicts of the random reads.)
// A rates pass whose block has one source mass and whose cs follows Tait
// (FAST) reads the first two only: the state record's 8-byte read was a
// fifth of the shared-memory wavefronts of a pair.
template <bool TABLE>
struct SrcRecords<true, TABLE> {
    uint32_t voff, soff;
    __device__ __forceinline__ float4 pos(int t) const {
        return *reinterpret_cast<const float4 *>(brick_smem + ((uint32_t)t << 4));
    }
    // rates pass: position (w = rho / 2), velocity, mass, alpha cs / 2
    template <bool FAST>
    __device__ __forceinline__ void rates_rec(int t, float mb, float tkc, float4 &p, float4 &v,
                                              float &mj, float &hac) const {
        p = *reinterpret_cast<const float4 *>(brick_smem + ((uint32_t)t << 4));
        v = *reinterpret_cast<const float4 *>(brick_smem + voff + ((uint32_t)t << 4));
        if (FAST) {
            // cs = co (rho / ro)^3
            mj = mb;
            hac = tkc * (p.w * p.w) * p.w;
        } else {
            const float2 s = *reinterpret_cast<const float2 *>(brick_smem + soff + ((uint32_t)t << 3));
            mj = s.x;
            hac = s.y;
        }
    }
};

// recomputed from the sorted arrays with the staging's operations
template <bool TABLE>
struct SrcRecords<false, TABLE> {
    const BrickSrcDev *src;
    StageTab<TABLE> tab;
    float csf;
    int T;
    float halpha;
    __device__ __forceinline__ float4 pos(int t) const {
        if (t >= T) return pad_pos();
        const int2 e = tab[t];
        return rel_pos(src->pm[e.x], e.y, csf);
    }
    template <bool FAST>
    __device__ __forceinline__ void rates_rec(int t, float, float, float4 &p, float4 &v, float &mj,
                                              float &hac) const {
        if (t >= T) {
            p = pad_rpos();
            v = pad_vel();
            mj = 0.f;
            hac = 0.f;
            return;
        }
        const int2 e = tab[t];
        const int j = e.x;
        p = rel_pos(src->pm[j], e.y, csf);
        const float4 vh = src->velh[j], st = src->st[j];
        mj = p.w;
        p.w = 0.5f * st.x;
        v = make_float4(vh.x, vh.y, vh.z, st.y);
        hac = halpha * st.z;
    }
};

template <bool STAGED, bool TABLE>
__device__ __forceinline__ SrcRecords<STAGED, TABLE> make_records(const BrickSmem &sm,
                                                                  const BrickSrcDev &S, float csf,
                                                                  const StageTab<TABLE> &tab, int T,
                                                                  float halpha) {
    if constexpr (STAGED)
        return SrcRecords<true, TABLE>{(uint32_t)sm.off_v, (uint32_t)sm.off_s};
    else
        return SrcRecords<false, TABLE>{&S, tab, csf, T, halpha};
}

// Asynchronous copies from global to shared memory (completed by the issuing
// thread's cp_async_wait): 16 and 8 bytes.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The records of stage, row by row (a build without the table of entries).
template <bool RATES>
__device__ __forceinline__ bool stage_rows(const StageTab<false> &tab, float csf,
                                           const BrickSmem &sm, bool state, float halpha,
                                           float mref) {
    const BrickSrcDev &S = *tab.S;
    const BlockGeo G = block_geo(*tab.g, *tab.bk, blockIdx.x);
    const int2 *rows = S.brow + (size_t)blockIdx.x * tab.bk->nrmax;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    bool same = true;
    for (int r = threadIdx.x >> 5; r < G.nr; r += nw) {
        const int2 e = rows[r];
        const int cy = G.ys0 + r % G.ry - G.cyc, cz = G.zs0 + r / G.ry - G.czc;
        for (int i = lane; i < row_len(e); i += 32) {
            const int j = e.x + i;
            const uint32_t t = (uint32_t)(row_off(e) + i);
            float4 pr = rel_pos(S.pm[j], pack_cell((int)S.scx[j] - G.cxc, cy, cz), csf);
            if (RATES) {
                const float4 vh = S.velh[j], st = S.st[j];
                same = same && pr.w == mref;
                *reinterpret_cast<float4 *>(brick_smem + sm.off_v + (t << 4)) =
                    make_float4(vh.x, vh.y, vh.z, st.y);
                if (state)
                    *reinterpret_cast<float2 *>(brick_smem + sm.off_s + (t << 3)) =
                        make_float2(pr.w, halpha * st.z);
                pr.w = 0.5f * st.x;
            }
            *reinterpret_cast<float4 *>(brick_smem + (t << 4)) = pr;
        }
    }
    return same;
}

// Copy the block's source records into shared memory (the layout of
// SrcRecords<true>).  The raw records (position; rates: velocity, rho and
// p / rho^2) are copied asynchronously, so that a thread has all its copies in
// flight and holds none in registers; then every thread finishes the records
// that it copied: the position from the block's origin cell, and in the rates
// pass (x, y, z, rho / 2), (u, v, w, p / rho^2) and, with STATE, (m, alpha cs /
// 2), with the halves that the pair averages of the artificial viscosity add.
// Returns whether every record this thread staged has mass mref.
template <bool RATES, bool TABLE>
__device__ __forceinline__ bool stage(const BrickSrcDev &S, const StageTab<TABLE> &tab, int T,
                                      float csf, const BrickSmem &sm, bool state, float halpha,
                                      float mref) {
    constexpr int U = 6;        // records of a thread in flight
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(brick_smem);
    const uint32_t vb = base + sm.off_v, sb = base + sm.off_s;
    const int nt = blockDim.x;
    if (threadIdx.x == 0) {
        // the padding record after the staged ones
        *reinterpret_cast<float4 *>(brick_smem + ((uint32_t)T << 4)) = RATES ? pad_rpos() : pad_pos();
        if (RATES) {
            *reinterpret_cast<float4 *>(brick_smem + sm.off_v + ((uint32_t)T << 4)) = pad_vel();
            *reinterpret_cast<float2 *>(brick_smem + sm.off_s + ((uint32_t)T << 3)) = pad_rstate();
        }
    }
    if constexpr (!TABLE) return stage_rows<RATES>(tab, csf, sm, state, halpha, mref);
    bool same = true;
    for (int t0 = threadIdx.x; t0 < T; t0 += U * nt) {
        int2 e[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t0 + u * nt < T) e[u] = tab[t0 + u * nt];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t t = (uint32_t)(t0 + u * nt);
            if (t < (uint32_t)T) {
                cp_async16(base + (t << 4), S.pm + e[u].x);
                if (RATES) {
                    cp_async16(vb + (t << 4), S.velh + e[u].x);
                    cp_async8(sb + (t << 3), S.st + e[u].x);
                }
            }
        }
        cp_async_wait();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t t = (uint32_t)(t0 + u * nt);
            if (t < (uint32_t)T) {
                float4 *prec = reinterpret_cast<float4 *>(brick_smem + (t << 4));
                float4 pr = rel_pos(*prec, e[u].y, csf);
                if (RATES) {
                    float2 *srec = reinterpret_cast<float2 *>(brick_smem + sm.off_s + (t << 3));
                    const float2 rp = *srec;
                    same = same && pr.w == mref;
                    if (state) *srec = make_float2(pr.w, halpha * S.st[e[u].x].z);
                    *reinterpret_cast<float *>(brick_smem + sm.off_v + (t << 4) + 12) = rp.y;
                    pr.w = 0.5f * rp.x;
                }
                *prec = pr;
            }
        }
    }
    return same;
}

// The state records (m, alpha cs / 2) of a block whose sources turned out not
// to share one mass.
template <bool TABLE>
__device__ __noinline__ void stage_state(const BrickSrcDev &S, StageTab<TABLE> tab, int T,
                                         uint32_t soff, float halpha) {
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        const int j = tab[t].x;
        *reinterpret_cast<float2 *>(brick_smem + soff + ((uint32_t)t << 3)) =
            make_float2(S.pm[j].w, halpha * S.st[j].z);
    }
}

// Staging offset of the first particle of every cell of every staged row
// (scell[r * (lx + 1) + i], i = 0 .. lx): the ranges a stencil traversal
// visits.
__device__ __forceinline__ void cell_table(const Grid &g, const BlockGeo &G, const int *scst,
                                           const int2 *brow, int *scell) {
    const int w = G.lx + 1;
    const int rowz = g.nx * g.ny;
    for (int idx = threadIdx.x; idx < G.nr * w; idx += blockDim.x) {
        const int r = idx / w, i = idx - r * w;
        const int cy = G.ys0 + r % G.ry, cz = G.zs0 + r / G.ry;
        const int2 e = brow[r];
        scell[idx] = row_off(e) + (scst[cz * rowz + cy * g.nx + G.xs0 + i] - e.x);
    }
}

// The 16-bit entry i (0..7) of a group.
__device__ __forceinline__ int group_entry(const uint4 &q, int i) {
    const unsigned w = i < 2 ? q.x : (i < 4 ? q.y : (i < 6 ? q.z : q.w));
    return (int)((i & 1) ? (w >> 16) : (w & 0xffffu));
}

// One destination of the block: slot, original index, cell, the cell-local
// offsets that prune the stencil and the brick-relative position and mass.
struct BrickDest {
    int s, orig;
    int cx, cy, cz;
    float4 xi, P;
};

__device__ __forceinline__ BrickDest brick_dest(const BrickDstDev &D, const BlockGeo &G, float csf,
                                                const int2 &e) {
    BrickDest q;
    q.s = e.x;
    q.cx = G.cxc + cell_int<0>(e.y);
    q.cy = G.cyc + cell_int<1>(e.y);
    q.cz = G.czc + cell_int<2>(e.y);
    q.orig = D.perm[q.s];
    q.xi = D.pm[q.s];
    q.P = rel_pos(q.xi, e.y, csf);
    return q;
}

__device__ __forceinline__ bool is_real(const BrickDstDev &D, int orig) {
    return D.tag == nullptr || D.tag[orig] == SPH_TAG_LOCAL_REAL;
}

// FP64 neighbour test of a source slot, inside the FP32 band
__device__ __noinline__ bool exact_hit(const BrickSrcDev &S, const BrickDstDev &D, int slot, int orig,
                                       double radius2) {
    const int oj = S.perm[slot];
    return exact_within(ld0(S.x, oj), ld0(S.y, oj), ld0(S.z, oj), ld0(D.x, orig), ld0(D.y, orig),
                        ld0(D.z, orig), radius2);
}

// Visit the sources of destination q that its list holds, in the staged
// records, in the order of the list-streaming kernels: stencil rows [r0, r1)
// in (dz, dy) order, each clipped to the chord of the search sphere,
// ascending slot within a row.  fn(t0, m): the listed ones among staging
// indices t0 .. t0 + 31, as bits.  (A listed source costs several times a
// candidate, one in four or five is listed, and a warp that handled each as it
// came paid for it at nearly every candidate: list build of 275 K particles
// 218 us, 195 by masks.)  With a list skin every source within the list radius is listed,
// without one the neighbours.  The ranges come from the block's cell table
// (scell) or, without one, from the grid's cell table.
template <bool SKIN, bool STAGED, bool TABLE, class Fn>
__device__ __forceinline__ void brick_rows(const Grid &g, const BlockGeo &G, const BrickSrcDev &S,
                                               const BrickDstDev &D, const SrcRecords<STAGED, TABLE> &R,
                                               const BrickRadius &rad, const int2 *brow,
                                               const StageTab<TABLE> &tab, const int *scell,
                                               const BrickDest &q, int r0, int r1,
                                               Fn &&fn) {
    const float csf = g.cs_f;
    const float inv_cs = 1.f / csf;
    const float R2 = fmaxf(rad.r2hi, rad.r2list) * 1.0002f;
    // listed below rl, without a skin up to r2hi where the FP64 test says so
    const float rl = SKIN ? rad.r2list : rad.r2lo;
    const int w = G.lx + 1;
    const int K = g.kx, wy = 2 * g.ky + 1;
    int dz = r0 / wy, dy = r0 - dz * wy - g.ky;
    dz -= g.kz;
#pragma unroll 1
    for (int rr = r0; rr < r1; ++rr, dz += dy == g.ky ? 1 : 0, dy = dy == g.ky ? -g.ky : dy + 1) {
        const int czz = q.cz + dz, cyy = q.cy + dy;
        if (czz < G.zs0 || czz >= G.zs1 || cyy < G.ys0 || cyy >= G.ys1) continue;
        const float ez = fmaxf(0.f, dz > 0 ? (float)dz * csf - q.xi.z
                                           : (dz < 0 ? q.xi.z - (float)(dz + 1) * csf : 0.f));
        const float ey = fmaxf(0.f, dy > 0 ? (float)dy * csf - q.xi.y
                                           : (dy < 0 ? q.xi.y - (float)(dy + 1) * csf : 0.f));
        const float rem = R2 - fmaf(ey, ey, ez * ez);
        if (rem < 0.f) continue;
        const float half = fmaf(rem * rsqrtf(fmaxf(rem, 1e-30f)), 1.0001f, 1e-5f * csf);
        const int tlo = max(-K, __float2int_rd((q.xi.x - half) * inv_cs));
        const int thi = min(K, __float2int_rd((q.xi.x + half) * inv_cs));
        const int clo = max(q.cx + tlo, G.xs0);
        const int chi = min(q.cx + thi, G.xs1 - 1);
        if (clo > chi) continue;
        const int r = (cyy - G.ys0) + G.ry * (czz - G.zs0);
        int ta, tb;
        if (scell != nullptr) {
            ta = scell[r * w + (clo - G.xs0)];
            tb = scell[r * w + (chi + 1 - G.xs0)];
        } else {
            const int2 e = brow[r];
            const int c = (czz * g.ny + cyy) * g.nx;
            ta = row_off(e) + (__ldg(S.cstart + c + clo) - e.x);
            tb = row_off(e) + (__ldg(S.cstart + c + chi + 1) - e.x);
        }
        for (int t0 = ta; t0 < tb; t0 += 32) {
            const int e = min(32, tb - t0);
            unsigned m = 0, band = 0;
            for (int u0 = 0; u0 < e; u0 += 8) {
                unsigned mm = 0, bb = 0;
                // (records past the row are read, not used: kSlack of them follow
                // the last)
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float4 pj = R.pos(t0 + u0 + u);
                    const float rx = q.P.x - pj.x, ry = q.P.y - pj.y, rz = q.P.z - pj.z;
                    const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
                    if (r2 < rl) mm |= 1u << u;
                    else if (!SKIN && r2 <= rad.r2hi) bb |= 1u << u;
                }
                m |= mm << u0;
                if (!SKIN) band |= bb << u0;
            }
            const unsigned row = 0xffffffffu >> (32 - e);
            m &= row;
            if (!SKIN) {
                for (band &= row; band; band &= band - 1) {
                    const int u = __ffs(band) - 1;
                    if (exact_hit(S, D, tab[t0 + u].x, q.orig, rad.radius2)) m |= 1u << u;
                }
            }
            fn(t0, m);
        }
    }
}

template <bool STAGED, bool TABLE, class Fn>
__device__ __forceinline__ void brick_traverse(const Grid &g, const BlockGeo &G, const BrickSrcDev &S,
                                               const BrickDstDev &D, const SrcRecords<STAGED, TABLE> &R,
                                               const BrickRadius &rad, const int2 *brow,
                                               const StageTab<TABLE> &tab, const int *scell,
                                               const BrickDest &q, int r0, int r1,
                                               Fn &&fn) {
    if (rad.r2list > 0.f) brick_rows<true, STAGED, TABLE>(g, G, S, D, R, rad, brow, tab, scell, q, r0, r1, fn);
    else brick_rows<false, STAGED, TABLE>(g, G, S, D, R, rad, brow, tab, scell, q, r0, r1, fn);
}

// Reciprocal square root and reciprocal, flushing subnormal inputs to zero
// (the pair terms' inputs are bounded away from the subnormal range: r^2 is
// clamped to 1e-30, the density sums are near the rest density).
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ---------------------------------------------------------------------------
// summation density (density_funcs.pyx:38-74) + Tait (eos_funcs.pyx:105-116)
// ---------------------------------------------------------------------------
// fac W(q) of the cubic spline (base/kernels.pyx:351-374), the normalisation
// (and any constant factor) folded into the coefficients: fac (1 - 1.5 q^2
// + 0.75 q^3) for q <= 1, fac / 4 (2 - q)^3 for 1 < q <= 2, else 0.
struct WCoef {
    float i0, i1, i2, o;
};

__device__ __forceinline__ WCoef w_coef(float fac, float scale) {
    const float f = fac * scale;
    return WCoef{f, -1.5f * f, 0.75f * f, 0.25f * f};
}

__device__ __forceinline__ float w_of(float q, const WCoef &c) {
    const float inner = fmaf(q * q, fmaf(c.i2, q, c.i1), c.i0);
    // (2 - q) clamped at 0: the outer branch is 0 beyond q = 2
    const float t = fmaxf(2.f - q, 0.f);
    const float outer = c.o * (t * t) * t;
    return q > 1.f ? outer : inner;
}

__device__ __forceinline__ float density_term(const float4 &pi, const float4 &pj, float ih,
                                              const WCoef &wc) {
    const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
    const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
    const float r = r2 * rsqrt_ftz(fmaxf(r2, 1e-30f));
    return w_of(r * ih, wc) * pj.w;
}

// Density of one destination (the compensated sum hi + lo) and, with
// Tait, its p and cs; the sorted state record when the pass writes the
// destination's own properties.  FP64 values are made by integer operations
// (f2d_exact): the FP64 pipe sees one addition per destination, not five
// instructions (8 of the 155 us of this pass at 1 M particles).
__device__ __forceinline__ void density_store(const BrickDensityArgs &A, int s, int orig, bool real,
                                              float mi, float hi, float lo) {
    const double r64 = f2d_exact(hi) + f2d_exact(lo);
    if (A.rho_out) A.rho_out[orig] = r64;
    const float rf = hi + lo;
    float pf = 0.f, cf = 0.f;
    if (A.tait) {
        if (real) {
            // p = B((rho/ro)^gamma - 1), cs = co (rho/ro)^((gamma-1)/2), through
            // log1p/expm1 of the density excess (relative accuracy of p as
            // rho -> ro); hi - ro is exact for hi within a factor 2 of ro
            const float Bt = A.co * A.co * A.ro / A.gamma;
            const float lr = log1pf(((hi - A.ro) + lo) * (1.f / A.ro));
            pf = Bt * expm1f(A.gamma * lr);
            cf = A.co * expf(0.5f * (A.gamma - 1.f) * lr);
        }
        A.p_out[orig] = f2d_exact(pf);
        A.cs_out[orig] = f2d_exact(cf);
    }
    if (A.st_out) {
        if (A.tait) {
            A.st_out[s] = make_float4(rf, pf / (rf * rf), cf, mi);
        } else {
            const float pold = d2f_rn(ld0(A.d.p, orig));
            A.st_out[s] = make_float4(rf, pold / (rf * rf), d2f_rn(ld0(A.d.cs, orig)), mi);
        }
    }
}

// Fold the batches that the S lanes of a destination have just summed into
// its compensated sum, in the order of the list: every lane adds all S of
// them, so all hold the sum that one thread would have.
// mask: the warp's lanes that fold together (a mask per destination would make
// the warp run each destination's shuffles by themselves).
template <int S>
__device__ __forceinline__ void fold_lanes(CSum &c, float part, unsigned mask) {
    if (S == 1) {
        c.add(part);
    } else {
#pragma unroll
        for (int s = 0; s < S; ++s) c.add(__shfl_sync(mask, part, s, S));
    }
}

// What a column (a lane of a destination) starts from: the destination's
// records, its count and the first two groups of the lane.  Every thread
// requests those of its first column before the block stages its sources, so
// their latency overlaps the staging.
struct DestPre {
    int s, orig;    // sorted slot, original index
    float4 P;       // brick-relative position, mass
    int c;
    uint4 b0, b1;
};

template <int S>
__device__ __forceinline__ void dest_prefetch(const BrickDstDev &Dd, float csf, const int2 &e,
                                              const int *cnt, const uint4 *lgrp, int cap, int D,
                                              int d, int lane, DestPre &p) {
    p.s = e.x;
    p.orig = Dd.perm[e.x];
    p.P = rel_pos(Dd.pm[e.x], e.y, csf);
    p.c = cnt[d];
    // every destination owns cap / 8 groups: those inside are read whatever
    // the count (used only as far as it reaches)
    const int ng = cap >> 3;
    const uint4 *lst = lgrp + d;
    p.b0 = lane < ng ? lst[(size_t)lane * D] : make_uint4(0, 0, 0, 0);
    p.b1 = lane + S < ng ? lst[(size_t)(lane + S) * D] : make_uint4(0, 0, 0, 0);
}

// The density sum of a destination over its groups of 8 entries, every lane
// taking every S-th group, each requested two ahead into one of three
// rotating buffers (the loop is unrolled over the three, so no buffer is
// copied).
template <int S, bool STAGED, bool TABLE>
__device__ __forceinline__ void density_group(CSum &rho, const SrcRecords<STAGED, TABLE> &R, bool mine,
                                              const uint4 &grp, const float4 &Pi, float ih,
                                              const WCoef &wc, unsigned mask) {
    float part = 0.f;
    if (S == 1 || mine) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float4 pj[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) pj[i] = R.pos(group_entry(grp, 4 * h + i));
#pragma unroll
            for (int i = 0; i < 4; ++i) part += density_term(Pi, pj[i], ih, wc);
        }
    }
    fold_lanes<S>(rho, part, mask);
}

template <int S, bool STAGED, bool TABLE>
__device__ __forceinline__ void density_stream(CSum &rho, const SrcRecords<STAGED, TABLE> &R,
                                               const uint4 *lst, int D, int ng, int lane,
                                               const float4 &Pi, float ih, const WCoef &wc, uint4 b0,
                                               uint4 b1, unsigned mask) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
    // the rounds of the warp's longest list (a batch of none adds 0)
    const int nr = S > 1 ? __reduce_max_sync(mask, ng) : ng;
    const size_t step = (size_t)D;
    uint4 b2;
    // g0: the first group of the round, gi: this lane's
    for (int g0 = 0, gi = lane;;) {
        if (g0 >= nr) break;
        b2 = gi + 2 * S < ng ? lst[(gi + 2 * S) * step] : zero;
        density_group<S, STAGED, TABLE>(rho, R, gi < ng, b0, Pi, ih, wc, mask);
        gi += S;
        if ((g0 += S) >= nr) break;
        b0 = gi + 2 * S < ng ? lst[(gi + 2 * S) * step] : zero;
        density_group<S, STAGED, TABLE>(rho, R, gi < ng, b1, Pi, ih, wc, mask);
        gi += S;
        if ((g0 += S) >= nr) break;
        b1 = gi + 2 * S < ng ? lst[(gi + 2 * S) * step] : zero;
        density_group<S, STAGED, TABLE>(rho, R, gi < ng, b2, Pi, ih, wc, mask);
        gi += S;
        g0 += S;
    }
}

// The list of one destination: its S lanes take consecutive shares of the
// stencil rows.  One lane: entries are collected eight at a time in a 128-bit
// shift register (the newest enters at the top) and written as one 16-byte
// store per group.  Several: each counts its share, a scan over the lanes
// gives its place in the list, and a second traversal writes the entries.
// The last group is padded with the zero record.  Returns the list's count.
template <int S, bool STAGED, bool TABLE>
__device__ __forceinline__ int build_list(const BrickDensityArgs &A, const BlockGeo &G,
                                          const SrcRecords<STAGED, TABLE> &R, const int2 *brow,
                                          const StageTab<TABLE> &tab, const int *scell,
                                          const BrickDest &q, bool active,
                                          int lane, int T, uint4 *out, int D) {
    const int cap = A.cap;
    const int rows = (2 * A.g.ky + 1) * (2 * A.g.kz + 1);
    int c = 0;
    if (S == 1) {
        if (!active) return 0;
        uint4 grp = make_uint4(0, 0, 0, 0);
        auto push = [&](unsigned t) {
            grp.x = __funnelshift_r(grp.x, grp.y, 16);
            grp.y = __funnelshift_r(grp.y, grp.z, 16);
            grp.z = __funnelshift_r(grp.z, grp.w, 16);
            grp.w = (grp.w >> 16) | (t << 16);
        };
        brick_traverse<STAGED, TABLE>(A.g, G, A.s, A.d, R, A.rad, brow, tab, scell, q, 0, rows,
            [&](int t0, unsigned m) {
                for (; m; m &= m - 1) {
                    push((unsigned)(t0 + __ffs(m) - 1));
                    ++c;
                    if ((c & 7) == 0 && c <= cap) out[(size_t)((c >> 3) - 1) * D] = grp;
                }
            });
        if (c < cap && (c & 7)) {
            for (int k = c; k & 7; ++k) push((unsigned)T);
            out[(size_t)(c >> 3) * D] = grp;
        }
        return c;
    }
    const int ra = rows * lane / S, rb = rows * (lane + 1) / S;
    if (active)
        brick_traverse<STAGED, TABLE>(A.g, G, A.s, A.d, R, A.rad, brow, tab, scell, q, ra, rb,
                               [&](int, unsigned m) { c += __popc(m); });
    __syncwarp();
    int end = c;
#pragma unroll
    for (int off = 1; off < S; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, end, off, S);
        if (lane >= off) end += y;
    }
    const int total = __shfl_sync(0xffffffffu, end, S - 1, S);
    if (active) {
        int k = end - c;
        uint16_t *o16 = reinterpret_cast<uint16_t *>(out);
        auto write = [&](unsigned t) {
            if (k < cap) o16[(size_t)(k >> 3) * D * 8 + (k & 7)] = (uint16_t)t;
            ++k;
        };
        brick_traverse<STAGED, TABLE>(A.g, G, A.s, A.d, R, A.rad, brow, tab, scell, q, ra, rb,
                               [&](int t0, unsigned m) {
                                   for (; m; m &= m - 1) write((unsigned)(t0 + __ffs(m) - 1));
                               });
        if (lane == S - 1)
            while (k & 7) write((unsigned)T);
    }
    // the lanes read each other's entries
    __threadfence_block();
    __syncwarp();
    return total;
}

// The density sum of a list build: plain FP32 batches of 8 neighbours (the
// listed sources that the skin adds do not count), each folded into the
// compensated sum; past the list's capacity the traversal goes on.
template <bool STAGED, bool TABLE>
__device__ __forceinline__ void build_sum(const BrickDensityArgs &A, const BlockGeo &G,
                                          const SrcRecords<STAGED, TABLE> &R, const int2 *brow,
                                          const StageTab<TABLE> &tab, const int *scell,
                                          const BrickDest &q, int c,
                                          const uint4 *lst, int D, float ih, const WCoef &wc,
                                          CSum &rho) {
    const int cap = A.cap;
    const float r2lo = A.rad.r2lo, r2hi = A.rad.r2hi;
    float part = 0.f;
    int nb = 0;
    auto add = [&](float r2, float m) {
        const float r = r2 * rsqrt_ftz(fmaxf(r2, 1e-30f));
        part += w_of(r * ih, wc) * m;
        if (++nb == 8) {
            rho.add(part);
            part = 0.f;
            nb = 0;
        }
    };
    auto dist2 = [&](const float4 &pj) {
        const float rx = q.P.x - pj.x, ry = q.P.y - pj.y, rz = q.P.z - pj.z;
        return fmaf(rx, rx, fmaf(ry, ry, rz * rz));
    };
    const int ng = (min(c, cap) + 7) >> 3;
    uint4 next = ng > 0 ? lst[0] : make_uint4(0, 0, 0, 0);
    for (int gi = 0; gi < ng; ++gi) {
        const uint4 grp = next;
        if (gi + 1 < ng) next = lst[(size_t)(gi + 1) * D];
        float r2[8], m[8];
        unsigned hit = 0, band = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 pj = R.pos(group_entry(grp, i));
            r2[i] = dist2(pj);
            m[i] = pj.w;
            if (r2[i] <= r2hi) hit |= 1u << i;
            if (!(r2[i] < r2lo) && r2[i] <= r2hi) band |= 1u << i;
        }
        if (band) {
#pragma unroll 1
            for (int i = 0; i < 8; ++i)
                if ((band >> i) & 1u) {
                    const unsigned w = i < 2 ? grp.x : (i < 4 ? grp.y : (i < 6 ? grp.z : grp.w));
                    const int t = (int)((i & 1) ? (w >> 16) : (w & 0xffffu));
                    if (!exact_hit(A.s, A.d, tab[t].x, q.orig, A.rad.radius2)) hit &= ~(1u << i);
                }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if ((hit >> i) & 1u) add(r2[i], m[i]);
    }
    if (c > cap) {
        int skip = cap;
        const int rows = (2 * A.g.ky + 1) * (2 * A.g.kz + 1);
        brick_traverse<STAGED, TABLE>(A.g, G, A.s, A.d, R, A.rad, brow, tab, scell, q, 0, rows,
            [&](int t0, unsigned bits) {
                for (; bits; bits &= bits - 1) {
                    if (skip > 0) { --skip; continue; }
                    const int t = t0 + __ffs(bits) - 1;
                    const float4 pj = R.pos(t);
                    const float d2 = dist2(pj);
                    bool hit = d2 < r2lo;
                    if (!hit && d2 <= r2hi)
                        hit = exact_hit(A.s, A.d, tab[t].x, q.orig, A.rad.radius2);
                    if (hit) add(d2, pj.w);
                }
            });
    }
    rho.add(part);
}

// Destinations with more neighbours than their list holds: the rest come
// from a traversal that skips the listed ones (in the order of the list
// build), added to the stored partial density.  A call of its own, so that
// the passes keep its registers out of their loops.
template <bool STAGED, bool TABLE>
__device__ __noinline__ void density_rest(const BrickDensityArgs &A) {
    const int b = blockIdx.x;
    const int2 dh = A.d.bdst[b];
    const int4 sh = A.s.bsrc[b];
    const Grid &g = A.g;
    const BlockGeo G = block_geo(g, A.bk, b);
    const int2 *brow = A.s.brow + (size_t)b * A.bk.nrmax;
    const StageTab<TABLE> tab = stage_tab<TABLE>(A, sh);
    const SrcRecords<STAGED, TABLE> R = make_records<STAGED, TABLE>(A.sm, A.s, g.cs_f, tab, sh.x, 0.f);
    const float ih = __fdividef(1.f, g.h_uniform);
    const float fac = cubic_fac(A.dim, ih);
    const int rows = (2 * g.ky + 1) * (2 * g.kz + 1);
    __syncthreads();    // the partial densities, another thread's with several lanes
    for (int d = threadIdx.x; d < dh.x; d += blockDim.x) {
        if (A.cnt[dh.y + d] <= A.cap) continue;
        const BrickDest q = brick_dest(A.d, G, g.cs_f, A.d.bdest[dh.y + d]);
        if (!is_real(A.d, q.orig)) continue;
        CSum rest;
        int skip = A.cap;
        brick_traverse<STAGED, TABLE>(g, G, A.s, A.d, R, A.rad, brow, tab, nullptr, q, 0, rows,
            [&](int t0, unsigned m) {
                for (; m; m &= m - 1) {
                    if (skip > 0) { --skip; continue; }
                    const float4 pj = R.pos(t0 + __ffs(m) - 1);
                    const float rx = q.P.x - pj.x, ry = q.P.y - pj.y, rz = q.P.z - pj.z;
                    const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
                    const float r = r2 > 0.f ? r2 * rsqrtf(r2) : 0.f;
                    rest.add(cubic_w(r * ih) * fac * pj.w);
                }
            });
        // the stored partial density (hi + lo of the listed part, in FP64)
        // plus the rest, as a compensated FP32 pair
        CSum tot = rest;
        const double part = A.rho_out[q.orig];
        const float phi = (float)part;
        tot.merge(phi, (float)(part - (double)phi));
        density_store(A, q.s, q.orig, true, q.P.w, tot.hi, tot.lo);
    }
}

// The density of destination d of the block (its prefetched records p).
template <int S, bool STAGED, bool TABLE>
__device__ __forceinline__ void density_dest(const BrickDensityArgs &A, const SrcRecords<STAGED, TABLE> &R,
                                             const uint4 *lst, int D, int lane, const DestPre &p,
                                             unsigned mask) {
    const float ih = __fdividef(1.f, A.g.h_uniform);
    const WCoef wc = w_coef(cubic_fac(A.dim, ih), 1.f);
    CSum rho;
    density_stream<S, STAGED, TABLE>(rho, R, lst, D, (min(p.c, A.cap) + 7) >> 3, lane, p.P, ih, wc, p.b0,
                              p.b1, mask);
    if (lane == 0) {
        const bool real = is_real(A.d, p.orig);
        density_store(A, p.s, p.orig, real, p.P.w, real ? rho.hi : 0.f, real ? rho.lo : 0.f);
    }
}

// Destinations past one per column of the block: a thread each while more than a
// quarter of the block's threads have one, the last ones shared by four lanes
// each.  (A wide support has a thousand destinations and more in a brick: RK2
// step of 49 091 particles in 2D, h / dx 4, 422 us, with four lanes for all of
// them 685; h / dx 1.7, some 120 past the block's 320 threads, 84, with four
// lanes up to half the block 92.)  A call of its own, so that the passes keep
// its registers out of their loops.
template <bool STAGED, bool TABLE>
__device__ __noinline__ void density_more(const BrickDensityArgs &A, int first) {
    constexpr int S = 4;
    const int b = blockIdx.x;
    const int2 dh = A.d.bdst[b];
    const int4 sh = A.s.bsrc[b];
    const SrcRecords<STAGED, TABLE> R =
        make_records<STAGED, TABLE>(A.sm, A.s, A.g.cs_f, stage_tab<TABLE>(A, sh), sh.x, 0.f);
    const uint4 *lgrp = reinterpret_cast<const uint4 *>(A.nbr) + (size_t)dh.y * (A.cap >> 3);
    const int lane = threadIdx.x % S, nt = blockDim.x;
    int r0 = first;
    for (; dh.x - r0 > nt / 4; r0 += nt) {
        const int d = r0 + threadIdx.x;
        if (d >= dh.x) continue;
        DestPre p;
        dest_prefetch<1>(A.d, A.g.cs_f, A.d.bdest[dh.y + d], A.cnt + dh.y, lgrp, A.cap, dh.x, d, 0,
                         p);
        density_dest<1, STAGED, TABLE>(A, R, lgrp + d, dh.x, 0, p, 0xffffffffu);
    }
    for (; r0 < dh.x; r0 += nt / S) {
        const int d = r0 + threadIdx.x / S;
        const unsigned mask = __ballot_sync(0xffffffffu, d < dh.x);
        if (d >= dh.x) continue;
        DestPre p;
        dest_prefetch<S>(A.d, A.g.cs_f, A.d.bdest[dh.y + d], A.cnt + dh.y, lgrp, A.cap, dh.x, d,
                         lane, p);
        density_dest<S, STAGED, TABLE>(A, R, lgrp + d, dh.x, lane, p, mask);
    }
}

template <int S, bool STAGED, bool TABLE>
__global__ void __maxnreg__(64) k_bdensity(const __grid_constant__ BrickDensityArgs A) {
    const int b = blockIdx.x;
    const int2 dh = A.d.bdst[b];        // destinations, first destination
    const int4 sh = A.s.bsrc[b];        // staged records, their table
    if (dh.x == 0) return;
    // read now, tested after the staging: everything up to there only reads
    // tables and lists of the last build and positions
    const unsigned off = A.gate != nullptr ? *A.gate : 0u;
    const int T = sh.x, D = dh.x;
    const StageTab<TABLE> tab = stage_tab<TABLE>(A, sh);
    const uint4 *lgrp = reinterpret_cast<const uint4 *>(A.nbr) + (size_t)dh.y * (A.cap >> 3);
    const int lane = threadIdx.x % S, d = threadIdx.x / S;
    // the destination of this thread, requested before the staging
    DestPre pre;
    if (d < D)
        dest_prefetch<S>(A.d, A.g.cs_f, A.d.bdest[dh.y + d], A.cnt + dh.y, lgrp, A.cap, D, d, lane,
                         pre);
    if (STAGED) stage<false, TABLE>(A.s, tab, T, A.g.cs_f, A.sm, false, 0.f, 0.f);
    __syncthreads();
    if (off != 0u) return;
    const SrcRecords<STAGED, TABLE> R = make_records<STAGED, TABLE>(A.sm, A.s, A.g.cs_f, tab, T, 0.f);
    const unsigned mask = S > 1 ? __ballot_sync(0xffffffffu, d < D) : 0xffffffffu;
    if (d < D) density_dest<S, STAGED, TABLE>(A, R, lgrp + d, D, lane, pre, mask);
    if (D > (int)blockDim.x / S) density_more<STAGED, TABLE>(A, blockDim.x / S);
    if (*A.maxcnt > A.cap && A.rho_out != nullptr) density_rest<STAGED, TABLE>(A);
}

// List build: every destination's list from a traversal, and (write_out) its
// density from the list just written.  Bound by issue, half the lanes idle in
// the traversal (the chords of a warp's destinations differ in length), so
// that loop only tests and lists; summing in it, under the same divergence,
// took 790 us at 1 M particles against 626 (both before the masks).
template <int S, bool STAGED, bool TABLE>
__global__ void __maxnreg__(64) k_bbuild(const __grid_constant__ BrickDensityArgs A) {
    const int b = blockIdx.x;
    const int2 dh = A.d.bdst[b];
    const int4 sh = A.s.bsrc[b];
    if (dh.x == 0) return;
    const unsigned off = A.gate != nullptr ? *A.gate : 0u;
    const Grid &g = A.g;
    const BlockGeo G = block_geo(g, A.bk, b);
    const int2 *brow = A.s.brow + (size_t)b * A.bk.nrmax;
    const StageTab<TABLE> tab = stage_tab<TABLE>(A, sh);
    const int T = sh.x, D = dh.x;
    const int cap = A.cap;              // a multiple of 8
    uint4 *lgrp = reinterpret_cast<uint4 *>(A.nbr) + (size_t)dh.y * (cap >> 3);
    int *cnt = A.cnt + dh.y;
    const int2 *bdest = A.d.bdest + dh.y;
    int *scell = reinterpret_cast<int *>(brick_smem + A.sm.off_scell);
    const int lane = threadIdx.x % S, d0 = threadIdx.x / S, step = blockDim.x / S;
    cell_table(g, G, A.s.cstart, brow, scell);
    if (STAGED) stage<false, TABLE>(A.s, tab, T, g.cs_f, A.sm, false, 0.f, 0.f);
    __syncthreads();
    if (off != 0u) return;
    const SrcRecords<STAGED, TABLE> R = make_records<STAGED, TABLE>(A.sm, A.s, g.cs_f, tab, T, 0.f);
    // every thread of a warp runs every round (build_list shuffles)
    for (int r0 = 0; r0 < D; r0 += step) {
        const int d = r0 + d0;
        const bool active = d < D;
        BrickDest q;
        bool real = false;
        if (active) {
            q = brick_dest(A.d, G, g.cs_f, bdest[d]);
            real = is_real(A.d, q.orig);
        }
        const int c = build_list<S, STAGED, TABLE>(A, G, R, brow, tab, scell, q, real, lane, T, lgrp + d, D);
        if (!active) continue;
        if (lane == 0) cnt[d] = c;
        const unsigned act = __activemask();
        const int wmax = __reduce_max_sync(act, c);
        if ((threadIdx.x & 31) == (__ffs(act) - 1)) atomicMax(A.maxcnt, wmax);
        if (!A.write_out || lane != 0) continue;
        const float ih = __fdividef(1.f, g.h_uniform);
        const WCoef wc = w_coef(cubic_fac(A.dim, ih), 1.f);
        CSum rho;
        if (real) build_sum<STAGED, TABLE>(A, G, R, brow, tab, scell, q, c, lgrp + d, D, ih, wc, rho);
        density_store(A, q.s, q.orig, real, q.P.w, real ? rho.hi : 0.f, real ? rho.lo : 0.f);
    }
}

// ---------------------------------------------------------------------------
// rates: PGrad (pressure_funcs.pyx:40-91) + Monaghan AV (viscosity_funcs.pyx:
// 41-124) [+ XSPH (xsph_funcs.pyx:31-88)], uniform h, one source, with
// gravity (external_force.pyx:39-45) and position stepping
// (position_funcs.pyx:32-60) folded into the store
// ---------------------------------------------------------------------------
struct RatesConst {
    float h, ih, beta, eta2h2;
    float gin0, gin1, gout;     // fac dW/dr / r: gin1 q + gin0 (q < 1), gout (2-q)^2 / r (q < 2)
    WCoef wx;                   // eps fac W(q) (XSPH)
    float mb, tkc;              // two-record blocks: the sources' mass, alpha cs / 2 per (rho / 2)^3
};

__device__ __forceinline__ RatesConst rates_const(float h, float fac, float beta, float eta2,
                                                  float eps) {
    RatesConst k;
    k.h = h;
    k.ih = __fdividef(1.f, h);
    k.beta = beta;
    k.eta2h2 = eta2 * h * h;
    // fac 3 (0.75 q - 1) / h^2 and -0.75 fac (2 - q)^2 / (h r) (base/kernels.pyx:376-413)
    k.gin1 = 2.25f * fac * k.ih * k.ih;
    k.gin0 = -3.f * fac * k.ih * k.ih;
    k.gout = -0.75f * fac * k.ih;
    k.wx = w_coef(fac, eps);
    k.mb = 0.f;
    k.tkc = 0.f;
    return k;
}

// destination state and the sums: plain FP32 partials of a batch, merged
// into the Neumaier-compensated totals by flush()
struct RatesAcc {
    float4 vi;
    float hrhoi, pri, haci;     // rho_i / 2, p_i / rho_i^2, alpha cs_i / 2
    float pax, pay, paz, pxx, pxy, pxz;
    CSum ax, ay, az, xx, xy, xz;
};

// One pair: pressure gradient -m_j (p_i/rho_i^2 + p_j/rho_j^2) grad W
// (pressure_funcs.pyx:67-91), Monaghan viscosity -m_j Pi_ab grad W with
// mu = h v_ab.r_ab / (r^2 + eta^2 h^2) for approaching pairs
// (viscosity_funcs.pyx:72-124; min(v.r, 0) gives mu = 0 otherwise, and
// with eta = 0, as the reference's class always has, 1/r^2 comes from the
// rsqrt already taken), and XSPH eps m_j W (v_j - v_i) / rho_ab
// (xsph_funcs.pyx:44-88), sharing 1 / rho_ab.
// Source record: pj = (position, rho_j / 2), vj = (velocity, p_j / rho_j^2),
// mj, hacj = alpha cs_j / 2.
template <bool XSPH, bool ETA0>
__device__ __forceinline__ void rates_pair(RatesAcc &a, const RatesConst &k, float rx, float ry,
                                           float rz, const float4 &pj, const float4 &vj,
                                           float mj, float hacj) {
    const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
    const float rinv = rsqrt_ftz(fmaxf(r2, 1e-30f));
    const float q = r2 * rinv * k.ih;
    const float dot = (a.vi.x - vj.x) * rx + (a.vi.y - vj.y) * ry + (a.vi.z - vj.z) * rz;
    const float hdot = k.h * fminf(dot, 0.f);
    const float mu = ETA0 ? hdot * rinv * rinv : __fdividef(hdot, r2 + k.eta2h2);
    const float inv_rhoab = rcp_ftz(a.hrhoi + pj.w);
    const float piab = mu * fmaf(k.beta, mu, -(a.haci + hacj)) * inv_rhoab;
    const float t = -mj * ((a.pri + vj.w) + piab);
    // (2 - q) clamped at 0: the outer branch is 0 beyond q = 2
    const float tq = fmaxf(2.f - q, 0.f);
    const float g = q >= 1.f ? k.gout * (tq * tq) * rinv : fmaf(k.gin1, q, k.gin0);
    const float gf = g * t;
    a.pax = fmaf(gf, rx, a.pax);
    a.pay = fmaf(gf, ry, a.pay);
    a.paz = fmaf(gf, rz, a.paz);
    if (XSPH) {
        const float temp = mj * w_of(q, k.wx) * inv_rhoab;
        a.pxx = fmaf(temp, vj.x - a.vi.x, a.pxx);
        a.pxy = fmaf(temp, vj.y - a.vi.y, a.pxy);
        a.pxz = fmaf(temp, vj.z - a.vi.z, a.pxz);
    }
}

template <int S, bool XSPH>
__device__ __forceinline__ void rates_flush(RatesAcc &a, unsigned mask) {
    fold_lanes<S>(a.ax, a.pax, mask); fold_lanes<S>(a.ay, a.pay, mask); fold_lanes<S>(a.az, a.paz, mask);
    a.pax = a.pay = a.paz = 0.f;
    if (XSPH) {
        fold_lanes<S>(a.xx, a.pxx, mask); fold_lanes<S>(a.xy, a.pxy, mask); fold_lanes<S>(a.xz, a.pxz, mask);
        a.pxx = a.pxy = a.pxz = 0.f;
    }
}

// The pairs of one group of 8 list entries, records two at a time, then
// the batch's partial sums folded into the compensated ones.
template <int S, bool XSPH, bool ETA0, bool FAST, bool STAGED, bool TABLE>
__device__ __forceinline__ void rates_group(RatesAcc &acc, const RatesConst &kc,
                                            const SrcRecords<STAGED, TABLE> &R, bool mine, const uint4 &grp,
                                            const float4 &Pi, unsigned mask) {
    if (S == 1 || mine) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            float4 pj[2], vj[2];
            float mj[2], hac[2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
                R.template rates_rec<FAST>(group_entry(grp, 2 * h + i), kc.mb, kc.tkc, pj[i], vj[i],
                                           mj[i], hac[i]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
                rates_pair<XSPH, ETA0>(acc, kc, Pi.x - pj[i].x, Pi.y - pj[i].y, Pi.z - pj[i].z,
                                       pj[i], vj[i], mj[i], hac[i]);
        }
    }
    rates_flush<S, XSPH>(acc, mask);
}

// The sums of a destination, its list streamed as in density_stream.
template <int S, bool XSPH, bool ETA0, bool FAST, bool STAGED, bool TABLE>
__device__ __forceinline__ void rates_stream(RatesAcc &acc, const RatesConst &kc,
                                             const SrcRecords<STAGED, TABLE> &R, const uint4 *lst, int D,
                                             int ng, int lane, const float4 &Pi, uint4 b0, uint4 b1,
                                             unsigned mask) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const int nr = S > 1 ? __reduce_max_sync(mask, ng) : ng;
    const size_t step = (size_t)D;
    uint4 b2;
    for (int g0 = 0, gi = lane;;) {
        if (g0 >= nr) break;
        b2 = gi + 2 * S < ng ? lst[(gi + 2 * S) * step] : zero;
        rates_group<S, XSPH, ETA0, FAST, STAGED, TABLE>(acc, kc, R, gi < ng, b0, Pi, mask);
        gi += S;
        if ((g0 += S) >= nr) break;
        b0 = gi + 2 * S < ng ? lst[(gi + 2 * S) * step] : zero;
        rates_group<S, XSPH, ETA0, FAST, STAGED, TABLE>(acc, kc, R, gi < ng, b1, Pi, mask);
        gi += S;
        if ((g0 += S) >= nr) break;
        b1 = gi + 2 * S < ng ? lst[(gi + 2 * S) * step] : zero;
        rates_group<S, XSPH, ETA0, FAST, STAGED, TABLE>(acc, kc, R, gi < ng, b2, Pi, mask);
        gi += S;
        g0 += S;
    }
}

__device__ __forceinline__ void rates_acc_init(RatesAcc &acc, const float4 &vi, const float4 &st,
                                               float halpha) {
    acc.pax = acc.pay = acc.paz = acc.pxx = acc.pxy = acc.pxz = 0.f;
    acc.vi = vi;
    acc.hrhoi = 0.5f * st.x;
    acc.pri = st.y;
    acc.haci = halpha * st.z;
}

// Store the destination's rates, the six components dealt out to its lanes.
template <int S, bool XSPH>
__device__ __forceinline__ void rates_store(const BrickRatesArgs &A, const RatesAcc &acc, int orig,
                                            int lane) {
    const bool real = is_real(A.d, orig);
    auto put = [&](int k, float sum, float shift, const double *vel, double grav) {
        if (A.acc[k] && (S == 1 || lane == (2 * k) % S)) {
            // the compensated sum rounded once to FP32 (far below the pair
            // terms' own FP32 error), then to FP64 by integer operations
            double v = real ? f2d_exact(sum) : 0.0;
            if (A.add_gravity && real) v += grav;
            A.acc[k][orig] = A.accumulate ? A.acc[k][orig] + v : v;
        }
        if (A.pos[k] && (S == 1 || lane == (2 * k + 1) % S)) {
            double v = 0.0;
            if (real) {
                if (XSPH) v = f2d_exact(shift);
                // exact FP64 velocity of the destination (position_funcs.pyx:47-50)
                if (A.add_velocity) v = XSPH ? v + ld0(vel, orig) : ld0(vel, orig);
            }
            A.pos[k][orig] = A.accumulate ? A.pos[k][orig] + v : v;
        }
    };
    put(0, acc.ax.fvalue(), acc.xx.fvalue(), A.d.u, A.gx);
    put(1, acc.ay.fvalue(), acc.xy.fvalue(), A.d.v, A.gy);
    put(2, acc.az.fvalue(), acc.xz.fvalue(), A.d.w, A.gz);
}

// Destinations with more neighbours than their list holds, as density_rest:
// the rest added to the stored sums.
template <bool XSPH, bool ETA0, bool STAGED, bool TABLE>
__device__ __noinline__ void rates_rest(const BrickRatesArgs &A) {
    const int b = blockIdx.x;
    const int2 dh = A.d.bdst[b];
    const int4 sh = A.s.bsrc[b];
    const Grid &g = A.g;
    const BlockGeo G = block_geo(g, A.bk, b);
    const int2 *brow = A.s.brow + (size_t)b * A.bk.nrmax;
    const StageTab<TABLE> tab = stage_tab<TABLE>(A, sh);
    const float halpha = 0.5f * A.alpha;
    const SrcRecords<STAGED, TABLE> R = make_records<STAGED, TABLE>(A.sm, A.s, g.cs_f, tab, sh.x, halpha);
    const float ih = __fdividef(1.f, g.h_uniform);
    const RatesConst kc = rates_const(g.h_uniform, cubic_fac(A.dim, ih), A.beta, A.eta2, A.eps);
    const int rows = (2 * g.ky + 1) * (2 * g.kz + 1);
    // a two-record block has staged no state records
    if (STAGED) {
        __syncthreads();
        stage_state<TABLE>(A.s, tab, sh.x, A.sm.off_s, halpha);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < dh.x; d += blockDim.x) {
        if (A.cnt[dh.y + d] <= A.cap) continue;
        const BrickDest q = brick_dest(A.d, G, g.cs_f, A.d.bdest[dh.y + d]);
        if (!is_real(A.d, q.orig)) continue;
        RatesAcc acc;
        rates_acc_init(acc, A.d.velh[q.s], A.d.st[q.s], halpha);
        int skip = A.cap;
        brick_traverse<STAGED, TABLE>(g, G, A.s, A.d, R, A.rad, brow, tab, nullptr, q, 0, rows,
            [&](int t0, unsigned m) {
                for (; m; m &= m - 1) {
                    if (skip > 0) { --skip; continue; }
                    float4 pj, vj;
                    float mj, hac;
                    R.template rates_rec<false>(t0 + __ffs(m) - 1, 0.f, 0.f, pj, vj, mj, hac);
                    rates_pair<XSPH, ETA0>(acc, kc, q.P.x - pj.x, q.P.y - pj.y, q.P.z - pj.z, pj, vj,
                                           mj, hac);
                    rates_flush<1, XSPH>(acc, 0u);
                }
            });
        const double a3[3] = {(double)acc.ax.fvalue(), (double)acc.ay.fvalue(),
                              (double)acc.az.fvalue()};
        const double p3[3] = {(double)acc.xx.fvalue(), (double)acc.xy.fvalue(),
                              (double)acc.xz.fvalue()};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (A.acc[k]) A.acc[k][q.orig] += a3[k];
            if (A.pos[k]) A.pos[k][q.orig] += p3[k];
        }
    }
}

// The rates of a destination (its prefetched records p, velocity, state).
template <int S, bool XSPH, bool ETA0, bool FAST, bool STAGED, bool TABLE>
__device__ __forceinline__ void rates_dest(const BrickRatesArgs &A, const SrcRecords<STAGED, TABLE> &R,
                                           float mb, const uint4 *lst, int D, int lane,
                                           const DestPre &p, const float4 &vi, const float4 &st,
                                           unsigned mask) {
    const float ih = __fdividef(1.f, A.g.h_uniform);
    RatesConst kc = rates_const(A.g.h_uniform, cubic_fac(A.dim, ih), A.beta, A.eta2, A.eps);
    kc.mb = mb;
    kc.tkc = A.tait_kc;
    RatesAcc acc;
    rates_acc_init(acc, vi, st, 0.5f * A.alpha);
    rates_stream<S, XSPH, ETA0, FAST, STAGED, TABLE>(acc, kc, R, lst, D, (min(p.c, A.cap) + 7) >> 3, lane,
                                              p.P, p.b0, p.b1, mask);
    rates_store<S, XSPH>(A, acc, p.orig, lane);
}

// Destinations past one per column of the block, as density_more.
template <bool XSPH, bool ETA0, bool FAST, bool STAGED, bool TABLE>
__device__ __noinline__ void rates_more(const BrickRatesArgs &A, float mb, int first) {
    constexpr int S = 4;
    const int b = blockIdx.x;
    const int2 dh = A.d.bdst[b];
    const int4 sh = A.s.bsrc[b];
    const SrcRecords<STAGED, TABLE> R = make_records<STAGED, TABLE>(A.sm, A.s, A.g.cs_f, stage_tab<TABLE>(A, sh), sh.x,
                                                      0.5f * A.alpha);
    const uint4 *lgrp = reinterpret_cast<const uint4 *>(A.nbr) + (size_t)dh.y * (A.cap >> 3);
    const int lane = threadIdx.x % S, nt = blockDim.x;
    int r0 = first;
    for (; dh.x - r0 > nt / 4; r0 += nt) {
        const int d = r0 + threadIdx.x;
        if (d >= dh.x) continue;
        DestPre p;
        dest_prefetch<1>(A.d, A.g.cs_f, A.d.bdest[dh.y + d], A.cnt + dh.y, lgrp, A.cap, dh.x, d, 0,
                         p);
        rates_dest<1, XSPH, ETA0, FAST, STAGED, TABLE>(A, R, mb, lgrp + d, dh.x, 0, p,
                                                       A.d.velh[p.s], A.d.st[p.s], 0xffffffffu);
    }
    for (; r0 < dh.x; r0 += nt / S) {
        const int d = r0 + threadIdx.x / S;
        const unsigned mask = __ballot_sync(0xffffffffu, d < dh.x);
        if (d >= dh.x) continue;
        DestPre p;
        dest_prefetch<S>(A.d, A.g.cs_f, A.d.bdest[dh.y + d], A.cnt + dh.y, lgrp, A.cap, dh.x, d,
                         lane, p);
        rates_dest<S, XSPH, ETA0, FAST, STAGED, TABLE>(A, R, mb, lgrp + d, dh.x, lane, p, A.d.velh[p.s],
                                                A.d.st[p.s], mask);
    }
}

template <int S, bool XSPH, bool ETA0, bool FAST, bool STAGED, bool TABLE>
__device__ __forceinline__ void rates_block(const BrickRatesArgs &A, const SrcRecords<STAGED, TABLE> &R,
                                            float mb, const uint4 *lgrp, int D, int d, int lane,
                                            const DestPre &pre, const float4 &vi, const float4 &st) {
    const unsigned mask = S > 1 ? __ballot_sync(0xffffffffu, d < D) : 0xffffffffu;
    if (d < D)
        rates_dest<S, XSPH, ETA0, FAST, STAGED, TABLE>(A, R, mb, lgrp + d, D, lane, pre, vi, st, mask);
    if (D > (int)blockDim.x / S) rates_more<XSPH, ETA0, FAST, STAGED, TABLE>(A, mb, blockDim.x / S);
    if (*A.maxcnt > A.cap) rates_rest<XSPH, ETA0, STAGED, TABLE>(A);
}

template <int S, bool XSPH, bool STAGED, bool TABLE>
__global__ void __maxnreg__(XSPH ? 80 : 64) k_brates(const __grid_constant__ BrickRatesArgs A) {
    const int b = blockIdx.x;
    const int2 dh = A.d.bdst[b];        // destinations, first destination
    const int4 sh = A.s.bsrc[b];        // staged records, their table, the first's slot
    if (dh.x == 0) return;
    const unsigned off = A.gate != nullptr ? *A.gate : 0u;   // tested after the staging
    const int T = sh.x, D = dh.x;
    const StageTab<TABLE> tab = stage_tab<TABLE>(A, sh);
    const uint4 *lgrp = reinterpret_cast<const uint4 *>(A.nbr) + (size_t)dh.y * (A.cap >> 3);
    const int lane = threadIdx.x % S, d = threadIdx.x / S;
    DestPre pre;
    float4 vi = pad_vel(), st = pad_vel();
    if (d < D) {
        dest_prefetch<S>(A.d, A.g.cs_f, A.d.bdest[dh.y + d], A.cnt + dh.y, lgrp, A.cap, D, d, lane,
                         pre);
        vi = A.d.velh[pre.s];
        st = A.d.st[pre.s];
    }
    const float halpha = 0.5f * A.alpha;
    // two-record blocks: staged sources of one mass (that of the first) whose
    // cs follows Tait
    const bool try_fast = STAGED && A.tait_state != 0 && A.eta2 == 0.f && T > 0;
    const float mref = try_fast ? A.s.pm[sh.z].w : 0.f;
    bool same = true;
    if (STAGED) same = stage<true, TABLE>(A.s, tab, T, A.g.cs_f, A.sm, !try_fast, halpha, mref);
    const bool fast = __syncthreads_and(try_fast && same) != 0;
    if (STAGED && try_fast && !fast) {
        stage_state<TABLE>(A.s, tab, T, A.sm.off_s, halpha);
        __syncthreads();
    }
    if (off != 0u) return;
    const SrcRecords<STAGED, TABLE> R = make_records<STAGED, TABLE>(A.sm, A.s, A.g.cs_f, tab, T, halpha);
    if (A.eta2 == 0.f) {
        if constexpr (STAGED) {
            if (fast) {
                rates_block<S, XSPH, true, true, STAGED, TABLE>(A, R, mref, lgrp, D, d, lane, pre, vi, st);
                return;
            }
        }
        rates_block<S, XSPH, true, false, STAGED, TABLE>(A, R, 0.f, lgrp, D, d, lane, pre, vi, st);
    } else {
        rates_block<S, XSPH, false, false, STAGED, TABLE>(A, R, 0.f, lgrp, D, d, lane, pre, vi, st);
    }
}

// ---------------------------------------------------------------------------
// tables of the blocks of one array (ArraySnap): first, a warp per block, the
// staged rows, the counts, and the places of its entries (one atomic per
// table; they differ from build to build, the results do not depend on
// them) and the list of the blocks that have any, then, the tables allocated,
// the entries of those, four warps per block (42 us
// at 1 M particles, once per full build; a warp per block took 20 us more at
// 275 000)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int warp_scan(int v) {     // inclusive
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// first slot and length of destination row r of a block (0 past the last)
__device__ __forceinline__ int dest_row(const Grid &g, const BlockGeo &G, const int *cstart, int r,
                                        int &lo) {
    const int dry = G.y1 - G.y0, ndr = dry * (G.z1 - G.z0);
    lo = 0;
    if (r >= ndr) return 0;
    const int c = ((G.z0 + r / dry) * g.ny + G.y0 + r % dry) * g.nx;
    lo = cstart[c + G.x0];
    return cstart[c + G.x1] - lo;
}

__global__ void __launch_bounds__(128) k_brick_count(Grid g, BrickGeom bk, const int *cstart,
                                                     int4 *bsrc, int2 *brow, int2 *bdst,
                                                     int *blist, unsigned *stats) {
    const int lane = threadIdx.x & 31;
    const int64_t b = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= bk.nbricks) return;
    const BlockGeo G = block_geo(g, bk, (int)b);
    // an empty block (most of the box of a splash) keeps no rows, and rows before
    // the first that has anything are zeros: the starts of an empty row's cells
    // are all the same, so a row of any first slot has nothing in it
    int2 *rows = brow + b * bk.nrmax;
    int T = 0, D = 0, first = 0, lo;
    for (int r0 = 0; r0 < G.nr; r0 += 32) {
        const int r = r0 + lane;
        int len = 0;
        lo = 0;
        if (r < G.nr) {
            const int c = ((G.zs0 + r / G.ry) * g.ny + G.ys0 + r % G.ry) * g.nx + G.xs0;
            lo = cstart[c];
            len = cstart[c + G.lx] - lo;
        }
        const unsigned some = __ballot_sync(0xffffffffu, len > 0);
        if (T == 0) {
            if (!some) continue;
            first = __shfl_sync(0xffffffffu, lo, __ffs(some) - 1);
            for (int q = lane; q < r0; q += 32) rows[q] = make_int2(0, 0);
        }
        const int inc = warp_scan(len);
        if (r < G.nr) rows[r] = make_int2(lo, (int)((unsigned)(T + inc - len) | ((unsigned)len << 16)));
        T += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (T == 0) {
        if (lane == 0) {
            bsrc[b] = make_int4(0, 0, 0, 0);
            bdst[b] = make_int2(0, 0);
        }
        return;
    }
    const int ndr = (G.y1 - G.y0) * (G.z1 - G.z0);
    for (int r0 = 0; r0 < ndr; r0 += 32)
        D += __reduce_add_sync(0xffffffffu, dest_row(g, G, cstart, r0 + lane, lo));
    if (lane == 0) {
        // every block: as a source this array is staged by the blocks that
        // hold destinations of any array
        const int tb = (int)atomicAdd(reinterpret_cast<unsigned long long *>(stats + 4),
                                      (unsigned long long)T);
        const int db = D > 0 ? (int)atomicAdd(stats + 2, (unsigned)D) : 0;
        atomicMax(stats, (unsigned)T);
        atomicMax(stats + 1, (unsigned)D);
        bsrc[b] = make_int4(T, tb, first, 0);
        bdst[b] = make_int2(D, db);
        blist[atomicAdd(stats + 3, 1u)] = (int)b;
    }
}

// blist null: every block; bstage null: the destinations only (brick_fill)
__global__ void __launch_bounds__(128) k_brick_fill(Grid g, BrickGeom bk, const int *cstart,
                                                    const float *scx, const int *blist,
                                                    const int4 *bsrc,
                                                    const int2 *brow, const int2 *bdst,
                                                    int2 *bstage, int2 *bdest) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int b = blist != nullptr ? blist[blockIdx.x] : blockIdx.x;
    const int D = bdst[b].x;
    const BlockGeo G = block_geo(g, bk, b);
    const int2 *rows = brow + (int64_t)b * bk.nrmax;
    int2 *stab = bstage + bsrc[b].y;
    const int nr = bstage != nullptr ? G.nr : 0;
    // a warp takes a row of cells at a time, its slots over the lanes
#pragma unroll 4
    for (int r = wid; r < nr; r += nw) {
        const int2 e = rows[r];
        const int c = pack_cell(-128, G.ys0 + r % G.ry - G.cyc, G.zs0 + r / G.ry - G.czc) -
                      G.cxc + 128;
        for (int i = lane; i < row_len(e); i += 32)
            stab[row_off(e) + i] = make_int2(e.x + i, c + (int)scx[e.x + i]);
    }
    if (D == 0) return;
    const int dry = G.y1 - G.y0, ndr = dry * (G.z1 - G.z0);
    int2 *dtab = bdest + bdst[b].y;
    for (int r0 = 0; r0 < ndr; r0 += 32) {
        int lo;
        const int len = dest_row(g, G, cstart, r0 + lane, lo);
        const int inc = warp_scan(len);
        const int cnt = min(32, ndr - r0);
        for (int k = wid; k < cnt; k += nw) {
            const int l = __shfl_sync(0xffffffffu, lo, k), n = __shfl_sync(0xffffffffu, len, k);
            const int at = __shfl_sync(0xffffffffu, inc - len, k);
            const int cy = G.y0 + (r0 + k) % dry - G.cyc, cz = G.z0 + (r0 + k) / dry - G.czc;
            for (int i = lane; i < n; i += 32)
                dtab[at + i] = make_int2(l + i, pack_cell((int)scx[l + i] - G.cxc, cy, cz));
        }
        dtab += __shfl_sync(0xffffffffu, inc, 31);
    }
}

// the largest source staging of any brick over every source array, as the
// staged-record capacity, if it fits the shared memory of a block
constexpr int kBrickSmemLimit = 200 * 1024;

// Shared-memory layout of a pass over the sources S.
int brick_layout(const sph_ctx *ctx, const ArraySnap &S, bool rates, bool cells, BrickSmem *sm,
                 size_t *bytes) {
    const BrickGeom &bk = ctx->bricks;
    const size_t ncell = cells ? (size_t)bk.nrmax * (bk.rowmax + 1) : 0;
    const size_t rec = rates ? (16 + 16 + 8) : 16;
    // the staged records and the padding record after them
    size_t cap = (size_t)std::max(S.b_tmax, 0) + 1;
    // environment SPH_BRICK_UNSTAGED=1 reads every record from global memory
    // (the path of bricks too populous for shared memory), to test it on
    // small sets
    static int unstaged = -1;
    if (unstaged < 0) {
        const char *e = getenv("SPH_BRICK_UNSTAGED");
        unstaged = (e && atoi(e) > 0) ? 1 : 0;
    }
    const bool staged = !unstaged && sizeof(int) * ncell + cap * rec + kSlack * 16 + 64 <=
                                         (size_t)kBrickSmemLimit;
    if (!staged) cap = 0;
    size_t off = 0;
    // position records, then (rates) velocity and state records
    off += staged ? (cap + kSlack) * 16 : 0;
    sm->off_v = (int)off;
    if (rates) off += cap * 16;
    sm->off_s = (int)off;
    if (rates) off += cap * 8;
    off = (off + 15) & ~(size_t)15;
    sm->off_scell = (int)off; off += sizeof(int) * ncell;
    *bytes = off;
    return staged ? 1 : 0;
}

BrickRadius brick_radius(const sph_ctx *ctx) {
    const Grid &g = ctx->grid;
    BrickRadius r;
    const double radius = ctx->build_h * g.radius_scale;
    r.radius2 = radius * radius;
    const float r2 = (float)r.radius2;
    r.r2lo = r2 * (1.f - 1e-5f);
    r.r2hi = r2 * (1.f + 1e-5f);
    r.r2list = 0.f;
    if (g.skin > 0.f) {
        const float rl = (float)radius + g.skin;
        r.r2list = rl * rl * (1.f + 2e-5f);
    }
    return r;
}

BrickSrcDev make_bsrc(const ArraySnap &S) {
    BrickSrcDev s;
    s.pm = S.pm; s.velh = S.velh; s.st = S.st; s.scx = S.scx;
    s.cstart = S.cstart; s.perm = S.perm;
    s.bsrc = S.bsrc; s.brow = S.brow; s.bstage = S.bstage;
    s.x = S.view.x; s.y = S.view.y; s.z = S.view.z;
    return s;
}

BrickDstDev make_bdst(const ArraySnap &D) {
    BrickDstDev d;
    d.pm = D.pm; d.velh = D.velh; d.st = D.st;
    d.perm = D.perm; d.bdst = D.bdst; d.bdest = D.bdest;
    d.tag = D.view.tag;
    d.x = D.view.x; d.y = D.view.y; d.z = D.view.z;
    d.u = D.view.u; d.v = D.view.v; d.w = D.view.w;
    d.p = D.view.p; d.cs = D.view.cs;
    return d;
}

// Threads per block: the columns (destinations times lanes) of the most
// populous block rounded to warps, at most 320 with one lane (three blocks of
// 64-register threads per SM) and 512 with more; a block with more columns
// takes them in rounds.
int brick_threads(const ArraySnap &D, int lanes) {
    // environment SPH_BRICK_MAX_THREADS: another ceiling (a multiple of 32
    // up to 512), to measure it
    static int ceiling = -1;
    if (ceiling < 0) {
        const char *e = getenv("SPH_BRICK_MAX_THREADS");
        const int v = e ? atoi(e) : 0;
        ceiling = (v >= 64 && v <= kBrickMaxThreads && v % 32 == 0) ? v : 0;
    }
    const int top = ceiling > 0 ? ceiling : (lanes == 1 ? 320 : kBrickMaxThreads);
    const int want = (std::max(D.b_dmax, 1) * lanes + 31) / 32 * 32;
    return std::min(std::max(want, 64), top);
}

template <class Kern>
int allow_smem(Kern *k, size_t bytes) {
    // raise each kernel's dynamic shared-memory limit to the largest layout,
    // once per kernel and device
    static std::mutex mu;
    static std::vector<std::pair<const void *, int>> done;
    if (bytes <= 48 * 1024) return SPH_OK;
    int dev = 0;
    SPH_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    for (const auto &d : done)
        if (d.first == (const void *)k && d.second == dev) return SPH_OK;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kBrickSmemLimit);
    if (e != cudaSuccess) return cuda_check(e, "cudaFuncSetAttribute (brick shared memory)");
    done.emplace_back((const void *)k, dev);
    return SPH_OK;
}

}  // namespace

// Most blocks of a box whose destinations get several lanes.  A small set that
// fills its box has fewer (686 of 39 304 particles in 3D); one with a few
// particles far off has more, nearly all empty, and each part of a brick is a
// block to launch.  Step in us with lanes / one lane: 2D, 5 025 particles, four
// lanes, 434 bricks 75.3 / 75.9, 967 79.7 / 78.3, 2 664 95.1 / 81.6, 43 000 444 /
// 157; 3D, four lanes, 4 096 particles 567 bricks 102 / 107, 2 352 126 / 112,
// 8 000 particles 1 049 bricks 112 / 116, 2 352 132 / 137, 4 440 159 / 138; two
// lanes, 21 952 particles 2 701 bricks 129 / 139, 6 147 157 / 159, 11 713 190 /
// 166.
constexpr int64_t kLaneBlocks2 = 152 * 16, kLaneBlocks3 = 152 * 40;

// Brick geometry of the current grid: edge lengths (cells) per stencil
// half-width, chosen so a brick holds a few hundred destinations and its
// staging ~5-8 times as many sources.
void brick_geometry(sph_ctx *ctx) {
    const Grid &g = ctx->grid;
    BrickGeom &bk = ctx->bricks;
    const int K = g.kx;
    // environment SPH_BRICK_EDGE: the brick edge in cells (3D), to measure
    // other brick sizes
    static int edge = -1;
    // environment SPH_BRICK_SHAPE=bx,by,bz: a 3D brick shape, to measure it
    static int shape[3] = {0, 0, 0};
    if (edge < 0) {
        const char *e = getenv("SPH_BRICK_EDGE");
        edge = e ? std::max(1, atoi(e)) : 0;
        const char *sh = getenv("SPH_BRICK_SHAPE");
        int a = 0, b = 0, c = 0;
        if (sh && sscanf(sh, "%d,%d,%d", &a, &b, &c) == 3 && a > 0 && b > 0 && c > 0 && a <= 16 &&
            b <= 16 && c <= 16) {
            shape[0] = a; shape[1] = b; shape[2] = c;
        }
    }
    if (g.kz > 0) {
        const int e = edge > 0 ? edge : (K == 1 ? 3 : (K == 2 ? 5 : 8));
        bk.bx = bk.by = bk.bz = e;
        // stencil half-width 2: 6 x 5 x 5 cells (1 M-particle lattice, rates
        // pass 0.276 ms against 0.283 ms with 5^3 cells)
        if (K == 2 && edge <= 0) bk.bx = 6;
        if (shape[0] > 0) {
            bk.bx = shape[0]; bk.by = shape[1]; bk.bz = shape[2];
        }
    } else if (g.ky > 0) {
        const int e = K == 1 ? 8 : (K == 2 ? 12 : 16);
        bk.bx = bk.by = e;
        bk.bz = 1;
    } else {
        bk.bx = 64;
        bk.by = bk.bz = 1;
    }
    // Lanes per destination and parts of a brick: a small simulation has fewer
    // bricks than there are SMs and each thread a long chain, so its
    // destinations get 2 or 4 lanes and its bricks as many parts; a larger one
    // pays for the parts' wider staging and the second traversal of a list
    // build.  Measured, rates + density in us at 1 / 2 / 4 lanes -- 3D: 4 096
    // particles 26.3 / 22.4 / 19.1, 8 000 28.9 / 23.8 / 22.3, 21 952 29.0 /
    // 26.6 / 35.6, 64 000 50.3 / 49.6 / 68.2; 2D: 5 025 18.2 / 17.8 / 15.9,
    // 10 300 17.8 / 16.9 / 15.6, 20 106 17.9 / 18.4 / 22.4.  In 1D, whose lists are
    // short, two: RK2 step of 4 000 with h / dx 2 77 / 77 / 92, with 3 93 / 80 /
    // 94, with 6 119 / 104 / 104.  Environment SPH_BRICK_LANES forces the lanes (to
    // measure them, and to test them at any size).
    static int force_lanes = -1;
    if (force_lanes < 0) {
        const char *l = getenv("SPH_BRICK_LANES");
        const int v = l ? atoi(l) : 0;
        force_lanes = (v == 1 || v == 2 || v == 4) ? v : 0;
    }
    int64_t n = 0;
    for (const ArraySnap &A : ctx->arrays) n = std::max(n, A.n);
    bk.lanes = force_lanes ? force_lanes
                           : (n < 12000 ? (g.ky > 0 || g.kz > 0 ? 4 : 2) : (g.kz > 0 && n < 40000 ? 2 : 1));
    const int64_t whole = (int64_t)((g.nx + bk.bx - 1) / bk.bx) * ((g.ny + bk.by - 1) / bk.by) *
                          ((g.nz + bk.bz - 1) / bk.bz);
    if (!force_lanes && whole * bk.lanes > (g.kz > 0 ? kLaneBlocks3 : kLaneBlocks2)) bk.lanes = 1;
    bk.px = bk.lanes > 1 && bk.bx > 1 ? 2 : 1;
    bk.py = bk.lanes > 2 && bk.by > 1 ? 2 : 1;
    bk.pz = 1;
    bk.nbx = (g.nx + bk.bx - 1) / bk.bx * bk.px;
    bk.nby = (g.ny + bk.by - 1) / bk.by * bk.py;
    bk.nbz = (g.nz + bk.bz - 1) / bk.bz * bk.pz;
    const int sx = (bk.bx + bk.px - 1) / bk.px, sy = (bk.by + bk.py - 1) / bk.py,
              sz = (bk.bz + bk.pz - 1) / bk.pz;
    bk.nrmax = (sy + 2 * g.ky) * (sz + 2 * g.kz);
    bk.rowmax = sx + 2 * g.kx;
    bk.nbricks = (int64_t)bk.nbx * bk.nby * bk.nbz;
}

// Per-array brick tables for the current build (queued on the context's
// stream): the counts, whose statistics land in stats[0 .. kBrickStats), then,
// when those are known on the host, the entries.
int brick_count(sph_ctx *ctx, int a, unsigned *stats) {
    ArraySnap &A = ctx->arrays[a];
    const BrickGeom &bk = ctx->bricks;
    // one allocation for the four tables (a new simulation's first step pays for
    // each), the widest entries first
    const int64_t nb = bk.nbricks, nrow = nb * bk.nrmax;
    const int64_t bytes = nb * (int64_t)(sizeof(int4) + sizeof(int2) + sizeof(int)) +
                          nrow * (int64_t)sizeof(int2);
    if (bytes > A.bcount_cap || !A.bsrc) {
        cudaFree(A.bsrc);
        A.bsrc = nullptr;
        A.bcount_cap = 0;
        SPH_CUDA(cudaMalloc((void **)&A.bsrc, bytes));
        A.bcount_cap = bytes;
    }
    A.bdst = reinterpret_cast<int2 *>(A.bsrc + nb);
    A.brow = A.bdst + nb;
    A.blist = reinterpret_cast<int *>(A.brow + nrow);
    const int th = 128, per = th / 32;
    const int blocks = (int)((bk.nbricks + per - 1) / per);
    k_brick_count<<<blocks, th, 0, ctx->stream>>>(ctx->grid, bk, A.cstart, A.bsrc, A.brow, A.bdst,
                                                  A.blist, stats);
    count_launch();
    SPH_LAUNCH_CHECK("k_brick_count");
    return SPH_OK;
}

// The destinations are filled for every array: a pass over another, sparser
// source takes this array's blocks however populous they are.  The table of
// staged entries (bstage, some five entries per particle in 3D) is for arrays
// that a block can stage (the fields of brow hold 16 bits each), with fewer
// than 2^31 entries (32-bit indices) and where there is memory for it; without
// it the passes find the entries from the rows (environment
// SPH_BRICK_STAGE_TABLE=0: always, to test that on small sets).  That costs
// time only: RK2 step of 1 M particles 915 -> 1126 us, of 64 000 157 -> 180.
int brick_fill(sph_ctx *ctx, int a) {
    ArraySnap &A = ctx->arrays[a];
    const BrickGeom &bk = ctx->bricks;
    static int wanted = -1;
    if (wanted < 0) {
        const char *e = getenv("SPH_BRICK_STAGE_TABLE");
        wanted = (e && atoi(e) == 0) ? 0 : 1;
    }
    // (one allocation, the destinations first)
    A.b_table = wanted && A.b_tmax < 65535 && A.b_staged < INT32_MAX;
    const int64_t least = A.n, exact = A.n + A.b_staged;
    if ((A.b_table ? exact : least) > A.bfill_cap || !A.bdest) {
        cudaFree(A.bdest);
        A.bdest = nullptr;
        A.bfill_cap = 0;
        // (an eighth more of the staged entries, for the next builds)
        for (const int64_t want : {exact + A.b_staged / 8, exact}) {
            if (!A.b_table || A.bdest) break;
            if (cudaMalloc((void **)&A.bdest, sizeof(int2) * want) == cudaSuccess) {
                A.bfill_cap = want;
            } else {
                A.bdest = nullptr;
                cudaGetLastError();     // (not the build's error)
            }
        }
        if (!A.bdest) {
            A.b_table = false;
            SPH_CUDA(cudaMalloc((void **)&A.bdest, sizeof(int2) * least));
            A.bfill_cap = least;
        }
    }
    A.bstage = A.b_table ? A.bdest + A.n : nullptr;
    k_brick_fill<<<(unsigned)A.b_blocks, 128, 0, ctx->stream>>>(
        ctx->grid, bk, A.cstart, A.scx, A.b_blocks < bk.nbricks ? A.blist : nullptr, A.bsrc, A.brow,
        A.bdst, A.bstage, A.bdest);
    count_launch();
    SPH_LAUNCH_CHECK("k_brick_fill");
    return SPH_OK;
}

bool brick_density_eligible(const sph_ctx *ctx, int dst, const int *srcs, int nsrc,
                            const sph_density_params *prm) {
    const Grid &g = ctx->grid;
    if (!ctx->bricks_on || !ctx->bricks_ready || nsrc != 1 || !g.uniform_h || g.periodic ||
        g.symmetric || prm->h0 != 0.0)
        return false;
    const ArraySnap &S = ctx->arrays[srcs[0]];
    const ArraySnap &D = ctx->arrays[dst];
    return S.n > 0 && D.n > 0 && S.b_tmax < 65535;
}

bool brick_rates_eligible(const sph_ctx *ctx, int dst, const sph_source_term *terms, int nterms,
                          const sph_rates_params *prm) {
    const Grid &g = ctx->grid;
    if (!ctx->bricks_on || !ctx->bricks_ready || nterms != 1 || !g.uniform_h || g.periodic ||
        g.symmetric || prm->drho_out != nullptr)
        return false;
    const uint32_t f = terms[0].flags;
    if (f != (SPH_TERM_PGRAD | SPH_TERM_AVISC) && f != (SPH_TERM_PGRAD | SPH_TERM_AVISC | SPH_TERM_XSPH))
        return false;
    const ArraySnap &S = ctx->arrays[terms[0].src];
    const ArraySnap &D = ctx->arrays[dst];
    return S.n > 0 && D.n > 0 && S.b_tmax < 65535;
}

// Density pass (and, with build, the list build) of destination dst among
// source src; write_out = 0 builds the list only.
int brick_density(sph_ctx *ctx, int dst, int src, NbrList &L, bool build, bool write_out,
                  const sph_density_params *prm, double *rho, double *p, double *cs,
                  float4 *st_out) {
    ArraySnap &D = ctx->arrays[dst];
    ArraySnap &S = ctx->arrays[src];
    BrickDensityArgs a{};
    a.g = ctx->grid;
    a.bk = ctx->bricks;
    a.rad = brick_radius(ctx);
    a.d = make_bdst(D);
    a.s = make_bsrc(S);
    size_t bytes = 0;
    const bool staged = brick_layout(ctx, S, false, build, &a.sm, &bytes) != 0;
    a.nbr = L.nbr16;
    a.cnt = L.cnt;
    a.maxcnt = L.maxcnt;
    a.cap = L.cap;
    a.write_out = write_out ? 1 : 0;
    if (prm) {
        a.dim = prm->dim;
        a.tait = prm->tait;
        a.co = (float)prm->co; a.ro = (float)prm->ro; a.gamma = (float)prm->gamma;
    } else {
        a.dim = ctx->dim;
    }
    a.rho_out = rho; a.p_out = p; a.cs_out = cs;
    a.st_out = st_out;
    a.gate = ctx->gate;
    if (D.n == 0) return SPH_OK;
    // (without a table of entries: one lane, whatever the parts)
    const int lanes = S.b_table ? ctx->bricks.lanes : 1;
    const int nt = brick_threads(D, lanes);
    const int blocks = (int)ctx->bricks.nbricks;
#define BDL2(K_, L_, S_, T_)                                                              \
    do {                                                                                  \
        int rc_ = allow_smem(K_<L_, S_, T_>, bytes);                                      \
        if (rc_) return rc_;                                                              \
        K_<L_, S_, T_><<<blocks, nt, bytes, ctx->stream>>>(a);                            \
    } while (0)
#define BDL1(K_, L_, T_)                                                                  \
    do { if (staged) BDL2(K_, L_, true, T_); else BDL2(K_, L_, false, T_); } while (0)
#define BDL(L_, T_)                                                                       \
    do { if (build) BDL1(k_bbuild, L_, T_); else BDL1(k_bdensity, L_, T_); } while (0)
    if (!S.b_table) BDL(1, false);
    else if (lanes == 1) BDL(1, true);
    else if (lanes == 2) BDL(2, true);
    else BDL(4, true);
#undef BDL
#undef BDL1
#undef BDL2
    count_launch();
    SPH_LAUNCH_CHECK("k_bdensity");
    return SPH_OK;
}

int brick_rates(sph_ctx *ctx, int dst, const sph_source_term &term, NbrList &L,
                const sph_rates_params *prm, double *const *acc, double *const *pos,
                int accumulate) {
    ArraySnap &D = ctx->arrays[dst];
    ArraySnap &S = ctx->arrays[term.src];
    BrickRatesArgs a{};
    a.g = ctx->grid;
    a.bk = ctx->bricks;
    a.rad = brick_radius(ctx);
    a.d = make_bdst(D);
    a.s = make_bsrc(S);
    size_t bytes = 0;
    const bool staged = brick_layout(ctx, S, true, false, &a.sm, &bytes) != 0;
    a.nbr = L.nbr16;
    a.cnt = L.cnt;
    a.maxcnt = L.maxcnt;
    a.cap = L.cap;
    a.dim = prm->dim;
    a.alpha = (float)term.alpha;
    a.beta = (float)term.beta;
    a.eta2 = (float)(term.eta * term.eta);
    a.eps = (float)term.eps;
    a.add_velocity = prm->add_velocity;
    a.add_gravity = prm->add_gravity;
    a.accumulate = accumulate;
    // alpha cs / 2 = (alpha / 2) f (2 (rho / 2))^3 with cs = f rho^3; the
    // environment setting SPH_BRICK_TWO_RECORDS=0 keeps three records
    static int two = -1;
    if (two < 0) {
        const char *e = getenv("SPH_BRICK_TWO_RECORDS");
        two = (e && atoi(e) == 0) ? 0 : 1;
    }
    a.tait_state = two && S.st_tait_f > 0.0 ? 1 : 0;
    a.tait_kc = (float)(4.0 * term.alpha * S.st_tait_f);
    a.gx = prm->gx; a.gy = prm->gy; a.gz = prm->gz;
    for (int c = 0; c < 3; ++c) {
        a.acc[c] = acc ? acc[c] : nullptr;
        a.pos[c] = pos ? pos[c] : nullptr;
    }
    a.gate = ctx->gate;
    if (D.n == 0) return SPH_OK;
    const bool xsph = (term.flags & SPH_TERM_XSPH) != 0;
    // (without a table of entries: one lane, whatever the parts)
    const int lanes = S.b_table ? ctx->bricks.lanes : 1;
    const int nt = brick_threads(D, lanes);
    const int blocks = (int)ctx->bricks.nbricks;
#define BRL3(L_, X_, S_, T_)                                                              \
    do {                                                                                  \
        int rc_ = allow_smem(k_brates<L_, X_, S_, T_>, bytes);                            \
        if (rc_) return rc_;                                                              \
        k_brates<L_, X_, S_, T_><<<blocks, nt, bytes, ctx->stream>>>(a);                  \
    } while (0)
#define BRL2(L_, X_, T_)                                                                  \
    do { if (staged) BRL3(L_, X_, true, T_); else BRL3(L_, X_, false, T_); } while (0)
#define BRL(L_, T_)                                                                       \
    do { if (xsph) BRL2(L_, true, T_); else BRL2(L_, false, T_); } while (0)
    if (!S.b_table) BRL(1, false);
    else if (lanes == 1) BRL(1, true);
    else if (lanes == 2) BRL(2, true);
    else BRL(4, true);
#undef BRL
#undef BRL2
#undef BRL3
    count_launch();
    SPH_LAUNCH_CHECK("k_brates");
    return SPH_OK;
}

}  // namespace sphgb
