// rc_device.cuh -- sm_100a device code of the OERM Monte Carlo solver.
//
// Reference: src/montecarlo/mc_gpu_noint.cu
//   kernel_fluid   :55-243   per-cell bundle emission + OERM tally
//   march_ray      :245-658  multigrid ray march with the wall conditions
//   find_band(S)   :1103-1233 band / g-point bisection
//   emiss_ang(S)   :1077-1102 emission directions
//   kernel_surface :1316-1482 wall-flux kernel
//   kernel_results :1296-1314 copy-out
//
// Arithmetic contract (shared with the CPU oracle, which restates the same
// operations in the same order so that sampled bands, g points, visited
// cells and per-bundle tallies agree bit for bit):
//   * no automatic FMA contraction (nvcc -fmad=false, g++ -ffp-contract=off);
//     every fused multiply-add is written out (fma_ here, the same call in
//     the oracle, fmaf() in radchan_math.h), so both sides round alike;
//   * face distance ds = (face - p) * (1/s), the reciprocal formed once per
//     direction change; positions p = fma(ds, s, p) on the axes not crossed;
//   * table coordinate q = rint(256 * clamp((T - T0) * (1/dT), 0, nT-1)),
//     8 fractional bits (the weight precision of the texture unit the
//     reference interpolates with), stored as uint16 per cell of every
//     multigrid level; v = fma(col[i1], a, col[i0]*(1-a)) (rc_lerpf) with
//     i0 = q >> 8, i1 = min(i0 + 1, nT - 1), a = (q & 255) / 256;
//   * em = expm1(-(ds*k)), alpha = -em, tra = fma(tra, em, tra);
//   * step tally c = (((Ibmax*tra)*alpha)*ratioI)*fma(invTi4, Ib, -1) in the
//     march precision, accumulated into an FP64 bundle sum;
//   * per-bundle sums are added in bundle order within a chunk of
//     rays_per_thread bundles, chunk sums in chunk order, and replicate
//     sums in replicate order, whatever thread traced which bundle.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "radchan.h"
#include "radchan_math.h"

namespace rc {

constexpr int kWarp = 32;
constexpr int kRefill = 11;  // emitted bundles waiting below which a warp emits the next wave
constexpr int kRing = kRefill - 1 + kWarp;  // per-warp ring of emitted bundles: those, and a wave
constexpr int kTileBufs = 3;  // tiles a warp has in flight (tile_bufs): 2 -> 3 30% faster on 192x128x128, 4 slower on small grids (L1)
constexpr int kGuide = 1024; // buckets of the band-CDF guide tables
constexpr int kFeedIdle = 16; // idle lanes that make a warp leave its step loop to take new bundles (15, 17: 1-2% slower)
constexpr int kTurnGather = 5; // lanes waiting at scattering events that make a warp draw their turns
constexpr int kChunkMax = 8;  // tiles a warp claims per work-queue fetch (guided: fewer near the end)
constexpr int kPhaseGuide = 64;  // phase-CDF guide buckets per band (scattering turns)

// ---------------------------------------------------------------------------
// descriptors
// ---------------------------------------------------------------------------
template <typename R>
struct DLevel {
    int im, jm, km, maxs;
    int rx, ry, rz;           // ratio to the next (coarser) level
    unsigned mrx, mry, mrz;   // floor(2^32 / r) + 1 (0 for r = 1): (n + r - 1) / r as a multiply-high
    const R *xu, *yu, *zu;    // faces (views into DSolve::faces)
    const uint16_t *Pw[6];    // wall emission temperature coordinates (or null)
};

// Interleaved table row: k and I_b at temperature rows t and t+1 (the last
// row repeats itself), so one 16-byte load serves a step's interpolation.
template <typename R>
struct alignas(4 * sizeof(R)) KIRow {
    R k0, ib0, k1, ib1;
};

// Per-solve scalars written on the device by the set-up kernels.
struct DScalars {
    unsigned int tmax_bits;   // float bits of max T (non-negative)
    unsigned int tmin_bits;   // float bits of min T
    int status;               // bit 0 out of table, bit 1 non-finite, bit 2 T <= 0, bit 3 index out of bounds,
                              // bit 4 a coordinate beyond 16 bits (cell_coord)
    int tm, row;
    int bad_site;             // first out-of-bounds site (bounds-checked build)
    double Tmax, kappamax, Ibmax_f, Ibmax_w[2];
    double T0, inv_dT;        // first table temperature and 1/spacing
    int Pm;                   // table coordinate of Tmax
    int pad2;
    unsigned long long steps, bundles;
};

template <typename R>
struct DSolve {
    // what entering a level needs of it, two 16-byte loads:
    // lva = (offset of xu in faces, offset of the coordinates in Pall, im, jm);
    // lvb = (km, maxs, bits of dy, bits of dz): face j of y lies at j dy
    int4 lva[RC_MAX_LEVELS], lvb[RC_MAX_LEVELS];
    const R *faces;           // every level's xu | yu | zu, one after the other
    const uint16_t *Pall;     // every level's table coordinates with their halos (cell_index), one after the other
    DLevel<R> lev[RC_MAX_LEVELS];
    int nlev;
    int imax, jmax, kmax, kloc, kfirst;
    int wtype[6];
    int nT, nB, nQ;
    int nVar, photmax, rpt, nchunk, gsize, nparts;
    int sort;  // 1: emitted bundles enter the ring in ascending k (band-sorted order)
    int nwalls, wall_id[2];
    R Lx, Ly, Lz;
    R toll, tollS;
    // run-time values (copied from DScalars by the kernels)
    R Ibmax_f, Ibmax_w0, Ibmax_w1;
    int row;
    const R *xc, *yc, *zc;    // level-0 cell centres incl. ghosts
    const R *probg;           // [nT][nB][nQ]
    const R *cdf_f;           // [nB] fluid band CDF at the selected row
    const R *cdf_s;           // [nB] wall band CDF at the selected row
    const R *probq;           // [nQ]
    const R *Ibw;             // [6][nB] fixed wall spectra
    const uint16_t *Pw0[2];   // level-0 west/east face coordinates [kmax][jmax]
    const KIRow<R> *ki;       // [nB][nQ][nT] interleaved k / I_b rows
    const R *den_f;           // [nB][nQ] I_b(Tmax) k(Tmax) (fluid OERM weight denominator)
    const R *ibm;             // [nB] I_b(Tmax) (wall OERM weight denominator)
    const int *guide_f;       // [kGuide] first band with cdf_f > q/kGuide
    const int *guide_s;       // [kGuide] same for cdf_s
    // scattering particles (nA = 0: none)
    const R *ksca;            // [nB][nQ] scattering coefficient (scaled by chanHeight)
    const R *pcdf;            // [nB][nA] cumulative phase-function probability, last = 1
    const R *pth;             // [nA] scattering angles in turns (theta / 2 pi)
    const uint16_t *pguide;   // [nB][kPhaseGuide+1] phase-CDF search brackets (phase_index)
    int nA;
    DScalars *sc;
    double *partial;
    long long n_fluid_items, n_items, n_tiles;
    // multiply-high reciprocals of the item decomposition divisors
    unsigned long long mg_nchunk, mg_nvar, mg_imax, mg_jmax, mg_nwc;
    unsigned long long nwc;   // jmax * kloc
    // 32-bit reciprocals of nVar, imax, jmax (tile_item); small_div: all three are at most 2^15
    unsigned m_nvar, m_imax, m_jmax;
    int small_div;
    long long steps_to[RC_MAX_LEVELS];  // step budgets of the levels up to and including each
    uint32_t key0, key1;
    long long tile_base;      // first tile of this launch within the solve (server quanta)
    // extents for the bounds-checked build
    long long n_faces, n_P, n_partial;
};

// Bounds-checked indexing.  The product build compiles RC_IX to the plain
// index.  A build with RC_CHECKED=1 (libradchan_checked.so) checks every
// table, field and partial-sum index of the march against its array's
// extent: an index outside [0, n) sets status bit 3 and the first offending
// site in DScalars::bad_site, and is replaced by 0 so the access stays
// inside the array.  Nothing traps.
enum RcSite : int {
    SITE_FACE = 1, SITE_PYRAMID, SITE_ROW, SITE_IBW, SITE_WALL_T, SITE_WALL_ROW, SITE_CENTRE, SITE_EMIT_T,
    SITE_WALL_EMIT_T, SITE_FACE_SHIFT, SITE_EMIT_ROW, SITE_DEN, SITE_IBM, SITE_PROBG, SITE_PARTIAL, SITE_LEVEL,
    SITE_CDF, SITE_KSCA, SITE_PHASE
};
#if RC_CHECKED
__device__ __forceinline__ long long rc_ix(long long i, long long n, int site, DScalars *sc) {
    if (i >= 0 && i < n) return i;
    atomicOr(&sc->status, 8);
    atomicCAS(&sc->bad_site, 0, site);
    return 0;
}
#define RC_IX(i, n, site, S) rc_ix((long long)(i), (long long)(n), (site), (S).sc)
#define RC_IX_IF(go, i, n, site, S) ((go) ? RC_IX(i, n, site, S) : 0)
#else
#define RC_IX(i, n, site, S) (i)
#define RC_IX_IF(go, i, n, site, S) (i)  // the lanes without `go` do not use the address
#endif

// ---------------------------------------------------------------------------
// precision traits
// ---------------------------------------------------------------------------
template <typename R> struct RT;
template <> struct RT<float> {
    static __device__ __forceinline__ float expm1_(float x) { return rc_expm1f(x); }
    static __device__ __forceinline__ float log_(float x) { return rc_logf(x); }
    static __device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
    static __device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }
    static __device__ __forceinline__ float lerp_(float a0, float a1, float w) { return rc_lerpf(a0, a1, w); }
    static __device__ __forceinline__ void sincos2pi_(float u, float *s, float *c) { rc_sincos2pif(u, s, c); }
    static __device__ __forceinline__ float fmin_(float a, float b) { return fminf(a, b); }
    static __device__ __forceinline__ float fmax_(float a, float b) { return fmaxf(a, b); }
    static __device__ __forceinline__ float fabs_(float a) { return fabsf(a); }
};
template <> struct RT<double> {
    static __device__ __forceinline__ double expm1_(double x) { return rc_expm1(x); }
    static __device__ __forceinline__ double log_(double x) { return rc_log(x); }
    static __device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }
    static __device__ __forceinline__ double fma_(double a, double b, double c) { return fma(a, b, c); }
    static __device__ __forceinline__ double lerp_(double a0, double a1, double w) { return rc_lerp(a0, a1, w); }
    static __device__ __forceinline__ void sincos2pi_(double u, double *s, double *c) { rc_sincos2pi(u, s, c); }
    static __device__ __forceinline__ double fmin_(double a, double b) { return fmin(a, b); }
    static __device__ __forceinline__ double fmax_(double a, double b) { return fmax(a, b); }
    static __device__ __forceinline__ double fabs_(double a) { return fabs(a); }
};

// Table coordinate of a temperature with 8 fractional bits, the weight
// precision of the texture unit the reference interpolates with:
// q = rint(256 * clamp((T - T0)/dT, 0, nT-1)); NaN -> 0.
template <typename R>
__device__ __forceinline__ int table_coord(R T, R T0, R inv_dT, int nT) {
    const R p = RT<R>::fmin_(RT<R>::fmax_((T - T0) * inv_dT, (R)0), (R)(nT - 1));
    return (int)rint(p * (R)256);
}

// One interleaved table row through the read-only path.
__device__ __forceinline__ KIRow<float> load_row(const KIRow<float> *p) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
    KIRow<float> r;
    r.k0 = v.x;
    r.ib0 = v.y;
    r.k1 = v.z;
    r.ib1 = v.w;
    return r;
}
__device__ __forceinline__ KIRow<double> load_row(const KIRow<double> *p) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    KIRow<double> r;
    r.k0 = a.x;
    r.ib0 = a.y;
    r.k1 = b.x;
    r.ib1 = b.y;
    return r;
}

// The same by the lanes with `go` only; the others get anything.
__device__ __forceinline__ void load_row_if(bool go, const KIRow<float> *p, KIRow<float> &r) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=f"(r.k0), "=f"(r.ib0), "=f"(r.k1), "=f"(r.ib1)
        : "l"(p), "r"((int)go));
}
__device__ __forceinline__ void load_row_if(bool go, const KIRow<double> *p, KIRow<double> &r) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p ld.global.nc.v2.f64 {%0, %1}, [%4];\n\t"
        "@p ld.global.nc.v2.f64 {%2, %3}, [%4+16];\n\t}"
        : "=&d"(r.k0), "=&d"(r.ib0), "=&d"(r.k1), "=&d"(r.ib1)
        : "l"(p), "r"((int)go));
}

// Fraction of a table coordinate: (q mod 256) / 256, exact: the low byte in
// the mantissa of 2^15 (unit 2^-8), 2^15 subtracted.
template <typename R>
__device__ __forceinline__ R coord_frac(int q) {
    return (R)(__int_as_float(__byte_perm(q, 0x47000000, 0x7440)) - 32768.0f);
}

// Offset of cell (i,j,k) (1-based) of a level of im x jm cells per plane, i
// fastest, one halo cell on every side (halo_code).  The offsets of all levels
// together fit 32 bits without a sign (params_validate).
// (A 4x4x4-brick layout was measured 2-3% slower: its index arithmetic
// costs more issue slots than its locality saves in L1 misses.)
__host__ __device__ __forceinline__ unsigned cell_index(int i, int j, int k, int im, int jm) {
    return i + (unsigned)(im + 2) * (j + (unsigned)(jm + 2) * k);
}

// Linear interpolation in temperature along one table column at a clamped
// coordinate (the reference does this with a clamped linear-filter texture,
// mc_gpu_noint.cu:341-345, memory_copy_noint.cu:241-245).
template <typename R>
__device__ __forceinline__ R lerp_at(const R *col, int i0, int i1, R a) {
    return RT<R>::lerp_(col[i0], col[i1], a);
}
template <typename R>
__device__ __forceinline__ R tab_lerp(const R *col, int nT, int q) {
    const int i0 = q >> 8;
    const int i1 = min(i0 + 1, nT - 1);
    return lerp_at(col, i0, i1, coord_frac<R>(q));
}

// Inverse-CDF bisection with the reference's edge rules
// (mc_gpu_noint.cu:1113-1127): R < cdf[0] -> 0, R == 1 -> n-1.
template <typename R>
__device__ __forceinline__ int bisect(const R *cdf, int n, R u) {
    int lo = 0, w = n;
    while (w > lo + 1) {
        int d = (lo + w) >> 1;
        if (u < cdf[d]) w = d;
        else lo = d;
    }
    int r = lo + 1;
    if (u < cdf[0]) r = 0;
    if (u == (R)1) r = n - 1;
    return min(r, n - 1);
}

// Band index of a uniform u on a cumulative table: the first b with
// u < cdf[b], with the reference's edge rules (R < cdf[0] -> 0, R == 1 ->
// n-1, mc_gpu_noint.cu:1113-1127).  For a non-decreasing cdf this is the
// same index the reference's bisection returns; the guide table gives the
// first band with cdf > q/kGuide, from which a short linear scan finishes.
template <typename R>
__device__ __forceinline__ int guided_index(const R *cdf, const int *guide, int n, R u) {
    const int q = min((int)(u * (R)kGuide), kGuide - 1);
    int b = guide[q];
    while (b < n - 1 && !(u < cdf[b])) ++b;
    return u == (R)1 ? n - 1 : b;
}

// Index of a uniform u on a short non-decreasing cumulative table: the number
// of its entries (the last left out) at or below u, the index the bisection
// returns, from independent loads.
template <typename R>
__device__ __forceinline__ int count_index(const R *cdf, int n, R u) {
    int g = 0;
#pragma unroll 4
    for (int d = 0; d < n - 1; ++d) g += !(u < cdf[d]);
    return u == (R)1 ? n - 1 : g;
}
constexpr int kCountMax = 16;  // g points up to which counting replaces the bisection

// Band and g point of an emitted bundle from its two uniforms: fluid bundles
// (kind 0) search the band CDF at the table row nearest Tmax and then the
// g CDF of that band and row (find_band, mc_gpu_noint.cu:1103-1169); wall
// bundles (kind 1, 2) the Planck-only wall band CDF and the constant g CDF
// probq (find_bandS :1170-1233, with the wall CDF's own edge rule).  The
// fluid's tables are checked to be non-decreasing when they are set; probq
// is not, so it keeps the bisection.
template <typename R>
__device__ __forceinline__ void select_band_g(const DSolve<R> &S, int row, int kind, R u_b, R u_g, int &nb, int &g) {
    const bool wall = kind != 0;
    nb = (int)RC_IX(guided_index(wall ? S.cdf_s : S.cdf_f, wall ? S.guide_s : S.guide_f, S.nB, u_b), S.nB, SITE_CDF, S);
    const R *cg = S.probg + RC_IX(((size_t)row * S.nB + nb) * S.nQ, (long long)S.nT * S.nB * S.nQ, SITE_PROBG, S);
    g = S.nQ == 1 ? 0 : S.nQ <= kCountMax ? count_index(cg, S.nQ, u_g) : bisect(cg, S.nQ, u_g);
    if (wall) g = S.nQ > 1 ? bisect(S.probq, S.nQ, u_g) : 0;
}

// The i and j of a cell in one word, 16 bits each.
__host__ __device__ __forceinline__ unsigned pack_ij(int i, int j) { return (unsigned)i | (unsigned)j << 16; }
__host__ __device__ __forceinline__ int unpack_i(unsigned ij) { return (int)(ij & 0xffffu); }
__host__ __device__ __forceinline__ int unpack_j(unsigned ij) { return (int)(ij >> 16); }

// A bundle after emission, placed at its start point: position, cell,
// direction, sampled band/g and OERM weights.  The edges, bands and g points
// that the packed words hold are the limits of params_validate.
template <typename R>
struct alignas(16) Emitted {
    R sx, sy, sz, ratioI, invTi4;
    unsigned ij;  // ic | jc << 16: the emitting cell (fluid) or wall cell
    int kk;    // kc | kind << 16 | pool index << 18 | pool parity << 29
    int nbg;   // nb | g << 20
};

// A traced ray.  What a step reads is kept ready in registers: the exit face
// of every axis (x: its coordinate fx and its index fi in DSolve::faces; y, z:
// the index as a float and the level's spacing, whose product is the face
// coordinate exactly as the grid builds it), the cell's offset in
// DSolve::Pall with the signed offsets of the three possible neighbours, and
// the cell's table coordinate.  A step moves one of the three axes, so it
// loads one coordinate (and one x face) for the step after it, early enough
// that the absorption of the current step hides their latency.
template <typename R>
struct Ray {
    R xp, yp, zp;
    R sx, sy, sz;
    R isx, isy, isz;
    R tra;
    R Ibmax, ratioI, invTi4, tol;
    R dI;                 // Ib / Ib(Ti) - 1 of the last step (the cutoff deposit of retire_ray)
    R fx;
    int fi;
    float fj, fk, dy, dz;
    unsigned cidx;        // cell offset in Pall
    int dx, dj, dk;       // offsets of the neighbours through the exit faces
    int q;                // coordinate of the cell, the halo code beyond a wall
    int kio;              // first table row of the bundle's band and g point
    int ln;               // band | level << 20
    int rem;              // steps left on the level
    double De;
};
// Coordinates of the halo cells around every level say what the wall between
// does with a ray: reflect it, let it re-enter through the opposite face, or
// end it (kBlack + wall: black walls, and any other type, whose rays are
// lost).  256 table rows end at 65280; a grey table may have more, and a cell
// that lies among its further rows must not read as a wall (cell_coord).
constexpr int kSpecular = 0xfff8, kPeriodic = 0xfff9, kBlack = 0xfffa;

__host__ __device__ __forceinline__ int halo_code(int wtype, int w) {
    return wtype == 1 ? kPeriodic : wtype == 3 ? kSpecular : kBlack + w;
}

// A coordinate as the 16-bit arrays hold it: the cells' below the halo codes,
// the walls' of all 16 bits.  One above (a grey table of more than 256 rows,
// a hot cell) is cut to the largest and reported (bit 4 of the status word).
__host__ __device__ __forceinline__ uint16_t cell_coord(int q, bool wall, bool &cut) {
    const int most = wall ? 0xffff : kSpecular - 1;
    cut = q > most;
    return (uint16_t)(cut ? most : q);
}

// Philox counter of one bundle: (h, v | kind << 24, cell, 0).
__device__ __forceinline__ rc_u32x4 bundle_draws(uint32_t key0, uint32_t key1, int h, int v, int kind, uint32_t cell) {
    rc_u32x4 c;
    c.x = (uint32_t)h;
    c.y = (uint32_t)v | ((uint32_t)kind << 24);
    c.z = cell;
    c.w = 0u;
    return rc_philox4x32_10(c, key0, key1);
}

// Emission of one bundle, placed at its start point.  kind 0: fluid cell
// (i,j,k) from its centre (kernel_fluid :115-186); kind 1/2: west/east wall
// cell (j,k) from the wall (kernel_surface :1381-1441).  Returns false if
// the bundle carries no energy.
//
// OERM weights: invTi4 = 1/I_b(Ti); ratioI = (I_b(Ti) k(Ti)) / (I_b(Tmax)
// k(Tmax)) for the fluid (the reference's ((1/invTi4)/Ib(Tmax))*k(Ti)/
// k(Tmax), :180-186) and I_b(Ti)/I_b(Tmax) for walls (:1421-1424).
// S: the solve's descriptor; row: its run-time table row nearest Tmax.
template <typename R>
__device__ __forceinline__ bool emit_bundle(Emitted<R> &e, const DSolve<R> &S, int row, int kind, int i, int j, int k,
                                            int v, int h) {
    // one path for cells and walls (values selected): a warp's wave runs it
    // together, whatever its bundles are
    const bool wall = kind != 0, east = kind == 2;
    const uint32_t jk = (uint32_t)((j - 1) + S.jmax * (k - 1));
    const uint32_t cell = wall ? jk : (uint32_t)(i - 1) + (uint32_t)S.imax * jk;
    const rc_u32x4 d = bundle_draws(S.key0, S.key1, h, v, kind, cell);
    const R u_phi = (R)rc_u01(d.x), u_mu = (R)rc_u01(d.y), u_b = (R)rc_u01(d.z), u_g = (R)rc_u01(d.w);
    R sp, cp;
    RT<R>::sincos2pi_(u_phi, &sp, &cp);
    // cell, isotropic: cos(theta) = 1 - 2u (emiss_ang, :1077-1084); wall,
    // Lambertian: theta = acos(1 - 2u)/2 (+pi/2 on the east wall)
    // (emiss_angS, :1093-1102), i.e. cos = sqrt(1-u) / -sqrt(u)
    const R mu = (R)1 - (R)2 * u_mu, um1 = (R)1 - u_mu;
    const R st = RT<R>::sqrt_(wall ? (east ? um1 : u_mu) : ((R)1 - mu) * ((R)1 + mu));
    e.sx = mu;
    if (wall) e.sx = east ? -RT<R>::sqrt_(u_mu) : RT<R>::sqrt_(um1);
    e.sy = st * cp;
    e.sz = st * sp;
    // components floored (:132-137, walls :1395-1400)
    const R tiny = wall ? (R)1e-10 : (R)0;
    if (RT<R>::fabs_(e.sx) <= tiny) e.sx = (R)(east ? -1 : 1) * (R)1e-10;
    if (RT<R>::fabs_(e.sy) <= tiny) e.sy = (R)(wall && !(e.sy > (R)0) ? -1 : 1) * (R)1e-10;
    if (RT<R>::fabs_(e.sz) <= tiny) e.sz = (R)(wall && !(e.sz > (R)0) ? -1 : 1) * (R)1e-10;
    int nb, g;
    select_band_g(S, row, kind, u_b, u_g, nb, g);
    const int Pi = wall ? S.Pw0[east][RC_IX(jk, (long long)S.kmax * S.jmax, SITE_WALL_EMIT_T, S)]
                        : S.Pall[RC_IX((unsigned)S.lva[0].y + cell_index(i, j, k, S.imax, S.jmax), S.n_P, SITE_EMIT_T, S)];
    const int ic = wall ? (east ? S.imax : 1) : i;
    e.nbg = nb | (g << 20);
    e.ij = pack_ij(ic, j);
    e.kk = k | (kind << 16);
    // OERM weights
    const KIRow<R> ki =
        load_row(S.ki + RC_IX(((size_t)nb * S.nQ + g) * S.nT + (Pi >> 8), (long long)S.nB * S.nQ * S.nT, SITE_EMIT_ROW, S));
    const R fr = coord_frac<R>(Pi);
    const R Ib_i = RT<R>::lerp_(ki.ib0, ki.ib1, fr);
    const R k_i = RT<R>::lerp_(ki.k0, ki.k1, fr);
    const R den = wall ? S.ibm[RC_IX(nb, S.nB, SITE_IBM, S)]
                       : S.den_f[RC_IX((size_t)nb * S.nQ + g, (long long)S.nB * S.nQ, SITE_DEN, S)];
    e.invTi4 = (R)1 / Ib_i;
    e.ratioI = (wall ? Ib_i : Ib_i * k_i) / den;
    return Ib_i > (R)0 && den > (R)0;
}

// What a step of a ray in cell c of the level (A, B) reads: see Ray.
template <typename R>
__device__ __forceinline__ void set_cell(Ray<R> &r, const DSolve<R> &S, const int3 &c, const int4 &A, const int4 &B) {
#if RC_CHECKED
    // the cell must lie inside its level or in its halo
    if (c.x < 0 || c.x > A.z + 1 || c.y < 0 || c.y > A.w + 1 || c.z < 0 || c.z > B.x + 1)
        RC_IX(-1, 0, SITE_PYRAMID, S);
#endif
    const int sj = A.z + 2, sk = sj * (A.w + 2);
    const bool nx = r.sx < (R)0, ny = r.sy < (R)0, nz = r.sz < (R)0;
    r.cidx = (unsigned)A.y + c.x + (unsigned)sj * c.y + (unsigned)sk * c.z;
    r.q = __ldg(S.Pall + RC_IX(r.cidx, S.n_P, SITE_PYRAMID, S));
    r.fi = A.x + c.x - (int)nx;
    r.fx = __ldg(S.faces + RC_IX(r.fi, S.n_faces, SITE_FACE, S));
    r.dx = nx ? -1 : 1;
    r.dj = ny ? -sj : sj;
    r.dk = nz ? -sk : sk;
    r.fj = (float)(c.y - (int)ny);
    r.fk = (float)(c.z - (int)nz);
    r.dy = __int_as_float(B.z);
    r.dz = __int_as_float(B.w);
}

// Ray state of an emitted bundle.  D: the descriptor in device memory, which
// holds the run-time Ibmax (S may be its copy in the kernel's parameters).
template <typename R>
__device__ __forceinline__ void place_bundle(Ray<R> &r, const DSolve<R> &S, const DSolve<R> &D, const Emitted<R> &e) {
    const int kind = (e.kk >> 16) & 3;
    int ic = unpack_i(e.ij), jc = unpack_j(e.ij), kc = e.kk & 0xffff;
    // start point: the cell centre, or the wall cell's point on the wall
    // (kernel_fluid :117-122, kernel_surface :1381-1384)
    r.xp = kind == 0 ? S.xc[RC_IX(ic, S.imax + 2, SITE_CENTRE, S)] : (kind == 1 ? (R)0 : S.Lx);
    r.yp = S.yc[RC_IX(jc, S.jmax + 2, SITE_CENTRE, S)];
    r.zp = S.zc[RC_IX(kc, S.kmax + 2, SITE_CENTRE, S)];
    if (kind != 0) {
        // cell shift when the start point lies on a face (:1429-1441)
        const DLevel<R> &G = S.lev[0];
        const bool fx = e.sx < (R)0, fy = e.sy < (R)0, fz = e.sz < (R)0;
        const int i0 = ic, j0 = jc, k0 = kc;
        if (fx && r.xp == G.xu[RC_IX(i0 - 1, G.im + 1, SITE_FACE_SHIFT, S)]) ic = i0 - 1;
        if (fy && r.yp == G.yu[RC_IX(j0 - 1, G.jm + 1, SITE_FACE_SHIFT, S)]) jc = j0 - 1;
        if (fz && r.zp == G.zu[RC_IX(k0 - 1, G.km + 1, SITE_FACE_SHIFT, S)]) kc = k0 - 1;
        if (!fx && r.xp == G.xu[RC_IX(ic, G.im + 1, SITE_FACE_SHIFT, S)]) ic = ic + 1;
        if (!fy && r.yp == G.yu[RC_IX(jc, G.jm + 1, SITE_FACE_SHIFT, S)]) jc = jc + 1;
        if (!fz && r.zp == G.zu[RC_IX(kc, G.km + 1, SITE_FACE_SHIFT, S)]) kc = kc + 1;
    }
    r.sx = e.sx;
    r.sy = e.sy;
    r.sz = e.sz;
    r.isx = (R)1 / e.sx;
    r.isy = (R)1 / e.sy;
    r.isz = (R)1 / e.sz;
    r.ratioI = e.ratioI;
    r.invTi4 = e.invTi4;
    const int nb = e.nbg & 0xfffff, g = e.nbg >> 20;
    r.kio = (nb * S.nQ + g) * S.nT;
    r.ln = nb;
    set_cell(r, S, make_int3(ic, jc, kc), S.lva[0], S.lvb[0]);
    r.rem = S.lvb[0].y;
    r.tra = (R)1;
    r.De = 0.0;
    r.dI = (R)0;
    r.Ibmax = kind == 0 ? D.Ibmax_f : kind == 1 ? D.Ibmax_w0 : D.Ibmax_w1;
    r.tol = kind == 0 ? S.toll : S.tollS;
}

// Index of the coarse cell holding fine cell n (1-based): (n + r - 1) / r,
// as floor(n' m / 2^32) with m = floor(2^32 / r) + 1, exact for n' r < 2^32
// (the host checks it); m = 0 stands for r = 1.
__device__ __forceinline__ int coarse_index(int n, int r, unsigned m) {
    const unsigned np = (unsigned)(n + r - 1);
    return (int)(m ? __umulhi(np, m) : np);
}

// Integer cell coordinates of a ray on its level (0 and extent + 1: beyond a
// wall), from the indices of its exit faces.
template <typename R>
__device__ __forceinline__ int3 ray_cell(const Ray<R> &r, const int4 &A) {
    return make_int3(r.fi - A.x + (int)(r.sx < (R)0), (int)r.fj + (int)(r.sy < (R)0), (int)r.fk + (int)(r.sz < (R)0));
}

// Wall a ray beyond the extents of its level (A, B: its words of lva, lvb)
// has crossed.
__device__ __forceinline__ int crossed_wall(const int3 &c, const int4 &A, const int4 &B) {
    if (c.x == 0) return RC_WEST;
    if (c.x > A.z) return RC_EAST;
    if (c.y == 0) return RC_SOUTH;
    if (c.y > A.w) return RC_NORTH;
    return c.z == 0 ? RC_BOT : RC_TOP;
}

// Everything about a ray's next cell that is not the plain move to the
// neighbour: the wall condition when the cell lies beyond a wall (:375-654,
// with the y/z specular branches reflecting the right component and flag),
// the move to coarser levels once the step budget of the level is spent
// (:210-224), and the faces, offsets and table coordinate of the cell that
// results.  Returns false when the ray must stop: at a black wall or as a
// lost ray (the coordinate stays kBlack + wall; retire_ray deposits the rest) or
// when the budget of the last level is spent.
template <typename R>
__device__ __forceinline__ bool enter_cell(Ray<R> &r, const DSolve<R> &S) {
    int lev = r.ln >> 20;
    int4 A = S.lva[RC_IX(lev, S.nlev, SITE_LEVEL, S)];
    int4 B = S.lvb[RC_IX(lev, S.nlev, SITE_LEVEL, S)];
    int3 c = ray_cell(r, A);
    const int code = r.q;
    if (code >= kSpecular) {
        if (code >= kBlack) return false;
        const int w = crossed_wall(c, A, B);
        // periodic: re-enter through the opposite face; specular: stay in
        // the cell with the crossed component reversed
        const bool hi = w & 1, per = code == kPeriodic;
        if (w <= RC_EAST) {
            r.xp = hi != per ? S.Lx : (R)0;
            c.x = hi != per ? A.z : 1;
            if (!per) r.sx = -r.sx, r.isx = -r.isx;
        } else if (w <= RC_NORTH) {
            r.yp = hi != per ? S.Ly : (R)0;
            c.y = hi != per ? A.w : 1;
            if (!per) r.sy = -r.sy, r.isy = -r.isy;
        } else {
            r.zp = hi != per ? S.Lz : (R)0;
            c.z = hi != per ? B.x : 1;
            if (!per) r.sz = -r.sz, r.isz = -r.isz;
        }
    }
    while (r.rem <= 0) {
        if (lev >= S.nlev - 1) {
            // stopped without a deposit, whatever the transmissivity
            r.tol = (R)0;
            r.q = 0;
            return false;
        }
        const DLevel<R> &L = S.lev[lev];
        c.x = coarse_index(c.x, L.rx, L.mrx);
        c.y = coarse_index(c.y, L.ry, L.mry);
        c.z = coarse_index(c.z, L.rz, L.mrz);
        lev += 1;
        r.ln += 1 << 20;
        A = S.lva[lev];
        B = S.lvb[lev];
        r.rem = B.y;
    }
    set_cell(r, S, c, A, B);
    return true;
}

// Re-entry of a ray beyond a periodic wall (coordinate kPeriodic) through the
// opposite face, with steps left on its level: what enter_cell does for it,
// without rebuilding what stays.  A channel's rays cross the y and z
// boundaries in about half of a warp's iterations, one or two lanes at a time.
template <typename R>
__device__ __forceinline__ void wrap_cell(Ray<R> &r, const DSolve<R> &S) {
    const int lev = RC_IX(r.ln >> 20, S.nlev, SITE_LEVEL, S);
    const int4 A = S.lva[lev];
    const int km = S.lvb[lev].x;
    const float fjm = (float)A.w, fkm = (float)km;
    if (r.fj < 0.f || r.fj > fjm) {
        const bool hi = r.fj > 0.f;
        r.yp = hi ? (R)0 : S.Ly;
        r.fj = hi ? 1.f : fjm - 1.f;
        r.cidx -= (unsigned)A.w * r.dj;
    } else if (r.fk < 0.f || r.fk > fkm) {
        const bool hi = r.fk > 0.f;
        r.zp = hi ? (R)0 : S.Lz;
        r.fk = hi ? 1.f : fkm - 1.f;
        r.cidx -= (unsigned)km * r.dk;
    } else {
        const bool hi = r.dx > 0;
        r.xp = hi ? (R)0 : S.Lx;
        r.fi = A.x + (hi ? 1 : A.z - 1);
        r.cidx -= (unsigned)A.z * r.dx;
        r.fx = __ldg(S.faces + RC_IX(r.fi, S.n_faces, SITE_FACE, S));
    }
    r.q = __ldg(S.Pall + RC_IX(r.cidx, S.n_P, SITE_PYRAMID, S));
}

// Absorption along a path of length ds in a cell of absorption coefficient
// absco and blackbody intensity blackpow: the step's OERM tally and the
// transmissivity update (:358-364).
template <typename R>
__device__ __forceinline__ void absorb(Ray<R> &r, R ds, R absco, R blackpow, bool go) {
    // a lane that does not step: nothing absorbed, its last dI kept
    const R em = go ? RT<R>::expm1_(-(ds * absco)) : (R)0;
    const R alpha = -em;
    r.dI = go ? RT<R>::fma_(r.invTi4, blackpow, (R)-1) : r.dI;
    R c = r.Ibmax * r.tra;
    c = c * alpha;
    c = c * r.ratioI;
    c = c * r.dI;
    r.De -= (double)c;
    r.tra = RT<R>::fma_(r.tra, em, r.tra);
}

// Last deposit of a ray that has stopped: the rest of its energy in the cell
// where its transmissivity fell below the cutoff (:365-370), or on the black
// wall it has reached (:398-399 and its siblings), De -= Ibmax tra ratioI
// (invTi4 e - 1).  The march retires the stopped rays of a warp together.
// Returns whether the ray's energy is spent (its transmissivity is then 0).
template <typename R>
__device__ __forceinline__ bool retire_ray(Ray<R> &r, const DSolve<R> &S) {
    if (r.tra < r.tol) {
        R c2 = (r.Ibmax * r.tra) * r.ratioI;
        c2 = c2 * r.dI;
        r.De -= (double)c2;
        return true;
    }
    if (r.q < kBlack) return false;
    const int w = r.q - kBlack, t = S.wtype[w];
    R e;
    if (t == 2) {  // black wall at its own temperature
        e = S.Ibw[RC_IX((size_t)w * S.nB + (r.ln & 0xfffff), 6LL * S.nB, SITE_IBW, S)];
    } else if (t == 4 || t == 6) {  // black wall at a field temperature
        const int lev = RC_IX(r.ln >> 20, S.nlev, SITE_LEVEL, S);
        const int4 A = S.lva[lev], B = S.lvb[lev];
        const int im = A.z, jm = A.w, km = B.x;
        const int3 cell = ray_cell(r, A);
        const int idx = w <= RC_EAST    ? (cell.z - 1) * jm + (cell.y - 1)
                        : w <= RC_NORTH ? (cell.z - 1) * im + (cell.x - 1)
                                        : (cell.y - 1) * im + (cell.x - 1);
        const long long n = w <= RC_EAST ? (long long)jm * km : w <= RC_NORTH ? (long long)im * km : (long long)im * jm;
        const int q = S.lev[lev].Pw[w][RC_IX(idx, n, SITE_WALL_T, S)];
        const KIRow<R> row = S.ki[r.kio + RC_IX(q >> 8, S.nT, SITE_WALL_ROW, S)];
        e = RT<R>::lerp_(row.ib0, row.ib1, coord_frac<R>(q));
    } else {
        return true;  // lost ray
    }
    R c = (r.Ibmax * r.tra) * RT<R>::fma_(r.invTi4, e, (R)-1);
    c = c * r.ratioI;
    r.De -= (double)c;
    return true;
}

// ---------------------------------------------------------------------------
// scattering by suspended particles
// ---------------------------------------------------------------------------
// The reference's Monte Carlo path has no scattering; nbcorrk tabulates the
// particles' scattering coefficient per band and g point and their phase
// function per band (nbcorrk/write_tables.cpp:204-260, :326-336).  A bundle
// of a scattering medium carries, besides its Ray, the Philox counter words
// of its emission (h, v | kind << 24, cell): draw n (the fourth counter word
// n >= 1; emission uses 0) is its n-th draw after emission.  Draw 1 gives
// the free path to the first scattering event, -ln(u) / k_s with k_s the
// scattering coefficient of its band and g point (no event when k_s = 0);
// at event n draw n+1 gives the scattering angle (the band's cumulative
// phase probability inverted, linear in angle between table angles), the
// azimuth (uniform) and the free path to the next event.  The free path is
// sampled against the scattering coefficient alone; absorption stays the
// continuous OERM tally, so the emission-based reciprocity weights are
// unchanged (the exchange between two cells is reciprocal for a phase
// function of the scattering angle alone).
// What a step needs of a scattering bundle is one register: the distance
// left to its next event.  The counter words, event count and k_s (needed
// only at an event) are kept apart, in shared memory in the march.
constexpr float kNoEvent = 3.0e38f;  // free path of a bundle whose band does not scatter
template <typename R>
struct ScatState {
    R dist;  // distance left to the next event; < 0: stopped at an event,
             // new direction not drawn yet
};

// Scattering coefficient of band nb, g point g (0 without particles).
template <typename R>
__device__ __forceinline__ R scatter_coef(const DSolve<R> &S, int nb, int g) {
    return (S.nA > 0) ? S.ksca[RC_IX((size_t)nb * S.nQ + g, (long long)S.nB * S.nQ, SITE_KSCA, S)] : (R)0;
}

// Philox counter words of a bundle (emission's: h, v | kind << 24, cell),
// with the event count in w.
__device__ __forceinline__ uint4 scatter_counter(uint32_t imax, uint32_t jmax, int kind, int i, int j, int k, int v,
                                                 int h, uint32_t nev) {
    const uint32_t cell = (kind == 0) ? (uint32_t)((i - 1) + imax * ((j - 1) + jmax * (k - 1)))
                                      : (uint32_t)((j - 1) + jmax * (k - 1));
    return make_uint4((uint32_t)h, (uint32_t)v | ((uint32_t)kind << 24), cell, nev);
}

// -ln(u) of draw 1 of a bundle with counter words ctr: its free path to the
// first event in units of 1/k_s.  The draw does not depend on the band, so
// the march takes it before the band is sampled (what is live at that
// point is small).
template <typename R>
__device__ __forceinline__ R scatter_first_lnu(const DSolve<R> &S, uint4 ctr) {
    rc_u32x4 c;
    c.x = ctr.x;
    c.y = ctr.y;
    c.z = ctr.z;
    c.w = 1u;
    const rc_u32x4 d = rc_philox4x32_10(c, S.key0, S.key1);
    return -RT<R>::log_((R)rc_u01(d.x));
}

// Free path to the first event: lnu / ks, kNoEvent when ks = 0.
template <typename R>
__device__ __forceinline__ R scatter_first_dist(R lnu, R ks) {
    return (ks > (R)0) ? lnu / ks : (R)kNoEvent;
}

// Angle index of a uniform u on the phase CDF of a band: the first a in
// [1, nA-1] with u < cdf[a] (nA-1 if none), which is what a bisection over
// the whole table returns for a CDF that starts at 0 and does not decrease.
// guide[q] (q = 0..kPhaseGuide) is the first a >= 1 with cdf[a] > q /
// kPhaseGuide (nA-1 if none), so for u in bucket q the answer lies in
// (guide[q] - 1, guide[q+1]] and the bisection runs over that bracket only:
// one or two table reads instead of log2(nA) dependent ones.
template <typename R>
__device__ __forceinline__ int phase_index(const R *cdf, const uint16_t *guide, R u) {
    const int q = min((int)(u * (R)kPhaseGuide), kPhaseGuide - 1);
    int lo = (int)guide[q] - 1, hi = (int)guide[q + 1];
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (u < cdf[mid]) hi = mid;
        else lo = mid;
    }
    return hi;
}

// New direction of a bundle travelling along (sx, sy, sz) in band nb at a
// scattering event (ctr: its counter words x, y, z and the number of the
// event in w; ks > 0 its scattering coefficient), with the reciprocals of
// the new direction and the free path to the event after it.  Everything is
// passed and returned by value: a reference would oblige the caller to keep
// the ray in local memory.
template <typename R>
struct TurnOut {
    R sx, sy, sz, isx, isy, isz, dist;
};
template <typename R>
__device__ __forceinline__ TurnOut<R> scatter_turn_v(R sx, R sy, R sz, int nb, uint4 ctr, R ks, const DSolve<R> *Sp) {
    const DSolve<R> &S = *Sp;
    rc_u32x4 c;
    c.x = ctr.x;
    c.y = ctr.y;
    c.z = ctr.z;
    c.w = ctr.w + 1u;
    const rc_u32x4 d = rc_philox4x32_10(c, S.key0, S.key1);
    const R u_t = (R)rc_u01(d.x), u_p = (R)rc_u01(d.y), u_s = (R)rc_u01(d.z);
    const int nA = S.nA;
    const R *cdf = S.pcdf + RC_IX((size_t)nb * nA, (long long)S.nB * nA, SITE_PHASE, S);
    const int hi = phase_index(cdf, S.pguide + RC_IX((size_t)nb * (kPhaseGuide + 1),
                                                     (long long)S.nB * (kPhaseGuide + 1), SITE_PHASE, S), u_t);
    const R c0 = cdf[hi - 1], c1 = cdf[hi];
    R fr = (c1 > c0) ? (u_t - c0) / (c1 - c0) : (R)0;
    if (fr > (R)1) fr = (R)1;
    const R t0 = S.pth[hi - 1], t1 = S.pth[hi];
    const R th = RT<R>::fma_(fr, t1 - t0, t0);
    R st, ct, sp, cp;
    RT<R>::sincos2pi_(th, &st, &ct);
    RT<R>::sincos2pi_(u_p, &sp, &cp);
    R nx, ny, nz;
    if (RT<R>::fabs_(sz) > (R)0.99999) {
        nx = st * cp;
        ny = st * sp;
        nz = (sz > (R)0) ? ct : -ct;
    } else {
        const R w = RT<R>::sqrt_((R)1 - sz * sz);
        const R a = st / w;
        nx = a * (sx * sz * cp - sy * sp) + sx * ct;
        ny = a * (sy * sz * cp + sx * sp) + sy * ct;
        nz = sz * ct - st * cp * w;
    }
    if (nx == (R)0) nx = (R)1e-10;
    if (ny == (R)0) ny = (R)1e-10;
    if (nz == (R)0) nz = (R)1e-10;
    TurnOut<R> o;
    o.sx = nx;
    o.sy = ny;
    o.sz = nz;
    o.isx = (R)1 / nx;
    o.isy = (R)1 / ny;
    o.isz = (R)1 / nz;
    o.dist = -RT<R>::log_(u_s) / ks;
    return o;
}

// The next scattering event of ray r: the event count in ctr.w advances,
// the direction turns, and q receives the free path to the event after it.
template <typename R>
__device__ __forceinline__ void scatter_turn(Ray<R> &r, uint4 &ctr, R ks, ScatState<R> &q, const DSolve<R> &S) {
    ctr.w += 1u;
    const TurnOut<R> o = scatter_turn_v(r.sx, r.sy, r.sz, r.ln & 0xfffff, ctr, ks, &S);
    // the cell stays; its exit faces and neighbours follow the new signs
    const bool nx = o.sx < (R)0, ny = o.sy < (R)0, nz = o.sz < (R)0;
    const bool fx = nx != (r.sx < (R)0), fy = ny != (r.sy < (R)0), fz = nz != (r.sz < (R)0);
    r.fi += fx ? (nx ? -1 : 1) : 0;
    r.fj += fy ? (ny ? -1.f : 1.f) : 0.f;
    r.fk += fz ? (nz ? -1.f : 1.f) : 0.f;
    r.dx = nx ? -1 : 1;
    r.dj = fy ? -r.dj : r.dj;
    r.dk = fz ? -r.dk : r.dk;
    r.fx = __ldg(S.faces + RC_IX(r.fi, S.n_faces, SITE_FACE, S));
    r.sx = o.sx;
    r.sy = o.sy;
    r.sz = o.sz;
    r.isx = o.isx;
    r.isy = o.isy;
    r.isz = o.isz;
    q.dist = o.dist;
}

// One ray-cell crossing (one iteration of the while loop of march_ray,
// :252-656) of a ray whose cell lies inside the level (enter_cell).  The side
// of the cell a ray leaves through on each axis follows from the sign of its
// direction component (never 0: emission floors it at 1e-10).  The geometry
// does not depend on the absorption, so the move to the neighbouring cell and
// the loads of its table coordinate and its new exit face come first; the
// absorption of this cell covers their latency.  All lanes of a warp run
// through it together, without a branch; those without `go` keep their ray and
// load their own cell again.  Returns whether the ray's transmissivity is still above
// the cutoff.
// With SCAT, a bundle whose step is longer than the distance left to its next
// event stops at the event inside the cell (absorbing along the shortened
// path), counts the event as a step and sets qs.dist < 0: the caller draws the
// new direction (scatter_turn) before the next step.  The turn depends neither
// on the cell nor on the level, so a caller may gather the turns of several
// lanes into one pass.
template <typename R, bool SCAT>
__device__ __forceinline__ bool march_step(Ray<R> &r, ScatState<R> &qs, const DSolve<R> &S, bool go) {
    KIRow<R> row;
    load_row_if(go, S.ki + r.kio + RC_IX_IF(go, r.q >> 8, S.nT, SITE_ROW, S), row);
    const R a = coord_frac<R>(r.q);
    const R fy = (R)(r.fj * r.dy), fz = (R)(r.fk * r.dz);
    const R dsx = (r.fx - r.xp) * r.isx;
    const R dsy = (fy - r.yp) * r.isy;
    const R dsz = (fz - r.zp) * r.isz;
    const R ds = RT<R>::fmin_(RT<R>::fmin_(dsx, dsy), dsz);
    // with SCAT, ev: the next scattering event lies inside this cell; the
    // bundle stops there (one absorption path shared with the plain step,
    // so the step loop's code does not grow)
    R dstep = ds;
    bool mv = go;
    if constexpr (SCAT) {
        const bool ev = ds > qs.dist;
        dstep = go ? (ev ? qs.dist : ds) : (R)0;
        qs.dist = go ? (ev ? (R)-1 : qs.dist - ds) : qs.dist;
        mv = go && !ev;
    }
    // a lane that does not step needs its position only if it waits for a turn
    const bool snap = SCAT ? mv : true;
    r.xp = (snap && ds == dsx) ? r.fx : RT<R>::fma_(dstep, r.sx, r.xp);
    r.yp = (snap && ds == dsy) ? fy : RT<R>::fma_(dstep, r.sy, r.yp);
    r.zp = (snap && ds == dsz) ? fz : RT<R>::fma_(dstep, r.sz, r.zp);
    // crossed axis (ties: x only if strictly smallest, :375-377, 524)
    const bool lt = dsx < dsy, lz = (lt ? dsx : dsy) < dsz;
    const int mvd = lz ? (lt ? r.dx : r.dj) : r.dk;
    r.cidx += mv ? mvd : 0;
    r.fi += mv && lz && lt ? r.dx : 0;
    r.fj += mv && lz && !lt ? copysignf(1.f, (float)r.sy) : 0.f;
    r.fk += mv && !lz ? copysignf(1.f, (float)r.sz) : 0.f;
    r.q = __ldg(S.Pall + RC_IX(r.cidx, S.n_P, SITE_PYRAMID, S));
    r.fx = __ldg(S.faces + RC_IX(r.fi, S.n_faces, SITE_FACE, S));
    r.rem -= (int)go;
    absorb(r, dstep, RT<R>::lerp_(row.k0, row.k1, a), RT<R>::lerp_(row.ib0, row.ib1, a), go);
    return r.tra > r.tol;
}

// n / d for a divisor fixed per solve: with M = floor((2^64 - 1)/d) + 1,
// floor(n M / 2^64) = floor(n / d) whenever n d < 2^64 (the host checks the
// bound when it builds the descriptor); M = 0 encodes d = 1.
__device__ __forceinline__ unsigned long long fdiv(unsigned long long n, unsigned long long M) {
    return M ? __umul64hi(n, M) : n;
}

// Decoded work item: item = ((cell*nVar + v)*nchunk + q); the wall items
// follow the fluid items.  kind = -1 marks an item past the end.
struct ItemId {
    int kind, i, j, k, v, h0;
};

template <typename R>
__device__ __forceinline__ ItemId decode_item(const DSolve<R> &S, long long item) {
    ItemId d;
    d.kind = -1;
    d.i = d.j = d.k = d.v = d.h0 = 0;
    if (item >= S.n_items) return d;
    unsigned long long it = (unsigned long long)item;
    int kind = 0;
    if (item >= S.n_fluid_items) {
        it -= (unsigned long long)S.n_fluid_items;
        kind = 1;
    }
    const unsigned long long t = fdiv(it, S.mg_nchunk);
    const int q = (int)(it - t * (unsigned long long)S.nchunk);
    const unsigned long long c = fdiv(t, S.mg_nvar);
    d.v = (int)(t - c * (unsigned long long)S.nVar);
    d.h0 = q * S.rpt;
    if (kind == 0) {
        const unsigned long long cj = fdiv(c, S.mg_imax);
        d.i = (int)(c - cj * (unsigned long long)S.imax) + 1;
        const unsigned long long ck = fdiv(cj, S.mg_jmax);
        d.j = (int)(cj - ck * (unsigned long long)S.jmax) + 1;
        d.k = (int)ck + S.kfirst;
        d.kind = 0;
    } else {
        const unsigned long long slot = fdiv(c, S.mg_nwc);
        const unsigned long long wc = c - slot * S.nwc;
        const unsigned long long kw = fdiv(wc, S.mg_jmax);
        d.j = (int)(wc - kw * (unsigned long long)S.jmax) + 1;
        d.k = (int)kw + S.kfirst;
        d.kind = 1 + S.wall_id[(int)slot];
    }
    return d;
}

// A tile in flight: its first item, how many of its emitted bundles have not
// finished, and the first item decoded (0-based i, j, k; q its chunk).  fluid:
// every item is a cell's, so the others follow from the first by 32-bit
// arithmetic on small numbers (tile_item).
struct TileBuf {
    long long item0;
    int out, fluid;
    int i, j, k, v, q, pad;
};

template <typename R>
__device__ __forceinline__ void decode_tile(const DSolve<R> &S, long long item0, TileBuf &t) {
    const ItemId d = decode_item(S, item0);
    t.item0 = item0;
    t.out = 0;
    t.fluid = S.small_div && item0 + kWarp <= S.n_fluid_items;
    t.i = d.i - 1;
    t.j = d.j - 1;
    t.k = d.k;
    t.v = d.v;
    t.q = d.h0 >> (__ffs(S.rpt) - 1);  // rpt: a power of two
}

// n / d for n < 2^16, d <= 2^15 with m = magic32(d): exact (n d < 2^32).
__device__ __forceinline__ int sdiv(int n, unsigned m) { return m ? (int)__umulhi((unsigned)n, m) : n; }

// Item it (0..31) of a tile.  The chunks of one (cell, replicate) are a power
// of two up to 32, or a multiple of 32: a tile starts at the first chunk of a
// (cell, replicate), or holds one only.
template <typename R>
__device__ __forceinline__ ItemId tile_item(const DSolve<R> &S, const TileBuf &t, int it) {
    if (!t.fluid) return decode_item(S, t.item0 + it);
    ItemId d;
    d.kind = 0;
    d.h0 = (t.q + (it & (S.gsize - 1))) * S.rpt;
    d.v = t.v;
    int i = t.i, j = t.j, k = t.k;
    if (S.gsize < kWarp) {
        const int x = t.v + (it >> (__ffs(S.gsize) - 1));
        const int c = sdiv(x, S.m_nvar);
        d.v = x - c * S.nVar;
        i += c;
        const int ci = sdiv(i, S.m_imax);
        i -= ci * S.imax;
        j += ci;
        const int cj = sdiv(j, S.m_jmax);
        j -= cj * S.jmax;
        k += cj;
    }
    d.i = i + 1;
    d.j = j + 1;
    d.k = k;
    return d;
}

}  // namespace rc
