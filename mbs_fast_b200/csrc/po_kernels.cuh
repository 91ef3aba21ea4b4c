// po_kernels.cuh — the sm_100a kernels of the PO diffraction path.
//
//   po_pack_kernel       flat mbs_po_beams arrays -> device beam records
//   po_diffract_kernel   fused aperture integral -> coherent Jones sum ->
//                        Mueller -> orientation average (one CTA per azimuth
//                        bin x zenith tile x orientation chunk)
//   po_pole_kernel       the polar zenith rows, whose direction and basis are
//                        the same for every azimuth bin
//   po_reduce_kernel     deterministic sum of the chunk partials
//   po_extinction_kernel optical-theorem extinction per orientation
#pragma once

#include "mbs_po_b200.h"
#include "po_device.cuh"

namespace mbs {

// ------------------------------------------------------------------ records

// A beam record: azimuth-independent coefficients, precomputed at staging.
//   A(t, phi) = sin t (-(cos phi h0 + sin phi h1)) + cos t h2 + a0, B likewise.
//   With vf = (-sin phi, cos phi, 0) off the poles, u = vt = -(cos phi cos t,
//   sin phi cos t, sin t) and w = vt x dir = -vf, so the rotation of
//   GpuDiffraction.cu:831-856 is R = R0 + cos t Rc + sin t Rs with
//     R0 = sin phi X1 + cos phi X2,  Rc = -(cos phi Y1 + sin phi Y2),  Rs = Z
//   X1 = [[NTx, NPx], [-DTx, -DPx]], X2 = [[-NTy, -NPy], [DTy, DPy]],
//   Y1 = [[DTx, DPx], [NTx, NPx]],   Y2 = [[DTy, DPy], [NTy, NPy]],
//   Z  = [[-DTz, -DPz], [-NTz, -NPz]]  (NT, NP, DT = nxDT, DP = nxDP).
//   Q holds complWave * (X J_phased) for X1, X2, Y1, Y2, Z (4 complex
//   entries each), so d = s m (P0 + cos t Pc + sin t Ps) with
//   P0 = sin phi Q1 + cos phi Q2, Pc = -(cos phi Q3 + sin phi Q4), Ps = Q5.
//   slab: k (xa, ya) / 1.25e-3, k (xb, yb) / 1.25e-3, the small-phase candidate
//   test (see the pack kernel); nearr2 (float): FP32C near-forward zone,
//   A^2+B^2 <= nearr2.

// Per vertex, azimuth-independent parts of the phase in turns:
//   phase(t, phi) = sin t ps + cos t pc + p0,  ps = -(cos phi X + sin phi Y)
// (internal beams include the common beam-centre phase, GpuDiffraction.cu:1110-1122).
// Slopes of the x and y branches; an edge invalid for a branch (|dx| or |dy|
// below the geometry tolerance, Handler.cpp:674-692) gets the slope 1e30, so
// its coefficient is ~1e30 |B| (or |A|) and its term ~1e-30 of the others:
// the reference skips it.
struct __align__(16) VertRec {
    double X, Y, pc, p0;
    double syx, sxy;
};

// Both record arrays are stored as structures of arrays: word w of record i
// at base[w * stride + i], so the lanes of a warp that fill consecutive
// records read consecutive words (full 32-byte sectors) instead of one
// scattered sector per lane.
// Words of a beam record (low | high half of the last two): h0 h1 h2 a0 v0 v1 v2
// b0, Q[40], slab[4], (nearr2 | vbeg), (nv | beam flags).
constexpr int kBrecWords = 54;
constexpr int kVrecWords = 6;    // X Y pc p0 syx sxy

struct BrecRef {
    const double *p;   // word 0 of the record
    int64_t s;         // stride between words
    __device__ __forceinline__ double ab(int i) const { return p[i * s]; }
    __device__ __forceinline__ double Q(int i) const { return p[(8 + i) * s]; }
    __device__ __forceinline__ double slab(int i) const { return p[(48 + i) * s]; }
    __device__ __forceinline__ float nearr2() const { return __int_as_float(__double2loint(p[52 * s])); }
    __device__ __forceinline__ int nv() const { return __double2loint(p[53 * s]); }
    __device__ __forceinline__ bool external() const
    {
        return (__double2hiint(p[53 * s]) & MBS_PO_BEAM_EXTERNAL) != 0;
    }
};

struct VrecRef {
    const double *p;
    int64_t s;
    __device__ __forceinline__ double X() const { return p[0]; }
    __device__ __forceinline__ double Y() const { return p[s]; }
    __device__ __forceinline__ double pc() const { return p[2 * s]; }
    __device__ __forceinline__ double p0() const { return p[3 * s]; }
    __device__ __forceinline__ double syx() const { return p[4 * s]; }
    __device__ __forceinline__ double sxy() const { return p[5 * s]; }
};

__device__ __forceinline__ void store_vrec(double *base, int64_t s, int64_t i, const VertRec &r)
{
    double *p = base + i;
    p[0] = r.X;
    p[s] = r.Y;
    p[2 * s] = r.pc;
    p[3 * s] = r.p0;
    p[4 * s] = r.syx;
    p[5 * s] = r.sxy;
}

constexpr double kInvalidSlope = 1.0e30;
constexpr int kMomentOrder = 6;      // near-forward expansion order
constexpr int kNumMoments = 28;      // (6+1)(6+2)/2
// Angular half-width of the FP32C near-forward zone in radians of vertex
// phase.  Inside it every |q.r| <= kNearPhase and the edge sum cancels
// badly in FP32; the sixth-order moment expansion there truncates at
// kNearPhase^7/7! < 1.3e-8.
constexpr double kNearPhase = 0.25;

struct KParams {
    const DevBeam *beams;
    const DevVert *verts;
    const double *brec;        // [kBrecWords][brec_stride]
    const double *vrec;        // [kVrecWords][vrec_stride]
    int64_t brec_stride, vrec_stride;
    const double *moments;     // [n_beams][kNumMoments] c_pq = <x^p y^q>/(p! q!)
    const int32_t *vbeg;       // [n_beams+1]
    const int32_t *beam_off;   // [n_orient+1]
    const double *weight;      // [n_orient]
    const double *st, *ct, *sphi, *cphi, *vf;
    const int8_t *row_kind;    // [n_t] 0 regular, 1 polar (po_pole_kernel), 2 general
    int n_az, n_t;             // n_t = n_zen+1
    int row0, row1;            // zenith rows of this launch
    int n_orient;
    int orient_per_chunk;
    int tiles_per_row;
    // Output sets (size instances of a multi-size batch): set s owns the
    // orientations [s*orient_per_set, (s+1)*orient_per_set) and the chunks
    // [s*chunks_per_set, (s+1)*chunks_per_set).  One set: the whole batch.
    int orient_per_set;
    int chunks_per_set;
    // Work items (chunk, azimuth bin, zenith tile), chunk-major: the
    // persistent CTAs of po_diffract_kernel take them in order from *work.
    int *work;
    int n_items;
    WaveConst wc;
    double *partial;           // [n_chunks][16][G]
    double *partial_ns;        // [n_chunks][16][G] or null
};

// Orientation range [o0, o1) of an orientation chunk; chunks never span
// two output sets.
__device__ __forceinline__ void chunk_range(const KParams &P, int chunk, int &o0, int &o1)
{
    const int set = chunk / P.chunks_per_set;
    const int base = set * P.orient_per_set;
    o0 = base + (chunk - set * P.chunks_per_set) * P.orient_per_chunk;
    o1 = min(min(base + P.orient_per_set, P.n_orient), o0 + P.orient_per_chunk);
}

// ------------------------------------------------------------ pack kernel

// Size scaling of a staged instance (multi-size scan): the reference's
// ScalePreparedOrientation (TracerPOTotal.cpp:2682-2747) and the scaled
// packing of pack_prepared_gpu_beam (GpuDiffraction.cu:281-357): vertex
// coordinates and the beam centre times s, area times s^2, and the Jones
// matrix re-phased from the unphased one,
//   J_phased = sign * absorption(s) * J * exp(i k s path),
//   absorption(s) = mean over absorption paths L of (L > DBL_EPSILON ?
//                   exp(cAbs L s) : 1)   (GpuDiffraction.cu:257-271).
struct ScaleParams {
    const double *scales;       // [n_inst] or null (one instance, s = 1, no re-phasing)
    const double *raw;          // [n_beams][MBS_PO_RAW_STRIDE]
    const int64_t *abs_off;     // [n_beams+1] or null
    const double *abs_paths;
    double k_rephase;           // wave number of the re-phasing
    double abs_coeff;
};

struct PackParams {
    int64_t n_beams;            // beams of one instance
    int64_t n_verts;            // vertices of one instance
    const int64_t *vert_off;
    const double *vx, *vy, *syx, *sxy;
    const uint8_t *eflags;
    const double *geom;
    const uint8_t *bflags;
    ScaleParams sc;
    WaveConst wc;
    DevBeam *beams;
    DevVert *verts;
    double *brec;               // [kBrecWords][brec_stride], null: not built
    double *vrec;               // [kVrecWords][vrec_stride], null: not built
    int64_t brec_stride, vrec_stride;
    double *moments;            // null: not built
    int32_t *vbeg;
    int *status;   // set to 1 on a malformed beam
};

// Grid: x over groups of kPackBeams beams of one instance, y = instance.
// Instance i writes beams [i n_beams, (i+1) n_beams) and vertices
// [i n_verts, (i+1) n_verts) of the record arrays.
//
// A CTA packs 16 consecutive beams: their geometry and vertices (contiguous in
// the flat arrays) come into shared memory in coalesced loads, 8 lanes share
// a beam's reductions and moments (a lane per edge), and the records go out
// word by word, 16 beams side by side.  With one thread per beam the kernel
// took 59 us whatever the batch, the length of one thread's chain (about
// 4,000 FP64 operations of moment sums for a quadrangle, in local arrays),
// and 210 us for 89,000 beams; now 7 us for 80 beams, 30 us for 26,000 and,
// without the records that extinction does not read, 49 us for 89,000.
constexpr int kPackBeams = 16;
constexpr int kPackLanes = 8;
constexpr int kPackThreads = kPackBeams * kPackLanes;
constexpr int kDevWords = sizeof(DevBeam) / 8;

// Sum of v over the 8 lanes of a beam, the same value in every lane.
__device__ __forceinline__ double pack_sum(double v)
{
#pragma unroll
    for (int off = 1; off < kPackLanes; off <<= 1)
        v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// First index (over the lanes' candidates) of the largest value.
__device__ __forceinline__ void pack_argmax(double &v, int &i)
{
#pragma unroll
    for (int off = 1; off < kPackLanes; off <<= 1) {
        const double v2 = __shfl_xor_sync(0xffffffffu, v, off);
        const int i2 = __shfl_xor_sync(0xffffffffu, i, off);
        if (v2 > v || (v2 == v && i2 < i)) {
            v = v2;
            i = i2;
        }
    }
}

__global__ void __launch_bounds__(kPackThreads) po_pack_kernel(PackParams P)
{
    __shared__ double sg[kPackBeams * MBS_PO_GEOM_STRIDE];
    __shared__ double sd[kPackBeams][kDevWords];                     // DevBeam images
    __shared__ double svx[kPackBeams * kMaxNv], svy[kPackBeams * kMaxNv];
    __shared__ double sslab[kPackBeams][4];
    __shared__ int svo[kPackBeams + 1];
    __shared__ unsigned char svb[kPackBeams * kMaxNv];               // beam of a vertex
    const int64_t bl0 = (int64_t)blockIdx.x * kPackBeams;
    const int nb = (int)min((int64_t)kPackBeams, P.n_beams - bl0);
    const int inst = blockIdx.y;
    const int64_t ob = (int64_t)inst * P.n_beams, ov = (int64_t)inst * P.n_verts;
    const int64_t vg0 = P.vert_off[bl0];
    const int sub = threadIdx.x & (kPackLanes - 1), il = threadIdx.x / kPackLanes;
    for (int i = threadIdx.x; i <= nb; i += kPackThreads) {
        const int64_t v = P.vert_off[bl0 + i];
        svo[i] = (int)(v - vg0);
        if (i < nb || bl0 + nb == P.n_beams)   // the last group also writes the terminal offset
            P.vbeg[ob + bl0 + i] = (int32_t)(ov + v);
    }
    for (int i = threadIdx.x; i < nb * MBS_PO_GEOM_STRIDE; i += kPackThreads)
        sg[i] = P.geom[bl0 * MBS_PO_GEOM_STRIDE + i];
    __syncthreads();
    int bad = 0;
    for (int i = threadIdx.x; i < nb; i += kPackThreads) {
        const int nv = svo[i + 1] - svo[i];
        bad |= nv < 3 || nv > kMaxNv;
    }
    if (__syncthreads_or(bad)) {   // the whole batch is refused: no record is read
        if (threadIdx.x == 0)
            atomicExch(P.status, 1);
        return;
    }
    const double scl = P.sc.scales ? P.sc.scales[inst] : 1.0;
    const int nvs = svo[nb];
    for (int e = threadIdx.x; e < nvs; e += kPackThreads) {          // scaled vertices
        svx[e] = P.vx[vg0 + e] * scl;
        svy[e] = P.vy[vg0 + e] * scl;
    }
    const WaveConst &wc = P.wc;
    const double k = wc.k, kt = wc.k * kInvTwoPi;
    const bool has = il < nb;
    const double *g = sg + (has ? il : 0) * MBS_PO_GEOM_STRIDE;
    const int64_t bl = bl0 + (has ? il : 0);
    const int vo = svo[has ? il : 0], nv = svo[has ? il + 1 : 1] - vo;
    // a0 = bd.hor, b0 = bd.ver (GpuDiffraction.cu:301-302)
    const double a0 = g[MBS_PO_G_BD] * g[MBS_PO_G_HOR] + g[MBS_PO_G_BD + 1] * g[MBS_PO_G_HOR + 1]
                    + g[MBS_PO_G_BD + 2] * g[MBS_PO_G_HOR + 2];
    const double b0 = g[MBS_PO_G_BD] * g[MBS_PO_G_VER] + g[MBS_PO_G_BD + 1] * g[MBS_PO_G_VER + 1]
                    + g[MBS_PO_G_BD + 2] * g[MBS_PO_G_VER + 2];
    if (has) {
        double *d = sd[il];
        for (int w = sub; w < 32; w += kPackLanes) {   // the words that are copied or scaled
            if (w >= 2 && w < 8)
                d[w] = g[MBS_PO_G_HOR + (w - 2)];                    // h, v
            else if (w >= 8 && w < 11)
                d[w] = g[MBS_PO_G_CEN + (w - 8)] * scl;
            else if (w >= 12 && w < 24)
                d[w] = g[MBS_PO_G_NT + (w - 12)];
            else if (w >= 24 && !P.sc.scales)
                d[w] = g[MBS_PO_G_JP + (w - 24)];
        }
        for (int e = sub; e < nv; e += kPackLanes)
            svb[vo + e] = (unsigned char)il;
        if (sub == 0) {
            d[0] = a0;
            d[1] = b0;
            d[11] = g[MBS_PO_G_AREA] * (scl * scl);
            d[32] = g[MBS_PO_G_OPATH] * scl;
            d[33] = 0.0;
            d[34] = __hiloint2double(nv, (int32_t)(ov + vg0 + vo));
        }
        if (sub == 1 && P.sc.scales) {
            const double *raw = P.sc.raw + bl * MBS_PO_RAW_STRIDE;
            double sn, cs;
            sincos(P.sc.k_rephase * raw[MBS_PO_R_PATH] * scl, &sn, &cs);
            double absorption = 1.0;
            if (P.sc.abs_off) {
                const int64_t p0 = P.sc.abs_off[bl], p1 = P.sc.abs_off[bl + 1];
                if (p1 > p0) {
                    double sum = 0.0;
                    for (int64_t a = p0; a < p1; ++a) {
                        const double path = P.sc.abs_paths[a];
                        sum += (path > 2.220446049250313e-16) ? exp(P.sc.abs_coeff * path * scl) : 1.0;
                    }
                    absorption = sum / (double)(p1 - p0);
                }
            }
            const double f = raw[MBS_PO_R_SIGN] * absorption;
            for (int i = 0; i < 4; ++i) {
                const double jr = raw[MBS_PO_R_J + 2 * i], ji = raw[MBS_PO_R_J + 2 * i + 1];
                d[24 + 2 * i] = f * (jr * cs - ji * sn);
                d[25 + 2 * i] = f * (jr * sn + ji * cs);
            }
        }
    }
    __syncthreads();   // vertices and DevBeam words are in shared memory
    const double *vx = svx + vo, *vy = svy + vo;
    // Small-phase candidates.  The reference's moment branch needs every
    // vertex phase |k(A x_v + B y_v)| <= 1e-3 (HandlerPO_fast.h:161-173); in
    // particular for the vertex a farthest from the origin and the vertex b
    // farthest from the line through a.  Those two slabs in (A, B), widened
    // by 25% for rounding, bound the candidates tightly even for sliver
    // apertures; candidates take the exact FP64 test.
    double r2 = -1.0;
    int ia = kMaxNv;
    for (int e = sub; e < nv; e += kPackLanes) {
        const double v = vx[e] * vx[e] + vy[e] * vy[e];
        if (v > r2) {
            r2 = v;
            ia = e;
        }
    }
    pack_argmax(r2, ia);
    if (ia >= nv)
        ia = 0;                               // every vertex NaN
    const double xa = vx[ia], ya = vy[ia];
    double cmax = -1.0;
    int ib = kMaxNv;
    for (int e = sub; e < nv; e += kPackLanes) {
        const double v = fabs(xa * vy[e] - ya * vx[e]);
        if (v > cmax) {
            cmax = v;
            ib = e;
        }
    }
    pack_argmax(cmax, ib);
    const int ib0 = ia == 0 ? 1 : 0;
    if (ib >= nv || !(cmax > fabs(xa * vy[ib0] - ya * vx[ib0])))
        ib = ib0;
    // FP32C near-forward zone: |q| rmax <= kNearPhase, so every vertex phase
    // is within kNearPhase and the moment expansion converges; 0.9 keeps the
    // zone inside that bound after the FP32 rounding of A and B.
    const double kr2 = k * k * fmax(0.0, r2);
    const float near2 = (float)((kr2 > 1e-300) ? 0.9 * kNearPhase * kNearPhase / kr2 : 0.0);
    if (has && sub == 0) {
        const double slab_scale = k / (1.25 * kSmallPhase);
        sslab[il][0] = xa * slab_scale;
        sslab[il][1] = ya * slab_scale;
        sslab[il][2] = vx[ib] * slab_scale;
        sslab[il][3] = vy[ib] * slab_scale;
        sd[il][35] = __hiloint2double(__float_as_int(near2), P.bflags[bl]);
    }
    __syncthreads();   // the DevBeam images and slabs are complete
    // general records: 16 consecutive beams are contiguous
    double *dst = reinterpret_cast<double *>(P.beams + ob + bl0);
    for (int i = threadIdx.x; i < nb * kDevWords; i += kPackThreads)
        dst[i] = sd[i / kDevWords][i % kDevWords];
    // vertices: general records and phase coefficients
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    for (int e = threadIdx.x; e < nvs; e += kPackThreads) {
        const double *d = sd[svb[e]];
        const double x = svx[e], y = svy[e];
        const bool internal = !(__double2loint(d[35]) & MBS_PO_BEAM_EXTERNAL);
        const uint8_t f = P.eflags[vg0 + e];
        const double syx = P.syx[vg0 + e], sxy = P.sxy[vg0 + e];
        DevVert dv;
        dv.x = x;
        dv.y = y;
        dv.syx = (f & MBS_PO_EDGE_VALID_X) ? syx : nan;
        dv.sxy = (f & MBS_PO_EDGE_VALID_Y) ? sxy : nan;
        P.verts[ov + vg0 + e] = dv;
        if (P.vrec) {
            VertRec vr;
            vr.X = kt * (d[2] * x + d[5] * y) + (internal ? kt * d[8] : 0.0);
            vr.Y = kt * (d[3] * x + d[6] * y) + (internal ? kt * d[9] : 0.0);
            vr.pc = kt * (d[4] * x + d[7] * y) + (internal ? kt * d[10] : 0.0);
            vr.p0 = kt * (d[0] * x + d[1] * y);
            vr.syx = (f & MBS_PO_EDGE_VALID_X) ? syx : kInvalidSlope;
            vr.sxy = (f & MBS_PO_EDGE_VALID_Y) ? sxy : kInvalidSlope;
            store_vrec(P.vrec, P.vrec_stride, ov + vg0 + e, vr);
        }
    }
    if (P.brec) {
        // beam records, a word of 16 beams at a time: A/B coefficients, the
        // entries of complWave (X J) as (row, column) pairs, slabs, counts
        constexpr int kItems = 8 + 20 + 4 + 2;
        for (int i = threadIdx.x; i < kItems * kPackBeams; i += kPackThreads) {
            const int w = i / kPackBeams, j = i - w * kPackBeams;
            if (j >= nb)
                continue;
            const double *d = sd[j];
            double *out = P.brec + ob + bl0 + j;
            if (w < 8) {   // h0 h1 h2 a0 v0 v1 v2 b0
                out[w * P.brec_stride] = d[(w & 3) == 3 ? w >> 2 : 2 + 3 * (w >> 2) + (w & 3)];
            } else if (w < 28) {
                // group q of X1, X2, Y1, Y2, Z (rows r of the real 2x2
                // matrix X, see kBrecWords), entry e = 2 r + c of X J
                const int q = (w - 8) >> 2, e = (w - 8) & 3, r = e >> 1, c = e & 1;
                const int comp = q == 4 ? 2 : q & 1;       // x, y or z component
                // vectors of row 0 / 1: (NT, NP) or (DT, DP); sign per group and row
                const bool dt = (q < 2) == (r == 1);
                const double sgn = q == 4 ? -1.0 : q < 2 ? ((q == 0) == (r == 0) ? 1.0 : -1.0) : 1.0;
                const double *T = d + 12 + ((q == 4 ? r == 0 : dt) ? 6 : 0) + comp;
                const double x0 = sgn * T[0], x1 = sgn * T[3];
                const double *jp = d + 24;
                const double mr = x0 * jp[2 * c] + x1 * jp[4 + 2 * c];
                const double mi = x0 * jp[2 * c + 1] + x1 * jp[5 + 2 * c];
                out[(8 + q * 8 + 2 * e) * P.brec_stride] = wc.cw_re * mr - wc.cw_im * mi;
                out[(9 + q * 8 + 2 * e) * P.brec_stride] = wc.cw_re * mi + wc.cw_im * mr;
            } else if (w < 32) {
                out[(48 + w - 28) * P.brec_stride] = sslab[j][w - 28];
            } else if (w == 32) {
                out[52 * P.brec_stride] = __hiloint2double(__double2loint(d[34]), __double2hiint(d[35]));
            } else {
                out[53 * P.brec_stride] = __hiloint2double(__double2loint(d[35]), __double2hiint(d[34]));
            }
        }
    }
    if (!P.moments)
        return;
    // Polygon moments I(p,q) = integral of x^p y^q over the aperture, by
    // Green's theorem over the edges (exact for polygons), normalised by
    // the signed area: c_pq = <x^p y^q> / (p! q!).  Per edge (i -> j):
    //   I(p,q) += p! q!/(p+q+2)! (x_i y_j - x_j y_i) H(p,q),
    //   H(p,q) = sum_{a<=p, c<=q} C(a+c, c) C(p+q-a-c, q-c) x_i^a x_j^(p-a) y_i^c y_j^(q-c),
    // the coefficients of 1 / ((1 - s x_i - t y_i) (1 - s x_j - t y_j)), so with
    // those of 1 / (1 - s x_j - t y_j), G, two recurrences give each degree from
    // the one below (140 operations an edge for all 28 moments; the sums
    // written out are about 1,000):
    //   G(p,q) = x_j G(p-1,q) + y_j G(p,q-1),  H(p,q) = x_i H(p-1,q) + y_i H(p,q-1) + G(p,q).
    double I[kNumMoments];
#pragma unroll
    for (int i = 0; i < kNumMoments; ++i)
        I[i] = 0.0;
    double minX = 1e300, maxX = -1e300, minY = 1e300, maxY = -1e300;
    for (int e = sub; e < nv; e += kPackLanes) {
        const int en = (e + 1 < nv) ? e + 1 : 0;
        const double xi = vx[e], yi = vy[e], xj = vx[en], yj = vy[en];
        minX = fmin(minX, xi); maxX = fmax(maxX, xi);
        minY = fmin(minY, yi); maxY = fmax(maxY, yi);
        const double cross = xi * yj - xj * yi;
        double Gd[kMomentOrder + 1], Hd[kMomentOrder + 1];   // degree n: p = n .. 0
        Gd[0] = Hd[0] = 1.0;
        I[0] += cross;
#pragma unroll
        for (int n = 1; n <= kMomentOrder; ++n) {
            // entry m (p = n - m) from entries m (p - 1) and m - 1 (q - 1) of
            // degree n - 1; from the last entry down, so each is read before
            // it is overwritten
#pragma unroll
            for (int m = n; m >= 0; --m) {
                const double gx = m < n ? Gd[m] : 0.0, gy = m > 0 ? Gd[m - 1] : 0.0;
                const double hx = m < n ? Hd[m] : 0.0, hy = m > 0 ? Hd[m - 1] : 0.0;
                Gd[m] = xj * gx + yj * gy;
                Hd[m] = xi * hx + yi * hy + Gd[m];
                I[n * (n + 1) / 2 + m] += cross * Hd[m];
            }
        }
    }
#pragma unroll
    for (int off = 1; off < kPackLanes; off <<= 1) {
        minX = fmin(minX, __shfl_xor_sync(0xffffffffu, minX, off));
        maxX = fmax(maxX, __shfl_xor_sync(0xffffffffu, maxX, off));
        minY = fmin(minY, __shfl_xor_sync(0xffffffffu, minY, off));
        maxY = fmax(maxY, __shfl_xor_sync(0xffffffffu, maxY, off));
    }
    __syncthreads();   // the DevBeam images are read: sd takes the moments
#pragma unroll
    for (int i = 0; i < kNumMoments; ++i)
        I[i] = pack_sum(I[i]);
    const double area2 = I[0];
    const bool degenerate = fabs(area2) <= 0x1p-40 * fmax((maxX - minX) * (maxY - minY), 2.2250738585072014e-308);
    if (has && sub == 0) {
        double f = 1.0 / (0.5 * area2);   // times 1 / (n + 2)!
#pragma unroll
        for (int n = 0; n <= kMomentOrder; ++n) {
            f /= (double)(n + 2);
#pragma unroll
            for (int m = 0; m <= n; ++m)
                sd[il][n * (n + 1) / 2 + m] = degenerate ? (n == 0 ? 1.0 : 0.0) : I[n * (n + 1) / 2 + m] * f;
        }
    }
    __syncthreads();
    double *mom = P.moments + (ob + bl0) * kNumMoments;
    for (int i = threadIdx.x; i < nb * kNumMoments; i += kPackThreads)
        mom[i] = sd[i / kNumMoments][i % kNumMoments];
}

// ----------------------------------------------------- general FP64 path
// Used for the rare (beam, direction) pairs that leave the vectorised path:
// irregular polar rows, near-singular FP32 edges and the small-phase
// candidates of the FP64 kernel.  Everything is recomputed in FP64 from the
// general records, as compute_beam_jones_context does
// (GpuDiffraction.cu:1064-1165).

struct DirFull {
    double st, ct, cp, sp;
    double dir[3], vf[3], vt[3], u[3], w[3];
};

__device__ __forceinline__ void cross3(const double *a, const double *b, double *o)
{
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ void dir_full(const KParams &P, int p, int t, DirFull &d)
{
    d.st = P.st[t];
    d.ct = P.ct[t];
    d.cp = P.cphi[p];
    d.sp = P.sphi[p];
    d.dir[0] = d.st * d.cp;
    d.dir[1] = d.st * d.sp;
    d.dir[2] = -d.ct;
    const double *vfp = P.vf + ((size_t)p * P.n_t + t) * 3;
    d.vf[0] = vfp[0]; d.vf[1] = vfp[1]; d.vf[2] = vfp[2];
    cross3(d.vf, d.dir, d.u);                 // u = vf x dir
    const double l2 = d.u[0] * d.u[0] + d.u[1] * d.u[1] + d.u[2] * d.u[2];
    const double il = (l2 > 1e-30) ? rsqrt(l2) : 1.0;   // transverse_basis_gpu
    d.vt[0] = d.u[0] * il; d.vt[1] = d.u[1] * il; d.vt[2] = d.u[2] * il;
    cross3(d.vt, d.dir, d.w);                 // w = vt x dir
}

// One beam's Jones contribution d[8] to one direction in FP64.  Returns
// false when the reference would skip the beam (NaN integral).
// `singular` = false drops nearly singular edges (|C_e| <= eps1) instead of
// taking their stable quotient, the reference's singularCorrection = 0;
// `common` = false leaves out an internal beam's common phase.
__device__ __noinline__ bool beam_general(const DevBeam &g, const DevVert *gv, const DirFull &dc,
                                          const WaveConst &wc, double *d, bool singular = true,
                                          bool common = true)
{
    const double k = wc.k;
    const double a_sin = -dc.cp * g.h[0] - dc.sp * g.h[1];
    const double b_sin = -dc.cp * g.v[0] - dc.sp * g.v[1];
    const double A = fma(dc.st, a_sin, fma(dc.ct, g.h[2], g.a0));
    const double B = fma(dc.st, b_sin, fma(dc.ct, g.v[2], g.b0));
    const bool internal = common && !(g.flags & MBS_PO_BEAM_EXTERNAL);
    const double cm = internal ? -k * (dc.st * (dc.cp * g.c[0] + dc.sp * g.c[1]) + dc.ct * (-g.c[2])) : 0.0;
    const DevVert *v = gv + g.vbeg;
    const int nv = g.nv;
    double fr, fi, pr, pi;
    if (small_phase_factor(v, nv, A, B, k, pr, pi)) {
        const double sgn = wc.legacy_sign ? 1.0 : -1.0;
        const double ar = sgn * wc.icw_re * g.area, ai = sgn * wc.icw_im * g.area;
        fr = ar * pr - ai * pi;
        fi = ar * pi + ai * pr;
        if (internal) {
            double s, c;
            sincos_rad(cm, s, c);
            const double tr = fr * c - fi * s;
            fi = fr * s + fi * c;
            fr = tr;
        }
    } else {
        const bool useX = fabs(B) > fabs(A);
        const double qx = k * A * kInvTwoPi, qy = k * B * kInvTwoPi, cmt = cm * kInvTwoPi;
        double s0, c0;
        sincos_turns(fma(qx, v[0].x, fma(qy, v[0].y, cmt)), s0, c0);
        double cprev = c0, sprev = s0, sr = 0.0, si = 0.0;
        for (int e = 0; e < nv; ++e) {
            const int en = (e + 1 < nv) ? e + 1 : 0;
            double cn = c0, sn = s0;
            if (en != 0)
                sincos_turns(fma(qx, v[en].x, fma(qy, v[en].y, cmt)), sn, cn);
            const double coef = useX ? fma(v[e].syx, B, A) : fma(v[e].sxy, A, B);
            const double ac = fabs(coef);
            if (ac > wc.eps1) {
                const double inv = 1.0 / coef;
                sr = fma(cn - cprev, inv, sr);
                si = fma(sn - sprev, inv, si);
            } else if (singular && ac <= wc.eps1) {   // valid, nearly singular edge (NaN: invalid edge)
                const double delta = useX ? (v[en].x - v[e].x) : (v[en].y - v[e].y);
                stable_edge(cprev, sprev, delta, coef, k, sr, si);
            }
            cprev = cn;
            sprev = sn;
        }
        const double m = useX ? 1.0 / B : -1.0 / A;
        sr *= m;
        si *= m;
        fr = wc.cw_re * sr - wc.cw_im * si;
        fi = wc.cw_re * si + wc.cw_im * sr;
    }
    if (isnan(fr))
        return false;
    // rotation (GpuDiffraction.cu:831-856) with w = vt x dir, u = vf x dir:
    // (dir x NT).vt = NT.w and (dir x NT).vf = NT.u; the dir(dir.nxDT)
    // terms vanish since vt and vf are orthogonal to dir.
    const double *NT = g.rot, *NP = g.rot + 3, *DT = g.rot + 6, *DP = g.rot + 9;
    const double r00 = NT[0] * dc.w[0] + NT[1] * dc.w[1] + NT[2] * dc.w[2] + DT[0] * dc.vt[0] + DT[1] * dc.vt[1] + DT[2] * dc.vt[2];
    const double r01 = NP[0] * dc.w[0] + NP[1] * dc.w[1] + NP[2] * dc.w[2] + DP[0] * dc.vt[0] + DP[1] * dc.vt[1] + DP[2] * dc.vt[2];
    const double r10 = NT[0] * dc.u[0] + NT[1] * dc.u[1] + NT[2] * dc.u[2] + DT[0] * dc.vf[0] + DT[1] * dc.vf[1] + DT[2] * dc.vf[2];
    const double r11 = NP[0] * dc.u[0] + NP[1] * dc.u[1] + NP[2] * dc.u[2] + DP[0] * dc.vf[0] + DP[1] * dc.vf[1] + DP[2] * dc.vf[2];
    const double *jp = g.jp;
    const double s00r = fr * r00, s00i = fi * r00, s01r = fr * r01, s01i = fi * r01;
    const double s10r = fr * r10, s10i = fi * r10, s11r = fr * r11, s11i = fi * r11;
    d[0] = s00r * jp[0] - s00i * jp[1] + s01r * jp[4] - s01i * jp[5];
    d[1] = s00r * jp[1] + s00i * jp[0] + s01r * jp[5] + s01i * jp[4];
    d[2] = s00r * jp[2] - s00i * jp[3] + s01r * jp[6] - s01i * jp[7];
    d[3] = s00r * jp[3] + s00i * jp[2] + s01r * jp[7] + s01i * jp[6];
    d[4] = s10r * jp[0] - s10i * jp[1] + s11r * jp[4] - s11i * jp[5];
    d[5] = s10r * jp[1] + s10i * jp[0] + s11r * jp[5] + s11i * jp[4];
    d[6] = s10r * jp[2] - s10i * jp[3] + s11r * jp[6] - s11i * jp[7];
    d[7] = s10r * jp[3] + s10i * jp[2] + s11r * jp[7] + s11i * jp[6];
    return true;
}

// FP32C near-forward zone: the aperture integral from the sixth-order
// moment expansion in FP64,  F = areaLimit sum_pq i^(p+q) qx^p qy^q c_pq,
// times the internal-beam common phase, returned as the edge-sum
// equivalent s = F / complWave so the caller applies P0 + cos t Pc + sin t Ps.
__device__ __noinline__ void near_forward_s(const DevBeam &g, const double *mom, double st, double ct,
                                            double cp, double sp, const WaveConst &wc,
                                            float &sr, float &si)
{
    const double k = wc.k;
    const double a_sin = -cp * g.h[0] - sp * g.h[1];
    const double b_sin = -cp * g.v[0] - sp * g.v[1];
    const double qx = k * fma(st, a_sin, fma(ct, g.h[2], g.a0));
    const double qy = k * fma(st, b_sin, fma(ct, g.v[2], g.b0));
    double px[kMomentOrder + 1], py[kMomentOrder + 1];
    px[0] = 1.0; py[0] = 1.0;
    for (int i = 1; i <= kMomentOrder; ++i) {
        px[i] = px[i - 1] * qx;
        py[i] = py[i - 1] * qy;
    }
    double re = 0.0, im = 0.0;
    int idx = 0;
    for (int n = 0; n <= kMomentOrder; ++n) {
        double s = 0.0;
        for (int p = n; p >= 0; --p, ++idx)
            s = fma(mom[idx], px[p] * py[n - p], s);
        switch (n & 3) {
        case 0: re += s; break;
        case 1: im += s; break;
        case 2: re -= s; break;
        default: im -= s; break;
        }
    }
    const double sgn = wc.legacy_sign ? 1.0 : -1.0;
    const double ar = sgn * wc.icw_re * g.area, ai = sgn * wc.icw_im * g.area;
    double fr = ar * re - ai * im, fi = ar * im + ai * re;
    if (!(g.flags & MBS_PO_BEAM_EXTERNAL)) {
        const double cm = -k * (st * (cp * g.c[0] + sp * g.c[1]) + ct * (-g.c[2]));
        double s, c;
        sincos_rad(cm, s, c);
        const double tr = fr * c - fi * s;
        fi = fr * s + fi * c;
        fr = tr;
    }
    // s = F / complWave
    const double n2 = wc.cw_re * wc.cw_re + wc.cw_im * wc.cw_im;
    sr = (float)((fr * wc.cw_re + fi * wc.cw_im) / n2);
    si = (float)((fi * wc.cw_re - fr * wc.cw_im) / n2);
}

// ----------------------------------------------- shared-memory records
// Per (beam, azimuth of the CTA), laid out for 16-byte vector loads: every
// lane of a warp reads the same record (a broadcast), so a beam costs ten
// (FP32C) or eighteen (FP64) shared loads per thread for all DPT directions.
//   A(t) = sin t a[0] + cos t a[1] + a[2],  B(t) = sin t a[3] + cos t a[4] + a[5]
//   P0, Pc, Ps: complWave (R J) parts, 4 complex entries each (see kBrecWords)
//   slab: small-phase candidate test, nearr2: FP32C near-forward zone

//   zone: nonzero when some direction of the CTA's zenith tile may fall in
//   the near-forward zone or pass the slab test (tile_zone_possible)

template <typename T>
struct BeamRegs {
    T a[6];
    T slab[4];
    float nearr2;
    int nv, vs, gbeam, zone;
    bool external;
};

template <typename T>
struct SBeamRaw;

template <>
struct __align__(16) SBeamRaw<float> {
    float4 q[10];   // a0 a3 a1 a4 | a2 a5 slab0 slab1 | slab2 slab3 nearr2 nv | P[24] | gbeam vs zone external
                    // ((a0, a3), (a1, a4), (a2, a5): operand pairs of the packed A, B;
                    // P entries 2h, 2h+1 of P0, Pc, Ps as (re, re, im, im): the
                    // real and the imaginary operand pairs of the packed Jones update)
};

template <>
struct __align__(16) SBeamRaw<double> {
    double2 q[18];  // a0a1 a2a3 a4a5 | slab | slab | P[24] | (zone + 2 external,nv) (gbeam,vs)
                    // (FP64 has no near-forward zone: the nearr2 word holds the flags)
};

// The zenith tile of a work item seen from the stage fill: every direction
// w = (sin t, cos t) the CTA evaluates lies within del of wc = (stc, ctc).
struct TileZone {
    double stc, ctc, del;
};

// Whether some direction of the tile can pass the per-pair zone tests of
// the hot loop for a beam with azimuth-folded coefficients a (A = sin t a0
// + cos t a1 + a2, B = sin t a3 + cos t a4 + a5): the FP32C near-forward
// test A^2 + B^2 <= nearr2 and the slab test |A s0 + B s1| <= 1 and
// |A s2 + B s3| <= 1.  A, B and the slab forms are affine in w, so over
// the tile they stay within |gradient| del of their values at wc.  The
// margins cover the hot loop's FP32 rounding of the coefficients, of
// sin t, cos t and of the sums (below 2.5e-7 of sum |a_i| for A and B), so
// a tile reported clear holds no pair that the per-pair tests would mark,
// and skipping those tests there leaves every result unchanged.
__device__ __forceinline__ bool tile_zone_possible(const double *a, const double *slab, float nearr2,
                                                   bool f32, const TileZone &z)
{
    const double Ac = fma(a[0], z.stc, fma(a[1], z.ctc, a[2]));
    const double Bc = fma(a[3], z.stc, fma(a[4], z.ctc, a[5]));
    const double amax = fabs(a[0]) + fabs(a[1]) + fabs(a[2]) + fabs(a[3]) + fabs(a[4]) + fabs(a[5]);
    const double marg = 1e-6 * amax + 1e-300;
    if (f32) {
        const double gq = sqrt(a[0] * a[0] + a[1] * a[1] + a[3] * a[3] + a[4] * a[4]);
        const double ql = sqrt(Ac * Ac + Bc * Bc) - gq * z.del - 2.0 * marg;
        if (!(ql > 0.0 && ql * ql > (double)nearr2 * (1.0 + 1e-5)))
            return true;
    }
    bool clear = false;
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        const double s0 = slab[k], s1 = slab[k + 1];
        const double uc = fma(Ac, s0, Bc * s1);
        const double g0 = fma(a[0], s0, a[3] * s1), g1 = fma(a[1], s0, a[4] * s1);
        const double mu = 2.0 * marg * (fabs(s0) + fabs(s1)) + 1e-6;
        clear = clear || fabs(uc) - sqrt(g0 * g0 + g1 * g1) * z.del > 1.0 + mu;
    }
    return !clear;
}

template <typename T>
struct SVertRaw;

template <>
struct __align__(16) SVertRaw<float> {
    double2 q[2];   // (ps, pc) (p0, slopes syx|sxy as two floats)
};

template <>
struct __align__(16) SVertRaw<double> {
    double2 q[3];   // (ps, pc) (p0, syx) (sxy, unused)
};

// Beams a stage holds.  FP64: 64 whatever the CTA (a record is 288 bytes, and
// the sine table takes 8 KB).  FP32C: the stage ends set where the FP32 block
// sums are folded, so shapes that must agree bit for bit have the same.
template <typename T>
constexpr int default_stage(int tpb) { return sizeof(T) == 8 ? 64 : tpb; }

template <typename T, int BEAMS>
struct StageCfg {
    static constexpr int kBeams = BEAMS;
    static constexpr int kVerts = 4 * kBeams;
    static constexpr size_t kBytes = kBeams * sizeof(SBeamRaw<T>) + kVerts * sizeof(SVertRaw<T>);
};

__device__ __forceinline__ void fill_beam(const BrecRef &r, double cp, double sp, int vs, int gbeam,
                                          const TileZone &z, SBeamRaw<float> &s)
{
    float a[6], P[24];
    const double ad[6] = {-(cp * r.ab(0) + sp * r.ab(1)), r.ab(2), r.ab(3),
                          -(cp * r.ab(4) + sp * r.ab(5)), r.ab(6), r.ab(7)};
    const double sl[4] = {r.slab(0), r.slab(1), r.slab(2), r.slab(3)};
    const int zone = tile_zone_possible(ad, sl, r.nearr2(), true, z) ? 1 : 0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
        a[i] = (float)ad[i];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        P[e] = (float)(sp * r.Q(e) + cp * r.Q(8 + e));
        P[8 + e] = (float)(-(cp * r.Q(16 + e) + sp * r.Q(24 + e)));
        P[16 + e] = (float)r.Q(32 + e);
    }
    s.q[0] = make_float4(a[0], a[3], a[1], a[4]);
    s.q[1] = make_float4(a[2], a[5], (float)sl[0], (float)sl[1]);
    s.q[2] = make_float4((float)sl[2], (float)sl[3], r.nearr2(), __int_as_float(r.nv()));
#pragma unroll
    for (int i = 0; i < 6; ++i)
        s.q[3 + i] = make_float4(P[4 * i], P[4 * i + 2], P[4 * i + 1], P[4 * i + 3]);
    s.q[9] = make_float4(__int_as_float(gbeam), __int_as_float(vs), __int_as_float(zone),
                         __int_as_float(r.external() ? 1 : 0));
}

__device__ __forceinline__ void fill_beam(const BrecRef &r, double cp, double sp, int vs, int gbeam,
                                          const TileZone &z, SBeamRaw<double> &s)
{
    const double ad[6] = {-(cp * r.ab(0) + sp * r.ab(1)), r.ab(2), r.ab(3),
                          -(cp * r.ab(4) + sp * r.ab(5)), r.ab(6), r.ab(7)};
    const double sl[4] = {r.slab(0), r.slab(1), r.slab(2), r.slab(3)};
    const int zone = tile_zone_possible(ad, sl, 0.f, false, z) ? 1 : 0;
    s.q[0] = make_double2(ad[0], ad[1]);
    s.q[1] = make_double2(ad[2], ad[3]);
    s.q[2] = make_double2(ad[4], ad[5]);
    s.q[3] = make_double2(sl[0], sl[1]);
    s.q[4] = make_double2(sl[2], sl[3]);
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
        s.q[5 + e / 2] = make_double2(sp * r.Q(e) + cp * r.Q(8 + e), sp * r.Q(e + 1) + cp * r.Q(9 + e));
        s.q[9 + e / 2] = make_double2(-(cp * r.Q(16 + e) + sp * r.Q(24 + e)),
                                      -(cp * r.Q(17 + e) + sp * r.Q(25 + e)));
        s.q[13 + e / 2] = make_double2(r.Q(32 + e), r.Q(33 + e));
    }
    s.q[17] = make_double2(__hiloint2double(r.nv(), zone + (r.external() ? 2 : 0)), __hiloint2double(vs, gbeam));
}

// FP32C: p0 carries the range-reduction constant 1.5*2^29 + 1/2, so the
// phase sum st ps + ct pc + p0 lands directly in [2^29, 2^30), where the low
// 23 mantissa bits hold frac(u + 1/2) (three roundings of at most 2^-24 turn).
__device__ __forceinline__ void fill_vert(const VrecRef &r, double cp, double sp, SVertRaw<float> &w)
{
    w.q[0] = make_double2(-(cp * r.X() + sp * r.Y()), r.pc());
    w.q[1] = make_double2(r.p0() + (kMagic29 + 0.5),
                          __hiloint2double(__float_as_int((float)r.sxy()), __float_as_int((float)r.syx())));
}

__device__ __forceinline__ void fill_vert(const VrecRef &r, double cp, double sp, SVertRaw<double> &w)
{
    w.q[0] = make_double2(-(cp * r.X() + sp * r.Y()), r.pc());
    w.q[1] = make_double2(r.p0(), r.syx());
    w.q[2] = make_double2(r.sxy(), 0.0);
}

__device__ __forceinline__ void load_beam(const SBeamRaw<float> &s, BeamRegs<float> &b)
{
    const float4 q0 = s.q[0], q1 = s.q[1], q2 = s.q[2], q9 = s.q[9];
    b.a[0] = q0.x; b.a[3] = q0.y; b.a[1] = q0.z; b.a[4] = q0.w; b.a[2] = q1.x; b.a[5] = q1.y;
    b.slab[0] = q1.z; b.slab[1] = q1.w; b.slab[2] = q2.x; b.slab[3] = q2.y;
    b.nearr2 = q2.z;
    b.nv = __float_as_int(q2.w);
    b.gbeam = __float_as_int(q9.x);
    b.vs = __float_as_int(q9.y);
    b.zone = __float_as_int(q9.z);
    b.external = __float_as_int(q9.w) != 0;
}

__device__ __forceinline__ void load_beam(const SBeamRaw<double> &s, BeamRegs<double> &b)
{
    const double2 q0 = s.q[0], q1 = s.q[1], q2 = s.q[2], q3 = s.q[3], q4 = s.q[4], q17 = s.q[17];
    b.a[0] = q0.x; b.a[1] = q0.y; b.a[2] = q1.x; b.a[3] = q1.y; b.a[4] = q2.x; b.a[5] = q2.y;
    b.slab[0] = q3.x; b.slab[1] = q3.y; b.slab[2] = q4.x; b.slab[3] = q4.y;
    b.nearr2 = 0.f;
    b.zone = __double2loint(q17.x) & 1;
    b.external = (__double2loint(q17.x) & 2) != 0;
    b.nv = __double2hiint(q17.x);
    b.vs = __double2hiint(q17.y);
    b.gbeam = __double2loint(q17.y);
}

__device__ __forceinline__ void load_P(const SBeamRaw<float> &s, float *P)
{
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const float4 q = s.q[3 + i];
        P[4 * i] = q.x; P[4 * i + 1] = q.z; P[4 * i + 2] = q.y; P[4 * i + 3] = q.w;
    }
}

__device__ __forceinline__ void load_P(const SBeamRaw<double> &s, double *P)
{
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        const double2 q = s.q[5 + i];
        P[2 * i] = q.x; P[2 * i + 1] = q.y;
    }
}

// P0, Pc, Ps entries 2h and 2h+1 of an FP32C beam record as (re 2h, re 2h+1)
// and (im 2h, im 2h+1) operand pairs, straight from the record's layout.
__device__ __forceinline__ void load_P_packed(const SBeamRaw<float> &s, int h, float2 &p0r, float2 &p0i,
                                              float2 &pcr, float2 &pci, float2 &psr, float2 &psi)
{
    const float4 a = s.q[3 + h], b = s.q[5 + h], c = s.q[7 + h];
    p0r = make_float2(a.x, a.y); p0i = make_float2(a.z, a.w);
    pcr = make_float2(b.x, b.y); pci = make_float2(b.z, b.w);
    psr = make_float2(c.x, c.y); psi = make_float2(c.z, c.w);
}

// The same of an FP64 record, (re, im) each.
__device__ __forceinline__ void load_P_pair(const SBeamRaw<double> &s, int h, double *p0, double *pc,
                                            double *ps)
{
    const double2 a0 = s.q[5 + 2 * h], a1 = s.q[6 + 2 * h];
    const double2 b0 = s.q[9 + 2 * h], b1 = s.q[10 + 2 * h];
    const double2 c0 = s.q[13 + 2 * h], c1 = s.q[14 + 2 * h];
    p0[0] = a0.x; p0[1] = a0.y; p0[2] = a1.x; p0[3] = a1.y;
    pc[0] = b0.x; pc[1] = b0.y; pc[2] = b1.x; pc[3] = b1.y;
    ps[0] = c0.x; ps[1] = c0.y; ps[2] = c1.x; ps[3] = c1.y;
}

struct VertRegs {
    double ps, pc, p0;
};

__device__ __forceinline__ void load_vert(const SVertRaw<float> &w, VertRegs &v, float &syx, float &sxy)
{
    const double2 q0 = w.q[0], q1 = w.q[1];
    v.ps = q0.x; v.pc = q0.y; v.p0 = q1.x;
    syx = __int_as_float(__double2loint(q1.y));
    sxy = __int_as_float(__double2hiint(q1.y));
}

__device__ __forceinline__ void load_vert(const SVertRaw<double> &w, VertRegs &v, double &syx, double &sxy)
{
    const double2 q0 = w.q[0], q1 = w.q[1], q2 = w.q[2];
    v.ps = q0.x; v.pc = q0.y; v.p0 = q1.x;
    syx = q1.y;
    sxy = q2.x;
}

// Vertex phasor (cos, sin) of 2 pi u, u = st ps + ct pc + p0 in turns.
__device__ __forceinline__ void vertex_phasor(double st, double ct, const VertRegs &w, double &s,
                                              double &c)
{
    sincos_turns(fma(st, w.ps, fma(ct, w.pc, w.p0)), s, c);
}

// FP32C: the offset sum (p0 holds 1.5*2^29 + 1/2, see fill_vert) leaves
// frac(u + 1/2) in the low 23 mantissa bits; as a float y = 1.f in [1, 2),
// 2 pi (y - 3/2) = y 2 pi - 3 pi is the reduced angle in [-pi, pi) (one FFMA,
// no FP64->FP32 conversion); then the hardware sine and cosine.
__device__ __forceinline__ void vertex_phasor(double st, double ct, const VertRegs &w, float &s,
                                              float &c)
{
    const double t = fma(st, w.ps, fma(ct, w.pc, w.p0));
    const unsigned lo = (unsigned)__double2loint(t);
    const float x = fmaf(__int_as_float(0x3F800000u | (lo & 0x007FFFFFu)), 6.28318530717958647f,
                         -9.42477796076937972f);
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(x));
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(x));
}

// FP64 phasor through the kernel's sine table.
__device__ __forceinline__ void vertex_phasor_t(double st, double ct, const VertRegs &w,
                                                const double2 *tab, double &s, double &c)
{
    sincos_turns_tab(fma(st, w.ps, fma(ct, w.pc, w.p0)), tab, s, c);
}

// The same for two directions of one vertex: the two reductions to the
// angle in one FFMA2 (each lane rounds as the FFMA above, so the phasors are
// bitwise those of two single calls).
__device__ __forceinline__ void vertex_phasor2(double st0, double ct0, double st1, double ct1,
                                               const VertRegs &w, float2 &cs0, float2 &cs1)
{
    const double t0 = fma(st0, w.ps, fma(ct0, w.pc, w.p0));
    const double t1 = fma(st1, w.ps, fma(ct1, w.pc, w.p0));
    const unsigned lo0 = (unsigned)__double2loint(t0), lo1 = (unsigned)__double2loint(t1);
    const float2 y = make_float2(__int_as_float(0x3F800000u | (lo0 & 0x007FFFFFu)),
                                 __int_as_float(0x3F800000u | (lo1 & 0x007FFFFFu)));
    const float2 x = __ffma2_rn(y, make_float2(6.28318530717958647f, 6.28318530717958647f),
                                make_float2(-9.42477796076937972f, -9.42477796076937972f));
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(cs0.y) : "f"(x.x));
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(cs0.x) : "f"(x.x));
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(cs1.y) : "f"(x.y));
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(cs1.x) : "f"(x.y));
}

// Phasors (cos, sin) of one vertex for a thread's DPT directions, handed to
// out(d, phasor): directions in pairs, an odd last one alone.
template <int DPT, typename Out>
__device__ __forceinline__ void vertex_phasors(const double *st, const double *ct, const VertRegs &w,
                                               Out &&out)
{
#pragma unroll
    for (int d = 0; d + 1 < DPT; d += 2) {
        float2 a, b;
        vertex_phasor2(st[d], ct[d], st[d + 1], ct[d + 1], w, a, b);
        out(d, a);
        out(d + 1, b);
    }
    if (DPT & 1) {
        float2 c;
        vertex_phasor(st[DPT - 1], ct[DPT - 1], w, c.y, c.x);
        out(DPT - 1, c);
    }
}

__device__ __forceinline__ double rcp_t(double x) { return rcp64(x); }
__device__ __forceinline__ float rcp_t(float x) { return rcp32(x); }

// FP64 edge sums S_d = sum_e (P(e+1) - P(e)) / C_e of one beam for the DPT
// directions of a thread.  The reference's two branches share one form,
// C_e = X2 + slope_e X1 with (X1, X2, slope) = (B, A, slope_yx) when |B| > |A|
// (x branch) and (A, B, slope_xy) otherwise (y branch).  All vertex phasors
// are independent, so the NV*DPT chains interleave.  mn[d] receives the
// smallest high word of |C_e| (nearly singular edges go to the FP64 pass): the
// comparison runs on the integer pipe, the FP64 pipe is what bounds the kernel
// (96 orientations of 87 beams on 48 x 1801 directions: 10.8 ms with FP64
// minima, two Newton steps and the table of 128; 9.5 ms so).  The sum regrouped by
// vertices, sum_v P(v) (1/C_{v-1} - 1/C_v), is 2 % shorter, but near the forward
// direction the differences P(e+1) - P(e) are small and exact and the weights'
// are neither: 16 % more error on a size scan.
__device__ __forceinline__ uint32_t abs_hi(double x)
{
    return (uint32_t)__double2hiint(x) & 0x7fffffffu;
}

// With kDrop an edge with |C_e| <= eps is left out instead (its coefficient
// becomes kDropped, its term 1e-100 of the others).
constexpr double kDropped = 1e100;

template <int DPT, int NV, bool kDrop>
__device__ __forceinline__ void edge_sums_fixed(const SVertRaw<double> *v, const double *st, const double *ct,
                                                const double *X1, const double *X2, const bool *useX,
                                                double *sr, double *si, uint32_t *mn, const double2 *tab,
                                                double eps)
{
    double c[DPT][NV], s[DPT][NV], syx[NV], sxy[NV];
#pragma unroll
    for (int e = 0; e < NV; ++e) {
        VertRegs w;
        load_vert(v[e], w, syx[e], sxy[e]);
#pragma unroll
        for (int d = 0; d < DPT; ++d)
            vertex_phasor_t(st[d], ct[d], w, tab, s[d][e], c[d][e]);
    }
#pragma unroll
    for (int d = 0; d < DPT; ++d) {
        mn[d] = 0xffffffffu;
        // 1 / C_e; consecutive edges share one reciprocal: 1/a = b/(ab),
        // 1/b = a/(ab) (coefficients between eps1 and about 1e30 |X1| keep the
        // product far from overflow and underflow; a pair with a smaller one
        // is marked and its sums discarded)
        double inv[NV];
#pragma unroll
        for (int e = 0; e < NV; e += 2) {
            double ca = fma(useX[d] ? syx[e] : sxy[e], X1[d], X2[d]);
            mn[d] = min(mn[d], abs_hi(ca));
            if (kDrop && fabs(ca) <= eps)
                ca = kDropped;
            if (e + 1 < NV) {
                double cb = fma(useX[d] ? syx[e + 1] : sxy[e + 1], X1[d], X2[d]);
                mn[d] = min(mn[d], abs_hi(cb));
                if (kDrop && fabs(cb) <= eps)
                    cb = kDropped;
                const double r = rcp64(ca * cb);
                inv[e] = cb * r;
                inv[e + 1] = ca * r;
            } else {
                inv[e] = rcp64(ca);
            }
        }
        sr[d] = (c[d][1] - c[d][0]) * inv[0];
        si[d] = (s[d][1] - s[d][0]) * inv[0];
#pragma unroll
        for (int e = 1; e < NV; ++e) {
            const int n = e + 1 < NV ? e + 1 : 0;
            sr[d] = fma(c[d][n] - c[d][e], inv[e], sr[d]);
            si[d] = fma(s[d][n] - s[d][e], inv[e], si[d]);
        }
    }
}

// FP32C edge sums in two parts.  The head (vertices 0-2, edges 0 and 1:
// every aperture has at least three vertices) sits in the beam loop's
// straight-line code with the beam's A, B and zone tests, so their chains
// interleave; the tail (the remaining vertices and edges, the closing edge
// back to vertex 0) follows the warp-uniform switch on the vertex count.
// The sums add the edges in order (edge e from vertex e to e + 1, the last
// back to vertex 0); consecutive edges share one reciprocal (rcp_pair).  The
// edge differences are one packed FP32x2 operation each (the same rounding
// as two subtractions: (-1) c_e + c_{e+1} is exact before its single
// rounding).
__device__ __forceinline__ void edge_step_f32(float2 a, float2 b, float slope, float X1, float X2,
                                              float &sr, float &si, float &mn)
{
    const float coef = fmaf(slope, X1, X2);
    const float inv = rcp32(coef);
    mn = fminf(mn, fabsf(coef));
    const float2 df = __ffma2_rn(a, make_float2(-1.f, -1.f), b);
    sr = fmaf(df.x, inv, sr);
    si = fmaf(df.y, inv, si);
}

// 1/a and 1/b from one reciprocal: r = 1/(a b), 1/a = b r, 1/b = a r (one
// MUFU instead of two, three more multiplications).  An edge reaches the hot
// loop's sums only with |a|, |b| > eps (else the pair goes to the FP64 pass),
// so the product does not underflow.  An invalid edge's coefficient (slope
// 1e30: about 1e30 |X1|) overflows the product only when the other one
// exceeds about 3e8; both quotients are then 0 instead of below 1e-30 and
// 3e-9, terms far below the FP32 rounding of the sum.
__device__ __forceinline__ void rcp_pair(float a, float b, float &ia, float &ib)
{
    const float r = rcp32(a * b);
    ia = b * r;
    ib = a * r;
}

// Two consecutive edges (vertex phasors a -> b -> c, slopes sa, sb) with
// one reciprocal for both coefficients; otherwise edge_step_f32 twice.
__device__ __forceinline__ void edge_pair_f32(float2 a, float2 b, float2 c, float sa, float sb, float X1,
                                              float X2, float &sr, float &si, float &mn)
{
    const float ca = fmaf(sa, X1, X2), cb = fmaf(sb, X1, X2);
    float ia, ib;
    rcp_pair(ca, cb, ia, ib);
    mn = fminf(mn, fminf(fabsf(ca), fabsf(cb)));
    const float2 da = __ffma2_rn(a, make_float2(-1.f, -1.f), b);
    const float2 db = __ffma2_rn(b, make_float2(-1.f, -1.f), c);
    sr = fmaf(da.x, ia, sr);
    si = fmaf(da.y, ia, si);
    sr = fmaf(db.x, ib, sr);
    si = fmaf(db.y, ib, si);
}

template <int DPT>
struct EdgeHead {
    float2 c0[DPT], c2[DPT];   // phasors of vertices 0 and 2
    float syx2, sxy2;          // slopes of vertex 2's edge
};

template <int DPT>
__device__ __forceinline__ void edge_head_f32(const SVertRaw<float> *v, const double *st, const double *ct,
                                              const float *X1, const float *X2, const bool *useX,
                                              EdgeHead<DPT> &h, float *sr, float *si, float *mn)
{
    float2 c1[DPT];
    float syx0, sxy0, syx1, sxy1;
    VertRegs w0, w1, w2;
    load_vert(v[0], w0, syx0, sxy0);
    load_vert(v[1], w1, syx1, sxy1);
    load_vert(v[2], w2, h.syx2, h.sxy2);
    // the head's phasors with the reductions of two directions paired (the
    // tail keeps single ones: pairing there too made the step 3 % longer)
    vertex_phasors<DPT>(st, ct, w0, [&](int d, float2 p) { h.c0[d] = p; });
    vertex_phasors<DPT>(st, ct, w1, [&](int d, float2 p) { c1[d] = p; });
    vertex_phasors<DPT>(st, ct, w2, [&](int d, float2 p) { h.c2[d] = p; });
#pragma unroll
    for (int d = 0; d < DPT; ++d) {
        mn[d] = 1e30f;
        sr[d] = 0.f;
        si[d] = 0.f;
        edge_pair_f32(h.c0[d], c1[d], h.c2[d], useX[d] ? syx0 : sxy0, useX[d] ? syx1 : sxy1, X1[d], X2[d],
                      sr[d], si[d], mn[d]);
    }
}

template <int DPT, int NV>
__device__ __forceinline__ void edge_tail_fixed_f32(const SVertRaw<float> *v, const double *st, const double *ct,
                                                    const float *X1, const float *X2, const bool *useX,
                                                    const EdgeHead<DPT> &h, float *sr, float *si, float *mn)
{
    constexpr int kM = NV > 3 ? NV - 3 : 1;
    float2 cs[DPT][kM];
    float syx[kM], sxy[kM];
#pragma unroll
    for (int e = 3; e < NV; ++e) {
        VertRegs w;
        load_vert(v[e], w, syx[e - 3], sxy[e - 3]);
#pragma unroll
        for (int d = 0; d < DPT; ++d)
            vertex_phasor(st[d], ct[d], w, cs[d][e - 3].y, cs[d][e - 3].x);
    }
    // edges in pairs (2, 3), (4, 5); an odd last edge alone
#pragma unroll
    for (int e = 2; e < NV; e += 2) {
#pragma unroll
        for (int d = 0; d < DPT; ++d) {
            const float2 a = e == 2 ? h.c2[d] : cs[d][e - 3];
            const float2 b = e + 1 < NV ? cs[d][e - 2] : h.c0[d];
            const float slope = e == 2 ? (useX[d] ? h.syx2 : h.sxy2)
                                       : (useX[d] ? syx[e - 3] : sxy[e - 3]);
            if (e + 1 < NV) {
                const float2 c = e + 2 < NV ? cs[d][e - 1] : h.c0[d];
                edge_pair_f32(a, b, c, slope, useX[d] ? syx[e - 2] : sxy[e - 2], X1[d], X2[d], sr[d],
                              si[d], mn[d]);
            } else {
                edge_step_f32(a, b, slope, X1[d], X2[d], sr[d], si[d], mn[d]);
            }
        }
    }
}

template <int DPT>
__device__ __forceinline__ void edge_tail_loop_f32(const SVertRaw<float> *v, int nv, const double *st,
                                                   const double *ct, const float *X1, const float *X2,
                                                   const bool *useX, const EdgeHead<DPT> &h, float *sr,
                                                   float *si, float *mn)
{
    float2 prev[DPT];
#pragma unroll
    for (int d = 0; d < DPT; ++d)
        prev[d] = h.c2[d];
    float syx = h.syx2, sxy = h.sxy2;
    for (int e = 2; e < nv; ++e) {
        const bool last = e + 1 == nv;
        const float syx_e = syx, sxy_e = sxy;
        VertRegs w;
        if (!last)
            load_vert(v[e + 1], w, syx, sxy);
#pragma unroll
        for (int d = 0; d < DPT; ++d) {
            float2 nx = h.c0[d];
            if (!last)
                vertex_phasor(st[d], ct[d], w, nx.y, nx.x);
            edge_step_f32(prev[d], nx, useX[d] ? syx_e : sxy_e, X1[d], X2[d], sr[d], si[d], mn[d]);
            prev[d] = nx;
        }
    }
}

template <int DPT, bool kDrop>
__device__ __forceinline__ void edge_sums_loop(const SVertRaw<double> *v, int nv, const double *st,
                                               const double *ct, const double *X1, const double *X2,
                                               const bool *useX, double *sr, double *si, uint32_t *mn,
                                               const double2 *tab, double eps)
{
    double c0[DPT], s0[DPT], cp_[DPT], sp_[DPT];
    double syx, sxy;
    VertRegs w;
    load_vert(v[0], w, syx, sxy);
#pragma unroll
    for (int d = 0; d < DPT; ++d) {
        vertex_phasor_t(st[d], ct[d], w, tab, s0[d], c0[d]);
        cp_[d] = c0[d];
        sp_[d] = s0[d];
        mn[d] = 0xffffffffu;
        sr[d] = 0.0;
        si[d] = 0.0;
    }
    for (int e = 0; e < nv; ++e) {
        const bool last = e + 1 == nv;
        const double syx_e = syx, sxy_e = sxy;
        if (!last)
            load_vert(v[e + 1], w, syx, sxy);
#pragma unroll
        for (int d = 0; d < DPT; ++d) {
            double cn = c0[d], sn = s0[d];
            if (!last)
                vertex_phasor_t(st[d], ct[d], w, tab, sn, cn);
            double coef = fma(useX[d] ? syx_e : sxy_e, X1[d], X2[d]);
            mn[d] = min(mn[d], abs_hi(coef));
            if (kDrop && fabs(coef) <= eps)
                coef = kDropped;
            const double inv = rcp64(coef);
            sr[d] = fma(cn - cp_[d], inv, sr[d]);
            si[d] = fma(sn - sp_[d], inv, si[d]);
            cp_[d] = cn;
            sp_[d] = sn;
        }
    }
}

// FP64 edge sums of one beam (the FP32C path uses edge_head_f32 and the
// tails above): fixed vertex counts unrolled, longer apertures in a loop.
template <int DPT, bool kDrop = false>
__device__ __forceinline__ void edge_sums(const SVertRaw<double> *v, int nv, const double *st,
                                          const double *ct, const double *X1, const double *X2,
                                          const bool *useX, double *sr, double *si, uint32_t *mn,
                                          const double2 *tab, double eps = 0.0)
{
    switch (nv) {   // warp-uniform: every lane evaluates the same beam
    case 3: edge_sums_fixed<DPT, 3, kDrop>(v, st, ct, X1, X2, useX, sr, si, mn, tab, eps); break;
    case 4: edge_sums_fixed<DPT, 4, kDrop>(v, st, ct, X1, X2, useX, sr, si, mn, tab, eps); break;
    case 5: edge_sums_fixed<DPT, 5, kDrop>(v, st, ct, X1, X2, useX, sr, si, mn, tab, eps); break;
    case 6: edge_sums_fixed<DPT, 6, kDrop>(v, st, ct, X1, X2, useX, sr, si, mn, tab, eps); break;
    default: edge_sums_loop<DPT, kDrop>(v, nv, st, ct, X1, X2, useX, sr, si, mn, tab, eps); break;
    }
}

// The rare pairs of one direction, in FP64: the near-forward moment
// expansion (FP32C), or the complete general evaluation (small-phase
// candidates, nearly singular edges, irregular polar rows).  Writes the
// Jones contribution to the thread's shared-memory slot out[0..7] (stride
// `stride`), so the caller's registers never leave the register file;
// returns false when the beam contributes nothing.
template <typename T>
__device__ __noinline__ bool beam_rare(const KParams &P, int gbeam, const SBeamRaw<T> *sbr, int p,
                                       int t, bool near, T *out, int stride)
{
    constexpr bool kF32 = sizeof(T) == 4;
    const double st = P.st[t], ct = P.ct[t], cp = P.cphi[p], sp = P.sphi[p];
    if (kF32 && near) {
        float sr, si;
        near_forward_s(P.beams[gbeam], P.moments + (size_t)gbeam * kNumMoments, st, ct, cp, sp,
                       P.wc, sr, si);
        T Pm[24];
        load_P(*sbr, Pm);
        const T stT = (T)st, ctT = (T)ct;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const T rr = fma(stT, Pm[16 + 2 * e], fma(ctT, Pm[8 + 2 * e], Pm[2 * e]));
            const T ri = fma(stT, Pm[17 + 2 * e], fma(ctT, Pm[9 + 2 * e], Pm[2 * e + 1]));
            out[(2 * e) * stride] = fma((T)sr, rr, -(T)si * ri);
            out[(2 * e + 1) * stride] = fma((T)sr, ri, (T)si * rr);
        }
        return true;
    }
    DirFull dc;
    dir_full(P, p, t, dc);
    double dd[8];
    const bool ok = beam_general(P.beams[gbeam], P.verts, dc, P.wc, dd);
#pragma unroll
    for (int q = 0; q < 8; ++q)
        out[q * stride] = (T)dd[q];
    return ok;
}

// A pair marked only for a nearly singular edge (|C_e| <= eps): the fast
// path's arithmetic from the shared-memory records, with every edge whose
// |C_e| <= eps taken in the stable form of the same quotient,
//   (e^{i phi_{e+1}} - e^{i phi_e}) / C_e = e^{i phi_e} (e^{iz} - 1) / C_e,
//   z = k C_e delta_e (delta_e: the edge's x or y extent on the branch),
// in FP64 (stable_edge, the reference's singular correction,
// GpuDiffraction.cu:951-970).  The result equals the general evaluation
// (beam_general) without its global-memory walk over the beam; the edge
// extents come from the two vertices' general records.  Writes the Jones
// contribution to out[0..7] (stride `stride`); returns false when the sum
// is not finite, where the general evaluation drops the beam.
template <typename T>
__device__ __noinline__ bool beam_sing(const KParams &P, const SBeamRaw<T> *sbr, const SVertRaw<T> *sv,
                                       int vglob, double st, double ct, T *out, int stride)
{
    constexpr bool kF32 = sizeof(T) == 4;
    BeamRegs<T> b;
    load_beam(*sbr, b);
    const T stT = (T)st, ctT = (T)ct;
    const T A = fma(stT, b.a[0], fma(ctT, b.a[1], b.a[2]));
    const T B = fma(stT, b.a[3], fma(ctT, b.a[4], b.a[5]));
    const bool useX = fabs(B) > fabs(A);
    const T X1 = useX ? B : A, X2 = useX ? A : B;
    const T eps = (T)(kF32 ? P.wc.eps1_f32 : P.wc.eps1);
    const SVertRaw<T> *v = sv + b.vs;
    const DevVert *gv = P.verts + vglob + b.vs;
    VertRegs w;
    T syx, sxy, c0, s0;
    load_vert(v[0], w, syx, sxy);
    vertex_phasor(st, ct, w, s0, c0);
    T cprev = c0, sprev = s0, sr = T(0), si = T(0);
    double dr = 0.0, di = 0.0;
    for (int e = 0; e < b.nv; ++e) {
        const int en = (e + 1 < b.nv) ? e + 1 : 0;
        const T syx_e = syx, sxy_e = sxy;
        T cn = c0, sn = s0;
        if (en != 0) {
            load_vert(v[en], w, syx, sxy);
            vertex_phasor(st, ct, w, sn, cn);
        }
        const T coef = fma(useX ? syx_e : sxy_e, X1, X2);
        if (fabs(coef) > eps) {
            const T inv = rcp_t(coef);
            sr = fma(cn - cprev, inv, sr);
            si = fma(sn - sprev, inv, si);
        } else if (fabs(coef) <= eps) {           // NaN: invalid edge, dropped
            const double delta = useX ? gv[en].x - gv[e].x : gv[en].y - gv[e].y;
            stable_edge((double)cprev, (double)sprev, delta, (double)coef, P.wc.k, dr, di);
        }
        cprev = cn;
        sprev = sn;
    }
    const T m = rcp_t(useX ? B : -A);
    const T s_r = (sr + (T)dr) * m, s_i = (si + (T)di) * m;
    if (!isfinite(s_r) || !isfinite(s_i))
        return false;
    T Pm[24];
    load_P(*sbr, Pm);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const T rr = fma(stT, Pm[16 + 2 * e], fma(ctT, Pm[8 + 2 * e], Pm[2 * e]));
        const T ri = fma(stT, Pm[17 + 2 * e], fma(ctT, Pm[9 + 2 * e], Pm[2 * e + 1]));
        out[(2 * e) * stride] = fma(s_r, rr, -s_i * ri);
        out[(2 * e + 1) * stride] = fma(s_r, ri, s_i * rr);
    }
    return true;
}

// Accumulator of the coherent Jones sum of one orientation for one
// direction.  FP32: plain sums over blocks of kFlushEvery beams in
// registers, folded into a Kahan-compensated running sum kept in shared
// memory (s, c with stride) at every block end.  FP64: plain sums.  Blocks
// of 32 beams: against 16 the step is 1.7 % shorter and the FP32C error
// against FP64 unchanged (it comes from the FP32 trigonometry, not from the
// block sums).
constexpr int kFlushEvery = 32;

template <typename T>
struct JonesAcc {
    T b[8];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] = T(0);
    }
    __device__ __forceinline__ void add(const T *d) {
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] += d[i];
    }
    __device__ __forceinline__ void fold(float *s, float *c, int stride) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float si = s[i * stride], ci = c[i * stride];
            const float y = __fsub_rn((float)b[i], ci);
            const float t = __fadd_rn(si, y);
            c[i * stride] = __fsub_rn(__fsub_rn(t, si), y);
            s[i * stride] = t;
            b[i] = T(0);
        }
    }
};

// J += s x (P0 + cos t Pc + sin t Ps) for DPT directions, two complex entries
// at a time.
template <typename T, int DPT>
__device__ __forceinline__ void jones_update(const SBeamRaw<T> &rec, const T *s_r, const T *s_i, const T *stT,
                                             const T *ctT, const float2 *st2, const float2 *ct2, JonesAcc<T> *J)
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if constexpr (sizeof(T) == 4) {
            // entries 2h and 2h+1 side by side: R = P0 + cos t Pc + sin t Ps
            // as (re, re) and (im, im) pairs, then J_re += -s_i R_i + s_r R_r
            // and J_im += s_i R_r + s_r R_i, the scalar form's operations
            // lane by lane (no operand pair needs its halves swapped)
            float2 p0r, p0i, pcr, pci, psr, psi;
            load_P_packed(rec, h, p0r, p0i, pcr, pci, psr, psi);
#pragma unroll
            for (int d = 0; d < DPT; ++d) {
                const float2 srr = make_float2(s_r[d], s_r[d]);
                const float2 sii = make_float2(s_i[d], s_i[d]);
                const float2 nsi = make_float2(-s_i[d], -s_i[d]);
                const float2 Rr = __ffma2_rn(st2[d], psr, __ffma2_rn(ct2[d], pcr, p0r));
                const float2 Ri = __ffma2_rn(st2[d], psi, __ffma2_rn(ct2[d], pci, p0i));
                float2 jr = make_float2(J[d].b[4 * h], J[d].b[4 * h + 2]);
                float2 ji = make_float2(J[d].b[4 * h + 1], J[d].b[4 * h + 3]);
                jr = __ffma2_rn(nsi, Ri, jr);
                jr = __ffma2_rn(srr, Rr, jr);
                ji = __ffma2_rn(sii, Rr, ji);
                ji = __ffma2_rn(srr, Ri, ji);
                J[d].b[4 * h] = jr.x;
                J[d].b[4 * h + 2] = jr.y;
                J[d].b[4 * h + 1] = ji.x;
                J[d].b[4 * h + 3] = ji.y;
            }
        } else {
            T p0[4], pc[4], ps[4];
            load_P_pair(rec, h, p0, pc, ps);
#pragma unroll
            for (int d = 0; d < DPT; ++d) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int q = 4 * h + 2 * e;
                    const T rr = fma(stT[d], ps[2 * e], fma(ctT[d], pc[2 * e], p0[2 * e]));
                    const T ri = fma(stT[d], ps[2 * e + 1], fma(ctT[d], pc[2 * e + 1], p0[2 * e + 1]));
                    J[d].b[q] = fma(s_r[d], rr, fma(-s_i[d], ri, J[d].b[q]));
                    J[d].b[q + 1] = fma(s_r[d], ri, fma(s_i[d], rr, J[d].b[q + 1]));
                }
            }
        }
    }
}

// Fused diffraction kernel, persistent: each CTA takes work items
// (orientation chunk, azimuth bin, zenith tile) from a global counter.  Each
// thread owns DPT directions of an item (rows trow + d*TPB + thread of the
// item's azimuth).  T = float selects FP32C.
template <typename T, int TPB, int DPT, bool NS, int MINB, int BEAMS = default_stage<T>(TPB)>
__global__ void __launch_bounds__(TPB, MINB) po_diffract_kernel(KParams P)
{
    using Cfg = StageCfg<T, BEAMS>;
    constexpr int kDirs = TPB * DPT;
    constexpr bool kF32 = sizeof(T) == 4;
    constexpr int kSets = NS ? 2 : 1;        // full and no-shadow sums
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SBeamRaw<T> *sb = reinterpret_cast<SBeamRaw<T> *>(smem_raw);
    SVertRaw<T> *sv = reinterpret_cast<SVertRaw<T> *>(smem_raw + Cfg::kBeams * sizeof(SBeamRaw<T>));
    // rare-path result slot per thread: [8][TPB]
    T *rsm = reinterpret_cast<T *>(smem_raw + Cfg::kBytes);
    // FP32C: Kahan running sums of the Jones matrices, [kSets][s, c][8][kDirs]
    float *Ksm = reinterpret_cast<float *>(rsm + 8 * TPB);
    // per thread: bit masks of the stage's pairs for the FP64 pass, [DPT][words][TPB]
    constexpr int kMaskWords = (Cfg::kBeams + 31) / 32;
    uint32_t *rmask = reinterpret_cast<uint32_t *>(Ksm + (kF32 ? kSets * 16 * kDirs : 0));

    const T eps = (T)(kF32 ? P.wc.eps1_f32 : P.wc.eps1);
    T *rslot = rsm + threadIdx.x;
    const int items_per_chunk = P.n_az * P.tiles_per_row;
    __shared__ int s_item;
    __shared__ double s_zdel[TPB / 32];
    __shared__ int s_rwarp[TPB / 32], s_rbase[TPB], s_rok[TPB];   // the spread FP64 pass
    // FP64: the sine table of the vertex phasors
    __shared__ double2 s_sincos[kF32 ? 1 : kSinTab];
    if constexpr (!kF32)
        fill_sincos_tab(s_sincos, TPB);

    // Persistent: take work items until none are left, so CTAs of uneven
    // cost (rare FP64 pairs, ragged beam counts) balance across the SMs.
    for (;;) {
    __syncthreads();   // the previous item is finished with s_item and the stage
    if (threadIdx.x == 0)
        s_item = atomicAdd(P.work, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= P.n_items)
        break;
    const int chunk = item / items_per_chunk;
    const int pt = item - chunk * items_per_chunk;
    const int p = pt / P.tiles_per_row;
    const int tile = pt - p * P.tiles_per_row;
    const int trow = P.row0 + tile * kDirs;   // the tile's first zenith row
    int o0, o1;
    chunk_range(P, chunk, o0, o1);
    const double cp = P.cphi[p], sp = P.sphi[p];

    int t[DPT];
    bool active[DPT], general[DPT];
    double st[DPT], ct[DPT];
    T stT[DPT], ctT[DPT];
#pragma unroll
    for (int d = 0; d < DPT; ++d) {
        const int tr = trow + d * TPB + threadIdx.x;
        t[d] = tr < P.row1 ? tr : P.row1 - 1;
        const int kind = P.row_kind[t[d]];
        active[d] = tr < P.row1 && kind != 1;
        general[d] = kind == 2;
        st[d] = P.st[t[d]];
        ct[d] = P.ct[t[d]];
        stT[d] = (T)st[d];
        ctT[d] = (T)ct[d];
    }
    float2 st2[DPT], ct2[DPT];   // FP32C: (sin t, sin t), (cos t, cos t) operand pairs
#pragma unroll
    for (int d = 0; d < DPT; ++d) {
        st2[d] = make_float2((float)stT[d], (float)stT[d]);
        ct2[d] = make_float2((float)ctT[d], (float)ctT[d]);
    }
    const size_t G = (size_t)P.n_az * P.n_t;
    // spread of the tile's directions around its middle row, for the zone
    // flags of the stage fill (read there after the fill's first barrier)
    {
        const int tm = min(trow + kDirs / 2, P.row1 - 1);
        const double stc = P.st[tm], ctc = P.ct[tm];
        double dd = 0.0;
#pragma unroll
        for (int d = 0; d < DPT; ++d)
            dd = fmax(dd, (st[d] - stc) * (st[d] - stc) + (ct[d] - ctc) * (ct[d] - ctc));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            dd = fmax(dd, __shfl_xor_sync(0xffffffffu, dd, off));
        if ((threadIdx.x & 31) == 0)
            s_zdel[threadIdx.x >> 5] = dd;
    }

    for (int o = o0; o < o1; ++o) {
        JonesAcc<T> J[DPT], Jn[NS ? DPT : 1];
#pragma unroll
        for (int d = 0; d < DPT; ++d) {
            J[d].zero();
            if (NS) Jn[d].zero();
        }
        if (kF32) {
            for (int i = threadIdx.x; i < kSets * 16 * kDirs; i += TPB)
                Ksm[i] = 0.f;
        }
        const int b0 = P.beam_off[o], b1 = P.beam_off[o + 1];
        for (int bs = b0; bs < b1;) {
            // stage [bs, be): at most kBeams beams and kVerts vertices
            const int vb0 = P.vbeg[bs];
            int be = min(b1, bs + Cfg::kBeams);
            if (P.vbeg[be] - vb0 > Cfg::kVerts) {
                int lo = bs + 1, hi = be;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (P.vbeg[mid] - vb0 <= Cfg::kVerts) lo = mid; else hi = mid - 1;
                }
                be = lo;
            }
            const int nb = be - bs;
            const int nvs = P.vbeg[be] - vb0;
            __syncthreads();   // previous stage fully consumed
            TileZone tz;
            {
                const int tm = min(trow + kDirs / 2, P.row1 - 1);
                double dd = 0.0;
#pragma unroll
                for (int w = 0; w < TPB / 32; ++w)
                    dd = fmax(dd, s_zdel[w]);
                tz.stc = P.st[tm];
                tz.ctc = P.ct[tm];
                tz.del = sqrt(dd) * (1.0 + 1e-12);
            }
            for (int i = threadIdx.x; i < nb; i += TPB)
                fill_beam(BrecRef{P.brec + bs + i, P.brec_stride}, cp, sp, P.vbeg[bs + i] - vb0, bs + i, tz,
                          sb[i]);
            for (int i = threadIdx.x; i < nvs; i += TPB)
                fill_vert(VrecRef{P.vrec + vb0 + i, P.vrec_stride}, cp, sp, sv[i]);
            __syncthreads();
            // Hot loop: every (beam, direction) pair on the vectorised path;
            // pairs that need FP64 (near-forward zone, small-phase candidates,
            // nearly singular edges, irregular rows) contribute nothing here
            // and are marked in the thread's bit mask for the pass below.
            uint32_t bits[DPT];
#pragma unroll
            for (int d = 0; d < DPT; ++d)
                bits[d] = 0u;
            // blocks of kFlushEvery beams: the mask store and the Kahan fold
            // run between blocks, not as tests inside the beam loop
            static_assert(32 % kFlushEvery == 0, "mask words hold whole blocks");
            for (int j0 = 0; j0 < nb; j0 += kFlushEvery) {
            const int j1 = min(nb, j0 + kFlushEvery);
            // Two beams per iteration where the shape leaves registers for it: one
            // beam's loads and edge head then overlap the other's chain, which
            // a thread with one or two directions cannot fill by itself.  300
            // orientations of 87 beams, 48 azimuths, FP32C: 64 rows (64x1) 1108 ->
            // 1032 us, 96 (96x1) 1219 -> 1174, 128 (128x1) 1451 -> 1353, 192 (96x2)
            // 1790 -> 1768, 256 (128x2) 2301 -> 2246, no-shadow sums (128x3) 1041
            // -> 1012; FP64, 150 orientations: 64 rows (64x1) 797 -> 782, 96 (96x1)
            // 1021 -> 1013, no-shadow sums (128x1 with 168 registers) of 61
            // orientations on 47 x 358 1645 -> 1605.  Slower
            // where it adds spills or the directions fill the chain: FP32C 128x3
            // 3043 -> 3066, FP64 64x3 1762 -> 1905, 128x1 with 128 registers 1176 ->
            // 1215; four beams: 64x1 1143, 96x1 1311.
            constexpr bool kRoomy = TPB * MINB <= 384;   // 168 registers or more
            constexpr int kUnroll = (kF32 ? DPT == 1 || NS || (DPT == 2 && kRoomy) : DPT == 1 && kRoomy) ? 2 : 1;
#pragma unroll kUnroll
            for (int j = j0; j < j1; ++j) {
                BeamRegs<T> b;
                load_beam(sb[j], b);
                T X1[DPT], X2[DPT], sr[DPT], si[DPT], mden[DPT], Av[DPT], Bv[DPT];
                bool useX[DPT], rare[DPT], sing[DPT];   // sing: a nearly singular edge
#pragma unroll
                for (int d = 0; d < DPT; ++d) {
                    T A, B;
                    if constexpr (kF32) {
                        const float2 ab = __ffma2_rn(st2[d], make_float2(b.a[0], b.a[3]),
                                                     __ffma2_rn(ct2[d], make_float2(b.a[1], b.a[4]),
                                                                make_float2(b.a[2], b.a[5])));
                        A = ab.x;
                        B = ab.y;
                    } else {
                        A = fma(stT[d], b.a[0], fma(ctT[d], b.a[1], b.a[2]));
                        B = fma(stT[d], b.a[3], fma(ctT[d], b.a[4], b.a[5]));
                    }
                    useX[d] = fabs(B) > fabs(A);
                    X1[d] = useX[d] ? B : A;
                    X2[d] = useX[d] ? A : B;
                    mden[d] = useX[d] ? B : -A;          // x branch: 1/B, y branch: -1/A
                    Av[d] = A;
                    Bv[d] = B;
                    rare[d] = general[d];
                }
                // the zone tests only where the stage fill found the tile
                // may reach the zone (warp-uniform: one beam per iteration)
                if (b.zone) {
#pragma unroll
                    for (int d = 0; d < DPT; ++d) {
                        const T A = Av[d], B = Bv[d];
                        const bool near = kF32 && (float)(A * A + B * B) <= b.nearr2;
                        const bool cand = fabs(fma(A, b.slab[0], B * b.slab[1])) <= T(1)
                                       && fabs(fma(A, b.slab[2], B * b.slab[3])) <= T(1);
                        rare[d] = rare[d] || near || cand;
                    }
                }
                if constexpr (kF32) {
                    float mn[DPT];
                    EdgeHead<DPT> eh;
                    const SVertRaw<float> *vb = sv + b.vs;
                    edge_head_f32<DPT>(vb, st, ct, X1, X2, useX, eh, sr, si, mn);
                    switch (b.nv) {   // warp-uniform: every lane evaluates the same beam
                    case 3: edge_tail_fixed_f32<DPT, 3>(vb, st, ct, X1, X2, useX, eh, sr, si, mn); break;
                    case 4: edge_tail_fixed_f32<DPT, 4>(vb, st, ct, X1, X2, useX, eh, sr, si, mn); break;
                    case 5: edge_tail_fixed_f32<DPT, 5>(vb, st, ct, X1, X2, useX, eh, sr, si, mn); break;
                    case 6: edge_tail_fixed_f32<DPT, 6>(vb, st, ct, X1, X2, useX, eh, sr, si, mn); break;
                    default: edge_tail_loop_f32<DPT>(vb, b.nv, st, ct, X1, X2, useX, eh, sr, si, mn); break;
                    }
#pragma unroll
                    for (int d = 0; d < DPT; ++d)
                        sing[d] = mn[d] <= eps;
                } else {
                    // high words: a coefficient within 2^-20 above eps is marked
                    // too (the pass takes its plain quotient)
                    uint32_t mn[DPT];
                    edge_sums<DPT>(sv + b.vs, b.nv, st, ct, X1, X2, useX, sr, si, mn, s_sincos);
#pragma unroll
                    for (int d = 0; d < DPT; ++d)
                        sing[d] = mn[d] <= abs_hi(eps);
                }
                T s_r[DPT], s_i[DPT];
#pragma unroll
                for (int d = 0; d < DPT; ++d) {
                    rare[d] = (rare[d] || sing[d]) && active[d];
                    bits[d] |= (rare[d] ? 1u : 0u) << (j & 31);
                    // select, not multiply: a marked pair may hold inf or NaN sums
                    const T m = rcp_t(mden[d]);
                    s_r[d] = rare[d] ? T(0) : sr[d] * m;
                    s_i[d] = rare[d] ? T(0) : si[d] * m;
                }
                // J += s x (P0 + cos t Pc + sin t Ps).  With no-shadow sums: FP32C
                // adds every beam to J and the internal ones to Jn (two sums, each
                // in beam order); FP64 adds external beams to J and internal ones
                // to Jn, and the full sum is J + Jn.  The branches are warp-uniform
                // (scalar updates weighted by a flag read per pair from global memory
                // took 1,157 us on 61 x 93 beams, 47 x 358 directions; now 1,039).
                if constexpr (!NS) {
                    jones_update<T, DPT>(sb[j], s_r, s_i, stT, ctT, st2, ct2, J);
                } else if constexpr (kF32) {
                    jones_update<T, DPT>(sb[j], s_r, s_i, stT, ctT, st2, ct2, J);
                    if (!b.external)
                        jones_update<T, DPT>(sb[j], s_r, s_i, stT, ctT, st2, ct2, Jn);
                } else {
                    if (b.external)
                        jones_update<T, DPT>(sb[j], s_r, s_i, stT, ctT, st2, ct2, J);
                    else
                        jones_update<T, DPT>(sb[j], s_r, s_i, stT, ctT, st2, ct2, Jn);
                }
            }
            if ((j1 & 31) == 0 || j1 == nb) {
#pragma unroll
                for (int d = 0; d < DPT; ++d) {
                    rmask[(d * kMaskWords + ((j1 - 1) >> 5)) * TPB + threadIdx.x] = bits[d];
                    bits[d] = 0u;
                }
            }
            if (kF32 && j1 - j0 == kFlushEvery) {
#pragma unroll
                for (int d = 0; d < DPT; ++d) {
                    const int slot = d * TPB + threadIdx.x;
                    J[d].fold(Ksm + slot, Ksm + 8 * kDirs + slot, kDirs);
                    if (NS)
                        Jn[NS ? d : 0].fold(Ksm + 16 * kDirs + slot, Ksm + 24 * kDirs + slot, kDirs);
                }
            }
            }
            // FP64 pass over the stage's marked pairs, spread over all the
            // CTA's threads: a pair's owner (the thread whose direction it
            // is) seldom has company in its warp, so per-owner loops left most
            // lanes idle and the CTA waiting at the next stage for its
            // busiest warp.  The marked pairs are numbered owner by owner in
            // the owners' (direction, beam) order; in rounds of TPB, thread i
            // evaluates pair r0 + i into its result slot, then every owner
            // adds its own results in that order, the order of a per-owner
            // loop, so the sums are the same bit for bit.
            {
                const int words = (nb + 31) >> 5;
                const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
                int cnt = 0;
#pragma unroll
                for (int d = 0; d < DPT; ++d)
                    for (int w = 0; w < words; ++w)
                        cnt += __popc(rmask[(d * kMaskWords + w) * TPB + threadIdx.x]);
                int incl = cnt;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, off);
                    if (lane >= off)
                        incl += v;
                }
                if (lane == 31)
                    s_rwarp[warp] = incl;
                __syncthreads();   // the warp totals and every thread's masks are visible
                int base = incl - cnt, total = 0;
#pragma unroll
                for (int w2 = 0; w2 < TPB / 32; ++w2) {
                    const int v = s_rwarp[w2];
                    base += w2 < warp ? v : 0;
                    total += v;
                }
                s_rbase[threadIdx.x] = base;
                __syncthreads();
                // the owner's cursor over its own marked pairs
                int cd = 0, cw = 0;
                uint32_t cm = words > 0 ? rmask[threadIdx.x] : 0u;
                for (int r0 = 0; r0 < total; r0 += TPB) {
                    const int q = r0 + threadIdx.x;
                    int okv = 0;
                    if (q < total) {
                        int lo = 0, hi = TPB - 1;   // owner: the last o with s_rbase[o] <= q
                        while (lo < hi) {
                            const int mid = (lo + hi + 1) >> 1;
                            if (s_rbase[mid] <= q) lo = mid; else hi = mid - 1;
                        }
                        const int o = lo;
                        int k = q - s_rbase[o], od = 0, j = 0;
                        bool found = false;
                        for (int d2 = 0; d2 < DPT && !found; ++d2)
                            for (int w = 0; w < words && !found; ++w) {
                                uint32_t m = rmask[(d2 * kMaskWords + w) * TPB + o];
                                const int c = __popc(m);
                                if (k < c) {
                                    for (int i = 0; i < k; ++i)
                                        m &= m - 1;
                                    j = w * 32 + __ffs(m) - 1;
                                    od = d2;
                                    found = true;
                                } else {
                                    k -= c;
                                }
                            }
                        const int to = trow + od * TPB + o;   // < row1: marked pairs are active
                        const double sto = P.st[to], cto = P.ct[to];
                        const bool gen = P.row_kind[to] == 2;
                        const T stTo = (T)sto, ctTo = (T)cto;
                        BeamRegs<T> b;
                        load_beam(sb[j], b);
                        const T A = fma(stTo, b.a[0], fma(ctTo, b.a[1], b.a[2]));
                        const T B = fma(stTo, b.a[3], fma(ctTo, b.a[4], b.a[5]));
                        const bool near = kF32 && !gen && (float)(A * A + B * B) <= b.nearr2;
                        const bool cand = fabs(fma(A, b.slab[0], B * b.slab[1])) <= T(1)
                                       && fabs(fma(A, b.slab[2], B * b.slab[3])) <= T(1);
                        okv = ((gen || near || cand)
                                   ? beam_rare<T>(P, b.gbeam, &sb[j], p, to, near, rslot, TPB)
                                   : beam_sing<T>(P, &sb[j], sv, vb0, sto, cto, rslot, TPB)) ? 1 : 0;
                    }
                    s_rok[threadIdx.x] = okv;
                    __syncthreads();   // this round's results are in the slots
                    const int q0 = max(base, r0), q1 = min(base + cnt, r0 + TPB);
                    for (int qq = q0; qq < q1; ++qq) {
                        while (cm == 0u) {
                            if (++cw == words) {
                                cw = 0;
                                ++cd;
                            }
                            cm = rmask[(cd * kMaskWords + cw) * TPB + threadIdx.x];
                        }
                        const int j = cw * 32 + __ffs(cm) - 1;
                        cm &= cm - 1;
                        const int slot = qq - r0;
                        if (s_rok[slot]) {
                            T dj[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                dj[i] = rsm[slot + i * TPB];
#pragma unroll
                            for (int d2 = 0; d2 < DPT; ++d2)
                                if (d2 == cd) {
                                    if (NS) {
                                        BeamRegs<T> bj;
                                        load_beam(sb[j], bj);
                                        if (kF32 || bj.external)
                                            J[d2].add(dj);
                                        if (!bj.external)
                                            Jn[NS ? d2 : 0].add(dj);
                                    } else {
                                        J[d2].add(dj);
                                    }
                                }
                        }
                    }
                    __syncthreads();   // the slots are read before the next round
                }
            }
            if (kF32) {
#pragma unroll
                for (int d = 0; d < DPT; ++d) {
                    const int slot = d * TPB + threadIdx.x;
                    J[d].fold(Ksm + slot, Ksm + 8 * kDirs + slot, kDirs);
                    if (NS)
                        Jn[NS ? d : 0].fold(Ksm + 16 * kDirs + slot, Ksm + 24 * kDirs + slot, kDirs);
                }
            }
            bs = be;
        }
        // Mueller of this orientation, weighted, added to the chunk's
        // partial plane in global memory (coalesced: consecutive threads
        // own consecutive directions; the first orientation initialises).
        // The adds are reductions performed in L2 (no load on the thread's
        // path); each partial element has a single owner thread, whose adds
        // reach it in program order, so the sums are deterministic.
        const double wgt = P.weight[o] * 0.25;
#pragma unroll
        for (int d = 0; d < DPT; ++d) {
            if (!active[d])
                continue;
            const int slot = d * TPB + threadIdx.x;
            const size_t g = (size_t)p * P.n_t + t[d];
            for (int set = 0; set < kSets; ++set) {
                double j[8];
                if (kF32) {
                    const float *s = Ksm + set * 16 * kDirs + slot;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        j[i] = (double)s[i * kDirs] - (double)s[(8 + i) * kDirs];
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        j[i] = NS ? (double)Jn[NS ? d : 0].b[i] + (set == 0 ? (double)J[d].b[i] : 0.0)
                                  : (double)J[d].b[i];
                }
                double m[16];
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    m[i] = 0.0;
                mueller_add(j, wgt, m);
                double *out = (set == 0 ? P.partial : P.partial_ns) + (size_t)chunk * 16 * G + g;
                if (o == o0) {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        out[i * G] = m[i];
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        atomicAdd(out + i * G, m[i]);
                }
            }
        }
    }
    }   // work items
}

template <typename T, int TPB, int DPT, bool NS, int BEAMS>
constexpr size_t diffract_smem_bytes()
{
    return StageCfg<T, BEAMS>::kBytes + 8 * TPB * sizeof(T)
         + (sizeof(T) == 4 ? (NS ? 2 : 1) * 16 * TPB * DPT * sizeof(float) : 0)
         + (size_t)DPT * ((BEAMS + 31) / 32) * TPB * sizeof(uint32_t);
}

// Polar zenith rows (row_kind 1): every azimuth bin has the same direction
// and polarisation basis there (Handler.h:147-160), so the row is evaluated
// once per orientation in FP64 and written to all azimuth bins.  Grid:
// x = orientation chunk, y = polar row index.  An orientation's beams are
// spread over `slices` warps (lanes stride over the beams, shuffle sums), the
// CTA's warp groups take the chunk's orientations in turn, and every sum runs
// in a fixed order (deterministic).  The beams' general evaluation is a chain
// of loads and FP64 operations of a few microseconds, so what bounds the
// kernel is how many beams one lane walks in turn (18 us for one orientation of
// 80 beams, 118 us for 12 of 1,200): with one thread per
// orientation (all its beams in turn) it took 204 us for one orientation of
// 80 beams, longer than the diffraction kernel beside it (176 us), and
// 5,990 us for 12 orientations of 1,200 beams.
constexpr int kPoleThreads = 256;

template <bool NS>
__global__ void __launch_bounds__(kPoleThreads) po_pole_kernel(KParams P, const int32_t *pole_rows, int slices)
{
    constexpr int kN = NS ? 16 : 8;
    __shared__ double part[kPoleThreads / 32][kN];    // Jones sums per warp
    __shared__ double msum[kPoleThreads / 32][2 * kN];  // Mueller sums per warp group
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = (blockDim.x >> 5) / slices;     // orientations in flight
    const int grp = warp / slices, slice = warp - grp * slices;
    const int chunk = blockIdx.x;
    const int t = pole_rows[blockIdx.y];
    int o0, o1;
    chunk_range(P, chunk, o0, o1);
    DirFull dc;
    dir_full(P, 0, t, dc);
    // Mueller sums of this group's orientations, held by the group's first lane
    double M[2 * kN];
#pragma unroll
    for (int i = 0; i < 2 * kN; ++i) M[i] = 0.0;
    for (int ob = o0; ob < o1; ob += groups) {
        const int o = ob + grp;
        double J[kN];
#pragma unroll
        for (int q = 0; q < kN; ++q) J[q] = 0.0;
        if (o < o1) {
            const int b1 = P.beam_off[o + 1];
            for (int b = P.beam_off[o] + slice * 32 + lane; b < b1; b += slices * 32) {
                double d[8];
                if (beam_general(P.beams[b], P.verts, dc, P.wc, d)) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) J[q] += d[q];
                    if (NS && !(P.beams[b].flags & MBS_PO_BEAM_EXTERNAL)) {
#pragma unroll
                        for (int q = 0; q < 8; ++q) J[NS ? 8 + q : q] += d[q];
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < kN; ++q) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                J[q] += __shfl_xor_sync(0xffffffffu, J[q], off);
            if (lane == 0)
                part[warp][q] = J[q];
        }
        __syncthreads();
        if (slice == 0 && lane == 0 && o < o1) {
            for (int s = 1; s < slices; ++s)
#pragma unroll
                for (int q = 0; q < kN; ++q)
                    J[q] += part[warp + s][q];
            const double wgt = P.weight[o] * 0.25;
            mueller_add(J, wgt, M);
            if (NS)
                mueller_add(J + (NS ? 8 : 0), wgt, M + (NS ? 16 : 0));
        }
        __syncthreads();   // the partial sums are read before the next round
    }
    if (slice == 0 && lane == 0)
#pragma unroll
        for (int i = 0; i < 2 * kN; ++i)
            msum[grp][i] = M[i];
    __syncthreads();
    const size_t G = (size_t)P.n_az * P.n_t;
    for (int i = threadIdx.x; i < 2 * kN * P.n_az; i += blockDim.x) {
        const int e = i / P.n_az, pp = i - e * P.n_az;
        double v = msum[0][e];
        for (int g = 1; g < groups; ++g)
            v += msum[g][e];
        double *out = (e < 16 ? P.partial : P.partial_ns) + (size_t)chunk * 16 * G;
        out[(size_t)(e & 15) * G + (size_t)pp * P.n_t + t] = v;
    }
}

// out[set][g*16+k] (+)= sum_c partial[set chunks c][k][g], in chunk order
// (deterministic).  Grid: x over 32 directions, y = output set; a warp sums
// two of the 16 elements of 32 consecutive directions (coalesced), and the
// tile goes out through shared memory as 512 consecutive doubles.  `add` false
// stores instead (nothing to clear or read first).  Bound by HBM: the planes
// are read once; writing out[g*16+k] directly from the summing lanes, 128 bytes
// apart, took 522 us for 300 planes of 4,608 directions (177 MB).
__global__ void __launch_bounds__(256) po_reduce_kernel(const double *__restrict__ partial, int chunks_per_set,
                                                        int64_t G, bool add, double *__restrict__ out)
{
    __shared__ double tile[16][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t g0 = (int64_t)blockIdx.x * 32, g = g0 + lane;
    const double *p = partial + (int64_t)blockIdx.y * chunks_per_set * 16 * G + warp * G + g;
    double s0 = 0.0, s1 = 0.0;
    if (g < G) {
#pragma unroll 4
        for (int c = 0; c < chunks_per_set; ++c) {
            s0 += p[(int64_t)c * 16 * G];
            s1 += p[(int64_t)c * 16 * G + 8 * G];
        }
    }
    tile[warp][lane] = s0;
    tile[warp + 8][lane] = s1;
    __syncthreads();
    out += ((int64_t)blockIdx.y * G + g0) * 16;
    const int n = (int)min((int64_t)32, G - g0) * 16;
    for (int i = threadIdx.x; i < n; i += 256) {
        const double v = tile[i & 15][i >> 4];
        out[i] = add ? out[i] + v : v;
    }
}

// Azimuth interpolation of a Mueller grid (the FFT-phi path): for every output
// azimuth p, out[p][r] += sum_m W[p][m] low[m][r], r running over the
// (zenith row, element) entries of one azimuth plane (plane = rows * 16
// doubles, coalesced across the block).  W [n_full][n_low] is the linear map
// of the zero-padded DFT upsampling (see phi_weights on the host); the
// block keeps its output azimuth's row of W in shared memory.
__global__ void __launch_bounds__(256) po_phi_interp_kernel(const double *__restrict__ low,
                                                            const double *__restrict__ W, int n_low,
                                                            int64_t plane, double *__restrict__ out)
{
    extern __shared__ double w_row[];
    const int p = blockIdx.y;
    for (int m = threadIdx.x; m < n_low; m += blockDim.x)
        w_row[m] = W[(size_t)p * n_low + m];
    __syncthreads();
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= plane)
        return;
    double acc = 0.0;
    for (int m = 0; m < n_low; ++m)
        acc = fma(w_row[m], low[(size_t)m * plane + r], acc);
    out[(size_t)p * plane + r] += acc;
}

// ------------------------------------------------------- azimuth average
// Per zenith row t the azimuth average of M(p, t) L(2 az_p), az_p = -p 2 pi / n_az
// (L the Stokes rotation [1 0 0 0; 0 c s 0; 0 -s c 0; 0 0 0 1]), the polar
// rows unrotated and projected (PoleMueller ApplyForward / ApplyBackward),
// as HandlerPOTotal::WriteMatricesToFile writes them (reference
// src/handler/HandlerPOTotal.cpp:49-96).  One CTA per row; threads stride over
// azimuth bins, fixed-order tree sum (deterministic).  rows[t][16].
__global__ void __launch_bounds__(128) po_phi_average_kernel(const double *__restrict__ M, int n_az,
                                                            int n_t, const double *__restrict__ theta,
                                                            double *__restrict__ rows)
{
    __shared__ double red[16][128];
    const int t = blockIdx.x;
    const double th = theta[t];
    const double tol = 256.0 * 2.220446049250313e-16;   // PoleMueller angular tolerance
    const bool fwd = fabs(th) <= tol;
    const bool bwd = fabs(th - kPi) <= tol;
    double S[16];
#pragma unroll
    for (int q = 0; q < 16; ++q)
        S[q] = 0.0;
    for (int p = threadIdx.x; p < n_az; p += blockDim.x) {
        const double *m = M + ((size_t)p * n_t + t) * 16;
        if (fwd || bwd) {
#pragma unroll
            for (int q = 0; q < 16; ++q)
                S[q] += m[q];
            continue;
        }
        double sn, c;
        sincos(2.0 * (-p * (2.0 * kPi / n_az)), &sn, &c);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const double m0 = m[4 * r], m1 = m[4 * r + 1], m2 = m[4 * r + 2], m3 = m[4 * r + 3];
            S[4 * r + 0] += m0;
            S[4 * r + 1] += m1 * c - m2 * sn;
            S[4 * r + 2] += m1 * sn + m2 * c;
            S[4 * r + 3] += m3;
        }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q)
        red[q][threadIdx.x] = S[q];
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int q = 0; q < 16; ++q)
                red[q][threadIdx.x] += red[q][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double R[16];
        for (int q = 0; q < 16; ++q)
            R[q] = red[q][0] / n_az;
        if (fwd || bwd) {
            const double M00 = R[0], M33 = R[15], M03 = R[3];
            const double M11 = bwd ? 0.5 * (R[5] - R[10]) : 0.5 * (R[5] + R[10]);
            for (int q = 0; q < 16; ++q)
                R[q] = 0.0;
            R[0] = M00; R[5] = M11; R[10] = bwd ? -M11 : M11; R[15] = M33;
            R[3] = M03; R[12] = M03;
        }
        for (int q = 0; q < 16; ++q)
            rows[(size_t)t * 16 + q] = R[q];
    }
}

// The same average straight from chunk partial planes [set][16][G] with one
// chunk per set (per-orientation rows): rows[set][t][16].  Grid: x over 32
// zenith rows, y = set; lanes hold consecutive rows (coalesced reads of the
// planes, each read once), the 8 warps take the azimuth bins in turn, and
// their sums meet in a fixed order.  Without it the planes went through
// po_reduce_kernel into cleared grids and from there through
// po_phi_average_kernel: 522 + 33 + 237 us for 300 planes of 96 x 48
// directions; now 48 us in one pass.
__global__ void __launch_bounds__(256) po_phi_rows_kernel(const double *__restrict__ partial, int n_az, int n_t,
                                                         const double *__restrict__ theta,
                                                         double *__restrict__ rows)
{
    __shared__ double red[8][16][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * 32 + lane;
    const size_t G = (size_t)n_az * n_t;
    const double th = theta[min(t, n_t - 1)];
    const double tol = 256.0 * 2.220446049250313e-16;   // PoleMueller angular tolerance
    const bool fwd = fabs(th) <= tol, bwd = fabs(th - kPi) <= tol;
    double S[16];
#pragma unroll
    for (int q = 0; q < 16; ++q)
        S[q] = 0.0;
    if (t < n_t) {
        const double *base = partial + (size_t)blockIdx.y * 16 * G + t;
        for (int p = warp; p < n_az; p += 8) {
            double m[16];
#pragma unroll
            for (int q = 0; q < 16; ++q)
                m[q] = base[q * G + (size_t)p * n_t];
            double sn = 0.0, c = 1.0;
            if (!fwd && !bwd)
                sincos(2.0 * (-p * (2.0 * kPi / n_az)), &sn, &c);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                S[4 * r + 0] += m[4 * r];
                S[4 * r + 1] += m[4 * r + 1] * c - m[4 * r + 2] * sn;
                S[4 * r + 2] += m[4 * r + 1] * sn + m[4 * r + 2] * c;
                S[4 * r + 3] += m[4 * r + 3];
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q)
        red[warp][q][lane] = S[q];
    __syncthreads();
    // element q of row r: the 8 warps' sums in order, then the polar
    // projection (PoleMueller ApplyForward / ApplyBackward)
    for (int i = threadIdx.x; i < 512; i += 256) {
        const int q = i >> 5, r = i & 31;
        double v = red[0][q][r];
        for (int w = 1; w < 8; ++w)
            v += red[w][q][r];
        red[0][q][r] = v / n_az;
    }
    __syncthreads();
    rows += ((size_t)blockIdx.y * n_t + (size_t)blockIdx.x * 32) * 16;
    const int n = min(32, n_t - (int)blockIdx.x * 32) * 16;
    for (int i = threadIdx.x; i < n; i += 256) {
        const int q = i & 15, r = i >> 4;
        const double thr = theta[blockIdx.x * 32 + r];
        const bool f = fabs(thr) <= tol, bw = fabs(thr - kPi) <= tol;
        double v = red[0][q][r];
        if (f || bw) {
            const double m11 = 0.5 * (bw ? red[0][5][r] - red[0][10][r] : red[0][5][r] + red[0][10][r]);
            v = q == 0 || q == 15 || q == 3 ? v : q == 12 ? red[0][3][r] : q == 5 ? m11
              : q == 10 ? (bw ? -m11 : m11) : 0.0;
        }
        rows[i] = v;
    }
}

// Scattering cross-section sum_t M11(t) dcos2pi(t) and the asymmetry
// parameter g = sum_t cos(theta_t) M11(t) dcos2pi(t) / that sum over the
// averaged rows.  One CTA, fixed-order tree sum; out[0] = C_sca, out[1] = g.
__global__ void __launch_bounds__(256) po_csca_kernel(const double *__restrict__ rows, int n_t,
                                                     const double *__restrict__ theta,
                                                     const double *__restrict__ dcos2pi,
                                                     double *__restrict__ out)
{
    __shared__ double a[256], b[256];
    double sa = 0.0, sb = 0.0;
    for (int t = threadIdx.x; t < n_t; t += blockDim.x) {
        const double v = rows[(size_t)t * 16] * dcos2pi[t];
        sa += v;
        sb += cos(theta[t]) * v;
    }
    a[threadIdx.x] = sa;
    b[threadIdx.x] = sb;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            a[threadIdx.x] += a[threadIdx.x + w];
            b[threadIdx.x] += b[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = a[0];
        out[1] = a[0] != 0.0 ? b[0] / a[0] : 0.0;
    }
}

// ------------------------------------------------------------ theta scan
// Incoherent, azimuth-summed M11 on a list of zenith angles (reference
// theta_m11_kernel, GpuDiffraction.cu:1909-1956, called by DiffractThetasGpu
// :4780-4970).  Grid: x = (azimuth bin, tile of TPB * DPT zenith points),
// y = beam chunk.  As in po_diffract_kernel the CTA folds its azimuth into
// per-beam records in shared memory once and every thread evaluates its
// points' edge sums from them.  No common phase is needed, so the vertex phases
// are k (A x + B y) / 2 pi: the rounding of A and B is the same in them and in
// the edge coefficients (phases folded over the azimuth like
// po_diffract_kernel's left 40 times the error at an edge just above eps1).
// Per pair only |s|^2 |R|^2 is
// needed, R = P0 + cos t Pc + sin t Ps having eight real components: the record
// holds the triangular factor U of the 8 x 3 matrix (P0, Pc, Ps), and
// |R| = |U (1, cos t, sin t)| takes 8 operations instead of 24, with the same
// error of some eps |P| in R (opposite to a beam's direction R vanishes by
// cancellation: |R|^2 as a quadratic form in (cos t, sin t) is wrong by eps |P|^2
// there, 13 % of a shadow beam's value at 179.99 degrees).  Small-phase
// candidates are marked and evaluated in general form after the stage.
// Bound by the FP64 pipe.  One thread per (point, beam, azimuth) with the
// general evaluation took 1,225 us for 2,088 beams x 48 x 181 points, now
// 245 us (229 with the quadratic form).
struct __align__(16) ThetaBeam {
    double a[6];        // A, B coefficients (see BeamRegs)
    double u[6];        // U by rows: u00 u01 u02 u11 u12 u22
    double slab[4];
    double w;           // 0.5 weight
    int nv, vs;
};
// Modified Gram-Schmidt steps over 8 components: x becomes a unit vector, its
// length returned (the zero vector stays); y loses its component along the unit
// vector x, returned.
__device__ __forceinline__ double take_column(double *x)
{
    double n = 0.0;
#pragma unroll
    for (int e = 0; e < 8; ++e)
        n = fma(x[e], x[e], n);
    n = sqrt(n);
    const double inv = n > 0.0 ? 1.0 / n : 0.0;
#pragma unroll
    for (int e = 0; e < 8; ++e)
        x[e] *= inv;
    return n;
}

__device__ __forceinline__ double take_component(const double *x, double *y)
{
    double c = 0.0;
#pragma unroll
    for (int e = 0; e < 8; ++e)
        c = fma(x[e], y[e], c);
#pragma unroll
    for (int e = 0; e < 8; ++e)
        y[e] = fma(-c, x[e], y[e]);
    return c;
}

constexpr int kThetaTpb = 64;
constexpr int kThetaBeams = 64;                // beams and vertices of a stage
constexpr int kThetaVerts = 4 * kThetaBeams;

template <int DPT>
__global__ void __launch_bounds__(kThetaTpb, 4) po_thetas_kernel(
    KParams P, int64_t n_beams, int beams_per_chunk, int tiles, const double *st_tab, const double *ct_tab,
    int n_points, double *out_partial)
{
    constexpr int TPB = kThetaTpb;
    __shared__ ThetaBeam sb[kThetaBeams];
    __shared__ SVertRaw<double> sv[kThetaVerts];
    __shared__ double2 s_sincos[kSinTab];
    fill_sincos_tab(s_sincos, TPB);
    const int p = blockIdx.x / tiles, tile = blockIdx.x - p * tiles;
    const double cp = P.cphi[p], sp = P.sphi[p], kt = P.wc.k * kInvTwoPi;
    const int64_t b0 = (int64_t)blockIdx.y * beams_per_chunk;
    const int64_t b1 = min(n_beams, b0 + beams_per_chunk);
    const int t0 = tile * TPB * DPT + threadIdx.x;
    double st[DPT], ct[DPT], acc[DPT];
#pragma unroll
    for (int d = 0; d < DPT; ++d) {
        const int t = min(t0 + d * TPB, n_points - 1);
        st[d] = st_tab[t];
        ct[d] = ct_tab[t];
        acc[d] = 0.0;
    }
    for (int64_t bs = b0; bs < b1;) {
        // stage [bs, be): at most kThetaBeams beams and kThetaVerts vertices
        const int vb0 = P.vbeg[bs];
        int64_t be = min(b1, bs + kThetaBeams);
        if (P.vbeg[be] - vb0 > kThetaVerts) {
            int64_t lo = bs + 1, hi = be;
            while (lo < hi) {
                const int64_t mid = (lo + hi + 1) >> 1;
                if (P.vbeg[mid] - vb0 <= kThetaVerts) lo = mid; else hi = mid - 1;
            }
            be = lo;
        }
        const int nb = (int)(be - bs), nvs = P.vbeg[be] - vb0;
        __syncthreads();   // the previous stage is consumed
        for (int i = threadIdx.x; i < nb; i += TPB) {
            const BrecRef r{P.brec + bs + i, P.brec_stride};
            ThetaBeam &s = sb[i];
            s.a[0] = -(cp * r.ab(0) + sp * r.ab(1)); s.a[1] = r.ab(2); s.a[2] = r.ab(3);
            s.a[3] = -(cp * r.ab(4) + sp * r.ab(5)); s.a[4] = r.ab(6); s.a[5] = r.ab(7);
            // orientation of the beam: last o with beam_off[o] <= b
            int lo = 0, hi = P.n_orient;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (P.beam_off[mid] <= bs + i) lo = mid; else hi = mid;
            }
            const double w = 0.5 * P.weight[lo];
            double p0[8], pc[8], ps[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                p0[e] = sp * r.Q(e) + cp * r.Q(8 + e);
                pc[e] = -(cp * r.Q(16 + e) + sp * r.Q(24 + e));
                ps[e] = r.Q(32 + e);
            }
            s.u[0] = take_column(p0);
            s.u[1] = take_component(p0, pc);
            s.u[2] = take_component(p0, ps);
            s.u[3] = take_column(pc);
            s.u[4] = take_component(pc, ps);
            s.u[5] = take_column(ps);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                s.slab[e] = r.slab(e);
            s.w = w;
            s.nv = r.nv();
            s.vs = P.vbeg[bs + i] - vb0;
        }
        for (int i = threadIdx.x; i < nvs; i += TPB) {
            const DevVert v = P.verts[vb0 + i];
            sv[i].q[0] = make_double2(kt * v.x, kt * v.y);
            sv[i].q[1] = make_double2(0.0, isnan(v.syx) ? kInvalidSlope : v.syx);
            sv[i].q[2] = make_double2(isnan(v.sxy) ? kInvalidSlope : v.sxy, 0.0);
        }
        __syncthreads();
        uint64_t marked[DPT];
#pragma unroll
        for (int d = 0; d < DPT; ++d)
            marked[d] = 0;
        for (int j = 0; j < nb; ++j) {
            const ThetaBeam &b = sb[j];
            double A_[DPT], B_[DPT], X1[DPT], X2[DPT], sr[DPT], si[DPT], m[DPT];
            uint32_t mn[DPT];
            bool useX[DPT], cand[DPT];
#pragma unroll
            for (int d = 0; d < DPT; ++d) {
                const double A = fma(st[d], b.a[0], fma(ct[d], b.a[1], b.a[2]));
                const double B = fma(st[d], b.a[3], fma(ct[d], b.a[4], b.a[5]));
                A_[d] = A;
                B_[d] = B;
                useX[d] = fabs(B) > fabs(A);
                X1[d] = useX[d] ? B : A;
                X2[d] = useX[d] ? A : B;
                m[d] = X1[d];                       // |s|^2 takes 1 / X1^2
                cand[d] = fabs(fma(A, b.slab[0], B * b.slab[1])) <= 1.0
                       && fabs(fma(A, b.slab[2], B * b.slab[3])) <= 1.0;
            }
            // the phases' factors are (A, B) in place of (sin t, cos t)
            edge_sums<DPT, true>(sv + b.vs, b.nv, A_, B_, X1, X2, useX, sr, si, mn, s_sincos, P.wc.eps1);
#pragma unroll
            for (int d = 0; d < DPT; ++d) {
                const double y0 = fma(st[d], b.u[2], fma(ct[d], b.u[1], b.u[0]));
                const double y1 = fma(st[d], b.u[4], ct[d] * b.u[3]), y2 = st[d] * b.u[5];
                const double q = fma(y0, y0, fma(y1, y1, y2 * y2));   // |R|^2
                const double r = rcp64(m[d]);
                const double xr = sr[d] * r, xi = si[d] * r;
                const double s2 = fma(xr, xr, xi * xi);
                // a candidate's sums may be inf or NaN: select; a beam without a
                // finite integral is left out, a NaN weight or Jones matrix is not
                acc[d] += cand[d] || !isfinite(s2) ? 0.0 : s2 * q * b.w;
                if (cand[d])
                    marked[d] |= 1ull << j;
            }
        }
#pragma unroll
        for (int d = 0; d < DPT; ++d) {
            if (marked[d] == 0)
                continue;
            DirFull dc;
            dc.st = st[d];
            dc.ct = ct[d];
            dc.cp = cp;
            dc.sp = sp;
            dc.dir[0] = dc.st * dc.cp;
            dc.dir[1] = dc.st * dc.sp;
            dc.dir[2] = -dc.ct;
            dc.vf[0] = -dc.sp; dc.vf[1] = dc.cp; dc.vf[2] = 0.0;
            cross3(dc.vf, dc.dir, dc.u);
            const double l2 = dc.u[0] * dc.u[0] + dc.u[1] * dc.u[1] + dc.u[2] * dc.u[2];
            const double il = (l2 > 1e-30) ? rsqrt(l2) : 1.0;
            dc.vt[0] = dc.u[0] * il; dc.vt[1] = dc.u[1] * il; dc.vt[2] = dc.u[2] * il;
            cross3(dc.vt, dc.dir, dc.w);
            while (marked[d]) {
                const int j = __ffsll((long long)marked[d]) - 1;
                marked[d] &= marked[d] - 1;
                double x[8];
                if (beam_general(P.beams[bs + j], P.verts, dc, P.wc, x, false)) {
                    double e = 0.0;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        e = fma(x[q], x[q], e);
                    acc[d] = fma(e, sb[j].w, acc[d]);
                }
            }
        }
        bs = be;
    }
    double *out = out_partial + ((size_t)blockIdx.y * P.n_az + p) * n_points;
#pragma unroll
    for (int d = 0; d < DPT; ++d)
        if (t0 + d * TPB < n_points)
            out[t0 + d * TPB] = acc[d];
}

// m11[t] = sum over rows r of partial[r][t], over n_az + 1: 32 points per CTA, the 32 warps
// take rows in turn, four sums a thread, and the 32 sums of a point meet in a
// tree (deterministic).  Around the poles every azimuth bin adds the same
// value, whose roundings go the same way: added one after the other they
// reach ten units of the last place.
__global__ void __launch_bounds__(1024) po_thetas_sum_kernel(const double *partial, int64_t n_rows, int n_points,
                                                            int n_az, double *m11)
{
    __shared__ double red[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * 32 + lane;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    if (t < n_points) {
        for (int64_t r = warp; r < n_rows; r += 128)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (r + 32 * i < n_rows)
                    s[i] += partial[(r + 32 * i) * n_points + t];
    }
    red[warp][lane] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    double v = red[lane][warp];              // point `warp` of the CTA
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0 && blockIdx.x * 32 + warp < n_points)
        m11[blockIdx.x * 32 + warp] = v / (double)(n_az + 1);
}

// --------------------------------------------------------- extinction
// HandlerPO::ComputeForwardExtinctionOt (reference HandlerPO.cpp:1812-2009) at
// zenith 0, azimuth 0: `slices` warps per orientation, lanes striding over its
// beams, sums in a fixed order.  Each beam is one general evaluation (a chain
// of loads and FP64 operations), so the time is the number of beams a lane
// takes in turn: one thread per orientation took 1,186 us for 1,024
// orientations of 87 beams.
constexpr int kExtThreads = 128;

__global__ void __launch_bounds__(kExtThreads) po_extinction_kernel(
    const DevBeam *beams, const DevVert *verts, const int32_t *beam_off, const double *weight,
    int n_orient, int slices, WaveConst wc, double *cext)
{
    __shared__ double part[kExtThreads / 32][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = warp / slices, slice = warp - grp * slices;
    const int o = blockIdx.x * ((kExtThreads / 32) / slices) + grp;
    const double k = wc.k;
    DirFull dc;
    dc.st = 0.0; dc.ct = 1.0; dc.cp = 1.0; dc.sp = 0.0;
    dc.dir[0] = 0.0; dc.dir[1] = 0.0; dc.dir[2] = -1.0;
    dc.vf[0] = 0.0; dc.vf[1] = 1.0; dc.vf[2] = 0.0;
    cross3(dc.vf, dc.dir, dc.u);
    dc.vt[0] = dc.u[0]; dc.vt[1] = dc.u[1]; dc.vt[2] = dc.u[2];
    cross3(dc.vt, dc.dir, dc.w);
    double f[4] = {0.0, 0.0, 0.0, 0.0};   // S00 and S11 (re, im)
    const int b1 = o < n_orient ? beam_off[o + 1] : 0;
    for (int b = (o < n_orient ? beam_off[o] : 0) + slice * 32 + lane; b < b1; b += slices * 32) {
        const DevBeam &g = beams[b];
        const bool external = (g.flags & MBS_PO_BEAM_EXTERNAL) != 0;
        if (wc.ot_phase_avg && !external)
            continue;
        // The extinction phase reference differs from the scattering one
        // (HandlerPO.cpp:1965-1977): external beams take exp(-ik opticalPath),
        // internal ones exp(-ik(cos t dp_cos + farReference)), so beam_general
        // runs without the common phase and that factor is applied here.
        const double ref = external ? g.opath : wc.ot_far_ref;
        // The reference drops beams whose 1/A or 1/B divisor is nearly
        // singular at this direction (HandlerPO.cpp:1920-1921, 1945-1946).
        const double A = g.h[2] + g.a0, B = g.v[2] + g.b0;
        double dd[8], pr, pi;
        if (((fabs(B) > fabs(A)) ? fabs(B) <= wc.eps1 : fabs(A) <= wc.eps1)
            && !small_phase_factor(verts + g.vbeg, g.nv, A, B, k, pr, pi))
            continue;
        if (!beam_general(g, verts, dc, wc, dd, true, false))
            continue;
        double ph = 0.0;
        if (!external)
            ph = -k * (1.0 * (-g.c[2]) + ref);
        else if (ref != 0.0)
            ph = -k * ref;
        double s = 0.0, c = 1.0;
        if (ph != 0.0)
            sincos_rad(ph, s, c);
        // the CPU rotation carries 0.5 (HandlerPO_fast.h:643-646)
        f[0] += 0.5 * (dd[0] * c - dd[1] * s); f[1] += 0.5 * (dd[0] * s + dd[1] * c);
        f[2] += 0.5 * (dd[6] * c - dd[7] * s); f[3] += 0.5 * (dd[6] * s + dd[7] * c);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            f[i] += __shfl_xor_sync(0xffffffffu, f[i], off);
        if (lane == 0)
            part[warp][i] = f[i];
    }
    __syncthreads();
    if (slice != 0 || lane != 0 || o >= n_orient)
        return;
    for (int s = 1; s < slices; ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            f[i] += part[warp + s][i];
    const double fwr = f[0] + f[2], fwi = f[1] + f[3];
    double amp = fwi;
    if (wc.ot_ping != 0.0) {
        double sn, cs;
        sincos_rad(2.0 * k * wc.ot_ping, sn, cs);
        amp = fwi * cs - fwr * sn;
    }
    const double cv = wc.wavelength * amp * weight[o];
    cext[o] = isfinite(cv) ? cv : 0.0;
}

// ------------------------------------------------------------ peak probe
// Independent FFMA chains: this device's FP32 FMA throughput, the
// denominator of the diffraction kernels' roofline fraction.
__global__ void __launch_bounds__(256) po_fp32_probe_kernel(float *out, int iters, float a, float b)
{
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        x[i] = threadIdx.x * 1e-3f + i;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                x[i] = fmaf(x[i], a, b);
        }
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        s += x[i];
    if (s == 1234.5f)
        out[blockIdx.x] = s;
}

// Independent DFMA chains: this device's FP64 FMA throughput, the
// denominator of the FP64 diffraction kernel's roofline fraction.
__global__ void __launch_bounds__(256) po_fp64_probe_kernel(double *out, int iters, double a, double b)
{
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        x[i] = threadIdx.x * 1e-3 + i;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                x[i] = fma(x[i], a, b);
        }
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        s += x[i];
    if (s == 1234.5)
        out[blockIdx.x] = s;
}

}  // namespace mbs
