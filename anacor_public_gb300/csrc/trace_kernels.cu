// sm_103a kernels of the absorption-factor path.
//
// One warp processes one work item = (sample, reflection, tile of consecutive
// voxels of the packed list) taken from an atomic counter, so a warp that
// finishes early takes the next item instead of waiting for its CTA.  Lane k
// takes voxels tile*t + k + 32*j: the 32 lanes hold 32 consecutive entries of
// the Morton-ordered list (a compact 3-D block) and march them along the same
// two directions.
//
// Per voxel (the body of AnACor/src/ray_tracing.c:199-278), per leg:
//   exit face  (cube_face, ray_tracing_basic.c:69-186): FP32 estimate of the
//              three candidate distances, exact FP64 division only when the
//              two smallest are within 2^-20 relative.
//   march      (cal_coord, :396-1460), warp-cooperative: lanes leaving through
//              the same face share its step rule and differ only by an integer
//              start offset, so one lane per increment computes the 32.32
//              fixed-point displacement and the warp broadcasts it; each lane
//              loads its label at base + displacement, eight increments in
//              flight, and checks four labels per packed word.  Increments
//              whose fraction lies within kAmbiguityMargin of a rounding
//              boundary are recomputed with the reference's FP64 expression.
//              Lanes that may touch a volume wall, faces with ratios beyond
//              fixed-point range and full_iteration march per lane in FP64.
//              Field variants: each lane marches alone on a packed label +
//              chessboard-distance field (centred, or one per direction
//              octant) and steps over the increments the field proves to keep
//              their label; stops, class changes and len_path_2 are those of
//              the per-increment march.
//   lengths    (cal_path2_plus, :1462-1552): for A_h in FP32 (the segments and
//              len_path_2 come from the exact march; A_h needs 1e-6); for the
//              per-voxel detail and the gridding map in FP64 with the
//              reference's operation order, the per-segment quotient
//              fl(span / (len-1)) from a table of correctly rounded quotients,
//              or a correctly rounded reciprocal and one FMA correction.  A
//              leg that stopped at vacuum takes its last point from the march.
//   rate       (cal_rate, :1554-1583): FP32 exponent and exp; sums of three
//              floats (FloatSum) a lane, warp, tile and reflection, rounded
//              once (the same bits for any schedule and cut into tiles).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <cstdlib>

#include "anacor_internal.h"
#include "device_math.cuh"
#include "trace_launch.h"

namespace anacor {

// g_num_rcp[d] = {(double)d, fl(1 / d)}: the quotient's operands without an
// integer-to-double conversion on the FP64 pipe
__device__ double2 g_num_rcp[kMaxDim + 2];

namespace {

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
// CTAs per SM the absorption kernel's register budget is sized for: the
// kernel is instantiated for 1..4 (times the two marches); the plan's
// variant, or the process default (ANACOR_CTAS_PER_SM, default
// kDefaultMinBlocks), picks one.
constexpr int kDefaultMinBlocks = 4;
// Label loads a lane has in flight before checking them (divides 32).
constexpr int kMarchBatch = 8;
constexpr unsigned kAll = 0xffffffffu;

// The kernels' shared arrays (per-warp tables, segment lists, lane sums) are
// sized for kBlock threads.  A launch with any other block shape sets the
// ANACOR_ERR_ARGS bit in `status` (from one thread) and returns before any
// shared or global access; the test is uniform over the block, so no thread
// is left waiting at a barrier.
__device__ __forceinline__ bool block_shape_ok(int *status)
{
    if (blockDim.x == kBlock && blockDim.y == 1 && blockDim.z == 1)
        return true;
    if (status && threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0)
        atomicOr(status, 1 << kErrArgs);
    return false;
}

struct Vol {
    const int8_t *p;
    int dz, dy, dx;
    const uint8_t *field = nullptr;   // label | distance << 3, for the distance-field march
    long long field_stride = 0;       // 0: one centred field; else 8 octant fields this far apart
    int bsy = 0, bsz = 0;             // bricked fields: byte strides of a brick step in y and z
};

// Offset of voxel (z, y, x) in a field stored in 4x4x4 bricks of 64 bytes:
// bricks in (z, y, x) order, bytes inside a brick (z, y, x) with x fastest, so
// a 32-byte sector holds a 2x4x4 (z, y, x) box.  A ray that steps by one voxel
// along any axis mostly stays in the sector its previous load brought into L1
// (in the linear layout only steps along x do).
//
// Axis coordinate u = 4 U + w contributes U * BS + w * IS (BS the axis's
// brick stride, IS its stride inside a brick), which equals
// (u & ~3) * K + u * IS with K = BS / 4 - IS: a mask and two multiply-adds.
__device__ __forceinline__ int brick_term(int u, int k, int is)
{
    return (u & ~3) * k + u * is;
}

// K and IS of axis a (0 z, 1 y, 2 x)
__device__ __forceinline__ int brick_k(int a, const Vol &v)
{
    return a == 0 ? v.bsz / 4 - 16 : (a == 1 ? v.bsy / 4 - 4 : 64 / 4 - 1);
}

__device__ __forceinline__ int brick_is(int a)
{
    return 16 >> (2 * a);
}

__device__ __forceinline__ int brick_offset(int z, int y, int x, const Vol &v)
{
    return brick_term(z, brick_k(0, v), 16) + brick_term(y, brick_k(1, v), 4) + brick_term(x, brick_k(2, v), 1);
}

__device__ __forceinline__ int pick3(int k, int z, int y, int x)
{
    return k == 0 ? z : (k == 1 ? y : x);
}

// C's `int64_t n = floor(v)` / `round(v)`, then the reference's clamp.
// Out-of-range and NaN conversions give INT64_MIN (x86-64 behaviour).
__device__ __noinline__ int exact_axis(int c, int i, double q, bool use_round, int dim)
{
    const double v = __dadd_rn((double)c, __dmul_rn((double)i, q));
    const double r = use_round ? round(v) : floor(v);
    long long n;
    if (!(r >= -9223372036854775808.0 && r < 9223372036854775808.0))
        n = LLONG_MIN;
    else
        n = (long long)r;
    if (n >= dim)
        n = dim - 1;
    else if (n < 0)
        n = 0;
    return (int)n;
}

// Exit face of the ray from (cz, cy, cx).  Returns the face code 1..6 or 0.
__device__ __forceinline__ int exit_face(const LegHead &h, int cz, int cy, int cx, const Vol &v)
{
    // A zero distance (origin on a min plane, non-zero component) wins; ties
    // follow the reference's test order x_min, y_min, z_min.
    const uint32_t sb = h.sign_bits;
    const bool hx = (sb & (4u | 32u)) != 0, hy = (sb & (2u | 16u)) != 0, hz = (sb & (1u | 8u)) != 0;
    if (cx == 0 && hx) return 6;
    if (cy == 0 && hy) return 4;
    if (cz == 0 && hz) return 2;
    // one candidate per axis: numerator n_a
    const int nx = (sb & 4u) ? v.dx - cx : cx;
    const int ny = (sb & 2u) ? v.dy - cy : cy;
    const int nz = (sb & 1u) ? v.dz - cz : cz;
    const float inf = __int_as_float(0x7f800000);
    const float tx = hx ? (float)nx * h.inv[2] : inf;
    const float ty = hy ? (float)ny * h.inv[1] : inf;
    const float tz = hz ? (float)nz * h.inv[0] : inf;
    // argmin with ties to the earlier axis (x, y, z)
    int best = 2;
    float t1 = tx, t2;
    if (ty < t1) { t2 = t1; t1 = ty; best = 1; } else { t2 = ty; }
    if (tz < t1) { t2 = t1; t1 = tz; best = 0; } else { t2 = fminf(t2, tz); }
    if ((sb & 64u) || !(t1 < inf && t2 > t1 * (1.0f + 0x1p-20f))) {
        // close call: the reference's FP64 quotients decide
        const double dinf = __longlong_as_double(0x7ff0000000000000ll);
        const double ex = hx ? __ddiv_rn((double)nx, fabs(h.e[2])) : dinf;
        const double ey = hy ? __ddiv_rn((double)ny, fabs(h.e[1])) : dinf;
        const double ez = hz ? __ddiv_rn((double)nz, fabs(h.e[0])) : dinf;
        best = 2;
        double b = ex;
        if (ey < b) { b = ey; best = 1; }
        if (ez < b) { b = ez; best = 0; }
        if (!(b < dinf))
            return 0;
    }
    const bool pos = (sb >> best) & 1u;
    // faces: x: 1 max / 6 min, y: 5 max / 4 min, z: 3 max / 2 min
    if (best == 2) return pos ? 1 : 6;
    if (best == 1) return pos ? 5 : 4;
    return pos ? 3 : 2;
}

// fl(span / den): from the quotient table (row den holds span = 1 .. den+1)
// or from rcp = fl(1/den) with one FMA-exact remainder and one correction.
__device__ __forceinline__ double seg_quotient(const double *qtab, int den_i, int span, double den, double rcp)
{
    if (qtab)
        return __ldg(qtab + ((den_i - 1) * (den_i + 2)) / 2 + (span - 1));
    const double s = g_num_rcp[span].x;
    const double q0 = __dmul_rn(s, rcp);
    const double r = __fma_rn(-q0, den, s);
    return __fma_rn(r, rcp, q0);
}

// L[cls-1] += term in segment order.  The first term of a class is stored
// as is (0.0 + term == term for the non-negative terms of cal_path2_plus).
__device__ __forceinline__ void add_class(int cls, double term, int &seen, double *L)
{
    if (cls < 1 || cls > 4)
        return;
    const int bit = 1 << cls;
    double nv = term;
    if (seen & bit) {
        const double cur = cls == 1 ? L[0] : (cls == 2 ? L[1] : (cls == 3 ? L[2] : L[3]));
        nv = __dadd_rn(cur, term);
    }
    seen |= bit;
    L[0] = cls == 1 ? nv : L[0];
    L[1] = cls == 2 ? nv : L[1];
    L[2] = cls == 3 ? nv : L[2];
    L[3] = cls == 4 ? nv : L[3];
}

// Per-leg march state.  Accepted path points are the increments 0..last_i
// (the march never skips one), so len_path_2 = last_i + 1.
struct March {
    int last_i, nseg, prev, vac;
};

// Where class changes go: mode 0 records (class, start) in shared memory;
// mode 1 (second pass, when a leg has more class changes than the shared
// buffer holds) accumulates the lengths directly.
struct Sink {
    uint16_t *seg;      // stride kBlock
    const double *qtab;
    double tot, den, rcp;
    int den_i;
    double L[4];
    int open_cls, open_pos, seen;
};

template <int kMode>
__device__ __forceinline__ bool visit(March &m, Sink &sk, int i, int lab, int full, int vac_limit)
{
    if (!full) {
        if (lab == 0)
            return false;
    } else {
        m.vac = lab == 0 ? m.vac + 1 : 0;
        if (m.vac > vac_limit)
            return false;
    }
    if (lab != m.prev && (unsigned)lab <= 4u) {
        if (kMode == 0) {
            if (m.nseg < kMaxSegments)
                sk.seg[m.nseg * kBlock] = (uint16_t)((lab << 13) | i);
        } else {
            const double q = seg_quotient(sk.qtab, sk.den_i, i - sk.open_pos, sk.den, sk.rcp);
            add_class(sk.open_cls, __dmul_rn(sk.tot, q), sk.seen, sk.L);
            sk.open_cls = lab;
            sk.open_pos = i;
        }
        m.nseg++;
    }
    m.last_i = i;
    m.prev = lab;
    return true;
}

// Geometry of one leg through one exit face in the face's own axis order:
// s = the step axis (the reference's loop axis, ratio exactly +-1), a and b
// the two other axes (32.32 fixed point).
struct LegGeom {
    int cs, ca, cb;          // start coordinates
    int hs, ha, hb;          // dim - 1
    int Ss, Sa, Sb;          // element strides
    int ds;                  // step direction (+1 / -1)
    int ia, ib;              // axis index (0 z, 1 y, 2 x) of a and b
    long long Qa, Qb;
    uint32_t Ma, Mb;         // ambiguity margins (0 for exact axes)
    long long off;           // 2^31 for round mode
};

__device__ __forceinline__ void leg_geom(const FaceRule &R, int cz, int cy, int cx, const Vol &v, LegGeom &g)
{
    const int s = R.count_axis;
    const int a = s == 0 ? 1 : 0;
    const int b = s == 2 ? 1 : 2;
    g.ia = a; g.ib = b;
    g.cs = pick3(s, cz, cy, cx); g.ca = pick3(a, cz, cy, cx); g.cb = pick3(b, cz, cy, cx);
    g.hs = pick3(s, v.dz, v.dy, v.dx) - 1; g.ha = pick3(a, v.dz, v.dy, v.dx) - 1;
    g.hb = pick3(b, v.dz, v.dy, v.dx) - 1;
    const int sz = v.dy * v.dx, sy = v.dx;
    g.Ss = pick3(s, sz, sy, 1); g.Sa = pick3(a, sz, sy, 1); g.Sb = pick3(b, sz, sy, 1);
    g.ds = R.Q[s] > 0 ? 1 : -1;   // the step axis's ratio is exactly +-1, so Q[s] = +-2^32
    g.Qa = R.Q[a]; g.Qb = R.Q[b];
    g.Ma = ((R.exact_mask >> a) & 1) ? 0u : kAmbiguityMargin;
    g.Mb = ((R.exact_mask >> b) & 1) ? 0u : kAmbiguityMargin;
    g.off = R.use_round ? 0x80000000ll : 0ll;
}

// Path point at increment i, (z, y, x).
__device__ __forceinline__ void point_at(const FaceRule &R, const LegGeom &g, int i, int cz, int cy, int cx,
                                         const Vol &v, int &pz, int &py, int &px)
{
    if (R.fast) {
        const int ps = min(max(g.cs + i * g.ds, 0), g.hs);
        const long long Ea = ((long long)g.ca << 32) + g.off + (long long)i * g.Qa;
        const long long Eb = ((long long)g.cb << 32) + g.off + (long long)i * g.Qb;
        int pa, pb;
        if (((uint32_t)Ea + g.Ma < 2u * g.Ma) | ((uint32_t)Eb + g.Mb < 2u * g.Mb)) {
            pa = exact_axis(g.ca, i, R.q[g.ia], R.use_round, g.ha + 1);
            pb = exact_axis(g.cb, i, R.q[g.ib], R.use_round, g.hb + 1);
        } else {
            pa = min(max((int)(Ea >> 32), 0), g.ha);
            pb = min(max((int)(Eb >> 32), 0), g.hb);
        }
        const int s = R.count_axis;
        pz = s == 0 ? ps : pa;
        py = s == 1 ? ps : (s == 0 ? pa : pb);
        px = s == 2 ? ps : pb;
    } else {
        pz = exact_axis(cz, i, R.q[0], R.use_round, v.dz);
        py = exact_axis(cy, i, R.q[1], R.use_round, v.dy);
        px = exact_axis(cx, i, R.q[2], R.use_round, v.dx);
    }
}

// Per-lane march (cal_coord) for the lanes the cooperative march does not
// take: walls within reach, huge ratios, full_iteration; the second pass; and
// (i_begin > 0) the increments after the cooperative part of a leg that did
// not stop before the cooperative march's wall limit, continuing `m`.
//
// Out of line, with everything it needs passed by value or recomputed: a
// by-reference argument whose object lives in the caller's registers would
// move that object to the stack for the whole of the caller.
template <int kMode>
__device__ __noinline__ void march_lane(const FaceRule &R, int cz, int cy, int cx, int steps, const Vol v, int full,
                                        March &m, Sink &sk, int i_begin = 0)
{
    LegGeom g;
    leg_geom(R, cz, cy, cx, v, g);
    const int sz = v.dy * v.dx, sy = v.dx;
    int z, y, x;
    if (i_begin > 0) {
        for (int i = i_begin; i < steps; i++) {
            point_at(R, g, i, cz, cy, cx, v, z, y, x);
            if (!visit<kMode>(m, sk, i, __ldg(v.p + (z * sz + y * sy + x)), full, R.vac_limit))
                return;
        }
        return;
    }
    m.last_i = 0; m.nseg = 1; m.vac = 0;
    if (kMode == 0)
        sk.seg[0] = (uint16_t)(3 << 13);
    if (steps <= 0)
        return;
    point_at(R, g, 0, cz, cy, cx, v, z, y, x);
    const int lab = __ldg(v.p + (z * sz + y * sy + x));
    if (!full) {
        if (lab == 0)
            return;
    } else {
        m.vac = lab == 0;
        if (m.vac > R.vac_limit)
            return;
    }
    m.prev = lab;
    for (int i = 1; i < steps; i++) {
        point_at(R, g, i, cz, cy, cx, v, z, y, x);
        if (!visit<kMode>(m, sk, i, __ldg(v.p + (z * sz + y * sy + x)), full, R.vac_limit))
            return;
    }
}

// Byte of `bytes` (the label volume or its packed distance field) at
// increment `inc`, from the reference's FP64 expression (an increment whose
// fixed-point fraction lies near a rounding boundary).
__device__ __noinline__ uint32_t exact_byte(const FaceRule &G, int cz, int cy, int cx, int inc, const Vol v,
                                            const uint8_t *bytes, bool brick)
{
    int pz, py, px;
    const int s = G.count_axis;
    const int ds = G.q[s] > 0.0 ? 1 : -1;
    pz = s == 0 ? cz + inc * ds : exact_axis(cz, inc, G.q[0], G.use_round, v.dz);
    py = s == 1 ? cy + inc * ds : exact_axis(cy, inc, G.q[1], G.use_round, v.dy);
    px = s == 2 ? cx + inc * ds : exact_axis(cx, inc, G.q[2], G.use_round, v.dx);
    return (uint32_t)__ldg(bytes + (brick ? brick_offset(pz, py, px, v) : (pz * v.dy + py) * v.dx + px));
}

__device__ __forceinline__ uint32_t exact_label(const FaceRule &G, int cz, int cy, int cx, int inc, const Vol &v)
{
    return exact_byte(G, cz, cy, cx, inc, v, reinterpret_cast<const uint8_t *>(v.p), false);
}

// Increments i >= 0 for which c + i*q stays at least 2 voxels inside [0, h]
// (an estimate in FP32 with a margin; -1 when increment 0 is already too
// close).  The cooperative march's end-point test decides; this only picks
// the end point.
__device__ __forceinline__ int wall_increments(double q, int c, int h)
{
    const float qf = (float)q;
    float k;
    if (qf > 0.0f)
        k = __fdiv_rn((float)(h - 2 - c), qf);
    else if (qf < 0.0f)
        k = __fdiv_rn((float)(c - 2), -qf);
    else
        return (c >= 1 && c <= h - 1) ? 0x3fffffff : -1;
    if (!(k >= 0.0f))
        return -1;
    return (int)fminf(floorf(k * 0.9999f), 1.0e9f);
}

// fl(fl(d * v_axis)^2), from the sample's table when it has one
__device__ __forceinline__ double sq_len(const double *sq, int stride, int axis, int d, double vox)
{
    if (sq)
        return __ldg(sq + axis * stride + d);
    const double t = __dmul_rn((double)d, vox);
    return __dmul_rn(t, t);
}

struct L4 {
    double v[4];
};

// cal_path2_plus by a second march, accumulating segments as they close (a
// leg with more class changes than the shared buffer holds), out of line.
__device__ __noinline__ L4 lengths_second_pass(const FaceRule &R, int cz, int cy, int cx, int steps, const Vol v,
                                               int full, int len, int fz, int fy, int fx, int lz, int ly, int lx,
                                               const double *voxel, const double *sq, int sq_stride,
                                               const double *qtab, uint16_t *seg)
{
    const double yy = sq_len(sq, sq_stride, 1, abs(ly - fy), voxel[1]);
    const double zz = sq_len(sq, sq_stride, 0, abs(lz - fz), voxel[0]);
    const double xx = sq_len(sq, sq_stride, 2, abs(lx - fx), voxel[2]);
    const double tot = __dsqrt_rn(__dadd_rn(__dadd_rn(yy, zz), xx));
    const int den_i = len - 1;
    const double2 dr = g_num_rcp[den_i];
    March m2;
    Sink s2;
    s2.seg = seg;
    s2.qtab = qtab;
    s2.tot = tot; s2.den = dr.x; s2.rcp = dr.y; s2.den_i = den_i;
    s2.L[0] = s2.L[1] = s2.L[2] = s2.L[3] = 0.0;
    s2.open_cls = 3; s2.open_pos = 0; s2.seen = 0;
    march_lane<1>(R, cz, cy, cx, steps, v, full, m2, s2);
    const double q = seg_quotient(qtab, den_i, len - s2.open_pos, dr.x, dr.y);
    add_class(s2.open_cls, __dmul_rn(tot, q), s2.seen, s2.L);
    L4 r;
    for (int k = 0; k < 4; k++)
        r.v[k] = s2.L[k];
    return r;
}

struct LegResult {
    double L[4];       // FP64 lengths (kF32 == false)
    float Lf[4];       // FP32 lengths (kF32 == true)
    int face, len, nseg, status;
    int first[3], last[3];
};


// cal_path2_plus in FP32 for A_h: total = |(dz, dy, dx) * voxel| (y, z, x
// order) and tot * (span / (len - 1)) per class segment of the shared buffer.
__device__ __forceinline__ void lengths_f32(int dz, int dy, int dx, int len, int nseg, const uint16_t *seg,
                                            const double *voxel, const float *voxelf, LegResult &out)
{
    const float vy = voxelf ? voxelf[1] : (float)voxel[1];
    const float vz = voxelf ? voxelf[0] : (float)voxel[0];
    const float vx = voxelf ? voxelf[2] : (float)voxel[2];
    const float ty = __fmul_rn((float)dy, vy);
    const float tz = __fmul_rn((float)dz, vz);
    const float tx = __fmul_rn((float)dx, vx);
    const float totf = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(ty, ty), __fmul_rn(tz, tz)), __fmul_rn(tx, tx)));
    const float scale = __fdiv_rn(totf, (float)(len - 1));
    int cur = seg[0];
    for (int j = 0; j < nseg; j++) {
        const int nxt = (j + 1 < nseg) ? (int)seg[(j + 1) * kBlock] : -1;
        const int start = cur & 0x1fff;
        const int end = (j + 1 < nseg) ? (nxt & 0x1fff) : len;
        const int cls = cur >> 13;
        const float term = scale * (float)(end - start);
        out.Lf[0] += cls == 1 ? term : 0.0f;
        out.Lf[1] += cls == 2 ? term : 0.0f;
        out.Lf[2] += cls == 3 ? term : 0.0f;
        out.Lf[3] += cls == 4 ? term : 0.0f;
        cur = nxt;
    }
}

// cal_path2_plus in FP64, bit for bit as the reference: total from the
// squares fl(fl(d * voxel)^2) summed y, z, x, then tot * fl(span / (len - 1))
// per class segment of the shared buffer, added in segment order.
__device__ __forceinline__ void lengths_f64(int dz, int dy, int dx, int len, int nseg, const uint16_t *seg,
                                            const double *voxel, const double *sq, int sq_stride, const double *qtab,
                                            LegResult &out)
{
    const double yy = sq_len(sq, sq_stride, 1, dy, voxel[1]);
    const double zz = sq_len(sq, sq_stride, 0, dz, voxel[0]);
    const double xx = sq_len(sq, sq_stride, 2, dx, voxel[2]);
    const double tot = __dsqrt_rn(__dadd_rn(__dadd_rn(yy, zz), xx));
    const int den_i = len - 1;
    const double2 dr = g_num_rcp[den_i];
    int seen = 0;
    int cur = seg[0];
    for (int j = 0; j < nseg; j++) {
        const int nxt = (j + 1 < nseg) ? (int)seg[(j + 1) * kBlock] : -1;
        const int start = cur & 0x1fff;
        const int end = (j + 1 < nseg) ? (nxt & 0x1fff) : len;
        const double q = seg_quotient(qtab, den_i, end - start, dr.x, dr.y);
        add_class(cur >> 13, __dmul_rn(tot, q), seen, out.L);
        cur = nxt;
    }
}

// State of one leg between its set-up, its march and its lengths.
struct LegState {
    March m;
    int face, lim, base;
    bool need, coop, stopped, live;
    int dlast;     // stopped at vacuum: |displacement| of the last accepted increment on the two non-step
                   // axes (a | b << 16) unless its position is near a rounding boundary, else -1
};

// cube_face and the march set-up of one leg (warp-synchronous).
template <bool kDetail>
__device__ __forceinline__ void leg_setup(const LegHead &h, const FaceRule *rules, int cz, int cy, int cx, bool valid,
                                          const Vol &v, int full, uint16_t *seg, LegResult &out, LegState &S)
{
    out.L[0] = out.L[1] = out.L[2] = out.L[3] = 0.0;
    out.Lf[0] = out.Lf[1] = out.Lf[2] = out.Lf[3] = 0.0f;
    out.len = 1; out.nseg = 1; out.status = kOk;
    if (kDetail) {
        out.first[0] = cz; out.first[1] = cy; out.first[2] = cx;
        out.last[0] = cz; out.last[1] = cy; out.last[2] = cx;
    }
    const int face = valid ? exit_face(h, cz, cy, cx, v) : 0;
    out.face = face;
    bool need = valid;
    if (valid && face == 0) {
        out.status = kErrNoFace;
        need = false;
    }
    if (need && rules[face - 1].status) {
        out.status = rules[face - 1].status;
        need = false;
    }
    March m;
    m.last_i = 0; m.nseg = 1; m.vac = 0; m.prev = 0;

    // ---- set-up: step count, cooperative eligibility, increment 0.  Only a
    // few values cross the cooperative loop; the geometry is recomputed after.
    bool coop = false, stopped = false, live = false;
    int lim = 0, base = 0;
    if (need) {
        const FaceRule &R = rules[face - 1];
        LegGeom g;
        leg_geom(R, cz, cy, cx, v, g);
        const int cc = pick3(R.count_axis, cz, cy, cx);
        const int dd = pick3(R.count_axis, v.dz, v.dy, v.dx);
        const int steps = R.count_kind == 0 ? cc + 1 : (R.count_kind == 1 ? dd - cc : dd - cc + 1);
        // the last increment of a count_kind 2 face clamps the step axis; it is
        // taken separately after the cooperative part
        const int steps_eff = R.count_kind == 2 ? steps - 1 : steps;
        coop = R.fast && !full && steps >= 1;
        lim = steps_eff;
        if (coop && steps_eff > 1) {
            // No increment of the cooperative part may clamp: its first and last
            // points (the path is monotone on every axis) lie at least one voxel
            // inside the volume.  When the volume's far wall is within reach of
            // the full leg, the cooperative part ends at the last increment that
            // stays clear of it; a leg still running there continues per lane.
            int kend = steps_eff - 1;
            for (int pass = 0; pass < 2; pass++) {
                const long long ena = g.off + (long long)kend * g.Qa;
                const long long enb = g.off + (long long)kend * g.Qb;
                const int a1 = g.ca + (int)((g.off + g.Qa) >> 32), an = g.ca + (int)(ena >> 32);
                const int b1 = g.cb + (int)((g.off + g.Qb) >> 32), bn = g.cb + (int)(enb >> 32);
                coop = min(a1, an) >= 1 && max(a1, an) <= g.ha - 1 && min(b1, bn) >= 1 && max(b1, bn) <= g.hb - 1;
                if (coop || pass == 1)
                    break;
                kend = min(kend, min(wall_increments(R.q[g.ia], g.ca, g.ha), wall_increments(R.q[g.ib], g.cb, g.hb)));
                if (kend < 1)
                    break;
            }
            lim = kend + 1;
        }
        if (coop) {
            base = g.cs * g.Ss + g.ca * g.Sa + g.cb * g.Sb;
            seg[0] = (uint16_t)(3 << 13);
            const int lab0 = __ldg(v.p + base);
            if (lab0 == 0) {
                stopped = true;
            } else {
                m.prev = lab0;
                live = lim > 1;
            }
        }
    }

    S.m = m;
    S.face = face;
    S.lim = lim;
    S.base = base;
    S.need = need;
    S.coop = coop;
    S.stopped = stopped;
    S.live = live;
    S.dlast = -1;
}

// The warp-cooperative march of the legs set up by leg_setup.
__device__ __forceinline__ void leg_coop(const FaceRule *rules, int cz, int cy, int cx, const Vol &v, uint16_t *seg,
                                         LegState &S)
{
    const int lane = threadIdx.x & 31;
    const int face = S.face, lim = S.lim, base = S.base;
    const bool coop = S.coop, live = S.live;
    bool stopped = S.stopped;
    March m = S.m;
    // ---- cooperative march, one exit-face group at a time
    unsigned pend = __ballot_sync(kAll, coop);
    while (pend) {
        const int f = __shfl_sync(kAll, face, __ffs(pend) - 1);
        const unsigned grp = __ballot_sync(kAll, coop && face == f);
        pend &= ~grp;
        const bool mine = (grp >> lane) & 1u;
        const FaceRule &G = rules[f - 1];
        const int glim = mine ? lim : 0;
        const int gmax = __reduce_max_sync(kAll, glim);
        const uint8_t *p = reinterpret_cast<const uint8_t *>(v.p) + base;
        bool on = mine && live;
        uint32_t prev4 = (uint32_t)(uint8_t)m.prev * 0x01010101u;
        for (int i0 = 1; i0 < gmax; i0 += 32) {
            if (!__any_sync(kAll, on))
                break;
            int delta;
            unsigned ambm;
            {
                // group constants, re-read from shared memory per chunk
                const int gs = G.count_axis, ga = gs == 0 ? 1 : 0, gb = gs == 2 ? 1 : 2;
                const int sz = v.dy * v.dx, sy = v.dx;
                const int ds = G.Q[gs] > 0 ? 1 : -1;
                const long long off = G.use_round ? 0x80000000ll : 0ll;
                const uint32_t Ma = ((G.exact_mask >> ga) & 1) ? 0u : kAmbiguityMargin;
                const uint32_t Mb = ((G.exact_mask >> gb) & 1) ? 0u : kAmbiguityMargin;
                const int i = i0 + lane;
                const long long ea = off + (long long)i * G.Q[ga], eb = off + (long long)i * G.Q[gb];
                const bool amb = ((uint32_t)ea + Ma < 2u * Ma) | ((uint32_t)eb + Mb < 2u * Mb);
                delta = i * ds * pick3(gs, sz, sy, 1) + (int)(ea >> 32) * pick3(ga, sz, sy, 1) +
                        (int)(eb >> 32) * pick3(gb, sz, sy, 1);
                ambm = __ballot_sync(kAll, amb);
            }
#pragma unroll 1
            for (int t = 0; t < 32; t += kMarchBatch) {
                if (!__any_sync(kAll, on))
                    break;
                const int ib = i0 + t;
                const int n = on ? glim - ib : 0;   // increments this lane still takes
                // kMarchBatch label loads in flight per lane before any is checked
                uint32_t lb[kMarchBatch];
#pragma unroll
                for (int k = 0; k < kMarchBatch; k++) {
                    const int dk = __shfl_sync(kAll, delta, t + k);
                    lb[k] = k < n ? (uint32_t)__ldg(p + dk) : 0u;
                }
                const unsigned amb_here = (ambm >> t) & ((1u << kMarchBatch) - 1u);
                if (amb_here) {
                    // the reference's FP64 expression decides, per lane (c enters its rounding)
#pragma unroll
                    for (int k = 0; k < kMarchBatch; k++)
                        if (((amb_here >> k) & 1u) && k < n)
                            lb[k] = exact_label(G, cz, cy, cx, ib + k, v);
                }
                if (n > 0) {
                    // Four increments per packed word.  prev is never 0 here, so
                    // a word equal to prev4 holds neither a stop nor a class
                    // change: the common case costs one compare per word.
                    const uint32_t w0 = lb[0] | (lb[1] << 8) | (lb[2] << 16) | (lb[3] << 24);
                    const uint32_t w1 = lb[4] | (lb[5] << 8) | (lb[6] << 16) | (lb[7] << 24);
                    if (n >= kMarchBatch && w0 == prev4 && w1 == prev4) {
                        m.last_i = ib + kMarchBatch - 1;
                    } else {
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const int nq = n - 4 * q;
                            if (stopped || nq <= 0)
                                break;
                            const uint32_t w = q == 0 ? w0 : w1;
                            const int b4 = ib + 4 * q;
                            const uint32_t valid_bytes = nq >= 4 ? 0xffffffffu : (1u << (8 * nq)) - 1u;
                            // the lowest set bit of w ^ prev4 lies in the first byte
                            // that differs: a stop (0) or a class change
                            uint32_t x = (w ^ prev4) & valid_bytes;
                            while (x) {
                                const int byte = (__ffs(x) - 1) >> 3;
                                const int lab = (int)(signed char)(w >> (8 * byte));
                                const int inc = b4 + byte;
                                if (lab == 0) {
                                    stopped = true;
                                    m.last_i = inc - 1;
                                    break;
                                }
                                if ((unsigned)lab <= 4u) {
                                    if (m.nseg < kMaxSegments)
                                        seg[m.nseg * kBlock] = (uint16_t)((lab << 13) | inc);
                                    m.nseg++;
                                }
                                m.prev = lab;
                                prev4 = (uint32_t)(uint8_t)lab * 0x01010101u;
                                const uint32_t above = byte == 3 ? 0u : (0xffffffffu << (8 * (byte + 1)));
                                x = (w ^ prev4) & valid_bytes & above;
                            }
                            if (!stopped)
                                m.last_i = b4 + min(nq, 4) - 1;
                        }
                    }
                    if (stopped || n <= kMarchBatch)
                        on = false;
                }
            }
        }
    }
    S.m = m;
    S.stopped = stopped;
    if (coop && stopped) {
        // the last point of a leg that stopped at vacuum (LegState::dlast)
        const FaceRule &R = rules[face - 1];
        const int s = R.count_axis, a = s == 0 ? 1 : 0, b = s == 2 ? 1 : 2;
        const long long off = R.use_round ? 0x80000000ll : 0ll;
        const uint32_t Ma = ((R.exact_mask >> a) & 1) ? 0u : kAmbiguityMargin;
        const uint32_t Mb = ((R.exact_mask >> b) & 1) ? 0u : kAmbiguityMargin;
        const long long ea = off + (long long)m.last_i * R.Q[a], eb = off + (long long)m.last_i * R.Q[b];
        const bool amb = ((uint32_t)ea + Ma < 2u * Ma) | ((uint32_t)eb + Mb < 2u * Mb);
        S.dlast = amb ? -1 : (abs((int)(ea >> 32)) | abs((int)(eb >> 32)) << 16);
    }
}

// After the march: the per-lane remainder of the path and cal_path2_plus.
template <bool kDetail, bool kF32>
__device__ __forceinline__ void leg_finish(const FaceRule *rules, int cz, int cy, int cx, const Vol &v, int full,
                                           const double *voxel, const double *sq, int sq_stride, const double *qtab,
                                           uint16_t *seg, LegState &S, LegResult &out, const float *voxelf)
{
    const int face = S.face, lim = S.lim;
    const bool need = S.need, coop = S.coop, stopped = S.stopped;
    March m = S.m;
    Sink sk;
    sk.seg = seg;
    if (!need)
        return;

    if (!kDetail && coop && stopped && S.dlast >= 0 && m.nseg <= kMaxSegments) {
        // a leg that stopped at vacuum: the last point is known
        // (step axis: last_i increments; the others: dlast), so the lengths
        // need neither the geometry nor the point
        const int len = m.last_i + 1;
        out.len = len;
        out.nseg = m.nseg;
        if (len == 1)
            return;
        const int s = rules[face - 1].count_axis;
        const int da = S.dlast & 0xffff, db = S.dlast >> 16;
        const int d0 = s == 0 ? m.last_i : da;
        const int d1 = s == 1 ? m.last_i : (s == 0 ? da : db);
        const int d2 = s == 2 ? m.last_i : db;
        if (kF32)
            lengths_f32(d0, d1, d2, len, m.nseg, seg, voxel, voxelf, out);
        else
            lengths_f64(d0, d1, d2, len, m.nseg, seg, voxel, sq, sq_stride, qtab, out);
        return;
    }

    // ---- after the march: geometry again, the per-lane paths, lengths
    const FaceRule &R = rules[face - 1];
    LegGeom g;
    leg_geom(R, cz, cy, cx, v, g);
    const int cc = pick3(R.count_axis, cz, cy, cx);
    const int dd = pick3(R.count_axis, v.dz, v.dy, v.dx);
    const int steps = R.count_kind == 0 ? cc + 1 : (R.count_kind == 1 ? dd - cc : dd - cc + 1);
    if (coop && !stopped && lim < (R.count_kind == 2 ? steps - 1 : steps)) {
        // the cooperative part ended at the wall limit: the rest per lane
        March mc = m;
        Sink sc;
        sc.seg = seg;
        march_lane<0>(R, cz, cy, cx, steps, v, full, mc, sc, lim);
        m = mc;
    } else if (coop && !stopped && R.count_kind == 2) {
        // the clamped last increment of a count_kind 2 face
        int pz, py, px;
        const int inc = steps - 1;
        point_at(R, g, inc, cz, cy, cx, v, pz, py, px);
        const int lab = __ldg(v.p + (pz * v.dy * v.dx + py * v.dx + px));
        if (inc >= 1)
            visit<0>(m, sk, inc, lab, 0, R.vac_limit);
    }
    if (!coop) {
        // separate objects for the out-of-line call (see march_lane)
        March mc = m;
        Sink sc;
        sc.seg = seg;
        march_lane<0>(R, cz, cy, cx, steps, v, full, mc, sc);
        m = mc;
    }

    // ---- cal_path2_plus
    const int len = m.last_i + 1;
    out.len = len;
    out.nseg = m.nseg;
    if (len == 1 && !kDetail)
        return;
    int fz = cz, fy = cy, fx = cx;
    if (!R.fast)
        point_at(R, g, 0, cz, cy, cx, v, fz, fy, fx);
    int lz, ly, lx;
    point_at(R, g, m.last_i, cz, cy, cx, v, lz, ly, lx);
    if (kDetail) {
        out.first[0] = fz; out.first[1] = fy; out.first[2] = fx;
        out.last[0] = lz; out.last[1] = ly; out.last[2] = lx;
        if (len == 1)
            return;
    }
    if (kF32 && m.nseg <= kMaxSegments) {
        lengths_f32(abs(lz - fz), abs(ly - fy), abs(lx - fx), len, m.nseg, seg, voxel, voxelf, out);
        return;
    }
    if (kF32) {
        const L4 r = lengths_second_pass(R, cz, cy, cx, steps, v, full, len, fz, fy, fx, lz, ly, lx, voxel, sq,
                                         sq_stride, qtab, seg);
        for (int k = 0; k < 4; k++)
            out.Lf[k] = (float)r.v[k];
        return;
    }
    if (m.nseg <= kMaxSegments) {
        lengths_f64(abs(lz - fz), abs(ly - fy), abs(lx - fx), len, m.nseg, seg, voxel, sq, sq_stride, qtab, out);
    } else {
        // total from the first and last path points, y then z then x
        const double yy = sq_len(sq, sq_stride, 1, abs(ly - fy), voxel[1]);
        const double zz = sq_len(sq, sq_stride, 0, abs(lz - fz), voxel[0]);
        const double xx = sq_len(sq, sq_stride, 2, abs(lx - fx), voxel[2]);
        const double tot = __dsqrt_rn(__dadd_rn(__dadd_rn(yy, zz), xx));
        const int den_i = len - 1;
        const double2 dr = g_num_rcp[den_i];
        // more class changes than the shared buffer holds: march again and
        // accumulate as segments close (same terms, same order)
        March m2;
        Sink s2;
        s2.seg = seg;
        s2.qtab = qtab;
        s2.tot = tot; s2.den = dr.x; s2.rcp = dr.y; s2.den_i = den_i;
        s2.L[0] = s2.L[1] = s2.L[2] = s2.L[3] = 0.0;
        s2.open_cls = 3; s2.open_pos = 0; s2.seen = 0;
        march_lane<1>(R, cz, cy, cx, steps, v, full, m2, s2);
        const double q = seg_quotient(qtab, den_i, len - s2.open_pos, dr.x, dr.y);
        add_class(s2.open_cls, __dmul_rn(tot, q), s2.seen, s2.L);
        for (int k = 0; k < 4; k++) {
            out.L[k] = s2.L[k];
            out.Lf[k] = (float)s2.L[k];
        }
    }
}

// cube_face + cal_coord + cal_path2_plus for one leg.  Called by all 32 lanes
// of a warp together (warp-synchronous); `valid` marks lanes that hold a voxel.
//
// Warp-cooperative march: lanes whose rays leave through the same face share
// that face's step rule, and their 32.32 positions differ only in the integer
// part (c * 2^32).  So the displacement of increment i -- and whether its
// fraction is near a rounding boundary -- is the same for every lane of the
// group: lane j computes it for increment i0 + j, the warp broadcasts it with
// shuffles, and each lane only adds it to its own start address, loads the
// label and checks it.  A lane joins the group only if no clamp can occur on
// its increments (both end points at least one voxel inside the volume) and
// the face has fixed-point ratios; other lanes, and full_iteration, use the
// per-lane march.
// kF32: the per-class lengths in FP32 (for A_h, which needs 1e-6; the march
// itself, and hence the visited voxels, segments and len_path_2, is the same);
// otherwise FP64 in the reference's order (bit-exact lengths).
template <bool kDetail, bool kF32 = false>
__device__ __forceinline__ void trace_leg(const LegHead &h, const FaceRule *rules, int cz, int cy, int cx,
                                          bool valid, const Vol &v, int full, const double *voxel,
                                          const double *sq, int sq_stride, const double *qtab, uint16_t *seg,
                                          LegResult &out, const float *voxelf = nullptr)
{
    LegState S;
    leg_setup<kDetail>(h, rules, cz, cy, cx, valid, v, full, seg, out, S);
    leg_coop(rules, cz, cy, cx, v, seg, S);
    leg_finish<kDetail, kF32>(rules, cz, cy, cx, v, full, voxel, sq, sq_stride, qtab, seg, S, out, voxelf);
}

// ---- field march ----------------------------------------------------------
//
// The A_h kernel's march on the packed fields: one lane walks one leg as a
// chain of dependent byte loads (about 12, 16 for the slowest lane of a warp),
// each an L2 access of some 450 cycles, so a warp alone needs 12,500 cycles a
// leg and what counts is how many warps an SM holds and how many instructions
// and L1 misses a step costs.  Hence:
//  * what a step needs is prepared once per work item (32 voxels x tile / 32 x
//    2 legs share it) in shared memory, one rule per leg and exit axis; a
//    leg's own set-up is the exit face and a few shared loads;
//  * a leg whose non-vacuum labels keep room from the walls ahead of it needs
//    no step count and no wall limit: it meets vacuum first;
//  * the inner loop holds no call (what lives across one is kept in local
//    memory: 92 local loads a warp and leg then), what a march need not hold
//    lies in shared memory at constant addresses (FieldShared; 10.2 -> 2.7
//    local loads), and the kernel fits 48 registers, five CTAs an SM (six, at
//    40 registers: 10 % slower, four 7 %);
//  * everything rare (close exit-face calls, ratios beyond fixed point,
//    full_iteration, legs that reach the wall limit, more than kMaxSegments
//    class changes) is out of line in leg_slow, which reads the full rule
//    from global memory.
// 512x512x400, 13,266 voxels, 20,000 reflections: 30.0 -> 18.6 ms (1,430 ->
// 852 warp instructions per 32 legs; L1 misses at 69 %, L2 at 60 % of their
// peak rates, issue slots at 53 %).  1024x1024x800, every crystal voxel (6.8 million),
// 32 reflections: 23.0 -> 17.7 ms on one box, 24.3 -> 19.9 on another (10 %
// more with those 10.2 local loads).

// One leg's rule for one exit axis.  q: the 32.32 ratios of the two other
// axes a and b (lo, hi words).  off: their initial low words -- the rounding
// offset plus kFieldMargin, so that a fraction near a rounding boundary reads
// below twice the margin (adding it changes the integer
// part only there, where the exact expression is used).  A whole-numbered
// ratio gets 2^31: its fraction stays one half, which is never ambiguous and
// rounds to the exact integer in both modes.  So does a ratio from 0 to 2^-33
// (Q = 0; a map's directions along an axis): i * q is below 2^-19, so c + i * q
// rounds to c either way.
struct alignas(16) HotRule {
    uint32_t qa_lo, qa_hi, qb_lo, qb_hi;
    uint32_t off_a, off_b;
    int dS, Sa;              // linear fields: signed stride of the step axis, stride of a
    int Sb;
    int rq;                  // skip multiplier (FaceRule::skip_rq)
    uint32_t flags;
    int face;
    const uint8_t *fld;      // the field of the leg's octant
    int ds;                  // +1 / -1 on the step axis
    int pad;
};
static_assert(sizeof(HotRule) == 64, "HotRule layout");
constexpr uint32_t kHotSimple = 1u;   // fixed point, no error status, no full_iteration
constexpr uint32_t kHotFree = 2u;     // a leg stops at vacuum before any increment can clamp at a wall

struct alignas(16) WarpTab {
    HotRule rule[2][3];      // [leg][exit axis]
    float inv[2][3];         // 1 / |e_a|; +inf for a zero component
    float sgn[2][3];         // exit distance on axis a is n_a inv_a with n_a = org_a + sgn_a c_a (exact)
    float org[2][3];
    uint32_t exact_face[2];  // the FP64 quotients decide for every lane
    float voxel[3];
    float mu[4];
    int dy, dx, is_exp, count_steps;
    const ReflTable *refl;
    const SampleDesc *desc;
    const short4 *coords;    // the item's voxels
    int n;
};

// Half-width of the ambiguous zone around a rounding boundary, in 2^-32
// units, for increments of a field march: i * Q differs from i * q * 2^32 by
// at most i / 2 <= 4096 units (Q is rounded, kMaxDim bounds i), and the
// reference's two FP64 roundings of values inside the volume (below 2^14) by
// less than one.
constexpr uint32_t kFieldMargin = 4096u + 16u;

// Fills a warp's table for reflection table T: lanes 0..5 a rule each (leg,
// axis), lanes 8..13 the exit-face operands, lanes 16..23 the sample's constants.
__device__ __forceinline__ void fill_warp_tab(WarpTab &w, const ReflTable *__restrict__ T, const SampleDesc &D,
                                              int tile, int lane)
{
    const int part = lane >> 3, k = lane & 7;
    if (part < 2 && k < 6) {
        const int leg = k / 3, a = k - 3 * leg;
        const uint32_t sb = __ldg(&T->head[leg].sign_bits);
        const bool pos = (sb >> a) & 1u, zero = !((sb >> a) & 9u);
        if (part == 1) {
            const int dim = a == 0 ? D.dim[0] : (a == 1 ? D.dim[1] : D.dim[2]);
            w.inv[leg][a] = __ldg(&T->head[leg].inv[a]);
            w.sgn[leg][a] = zero ? 0.0f : (pos ? -1.0f : 1.0f);
            w.org[leg][a] = zero ? 1.0f : (pos ? (float)dim : 0.0f);
            if (a == 0)
                w.exact_face[leg] = sb & 64u;
            return;
        }
        const int face = a == 2 ? (pos ? 1 : 6) : (a == 1 ? (pos ? 5 : 4) : (pos ? 3 : 2));
        const FaceRule &R = T->rule[leg][face - 1];
        HotRule h;
        const int ia = a == 0 ? 1 : 0, ib = a == 2 ? 1 : 2;
        const long long Qa = R.Q[ia], Qb = R.Q[ib];
        h.qa_lo = (uint32_t)Qa;
        h.qa_hi = (uint32_t)(Qa >> 32);
        h.qb_lo = (uint32_t)Qb;
        h.qb_hi = (uint32_t)(Qb >> 32);
        const uint32_t off = (R.use_round ? 0x80000000u : 0u) + kFieldMargin;
        h.off_a = (R.exact_mask >> ia) & 1 || (Qa == 0 && R.q[ia] >= 0.0) ? 0x80000000u : off;
        h.off_b = (R.exact_mask >> ib) & 1 || (Qb == 0 && R.q[ib] >= 0.0) ? 0x80000000u : off;
        h.ds = R.Q[a] > 0 ? 1 : -1;
        const int sz = D.dim[1] * D.dim[2], sy = D.dim[2];
        h.dS = h.ds * pick3(a, sz, sy, 1);
        h.Sa = pick3(ia, sz, sy, 1);
        h.Sb = pick3(ib, sz, sy, 1);
        h.rq = (int)R.skip_rq;   // at most 2^22, times 31
        h.pad = 0;
        h.fld = D.field + R.octant * D.field_stride;
        h.face = face;
        uint32_t f = 0u;
        if (R.fast && !R.status && !D.full_iteration && !zero) {
            f |= kHotSimple;
            // see free_leg_room; such a leg also stops before its face's last increment
            if (D.walls) {
                const int need = free_leg_room(max(Qa < 0 ? -Qa : Qa, Qb < 0 ? -Qb : Qb));
                bool free_leg = true;
#pragma unroll
                for (int x = 0; x < 3; x++)
                    free_leg = free_leg && __ldg(D.walls + wall_ahead(R.octant, x)) >= need;
                if (free_leg)
                    f |= kHotFree;
            }
        }
        h.flags = f;
        w.rule[leg][a] = h;
    } else if (part == 2) {
        if (k < 3)
            w.voxel[k] = D.voxelf[k];
        else if (k < 7)
            w.mu[k - 3] = D.muf[k - 3];
        else {
            w.dy = D.dim[1];
            w.dx = D.dim[2];
            w.is_exp = D.is_exp;
            w.count_steps = D.steps != nullptr;
            w.refl = T;
            w.desc = &D;
            w.coords = D.coords + (long long)tile * D.tile;
            w.n = min(D.tile, D.n_vox - tile * D.tile);
        }
    }
}

// integer part (the return value) and fraction of off + i * Q
__device__ __forceinline__ int fixed_at(int i, uint32_t q_lo, uint32_t q_hi, unsigned long long off, uint32_t &frac)
{
    const unsigned long long p = (unsigned long long)(uint32_t)i * q_lo + off;
    frac = (uint32_t)p;
    return (int)((uint32_t)(p >> 32) + (uint32_t)i * q_hi);
}

// The increment examined after i, whose field byte holds the distance d (>= 1)
// above its label: the ones the field proves to keep i's label, min(d - 1, floor((d - 2) / qmax))
// and never a negative number of them, are passed over.
__device__ __forceinline__ int next_increment(int i, uint32_t byte, int rq)
{
    const int d = (int)(byte >> 3);
    return i + max(min((((d - 2) * rq) >> 16) + 1, d), 1);
}

// Byte of increment i of a field whose displacement on the two non-step axes
// is (da, db): linear fields from the leg's start byte, bricked ones from the
// absolute coordinates.
template <bool kBrick>
__device__ __forceinline__ uint32_t field_byte(const uint8_t *start, const HotRule &R, const SampleDesc *D, int axis,
                                               int cz, int cy, int cx, int i, int da, int db, int dS, int Sa, int Sb)
{
    if (!kBrick)
        return __ldg(start + (i * dS + da * Sa + db * Sb));
    const Vol v{nullptr, D->dim[0], D->dim[1], D->dim[2], nullptr, 0, D->brick_sy, D->brick_sz};
    const int s = i * R.ds;
    const int pz = cz + (axis == 0 ? s : da);
    const int py = cy + (axis == 1 ? s : (axis == 0 ? da : db));
    const int px = cx + (axis == 2 ? s : db);
    return __ldg(R.fld + brick_offset(pz, py, px, v));
}

// Class changes go to rows 1.. of the lane's list in shared memory; a list
// that would be longer than kMaxSegments parks in the row after the last.
constexpr int kSegRows = kMaxSegments + 1;

// Shared memory of the field kernels.  It is dynamic, so that every function
// reaches it by a constant address, and a lane's place in it comes from its
// thread number, read anew where it is needed: the march's registers are what
// limits the warps an SM holds, and a pointer kept across a leg ended up in
// local memory, whose loads miss L1 among the field's.
struct FieldShared {
    WarpTab tabs[kWarps];
    uint16_t seg[kSegRows * kBlock];
    float4 incident[kBlock];     // the incident leg's lengths while the diffracted leg marches
    float2 total[kBlock];        // the lanes' sums (FloatSum)
    float total_low[kBlock];
    unsigned steps[kBlock];
    FloatPair consts[7];         // map kernel: squared voxel edges (z, y, x), mu
};
extern __shared__ __align__(16) uint8_t field_smem[];

__device__ __forceinline__ FieldShared &field_shared() { return *reinterpret_cast<FieldShared *>(field_smem); }

__device__ __forceinline__ int thread_now()
{
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

__device__ __forceinline__ WarpTab &warp_tab() { return field_shared().tabs[thread_now() >> 5]; }
__device__ __forceinline__ uint16_t *seg_list() { return field_shared().seg + thread_now(); }

struct SlowLeg {
    float4 L;
    int len;
};

// What leg_slow continues from: 0 the start; 1 the wall limit (increments
// 0..lim-1 accepted); 2 the stop at increment i (only the lengths are left).
enum SlowFrom { kFromStart = 0, kFromLimit = 1, kFromStop = 2 };

// The rest of a leg that the field march does not finish by itself: FP32
// lengths (out.Lf), or FP64 ones in the reference's order (out.L).
template <bool kF32>
__device__ __forceinline__ void leg_rest(int leg, int vi, int from, int axis, int i, int nseg, int prev, int lim,
                                         LegResult &out)
{
    const WarpTab &W = warp_tab();
    uint16_t *seg = seg_list();
    const short4 cv = __ldg(W.coords + vi);
    const SampleDesc &D = *W.desc;
    const ReflTable *T = W.refl;
    const Vol v{D.vol, D.dim[0], D.dim[1], D.dim[2]};
    for (int k = 0; k < 4; k++) {
        out.L[k] = 0.0;
        out.Lf[k] = 0.0f;
    }
    out.len = 1;
    out.status = kOk;
    const FaceRule *rules = T->rule[leg];
    const int face = from == kFromStart ? exit_face(T->head[leg], cv.x, cv.y, cv.z, v) : W.rule[leg][axis].face;
    if (face == 0)
        out.status = kErrNoFace;
    else if (rules[face - 1].status)
        out.status = rules[face - 1].status;
    if (out.status)
        return;
    LegState S;
    S.m.last_i = (from == kFromStop ? i : lim) - 1;
    S.m.nseg = nseg;
    S.m.prev = prev;
    S.m.vac = 0;
    S.face = face;
    S.lim = lim;
    S.base = 0;
    S.need = true;
    S.coop = from != kFromStart;
    S.stopped = from == kFromStop;
    S.live = false;
    S.dlast = -1;
    leg_finish<false, kF32>(rules, cv.x, cv.y, cv.z, v, D.full_iteration, D.voxel, D.sq, D.sq_stride, D.qtab, seg, S,
                            out, D.voxelf);
}

__device__ __noinline__ SlowLeg leg_slow(int leg, int vi, int from, int axis, int i, int nseg, int prev, int lim)
{
    LegResult out;
    leg_rest<true>(leg, vi, from, axis, i, nseg, prev, lim, out);
    if (out.status)
        atomicOr(warp_tab().desc->status, 1 << out.status);
    SlowLeg r;
    r.L = make_float4(out.Lf[0], out.Lf[1], out.Lf[2], out.Lf[3]);
    r.len = out.len;
    return r;
}

// Exit axis of a leg whose estimated distances do not decide it (the voxel
// lies as far from two walls, or on one), by the reference's quotients; -1
// when its rule is not the one the march keeps for the axis (a zero distance
// to the wall behind).  The march itself is as good for such a leg as for any:
// left to leg_slow, 4 in 10,000 legs of a regular grid of directions -- ties
// of whole-degree angles -- took 100 us each one after the other and
// 4,096 directions 2.2 ms, most of it one warp's.
__device__ __noinline__ int exact_axis(int leg, int vi)
{
    const WarpTab &W = warp_tab();
    const short4 cv = __ldg(W.coords + vi);
    const Vol v{nullptr, W.desc->dim[0], W.dy, W.dx};
    const int face = exit_face(W.refl->head[leg], cv.x, cv.y, cv.z, v);
    if (face == 0)
        return -1;
    const int axis = face == 1 || face == 6 ? 2 : (face == 4 || face == 5 ? 1 : 0);
    return W.rule[leg][axis].face == face ? axis : -1;
}

// Displacement of increment i on the two non-step axes from the reference's
// FP64 expression (a position near a rounding boundary, inside the volume).
__device__ __forceinline__ void exact_displacement(int leg, int axis, int vi, int i, int &da, int &db)
{
    const WarpTab &W = warp_tab();
    const short4 cv = __ldg(W.coords + vi);
    const FaceRule &F = W.refl->rule[leg][W.rule[leg][axis].face - 1];
    const int a = axis == 0 ? 1 : 0, b = axis == 2 ? 1 : 2;
    const int ca = axis == 0 ? cv.y : cv.x, cb = axis == 2 ? cv.y : cv.z;
    const double va = __dadd_rn((double)ca, __dmul_rn((double)i, F.q[a]));
    const double vb = __dadd_rn((double)cb, __dmul_rn((double)i, F.q[b]));
    const bool rnd = F.use_round;
    da = (int)(rnd ? round(va) : floor(va)) - ca;
    db = (int)(rnd ? round(vb) : floor(vb)) - cb;
}

// The number of leading increments of a leg that cannot clamp at a wall (the
// last one excluded where its face clamps it), or 0 when the leg is left to
// the per-lane march: the path is monotone on every axis, so its first and
// last points decide; where the far wall is within reach of the whole leg,
// the part ends at the last increment that stays clear of it.
__device__ __noinline__ int leg_limit(const FaceRule *R, int cz, int cy, int cx, int dz, int dy, int dx)
{
    Vol v{nullptr, dz, dy, dx};
    LegGeom g;
    leg_geom(*R, cz, cy, cx, v, g);
    const int cc = pick3(R->count_axis, cz, cy, cx);
    const int dd = pick3(R->count_axis, dz, dy, dx);
    const int steps = R->count_kind == 0 ? cc + 1 : (R->count_kind == 1 ? dd - cc : dd - cc + 1);
    const int steps_eff = R->count_kind == 2 ? steps - 1 : steps;
    if (steps_eff <= 1)
        return 0;
    int kend = steps_eff - 1;
    for (int pass = 0; pass < 2; pass++) {
        const long long ena = g.off + (long long)kend * g.Qa;
        const long long enb = g.off + (long long)kend * g.Qb;
        const int a1 = g.ca + (int)((g.off + g.Qa) >> 32), an = g.ca + (int)(ena >> 32);
        const int b1 = g.cb + (int)((g.off + g.Qb) >> 32), bn = g.cb + (int)(enb >> 32);
        if (min(a1, an) >= 1 && max(a1, an) <= g.ha - 1 && min(b1, bn) >= 1 && max(b1, bn) <= g.hb - 1)
            return kend + 1;
        kend = min(kend, min(wall_increments(R->q[g.ia], g.ca, g.ha), wall_increments(R->q[g.ib], g.cb, g.hb)));
        if (kend < 1)
            break;
    }
    return 0;
}

// Exit face and march of one leg of one voxel (not warp-synchronous).
// Returns `none()` for a leg without length (it starts in vacuum or stops at
// increment 1), `done(i, nseg, d0, d1, d2)` for one that stopped at vacuum at
// increment i with its class changes in the list and its last point's
// |displacement| (z, y, x), and `slow(from, axis, i, nseg, prev, lim)` for one
// that is left to the slow path.
//
// The inner loop is kept to one load, one exit branch and predicated
// bookkeeping (about 30 instructions) and holds no call: what lives across
// one would be kept in local memory.  A position near a rounding boundary is
// off by at most one voxel in the inner loop, still inside the volume (free
// legs keep a voxel of room, the others their wall limit); the outer loop
// takes that increment with the exact position.
// kTies: a leg whose exit face the estimates leave open marches too, on the
// face of exact_axis.  For the maps' regular directions; measured directions
// have a handful of such legs in a million and the call costs the A_h kernel
// 1 to 2 %.
template <bool kBrick, bool kTies, class None, class Done, class Slow>
__device__ __forceinline__ auto field_march(int leg, int vi, None none, Done done, Slow slow)
{
    const WarpTab &W = warp_tab();
    uint16_t *seg = seg_list();
    // the coordinates are loaded per leg (and again where they are rarely
    // needed) rather than kept across the march
    const short4 cv = __ldg(W.coords + vi);
    const int cz = cv.x, cy = cv.y, cx = cv.z;
    // ---- exit face: the smallest of the three distances n_a / |e_a| (n_a
    // exact, the estimates within 2^-22), when the next one is clearly larger
    // and the voxel is not on a min plane (a zero distance wins there)
    const float tx = __fmaf_rn(W.sgn[leg][2], (float)cx, W.org[leg][2]) * W.inv[leg][2];
    const float ty = __fmaf_rn(W.sgn[leg][1], (float)cy, W.org[leg][1]) * W.inv[leg][1];
    const float tz = __fmaf_rn(W.sgn[leg][0], (float)cz, W.org[leg][0]) * W.inv[leg][0];
    const float lo = fminf(tx, ty);
    const float t1 = fminf(lo, tz), t2 = fmaxf(lo, fminf(fmaxf(tx, ty), tz));
    int axis = tx == t1 ? 2 : (ty == t1 ? 1 : 0);
    bool go = t2 > t1 * (1.0f + 0x1p-20f) && !W.exact_face[leg] && min(cx, min(cy, cz)) > 0;
    if (kTies && !go) {
        axis = exact_axis(leg, vi);
        go = axis >= 0;
        axis = max(axis, 0);
    }
    const HotRule &R = W.rule[leg][axis];
    const uint32_t flags = R.flags;
    int from = kFromStart, i = 0, nseg = 1, prev = 0, lim = 0x7fffffff;
    go = go && (flags & kHotSimple);
    if (go && !(flags & kHotFree)) {
        lim = leg_limit(&W.refl->rule[leg][R.face - 1], cz, cy, cx, W.desc->dim[0], W.dy, W.dx);
        go = lim > 1;
    }
    if (go) {
        const uint8_t *start =
            R.fld + (kBrick ? brick_offset(cz, cy, cx, Vol{nullptr, W.desc->dim[0], W.dy, W.dx, nullptr, 0,
                                                           W.desc->brick_sy, W.desc->brick_sz})
                            : (cz * W.dy + cy) * W.dx + cx);
        uint32_t b = __ldg(start);
        if ((b & 7u) == 0u)
            return none();   // starts in vacuum
        const uint32_t qa_lo = R.qa_lo, qa_hi = R.qa_hi, qb_lo = R.qb_lo, qb_hi = R.qb_hi;
        const unsigned long long off_a = R.off_a, off_b = R.off_b;
        const int dS = R.dS, Sa = R.Sa, Sb = R.Sb, rq = R.rq;
        prev = (int)(b & 7u);
        i = next_increment(0, b, rq);
        auto take = [&](int lab) {   // class-change bookkeeping and the step
            if (lab != prev && lab <= 4) {
                seg[min(nseg, kMaxSegments) * kBlock] = (uint16_t)((lab << 13) | i);
                nseg++;
            }
            prev = lab;
            i = next_increment(i, b, rq);
        };
        from = kFromLimit;
        while (i < lim) {
            bool near;
            for (;;) {
                uint32_t fa, fb;
                const int da = fixed_at(i, qa_lo, qa_hi, off_a, fa);
                const int db = fixed_at(i, qb_lo, qb_hi, off_b, fb);
                b = field_byte<kBrick>(start, R, W.desc, axis, cz, cy, cx, i, da, db, dS, Sa, Sb);
                near = min(fa, fb) < 2u * kFieldMargin;
                const int lab = (int)(b & 7u);
                if (near | (lab == 0))
                    break;
                take(lab);
                if (i >= lim)
                    break;
            }
            if (i >= lim)
                break;
            if (near) {
                int da, db;
                exact_displacement(leg, axis, vi, i, da, db);
                b = field_byte<kBrick>(start, R, W.desc, axis, cz, cy, cx, i, da, db, dS, Sa, Sb);
                if (b & 7u) {
                    take((int)(b & 7u));
                    continue;
                }
            }
            from = kFromStop;
            break;
        }
        if (from == kFromStop && i == 1)
            return none();
        if (from == kFromStop && nseg <= kMaxSegments) {
            // the last point's displacement: last_i on the step axis
            const int last_i = i - 1;
            uint32_t fa, fb;
            int da = fixed_at(last_i, qa_lo, qa_hi, off_a, fa);
            int db = fixed_at(last_i, qb_lo, qb_hi, off_b, fb);
            if (min(fa, fb) < 2u * kFieldMargin)
                exact_displacement(leg, axis, vi, last_i, da, db);
            const int d0 = axis == 0 ? last_i : abs(da);
            const int d1 = axis == 1 ? last_i : (axis == 0 ? abs(da) : abs(db));
            const int d2 = axis == 2 ? last_i : abs(db);
            seg[0] = (uint16_t)(3 << 13);
            return done(i, nseg, d0, d1, d2);
        }
    }
    seg[0] = (uint16_t)(3 << 13);
    return slow(from, axis, i, nseg, prev, lim);
}

// One leg of voxel vi of the item: FP32 lengths (liquor, loop, crystal, bubble).
template <bool kBrick>
__device__ __forceinline__ float4 field_leg(int leg, int vi, int &len)
{
    len = 1;
    return field_march<kBrick, false>(
        leg, vi, [] { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); },
        [&](int i, int nseg, int d0, int d1, int d2) {
            len = i;
            LegResult out;
            out.Lf[0] = out.Lf[1] = out.Lf[2] = out.Lf[3] = 0.0f;
            lengths_f32(d0, d1, d2, i, nseg, seg_list(), nullptr, warp_tab().voxel, out);
            return make_float4(out.Lf[0], out.Lf[1], out.Lf[2], out.Lf[3]);
        },
        [&](int from, int axis, int i, int nseg, int prev, int lim) {
            const SlowLeg r = leg_slow(leg, vi, from, axis, i, nseg, prev, lim);
            len = r.len;
            return r.L;
        });
}

// A map value (cal_rate with a zero incident leg) of a leg
// in the reference's FP64 operations: legs the march leaves, and values too
// close to a rounding boundary of float.
__device__ __noinline__ float map_slow(int vi, int from, int axis, int i, int nseg, int prev, int lim, int d0, int d1,
                                       int d2)
{
    const SampleDesc &D = *warp_tab().desc;
    LegResult out;
    if (d0 >= 0) {   // marched to its stop: the lengths alone
        out.L[0] = out.L[1] = out.L[2] = out.L[3] = 0.0;
        out.status = kOk;
        lengths_f64(d0, d1, d2, i, nseg, seg_list(), D.voxel, D.sq, D.sq_stride, D.qtab, out);
    } else {
        leg_rest<false>(1, vi, from, axis, i, nseg, prev, lim, out);
    }
    if (out.status) {
        atomicOr(D.status, 1 << out.status);
        return __int_as_float(0x7fffffff);
    }
    const double t0 = __dmul_rn(D.mu[0], out.L[0]);
    const double t1 = __dmul_rn(D.mu[1], out.L[1]);
    const double t2 = __dmul_rn(D.mu[2], out.L[2]);
    const double t3 = __dmul_rn(D.mu[3], out.L[3]);
    const double ex = __dadd_rn(__dadd_rn(__dadd_rn(t0, t1), t2), t3);
    return (float)(D.is_exp ? exp(-ex) : ex);
}

__device__ __forceinline__ int find_sample(const SampleDesc *d, int n, long long item)
{
    int s = 0;
    while (s + 1 < n && item >= d[s + 1].work_begin)
        s++;
    return s;
}

// The end of an absorption work item: the warp's sum, the item's partial sum
// and, for the last tile of the reflection to arrive, the combination of the
// partials into A_h.  The sums stay three floats (FloatSum) to the end, exact as
// far as those go, so A_h has the same bits however the voxels are cut into
// items: for a full set of reflections, a part of it and in a batch.  (A launch
// without room for the third floats folds them in.)
__device__ __forceinline__ void finish_warp_item(FloatSum a, const SampleDesc &D, long long r, int t, int lane)
{
#pragma unroll 1   // inlined everywhere: unrolled, it costs the bisection 0.8 % in instruction fetches
    for (int o = 16; o > 0; o >>= 1)
        sum_merge(a, __shfl_down_sync(kAll, a.s, o), __shfl_down_sync(kAll, a.c, o), __shfl_down_sync(kAll, a.d, o));
    int last = 0;
    if (lane == 0) {
        const long long at = r * D.tiles + t;
        if (D.partial_low)
            D.partial_low[at] = a.d;
        else
            a.c += a.d;
        D.partial[at] = make_float2(a.s, a.c);
        __threadfence();
        last = atomicAdd(D.arrive + r, 1u) == (unsigned)(D.tiles - 1);
    }
    if (__shfl_sync(kAll, last, 0)) {
        __threadfence();
        const float2 *sc = D.partial + r * D.tiles;
        const float *low = D.partial_low ? D.partial_low + r * D.tiles : nullptr;
        a = {0.0f, 0.0f, 0.0f};
        // eight entries' loads together: a few reflections of many items wait for
        // this loop (6 of 64,000 voxels: 53 us a launch, 69 one after the other)
        constexpr int kAhead = 8;
        for (int k0 = lane; k0 < D.tiles; k0 += 32 * kAhead) {
            float2 p[kAhead];
            float d[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; j++) {
                const int k = k0 + 32 * j;
                const bool in = k < D.tiles;
                p[j] = in ? __ldcg(sc + k) : make_float2(0.0f, 0.0f);
                d[j] = in && low ? __ldcg(low + k) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < kAhead; j++)
                sum_merge(a, p[j].x, p[j].y, d[j]);
        }
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1)
            sum_merge(a, __shfl_down_sync(kAll, a.s, o), __shfl_down_sync(kAll, a.c, o), __shfl_down_sync(kAll, a.d, o));
        if (lane == 0) {
            double h, l;
            two_sum((double)a.s, (double)a.c, h, l);
            D.out[r] = (h + (l + (double)a.d)) / (double)D.n_vox;
            D.arrive[r] = 0u;   // ready for the next launch
        }
    }
}

// The A_h kernel with the warp-cooperative march.
template <int kMinBlocks>
__global__ void __launch_bounds__(kBlock, kMinBlocks) absorption_kernel(const SampleDesc *__restrict__ descs,
                                                                        int n_desc, long long total_items,
                                                                        unsigned long long *__restrict__ work_counter)
{
    __shared__ ReflTable tabs[kWarps];   // one per warp: items are taken per warp
    __shared__ uint16_t seg[kMaxSegments * kBlock];
    __shared__ float lsum[4][kBlock];

    if (!block_shape_ok(n_desc > 0 ? descs[0].status : nullptr))
        return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    ReflTable &tab = tabs[warp];
    for (;;) {
        unsigned long long it = 0;
        if (lane == 0)
            it = atomicAdd(work_counter, 1ull);
        const long long item = (long long)__shfl_sync(kAll, it, 0);
        if (item >= total_items)
            break;
        const int si = find_sample(descs, n_desc, item);
        const SampleDesc &D = descs[si];
        const long long local = item - D.work_begin;
        const long long k = local / D.tiles;
        const long long r = D.order ? (long long)__ldg(D.order + k) : k;
        const int t = (int)(local - k * D.tiles);
        __syncwarp();   // the previous item's reads of the table are done
        {
            const int4 *src = reinterpret_cast<const int4 *>(D.refl + r);
            int4 *dst = reinterpret_cast<int4 *>(&tab);
            for (int k = lane; k < (int)(sizeof(ReflTable) / 16); k += 32)
                dst[k] = __ldg(src + k);
        }
        __syncwarp();

        const Vol v{D.vol, D.dim[0], D.dim[1], D.dim[2]};
        FloatSum sum = {0.0f, 0.0f, 0.0f};
        int bad = kOk;
        unsigned nsteps = 0;
        const int v0 = t * D.tile;
        const int v1 = min(D.n_vox, v0 + D.tile);
        // every lane runs the same number of iterations (the march is warp-synchronous)
        for (int vb = v0; vb < v1; vb += 32) {
            const int vi = vb + lane;
            const bool valid = vi < v1;
            const short4 cv = valid ? __ldg(D.coords + vi) : make_short4(0, 0, 0, 0);
#pragma unroll 1
            for (int leg = 0; leg < 2; leg++) {
                LegResult a;
                trace_leg<false, true>(tab.head[leg], tab.rule[leg], cv.x, cv.y, cv.z, valid, v,
                                       D.full_iteration, D.voxel, D.sq, D.sq_stride, D.qtab, seg + tid, a,
                                       D.voxelf);
                bad |= a.status;
                nsteps += valid ? (unsigned)a.len : 0u;
                // the incident leg's lengths wait in shared memory while the
                // diffracted leg marches; then (L_incident + L_diffracted) per
                // class, as cal_rate adds them
#pragma unroll
                for (int k = 0; k < 4; k++)
                    lsum[k][tid] = leg == 0 ? a.Lf[k] : lsum[k][tid] + a.Lf[k];
            }
            if (valid) {
                // cal_rate's exponent (AnACor/src/ray_tracing_basic.c:1573-1576), in FP32
                const float ex = D.muf[0] * lsum[0][tid] + D.muf[1] * lsum[1][tid] + D.muf[2] * lsum[2][tid] +
                                 D.muf[3] * lsum[3][tid];
                const float term = D.is_exp ? expf(-ex) : ex;
                sum_add(sum, term);
            }
        }
        if (bad)
            atomicOr(D.status, 1 << bad);
        if (D.steps) {
            unsigned long long w = nsteps;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                w += __shfl_down_sync(kAll, w, o);
            if (lane == 0)
                atomicAdd(D.steps, w);
        }
        finish_warp_item(sum, D, r, t, lane);
    }
}

// The A_h kernel on packed fields (centred, octant or bricked octant).
template <int kMinBlocks, bool kBrick>
__global__ void __launch_bounds__(kBlock, kMinBlocks + 1) field_kernel(const SampleDesc *__restrict__ descs, int n_desc,
                                                                   long long total_items,
                                                                   unsigned long long *__restrict__ work_counter)
{
    if (!block_shape_ok(n_desc > 0 ? descs[0].status : nullptr))
        return;
    FieldShared &S = field_shared();
    for (;;) {
        const int lane = thread_now() & 31;
        unsigned long long it = 0;
        if (lane == 0)
            it = atomicAdd(work_counter, 1ull);
        const long long item = (long long)__shfl_sync(kAll, it, 0);
        if (item >= total_items)
            break;
        const SampleDesc &D = descs[find_sample(descs, n_desc, item)];
        if (!D.field || (D.brick_sz != 0) != kBrick) {
            // launched over a sample without its field (or with the other
            // layout): an error status, no reads
            if (lane == 0)
                atomicOr(D.status, 1 << kErrArgs);
            continue;
        }
        const long long local = item - D.work_begin;
        const long long k = local / D.tiles;
        const long long r = D.order ? (long long)__ldg(D.order + k) : k;
        const int t = (int)(local - k * D.tiles);
        __syncwarp();   // the previous item's reads of the table are done
        fill_warp_tab(warp_tab(), D.refl + r, D, t, lane);
        __syncwarp();

        S.total[thread_now()] = make_float2(0.0f, 0.0f);
        S.total_low[thread_now()] = 0.0f;
        S.steps[thread_now()] = 0u;
        for (int vi = lane; vi < warp_tab().n; vi += 32) {
            float4 L;
#pragma unroll 1
            for (int leg = 0; leg < 2; leg++) {
                int len;
                L = field_leg<kBrick>(leg, vi, len);
                const int tid = thread_now();
                if (warp_tab().count_steps)
                    S.steps[tid] += (unsigned)len;
                if (leg == 0)
                    S.incident[tid] = L;
            }
            // L_incident + L_diffracted per class and cal_rate's exponent
            // (AnACor/src/ray_tracing_basic.c:1573-1576), in FP32
            const int tid = thread_now();
            const WarpTab &W = warp_tab();
            const float4 I = S.incident[tid];
            const float ex = W.mu[0] * (I.x + L.x) + W.mu[1] * (I.y + L.y) + W.mu[2] * (I.z + L.z) +
                             W.mu[3] * (I.w + L.w);
            const float term = W.is_exp ? expf(-ex) : ex;
            const float2 sc = S.total[tid];
            FloatSum sum = {sc.x, sc.y, S.total_low[tid]};
            sum_add(sum, term);
            S.total[tid] = make_float2(sum.s, sum.c);
            S.total_low[tid] = sum.d;
        }
        __syncwarp();
        if (D.steps) {
            unsigned long long w = S.steps[thread_now()];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                w += __shfl_down_sync(kAll, w, o);
            if (lane == 0)
                atomicAdd(D.steps, w);
        }
        {
            const float2 sc = S.total[thread_now()];
            finish_warp_item({sc.x, sc.y, S.total_low[thread_now()]}, D, r, t, lane);
        }
    }
}

// ---- iterative bisection (the reference's ib_test) ------------------------

// One boundary search of AnACor/src/bisection.c:150-238 on the ray
// c + m * q (q = the face rule's signed ratios, which are the ratios of the
// reference's increments(), bisection.c:21-148): halve [shortest, longest]
// down to the resolution 1.0; boundary 0: a label equal to cls moves longest
// in, boundary 1: it moves shortest out.  The point is floor(c + floor(mid) q).
// A position outside the volume (undefined in the reference) fails the ray.
//
// The probe points floor(c + fl(mid * q)) come from fixed point where that is
// exact: mid in 24.40 (truncated) times the rule's Q = llrint(q * 2^32) is a
// 128-bit product read as 56.72; its error is below 1.1e-6 for |q| < 2^16 and
// |mid q| < 2^14 (every point inside the volume), and the FP64 expression's
// own rounding below 1e-11, so a fraction more than 2^-18 from an integer has
// the reference's floor.  Nearer than that (or a rule without Q) the FP64
// expression is evaluated; the range tests sit on integers and are covered by
// the same margin.  The FP64 pipe, which binds this kernel, keeps only the
// bisection of [shortest, longest] itself.
__device__ __forceinline__ bool bisect_dev(double longest, double shortest, int cz, int cy, int cx,
                                           const FaceRule &R, const Vol &v, int boundary, int cls, int *p,
                                           double &mid)
{
    const double *q = R.q;
    const double c[3] = {(double)cz, (double)cy, (double)cx};
    const int ci[3] = {cz, cy, cx};
    const int dim[3] = {v.dz, v.dy, v.dx};
    constexpr unsigned long long kMargin = 1ull << 46;   // 2^-18 of the 64-bit fraction
    double diff = __dadd_rn(longest, -shortest);
    mid = __dmul_rn(__dadd_rn(longest, shortest), 0.5);
    while (diff > 1.0) {
        mid = __dmul_rn(__dadd_rn(longest, shortest), 0.5);
        const long long mfx = R.fast ? __double2ll_rz(__dmul_rn(mid, 1099511627776.0)) : 0ll;   // mid * 2^40
        int pp[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            bool exact = !R.fast;
            long long x = 0;
            if (!exact) {
                const long long hi = __mul64hi(mfx, R.Q[a]);
                const unsigned long long lo = (unsigned long long)mfx * (unsigned long long)R.Q[a];
                const unsigned long long frac = ((unsigned long long)(hi & 0xff) << 56) | (lo >> 8);
                exact = frac < kMargin || frac > ~kMargin;
                x = (long long)ci[a] + (hi >> 8);
            }
            if (exact) {
                const double xd = floor(__dadd_rn(c[a], __dmul_rn(mid, q[a])));
                if (!(xd >= 0.0 && xd < (double)dim[a]))
                    return false;
                x = (long long)xd;
            } else if (x < 0 || x >= dim[a]) {
                return false;
            }
            pp[a] = (int)x;
        }
        const int lab = __ldg(v.p + ((long long)pp[0] * v.dy + pp[1]) * v.dx + pp[2]);
        const bool hit = lab == cls;
        if (boundary == 0) {
            if (hit) longest = mid; else shortest = mid;
        } else {
            if (hit) shortest = mid; else longest = mid;
        }
        diff = __dadd_rn(longest, -shortest);
    }
    const double fm = floor(mid);
#pragma unroll
    for (int a = 0; a < 3; a++)
        p[a] = (int)floor(__dadd_rn(c[a], __dmul_rn(fm, q[a])));
    return true;
}

__device__ __forceinline__ double abs_sum3(const int *a, const int *b)
{
    return __dadd_rn(__dadd_rn(fabs((double)(a[0] - b[0])), fabs((double)(a[1] - b[1]))), fabs((double)(a[2] - b[2])));
}

// difference_length (bisection.c:260-270): z, then y, then x
__device__ __forceinline__ double seg_len(const int *s, const int *e, const double *vox)
{
    const double dz = __dmul_rn((double)(s[0] - e[0]), vox[0]);
    const double dy = __dmul_rn((double)(s[1] - e[1]), vox[1]);
    const double dx = __dmul_rn((double)(s[2] - e[2]), vox[2]);
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dz, dz), __dmul_rn(dy, dy)), __dmul_rn(dx, dx)));
}

// iterative_bisection + cal_path_bisection (bisection.c:272-463) for one leg;
// returns a status.  L = [liquor, loop, crystal, bubble].
__device__ __noinline__ int ib_leg(const LegHead &h, const FaceRule *rules, int cz, int cy, int cx, const Vol &v,
                                   int num_cls, const double *vox, double *L)
{
    L[0] = L[1] = L[2] = L[3] = 0.0;
    const int face = exit_face(h, cz, cy, cx, v);
    if (face == 0)
        return kErrNoFace;
    const FaceRule &R = rules[face - 1];
    if (R.status)
        return R.status;
    double air_longest;
    switch (face) {
    case 4: air_longest = (double)cy; break;
    case 5: air_longest = (double)(v.dy - 1 - cy); break;
    case 6: air_longest = (double)cx; break;
    case 1: air_longest = (double)(v.dx - 1 - cx); break;
    case 2: air_longest = (double)cz; break;
    default: air_longest = (double)(v.dz - 1 - cz); break;
    }
    const int p0[3] = {cz, cy, cx};
    int air[3], cr[3], li[3], lo[3], bi[3], bo[3];
    double m_air, m_cr, m_li, m_lo, m_bi, m_bo;
    if (!bisect_dev(air_longest, 0.0, cz, cy, cx, R, v, 0, 0, air, m_air) ||
        !bisect_dev(m_air, 0.0, cz, cy, cx, R, v, 1, 3, cr, m_cr))
        return kErrArgs;
    int npts = 3;
    const int *pa = nullptr, *pb = nullptr, *pc = nullptr, *pd = nullptr;   // points 3..6
    do {
        if (!bisect_dev(m_air, m_cr, cz, cy, cx, R, v, 0, 2, li, m_li))
            return kErrArgs;
        if (__ddiv_rn(abs_sum3(li, air), 3.0) > 1.0) {
            if (!bisect_dev(m_air, m_li, cz, cy, cx, R, v, 1, 2, lo, m_lo))
                return kErrArgs;
            if (__ddiv_rn(abs_sum3(li, lo), 3.0) <= 2.0)
                break;
            pa = li;
            pb = lo;
            npts = 5;
        }
        if (num_cls > 3) {
            if (!bisect_dev(m_air, m_cr, cz, cy, cx, R, v, 0, 4, bi, m_bi))
                return kErrArgs;
            if (abs_sum3(bi, air) > 1.0) {
                if (!bisect_dev(m_air, m_bi, cz, cy, cx, R, v, 1, 4, bo, m_bo))
                    return kErrArgs;
                if (__ddiv_rn(abs_sum3(bi, bo), 3.0) <= 2.0)
                    break;
                if (npts == 3) {
                    pa = bi;
                    pb = bo;
                } else {
                    pc = bi;
                    pd = bo;
                }
                npts += 2;
            }
        }
    } while (false);
    const double total = seg_len(p0, air, vox);
    const double cr_l = seg_len(p0, cr, vox);
    double lo_l = 0.0, bu_l = 0.0;
    // the lengths are read from the path by its length (5 points: loop, 7: bubble)
    if (npts == 5)
        lo_l = seg_len(pa, pb, vox);
    else if (npts == 7)
        bu_l = seg_len(pc, pd, vox);
    L[0] = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(total, -lo_l), -bu_l), -cr_l), -0.0);
    L[1] = lo_l;
    L[2] = cr_l;
    L[3] = bu_l;
    return kOk;
}

// ib_single_gridding's value (AnACor/src/ray_tracing.c:427-481) for n voxels
// and one direction (leg 1 of `dir`): the diffracted leg's lengths by
// iterative bisection, then cal_rate's exponent with a zero incident leg,
// sum_m mu_m (0 + L_m) left to right.  vox_mu = voxel[3], mu[4].
__global__ void __launch_bounds__(kBlock) ib_direction_kernel(const ReflTable *__restrict__ dir, const int8_t *vol,
                                                              int dz, int dy, int dx, const short4 *coords, int n,
                                                              const double *vox_mu, int num_cls, double *out,
                                                              int *status)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n)
        return;
    const short4 cv = coords[k];
    const Vol v{vol, dz, dy, dx};
    double L[4];
    const int st = ib_leg(dir->head[1], dir->rule[1], cv.x, cv.y, cv.z, v, num_cls, vox_mu, L);
    status[k] = st;
    if (st) {
        out[k] = 0.0;
        return;
    }
    const double *mu = vox_mu + 3;
    double a = __dmul_rn(mu[0], __dadd_rn(0.0, L[0]));
    a = __dadd_rn(a, __dmul_rn(mu[1], __dadd_rn(0.0, L[1])));
    a = __dadd_rn(a, __dmul_rn(mu[2], __dadd_rn(0.0, L[2])));
    a = __dadd_rn(a, __dmul_rn(mu[3], __dadd_rn(0.0, L[3])));
    out[k] = a;
}

// ib_test over every work item: as absorption_kernel, with bisection paths.
// An item a warp, as plan_split cuts them (down to one voxel a lane): with an
// item a block, 20 reflections of 20,000 voxels (1100x220x210) left seven
// warps of eight idle.
__global__ void __launch_bounds__(kBlock, 2) bisection_kernel(const SampleDesc *__restrict__ descs, int n_desc,
                                                              long long total_items,
                                                              unsigned long long *__restrict__ work_counter,
                                                              int num_cls)
{
    __shared__ ReflTable tabs[kWarps];
    if (!block_shape_ok(n_desc > 0 ? descs[0].status : nullptr))
        return;
    const int tid = threadIdx.x, lane = tid & 31;
    ReflTable &tab = tabs[tid >> 5];
    for (;;) {
        unsigned long long it = 0;
        if (lane == 0)
            it = atomicAdd(work_counter, 1ull);
        const long long item = (long long)__shfl_sync(kAll, it, 0);
        if (item >= total_items)
            break;
        const int si = find_sample(descs, n_desc, item);
        const SampleDesc &D = descs[si];
        const long long local = item - D.work_begin;
        const long long k = local / D.tiles;
        const long long r = D.order ? (long long)__ldg(D.order + k) : k;
        const int t = (int)(local - k * D.tiles);
        __syncwarp();   // the previous item's reads of the table are done
        {
            const int4 *src = reinterpret_cast<const int4 *>(D.refl + r);
            int4 *dst = reinterpret_cast<int4 *>(&tab);
            for (int k = lane; k < (int)(sizeof(ReflTable) / 16); k += 32)
                dst[k] = __ldg(src + k);
        }
        __syncwarp();
        const Vol v{D.vol, D.dim[0], D.dim[1], D.dim[2]};
        FloatSum sum = {0.0f, 0.0f, 0.0f};
        const int v1 = min(D.n_vox, (t + 1) * D.tile);
        for (int vi = t * D.tile + lane; vi < v1; vi += 32) {
            const short4 cv = __ldg(D.coords + vi);
            double a[4], b[4];
            int st = ib_leg(tab.head[0], tab.rule[0], cv.x, cv.y, cv.z, v, num_cls, D.voxel, a);
            if (!st)
                st = ib_leg(tab.head[1], tab.rule[1], cv.x, cv.y, cv.z, v, num_cls, D.voxel, b);
            if (st) {
                atomicOr(D.status, 1 << st);
                continue;
            }
            // cal_rate, operand order of AnACor/src/ray_tracing_basic.c:1573-1576
            const double t0 = __dmul_rn(D.mu[0], __dadd_rn(a[0], b[0]));
            const double t1 = __dmul_rn(D.mu[1], __dadd_rn(a[1], b[1]));
            const double t2 = __dmul_rn(D.mu[2], __dadd_rn(a[2], b[2]));
            const double t3 = __dmul_rn(D.mu[3], __dadd_rn(a[3], b[3]));
            const double ex = __dadd_rn(__dadd_rn(__dadd_rn(t0, t1), t2), t3);
            sum_add(sum, exp_neg(ex));
        }
        __syncwarp();
        finish_warp_item(sum, D, r, t, lane);
    }
}

// ---- bisection in fixed point ----------------------------------------------
//
// The same searches for volumes with axes of at most kBisectFixedDim voxels.
// Every value a search halves is a dyadic number there: the first one starts
// from [0, n] with n < 2^10 and halves at most 10 times, each later one starts
// from earlier results and adds at most 10 bits, the deepest chain (sample
// boundary, crystal boundary, loop or bubble inner, outer boundary) ends on
// multiples of 2^-40.  The reference's FP64 halvings are exact on such values
// (at most 50 bits), so 24.40 integers take the same decisions.
//
// Probe points floor(c + mid q): on the step axis c +- mid exactly; on the
// others mid cut to 11.21 times the rule's 32.32 ratio, T = floor(product) in
// 2^-21 units (32-bit: the exit face is the nearest, so displacements stay
// below 2^10).  It is off by at most |q| + 1.25 units (mid's and T's cuts, Q's
// rounding); a fraction within `margin` >= |q| + 2 units of an integer is
// recomputed with the reference's FP64 expression.  Lengths and the exponent
// run on pairs of floats.
//
// What is left is a chain of about 45 dependent label loads per ray, one ray
// a lane, so the kernel is bound by load latency and the warps an SM holds.
// 288x240x257, 6,800 voxels, 701 reflections: a call 8.9 ms (FP64 searches,
// FP64 pipe) -> 1.27 ms, A_h bit for bit the same.  Longer axes keep the FP64
// searches: their halvings would need more than 40 fractional bits.

constexpr long long kBisectOne = 1ll << 40;

struct BisectRay {
    const int8_t *start;     // the voxel's label
    uint32_t qa_lo, qa_hi, qb_lo, qb_hi;
    uint32_t margin;         // in 2^-21 units
    int ds, Ss, Sa, Sb;      // step direction; element strides
    int cs, ca, cb;          // start coordinates
    int ns, na, nb;          // dimensions
};

// the reference's FP64 probe point of axis a (0 z, 1 y, 2 x)
__device__ __noinline__ int bisect_exact(const WarpTab &W, int leg, int face, int axis, int c, double mid)
{
    const double x = floor(__dadd_rn((double)c, __dmul_rn(mid, W.refl->rule[leg][face - 1].q[axis])));
    return x >= -1.0 && x <= 8192.0 ? (int)x : -1;
}

// One boundary search: longest moves in on a label equal to cls (boundary 0),
// or shortest moves out on one (boundary 1).  False when a probe leaves the
// volume.
__device__ __forceinline__ bool bisect_fixed(const BisectRay &r, const WarpTab &W, int leg, int axis,
                                             long long longest, long long shortest, bool boundary, int cls,
                                             long long &mid)
{
    mid = (longest + shortest) >> 1;
    while (longest - shortest > kBisectOne) {
        mid = (longest + shortest) >> 1;
        const uint32_t m = (uint32_t)(mid >> 19);
        const int ta = (int)(__umulhi(m, r.qa_lo) + m * r.qa_hi);
        const int tb = (int)(__umulhi(m, r.qb_lo) + m * r.qb_hi);
        const int whole = (int)(mid >> 40);
        const int sd = r.ds > 0 ? whole : -whole - ((mid & (kBisectOne - 1)) != 0);
        int da = ta >> 21, db = tb >> 21;
        constexpr uint32_t kFrac = (1u << 21) - 1u;
        if (min(((uint32_t)ta + r.margin) & kFrac, ((uint32_t)tb + r.margin) & kFrac) < 2u * r.margin) {
            const double md = (double)mid * 0x1p-40;
            const int face = W.rule[leg][axis].face;
            da = bisect_exact(W, leg, face, axis == 0 ? 1 : 0, r.ca, md) - r.ca;
            db = bisect_exact(W, leg, face, axis == 2 ? 1 : 2, r.cb, md) - r.cb;
        }
        if ((unsigned)(r.cs + sd) >= (unsigned)r.ns || (unsigned)(r.ca + da) >= (unsigned)r.na ||
            (unsigned)(r.cb + db) >= (unsigned)r.nb)
            return false;
        const int lab = __ldg(r.start + (sd * r.Ss + da * r.Sa + db * r.Sb));
        if ((lab == cls) != boundary)
            longest = mid;
        else
            shortest = mid;
    }
    return true;
}

// the search's point floor(c + floor(mid) q) as its displacement on (step
// axis, a, b)
struct BisectPoint {
    int s, a, b;
};

__device__ __forceinline__ BisectPoint bisect_point(const BisectRay &r, const WarpTab &W, int leg, int axis,
                                                    long long mid)
{
    const int i = (int)(mid >> 40);
    uint32_t fa, fb;
    BisectPoint p;
    p.s = r.ds * i;
    p.a = fixed_at(i, r.qa_lo, r.qa_hi, kFieldMargin, fa);
    p.b = fixed_at(i, r.qb_lo, r.qb_hi, kFieldMargin, fb);
    if (min(fa, fb) < 2u * kFieldMargin) {
        const int face = W.rule[leg][axis].face;
        p.a = bisect_exact(W, leg, face, axis == 0 ? 1 : 0, r.ca, (double)i) - r.ca;
        p.b = bisect_exact(W, leg, face, axis == 2 ? 1 : 2, r.cb, (double)i) - r.cb;
    }
    return p;
}

__device__ __forceinline__ BisectPoint operator-(const BisectPoint &x, const BisectPoint &y)
{
    return {x.s - y.s, x.a - y.a, x.b - y.b};
}

__device__ __forceinline__ int abs_sum(const BisectPoint &d) { return abs(d.s) + abs(d.a) + abs(d.b); }

// length of a displacement; v2: the squared voxel edges of (step axis, a, b)
__device__ __forceinline__ FloatPair pair_length(const BisectPoint &d, const FloatPair *v2)
{
    const FloatPair s = pair_add(pair_add(pair_mul(v2[0], (float)(d.s * d.s)), pair_mul(v2[1], (float)(d.a * d.a))),
                                 pair_mul(v2[2], (float)(d.b * d.b)));
    return pair_sqrt(s);
}

// iterative_bisection and cal_path_bisection (AnACor/src/bisection.c:272-463)
// for one leg; adds mu_m L_m to `sum`.  Returns a status.
__device__ __forceinline__ int bisect_leg_fixed(const BisectRay &r, const WarpTab &W, int leg, int axis, int reach,
                                                int num_cls, const FloatPair *v2, const FloatPair *mu, FloatPair *L)
{
    long long m_air, m_cr, m_in, m_out;
    if (!bisect_fixed(r, W, leg, axis, (long long)reach << 40, 0, false, 0, m_air) ||
        !bisect_fixed(r, W, leg, axis, m_air, 0, true, 3, m_cr))
        return kErrArgs;
    const BisectPoint air = bisect_point(r, W, leg, axis, m_air);
    FloatPair pair_l = {0.0f, 0.0f};   // the last pair of points found
    int pairs = 0;
    bool more = true;
    if (!bisect_fixed(r, W, leg, axis, m_air, m_cr, false, 2, m_in))
        return kErrArgs;
    BisectPoint in = bisect_point(r, W, leg, axis, m_in);
    if (abs_sum(in - air) > 3) {
        if (!bisect_fixed(r, W, leg, axis, m_air, m_in, true, 2, m_out))
            return kErrArgs;
        const BisectPoint d = in - bisect_point(r, W, leg, axis, m_out);
        if (abs_sum(d) <= 6) {
            more = false;
        } else {
            pair_l = pair_length(d, v2);
            pairs = 1;
        }
    }
    if (more && num_cls > 3) {
        if (!bisect_fixed(r, W, leg, axis, m_air, m_cr, false, 4, m_in))
            return kErrArgs;
        in = bisect_point(r, W, leg, axis, m_in);
        if (abs_sum(in - air) > 1) {
            if (!bisect_fixed(r, W, leg, axis, m_air, m_in, true, 4, m_out))
                return kErrArgs;
            const BisectPoint d = in - bisect_point(r, W, leg, axis, m_out);
            if (abs_sum(d) > 6) {
                pair_l = pair_length(d, v2);
                pairs++;
            }
        }
    }
    // read from the path by its length: one pair is counted as loop, of two
    // the second as bubble
    const FloatPair cr = pair_length(bisect_point(r, W, leg, axis, m_cr), v2);
    L[0] = pair_add(pair_add(pair_length(air, v2), pair_neg(pair_l)), pair_neg(cr));
    L[1] = pairs == 1 ? pair_l : FloatPair{0.0f, 0.0f};
    L[2] = cr;
    L[3] = pairs == 2 ? pair_l : FloatPair{0.0f, 0.0f};
    return kOk;
}

__global__ void __launch_bounds__(kBlock, 4) bisection_fixed_kernel(const SampleDesc *__restrict__ descs, int n_desc,
                                                                    long long total_items,
                                                                    unsigned long long *__restrict__ work_counter,
                                                                    int num_cls)
{
    __shared__ WarpTab tabs[kWarps];
    __shared__ FloatPair consts[kWarps][7];   // squared voxel edges (z, y, x), mu
    // third floats of the lanes' sums: a third register spills what a search
    // needs (701 reflections of 6,800 voxels: 1.0 % slower), all three here are
    // 2 KB more a block out of L1 (0.6 %)
    __shared__ float low[kBlock];
    if (!block_shape_ok(n_desc > 0 ? descs[0].status : nullptr))
        return;
    const int tid = threadIdx.x, lane = tid & 31;
    WarpTab &W = tabs[tid >> 5];
    FloatPair *K = consts[tid >> 5];
    for (;;) {
        unsigned long long it = 0;
        if (lane == 0)
            it = atomicAdd(work_counter, 1ull);
        const long long item = (long long)__shfl_sync(kAll, it, 0);
        if (item >= total_items)
            break;
        const SampleDesc &D = descs[find_sample(descs, n_desc, item)];
        const long long local = item - D.work_begin;
        const long long k = local / D.tiles;
        const long long refl = D.order ? (long long)__ldg(D.order + k) : k;
        const int t = (int)(local - k * D.tiles);
        __syncwarp();   // the previous item's reads of the table are done
        fill_warp_tab(W, D.refl + refl, D, t, lane);
        if (lane < 3)
            K[lane] = pair_of(__dmul_rn(D.voxel[lane], D.voxel[lane]));
        else if (lane < 7)
            K[lane] = pair_of(D.mu[lane - 3]);
        __syncwarp();
        float s = 0.0f, c = 0.0f;
        low[tid] = 0.0f;
        const int n = min(D.tile, D.n_vox - t * D.tile);
        const short4 *coords = D.coords + (long long)t * D.tile;
        for (int vi = lane; vi < n; vi += 32) {
            FloatPair L[2][4];
            int bad = kOk;
#pragma unroll 1
            for (int leg = 0; leg < 2 && !bad; leg++) {
                const short4 cv = __ldg(coords + vi);
                const Vol v{D.vol, D.dim[0], D.dim[1], D.dim[2]};
                const int face = exit_face(D.refl[refl].head[leg], cv.x, cv.y, cv.z, v);
                if (face == 0) {
                    bad = kErrNoFace;
                    break;
                }
                // the rule of the exit axis (of its own face: a start on a min
                // plane may leave against the direction of travel)
                const FaceRule &F = D.refl[refl].rule[leg][face - 1];
                if (F.status) {
                    bad = F.status;
                    break;
                }
                const int axis = F.count_axis;
                const HotRule &R = W.rule[leg][axis];
                const int dz = D.dim[0], dy = D.dim[1], dx = D.dim[2];
                int reach;
                switch (face) {
                case 4: reach = cv.y; break;
                case 5: reach = dy - 1 - cv.y; break;
                case 6: reach = cv.z; break;
                case 1: reach = dx - 1 - cv.z; break;
                case 2: reach = cv.x; break;
                default: reach = dz - 1 - cv.x; break;
                }
                const long long qm = max(F.Q[axis == 0 ? 1 : 0] < 0 ? -F.Q[axis == 0 ? 1 : 0] : F.Q[axis == 0 ? 1 : 0],
                                         F.Q[axis == 2 ? 1 : 2] < 0 ? -F.Q[axis == 2 ? 1 : 2] : F.Q[axis == 2 ? 1 : 2]);
                if (!F.fast || R.face != face || qm >= 64ll << 32) {
                    // ratios beyond the 32-bit products: the FP64 searches
                    double Ld[4];
                    bad = ib_leg(D.refl[refl].head[leg], D.refl[refl].rule[leg], cv.x, cv.y, cv.z, v, num_cls, D.voxel,
                                 Ld);
                    for (int m = 0; m < 4; m++)
                        L[leg][m] = pair_of(Ld[m]);
                    continue;
                }
                BisectRay r;
                r.start = D.vol + ((long long)cv.x * dy + cv.y) * dx + cv.z;
                r.qa_lo = R.qa_lo; r.qa_hi = R.qa_hi; r.qb_lo = R.qb_lo; r.qb_hi = R.qb_hi;
                r.margin = (uint32_t)(qm >> 32) + 3u;
                r.ds = R.ds;
                r.Ss = R.dS * R.ds; r.Sa = R.Sa; r.Sb = R.Sb;
                r.cs = pick3(axis, cv.x, cv.y, cv.z);
                r.ca = axis == 0 ? cv.y : cv.x;
                r.cb = axis == 2 ? cv.y : cv.z;
                r.ns = pick3(axis, dz, dy, dx);
                r.na = axis == 0 ? dy : dz;
                r.nb = axis == 2 ? dy : dx;
                const FloatPair v2[3] = {K[axis], K[axis == 0 ? 1 : 0], K[axis == 2 ? 1 : 2]};
                bad = bisect_leg_fixed(r, W, leg, axis, reach, num_cls, v2, K + 3, L[leg]);
            }
            if (bad) {
                atomicOr(D.status, 1 << bad);
                continue;
            }
            // cal_rate (AnACor/src/ray_tracing_basic.c:1573-1576)
            FloatPair ex = {0.0f, 0.0f};
#pragma unroll
            for (int m = 0; m < 4; m++)
                ex = pair_add(ex, pair_mul(pair_add(L[0][m], L[1][m]), K[3 + m]));
            FloatSum sum = {s, c, low[tid]};
            sum_add(sum, exp_neg(ex));
            s = sum.s;
            c = sum.c;
            low[tid] = sum.d;
        }
        __syncwarp();
        finish_warp_item({s, c, low[tid]}, D, refl, t, lane);
    }
}

// Absorption map: work item = (grid direction, tile of voxels); the
// diffracted leg of every voxel, one output per (direction, voxel).
__global__ void __launch_bounds__(kBlock, 2) gridding_map_kernel(const MapDesc *__restrict__ dp, long long total_items,
                                                                 unsigned long long *__restrict__ work_counter)
{
    __shared__ ReflTable tab;
    __shared__ uint16_t seg[kMaxSegments * kBlock];
    __shared__ long long item_s;
    const MapDesc &D = *dp;
    if (!block_shape_ok(D.status))
        return;
    const int tid = threadIdx.x;
    const Vol v{D.vol, D.dim[0], D.dim[1], D.dim[2]};
    for (;;) {
        if (tid == 0)
            item_s = (long long)atomicAdd(work_counter, 1ull);
        __syncthreads();
        const long long item = item_s;
        if (item >= total_items)
            break;
        const long long d = item / D.tiles;
        const int t = (int)(item - d * D.tiles);
        {
            const int4 *src = reinterpret_cast<const int4 *>(D.dirs + d);
            int4 *dst = reinterpret_cast<int4 *>(&tab);
            for (int k = tid; k < (int)(sizeof(ReflTable) / 16); k += kBlock)
                dst[k] = __ldg(src + k);
        }
        __syncthreads();
        int bad = kOk;
        const int v0 = t * D.tile;
        const int v1 = min(D.n_vox, v0 + D.tile);
        float *row = D.out + d * D.ld;
        for (int vb = v0; vb < v1; vb += kBlock) {
            const int vi = vb + tid;
            const bool valid = vi < v1;
            const short4 cv = valid ? __ldg(D.coords + vi) : make_short4(0, 0, 0, 0);
            LegResult a;
            trace_leg<false>(tab.head[1], tab.rule[1], cv.x, cv.y, cv.z, valid, v, D.full_iteration,
                                            D.voxel, D.sq, D.sq_stride, D.qtab, seg + tid, a);
            if (!valid)
                continue;
            double val;
            if (a.status) {
                bad |= a.status;
                val = __longlong_as_double(0x7ff8000000000000ll);
            } else {
                // cal_rate with a zero incident leg: (0 + L) == L per class
                const double t0 = __dmul_rn(D.mu[0], a.L[0]);
                const double t1 = __dmul_rn(D.mu[1], a.L[1]);
                const double t2 = __dmul_rn(D.mu[2], a.L[2]);
                const double t3 = __dmul_rn(D.mu[3], a.L[3]);
                const double ex = __dadd_rn(__dadd_rn(__dadd_rn(t0, t1), t2), t3);
                val = D.is_exp ? exp(-ex) : ex;
            }
            const long long o = D.col ? __ldg(D.col + vi) : vi;
            if (D.out64)
                D.out64[d * D.ld + o] = val;
            else
                row[o] = (float)val;
        }
        if (bad)
            atomicOr(D.status, 1 << bad);
        __syncthreads();   // the table and item_s are rewritten next
    }
}

// The absorption map on the octant fields, bit for bit the FP64 values rounded
// to float: the reference's sum mu_m L_m = total / (len - 1) * sum mu_m span_m
// is formed on pairs of floats (within 2^-43 of it, the squared displacements
// exact: those of an axis beyond 4,096 need 26 bits), and where that leaves the
// rounding to float open (a few in 10^5) map_slow evaluates the FP64
// expressions.  On GB300 those bound the kernel before (a square root, the
// quotients and the sums of every leg on an FP64 pipe of two lanes a cycle).
// 64,800 directions x 1,657 voxels of a 512x512x400 volume: 14.8 -> 4.9 ms
// in one launch; in the launches of a build 4.6, exit-face ties on the march
// (exact_axis), which left each of them a tail of 1 to 2 ms.
__global__ void __launch_bounds__(kBlock, 5) field_map_kernel(const SampleDesc *__restrict__ dp, long long total_items,
                                                              unsigned long long *__restrict__ work_counter,
                                                              float *__restrict__ out, long long ld,
                                                              const int *__restrict__ col)
{
    FloatPair *consts = field_shared().consts;
    const SampleDesc &D = *dp;
    if (!block_shape_ok(D.status))
        return;
    const int tid = threadIdx.x, lane = tid & 31;
    WarpTab &W = field_shared().tabs[tid >> 5];
    if (tid < 3)
        consts[tid] = pair_of(__dmul_rn(D.voxel[tid], D.voxel[tid]));
    else if (tid < 7)
        consts[tid] = pair_of(D.mu[tid - 3]);
    __syncthreads();
    // The error bound is relative to the sum: no cancellation between terms,
    // and squares that a float's range holds.  Every class counts, an absent
    // one with length zero: infinite or undefined coefficients give NaN for it.
    bool plain = true;
    for (int a = 0; a < 4; a++)
        plain = plain && D.mu[a] >= 0.0 && D.mu[a] < 1e300;
    for (int a = 0; a < 3; a++)
        plain = plain && fabs(D.voxel[a]) > 0x1p-40 && fabs(D.voxel[a]) < 0x1p40;
    for (;;) {
        unsigned long long it = 0;
        if (lane == 0)
            it = atomicAdd(work_counter, 1ull);
        const long long item = (long long)__shfl_sync(kAll, it, 0);
        if (item >= total_items)
            break;
        const long long d = item / D.tiles;
        const int t = (int)(item - d * D.tiles);
        __syncwarp();   // the previous item's reads of the table are done
        fill_warp_tab(W, D.refl + d, D, t, lane);
        __syncwarp();
        for (int vi = lane; vi < W.n; vi += 32) {
            const float val = field_march<false, true>(
                1, vi,
                [&] {
                    return !plain ? map_slow(vi, kFromStart, 0, 0, 1, 0, 0, -1, 0, 0) : (W.is_exp ? 1.0f : 0.0f);
                },
                [&](int i, int nseg, int d0, int d1, int d2) {
                    const FloatPair tot = pair_sqrt(
                        pair_add(pair_add(pair_mul(consts[0], pair_square((float)d0)),
                                          pair_mul(consts[1], pair_square((float)d1))),
                                 pair_mul(consts[2], pair_square((float)d2))));
                    FloatPair sum = {0.0f, 0.0f};
                    int cur = 3 << 13;
                    for (int j = 1; j <= nseg; j++) {
                        const int nxt = j < nseg ? (int)seg_list()[j * kBlock] : i;
                        const int cls = cur >> 13, span = (nxt & 0x1fff) - (cur & 0x1fff);
                        if (cls >= 1)
                            sum = pair_add(sum, pair_mul(consts[2 + cls], (float)span));
                        cur = nxt;
                    }
                    const FloatPair p = pair_mul(tot, sum);
                    const float den = (float)(i - 1);
                    const float q = __fdiv_rn(p.h, den);
                    const FloatPair r = pair_norm(q, __fdividef(__fadd_rn(__fmaf_rn(-q, den, p.h), p.l), den));
                    float v;
                    bool sure;
                    if (W.is_exp) {
                        const double ex = (double)r.h + (double)r.l, y = exp(-ex);
                        const double err = y * (fabs(ex) * 0x1p-40 + 0x1p-50);
                        v = (float)y;
                        sure = (float)(y + err) == v && (float)(y - err) == v;
                    } else {
                        // the float nearest to r, unless r is within 2^-40 of a tie
                        const float err = fabsf(r.h) * 0x1p-40f;
                        v = r.h;
                        sure = __fadd_rn(r.h, r.l + err) == r.h && __fadd_rn(r.h, r.l - err) == r.h && r.h > 0x1p-80f;
                    }
                    return plain && sure ? v
                                            : map_slow(vi, kFromStop, 0, i, nseg, 0, 0, d0, d1, d2);
                },
                [&](int from, int axis, int i, int nseg, int prev, int lim) {
                    return map_slow(vi, from, axis, i, nseg, prev, lim, -1, 0, 0);
                });
            const int k = t * D.tile + vi;
            out[d * ld + (col ? __ldg(col + k) : k)] = val;
        }
    }
}

// Per-voxel, per-leg detail for one reflection (path-level parity checks);
// same march code as the absorption kernel.
__global__ void __launch_bounds__(kBlock) leg_detail_kernel(const ReflTable *__restrict__ tabp, const int8_t *vol,
                                                            int dz, int dy, int dx, const short4 *coords, int n,
                                                            const double *voxel3, int full, const double *sq,
                                                            int sq_stride, const double *qtab, int *face, int *len,
                                                            int *nseg, int *first, int *last, double *L,
                                                            int *status)
{
    __shared__ ReflTable tab;
    __shared__ uint16_t seg[kMaxSegments * kBlock];
    __shared__ double vox[3];
    if (!block_shape_ok(status))
        return;
    {
        const int4 *src = reinterpret_cast<const int4 *>(tabp);
        int4 *dst = reinterpret_cast<int4 *>(&tab);
        for (int k = threadIdx.x; k < (int)(sizeof(ReflTable) / 16); k += kBlock)
            dst[k] = src[k];
        if (threadIdx.x < 3)
            vox[threadIdx.x] = voxel3[threadIdx.x];
    }
    __syncthreads();
    const int vi = blockIdx.x * kBlock + threadIdx.x;
    const bool valid = vi < n;
    const Vol v{vol, dz, dy, dx};
    const short4 cv = valid ? coords[vi] : make_short4(0, 0, 0, 0);
#pragma unroll 1
    for (int leg = 0; leg < 2; leg++) {
        LegResult a;
        trace_leg<true>(tab.head[leg], tab.rule[leg], cv.x, cv.y, cv.z, valid, v, full, vox, sq, sq_stride, qtab,
                        seg + threadIdx.x, a);
        if (!valid)
            continue;
        const int o = 2 * vi + leg;
        face[o] = a.face;
        len[o] = a.len;
        nseg[o] = a.nseg;
        status[o] = a.status;
        for (int k = 0; k < 3; k++) {
            first[3 * o + k] = a.first[k];
            last[3 * o + k] = a.last[k];
        }
        for (int k = 0; k < 4; k++)
            L[4 * o + k] = a.L[k];
    }
}

// int64 (z, y, x) coordinates -> short4; flags out-of-range voxels.
__global__ void pack_coords_kernel(const long long *__restrict__ c, int n, int dz, int dy, int dx,
                                   short4 *__restrict__ out, int *__restrict__ status_word)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const long long z = c[3 * i], y = c[3 * i + 1], x = c[3 * i + 2];
    if (z < 0 || z >= dz || y < 0 || y >= dy || x < 0 || x >= dx) {
        atomicOr(status_word, 1 << kErrArgs);
        out[i] = make_short4(0, 0, 0, 0);
        return;
    }
    out[i] = make_short4((short)z, (short)y, (short)x, 0);
}

// Quotient table: row d (1 <= d <= max_den) holds fl(s / d) for s = 1 .. d+1,
// rows packed one after another (row d starts at (d-1)(d+2)/2).
__global__ void quotient_table_kernel(double *__restrict__ q, int max_den)
{
    const long long total = (long long)max_den * (max_den + 3) / 2;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        // row d: the largest d with (d-1)(d+2)/2 <= k
        int d = (int)floor((sqrt(8.0 * (double)k + 9.0) - 1.0) / 2.0);
        if (d < 1)
            d = 1;
        while (d > 1 && (long long)(d - 1) * (d + 2) / 2 > k)
            d--;
        while ((long long)d * (d + 3) / 2 <= k)
            d++;
        const int s = (int)(k - (long long)(d - 1) * (d + 2) / 2) + 1;
        q[k] = __ddiv_rn((double)s, (double)d);
    }
}

}  // namespace

int rcp_table_init()
{
    static double2 host[kMaxDim + 2];
    host[0] = make_double2(0.0, 0.0);
    for (int d = 1; d < kMaxDim + 2; d++)
        host[d] = make_double2((double)d, 1.0 / (double)d);
    return cudaMemcpyToSymbol(g_num_rcp, host, sizeof(host)) == cudaSuccess ? kOk : kErrCuda;
}

size_t quotient_table_entries(int max_den)
{
    return max_den > 0 ? (size_t)max_den * (size_t)(max_den + 3) / 2 : 0;
}

cudaError_t launch_quotient_table(double *d_q, int max_den, cudaStream_t st)
{
    if (max_den <= 0)
        return cudaSuccess;
    quotient_table_kernel<<<1024, 256, 0, st>>>(d_q, max_den);
    return cudaGetLastError();
}

cudaError_t launch_pack_coords(const long long *d_c, int n, const int *dims, short4 *d_out, int *d_status,
                               cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    pack_coords_kernel<<<(n + 255) / 256, 256, 0, st>>>(d_c, n, dims[0], dims[1], dims[2], d_out, d_status);
    return cudaGetLastError();
}

int absorption_variant()
{
    static const int v = [] {
        const char *e = std::getenv("ANACOR_CTAS_PER_SM");
        const int x = e ? std::atoi(e) : kDefaultMinBlocks;
        return (x >= 1 && x <= 4) ? x : kDefaultMinBlocks;
    }();
    return v;
}

cudaError_t launch_absorption(const SampleDesc *d_descs, int n_desc, long long total_items,
                              unsigned long long *d_counter, int grid, cudaStream_t st, int variant)
{
    if (total_items <= 0)
        return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess)
        return e;
#define ANACOR_COOP(B) absorption_kernel<B><<<grid, kBlock, 0, st>>>(d_descs, n_desc, total_items, d_counter)
#define ANACOR_FIELD(B, K) field_kernel<B, K><<<grid, kBlock, sizeof(FieldShared), st>>>(d_descs, n_desc, total_items, d_counter)
    switch (variant > 0 ? variant : absorption_variant()) {
    case 1: ANACOR_COOP(1); break;
    case 3: ANACOR_COOP(3); break;
    case 4: ANACOR_COOP(4); break;
    case 5: ANACOR_FIELD(1, false); break;
    case 6: ANACOR_FIELD(2, false); break;
    case 7: ANACOR_FIELD(3, false); break;
    case 8: ANACOR_FIELD(4, false); break;
    case 9: ANACOR_FIELD(1, true); break;
    case 10: ANACOR_FIELD(2, true); break;
    case 11: ANACOR_FIELD(3, true); break;
    case 12: ANACOR_FIELD(4, true); break;
    default: ANACOR_COOP(2); break;
    }
#undef ANACOR_COOP
#undef ANACOR_FIELD
    return cudaGetLastError();
}

cudaError_t launch_leg_detail(const ReflTable *d_tab, const int8_t *d_vol, const int *dims, const short4 *d_coords,
                              int n, const double *d_voxel, int full, const double *d_sq, int sq_stride,
                              const double *d_qtab, int *face, int *len, int *nseg, int *first, int *last, double *L,
                              int *status, cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    leg_detail_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(d_tab, d_vol, dims[0], dims[1], dims[2],
                                                                    d_coords, n, d_voxel, full, d_sq, sq_stride,
                                                                    d_qtab, face, len, nseg, first, last, L, status);
    return cudaGetLastError();
}

cudaError_t launch_bisection(const SampleDesc *d_descs, int n_desc, long long total_items,
                             unsigned long long *d_counter, int grid, int num_cls, bool fixed, cudaStream_t st)
{
    if (total_items <= 0)
        return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess)
        return e;
    if (fixed)
        bisection_fixed_kernel<<<grid, kBlock, 0, st>>>(d_descs, n_desc, total_items, d_counter, num_cls);
    else
        bisection_kernel<<<grid, kBlock, 0, st>>>(d_descs, n_desc, total_items, d_counter, num_cls);
    return cudaGetLastError();
}

cudaError_t launch_ib_direction(const ReflTable *d_dir, const int8_t *d_vol, const int *dims, const short4 *d_coords,
                                int n, const double *d_vox_mu, int num_cls, double *d_out, int *d_status,
                                cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    ib_direction_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(d_dir, d_vol, dims[0], dims[1], dims[2],
                                                                      d_coords, n, d_vox_mu, num_cls, d_out,
                                                                      d_status);
    return cudaGetLastError();
}

int bisection_occupancy(int *blocks_per_sm, bool fixed)
{
    const cudaError_t e =
        fixed ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, bisection_fixed_kernel, kBlock, 0)
              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, bisection_kernel, kBlock, 0);
    return e == cudaSuccess ? kOk : kErrCuda;
}

cudaError_t launch_field_map(const SampleDesc *d_desc, long long total_items, unsigned long long *d_counter, int grid,
                             float *out, long long ld, const int *col, cudaStream_t st)
{
    if (total_items <= 0)
        return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess)
        return e;
    field_map_kernel<<<grid, kBlock, sizeof(FieldShared), st>>>(d_desc, total_items, d_counter, out, ld, col);
    return cudaGetLastError();
}

int field_map_occupancy(int *blocks_per_sm)
{
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, field_map_kernel, kBlock, sizeof(FieldShared)) == cudaSuccess
               ? kOk
               : kErrCuda;
}

cudaError_t launch_gridding_map(const MapDesc *d_desc, long long total_items, unsigned long long *d_counter, int grid,
                                cudaStream_t st)
{
    if (total_items <= 0)
        return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess)
        return e;
    gridding_map_kernel<<<grid, kBlock, 0, st>>>(d_desc, total_items, d_counter);
    return cudaGetLastError();
}

int gridding_map_occupancy(int *blocks_per_sm)
{
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, gridding_map_kernel, kBlock, 0) == cudaSuccess
               ? kOk
               : kErrCuda;
}

int absorption_block_threads() { return kBlock; }

int block_guard_selftest(int threads, int *status_out)
{
    // Launch the absorption kernel over no work with `threads` threads per
    // block, fewer than kBlock (a whole number of warps), and report the
    // status word it leaves.  The guard must refuse the launch before any
    // access; threads == kBlock must pass it and find no work.
    if (threads <= 0 || threads > kBlock || threads % 32 != 0 || !status_out)
        return kErrArgs;
    SampleDesc h{};
    SampleDesc *d = nullptr;
    unsigned long long *counter = nullptr;
    int *status = nullptr;
    if (cudaMalloc(&d, sizeof(SampleDesc)) != cudaSuccess)
        return kErrCuda;
    int rc = kErrCuda;
    if (cudaMalloc(&counter, sizeof(unsigned long long)) == cudaSuccess &&
        cudaMalloc(&status, sizeof(int)) == cudaSuccess && cudaMemset(status, 0, sizeof(int)) == cudaSuccess &&
        cudaMemset(counter, 0, sizeof(unsigned long long)) == cudaSuccess) {
        h.status = status;
        if (cudaMemcpy(d, &h, sizeof(h), cudaMemcpyHostToDevice) == cudaSuccess) {
            absorption_kernel<2><<<2, threads>>>(d, 1, 0, counter);
            if (cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess &&
                cudaMemcpy(status_out, status, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess)
                rc = kOk;
        }
    }
    cudaFree(status);
    cudaFree(counter);
    cudaFree(d);
    return rc;
}

// Preferred shared-memory carveout (percent of the unified L1/shared storage)
// of every absorption kernel; a hint to the driver.
int absorption_set_carveout(int pct, int field_pct)
{
    cudaError_t e = cudaSuccess;
#define ANACOR_CARVE(K, P) \
    if (e == cudaSuccess) \
        e = cudaFuncSetAttribute(K, cudaFuncAttributePreferredSharedMemoryCarveout, P)
    ANACOR_CARVE(absorption_kernel<1>, pct); ANACOR_CARVE(absorption_kernel<2>, pct);
    ANACOR_CARVE(absorption_kernel<3>, pct); ANACOR_CARVE(absorption_kernel<4>, pct);
#define ANACOR_CARVE2(B) \
    ANACOR_CARVE((field_kernel<B, false>), field_pct); ANACOR_CARVE((field_kernel<B, true>), field_pct)
    ANACOR_CARVE2(1); ANACOR_CARVE2(2); ANACOR_CARVE2(3); ANACOR_CARVE2(4);
#undef ANACOR_CARVE2
#undef ANACOR_CARVE
    return e == cudaSuccess ? kOk : kErrCuda;
}

int absorption_occupancy(int *blocks_per_sm, int variant)
{
    cudaError_t e;
#define ANACOR_OCC(K, S) cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, K, kBlock, S)
    switch (variant > 0 ? variant : absorption_variant()) {
    case 1: e = ANACOR_OCC(absorption_kernel<1>, 0); break;
    case 3: e = ANACOR_OCC(absorption_kernel<3>, 0); break;
    case 4: e = ANACOR_OCC(absorption_kernel<4>, 0); break;
    case 5: e = ANACOR_OCC((field_kernel<1, false>), sizeof(FieldShared)); break;
    case 6: e = ANACOR_OCC((field_kernel<2, false>), sizeof(FieldShared)); break;
    case 7: e = ANACOR_OCC((field_kernel<3, false>), sizeof(FieldShared)); break;
    case 8: e = ANACOR_OCC((field_kernel<4, false>), sizeof(FieldShared)); break;
    case 9: e = ANACOR_OCC((field_kernel<1, true>), sizeof(FieldShared)); break;
    case 10: e = ANACOR_OCC((field_kernel<2, true>), sizeof(FieldShared)); break;
    case 11: e = ANACOR_OCC((field_kernel<3, true>), sizeof(FieldShared)); break;
    case 12: e = ANACOR_OCC((field_kernel<4, true>), sizeof(FieldShared)); break;
    default: e = ANACOR_OCC(absorption_kernel<2>, 0); break;
    }
#undef ANACOR_OCC
    return e == cudaSuccess ? kOk : kErrCuda;
}

}  // namespace anacor
