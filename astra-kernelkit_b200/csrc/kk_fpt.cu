// Exact adjoint of the ray-driven forward projection (kk_fp.cu), as a
// voxel-driven gather: no atomics, every voxel sums its own terms.
//
// The forward projection adds, for ray (a, r, c) and every slice s along
// the ray's dominant axis A, the bilinear sample of slice s at in-slice
// coordinates (y_s, z_s), times corr * outputScale. Its transpose gives
// voxel (s, j, k) the sum, over the rays whose slice-s sample touches it, of
// proj[a, r, c] * corr * outputScale * (that sample's weight on the voxel).
// To be the exact transpose of the forward projector (not of an idealised
// one), each candidate ray is set up by the same ray_setup(), its slice-s
// coordinates are rebuilt by the same slab-restart-and-increment sequence
// in the same float32 operations, and its weights come from the same weight
// rule (texture-compatible 1/256 weights or exact ones).
//
// Candidates: the footprint of voxel (j, k) in slice s is the square of
// sample positions y in [j - 1/2, j + 3/2), z in [k - 1/2, k + 3/2); its
// four corners are projected onto the detector and every pixel whose
// centre falls inside their bounding box (widened by 0.05 pixel) is tested
// exactly. Ray set-ups are computed once per chunk of angles into a
// caller-provided work buffer, so any volume size fits by chunking.
#include "kk_cone.cuh"

#include <climits>
#include <type_traits>

namespace kk {

struct FptArgs {
    float* vol;
    int64_t vs[3];
    int vn[3];
    int m0, m1, m2;  // world axes from slowest to fastest in memory
    int rank[3];     // memory rank of each world axis: 0 fastest .. 2 slowest
    const float* proj;
    const uint64_t* table;
    int64_t ps[3];
    int rows, cols;
    const kk_fp_angle* angles;
    float os[9];
    int slab;
    // by how far slice coordinates may be off the straight line, e per world
    // axis: half a texel and e; the least D2 step of a walked column, 2 e or
    // more
    float margin[3], min_step[3];
    int rec0, nrec;  // records of this chunk
    int accumulate;  // add to the volume (later chunks, or additive)
    float4* ray_ab;  // per * nrec entries, laid out per record (RayRecord)
    float* ray_pc;   // projection value * corr * outputScale per ray
};

// Ray set-ups of one record of the chunk, by class. General records: (a1,
// b1, a2, b2) per ray and the folded projection values, rows fastest (a warp
// of the gather, consecutive voxels along the fastest volume axis, reads
// neighbouring entries). Records whose rows share their D1 coordinate: per
// ray its (a2, value) and those of the next row, as (a2, a2', value,
// value'), columns fastest (a warp of the column pass walks consecutive
// columns, two rays per load) and the rows in the order of v's D2
// component, and a1 per column. b1 and b2 follow from the source.
struct RayRecord {
    float4* ab;
    float* pc;  // general: the value per ray; shared: a1 per column
};

__device__ __forceinline__ RayRecord ray_record(const FptArgs& L, int k) {
    const int64_t per = (int64_t)L.rows * L.cols;
    RayRecord R;
    R.ab = L.ray_ab + k * per;
    R.pc = L.ray_pc + k * per;
    return R;
}

constexpr int FPT_TILE_2 = 32;
constexpr int FPT_TILE_1 = 8;

__device__ __forceinline__ void cross3(const float* a, const float* b, float* o) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ float dot3(const float* a, const float* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// Component k of the point whose coordinate along axis A is t, along D1
// is d1 and along D2 is d2 (selects, not an indexed array, so nothing goes
// to local memory).
__device__ __forceinline__ float place(int k, int A, int D1, float t, float d1, float d2) {
    return k == A ? t : (k == D1 ? d1 : d2);
}

// circular scans: the detector's v has no component along A and D1, so
// every row of a column has bit for bit the same D1 coordinate sequence
// (as in the forward projector's shared path)
__device__ __forceinline__ bool shared_record(const kk_fp_angle* P, int A, int D1) {
    const float vA = A == 0 ? __ldg(&P->v[0]) : (A == 1 ? __ldg(&P->v[1]) : __ldg(&P->v[2]));
    const float vD1 = D1 == 0 ? __ldg(&P->v[0]) : __ldg(&P->v[1]);
    return vA == 0.f && vD1 == 0.f;
}

// Ray set-up of every ray of the chunk, in its record's layout. The
// projection value is folded in here, times the ray's corr * outputScale.
__global__ void fpt_rays_kernel(const FptArgs L) {
    const int64_t per = (int64_t)L.rows * L.cols;
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= per * L.nrec) return;
    const int k = (int)(id / per);
    const int cr = (int)(id - (int64_t)k * per);
    const kk_fp_angle* P = L.angles + L.rec0 + k;
    const int A = __ldg(&P->axis);
    const int D1 = A == 1 ? 0 : 1, D2 = A == 2 ? 0 : 2;
    const bool shared = shared_record(P, A, D1);
    float src[3], cor[3], u[3], v[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        src[q] = __ldg(&P->src[q]);
        cor[q] = __ldg(&P->corner[q]);
        u[q] = __ldg(&P->u[q]);
        v[q] = __ldg(&P->v[q]);
    }
    const int a = __ldg(&P->index);
    const float* plane = L.table ? (const float*)L.table[a] : L.proj + (int64_t)a * L.ps[0];
    auto value = [&](const RaySetup& R, int r, int c) {
        return __ldg(plane + (int64_t)r * L.ps[1] + (int64_t)c * L.ps[2]) * (R.corr * L.os[3 * A + 2]);
    };
    const RayRecord O = ray_record(L, k);
    if (shared) {
        const int pos = cr / L.cols, c = cr % L.cols;
        const bool up = pick3(v, D2) >= 0.f;
        const int r0 = up ? pos : L.rows - 1 - pos;
        const int r1 = up ? min(pos + 1, L.rows - 1) : max(r0 - 1, 0);
        const RaySetup R = ray_setup(src, cor, u, v, A, D1, D2, r0, c, L.os[3 * A], L.os[3 * A + 1]);
        const RaySetup Q = ray_setup(src, cor, u, v, A, D1, D2, r1, c, L.os[3 * A], L.os[3 * A + 1]);
        O.ab[cr] = make_float4(R.a2, Q.a2, value(R, r0, c), value(Q, r1, c));
        if (pos == 0) O.pc[c] = R.a1;
    } else {
        const int r = cr % L.rows, c = cr / L.rows;
        const RaySetup R = ray_setup(src, cor, u, v, A, D1, D2, r, c, L.os[3 * A], L.os[3 * A + 1]);
        O.pc[cr] = value(R, r, c);
        O.ab[cr] = make_float4(R.a1, R.b1, R.a2, R.b2);
    }
}

// A ray's in-slice coordinate at slice off + nst: the slab-start value v0
// followed by nst rounded adds of the slope, exactly as the forward
// projector computes it. With texture-compatible weights the split only
// sees floor(256 v - 127.5); each rounded add errs by at most half an ulp
// (2^-24 relative), so the sequence ends within eps of fma(nst, a, v0), and
// when no boundary of floor() lies within eps of that direct value (for
// |v| < 2^13, q = 256 v - 127.5 and q - floor(q) are exact in float32) it
// splits exactly as the sequence would and is returned instead.
template <bool TEX8>
__device__ __forceinline__ float slice_coord(float v0, float a, int nst) {
    if (TEX8) {
        const float fn = (float)nst;
        const float vd = fmaf(fn, a, v0);
        const float eps = (fn + 1.f) * 1.2e-7f * (fabsf(vd) + fabsf(a) * fn + 1.f);
        const float q = 256.f * vd - 127.5f;
        const float f = q - floorf(q);
        const float e = 256.f * 1.01f * eps + 1e-6f;
        if (fabsf(vd) < 8192.f && f > e && f < 1.f - e) return vd;
    }
    float v = v0;
    for (int q = 0; q < nst; ++q) v = __fadd_rn(v, a);
    return v;
}

// Candidate pixel box on the detector of the sample-position rectangle
// y in [y0, y1), z in [z0, z1) (centred coordinates along D1, D2) of slice
// position t of record P: the corners are projected centrally from the
// source; pixel c is a candidate when its centre c + 1/2 lies in the
// projected range widened by 0.05 pixel. False when a corner does not
// project (behind the source), then every pixel is a candidate.
__device__ __forceinline__ bool footprint_box(const FptArgs& L, const kk_fp_angle* P, int A, int D1, float t, float y0,
                                              float y1, float z0, float z1, int& c0, int& c1, int& rlo, int& rhi) {
    float src[3], cor[3], u[3], v[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        src[q] = __ldg(&P->src[q]);
        cor[q] = __ldg(&P->corner[q]);
        u[q] = __ldg(&P->u[q]);
        v[q] = __ldg(&P->v[q]);
    }
    // detector coordinates (pixel units, centre of pixel c at c + 1/2)
    float nrm[3], e1[3], e2[3], tmp[3];
    cross3(u, v, nrm);
    cross3(v, nrm, tmp);
    const float ue = dot3(u, tmp);
    cross3(nrm, u, e2);
    const float ve = dot3(v, e2);
    // the candidate box only needs a few correct digits (it is widened by
    // 0.05 pixel), so the fast reciprocal and division suffice
    const float iue = __frcp_rn(ue), ive = __frcp_rn(ve);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        e1[q] = tmp[q] * iue;
        e2[q] = e2[q] * ive;
    }
    float cs_[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) cs_[q] = cor[q] - src[q];
    const float num = dot3(cs_, nrm);
    float amin = 1e30f, amax = -1e30f, bmin = 1e30f, bmax = -1e30f;
    bool ok = true;
#pragma unroll
    for (int corner = 0; corner < 4; ++corner) {
        const float d1 = (corner & 1) ? y1 : y0;
        const float d2 = (corner & 2) ? z1 : z0;
        float d[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) d[q] = place(q, A, D1, t, d1, d2) - src[q];
        const float den = dot3(d, nrm);
        const float lam = __fdividef(num, den);
        ok = ok && isfinite(lam) && lam > 0.f;
        float qc[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) qc[q] = src[q] + lam * d[q] - cor[q];
        const float al = dot3(qc, e1), be = dot3(qc, e2);
        amin = fminf(amin, al);
        amax = fmaxf(amax, al);
        bmin = fminf(bmin, be);
        bmax = fmaxf(bmax, be);
    }
    c0 = 0;
    c1 = L.cols - 1;
    rlo = 0;
    rhi = L.rows - 1;
    if (ok && isfinite(amin) && isfinite(amax) && isfinite(bmin) && isfinite(bmax)) {
        c0 = max(c0, (int)ceilf(fmaxf(amin - 0.55f, -1.f)));
        c1 = min(c1, (int)floorf(fminf(amax - 0.45f, (float)L.cols)));
        rlo = max(rlo, (int)ceilf(fmaxf(bmin - 0.55f, -1.f)));
        rhi = min(rhi, (int)floorf(fminf(bmax - 0.45f, (float)L.rows)));
        return true;
    }
    return false;
}

// Contribution of record k of the chunk to voxel (w0, w1, w2): every pixel
// of the voxel's candidate box is tested exactly.
template <bool TEX8>
__device__ float gather_record(const FptArgs& L, int k, int w0, int w1, int w2) {
    const kk_fp_angle* P = L.angles + L.rec0 + k;
    const int A = __ldg(&P->axis);
    const int D1 = A == 1 ? 0 : 1, D2 = A == 2 ? 0 : 2;
    const int s = A == 0 ? w0 : (A == 1 ? w1 : w2);
    const int jv = D1 == 0 ? w0 : w1;
    const int kv = D2 == 0 ? w0 : w2;
    const int nS = A == 0 ? L.vn[0] : (A == 1 ? L.vn[1] : L.vn[2]);
    const int n1 = D1 == 0 ? L.vn[0] : L.vn[1];
    const int n2 = D2 == 0 ? L.vn[0] : L.vn[2];
    const float half1 = 0.5f * (float)n1, half2 = 0.5f * (float)n2;
    const int rA = A == 0 ? L.rank[0] : (A == 1 ? L.rank[1] : L.rank[2]);
    const int r1 = D1 == 0 ? L.rank[0] : L.rank[1];
    const int r2 = D2 == 0 ? L.rank[0] : L.rank[2];
    const int rule = 2 - rA;
    const bool a_fast = r1 < r2;
    const float t = (float)s - 0.5f * (float)nS + 0.5f;
    const int off = (s / L.slab) * L.slab;
    const float t1 = __fadd_rn(__fsub_rn((float)off, 0.5f * (float)nS), 0.5f);
    const int nst = s - off;
    const float e1 = D1 == 0 ? L.margin[0] : L.margin[1], e2 = D2 == 0 ? L.margin[0] : L.margin[2];
    int c0, c1, rlo, rhi;
    footprint_box(L, P, A, D1, t, (float)jv - e1 - half1, (float)(jv + 1) + e1 - half1, (float)kv - e2 - half2,
                  (float)(kv + 1) + e2 - half2, c0, c1, rlo, rhi);
    const RayRecord O = ray_record(L, k);
    float acc = 0.f;
    for (int c = c0; c <= c1; ++c) {
        for (int r = rlo; r <= rhi; ++r) {
            const int64_t id = (int64_t)c * L.rows + r;
            const float4 ab = __ldg(&O.ab[id]);
            // the forward projector's coordinates for slice s
            const Split sy = split_coord<TEX8>(slice_coord<TEX8>(__fadd_rn(fmaf(ab.x, t1, ab.y), half1), ab.x, nst));
            const Split sz = split_coord<TEX8>(slice_coord<TEX8>(__fadd_rn(fmaf(ab.z, t1, ab.w), half2), ab.z, nst));
            const int di = jv - sy.i, dj = kv - sz.i;
            if ((unsigned)di > 1u || (unsigned)dj > 1u) continue;
            const W4 wt = weights4<TEX8>(sy.w, sz.w, rule, a_fast);
            float wgt = di == 0 ? (dj == 0 ? wt.w00 : wt.w01) : (dj == 0 ? wt.w10 : wt.w11);
            if (TEX8) wgt *= 1.f / 256.f;
            acc = fmaf(__ldg(&O.pc[id]), wgt, acc);
        }
    }
    return acc;
}

// General path: one thread per voxel, every record of the chunk that the
// column passes do not handle.
template <bool TEX8>
__global__ void __launch_bounds__(FPT_TILE_2* FPT_TILE_1) fpt_gather_kernel(const FptArgs L) {
    // nothing to do when the column passes handle every record of the chunk
    int todo = 0;
    for (int k = threadIdx.y * FPT_TILE_2 + threadIdx.x; k < L.nrec; k += FPT_TILE_2 * FPT_TILE_1) {
        const kk_fp_angle* P = L.angles + L.rec0 + k;
        const int A = __ldg(&P->axis);
        if (!shared_record(P, A, A == 1 ? 0 : 1)) todo = 1;
    }
    if (!__syncthreads_or(todo)) return;
    const int i2 = blockIdx.x * FPT_TILE_2 + threadIdx.x;
    const int i1 = blockIdx.y * FPT_TILE_1 + threadIdx.y;
    const int i0 = blockIdx.z;
    if (i2 >= L.vn[L.m2] || i1 >= L.vn[L.m1]) return;
    // world indices of the voxel
    const int w0 = L.m0 == 0 ? i0 : (L.m1 == 0 ? i1 : i2);
    const int w1 = L.m0 == 1 ? i0 : (L.m1 == 1 ? i1 : i2);
    const int w2 = L.m0 == 2 ? i0 : (L.m1 == 2 ? i1 : i2);
    float acc = 0.f;
    for (int k = 0; k < L.nrec; ++k) {
        const kk_fp_angle* P = L.angles + L.rec0 + k;
        const int A = __ldg(&P->axis);
        if (shared_record(P, A, A == 1 ? 0 : 1)) continue;
        acc += gather_record<TEX8>(L, k, w0, w1, w2);
    }
    float* out = L.vol + (int64_t)w0 * L.vs[0] + (int64_t)w1 * L.vs[1] + (int64_t)w2 * L.vs[2];
    *out = L.accumulate ? *out + acc : acc;
}

// ---------------------------------------------------------------------------
// column pass for circular scans
// ---------------------------------------------------------------------------
// Records whose dominant axis is A and whose rows share their D1
// coordinate. One warp owns FPC_TJ rows (along D1) x FPC_TK texels (along
// D2) of one slice and keeps their sums in shared memory, a lane per row,
// while it walks the records. Work is laid out so that every ray is set up once
// per warp and nothing is tested per texel:
//
//   * the detector columns whose D1 texel pair {i1, i1 + 1} meets the rows
//     are packed over the lanes, 32 (record, column) pairs at a time across
//     record boundaries, so the lanes stay busy whatever a record's share;
//   * down its column a lane's D2 coordinate only grows, so the texels are
//     visited in order and each takes the lane's next rays, evaluated two at a time in paired FP32,
//     as long as their left texel is the current one. A ray adds to the
//     current texel and to the carry of the next, for both texel rows: its
//     four weights, exactly the forward projector's;
//   * the two sums of the columns (rows i1 and i1 + 1) then move to the
//     rows' lanes by shuffles whose sources are found once per 32 pairs.
//
// Lane 0 is the row before the first owned one: it only hands its second
// row's sums on. A column whose D2 step per detector row is below 1/16
// texel, or so small that the rounding of its slab's slices might change the
// order of its rays (FptArgs.min_step), or above 1024 texels, or not finite, is
// handed round the warp and tested ray by ray.
//
// Bound by instruction issue (80 % of the issue slots used on 384^3 x 128 x
// 576^2) and then by the latency of the ray loads. 256^3 x 360 x 384^2: 256.5
// -> 36.6 ms against a per-texel gather from shared-memory tables, 64^3 x 96 x
// 96^2: 1.60 -> 0.36 ms. The
// sums live in shared memory, not in registers: a register per texel means
// unrolling the texel loop, whose code then misses the instruction cache
// (75 ms).
constexpr int FPC_TJ = 31;
constexpr int FPC_TK = 32;
constexpr int FPC_LD = 33;  // stride of a warp's sums: rows are read back along D2

// weight rule of a pass: any (weights4), or the two rules of a D2 axis
// faster than D1
enum FpcRule { FPC_ANY = 0, FPC_RULE0 = 1, FPC_RULE1 = 2 };

// n rounded adds of a slope, n the same for the whole warp.
template <typename T, typename Add>
__device__ __forceinline__ T add_steps(T v, T a, int n, Add add) {
    for (int q = n >> 4; q > 0; --q) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v = add(v, a);
    }
    if (n & 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v = add(v, a);
    }
    if (n & 4) v = add(add(add(add(v, a), a), a), a);
    if (n & 2) v = add(add(v, a), a);
    if (n & 1) v = add(v, a);
    return v;
}

template <bool TEX8, int RULE, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 36 / WARPS) fpt_column_kernel(const FptArgs L, int A) {
    __shared__ unsigned s_rows[WARPS][32];
    __shared__ float s_acc[WARPS][FPC_TK * FPC_LD];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int D1 = A == 1 ? 0 : 1, D2 = A == 2 ? 0 : 2;
    const int nS = L.vn[A], n1 = L.vn[D1], n2 = L.vn[D2];
    // the block's warps share the records (which alternate between the axes
    // in small groups: a warp's place among WARPS rotates). Slices fastest:
    // the blocks in flight read nearly the same rays
    const int ktiles = (n2 + FPC_TK - 1) / FPC_TK;
    const int s = blockIdx.x % nS, tile = blockIdx.x / nS;
    const int j0 = (tile / ktiles) * FPC_TJ, k0 = (tile % ktiles) * FPC_TK;
    const float half1 = 0.5f * (float)n1, half2 = 0.5f * (float)n2;
    const int rule = 2 - L.rank[A];
    const bool a_fast = L.rank[D1] < L.rank[D2];
    const int off = (s / L.slab) * L.slab;
    const float t1 = __fadd_rn(__fsub_rn((float)off, 0.5f * (float)nS), 0.5f);
    const int nst = s - off;
    const float t = (float)s - 0.5f * (float)nS + 0.5f;
    const int rows = L.rows, cols = L.cols;
    auto add1 = [](float a, float b) { return __fadd_rn(a, b); };
    auto addp = [](float2 a, float2 b) { return add2(a, b); };

    float* acc = &s_acc[warp][lane];  // texel kk of this lane's row: acc[FPC_LD kk]
#pragma unroll
    for (int q = 0; q < FPC_TK; ++q) acc[FPC_LD * q] = 0.f;
    auto record = [&](int i) { return i * WARPS + ((warp + 3 * i) & (WARPS - 1)); };
    bool touched = false;

    for (int g0 = 0; g0 * WARPS < L.nrec; g0 += 32) {
        // the candidate columns of 32 records, one per lane
        int first = 0, cnt = 0;
        if (record(g0 + lane) < L.nrec) {
            const kk_fp_angle* P = L.angles + L.rec0 + record(g0 + lane);
            if (__ldg(&P->axis) == A && shared_record(P, A, D1)) {
                int c0, c1, rl, rh;
                footprint_box(L, P, A, D1, t, (float)j0 - L.margin[D1] - half1, (float)(j0 + FPC_TJ) + L.margin[D1] - half1,
                              (float)k0 - L.margin[D2] - half2, (float)(k0 + FPC_TK) + L.margin[D2] - half2, c0, c1, rl, rh);
                first = c0;
                cnt = rh >= rl ? max(c1 - c0 + 1, 0) : 0;
            }
        }
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(full, incl, d);
            if (lane >= d) incl += v;
        }
        const int total = __shfl_sync(full, incl, 31);
        first -= incl - cnt;  // column of flat index f: first + f
        touched = touched || total > 0;
        for (int b = 0; b < total; b += 32) {
            // this lane's (record, column)
            const int f = b + lane;
            int m = 0;
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1)
                if (__shfl_sync(full, incl, m + d - 1) <= f) m += d;
            const int c = __shfl_sync(full, first, m) + f;
            const RayRecord O = ray_record(L, record(g0 + m));
            const float4* ray = O.ab + c;  // position 0 of the column
            // its D1 split, and its D2 coordinate at the first and last ray
            Split sy;
            sy.i = 0;
            sy.w = 0.f;
            bool in = f < total, ok = true;
            float z0 = 0.f, dz = 1.f, sA = 0.f, s2 = 0.f;
            if (in) {
                const kk_fp_angle* P = L.angles + L.rec0 + record(g0 + m);
                const float a1 = __ldg(&O.pc[c]);
                sA = __ldg(&P->src[A]);
                s2 = __ldg(&P->src[D2]);
                const float b1 = fmaf(-a1, sA, __ldg(&P->src[D1]));  // as ray_setup
                const float y = add_steps(__fadd_rn(fmaf(a1, t1, b1), half1), a1, nst, add1);
                sy = split_coord<TEX8>(y);
                in = (unsigned)(sy.i - (j0 - 1)) < 32u;
                const float e0 = __ldg(&ray->x), e1 = __ldg(&ray[(int64_t)(rows - 1) * cols].x);
                z0 = fmaf(e0, t, fmaf(-e0, sA, s2)) + half2;
                const float z1 = fmaf(e1, t, fmaf(-e1, sA, s2)) + half2;
                dz = rows > 1 ? (z1 - z0) / (float)(rows - 1) : 1.f;
                ok = fabsf(dz) >= L.min_step[D2] && fabsf(dz) <= 1024.f && isfinite(z0);
                if (dz < 0.f) z0 = z1;
            }
            const int v1 = sy.i - (j0 - 1);
            // the lanes of each row
            s_rows[warp][lane] = 0;
            __syncwarp();
            const unsigned peers = __match_any_sync(full, in && ok ? v1 : -1);
            if (in && ok && lane == __ffs(peers) - 1) s_rows[warp][v1] = peers;
            __syncwarp();
            const unsigned mine = s_rows[warp][lane], rest = mine & (mine - 1);
            __syncwarp();
            const int most = __reduce_max_sync(full, __popc(mine));
            const int l0 = __ffs(mine) - 1, l1 = __ffs(rest) - 1;
            // Walks the columns' rays in order of growing D2. BACK: some lane
            // meets them from the last position (a slice behind the source).
            auto walk = [&](auto back_tag) {
                constexpr bool BACK = decltype(back_tag)::value;
                // start two or less before the first ray whose left texel
                // may be k0 - 1 (coordinates are off by half a step at most:
                // the row in hand makes up for it)
                const bool back = BACK && dz < 0.f;
                const float pf = floorf(((float)k0 - 0.5f - z0) / fabsf(dz)) - 1.f;
                int left = in && ok ? rows - (int)fminf(fmaxf(pf, 0.f), (float)rows) : 0;  // rays from here on
                // lanes without rays keep reading an entry that exists
                const float S = sy.w, S256 = S * (1.f / 256.f);
                const float4* rp = left > 0 ? ray + (int64_t)(rows - left) * cols : L.ray_ab;
                int ia, ib;  // left texels of the next two rays, from k0
                float2 F, pc;
                auto eval = [&]() {
                    float4 e = __ldg(!BACK || left <= 0 || !back ? rp : ray + (int64_t)max(left - 2, 0) * cols);
                    if (BACK && back && left > 1) e = make_float4(e.y, e.x, e.w, e.z);
                    pc = f2(e.z, e.w);
                    const float2 a2 = f2(e.x, e.y);
                    // slab start as the forward projector: (a2 t1 + b2) + half2
                    const float2 z = add_steps(add2(fma2(a2, f2(t1), fma2(a2, f2(-sA), f2(s2))), f2(half2)), a2, nst, addp);
                    if (TEX8) {
                        const float2 q = add2_rd(fma2_rd(z, f2(256.f), f2(-127.5f)), f2(12582912.f));
                        const int b0 = __float_as_int(q.x), b1 = __float_as_int(q.y);
                        ia = b0 >> 8;
                        ib = b1 >> 8;
                        F = add2(f2(__int_as_float((b0 & 255) | 0x4B000000), __int_as_float((b1 & 255) | 0x4B000000)),
                                 f2(-8388608.f));
                    } else {
                        const Split sa = split_coord<false>(z.x), sb = split_coord<false>(z.y);
                        ia = sa.i;
                        ib = sb.i;
                        F = f2(left > 0 ? sa.w : 0.f, left > 1 ? sb.w : 0.f);
                    }
                };
                auto advance = [&](int n) {
                    left -= n;
                    if (left > 0) rp += n * cols;
                };
                auto weights = [&](float2& w00, float2& w01, float2& w10, float2& w11) {
                    if (RULE == FPC_ANY || !TEX8) {
                        const W4 a = weights4<TEX8>(S, F.x, rule, a_fast), b = weights4<TEX8>(S, F.y, rule, a_fast);
                        w00 = f2(a.w00, b.w00);
                        w01 = f2(a.w01, b.w01);
                        w10 = f2(a.w10, b.w10);
                        w11 = f2(a.w11, b.w11);
                    } else {
                        // x1 = round half up(F S / 256), x0 as weights4
                        w11 = add2(add2_rd(fma2(F, f2(S256), f2(0.5f)), f2(12582912.f)), f2(-12582912.f));
                        w01 = RULE == FPC_RULE1 ? add2(add2_rd(fma2(F, f2(-S256), f2(0.5f)), f2(12582912.f)),
                                                       add2(F, f2(-12582912.f)))
                                                : sub2(F, w11);
                        w00 = sub2(f2(256.f - S), w01);
                        w10 = sub2(f2(S), w11);
                    }
                };
                const int base = k0 + (TEX8 ? 0x4B4000 : 0);  // texel k0 as eval numbers it
                eval();
                while (__any_sync(full, left > 0 && ia < base - 1)) {
                    advance((left > 0 && ia < base - 1) + (left > 1 && ib < base - 1));
                    eval();
                }
                float2 n0 = f2(0.f), n1s = f2(0.f);  // carries of the next texel, rows i1 and i1 + 1
                float* ak = acc - FPC_LD;
#pragma unroll 1
                for (int kk = base - 1; kk < base + FPC_TK; ++kk, ak += FPC_LD) {
                    bool ta = left > 0 && ia == kk, tb = left > 1 && ib == kk;
                    float2 w = f2(ta ? pc.x : 0.f, tb ? pc.y : 0.f), w00, w01, w10, w11;
                    weights(w00, w01, w10, w11);
                    float2 g0s = fma2(w, w00, n0), g1s = fma2(w, w10, n1s);
                    n0 = mul2(w, w01);
                    n1s = mul2(w, w11);
                    advance((int)ta + (int)tb);
                    eval();
                    // more than two rays of this texel
                    while (__any_sync(full, ta = left > 0 && ia == kk)) {
                        tb = left > 1 && ib == kk;
                        w = f2(ta ? pc.x : 0.f, tb ? pc.y : 0.f);
                        weights(w00, w01, w10, w11);
                        g0s = fma2(w, w00, g0s);
                        n0 = fma2(w, w01, n0);
                        g1s = fma2(w, w10, g1s);
                        n1s = fma2(w, w11, n1s);
                        advance((int)ta + (int)tb);
                        eval();
                    }
                    if (kk < base) continue;
                    const float G0 = g0s.x + g0s.y, G1 = g1s.x + g1s.y;
                    float h0 = 0.f, h1 = 0.f;
                    const float a0 = __shfl_sync(full, G0, l0), a1 = __shfl_sync(full, G1, l0);
                    const float c0 = __shfl_sync(full, G0, l1), c1 = __shfl_sync(full, G1, l1);
                    if (mine) {
                        h0 = a0;
                        h1 = a1;
                    }
                    if (rest) {
                        h0 += c0;
                        h1 += c1;
                    }
                    if (most > 2) {
                        unsigned more = rest & (rest - 1);
                        for (int q = 2; q < most; ++q) {
                            const int l = __ffs(more) - 1;
                            const float d0 = __shfl_sync(full, G0, l), d1 = __shfl_sync(full, G1, l);
                            if (more) {
                                h0 += d0;
                                h1 += d1;
                            }
                            more &= more - 1;
                        }
                    }
                    *ak += h0 + __shfl_up_sync(full, h1, 1);
                }
            };
            if (most > 0) {
                if (__any_sync(full, in && ok && dz < 0.f))
                    walk(std::true_type{});
                else
                    walk(std::false_type{});
            }
            // columns that cannot be walked: every ray against every texel
            unsigned odd = __ballot_sync(full, in && !ok);
            while (odd) {
                const int l = __ffs(odd) - 1;
                odd &= odd - 1;
                const int cq = __shfl_sync(full, c, l), vq = __shfl_sync(full, v1, l);
                const float4* rq = ray_record(L, record(g0 + __shfl_sync(full, m, l))).ab + cq;
                const float S = __shfl_sync(full, sy.w, l);
                const float qA = __shfl_sync(full, sA, l), q2 = __shfl_sync(full, s2, l);
                const int dj = lane - vq;  // this lane's row: i1 (0) or i1 + 1 (1)
                for (int r = 0; (unsigned)dj < 2u && r < rows; ++r) {
                    const float4 ab = __ldg(rq + (int64_t)r * cols);
                    const float z =
                        add_steps(__fadd_rn(fmaf(ab.x, t1, fmaf(-ab.x, qA, q2)), half2), ab.x, nst, add1);
                    const Split sz = split_coord<TEX8>(z);
                    const int kk = sz.i - k0;
                    const W4 w = weights4<TEX8>(S, sz.w, rule, a_fast);
                    if (kk >= 0 && kk < FPC_TK) acc[FPC_LD * kk] += ab.z * (dj ? w.w10 : w.w00);
                    if (kk >= -1 && kk < FPC_TK - 1) acc[FPC_LD * (kk + 1)] += ab.z * (dj ? w.w11 : w.w01);
                }
            }
            __syncwarp();
        }
    }
    touched = __syncthreads_or(touched);
    if (!touched && L.accumulate) return;
    // lanes along the faster of the two axes
    const bool along2 = L.rank[D2] < L.rank[D1];
    float* out = L.vol + (int64_t)s * L.vs[A];
    for (int q = warp; q < 32; q += WARPS) {
        const int row = along2 ? q : lane, kk = along2 ? lane : q;
        const int j = j0 - 1 + row, k = k0 + kk;
        if (row == 0 || j >= n1 || k >= n2) continue;
        float v = s_acc[0][kk * FPC_LD + row];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) v += s_acc[w][kk * FPC_LD + row];
        v *= 1.f / weight_unit<TEX8>();
        float* o = out + (int64_t)j * L.vs[D1] + (int64_t)k * L.vs[D2];
        *o = L.accumulate ? *o + v : v;
    }
}

}  // namespace kk

// ===========================================================================
// host side
// ===========================================================================
using namespace kk;

// (slice, tile) pairs of a pass, a block each
static int64_t column_blocks(const FptArgs& L, int A) {
    const int D1 = A == 1 ? 0 : 1, D2 = A == 2 ? 0 : 2;
    return (int64_t)L.vn[A] * ((L.vn[D1] + FPC_TJ - 1) / FPC_TJ) * ((L.vn[D2] + FPC_TK - 1) / FPC_TK);
}

template <int WARPS>
static void launch_column_split(const FptArgs& L, int A, bool tex8, cudaStream_t st) {
    const int D1 = A == 1 ? 0 : 1, D2 = A == 2 ? 0 : 2;
    constexpr int threads = 32 * WARPS;
    const unsigned blocks = (unsigned)column_blocks(L, A);
    // rules 0 and 1 with D2 the faster in-slice axis have their own code;
    // the middle + slowest plane (rule 2) and permuted volumes go by weights4
    const bool d2_fast = L.rank[D2] < L.rank[D1];
    if (!tex8)
        fpt_column_kernel<false, FPC_ANY, WARPS><<<blocks, threads, 0, st>>>(L, A);
    else if (d2_fast && L.rank[A] == 2)
        fpt_column_kernel<true, FPC_RULE0, WARPS><<<blocks, threads, 0, st>>>(L, A);
    else if (d2_fast && L.rank[A] == 1)
        fpt_column_kernel<true, FPC_RULE1, WARPS><<<blocks, threads, 0, st>>>(L, A);
    else
        fpt_column_kernel<true, FPC_ANY, WARPS><<<blocks, threads, 0, st>>>(L, A);
}

// The records are split over the warps of a block, which add their sums in
// order: four ways (four slices' tiles take turns more evenly than one long
// warp each: 256^3 x 360 x 384^2 41.1 -> 36.7 ms), eight ways while the
// (slice, tile) pairs fill less than about four rounds of the GPU (128 x 128
// x 100 x 180 2.60 -> 2.43 ms, 64^3 x 96 0.54 -> 0.37 ms; 192 x 192 x 180 x
// 250, at 54 pairs per SM, 10.62 ms four ways and 10.88 eight ways).
static void launch_column_pass(const FptArgs& L, int A, bool tex8, cudaStream_t st) {
    if (column_blocks(L, A) < (int64_t)kk_sm_count() * 40)
        launch_column_split<8>(L, A, tex8, st);
    else
        launch_column_split<4>(L, A, tex8, st);
}

extern "C" int kk_cone_fp_adjoint(const kk_projections* proj, const kk_volume* vol, const kk_fp_angle* angles,
                                  const float* out_scale, int32_t interp, int32_t slab, int32_t additive,
                                  float* work, int64_t work_floats, void* stream) {
    const char* who = "kk_cone_fp_adjoint";
    int rc = check_volume(vol, who);
    if (rc) return rc;
    rc = check_projections(proj, who);
    if (rc) return rc;
    if (!angles || !out_scale) return kk_fail(KK_ERR_INVALID_ARGUMENT, "%s: angles or out_scale is NULL", who);
    if (interp != KK_INTERP_TEX8 && interp != KK_INTERP_EXACT)
        return kk_fail(KK_ERR_INVALID_ARGUMENT, "%s: unknown interpolation mode %d", who, interp);
    if (vol->dtype != KK_F32 || proj->dtype != KK_F32)
        return kk_fail(KK_ERR_UNSUPPORTED, "%s: float32 volume and projections only", who);
    if (proj->table && proj->table_axis != 0)
        return kk_fail(KK_ERR_UNSUPPORTED, "%s: pointer table along the angle axis only", who);
    const int64_t per = proj->rows * proj->cols;
    if (!work || ((uintptr_t)work & 15) != 0)
        return kk_fail(KK_ERR_INVALID_ARGUMENT, "%s: work must be a 16-byte aligned device buffer", who);
    const int64_t chunk = work_floats / (5 * per);
    if (chunk < 1)
        return kk_fail(KK_ERR_INVALID_ARGUMENT, "%s: work holds %lld floats, at least 5 * rows * cols = %lld needed",
                       who, (long long)work_floats, (long long)(5 * per));
    FptArgs L = {};
    L.vol = (float*)vol->data;
    for (int k = 0; k < 3; ++k) {
        L.vs[k] = vol->stride[k];
        L.vn[k] = (int)vol->shape[k];
        L.ps[k] = proj->stride[k];
    }
    for (int k = 0; k < 3; ++k) {
        L.rank[k] = 0;
        for (int j = 0; j < 3; ++j)
            if (j != k && (vol->stride[j] < vol->stride[k] || (vol->stride[j] == vol->stride[k] && j > k))) ++L.rank[k];
    }
    for (int k = 0; k < 3; ++k) {
        if (L.rank[k] == 2) L.m0 = k;
        if (L.rank[k] == 1) L.m1 = k;
        if (L.rank[k] == 0) L.m2 = k;
    }
    // (volumes of 8 TB and more have more tiles than a launch has blocks)
    if ((L.vn[L.m1] + FPT_TILE_1 - 1) / FPT_TILE_1 > MAX_GRID_Y || L.vn[L.m0] > MAX_GRID_Y ||
        std::max(column_blocks(L, 0), std::max(column_blocks(L, 1), column_blocks(L, 2))) > INT_MAX)
        return kk_fail(KK_ERR_UNSUPPORTED, "%s: volume too large for one launch", who);
    L.proj = (const float*)proj->data;
    L.table = proj->table;
    L.rows = (int)proj->rows;
    L.cols = (int)proj->cols;
    L.angles = angles;
    for (int k = 0; k < 9; ++k) L.os[k] = out_scale[k];
    L.slab = slab > 0 ? slab : FP_SLAB;
    for (int k = 0; k < 3; ++k) {
        const float e = slab_drift(L.slab, L.vn, k);
        L.margin[k] = 0.5f + e;
        L.min_step[k] = std::max(0.0625f, 2.f * e);
    }
    const int n = (int)proj->n_angles;
    const int ck = (int)std::min<int64_t>(chunk, n);
    L.ray_ab = (float4*)work;
    L.ray_pc = work + 4 * (int64_t)ck * per;
    const cudaStream_t st = (cudaStream_t)stream;
    const dim3 block(FPT_TILE_2, FPT_TILE_1);
    const dim3 grid((L.vn[L.m2] + FPT_TILE_2 - 1) / FPT_TILE_2, (L.vn[L.m1] + FPT_TILE_1 - 1) / FPT_TILE_1, L.vn[L.m0]);
    const bool tex8 = interp == KK_INTERP_TEX8;
    for (int r0 = 0; r0 < n; r0 += ck) {
        L.rec0 = r0;
        L.nrec = std::min(ck, n - r0);
        const int first = (r0 > 0 || additive) ? 1 : 0;
        const int64_t rays = (int64_t)L.nrec * per;
        fpt_rays_kernel<<<(unsigned)((rays + 255) / 256), 256, 0, st>>>(L);
        // every voxel is written by the first column pass (even where no
        // ray of its axis touches it), the later passes and the per-voxel
        // gather of the remaining records add
        for (int A = 0; A < 3; ++A) {
            L.accumulate = A > 0 ? 1 : first;
            launch_column_pass(L, A, tex8, st);
        }
        L.accumulate = 1;
        if (tex8)
            fpt_gather_kernel<true><<<grid, block, 0, st>>>(L);
        else
            fpt_gather_kernel<false><<<grid, block, 0, st>>>(L);
    }
    return kk_check_launch(who);
}
