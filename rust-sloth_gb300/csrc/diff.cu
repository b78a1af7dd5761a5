// diff.cu -- differentiable shading of a rendered batch and its hand-written adjoint.
//
// There is no counterpart in the reference: sloth only picks a character from the
// screen-space normal's z (src/rasterizer.rs:76).  The image defined here reduces to that
// quantity: for the winning sample (x, y) of a depth cell (the render's visibility, held
// fixed) and its triangle A, B, C in screen space,
//     rgb = (b0*c(A) + b1*c(B) + b2*c(C)) * clamp(n_hat . L, 0, 1)
// with b_i = w_i / orient(A,B,C) the barycentric weights of (x, y), c the f32 vertex
// colours, n_hat = unit((B-A) x (C-A)) and L the light direction in screen space; with
// L = (0,0,1) the shade factor is the reference's normal z.
//
// Both passes read a winner's triangle from its record (the render's transformed x and y,
// and the two depth differences the normal needs) and its colours by the mesh's indices.
//
// The backward pass walks the cells in sample order, so that the lanes of a warp hold
// consecutive samples of one row: their winners are mostly runs of one triangle.  For a
// fixed triangle everything the gradients need is affine in the sample, so a run
// contributes through two moments of the image gradient, sum(g) and sum(g*(x - x_head)):
// a segmented warp reduction of those six values, after which the run's head lane alone
// evaluates the triangle once.  The head maps the screen-space position gradients to
// object space through the draw's matrix (object = M3^T * screen; the vertex transform has
// no divide) and adds them, and the colour gradients, to the mesh's vertices.  The light
// gradient is reduced per block.
#include "diff_kernels.h"
#include "resolve_common.cuh"

namespace sloth {

namespace {

constexpr uint32_t kNoTri = 0xffffffffu;
constexpr int kDiffThreads = 256;
// A gradient whose components come to this or more, or are not finite, keeps to its own sample:
// the sums of a run of 32 (up to 496 times it) stay below the largest float.
constexpr float kRunMax = 1e35f;

struct Hit {
    uint32_t tri;      // frame-local triangle (draw order), kNoTri when none
    int32_t x, y;      // sample point
};

// Winning sample of depth cell id of frame f, decoded from its depth key.
__device__ __forceinline__ Hit hit_from_key(const BatchFrame &f, uint64_t id)
{
    const int r = (int)(id / f.g.w), cc = (int)(id - (uint64_t)r * f.g.w);
    const uint64_t key = key_at(f.g, f.fb, r, cc);
    if (key == kEmptyKey) return Hit{kNoTri, 0, 0};
    const uint32_t lo = (uint32_t)key;
    if (lo & 1u) return Hit{lo >> 1, cc >> 1, r};
    return Hit{lo >> 1, (cc + f.g.w) >> 1, r - 1};
}

__device__ __forceinline__ uint2 pack_hit(const Hit &h)
{
    return make_uint2(h.tri, (uint32_t)h.x | ((uint32_t)h.y << 16));
}

__device__ __forceinline__ Hit unpack_hit(uint2 v)
{
    return Hit{v.x, (int32_t)(v.y & 0xffffu), (int32_t)(v.y >> 16)};
}

// The draw of frame-local triangle `tri`: the last of the frame's draws whose first
// triangle is <= tri.
__device__ __forceinline__ uint32_t draw_of(const BatchDev &b, const BatchFrame &f, uint32_t tri)
{
    uint32_t lo = f.first_draw, hi = f.first_draw + f.ndraws - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (b.draws[mid].local_base <= tri) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// A winner's triangle: x and y of the transformed vertices, z relative to the first (only
// differences of z are used), and its mesh vertex ids.
struct Tri {
    float3 A, B, C;
    uint32_t i0, i1, i2;
};

// Rows 0, 1 and 5 of a winner's record (the rest is not written for every path).
struct TriRows {
    float4 q0, q1, q5;
};
__device__ __forceinline__ TriRows load_rows(const BatchFrame &f, uint32_t tri)
{
    const float4 *p = reinterpret_cast<const float4 *>(f.fb.records + tri);
    return TriRows{__ldg(p), __ldg(p + 1), __ldg(p + 5)};
}

__device__ __forceinline__ void load_ids(const BatchDraw &d, uint32_t t, Tri &g)
{
    if (d.mesh.idx) {
        g.i0 = __ldg(d.mesh.idx + 3 * (size_t)t);
        g.i1 = __ldg(d.mesh.idx + 3 * (size_t)t + 1);
        g.i2 = __ldg(d.mesh.idx + 3 * (size_t)t + 2);
    } else {
        g.i0 = 3 * t;
        g.i1 = 3 * t + 1;
        g.i2 = 3 * t + 2;
    }
}

__device__ __forceinline__ void set_vertices(const TriRows &r, Tri &g)
{
    g.A = make_float3(r.q0.x, r.q0.y, 0.0f);
    g.B = make_float3(r.q0.z, r.q0.w, r.q5.y);
    g.C = make_float3(r.q1.x, r.q1.y, r.q5.z);
}

__device__ __forceinline__ float orient2(float ax, float ay, float bx, float by, float cx, float cy)
{
    return (bx - ax) * (cy - ay) - (by - ay) * (cx - ax);
}
__device__ __forceinline__ float3 sub3(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b)
{
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 ld3(const float *p)
{
    return make_float3(__ldg(p), __ldg(p + 1), __ldg(p + 2));
}

struct Shade {
    bool ok;                 // non-degenerate triangle
    float b0, b1, b2, o;     // barycentrics, orient(A,B,C)
    float3 c0, c1, c2;       // vertex colours
    float3 col;              // interpolated colour
    float3 nhat;
    float nlen, ndl, s;      // |n|, n_hat . L, clamp(n_hat . L, 0, 1)
};

__device__ __forceinline__ Shade shade_at(const Tri &g, float px, float py, const float *vrgb, float3 L)
{
    Shade e;
    e.o = orient2(g.A.x, g.A.y, g.B.x, g.B.y, g.C.x, g.C.y);
    const float3 n = cross3(sub3(g.B, g.A), sub3(g.C, g.A));
    e.nlen = sqrtf(dot3(n, n));
    e.ok = e.o != 0.0f && e.nlen > 0.0f && isfinite(e.o) && isfinite(e.nlen);
    if (!e.ok) return e;
    const float io = 1.0f / e.o;
    e.b0 = orient2(g.B.x, g.B.y, g.C.x, g.C.y, px, py) * io;
    e.b1 = orient2(g.C.x, g.C.y, g.A.x, g.A.y, px, py) * io;
    e.b2 = orient2(g.A.x, g.A.y, g.B.x, g.B.y, px, py) * io;
    e.c0 = ld3(vrgb + 3 * (size_t)g.i0);
    e.c1 = ld3(vrgb + 3 * (size_t)g.i1);
    e.c2 = ld3(vrgb + 3 * (size_t)g.i2);
    e.col = make_float3(e.b0 * e.c0.x + e.b1 * e.c1.x + e.b2 * e.c2.x, e.b0 * e.c0.y + e.b1 * e.c1.y + e.b2 * e.c2.y,
                        e.b0 * e.c0.z + e.b1 * e.c1.z + e.b2 * e.c2.z);
    const float il = 1.0f / e.nlen;
    e.nhat = make_float3(n.x * il, n.y * il, n.z * il);
    e.ndl = dot3(e.nhat, L);
    e.s = fminf(fmaxf(e.ndl, 0.0f), 1.0f);
    return e;
}

// The shaded colour of a hit (0 without one, or for a degenerate triangle).
__device__ __forceinline__ float3 shade_hit(const Hit &h, const TriRows &rows, Tri &g, const float *vrgb, float3 L)
{
    if (h.tri == kNoTri) return make_float3(0.0f, 0.0f, 0.0f);
    set_vertices(rows, g);
    const Shade e = shade_at(g, (float)h.x, (float)h.y, vrgb, L);
    return e.ok ? make_float3(e.col.x * e.s, e.col.y * e.s, e.col.z * e.s) : make_float3(0.0f, 0.0f, 0.0f);
}

// A block shades kDiffChunk depth cells.  Even widths go by pairs of cells, kPairs of them
// per thread at once: the odd cell of a pair never has a winner, so no lane idles on one,
// and a pair's image and visibility go out in 8- and 16-byte stores when vec says they are
// aligned.  Bound by the latency of key -> record and ids -> colours, which the independent
// pairs overlap.
constexpr int kPairs = 2;
__global__ void __launch_bounds__(kDiffThreads)
batch_shade_kernel(BatchDev b, const int2 *__restrict__ blocks, const float *__restrict__ vrgb,
                   const float *__restrict__ light, float *__restrict__ rgb, uint2 *__restrict__ vis, int vec)
{
    const int2 blk = blocks[blockIdx.x];
    const BatchFrame &f = b.frames[blk.x];
    const uint64_t nz = (uint64_t)f.g.w * f.g.h;
    const uint64_t end = min(nz, (uint64_t)blk.y + kDiffChunk);
    const float3 L = ld3(light);
    if (!(f.g.w & 1)) {
        const bool v = vec && !(f.z_off & 1);
        for (uint64_t c = (uint64_t)blk.y + 2 * threadIdx.x; c < end; c += 2 * kPairs * kDiffThreads) {
            Hit h[kPairs];
            TriRows rows[kPairs];
            Tri g[kPairs];
#pragma unroll
            for (int j = 0; j < kPairs; ++j) {
                const uint64_t cj = c + 2 * j * kDiffThreads;
                h[j] = cj < end ? hit_from_key(f, cj) : Hit{kNoTri, 0, 0};
            }
#pragma unroll
            for (int j = 0; j < kPairs; ++j)
                if (h[j].tri != kNoTri) {
                    const BatchDraw &d = b.draws[draw_of(b, f, h[j].tri)];
                    rows[j] = load_rows(f, h[j].tri);
                    load_ids(d, h[j].tri - d.local_base, g[j]);
                }
#pragma unroll
            for (int j = 0; j < kPairs; ++j) {
                const uint64_t cj = c + 2 * j * kDiffThreads;
                if (cj >= end) continue;
                const float3 out = shade_hit(h[j], rows[j], g[j], vrgb, L);
                const uint64_t gc = f.z_off + cj;
                const uint2 hv = pack_hit(h[j]), none = pack_hit(Hit{kNoTri, 0, 0});
                float *o = rgb + 3 * gc;
                if (v) {
                    float2 *o2 = reinterpret_cast<float2 *>(o);
                    o2[0] = make_float2(out.x, out.y);
                    o2[1] = make_float2(out.z, 0.0f);
                    o2[2] = make_float2(0.0f, 0.0f);
                    if (vis) *reinterpret_cast<uint4 *>(vis + gc) = make_uint4(hv.x, hv.y, none.x, none.y);
                } else {
                    o[0] = out.x;
                    o[1] = out.y;
                    o[2] = out.z;
                    o[3] = o[4] = o[5] = 0.0f;
                    if (vis) {
                        vis[gc] = hv;
                        vis[gc + 1] = none;
                    }
                }
            }
        }
        return;
    }
    for (uint64_t c = (uint64_t)blk.y + threadIdx.x; c < end; c += kDiffThreads) {
        const uint64_t gc = f.z_off + c;
        const Hit h = hit_from_key(f, c);
        TriRows rows;
        Tri g;
        if (h.tri != kNoTri) {
            const BatchDraw &d = b.draws[draw_of(b, f, h.tri)];
            rows = load_rows(f, h.tri);
            load_ids(d, h.tri - d.local_base, g);
        }
        const float3 out = shade_hit(h, rows, g, vrgb, L);
        if (vis) vis[gc] = pack_hit(h);
        rgb[3 * gc + 0] = out.x;
        rgb[3 * gc + 1] = out.y;
        rgb[3 * gc + 2] = out.z;
    }
}

// v summed over the lanes [lane, seg_end) of the caller's run (all 32 lanes call).
__device__ __forceinline__ float run_sum(float v, int lane, int seg_end)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float o = __shfl_down_sync(0xffffffffu, v, d);
        if (lane + d < seg_end) v += o;
    }
    return v;
}

__device__ __forceinline__ void red_add(float *p, float a) { asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(a) : "memory"); }
__device__ __forceinline__ void red_add2(float *p, float a, float b)
{
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b) : "memory");
}

// a, b, c added to p[0..2]: a pair at its 8-byte boundary and a single, whichever comes first.
__device__ __forceinline__ void red_add3(float *p, float a, float b, float c)
{
    if (reinterpret_cast<uintptr_t>(p) & 7u) {
        red_add(p, a);
        red_add2(p + 1, b, c);
    } else {
        red_add2(p, a, b);
        red_add(p + 2, c);
    }
}

// One run's gradients, from its triangle at the head sample (px, py) and the moments of the
// image gradient over the run: S0 = sum(g), S1 = sum(g*(x - px)).
__device__ __forceinline__ void run_backward(const BatchDev &b, const BatchFrame &f, uint32_t tri, float px, float py,
                                             float3 S0, float3 S1, const float *vrgb, float3 L, float *gpos,
                                             float *gcol, float &gl0, float &gl1, float &gl2)
{
    const uint32_t draw = draw_of(b, f, tri);
    const BatchDraw &d = b.draws[draw];
    const TriRows rows = load_rows(f, tri);
    Tri g;
    load_ids(d, tri - d.local_base, g);
    set_vertices(rows, g);
    const Shade e = shade_at(g, px, py, vrgb, L);
    if (!e.ok) return;
    const float3 A = g.A, B = g.B, C = g.C;
    const float io = 1.0f / e.o;
    // T_i = sum(g*b_i): b_i is affine in x along the row
    const float db0 = (B.y - C.y) * io, db1 = (C.y - A.y) * io, db2 = (A.y - B.y) * io;
    const float3 T0 = make_float3(S0.x * e.b0 + S1.x * db0, S0.y * e.b0 + S1.y * db0, S0.z * e.b0 + S1.z * db0);
    const float3 T1 = make_float3(S0.x * e.b1 + S1.x * db1, S0.y * e.b1 + S1.y * db1, S0.z * e.b1 + S1.z * db1);
    const float3 T2 = make_float3(S0.x * e.b2 + S1.x * db2, S0.y * e.b2 + S1.y * db2, S0.z * e.b2 + S1.z * db2);
    const float G = dot3(e.c0, T0) + dot3(e.c1, T1) + dot3(e.c2, T2);   // sum(g . col)
    if (gcol) {
        const float3 T[3] = {T0, T1, T2};
        const uint32_t ids[3] = {g.i0, g.i1, g.i2};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float x = e.s * T[q].x, y = e.s * T[q].y, z = e.s * T[q].z;
            if (x != 0.0f || y != 0.0f || z != 0.0f) red_add3(gcol + 3 * (size_t)ids[q], x, y, z);
        }
    }
    const float gs = (e.ndl > 0.0f && e.ndl < 1.0f) ? G : 0.0f;
    gl0 += gs * e.nhat.x;
    gl1 += gs * e.nhat.y;
    gl2 += gs * e.nhat.z;
    if (!gpos) return;
    // barycentrics: b_i = w_i / o, d b_i = (d w_i - b_i d o) / o; g_i = sum of the gradient of
    // b_i over the run, h_i the same times x - px
    const float g0 = e.s * dot3(e.c0, S0), g1 = e.s * dot3(e.c1, S0), g2 = e.s * dot3(e.c2, S0);
    const float h0 = e.s * dot3(e.c0, S1), h1 = e.s * dot3(e.c1, S1), h2 = e.s * dot3(e.c2, S1);
    const float k = e.s * G;
    float v[9];
    v[0] = io * (g1 * (py - C.y) + g2 * (B.y - py) - k * (B.y - C.y));
    v[1] = io * (g1 * (C.x - px) - h1 + (g2 * (px - B.x) + h2) - k * (C.x - B.x));
    v[2] = 0.0f;
    v[3] = io * (g0 * (C.y - py) + g2 * (py - A.y) - k * (C.y - A.y));
    v[4] = io * (g0 * (px - C.x) + h0 + (g2 * (A.x - px) - h2) - k * (A.x - C.x));
    v[5] = 0.0f;
    v[6] = io * (g0 * (py - B.y) + g1 * (A.y - py) - k * (A.y - B.y));
    v[7] = io * (g0 * (B.x - px) - h0 + (g1 * (px - A.x) + h1) - k * (B.x - A.x));
    v[8] = 0.0f;
    if (gs != 0.0f) {
        // s = n_hat . L, n_hat = n / |n|, n = (B-A) x (C-A)
        const float il = 1.0f / e.nlen;
        const float3 gn = make_float3(gs * (L.x - e.ndl * e.nhat.x) * il, gs * (L.y - e.ndl * e.nhat.y) * il,
                                      gs * (L.z - e.ndl * e.nhat.z) * il);
        const float3 ge1 = cross3(sub3(C, A), gn), ge2 = cross3(gn, sub3(B, A));
        v[3] += ge1.x; v[4] += ge1.y; v[5] += ge1.z;
        v[6] += ge2.x; v[7] += ge2.y; v[8] += ge2.z;
        v[0] -= ge1.x + ge2.x; v[1] -= ge1.y + ge2.y; v[2] -= ge1.z + ge2.z;
    }
    const Mat4 &M = b.mats[draw];
    const uint32_t ids[3] = {g.i0, g.i1, g.i2};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const float sx = v[3 * q], sy = v[3 * q + 1], sz = v[3 * q + 2];
        if (sx != 0.0f || sy != 0.0f || sz != 0.0f)
            red_add3(gpos + 3 * (size_t)ids[q], M.m[0] * sx + M.m[4] * sy + M.m[8] * sz,
                     M.m[1] * sx + M.m[5] * sy + M.m[9] * sz, M.m[2] * sx + M.m[6] * sy + M.m[10] * sz);
    }
}

// A block takes the winners of kDiffChunk depth cells in sample order: of an even-width
// frame the even cells (the others never have one), of an odd-width frame each row's even
// columns, which the row's own samples write, then its odd ones.
__global__ void __launch_bounds__(kDiffThreads)
batch_shade_backward_kernel(BatchDev b, const int2 *__restrict__ blocks, const float *__restrict__ vrgb,
                            const float *__restrict__ light, const float *__restrict__ grad_rgb,
                            const uint2 *__restrict__ vis, float *__restrict__ gpos, float *__restrict__ gcol,
                            float *__restrict__ glight)
{
    __shared__ float sl[3][kDiffThreads / 32];
    const int2 blk = blocks[blockIdx.x];
    const BatchFrame &f = b.frames[blk.x];
    const int w = f.g.w;
    const uint64_t nz = (uint64_t)w * f.g.h;
    const float3 L = ld3(light);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool even = !(w & 1);
    const uint32_t slots = even ? kDiffChunk / 2 : kDiffChunk;
    float gl0 = 0.0f, gl1 = 0.0f, gl2 = 0.0f;
    // warp-uniform trip count: every lane takes part in the run reductions
    for (uint32_t i = threadIdx.x; i < slots; i += kDiffThreads) {
        uint64_t id = (uint64_t)blk.y + (even ? 2 * i : i);
        if (!even && id < nz) {
            const uint64_t r = id / w;
            const uint32_t k = (uint32_t)(id - r * w), half = (uint32_t)(w + 1) / 2;
            id = r * w + (k < half ? 2 * k : 2 * (k - half) + 1);
        }
        Hit h{kNoTri, 0, 0};
        float3 go = make_float3(0.0f, 0.0f, 0.0f);
        if (id < nz) {
            h = vis ? unpack_hit(vis[f.z_off + id]) : hit_from_key(f, id);
            if (h.tri != kNoTri) {
                go = ld3(grad_rgb + 3 * (f.z_off + id));
                if (go.x == 0.0f && go.y == 0.0f && go.z == 0.0f) h.tri = kNoTri;
            }
        }
        if (!__any_sync(0xffffffffu, h.tri != kNoTri)) continue;
        // a run: one triangle over consecutive samples of a row.  A gradient that is not
        // finite, or would overflow the run's sums, keeps to its own sample, so that it
        // reaches what it reached by itself.
        const bool wild = h.tri != kNoTri && !(fabsf(go.x) + fabsf(go.y) + fabsf(go.z) < kRunMax);
        const bool split = __any_sync(0xffffffffu, wild);
        const uint32_t pt = __shfl_up_sync(0xffffffffu, h.tri, 1);
        const int pxl = __shfl_up_sync(0xffffffffu, h.x, 1), pyl = __shfl_up_sync(0xffffffffu, h.y, 1);
        const bool head = lane == 0 || split || pt != h.tri || pyl != h.y || pxl + 1 != h.x;
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        const unsigned above = lane == 31 ? 0u : (heads & ~((2u << lane) - 1u));
        const int seg_end = above ? __ffs(above) - 1 : 32;
        const int first = 31 - __clz(heads & ((2u << lane) - 1u));   // the run's head lane
        const float j = (float)(lane - first);
        float m[6] = {go.x, go.y, go.z, 0.0f, 0.0f, 0.0f};
        if (lane != first) {
            m[3] = go.x * j;
            m[4] = go.y * j;
            m[5] = go.z * j;
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) m[q] = run_sum(m[q], lane, seg_end);
        if (head && h.tri != kNoTri)
            run_backward(b, f, h.tri, (float)h.x, (float)h.y, make_float3(m[0], m[1], m[2]),
                         make_float3(m[3], m[4], m[5]), vrgb, L, gpos, gcol, gl0, gl1, gl2);
    }
#pragma unroll
    for (int dd = 16; dd > 0; dd >>= 1) {
        gl0 += __shfl_xor_sync(0xffffffffu, gl0, dd);
        gl1 += __shfl_xor_sync(0xffffffffu, gl1, dd);
        gl2 += __shfl_xor_sync(0xffffffffu, gl2, dd);
    }
    if (lane == 0) {
        sl[0][wid] = gl0;
        sl[1][wid] = gl1;
        sl[2][wid] = gl2;
    }
    block_sync();
    if (glight && threadIdx.x < 3) {
        float s = 0.0f;
        for (int q = 0; q < kDiffThreads / 32; ++q) s += sl[threadIdx.x][q];
        if (s != 0.0f) atomicAdd(glight + threadIdx.x, s);
    }
}

__global__ void __launch_bounds__(kDiffThreads) clear_gradients_kernel(float *gpos, float *gcol, float *glight, uint64_t n)
{
    const uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = i0; i < n; i += step) {
        if (gpos) gpos[i] = 0.0f;
        if (gcol) gcol[i] = 0.0f;
    }
    if (glight && i0 < 3) glight[i0] = 0.0f;
}

}  // namespace

cudaError_t launch_clear_gradients(float *gpos, float *gcol, float *glight, uint32_t nvert, cudaStream_t s)
{
    const uint64_t n = 3ull * nvert, most = 8ull * (uint64_t)device_sm_count();
    const uint64_t blocks = (n + kDiffThreads - 1) / kDiffThreads;
    clear_gradients_kernel<<<(unsigned)(blocks < 1 ? 1 : blocks < most ? blocks : most), kDiffThreads, 0, s>>>(gpos, gcol,
                                                                                                         glight, n);
    return cudaGetLastError();
}

cudaError_t launch_batch_shade(const BatchDev &b, const int2 *blocks, uint32_t nblocks, const float *vrgb,
                               const float *light, float *rgb, uint2 *vis, cudaStream_t s)
{
    if (!nblocks) return cudaSuccess;
    const int vec = (reinterpret_cast<uintptr_t>(rgb) & 7u) == 0;   // vis starts an allocation
    batch_shade_kernel<<<nblocks, kDiffThreads, 0, s>>>(b, blocks, vrgb, light, rgb, vis, vec);
    return cudaGetLastError();
}

cudaError_t launch_batch_shade_backward(const BatchDev &b, const int2 *blocks, uint32_t nblocks, const float *vrgb,
                                        const float *light, const float *grad_rgb, const uint2 *vis, float *gpos,
                                        float *gcol, float *glight, cudaStream_t s)
{
    if (!nblocks) return cudaSuccess;
    batch_shade_backward_kernel<<<nblocks, kDiffThreads, 0, s>>>(b, blocks, vrgb, light, grad_rgb, vis, gpos, gcol,
                                                                 glight);
    return cudaGetLastError();
}

}  // namespace sloth
