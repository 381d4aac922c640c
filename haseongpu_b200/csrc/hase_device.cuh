// hase_device.cuh -- device-side building blocks of the phi-ASE hot path:
// Philox4x32-10, the packed prism-mesh view, and the FP32 prism walk.
//
// The walk follows the legacy HASEonGPU backward method (rays from a start
// point in a prism to the sample point, crossing triangle edges through the
// neighbour table and z levels), here parametrised by the remaining distance s
// to the (image) sample point, p(s) = S + s*u, walked from s = |start - S|
// down to 0.  The exits of a prism are the largest crossing parameters below
// s: edges (2-D lines n.x = c whose outward normal points against the motion)
// and the level planes z = k*h, all relative to the sample so that the last
// prism (the one touching the sample point) ends the walk at s = 0 exactly.
// Gain anchor: g = N_tot (beta (sigmaE + sigmaA) - sigmaA), cladding
// g = -claddingAbsorption (include/kernels/forward/rayWalk.hpp:170-182).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace hase {

constexpr uint32_t kTagRay = 0u;
constexpr uint32_t kTagMap = 1u;
constexpr uint32_t kTagFar = 2u;  // far rays of the local proposal: Philox counter word 3
constexpr uint32_t kWeylStep = 0x9E3779B9u;  // 2^32 / golden ratio: the rays' wavelength sequence step
constexpr int kMaxSteps = 10000;  // bounded walk (include/kernels/forward/policyRay.hpp:386)

// ---------------------------------------------------------------- Philox ----
// Philox4x32-10, Salmon, Moraes, Dror, Shaw, "Parallel Random Numbers: As Easy
// as 1, 2, 3", SC'11: 10 rounds of two 32x32->64 multiplies with a Weyl key
// schedule.
struct Philox4 {
    uint32_t x, y, z, w;
};

__host__ __device__ __forceinline__ Philox4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                                          uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int round = 0; round < 10; ++round) {
        if (round > 0) {
            k0 += 0x9E3779B9u;
            k1 += 0xBB67AE85u;
        }
#ifdef __CUDA_ARCH__
        const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
#else
        const uint64_t p0 = uint64_t(0xD2511F53u) * c0, p1 = uint64_t(0xCD9E8D57u) * c2;
        const uint32_t hi0 = uint32_t(p0 >> 32), lo0 = uint32_t(p0);
        const uint32_t hi1 = uint32_t(p1 >> 32), lo1 = uint32_t(p1);
#endif
        const uint32_t n0 = hi1 ^ c1 ^ k0;
        const uint32_t n2 = hi0 ^ c3 ^ k1;
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
    }
    return Philox4{c0, c1, c2, c3};
}

// 24-bit uniform in (0,1): (k + 1/2) 2^-24, exact in FP32.
__device__ __forceinline__ float unit24(uint32_t k24) { return (float(k24) + 0.5f) * (1.0f / 16777216.0f); }

// ------------------------------------------------------------ mesh view ----
// Packed per-triangle walk record, 3 x float4 = 48 B:
//   r0 = (nx0, ny0, c0, nx1), r1 = (ny1, c1, nx2, ny2), r2 = (c2, nb0, nb1, nb2)
// with nb_e = (neighbour << 2 | entry edge in the neighbour) as int bits, -1 at
// the mesh boundary.  Start-point record, 2 x float4 = 32 B:
//   g0 = (ax, ay, bx-ax, by-ay), g1 = (cx-ax, cy-ay, area, 0); centroid separate.
struct MeshView {
    const float4* tri;       // [T][3]
    const float4* win;       // [T][4]: the walks' edge windows (windowSlot)
    const float4* geo;       // [T][2]
    const int4* verts;       // [T] point ids of the triangle's vertices (w unused)
    const float2* centroid;  // [T]
    // [T][layers] the ray walk's value of each prism (WalkMode): g, or beta with
    // NaN in cladding prisms.  Triangle-major: the rays of a warp cross the same
    // triangles at different heights, so their reads share a column's one or two
    // lines; layer-major they were up to one line per lane.
    const float* walkTab;
    const float* gTab;       // [P] g of each prism for the solve's averaged (A, B) (a monochromatic solve: its pair)
    const float* srcBeta;    // [P] beta (source weight)
    const float2* points;    // [Np]
    const float* reflect;    // [T][2] or nullptr
    uint32_t T, layers, P, Np;
    uint32_t divTm, divTs;   // floor(p / T) = (p * divTm) >> divTs for p < 2^31 (invariantDivisor)
    uint32_t divNpm, divNps; // the same for division by Np
    float h;                 // level spacing
    float cladAbs;           // claddingAbsorption
    float tolEnd;            // |s| below which the target is reached
    float tirCos2[2];        // total internal reflection when uz^2 <= tirCos2[surface]
};

// The walks' edge windows.  An edge is one float4 (nx, ny, c, code), a
// triangle holds its edges in the four slots e0 e1 e2 e0, and a window is the
// pair of slots a ray that entered through the third edge can leave by:
// entered through e0: slots 1, 2; e1: slots 2, 3; e2: slots 0, 1.  code is the
// window on the other side, 4 neighbour + its first slot, so that one index,
// loaded with the edge, is the next triangle, its records' address and the
// edge that is left out.  The three-edge records cost a third edge test and a
// third 16-byte load per triangle for an edge that never is the exit.
// A mesh-boundary edge is (0, 0, 1, 0): its exit parameter is negative whatever
// the ray, so it is never chosen, and its code is a valid index.
__host__ __device__ __forceinline__ uint32_t windowSlot(uint32_t entryEdge) { return entryEdge == 2 ? 0u : entryEdge + 1u; }

// Layer of prism index p < 2^31 (p = t + layer T): an exact multiply-shift
// instead of a 32-bit division by the runtime T.
__device__ __forceinline__ uint32_t prismLayer(const MeshView& m, uint32_t p) {
    return uint32_t((uint64_t(p) * m.divTm) >> m.divTs);
}

// Level of sample index s < 2^31 (s = point + level Np), by multiply-shift.
__device__ __forceinline__ uint32_t sampleLevel(const MeshView& m, uint32_t s) {
    return uint32_t((uint64_t(s) * m.divNpm) >> m.divNps);
}

// Unfolded integer level of the image of sample level ls for reflection slice.
__device__ __forceinline__ int imageLevel(int ls, int layers, uint32_t slice) {
    switch (slice) {
        case 1: return -ls;                 // bottom
        case 2: return 2 * layers - ls;     // top
        case 3: return ls - 2 * layers;     // bottom, then top
        case 4: return ls + 2 * layers;     // top, then bottom
        default: return ls;
    }
}

__device__ __forceinline__ int expectedReflections(uint32_t slice) { return slice == 0 ? 0 : (slice <= 2 ? 1 : 2); }

// Legacy reflectivity index t*2 + surface (include/core/mesh.hpp:301-332), with
// total internal reflection above the critical angle.
__device__ __forceinline__ float reflectFactor(const MeshView& m, uint32_t t, int surf, float uz) {
    if (uz * uz <= m.tirCos2[surf]) return 1.0f;
    return m.reflect ? __ldg(m.reflect + 2 * t + surf) : 0.0f;
}

// One ray in flight.  The walk runs in the unfolded z coordinate (reflection
// images); `row` is the physical layer of the current unfolded layer and
// `rstep` the step to the next physical layer toward the image point, +1 or -1
// (it flips at every reflection), so no division or modulo is needed per
// crossing.
struct Ray {
    uint32_t w;     // edge window: 4 triangle + first slot (MeshView::win)
    int row;        // physical layer of the current unfolded layer
    int rstep;      // +1 / -1
    int reflLeft;   // reflections the slice still implies
    int steps;      // triangles left minus the first zl: with the current zl, the crossings so far (raySteps)
    float s;        // remaining distance to the image point
    float G;        // accumulated ln(gain) for the pair (A, B), including reflection factors
    float A, B;     // g = beta*A - B: the walk's reference pair
    float Jb;       // integral of beta dl over gain prisms (beta walks)
    float Lc;       // path length in cladding prisms (kWalkBeta)
    float D;        // path length, start to image point
    float ux, uy, uz;
    // the current layer's exit plane lies at s = zl hOverUz: zl is the plane's
    // unfolded level offset from the image point (a small integer, exact in
    // float) and hOverUz = h / uz, both times the layer step toward the image
    // (-1 when uz > 0, else +1), so that zl grows by 1 per plane
    float hOverUz;
    float zl;
};

// Crossings so far: triangles left plus level planes and reflections.
__device__ __forceinline__ int raySteps(const Ray& r) { return r.steps + int(r.zl); }

enum StepResult { kContinue = 0, kDone = 1, kDropped = 2 };

// How a walk obtains the gain coefficient g of the current prism.  The beta
// walks also keep the path integrals that make the gain of every wavelength
// (A_l, B_l) follow from the reference pair's: ln G_l = G + (A_l - A) Jb -
// (B_l - B)(D - Lc), so a ray's gain is known for the whole spectrum
// (rayMeanGain); for the reference pair it is G itself, bit for bit as the
// table walk gives it.
enum WalkMode {
    kWalkBeta = 0,         // m.walkTab holds beta; cladding prisms (NaN beta) add to Lc
    kWalkTable = 1,        // m.walkTab holds g (a monochromatic solve: the table is built for its pair)
    kWalkBetaNoClad = 2,   // as kWalkBeta for a medium without cladding prisms (beta is never NaN)
};

// Reciprocal with the hardware approximation (1 ulp; subnormal inputs give inf).
__device__ __forceinline__ float rcpApprox(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Initialise a ray from the start point, given as its offset (dx, dy, dz)
// from the image point (Sx, Sy, kImg*h), in physical layer `layer`.
// Returns |start - image|^2.
__device__ __forceinline__ float initRay(Ray& r, uint32_t t, int layer, float dx, float dy, float dz, int kImg,
                                         uint32_t slice, float A, float B, const MeshView& m) {
    const float h = m.h;
    if (dz == 0.0f) dz = 1e-6f * h;  // a ray inside a level plane: nudge it off the plane
    const float D2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float D = sqrtf(D2);
    const float inv = 1.0f / D;
    r.row = layer;
    r.reflLeft = expectedReflections(slice);
    r.s = D;
    r.G = 0.0f;
    r.Jb = 0.0f;
    r.Lc = 0.0f;
    r.D = D;
    r.ux = dx * inv;
    r.uy = dy * inv;
    r.uz = dz * inv;
    // moving toward the image: down (layer step -1) when uz > 0, up (+1) otherwise
    const float hu = h * rcpApprox(r.uz);
    r.hOverUz = r.uz > 0.0f ? -hu : hu;
    const int zl0 = r.uz > 0.0f ? kImg - layer : layer + 1 - kImg;
    r.zl = float(zl0);
    r.steps = -zl0;
    r.rstep = r.uz > 0.0f ? -1 : 1;
    r.A = A;
    r.B = B;
    // the first window leaves out an edge the ray does not move out through
    // (one of the three always is; a boundary edge's zero normal counts too)
    const float2* e = reinterpret_cast<const float2*>(m.win + 4 * size_t(t));
    const float2 e0 = __ldg(e), e1 = __ldg(e + 2);
    const bool out0 = -fmaf(e0.x, r.ux, e0.y * r.uy) > 0.0f, out1 = -fmaf(e1.x, r.ux, e1.y * r.uy) > 0.0f;
    r.w = 4 * t + (!out0 ? 1u : (!out1 ? 2u : 0u));
    return D2;
}

// One segment of length len in a prism whose table value (kWalkTable: g) or
// beta (NaN: cladding) is gb.
template <int WALK>
__device__ __forceinline__ void addSegment(Ray& r, float gb, float len, float cladAbs) {
    if constexpr (WALK == kWalkTable) {
        r.G = fmaf(gb, len, r.G);
    } else if constexpr (WALK == kWalkBetaNoClad) {
        r.G = fmaf(fmaf(gb, r.A, -r.B), len, r.G);
        r.Jb = fmaf(gb, len, r.Jb);
    } else {
        const bool gain = gb == gb;
        r.G = fmaf(gain ? fmaf(gb, r.A, -r.B) : -cladAbs, len, r.G);
        r.Jb = fmaf(gain ? gb : 0.0f, len, r.Jb);
        r.Lc += gain ? 0.0f : len;
    }
}

// ln gain of a finished ray (beta walks) for the pair (A_l, B_l): exact for
// the reference pair.
__device__ __forceinline__ float rayLnGain(const Ray& r, float Al, float Bl) {
    return fmaf(Al - r.A, r.Jb, fmaf(r.B - Bl, r.D - r.Lc, r.G));
}

// The mean over the nL wavelengths (A_l, B_l) of a finished ray's gain
// (beta walks), relative to the reference pair's exact exp(G) (FP64 above
// G = 80): one FP32 exponential per wavelength of the difference of its
// exponent from G, (A_l - A) Jb - (B_l - B)(D - Lc) (bounded by the spread
// of the cross sections along one path; clamped at 80).  One wavelength:
// exp(G), as the table walk.
__device__ __forceinline__ double rayMeanGain(const Ray& r, const float2* spec, uint32_t nL) {
    const double e = r.G < 80.0f ? double(expf(r.G)) : exp(double(r.G));
    if (nL == 1) return e;
    const float Lg = r.D - r.Lc;
    float sum = 0.0f;
    for (uint32_t l = 0; l < nL; ++l) {
        const float2 ab = __ldg(spec + l);
        sum += __expf(fminf(fmaf(ab.x - r.A, r.Jb, (r.B - ab.y) * Lg), 80.0f));
    }
    return e * double(sum) / double(nL);
}

// Exit parameter s = e / d of one window edge for a ray along -u to the sample:
// d the speed out through the edge, e the sample's signed distance from its
// line.  Negative unless the ray moves out: e takes d's sign bit where that is
// set.  (In through an edge, d < 0, the sample lies on its inner side, e < 0,
// up to the rounding of a ray that starts on the edge; without the sign such a
// ray could step back and forth around a vertex.  The 1e-30 gives a ray along
// the edge, d = 0, the same sign.)
__device__ __forceinline__ float edgeExit(const float4& a, float ux, float uy, float Sx, float Sy) {
    const float d = fmaf(-a.x, ux, fmaf(-a.y, uy, -1e-30f));
    const float e = fmaf(a.x, Sx, fmaf(a.y, Sy, -a.z));
    const float es = __uint_as_float(__float_as_uint(e) | (__float_as_uint(d) & 0x80000000u));
    return es * rcpApprox(fabsf(d));
}

// A ray that stepped past a physical bottom or top surface in triangle t:
// back into its layer, reflected (false: more reflections than the slice implies).
__device__ __forceinline__ bool reflectRay(const MeshView& m, Ray& r, uint32_t t) {
    if (r.reflLeft <= 0) return false;
    r.G += __logf(reflectFactor(m, t, r.row < 0 ? 0 : 1, r.uz));
    --r.reflLeft;
    r.row -= r.rstep;
    r.rstep = -r.rstep;
    return true;
}

// Walks up to K triangle columns per call.  Per column: the exit is the later
// crossing of the window's two edges, then the level planes before it.  Once the exit edge is known the next window's records are
// loaded, so that their latency is hidden behind the column's planes.
// The walk is bound by instruction issue and, within it, by the half-rate ALU
// pipe (compares, selects, min/max, integers), so a column is straight-line
// code with as few of those as it can do with:
// - an edge the ray moves in through gets a negative exit parameter, which
//   loses against any exit (edgeExit: two reciprocals on the idle
//   special-function pipe in place of sign tests, a cross multiplication and
//   their selects);
// - no lower clamp: what is not above tolEnd, NaN included, is the target's
//   column, whose end is 0;
// - the segment to the first plane or the exit, and the segment after one
//   plane (of no length where none is crossed: it adds exactly 0), are always
//   computed; only lanes with a second plane in the column enter a loop.  A
//   loop over the planes ran for the whole warp as often as its worst lane
//   needed.
// Crossings are counted by the columns and zl, the step bound is checked once
// per call, and kWalkTable walks a table of g = beta A - B.
// Boundary edges are never exits: the 2-D mesh is convex and the target lies
// in it, so only rounding could route a ray across one.
template <int K = 1, int WALK = kWalkBeta>
__device__ __forceinline__ int stepRay(const MeshView& m, float Sx, float Sy, Ray& r) {
    const float4* win = m.win;
    const auto value = [&](uint32_t t) { return __ldg(m.walkTab + (t * m.layers + uint32_t(r.row))); };
    float4 a = __ldg(win + r.w), b = __ldg(win + r.w + 1);
    // beta (kWalkTable: g) of the current prism, issued with the record so
    // that its latency overlaps the edge tests
    float gb = value(r.w >> 2);
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
        const uint32_t t = r.w >> 2;
        const float q1 = edgeExit(a, r.ux, r.uy, Sx, Sy), q2 = edgeExit(b, r.ux, r.uy, Sx, Sy);
        const float qm = fmaxf(q1, q2);
        const uint32_t code = __float_as_uint(q2 == qm ? b.w : a.w);
        a = __ldg(win + code);
        b = __ldg(win + code + 1);
        const float sEdge = fminf(qm, r.s);
        const float cut = fmaxf(sEdge, m.tolEnd);
        const bool last = !(sEdge > m.tolEnd);  // the target's column: its planes above tolEnd, then the rest of the path
        const float sEnd = last ? 0.0f : sEdge;
        float sz = r.zl * r.hOverUz;
        bool plane = sz > cut;
        float next = plane ? sz : sEnd;
        addSegment<WALK>(r, gb, r.s - next, m.cladAbs);
        r.s = next;
        if (plane) {
            r.row += r.rstep;
            r.zl += 1.0f;
        }
        if (uint32_t(r.row) >= m.layers) {
            if (!reflectRay(m, r, t)) {
                r.steps += k;
                return kDropped;
            }
        }
        if (plane) gb = value(t);
        sz = r.zl * r.hOverUz;
        plane = plane && sz > cut;
        next = plane ? sz : sEnd;
        addSegment<WALK>(r, gb, r.s - next, m.cladAbs);
        r.s = next;
        while (plane) {
            r.row += r.rstep;
            r.zl += 1.0f;
            if (uint32_t(r.row) >= m.layers && !reflectRay(m, r, t)) {
                r.steps += k;
                return kDropped;
            }
            gb = value(t);
            sz = r.zl * r.hOverUz;
            plane = sz > cut;
            next = plane ? sz : sEnd;
            addSegment<WALK>(r, gb, r.s - next, m.cladAbs);
            r.s = next;
        }
        if (last) {
            r.steps += k;
            return kDone;
        }
        r.w = code;
        gb = value(code >> 2);
    }
    r.steps += K;
    // the step bound, once per call: a call walks at most K columns of at most
    // 1 + 3 x layers segments each
    return raySteps(r) >= kMaxSteps ? kDropped : kContinue;
}

// After kDone: a reflection the slice implies but which happens at the target
// itself (a sample on the reflecting surface) is applied in the final triangle.
__device__ __forceinline__ void finishReflections(const MeshView& m, Ray& r) {
    if (r.reflLeft > 0) {
        r.G += __logf(reflectFactor(m, r.w >> 2, r.row + r.rstep < 0 ? 0 : 1, r.uz));
        r.reflLeft = 0;
    }
}

// Near-field start point for a prism (t, l) that touches the image point of
// sample point `pS` (a vertex of triangle t at image level kImg = l or l+1).
// Uniform start points give such prisms an infinite-variance 1/d^2 weight;
// here the direction from the image point is uniform in the prism's solid
// angle (azimuth uniform between the two triangle edges at the vertex,
// sin(elevation) uniform: the prism seen from its vertex is that lune
// segment, solid angle alpha) and the distance is uniform up to the prism
// exit L(Omega).  The density is 1/(alpha L d^2), so the ray weight
// beta G / d^2 / density = beta G alpha L stays bounded.
// Returns false when t does not have pS as a vertex.
__device__ __forceinline__ bool nearFieldStart(const MeshView& m, uint32_t t, int l, int kImg, uint32_t pS,
                                               float2 S, float uAz, float uEl, float uR, float& dx, float& dy,
                                               float& dz, float& alphaL) {
    const int4 v = __ldg(m.verts + t);
    const int iv = v.x == int(pS) ? 0 : (v.y == int(pS) ? 1 : (v.z == int(pS) ? 2 : -1));
    if (iv < 0) return false;
    const float4 g0 = __ldg(m.geo + 2 * t), g1 = __ldg(m.geo + 2 * t + 1);
    const float px[3] = {g0.x, g0.x + g0.z, g0.x + g1.x};
    const float py[3] = {g0.y, g0.y + g0.w, g0.y + g1.y};
    float e1x = (iv == 0 ? px[1] : (iv == 1 ? px[2] : px[0])) - S.x;
    float e1y = (iv == 0 ? py[1] : (iv == 1 ? py[2] : py[0])) - S.y;
    float e2x = (iv == 0 ? px[2] : (iv == 1 ? px[0] : px[1])) - S.x;
    float e2y = (iv == 0 ? py[2] : (iv == 1 ? py[0] : py[1])) - S.y;
    const float i1 = rsqrtf(e1x * e1x + e1y * e1y), i2 = rsqrtf(e2x * e2x + e2y * e2y);
    e1x *= i1;
    e1y *= i1;
    e2x *= i2;
    e2y *= i2;
    const float cosA = fminf(fmaxf(fmaf(e1x, e2x, e1y * e2y), -1.0f), 1.0f);
    const float alpha = acosf(cosA);
    const float sinA = sinf(alpha);
    // slerp weights: sin(u a)/sin a and sin((1-u) a)/sin a = cos(u a) - cos a sin(u a)/sin a
    float su, cu;
    sincosf(uAz * alpha, &su, &cu);
    const float w2 = __fdividef(su, sinA), w1 = fmaf(-cosA, w2, cu);
    const float cx = fmaf(w1, e1x, w2 * e2x), cy = fmaf(w1, e1y, w2 * e2y);
    const float se = uEl, ce = sqrtf(fmaxf(0.0f, 1.0f - se * se));
    // edge opposite the vertex: edge (iv + 1) % 3 of the walk record
    const int eo = iv == 2 ? 0 : iv + 1;
    const float4 r0 = __ldg(m.tri + 3 * t), r1 = __ldg(m.tri + 3 * t + 1), r2 = __ldg(m.tri + 3 * t + 2);
    const float nx = eo == 0 ? r0.x : (eo == 1 ? r0.w : r1.z);
    const float ny = eo == 0 ? r0.y : (eo == 1 ? r1.x : r1.w);
    const float cc = eo == 0 ? r0.z : (eo == 1 ? r1.y : r2.x);
    const float lxy = __fdividef(cc - fmaf(nx, S.x, ny * S.y), fmaf(nx, cx, ny * cy));
    const float L = fminf(__fdividef(lxy, ce), __fdividef(m.h, se));
    const float r = uR * L;
    const float zs = l == kImg ? 1.0f : -1.0f;
    dx = r * ce * cx;
    dy = r * ce * cy;
    dz = zs * r * se;
    alphaL = alpha * L;
    return true;
}

}  // namespace hase
