// Narrow phase (GJK + EPA) and contact force, warp-cooperative, for sm_103a.
//
// Algorithm: LIBRARIES/gpu_fine_contact_detection.cu (GJK driver :996-1288, simplex tests :103-268,
// EPA :270-603, force :647-871).  The decisions and the floating-point operation sequence are the
// reference's, so contact flags, depths, normals and forces round exactly as the reference kernel
// evaluated without FMA contraction.  The execution model is not:
//
//  * a group of LPP lanes (4/8/16/32) works on one pair; a block holds 128/LPP groups and the grid
//    strides over the pair list.  The device step runs two passes: GJK (gjk_pass_kernel, also one
//    lane per pair) writes the pairs in contact with the simplex it stopped on to a list, and EPA
//    with the force (epa_pass_kernel) continues from that list with a warp per pair;
//  * a GJK support query is a strided scan of the float4 hull vertices (staged in shared memory, or read
//    in place from the L1-cached vertex table) by the group's lanes, then a group argmax on (value
//    desc, index asc), which reproduces the reference's strict-'>' first-index tie break;
//  * the simplex logic runs identically on every lane of the group, so control flow stays group-uniform;
//    the three faces of a tetrahedron test have a lane each (tet_test_lanes), ballots combine them;
//  * EPA keeps an append-only face list of MWD_EPA_FACE_CAP faces, four to a lane (distances and vertex
//    numbers in its registers, normals in shared memory), like the reference's T[50]/n[50]/dist[50] (which
//    overflow past 50 faces); when it is full the removed faces are dropped from it; the face scan, the visibility test, the horizon edge count (the
//    reference's 50x50 delpair matrix, replaced by marks per vertex pair) and the new faces are computed
//    lane-parallel, with ballots to keep the reference's face order;
//  * force/torque are accumulated with float atomics (skipped for wall rows in table mode, whose
//    forces the reference discards, MWDiem.py:977-978).
#include <float.h>

#include "common.cuh"
#include "narrow.cuh"

namespace mwd {

namespace {

constexpr int FCAP = MWD_EPA_FACE_CAP;
constexpr int VCAP = MWD_EPA_VERT_CAP;

__device__ __forceinline__ int ft_v(uint32_t t, int k) { return (t >> (8 * k)) & 0xff; }
template <int LPP>
struct Group {
    int lane;
    unsigned mask;
    __device__ __forceinline__ unsigned ballot(bool p) const
    {
        unsigned b = __ballot_sync(mask, p);
        if (LPP < 32) b = (b & mask) >> (__ffs(mask) - 1);
        return b;
    }
};

// Order-preserving key of a float (-0 and +0 share the key of +0, as they compare equal): the
// group reductions below run on these keys with redux.sync.
__device__ __forceinline__ unsigned fkey(float f)
{
    const unsigned b = __float_as_uint(f + 0.f);
    return b ^ ((unsigned)((int)b >> 31) | 0x80000000u);
}

// Work queue of the EPA pass: a 64-bit counter after the EPA record count in the block epa_count points
// to (MWD_EPA_COUNT_INTS ints, 8-byte aligned), ints [2..3].  Zeroed with the record count before
// each narrow phase.
__device__ __forceinline__ unsigned long long* epa_queue(const NarrowArgs& a)
{
    return reinterpret_cast<unsigned long long*>(a.epa_count + 2);
}

// The next `amount` items of a queue for the calling warp: its first lane takes them with one atomic.
__device__ __forceinline__ int64_t claim(unsigned long long* next, int64_t amount)
{
    unsigned long long base = 0;
    if ((threadIdx.x & 31) == 0) base = atomicAdd(next, (unsigned long long)amount);
    return (int64_t)__shfl_sync(0xffffffffu, base, 0);
}

// work counted per pair when the caller asks for it: vertex dot products, EPA faces, support queries
struct Work3 {
    uint32_t dots, faces, queries;
};

// Vertices of a hull in order, two per 256-bit load where they share 32 bytes, eight in flight.  use(v, i):
// vertex i.  (One lane per pair waits on these loads, each lane's from a hull of its own; four in flight by
// 128-bit loads, a million random pairs took 4.53 ms in both passes instead of 4.38, a 256-scene batch 203 us
// instead of 196; sixteen in flight 237.)
template <class Use>
__device__ __forceinline__ void each_vertex(const float4* h, int n, Use&& use)
{
    int i = 0;
    if ((reinterpret_cast<uintptr_t>(h) & 16u) && n > 0) {
        use(h[0], 0);
        i = 1;
    }
#pragma unroll 4
    for (; i + 1 < n; i += 2) {
        float4 u, v;
        asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(u.x), "=f"(u.y), "=f"(u.z), "=f"(u.w), "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
            : "l"(__cvta_generic_to_global(h + i)));
        use(u, i);
        use(v, i + 1);
    }
    if (i < n) use(h[i], i);
}

// Two hulls read in place by one lane.  query: argmax of d.a over A and of (-d).b over B, first index on ties
// (.cu:55-101); both: the queries in the directions d and -d in one pass over the hulls (the second one's
// products are the first one's negated, exactly).
struct LaneHulls {
    const float4 *hA, *hB;
    int nA, nB;
    __device__ __forceinline__ void query(f3 d, f3& s, int& ia, int& ib) const
    {
        float bA = -1e30f, bB = -1e30f;
        int wA = 0, wB = 0;
        each_vertex(hA, nA, [&](float4 v, int i) {
            const float t = d.x * v.x + d.y * v.y + d.z * v.z;
            if (t > bA) { bA = t; wA = i; }
        });
        const f3 nd = d * (-1.f);
        each_vertex(hB, nB, [&](float4 v, int j) {
            const float t = nd.x * v.x + nd.y * v.y + nd.z * v.z;
            if (t > bB) { bB = t; wB = j; }
        });
        ia = wA;
        ib = wB;
        const float4 a = hA[ia], b = hB[ib];
        s = mk3(a.x - b.x, a.y - b.y, a.z - b.z);
    }
    __device__ __forceinline__ void both(f3 d, f3& S1, int& a1, int& b1, f3& S2, int& a2, int& b2) const
    {
        float tA = -1e30f, uA = -1e30f, tB = -1e30f, uB = -1e30f;
        int wA1 = 0, wA2 = 0, wB1 = 0, wB2 = 0;
        each_vertex(hA, nA, [&](float4 v, int i) {
            const float t = d.x * v.x + d.y * v.y + d.z * v.z;
            if (t > tA) { tA = t; wA1 = i; }
            if (-t > uA) { uA = -t; wA2 = i; }
        });
        each_vertex(hB, nB, [&](float4 v, int j) {
            const float t = d.x * v.x + d.y * v.y + d.z * v.z;
            if (t > tB) { tB = t; wB2 = j; }
            if (-t > uB) { uB = -t; wB1 = j; }
        });
        a1 = wA1;
        a2 = wA2;
        b1 = wB1;
        b2 = wB2;
        const float4 p1 = hA[a1], q1 = hB[b1], p2 = hA[a2], q2 = hB[b2];
        S1 = mk3(p1.x - q1.x, p1.y - q1.y, p1.z - q1.z);
        S2 = mk3(p2.x - q2.x, p2.y - q2.y, p2.z - q2.z);
    }
};

// ---- simplex tests, identical on every lane (.cu:103-268) ----
__device__ __forceinline__ void seg_test(f3 P1, f3 P2, int& coll, f3& d)
{
    coll = -1;
    d = mk3(0.f, 0.f, 0.f);
    f3 e = P2 - P1;
    if (dot(e, P2) < 0.f) { coll = 0; return; }
    f3 t = cross(e, P2);
    if (t.x == 0.f && t.y == 0.f && t.z == 0.f) { coll = 1; return; }
    f3 tmp = cross(e, P2 * (-1.f));
    d = cross(tmp, e);
}

__device__ __forceinline__ void tri_test(f3 P1, f3 P2, f3 P3, int& coll, f3& d)
{
    coll = -1;
    d = mk3(0.f, 0.f, 0.f);
    int c2, c3;
    seg_test(P2, P3, c2, d);
    if (c2 == 1) { coll = 1; return; }
    seg_test(P1, P3, c3, d);
    if (c3 == 1) { coll = 1; return; }
    if (c2 + c3 > -1) { coll = 0; return; }
    f3 e32 = P3 - P2, e13 = P1 - P3;
    f3 n = cross(e32, e13);
    f3 n2 = cross(e32, n);
    f3 n3 = cross(e13, n);
    if (dot(n2, P2) < 0.f) { d = n2; return; }
    if (dot(n3, P3) < 0.f) { d = n3; return; }
    if (dot(P3, n) == 0.f) { coll = 1; return; }
    if (dot(n, P3) > 0.f) d = n * (-1.f);
    else d = n;
}

__device__ __forceinline__ void tet_test(f3 P1, f3 P2, f3 P3, f3 P4, int& coll, f3& d, int& todel)
{
    coll = -1;
    d = mk3(0.f, 0.f, 0.f);
    todel = 0;
    int c1, c2, c3;
    tri_test(P1, P2, P4, c1, d);
    if (c1 == 1) { coll = 1; return; }
    tri_test(P2, P3, P4, c2, d);
    if (c2 == 1) { coll = 1; return; }
    tri_test(P3, P1, P4, c3, d);
    if (c3 == 1) { coll = 1; return; }
    if (c1 + c2 + c3 > -2) { coll = 0; return; }
    f3 e13 = P1 - P3, e21 = P2 - P1, e32 = P3 - P2, e41 = P4 - P1;
    f3 n2 = cross(e21, e41);
    f3 e42 = P4 - P2;
    f3 n3 = cross(e32, e42);
    f3 e43 = P4 - P3;
    f3 n4 = cross(e13, e43);
    if (dot(n2, P4) < 0.f) { d = n2; todel = 3; }
    else if (dot(n3, P4) < 0.f) { d = n3; todel = 1; }
    else if (dot(n4, P4) < 0.f) { d = n4; todel = 2; }
    else coll = 1;
}

// the outcome of seg_test and of tri_test, without their direction (which tet_test does not use)
__device__ __forceinline__ int seg_outcome(f3 P1, f3 P2)
{
    const f3 e = P2 - P1;
    const f3 t = cross(e, P2);
    return dot(e, P2) < 0.f ? 0 : (t.x == 0.f && t.y == 0.f && t.z == 0.f) ? 1 : -1;
}
__device__ __forceinline__ int tri_outcome(f3 P1, f3 P2, f3 P3)
{
    const int c2 = seg_outcome(P2, P3), c3 = seg_outcome(P1, P3);
    const f3 e13 = P1 - P3;
    const f3 e32 = P3 - P2;
    const f3 n = cross(e32, e13);
    const bool beside = dot(cross(e32, n), P2) < 0.f || dot(cross(e13, n), P3) < 0.f;
    if (c2 == 1 || c3 == 1) return 1;
    if (c2 == 0 && c3 == 0) return 0;
    return !beside && dot(P3, n) == 0.f ? 1 : -1;
}

// tet_test by each group of LPP >= 4 lanes of a full warp: lane f = 0, 1, 2 tests the face (P1,P2,P4),
// (P2,P3,P4), (P3,P1,P4) -- tri_test's outcome and the side the origin lies on -- and ballots combine them.
// (On every lane in turn, the three faces are about 400 instructions, and GJK's slow pairs run 50 such tests.)
template <int LPP>
__device__ __forceinline__ void tet_test_lanes(f3 P1, f3 P2, f3 P3, f3 P4, int& coll, f3& d, int& todel)
{
    static_assert(LPP >= 4, "a lane per face");
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, g0 = lane & ~(LPP - 1), f = lane & 3;
    const f3 a = f == 0 ? P1 : f == 1 ? P2 : P3;
    const f3 b = f == 0 ? P2 : f == 1 ? P3 : P1;
    const int c = tri_outcome(a, b, P4);
    const f3 n = cross(b - a, P4 - a);
    const unsigned inside = (__ballot_sync(ALL, c == 1) >> g0) & 7u, zero = (__ballot_sync(ALL, c == 0) >> g0) & 7u;
    const unsigned beyond = (__ballot_sync(ALL, dot(n, P4) < 0.f) >> g0) & 7u;
    const int first = beyond ? __ffs(beyond) - 1 : 0;
    // c1 + c2 + c3 > -2: two of them zero
    coll = inside ? 1 : __popc(zero) >= 2 ? 0 : beyond ? -1 : 1;
    todel = first == 0 ? 3 : first;
    d.x = __shfl_sync(ALL, n.x, g0 + first);
    d.y = __shfl_sync(ALL, n.y, g0 + first);
    d.z = __shfl_sync(ALL, n.z, g0 + first);
}

// (double)v < 1e-6 && (double)v > -1e-6 for a float v, without FP64: a float compares with the
// double 1e-6 as it compares with the smallest float not below it (0x358637be); NaN fails both
__device__ __forceinline__ bool within_1e6(float v)
{
    const float F = __uint_as_float(0x358637beu);
    return v < F && v > -F;
}

// CorrectFlat: both determinants inside a double +-1e-6 window (.cu:256-268)
__device__ __forceinline__ bool is_flat(f3 S1, f3 S2, f3 S3, f3 S4)
{
    float det1 = S1.x * (S2.y * S3.z - S3.y * S2.z) - S2.x * (S1.y * S3.z - S3.y * S1.z) + S3.x * (S1.y * S2.z - S2.y * S1.z);
    if (within_1e6(det1)) {
        float det2 = S1.x * (S2.y * S4.z - S4.y * S2.z) - S2.x * (S1.y * S4.z - S4.y * S1.z) + S4.x * (S1.y * S2.z - S2.y * S1.z);
        if (within_1e6(det2)) return true;
    }
    return false;
}

// The EPA's stop tests (.cu:437-439): x > p, or (double)x * 1.00001 > (double)p && (double)x * 0.99999 <
// (double)p.  For x > 0 the two together are (double)x * 1.00001 > (double)p, decided in FP32 unless p
// lies within 2^-22 x of the bound: the float product x * 1.00001f is within 7.5e-8 x of the double one
// and the shifted bounds round by at most 6e-8 x more (1.4e-7 x < 2^-22 x in all), so outside that band
// the float answer is the double one; inside it (and for x outside [1e-30, 1e37], NaN, or 0) the
// reference's tests run.
__device__ __noinline__ bool epa_stops_exactly(float x, float p)
{
    return x > p || ((double)x * 1.00001 > (double)p && (double)x * 0.99999 < (double)p);
}
__device__ __forceinline__ bool epa_stops(float x, float p)
{
    if (x > 1e-30f && x < 1e37f) {
        const float hi = x * 1.00001f, tol = x * 2.384185791015625e-7f;
        if (p < hi - tol) return true;
        if (p > hi + tol) return false;
    }
    return epa_stops_exactly(x, p);
}

// ---------------------------------------------------------------- the reference's double results in FP32
// A few per-contact quantities the reference computes in double and rounds to float (the barycentric
// weight of the contact point, .cu:583; the tangential stiffness and damping, .cu:746-749; the Coulomb
// test, .cu:774).  FP64 runs at a small fraction of the FP32 rate on this GPU and its long latency sat
// on every contact's path, so they are evaluated in float-float arithmetic (error-free sums, fused
// multiply-add remainders) and the float is taken when it is provably the double computation's result
// rounded to float: when the value lies farther from a float rounding boundary than the error bound of
// both computations.  Otherwise (a value within ~2^-18 of a boundary, or non-finite or extreme
// operands) the double computation runs.

// s + e = a + b exactly (Knuth)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// s + e = a + b exactly, for |a| >= |b| (or a = 0) (Dekker)
__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e)
{
    s = a + b;
    e = b - (s - a);
}

// true when every real within `err` of a + b rounds to the float a (round to nearest): |b| plus the
// error stays below half the spacing of the floats next to a on b's side (the spacing below a power
// of two, toward zero, is half the one above).  False for |a| outside [2^-102, 2^127) and non-finite a.
__device__ __forceinline__ bool rounds_to(float a, float b, float err)
{
    const uint32_t ua = __float_as_uint(a) & 0x7fffffffu;
    if (ua < 0x0c800000u || ua >= 0x7f000000u) return false;
    const float ulp = __uint_as_float(ua & 0x7f800000u) * 1.1920928955078125e-7f;  // 2^(exponent - 23)
    const bool toward_zero = (b < 0.f) != (a < 0.f);
    const float half = ((ua & 0x007fffffu) == 0u && toward_zero) ? 0.25f * ulp : 0.5f * ulp;
    return fabsf(b) + err < half * 0.99999f;
}

// spacing of the floats at x (2^-149 for subnormal x, +inf for 0 and non-finite x)
__device__ __forceinline__ float ulp_of(float x)
{
    const uint32_t ux = __float_as_uint(x) & 0x7fffffffu;
    if (ux == 0u || ux >= 0x7f800000u) return __int_as_float(0x7f800000);
    if (ux < 0x00800000u) return 1.401298464324817e-45f;
    return __uint_as_float(ux & 0x7f800000u) * 1.1920928955078125e-7f;
}

// (float)(1.0 - (double)bw - (double)bv).  The exact value is s2 + t + r (error-free sums) and a is the
// float nearest to s2 + t.  1, bw and bv are multiples of q = the smallest of their spacings, and so
// are 1 - bw and the result: below 2^53 q the double computation holds both exactly, and with r = 0 a is
// then its result rounded to float, ties included.  Otherwise a is certified against the double
// computation's error, at most 2^-53 (|1 - bw| + |result|).
__device__ __forceinline__ float one_minus_two(float bw, float bv)
{
    float s1, e1, s2, e2, t, r, a, b0;
    two_sum(1.f, -bw, s1, e1);
    two_sum(s1, -bv, s2, e2);
    two_sum(e2, e1, t, r);
    two_sum(s2, t, a, b0);
    if (fabsf(bw) < 1e30f && fabsf(bv) < 1e30f) {
        const float q = fminf(fminf(ulp_of(bw), ulp_of(bv)), 1.1920928955078125e-7f);
        const bool exact = fmaxf(fabsf(s1), fabsf(a)) < q * 2251799813685248.f;  // 2^51 q
        if (exact && r == 0.f) return a;
        const float b = b0 + r;
        const float err = (exact ? 0.f : (fabsf(s1) + fabsf(a)) * 2.220446049250313e-16f) +
                          fabsf(b) * 1.1920928955078125e-7f;
        if (rounds_to(a, b, err)) return a;
    }
    return (float)(1.0 - (double)bw - (double)bv);
}

// Kt = (float)(KtA * 1 / C) and Gt = (float)((-1) * 2 / C * (double)ln_et) with
// C = inv_mu + (double)x + (double)y (.cu:746-749; x, y the float quotients dA^2/IsA, dB^2/IsB).  C is
// formed as a float pair from non-negative terms; each quotient is a rounded float quotient (KtA_hi / ch,
// and -2 / ch as -2 RN(1 / ch), exact scaling), whose remainder a fused multiply-add gives exactly,
// corrected by that remainder times RN(1 / ch).  The pair values are within 2^-43 of the exact ones
// and the double results within 5 * 2^-53 of them: a margin of 2^-41 certifies the float.
__device__ __forceinline__ void tangential_coeffs(const mwd_material& M, float x, float y, float& Kt, float& Gt)
{
    bool okK = false, okG = false;
    if (x >= 0.f && x < 1e30f && y >= 0.f && y < 1e30f && M.inv_mu_hi > 0.f && M.inv_mu_hi < 1e30f) {
        float c1, e1, c2, e2, ch, cl;
        two_sum(M.inv_mu_hi, x, c1, e1);
        two_sum(c1, y, c2, e2);
        fast_two_sum(c2, (M.inv_mu_lo + e1) + e2, ch, cl);
        const float rc = 1.f / ch;
        // (KtA_hi + KtA_lo) / (ch + cl)
        const float q1 = M.KtA_hi / ch;
        const float rq = ((fmaf(-q1, ch, M.KtA_hi) + M.KtA_lo) - q1 * cl) * rc;
        float kh, kl;
        fast_two_sum(q1, rq, kh, kl);
        // -2 / (ch + cl), then times ln_et
        const float g1 = -2.f * rc;
        const float rg = (fmaf(-g1, ch, -2.f) - g1 * cl) * rc;
        float gh, gl;
        fast_two_sum(g1, rg, gh, gl);
        const float p = gh * M.ln_et;
        float Gh, Gl;
        fast_two_sum(p, fmaf(gh, M.ln_et, -p) + gl * M.ln_et, Gh, Gl);
        okK = rounds_to(kh, kl, fabsf(kh) * 4.547473508864641e-13f);  // 2^-41
        okG = rounds_to(Gh, Gl, fabsf(Gh) * 4.547473508864641e-13f);
        Kt = kh;
        Gt = Gh;
    }
    if (okK && okG) return;
    const double C = M.inv_mu + (double)x + (double)y;
    if (!okK) Kt = (float)(M.KtA * 1 / C);
    if (!okG) Gt = (float)((-1) * 2 / C * (double)M.ln_et);
}

// (double)Ftn > mu * (double)Fnn (.cu:774): 1 when greater, 0 when not greater, -1 when unordered (NaN).
// mu_f * Fnn is within 2.1 u of the double product (u = 2^-24): a margin of 4e-7 (~6.7 u) decides.
__device__ __forceinline__ int coulomb_compare(float Ftn, float Fnn, const mwd_material& M)
{
    const float t = M.mu_f * Fnn;
    if (t >= 1e-30f && t <= 1e30f) {
        const float e = t * 4e-7f;
        if (Ftn > t + e) return 1;
        if (Ftn < t - e) return 0;
    }
    const double X = (double)Ftn, P = M.mu * (double)Fnn;
    return X > P ? 1 : (X <= P ? 0 : -1);
}

struct EpaResult {
    float depth;
    f3 n, cpA, cpB;
    int fa[3], fb[3];
    uint32_t status;
};

// contact points of the final face (.cu:548-600): barycentric coordinates of n * depth on the face
// Va, Vb, Vc (winding swapped when its normal points the other way), applied to the support vertices of
// A and B (pa, pb, pc: index on A | index on B << 8)
__device__ __forceinline__ void epa_contact(f3 Va, f3 Vb, f3 Vc, int pa, int pb, int pc, const float4* hA,
                                            const float4* hB, f3 n, EpaResult& r)
{
    f3 Pr = n * r.depth;
    f3 v0 = Vb - Va, v1 = Vc - Va, v2 = Pr - Va;
    if (dot(cross(v0, v1), n) < 0.f) {
        v0 = Vc - Va;
        v1 = Vb - Va;
    }
    float v00 = dot(v0, v0), v01 = dot(v0, v1), v11 = dot(v1, v1), v20 = dot(v2, v0), v21 = dot(v2, v1);
    float den = v00 * v11 - v01 * v01;
    float bv = (v11 * v20 - v01 * v21) / den;
    float bw = (v00 * v21 - v01 * v20) / den;
    float bu = one_minus_two(bw, bv);
    r.fa[0] = pa & 0xff; r.fa[1] = pb & 0xff; r.fa[2] = pc & 0xff;
    r.fb[0] = pa >> 8; r.fb[1] = pb >> 8; r.fb[2] = pc >> 8;
    r.cpA = (xyz(hA[r.fa[0]]) * bu + xyz(hA[r.fa[1]]) * bv) + xyz(hA[r.fa[2]]) * bw;
    r.cpB = (xyz(hB[r.fb[0]]) * bu + xyz(hB[r.fb[1]]) * bv) + xyz(hB[r.fb[2]]) * bw;
    r.n = n;
}

// ------------------------------------------------------------------ EPA by one warp
//
// One pair per warp, laid out for the length of an iteration's dependent chain, which sets the time of
// a step with a few thousand contacts (its longest EPA runs 25 iterations): each lane keeps its
// hull vertices and the distances and vertex numbers of its faces of the append-only list (face f in lane
// f % 32, slot f / 32) in registers, so a support query and the minimum search read no memory; the new
// faces are computed in the lanes that will hold them.  Shared memory holds the polytope's vertices and the
// faces' normals (in registers too, 2M random pairs took 4% longer; with nothing of the faces in
// registers 1% less, but short lists 2-4% longer).  The forces wait until the warp has up to 32 of them, one
// per lane.
//
// An iteration alone on its scheduler takes about 1.2 us (some 560 instructions, partly waiting for their
// fetch).  Against groups of 8, 16 or 32 lanes with the polytope in shared memory, which it replaces: the pass
// on 3,001 random pairs 122 -> 50 us (8 lanes before), on four steps of 5,003 packed hulls 122 -> 56 us each
// (8 lanes and the rerun of the overflowing pairs), on 30,011 packed hulls 83 -> 70 us (32 lanes), on 2M random
// pairs 9.05 -> 7.6 ms (16 lanes), where it issues on 74% of the cycles.

// the two hulls over a warp: lanes 0-15 hold A's vertices, lanes 16-31 B's, `per` consecutive ones each
// (NaN past the end: such a product never wins)
struct WarpHulls {
    const float4 *hA, *hB;
    int nA, nB, per;
    float x[4], y[4], z[4];
    __device__ __forceinline__ void query(f3 d, f3& s, int& ia, int& ib) const;
    __device__ __forceinline__ void both(f3 d, f3& S1, int& a1, int& b1, f3& S2, int& a2, int& b2) const;
    __device__ __forceinline__ void load(const float4* a, int na, const float4* b, int nb)
    {
        hA = a;
        hB = b;
        nA = na;
        nB = nb;
        per = (max(na, nb) + 15) >> 4;
        const int lane = threadIdx.x & 31;
        const float4* h = lane < 16 ? a : b;
        const int n = lane < 16 ? na : nb, first = (lane & 15) * per;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float4 v = make_float4(__int_as_float(0x7fffffff), 0.f, 0.f, 0.f);
            if (j < per && first + j < n) v = h[first + j];
            x[j] = v.x;
            y[j] = v.y;
            z[j] = v.z;
        }
    }
};
static_assert(MWD_HULL_CAP <= 64, "four vertices per lane");

// support() by a warp: each half's largest product, then the smallest index among the lanes that hold it
__device__ __forceinline__ void warp_winners(float best, unsigned idx, int& ia, int& ib)
{
    const bool onB = (threadIdx.x & 16) != 0;
    const unsigned k = fkey(best);
    const unsigned kA = __reduce_max_sync(0xffffffffu, onB ? 0u : k);
    const unsigned kB = __reduce_max_sync(0xffffffffu, onB ? k : 0u);
    ia = (int)__reduce_min_sync(0xffffffffu, !onB && k == kA ? idx : 0xffffu);
    ib = (int)__reduce_min_sync(0xffffffffu, onB && k == kB ? idx : 0xffffu);
}

__device__ __forceinline__ void WarpHulls::query(f3 d, f3& s, int& ia, int& ib) const
{
    const int lane = threadIdx.x & 31;
    const f3 e = lane >= 16 ? d * (-1.f) : d;
    float best = -1e30f;
    int at = -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j < per) {
            const float t = e.x * x[j] + e.y * y[j] + e.z * z[j];
            if (t > best) { best = t; at = j; }
        }
    }
    warp_winners(best, at < 0 ? 0u : (unsigned)((lane & 15) * per + at), ia, ib);
    const float4 a = hA[ia], b = hB[ib];
    s = mk3(a.x - b.x, a.y - b.y, a.z - b.z);
}

// support_pair() by a warp: the second query's products are the first one's negated (exactly)
__device__ __forceinline__ void WarpHulls::both(f3 d, f3& S1, int& a1, int& b1, f3& S2, int& a2, int& b2) const
{
    const int lane = threadIdx.x & 31;
    const f3 e = lane >= 16 ? d * (-1.f) : d;
    float best = -1e30f, opp = -1e30f;
    int at = -1, oat = -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j < per) {
            const float t = e.x * x[j] + e.y * y[j] + e.z * z[j];
            if (t > best) { best = t; at = j; }
            if (-t > opp) { opp = -t; oat = j; }
        }
    }
    const unsigned first = (unsigned)((lane & 15) * per);
    warp_winners(best, at < 0 ? 0u : first + (unsigned)at, a1, b1);
    warp_winners(opp, oat < 0 ? 0u : first + (unsigned)oat, a2, b2);
    const float4 p1 = hA[a1], q1 = hB[b1], p2 = hA[a2], q2 = hB[b2];
    S1 = mk3(p1.x - q1.x, p1.y - q1.y, p1.z - q1.z);
    S2 = mk3(p2.x - q2.x, p2.y - q2.y, p2.z - q2.z);
}

constexpr uint32_t FACE_LIVE = 0x80000000u;
constexpr int FACE_SLOTS = FCAP / 32;

struct WarpEpaMem {
    float4 fn[FCAP];      // face normal xyz, distance (3e20 once removed)
    float4 pv[VCAP];      // polytope vertices
    uint32_t ft[FCAP];    // vertices T0 | T1 << 8 | T2 << 16, FACE_LIVE
    uint32_t del[FCAP];   // faces removed in this iteration, in index order
    uint16_t edge[FCAP];  // horizon edges, first vertex | second << 8
    uint16_t mark[VCAP * VCAP];  // by unordered vertex pair: the removed faces' edge that has it
    uint16_t pab[VCAP];   // support index on A | on B << 8
};

// AddTriangle (.cu:270-325) for the face a, b, c: its normal and distance (1e30 when the origin's
// projection falls outside it); flip: its winding is a, c, b
__device__ __forceinline__ float4 face_plane(f3 a, f3 b, f3 c, bool& flip)
{
    f3 n = cross(b - a, c - b);
    n = n / sqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
    float dist = dot(n, a);
    flip = dist < 0.f;
    if (flip) {
        const f3 t = b;
        b = c;
        c = t;
        dist = dist * (-1.f);
        n = n * (-1.f);
    }
    // (the reference's dot(., -a) < 0: the negated product is exact)
    const float ia = dot(cross(b - a, n), a), ib = dot(cross(c - b, n), b), ic = dot(cross(a - c, n), c);
    return f4(n, ia > 0.f && ib > 0.f && ic > 0.f ? dist : 1e30f);
}

// edge j of a removed face: its vertices, and the code of the unordered pair
__device__ __forceinline__ int edge_vertices(uint32_t t, int j, int& e0, int& e1)
{
    e0 = (int)((t >> (8 * j)) & 0xffu);
    e1 = (int)((t >> (j == 2 ? 0 : 8 * j + 8)) & 0xffu);
    return min(e0, e1) * VCAP + max(e0, e1);
}

// What an EPA seldom needs stays out of its loop, whose time on a short list is that of fetching its
// instructions.

// the horizon of more than ten removed faces (more edges than lanes), 32 edges at a time
__device__ __noinline__ int horizon_many(WarpEpaMem& m, int edges)
{
    const int lane = threadIdx.x & 31;
    int e0, e1, nnew = 0;
    for (int c = lane; c < edges; c += 32) m.mark[edge_vertices(m.del[c / 3], c % 3, e0, e1)] = (uint16_t)c;
    __syncwarp();
    for (int c = lane; c < edges; c += 32) {
        const int code = edge_vertices(m.del[c / 3], c % 3, e0, e1);
        if (m.mark[code] != c) m.mark[code] = 0xffffu;
    }
    __syncwarp();
    for (int base = 0; base < edges; base += 32) {
        const int c = base + lane;
        const bool keep = c < edges && m.mark[edge_vertices(m.del[c / 3], c % 3, e0, e1)] == c;
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        const int q = nnew + __popc(b & ((1u << lane) - 1u));
        if (keep && q < FCAP) m.edge[q] = (uint16_t)(e0 | (e1 << 8));
        nnew += __popc(b);
    }
    return nnew;
}

// the removed faces out of the list in shared memory, the first one excepted; returns the new length
__device__ __noinline__ int drop_removed(WarpEpaMem& m, int nt)
{
    const int lane = threadIdx.x & 31;
    int kept = 0;
    bool first = true;
    for (int base = 0; base < nt; base += 32) {
        const int f = base + lane;
        const bool in = f < nt;
        const float4 p = in ? m.fn[f] : make_float4(0.f, 0.f, 0.f, 0.f);
        const uint32_t t = in ? m.ft[f] : 0u;
        const unsigned gone = __ballot_sync(0xffffffffu, in && !(t & FACE_LIVE));
        const bool keep = in && ((t & FACE_LIVE) || (first && lane == __ffs(gone) - 1));
        if (gone) first = false;
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        const int o = kept + __popc(b & ((1u << lane) - 1u));  // at most f: nothing unread is overwritten
        __syncwarp();
        if (keep) {
            m.fn[o] = p;
            m.ft[o] = t;
        }
        kept += __popc(b);
    }
    __syncwarp();
    return kept;
}

struct WarpEpaOut {
    float4 face;      // the final face's normal; w: depth
    uint32_t t;       // its vertices in the polytope
    uint32_t status;
    int faces, queries;  // faces created, support queries
};

// EPA (.cu:328-603).  The list is append-only like the reference's: a removed face stays at distance
// 3e20 (.cu:541-542), where the first of them can still win the minimum search (.cu:41-53).  When the
// list is full the removed faces are dropped from it, the first one excepted, in order.
__device__ __forceinline__ void epa_warp(WarpEpaMem& m, const WarpHulls& h, f3 S1, int a1, int b1, f3 S2, int a2,
                                         int b2, f3 S3, int a3, int b3, f3 S4, int a4, int b4, WarpEpaOut& r)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int lane_face = lane / 3, lane_edge = lane % 3;  // of the first 32 edges of the removed faces
    constexpr unsigned ALL = 0xffffffffu;
    const float nan = __int_as_float(0x7fffffff);
    r.status = 0;
    __syncwarp();
    if (lane == 0) {
        m.pv[0] = f4(S1, 0.f); m.pv[1] = f4(S2, 0.f); m.pv[2] = f4(S3, 0.f); m.pv[3] = f4(S4, 0.f);
        m.pab[0] = (uint16_t)(a1 | (b1 << 8)); m.pab[1] = (uint16_t)(a2 | (b2 << 8));
        m.pab[2] = (uint16_t)(a3 | (b3 << 8)); m.pab[3] = (uint16_t)(a4 | (b4 << 8));
    }
    // this lane's faces: distance (NaN: no face), vertex numbers
    float fd[FACE_SLOTS];
    uint32_t ft[FACE_SLOTS];
#pragma unroll
    for (int s = 0; s < FACE_SLOTS; ++s) {
        fd[s] = nan;
        ft[s] = 0;
    }
    // face f of (0,1,2), (1,2,3), (2,0,3), (0,1,3) in lane f
    if (lane < 4) {
        const f3 a = lane == 1 ? S2 : lane == 2 ? S3 : S1;
        const f3 b = lane == 1 ? S3 : lane == 2 ? S1 : S2;
        const f3 c = lane == 0 ? S3 : S4;
        const uint32_t e = lane == 0 ? 0x020100u : lane == 1 ? 0x030201u : lane == 2 ? 0x030002u : 0x030100u;
        bool flip;
        const float4 p = face_plane(a, b, c, flip);
        fd[0] = p.w;
        ft[0] = (flip ? (e & 0xffu) | ((e >> 8) & 0xff00u) | ((e & 0xff00u) << 8) : e) | FACE_LIVE;
        m.fn[lane] = p;
        m.ft[lane] = ft[0];
    }
    __syncwarp();
    int nt = 4, nv = 4, counter = 0;
    r.faces = 4;
    r.queries = 0;
    float xmin_old = 1e29f;
    float proj = 2 * xmin_old + 1;
    float4 fm = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t tm = 0;
    while (xmin_old < proj) {
        // first index of the minimum distance (NaN never wins, except in face 0, where the search starts)
        float bv = fd[0];
        int bs = 0;
#pragma unroll
        for (int s = 1; s < FACE_SLOTS; ++s) {
            if (32 * s < nt && (fd[s] < bv || bv != bv)) { bv = fd[s]; bs = s; }
        }
        unsigned k = bv != bv ? 0xffffffffu : fkey(bv);
        if (lane == 0 && fd[0] != fd[0]) { k = 0u; bs = 0; }
        const unsigned km = __reduce_min_sync(ALL, k);
        const int bi = (int)__reduce_min_sync(ALL, k == km ? (unsigned)(32 * bs + lane) : 0x7fffffffu);
        fm = m.fn[bi];
        tm = m.ft[bi];
        xmin_old = fm.w;
        const f3 n = xyz(fm);
        f3 sp;
        int sa, sb;
        h.query(n, sp, sa, sb);
        r.queries += 1;
        proj = dot(n, sp);
        if (epa_stops(xmin_old, proj)) break;
        if (counter > 49) { r.status |= MWD_ST_EPA_NOCONV; break; }
        counter = counter + 1;
        if (nv >= VCAP) { r.status |= MWD_ST_EPA_OVERFLOW; break; }
        if (lane == 0) {
            m.pv[nv] = f4(sp, 0.f);
            m.pab[nv] = (uint16_t)(sa | (sb << 8));
        }
        nv++;
        __syncwarp();  // every lane has read the chosen face
        // faces that the new vertex sees are removed, collected in index order
        int ndel = 0;
#pragma unroll
        for (int s = 0; s < FACE_SLOTS; ++s) {
            if (32 * s < nt) {
                const bool dead = (ft[s] & FACE_LIVE) && dot(sp - xyz(m.pv[ft_v(ft[s], 0)]), xyz(m.fn[32 * s + lane])) >= 0.f;
                const unsigned b = __ballot_sync(ALL, dead);
                if (dead) {
                    m.del[ndel + __popc(b & lt)] = ft[s];
                    ft[s] &= ~FACE_LIVE;
                    fd[s] = 3e20f;
                    m.fn[32 * s + lane].w = 3e20f;
                    m.ft[32 * s + lane] = ft[s];
                }
                ndel += __popc(b);
            }
        }
        __syncwarp();
        // horizon edges of the removed faces, in face order then edge order (0,1),(1,2),(2,0); an edge is
        // kept when fewer than two delpair increments land on it (.cu:482-544), i.e. when its unordered
        // vertex pair occurs once among the removed faces' edges (a face's vertices are distinct).  Every
        // edge marks its pair with its number; one that finds another's number there spoils the mark; an
        // edge that still finds its own is alone.  (A match over the warp takes 390 cycles on this GPU;
        // comparing the lanes' pairs by exchanges took a quarter of the EPA's instructions.)
        int nnew = 0;
        const int edges = 3 * ndel;
        if (edges <= 32) {
            const bool has = lane < edges;
            int e0 = 0, e1 = 0, code = 0;
            if (has) {
                code = edge_vertices(m.del[lane_face], lane_edge, e0, e1);
                m.mark[code] = (uint16_t)lane;
            }
            __syncwarp();
            if (has && m.mark[code] != lane) m.mark[code] = 0xffffu;
            __syncwarp();
            const bool keep = has && m.mark[code] == lane;
            const unsigned b = __ballot_sync(ALL, keep);
            if (keep) m.edge[__popc(b & lt)] = (uint16_t)(e0 | (e1 << 8));
            nnew = __popc(b);
        } else {
            nnew = horizon_many(m, edges);
        }
        __syncwarp();
        if (nt + nnew > FCAP) {
            // the list is full (about one deep overlap in 120,000 of random hulls, some contacts of every
            // step of packed hulls or cubes): drop the removed faces, the first one excepted.  At most
            // 2 * 30 - 4 = 56 faces of a closed polytope are alive within the reference's iteration limit.
            nt = drop_removed(m, nt);
#pragma unroll
            for (int s = 0; s < FACE_SLOTS; ++s) {
                fd[s] = nan;
                ft[s] = 0;
                if (32 * s + lane < nt) {
                    const float4 p = m.fn[32 * s + lane];
                    ft[s] = m.ft[32 * s + lane];
                    fd[s] = p.w;
                }
            }
            __syncwarp();
            if (nt + nnew > FCAP) { r.status |= MWD_ST_EPA_OVERFLOW; break; }
        }
        // the new faces (edge q, new vertex) at list positions nt + q, each in the lane that holds it
        for (int q0 = 0; q0 < nnew; q0 += 32) {
            const int q = q0 + ((lane - nt - q0) & 31);
            const int pos = q < nnew ? nt + q : -1;
            f3 a = mk3(0.f, 0.f, 0.f);
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
            uint32_t t = 0;
            if (pos >= 0) {
                const uint32_t e = m.edge[q];
                const uint32_t e0 = e & 0xffu, e1 = e >> 8, e2 = (uint32_t)(nv - 1);
                a = xyz(m.pv[e0]);
                bool flip;
                p = face_plane(a, xyz(m.pv[e1]), sp, flip);
                t = e0 | (flip ? (e2 << 8) | (e1 << 16) : (e1 << 8) | (e2 << 16)) | FACE_LIVE;
                m.fn[pos] = p;
                m.ft[pos] = t;
            }
            const int s0 = (nt + q0) >> 5;  // the 32 positions lie in slots s0 and s0 + 1
#pragma unroll
            for (int s = 0; s < FACE_SLOTS; ++s) {
                if (s != s0 && s != s0 + 1) continue;
                const bool here = (pos >> 5) == s;  // selects, so that the arrays stay in registers
                fd[s] = here ? p.w : fd[s];
                ft[s] = here ? t : ft[s];
            }
        }
        nt += nnew;
        r.faces += nnew;
        counter = counter + 1;
        __syncwarp();
    }
    r.face = make_float4(fm.x, fm.y, fm.z, fm.w);
    r.t = tm;
}

// CorrectFlat (.cu:256-268) and EPA from the simplex GJK stopped on (ia, ib: its support indices, 8 bits each)
__device__ __forceinline__ void epa_from_simplex(WarpEpaMem& m, const WarpHulls& h, f3 S1, f3 S2, f3 S3, f3 S4,
                                                 uint32_t ia, uint32_t ib, WarpEpaOut& r)
{
    int a4 = ia >> 24, b4 = ib >> 24;
    const bool flat = is_flat(S1, S2, S3, S4);
    if (flat) h.query(cross(S1, S2), S4, a4, b4);
    epa_warp(m, h, S1, ia & 0xff, ib & 0xff, S2, (ia >> 8) & 0xff, (ib >> 8) & 0xff, S3, (ia >> 16) & 0xff,
             (ib >> 16) & 0xff, S4, a4, b4, r);
    r.queries += flat ? 1 : 0;
}

struct ForceResult {
    f3 F, TA, TB, dt;
};

// Force (.cu:647-871) with the pair-independent constants taken from mwd_material
// imA, imB: inverse masses (0 for a wall side), read only by the physical law.
__device__ __forceinline__ void contact_force(f3 cA, f3 cB, float depth, f3 n, f3 cpA, f3 cpB, const mwd_material& M,
                                              f3 vA, f3 vB, f3 wA, f3 wB, f3 dt, float4 qA, float dtn, float IsA,
                                              float IsB, float imA, float imB, ForceResult& o)
{
    f3 cp;
    float Kt, Gt, Gn;
    if (!M.physical) {
        cp = (cpA - cpB) / 2.f;
        f3 dA = cp - cA, dB = cp - cB;
        float dA2 = dA.x * dA.x + dA.y * dA.y + dA.z * dA.z;
        float dB2 = dB.x * dB.x + dB.y * dB.y + dB.z * dB.z;
        tangential_coeffs(M, dA2 / IsA, dB2 / IsB, Kt, Gt);
        Gn = M.Gn;
    } else {
        // effective masses from the pair; tc and the dampings follow from them (MWD_LAW_PHYSICAL)
        cp = (cpA + cpB) / 2.f;
        f3 dA = cp - cA, dB = cp - cB;
        float dA2 = dA.x * dA.x + dA.y * dA.y + dA.z * dA.z;
        float dB2 = dB.x * dB.x + dB.y * dB.y + dB.z * dB.z;
        const float im = imA + imB;
        const float mn = 1.f / im;
        const float tc2 = mn * M.Xn / M.Kn_f;
        const float tc = sqrtf(tc2);
        Gn = (-2.f) * mn * M.ln_en / tc;
        float C = im;
        if (imA != 0.f) C = C + dA2 / IsA;
        if (imB != 0.f) C = C + dB2 / IsB;
        const float mt = 1.f / C;
        Kt = mt * M.Xt / tc2;
        Gt = (-2.f) * mt * M.ln_et / tc;
    }
    if (dot(cB - cA, n) < 0.f) n = n * (-1.f);
    float nn = sqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
    n = n / nn;
    f3 disp_n = n * depth;
    f3 u = ((vA + cross(wA, cpA - cA)) - vB) - cross(wB, cpB - cB);
    f3 un = n * dot(u, n);
    f3 ut = u - un;
    float utn = sqrtf(ut.x * ut.x + ut.y * ut.y + ut.z * ut.z);
    f3 tij = mk3(0.f, 0.f, 0.f);
    if (utn != 0.f) tij = ut / utn;
    if (utn == 0.f && dtn != 0.f) tij = dt / dtn;
    f3 Fn = (disp_n * (-1.f)) * M.Kn_f - un * Gn;
    float Fnn = sqrtf(Fn.x * Fn.x + Fn.y * Fn.y + Fn.z * Fn.z);
    f3 Ft = dt * (-1.f) * Kt - ut * Gt;
    float Ftn = sqrtf(Ft.x * Ft.x + Ft.y * Ft.y + Ft.z * Ft.z);
    // two separate tests as in the reference, so a NaN norm takes the second (slip) branch
    const int coulomb = coulomb_compare(Ftn, Fnn, M);
    if (coulomb == 1) Ft = ((tij * Fnn) * (-1.f)) * M.mu_f;
    if (coulomb == 0) {
        float4 qi = qconj(qA);
        o.dt = qtrip(qA, dt, qi) + ut * M.dt_f;
    } else {
        f3 t = (((tij * Fnn) * M.mu_f) * (-1.f)) - ut * Gt;
        o.dt = (t * 1.f) / Kt;
    }
    f3 Ff = Ft + Fn;
    o.F = Fn;
    o.TA = cross(cp - cA, Ff);
    o.TB = cross(cp - cB, Ff * (-1.f));
}

// ------------------------------------------------------------------ pair sources

struct PairView {
    f3 cA, cB, vA, vB, wA, wB, dt;
    float4 qA;
    float IsA, IsB, dtn;
    int idA, idB, nA, nB;
    int wall;
};

// Both hulls of a pair into the group's staging area, 32 vertices of each at a time, all their loads in
// flight at once (a vertex per lane and round trip, the drop-in kernel waited for nine of them in a row:
// 122k candidate pairs 122 us).  at(v, i): vertex i of hull v.
template <int LPP, class At>
__device__ __forceinline__ void stage_hulls(float4* hA, int nA, float4* hB, int nB, int lane, At&& at)
{
    constexpr int U = LPP < 32 ? 32 / LPP : 2;
    const int most = max(nA, nB);
    for (int base = lane; base < most; base += U * LPP) {
        float4 x[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = base + u * LPP;
            x[u] = y[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < nA) x[u] = at(0, i);
            if (i < nB) y[u] = at(1, i);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = base + u * LPP;
            if (i < nA) hA[i] = x[u];
            if (i < nB) hB[i] = y[u];
        }
    }
}

// LPP: lanes of the group that stages the hulls (0: not staged)
template <int MODE, int LPP>
__device__ __forceinline__ bool load_pair(const NarrowArgs& a, int64_t P, PairView& p, float4* hA, float4* hB, int lane)
{
    if (MODE == 0) {
        const float* c;
        c = a.A_com + 3 * P; p.cA = mk3(c[0], c[1], c[2]);
        c = a.B_com + 3 * P; p.cB = mk3(c[0], c[1], c[2]);
        c = a.A_vel + 3 * P; p.vA = mk3(c[0], c[1], c[2]);
        c = a.B_vel + 3 * P; p.vB = mk3(c[0], c[1], c[2]);
        c = a.A_w + 3 * P; p.wA = mk3(c[0], c[1], c[2]);
        c = a.B_w + 3 * P; p.wB = mk3(c[0], c[1], c[2]);
        c = a.qA + 4 * P; p.qA = make_float4(c[0], c[1], c[2], c[3]);
        p.IsA = a.IsA[P];
        p.IsB = a.IsB[P];
        p.idA = a.A_id[P];
        p.idB = a.B_id[P];
        p.nA = a.A_nv[P];
        p.nB = a.B_nv[P];
        p.wall = (p.idA < a.n_wall || p.idB < a.n_wall) ? 1 : 0;
        const int64_t hb = a.hist_mode ? 4 * P : P;
        p.dt = mk3(a.hist_in[hb], a.hist_in[hb + 1], a.hist_in[hb + 2]);
        if (p.nA < 0 || p.nB < 0 || p.nA > a.hull_cap || p.nB > a.hull_cap) return false;
        const float* va = a.A_verts + P * a.V * 3;
        const float* vb = a.B_verts + P * a.V * 3;
        if constexpr (LPP > 0)
            stage_hulls<LPP>(hA, p.nA, hB, p.nB, lane, [&](int v, int i) {
                const float* x = (v ? vb : va) + 3 * i;
                return make_float4(x[0], x[1], x[2], 0.f);
            });
    } else {
        int2 pr = reinterpret_cast<const int2*>(a.pairs)[P];
        p.idA = pr.x;
        p.idB = pr.y;
        const double4 pa = reinterpret_cast<const double4*>(a.st.pos)[p.idA];
        const double4 pb = reinterpret_cast<const double4*>(a.st.pos)[p.idB];
        p.cA = mk3((float)pa.x, (float)pa.y, (float)pa.z);
        p.cB = mk3((float)pb.x, (float)pb.y, (float)pb.z);
        const float4* vel = reinterpret_cast<const float4*>(a.st.vel);
        const float4* w = reinterpret_cast<const float4*>(a.st.w);
        p.vA = xyz(vel[p.idA]);
        p.vB = xyz(vel[p.idB]);
        p.wA = xyz(w[p.idA]);
        p.wB = xyz(w[p.idB]);
        p.qA = reinterpret_cast<const float4*>(a.st.q)[p.idA];
        p.IsA = reinterpret_cast<const float4*>(a.st.inertia)[p.idA].w;
        p.IsB = reinterpret_cast<const float4*>(a.st.inertia)[p.idB].w;
        p.wall = ((a.st.info[p.idA] | a.st.info[p.idB]) & 1);
        p.dt = mk3(0.f, 0.f, 0.f);
        const int oa = a.st.vert_off[p.idA], ob = a.st.vert_off[p.idB];
        p.nA = a.st.vert_off[p.idA + 1] - oa;
        p.nB = a.st.vert_off[p.idB + 1] - ob;
        if (p.nA > a.hull_cap || p.nB > a.hull_cap) return false;
        if constexpr (LPP > 0) {
            const float4* wv = reinterpret_cast<const float4*>(a.st.world_verts);
            stage_hulls<LPP>(hA, p.nA, hB, p.nB, lane, [&](int v, int i) { return wv[(v ? ob : oa) + i]; });
        }
    }
    p.dtn = sqrtf(p.dt.x * p.dt.x + p.dt.y * p.dt.y + p.dt.z * p.dt.z);
    return true;
}

// Inverse masses of a pair's two rows for the physical law (0 for a wall row); the per-pair layout
// (MODE 0) carries no masses and only runs the reference law.
template <int MODE>
__device__ __forceinline__ void pair_inv_mass(const NarrowArgs& a, const PairView& p, const mwd_material& M,
                                              float& imA, float& imB)
{
    imA = 0.f;
    imB = 0.f;
    if (MODE == 0 || !M.physical) return;
    const float4* ii = reinterpret_cast<const float4*>(a.st.inv_inertia);
    if (!(a.st.info[p.idA] & 1)) imA = ii[p.idA].w;
    if (!(a.st.info[p.idB] & 1)) imB = ii[p.idB].w;
}

template <int MODE>
__device__ __forceinline__ void write_hist(const NarrowArgs& a, int64_t P, f3 v, float flag)
{
    if (MODE != 0) return;
    if (a.hist_mode) {
        float* h = a.hist_out + 4 * P;
        h[0] = v.x; h[1] = v.y; h[2] = v.z; h[3] = flag;
    } else {
        reinterpret_cast<float4*>(a.hist_stage)[P] = make_float4(v.x, v.y, v.z, flag);
        a.hist_wrote[P] = 1;
    }
}

template <int MODE>
__device__ __forceinline__ void accumulate(const NarrowArgs& a, const PairView& p, const ForceResult& fo)
{
    if (MODE == 0) {
        atomicAdd(a.force + 3 * p.idA + 0, fo.F.x);
        atomicAdd(a.force + 3 * p.idA + 1, fo.F.y);
        atomicAdd(a.force + 3 * p.idA + 2, fo.F.z);
        atomicAdd(a.force + 3 * p.idB + 0, -1 * fo.F.x);
        atomicAdd(a.force + 3 * p.idB + 1, -1 * fo.F.y);
        atomicAdd(a.force + 3 * p.idB + 2, -1 * fo.F.z);
        atomicAdd(a.torque + 3 * p.idA + 0, fo.TA.x);
        atomicAdd(a.torque + 3 * p.idA + 1, fo.TA.y);
        atomicAdd(a.torque + 3 * p.idA + 2, fo.TA.z);
        atomicAdd(a.torque + 3 * p.idB + 0, fo.TB.x);
        atomicAdd(a.torque + 3 * p.idB + 1, fo.TB.y);
        atomicAdd(a.torque + 3 * p.idB + 2, fo.TB.z);
    } else {
        float* F = a.st.force;
        float* T = a.st.torque;
        if (!(a.st.info[p.idA] & 1)) {
            atomicAdd(F + 4 * p.idA + 0, fo.F.x);
            atomicAdd(F + 4 * p.idA + 1, fo.F.y);
            atomicAdd(F + 4 * p.idA + 2, fo.F.z);
            atomicAdd(T + 4 * p.idA + 0, fo.TA.x);
            atomicAdd(T + 4 * p.idA + 1, fo.TA.y);
            atomicAdd(T + 4 * p.idA + 2, fo.TA.z);
        }
        if (!(a.st.info[p.idB] & 1)) {
            atomicAdd(F + 4 * p.idB + 0, -1 * fo.F.x);
            atomicAdd(F + 4 * p.idB + 1, -1 * fo.F.y);
            atomicAdd(F + 4 * p.idB + 2, -1 * fo.F.z);
            atomicAdd(T + 4 * p.idB + 0, fo.TB.x);
            atomicAdd(T + 4 * p.idB + 1, fo.TB.y);
            atomicAdd(T + 4 * p.idB + 2, fo.TB.z);
        }
    }
}

// GJK (.cu:996-1288) between its tetrahedron tests: three simplex points with their support indices (A | B << 8),
// the fourth one on a hit, and the next direction
struct GjkState {
    f3 S1, S2, S3, S4, d;
    int i1, i2, i3, i4;
    __device__ __forceinline__ void drop(int todel)  // the point (of 1, 2, 3) that S4 replaces, order kept
    {
        if (todel == 1) {
            S1 = S2;
            i1 = i2;
            S2 = S3;
            i2 = i3;
        } else if (todel == 2) {
            const f3 t = S1;
            const int it = i1;
            S1 = S3;
            i1 = i3;
            S2 = t;
            i2 = it;
        }
        S3 = S4;
        i3 = i4;
    }
};

constexpr int GJK_TESTS = 50;   // tetrahedron tests before the reference gives up (.cu:1104)
constexpr int GJK_OPEN = 2;     // not decided yet

// The first three queries, by one lane or by a warp: 0 separated, else GJK_OPEN
template <class Hulls>
__device__ __forceinline__ int gjk_start(const Hulls& h, f3 cA, f3 cB, GjkState& g, int& queries)
{
    const f3 d1 = cB - cA;
    const f3 d2 = d1 * (-1.f);
    int a1, b1, a2, b2, a3, b3, coll = -1;
    h.both(d1, g.S1, a1, b1, g.S2, a2, b2);
    queries = 1;
    if (dot(d1, g.S1) < 0.f) return 0;
    queries = 2;
    if (dot(d2, g.S2) < 0.f) return 0;
    f3 d3;
    seg_test(g.S1, g.S2, coll, d3);
    if (coll == 0) return 0;
    h.query(d3, g.S3, a3, b3);
    queries = 3;
    if (dot(d3, g.S3) < 0.f) return 0;
    tri_test(g.S1, g.S2, g.S3, coll, g.d);
    g.i1 = a1 | (b1 << 8);
    g.i2 = a2 | (b2 << 8);
    g.i3 = a3 | (b3 << 8);
    return coll == 0 ? 0 : GJK_OPEN;
}

// Tetrahedron tests from..to - 1, by one lane or by a warp (LPP 1 or 32): 0 separated, 1 in contact, else GJK_OPEN
template <int LPP, class Hulls>
__device__ __forceinline__ int gjk_search(const Hulls& h, GjkState& g, int from, int to, int& queries)
{
    for (int zz = from; zz < to; ++zz) {
        int a4, b4, coll = -1, todel = 0;
        h.query(g.d, g.S4, a4, b4);
        g.i4 = a4 | (b4 << 8);
        ++queries;
        if (dot(g.d, g.S4) < 0.f) return 0;
        if (g.S4.x == 0.f && g.S4.y == 0.f && g.S4.z == 0.f) return 1;
        if constexpr (LPP >= 4) tet_test_lanes<LPP>(g.S1, g.S2, g.S3, g.S4, coll, g.d, todel);
        else tet_test(g.S1, g.S2, g.S3, g.S4, coll, g.d, todel);
        if (coll >= 0) return coll;
        g.drop(todel);
    }
    return GJK_OPEN;
}

// The pairs (one per aligned group of LPP lanes) still open after `from` tests, one after another by the whole
// warp: an iteration of the warp takes a fifth of the time of one of a lane or of a group, and a pass ends
// with its slowest pair, which runs 50.  open: this lane's pair is one of them.
template <int LPP>
__device__ __forceinline__ void gjk_finish(const float4* hA, int nA, const float4* hB, int nB, GjkState& g, int from,
                                           bool open, int& out, int& queries)
{
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (unsigned todo = __ballot_sync(ALL, open && (lane & (LPP - 1)) == 0); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        auto from3 = [&](f3 v) {
            return mk3(__shfl_sync(ALL, v.x, src), __shfl_sync(ALL, v.y, src), __shfl_sync(ALL, v.z, src));
        };
        GjkState w;
        w.S1 = from3(g.S1);
        w.S2 = from3(g.S2);
        w.S3 = from3(g.S3);
        w.d = from3(g.d);
        w.i1 = __shfl_sync(ALL, g.i1, src);
        w.i2 = __shfl_sync(ALL, g.i2, src);
        w.i3 = __shfl_sync(ALL, g.i3, src);
        const float4* a = reinterpret_cast<const float4*>(__shfl_sync(ALL, reinterpret_cast<unsigned long long>(hA), src));
        const float4* b = reinterpret_cast<const float4*>(__shfl_sync(ALL, reinterpret_cast<unsigned long long>(hB), src));
        WarpHulls h;
        h.load(a, __shfl_sync(ALL, nA, src), b, __shfl_sync(ALL, nB, src));
        int more = 0;
        const int o = gjk_search<32>(h, w, from, GJK_TESTS, more);
        if ((lane & ~(LPP - 1)) == src) {
            g = w;
            out = o == GJK_OPEN ? -1 : o;
            queries += more;
        }
    }
}

__device__ __forceinline__ void gjk_record(const GjkState& g, SimplexRec& rec)
{
    rec.S[0] = f4(g.S1, 0.f); rec.S[1] = f4(g.S2, 0.f); rec.S[2] = f4(g.S3, 0.f); rec.S[3] = f4(g.S4, 0.f);
    auto pack = [&](int shift) {
        return (uint32_t)((g.i1 >> shift) & 0xff) | (uint32_t)((g.i2 >> shift) & 0xff) << 8 |
               (uint32_t)((g.i3 >> shift) & 0xff) << 16 | (uint32_t)((g.i4 >> shift) & 0xff) << 24;
    };
    rec.ia = pack(0);
    rec.ib = pack(8);
}

// ------------------------------------------------------------------ GJK by lane groups in lockstep
//
// The groups of a warp (LPP = 4, 8, 16 or 32 lanes, a pair each) run GJK together: every exchange between
// lanes names the whole warp, so one instruction serves all the pairs of the warp until the last of them
// is decided.  (Groups that exchange under masks of their own run one after another from the first
// exchange on: 13,000 candidates of a pour took 20 us with them.)

// (largest v, then smallest i) over aligned runs of H lanes
template <int H>
__device__ __forceinline__ int run_argmax(float v, int i)
{
    const unsigned k = fkey(v);
    unsigned m = k;
#pragma unroll
    for (int o = H / 2; o > 0; o /= 2) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    int w = k == m ? i : 0x7fffffff;
#pragma unroll
    for (int o = H / 2; o > 0; o /= 2) w = min(w, __shfl_xor_sync(0xffffffffu, w, o));
    return w;
}

// the hulls of a group, read in place or staged: the lower half of its lanes scans A's vertices, the upper
// half B's
template <int LPP>
struct LockHulls {
    const float4 *hA, *hB;
    int nA, nB;
    // support() of the groups that are on
    __device__ __forceinline__ void query(f3 d, bool on, f3& s, int& ia, int& ib) const
    {
        constexpr int H = LPP / 2;
        const int lane = threadIdx.x & 31, g0 = lane & ~(LPP - 1);
        const bool onB = (lane & H) != 0;
        const float4* h = onB ? hB : hA;
        const int n = !on ? 0 : onB ? nB : nA;
        const f3 e = onB ? d * (-1.f) : d;
        float best = -1e30f;
        int at = 0;
#pragma unroll 4
        for (int i = lane & (H - 1); i < n; i += H) {
            const float4 v = h[i];
            const float t = e.x * v.x + e.y * v.y + e.z * v.z;
            if (t > best) { best = t; at = i; }
        }
        at = run_argmax<H>(best, at);
        const int wA = __shfl_sync(0xffffffffu, at, g0), wB = __shfl_sync(0xffffffffu, at, g0 + H);
        if (on) {  // (a decided group keeps what it has)
            ia = wA;
            ib = wB;
            const float4 a = hA[ia], b = hB[ib];
            s = mk3(a.x - b.x, a.y - b.y, a.z - b.z);
        }
    }
    // the queries in the directions d and -d: the second one's products are the first one's negated (exactly)
    __device__ __forceinline__ void both(f3 d, bool on, f3& S1, int& a1, int& b1, f3& S2, int& a2, int& b2) const
    {
        constexpr int H = LPP / 2;
        const int lane = threadIdx.x & 31, g0 = lane & ~(LPP - 1);
        const bool onB = (lane & H) != 0;
        const float4* h = onB ? hB : hA;
        const int n = !on ? 0 : onB ? nB : nA;
        const f3 e = onB ? d * (-1.f) : d;
        float best = -1e30f, opp = -1e30f;
        int at = 0, oat = 0;
#pragma unroll 4
        for (int i = lane & (H - 1); i < n; i += H) {
            const float4 v = h[i];
            const float t = e.x * v.x + e.y * v.y + e.z * v.z;
            if (t > best) { best = t; at = i; }
            if (-t > opp) { opp = -t; oat = i; }
        }
        at = run_argmax<H>(best, at);
        oat = run_argmax<H>(opp, oat);
        a1 = __shfl_sync(0xffffffffu, at, g0);
        b1 = __shfl_sync(0xffffffffu, at, g0 + H);
        a2 = __shfl_sync(0xffffffffu, oat, g0);
        b2 = __shfl_sync(0xffffffffu, oat, g0 + H);
        if (on) {
            const float4 p1 = hA[a1], q1 = hB[b1], p2 = hA[a2], q2 = hB[b2];
            S1 = mk3(p1.x - q1.x, p1.y - q1.y, p1.z - q1.z);
            S2 = mk3(p2.x - q2.x, p2.y - q2.y, p2.z - q2.z);
        }
    }
};

// tetrahedron tests that the groups of a warp run in lockstep before the whole warp takes over what is still
// open (2 and 8 measured the same within 3%)
constexpr int GJK_GROUP_TESTS = 4;

// GJK of every group that is on, by a full warp: 0 separated, 1 in contact, -1 undecided after 50 tests;
// queries: the group's support queries
template <int LPP>
__device__ __forceinline__ int gjk_lockstep(const LockHulls<LPP>& h, bool on, f3 cA, f3 cB, GjkState& g, int& queries)
{
    constexpr unsigned ALL = 0xffffffffu;
    int a1, b1, a2, b2, a3 = 0, b3 = 0, a4 = 0, b4 = 0, coll = -1, out = 0;
    g.S1 = g.S2 = g.S3 = g.S4 = g.d = mk3(0.f, 0.f, 0.f);
    f3 d3 = g.S1;
    queries = 0;
    const f3 d1 = cB - cA;
    const f3 d2 = d1 * (-1.f);
    h.both(d1, on, g.S1, a1, b1, g.S2, a2, b2);
    if (on) {
        queries = 1;
        on = !(dot(d1, g.S1) < 0.f);
        if (on) {
            queries = 2;
            on = !(dot(d2, g.S2) < 0.f);
        }
        if (on) {
            seg_test(g.S1, g.S2, coll, d3);
            on = coll != 0;
        }
    }
    if (!__any_sync(ALL, on)) return 0;
    h.query(d3, on, g.S3, a3, b3);
    g.i1 = a1 | (b1 << 8);
    g.i2 = a2 | (b2 << 8);
    g.i3 = a3 | (b3 << 8);
    if (on) {
        ++queries;
        on = !(dot(d3, g.S3) < 0.f);
        if (on) {
            tri_test(g.S1, g.S2, g.S3, coll, g.d);
            on = coll != 0;
        }
    }
    for (int zz = 0; zz < GJK_GROUP_TESTS && __any_sync(ALL, on); ++zz) {
        h.query(g.d, on, g.S4, a4, b4);
        bool hit = false;
        if (on) {
            ++queries;
            g.i4 = a4 | (b4 << 8);
            on = !(dot(g.d, g.S4) < 0.f);
            hit = g.S4.x == 0.f && g.S4.y == 0.f && g.S4.z == 0.f;
        }
        f3 n;
        int todel;
        tet_test_lanes<LPP>(g.S1, g.S2, g.S3, g.S4, coll, n, todel);
        if (on) {
            hit = hit || coll == 1;
            if (hit) out = 1;
            on = !hit && coll != 0;
        }
        if (on) {
            g.d = n;
            g.drop(todel);
        }
    }
    gjk_finish<LPP>(h.hA, h.nA, h.hB, h.nB, g, GJK_GROUP_TESTS, on, out, queries);
    return out;
}

// ------------------------------------------------------------------ single-pass narrow phase
// GJK by the groups of a warp, each on its own pair, then EPA by the whole warp on one after another of
// the pairs they found in contact; the lane that leads a pair's group evaluates its force.
template <int LPP, int MODE>
__device__ __forceinline__ void narrow_pairs(const NarrowArgs& a, int64_t P, bool in, const Group<LPP>& g,
                                             WarpEpaMem& em, float4* hA, float4* hB)
{
    const int lane = threadIdx.x & 31;
    PairView p;
    Work3 wk = {0u, 0u, 0u};
    GjkState gs;
    int out = 0;  // 0 separated, 1 in contact, -1 undecided
    bool ok = false;
    if (in) ok = load_pair<MODE, LPP>(a, P, p, hA, hB, g.lane);
    __syncwarp();
    int queries;
    out = gjk_lockstep<LPP>(LockHulls<LPP>{hA, hB, p.nA, p.nB}, ok, p.cA, p.cB, gs, queries);
    wk.queries = (uint32_t)queries;
    wk.dots = ok ? (uint32_t)queries * (uint32_t)(p.nA + p.nB) : 0u;
    EpaResult er;
    er.status = 0;
    for (unsigned hits = __ballot_sync(0xffffffffu, out == 1 && g.lane == 0); hits; hits &= hits - 1) {
        const int src = __ffs(hits) - 1;
        if (lane == src) {
            SimplexRec rec;
            gjk_record(gs, rec);
            for (int k = 0; k < 4; ++k) em.pv[k] = rec.S[k];
            em.ft[0] = rec.ia;
            em.ft[1] = rec.ib;
        }
        const float4* ha = hA + (src / LPP - lane / LPP) * 2 * a.hull_cap;  // the group's staged hulls
        WarpHulls h;
        h.load(ha, __shfl_sync(0xffffffffu, p.nA, src), ha + a.hull_cap, __shfl_sync(0xffffffffu, p.nB, src));
        __syncwarp();
        const f3 S1 = xyz(em.pv[0]), S2 = xyz(em.pv[1]), S3 = xyz(em.pv[2]);
        f3 S4 = xyz(em.pv[3]);
        const uint32_t ia = em.ft[0], ib = em.ft[1];
        WarpEpaOut o;
        epa_from_simplex(em, h, S1, S2, S3, S4, ia, ib, o);
        if (lane == src) {
            wk.queries += (uint32_t)o.queries;
            wk.faces += (uint32_t)o.faces;
            wk.dots += (uint32_t)o.queries * (uint32_t)(p.nA + p.nB);
            const int ta = ft_v(o.t, 0), tb = ft_v(o.t, 1), tc = ft_v(o.t, 2);
            er.status = o.status;
            er.depth = o.face.w;
            epa_contact(xyz(em.pv[ta]), xyz(em.pv[tb]), xyz(em.pv[tc]), em.pab[ta], em.pab[tb], em.pab[tc], hA, hB,
                        xyz(o.face), er);
        }
        __syncwarp();
    }
    if (!in || g.lane != 0) return;
    if (!ok) {
        set_status(a.status, MWD_ST_BAD_SHAPE);
        if (a.collision) a.collision[P] = -1;
        return;
    }
    const bool resolved = out == 1;
    ForceResult fo;
    fo.F = fo.TA = fo.TB = mk3(0.f, 0.f, 0.f);
    fo.dt = p.dt;
    if (resolved) {
        const mwd_material& M = MODE == 0 ? a.mat[p.wall] : a.scenes[a.st.info[p.idA] >> 1].mat[p.wall];
        float imA, imB;
        pair_inv_mass<MODE>(a, p, M, imA, imB);
        contact_force(p.cA, p.cB, er.depth, er.n, er.cpA, er.cpB, M, p.vA, p.vB, p.wA, p.wB, p.dt, p.qA, p.dtn, p.IsA,
                      p.IsB, imA, imB, fo);
    }
    set_status(a.status, out == -1 ? (uint32_t)MWD_ST_GJK_NOCONV : er.status);
    if (a.work_counters) {
        atomicAdd(a.work_counters + 0, (unsigned long long)wk.dots);
        atomicAdd(a.work_counters + 1, (unsigned long long)wk.faces);
        atomicAdd(a.work_counters + 2, (unsigned long long)wk.queries);
    }
    if (a.collision) a.collision[P] = out;
    if (out == 0) {
        write_hist<MODE>(a, P, mk3(0.f, 0.f, 0.f), 0.f);
    } else {
        if (resolved) write_hist<MODE>(a, P, fo.dt, 1.f);
        accumulate<MODE>(a, p, fo);
    }
    if (a.diag) {
        float* dg = a.diag + 10 * P;
        if (resolved) {
            dg[0] = er.depth;
            dg[1] = er.n.x; dg[2] = er.n.y; dg[3] = er.n.z;
            dg[4] = er.cpA.x; dg[5] = er.cpA.y; dg[6] = er.cpA.z;
            dg[7] = er.cpB.x; dg[8] = er.cpB.y; dg[9] = er.cpB.z;
        } else {
            for (int k = 0; k < 10; ++k) dg[k] = 0.f;
        }
    }
    if (a.face_ids) {
        int* fid = a.face_ids + 6 * P;
        for (int k = 0; k < 3; ++k) {
            fid[k] = resolved ? er.fa[k] : -1;
            fid[3 + k] = resolved ? er.fb[k] : -1;
        }
    }
}

template <int LPP, int MODE>
__global__ void __launch_bounds__(NARROW_THREADS) narrow_kernel(NarrowArgs a)
{
    extern __shared__ float4 smem[];
    constexpr int GPB = NARROW_THREADS / LPP;
    const int grp = threadIdx.x / LPP;
    Group<LPP> g;
    g.lane = threadIdx.x % LPP;
    g.mask = LPP == 32 ? 0xffffffffu : (((1u << LPP) - 1u) << ((threadIdx.x & 31) / LPP * LPP));
    WarpEpaMem& em = reinterpret_cast<WarpEpaMem*>(smem)[threadIdx.x / 32];
    float4* hA = reinterpret_cast<float4*>(reinterpret_cast<WarpEpaMem*>(smem) + NARROW_THREADS / 32) +
                 (size_t)grp * 2 * a.hull_cap;
    float4* hB = hA + a.hull_cap;
    int64_t n = a.n_pairs;
    if (MODE == 1) {
        int64_t m = *a.n_pairs_dev;
        n = m < a.pair_cap ? m : a.pair_cap;
        // sphere pre-test (spheres_apart), LPP candidate pairs at a time per group (one per lane); pairs it
        // settles get the reference's outcome (collision 0, no force) without running GJK
        const double4* pos = reinterpret_cast<const double4*>(a.st.pos);
        const int2* pairs = reinterpret_cast<const int2*>(a.pairs);
        const int64_t stride = (int64_t)gridDim.x * GPB * LPP;
        for (int64_t b0 = (int64_t)blockIdx.x * GPB * LPP; b0 < n; b0 += stride) {
            const int64_t base = b0 + (int64_t)grp * LPP;
            const int64_t Pl = base + g.lane;
            bool live = false;
            if (Pl < n) {
                const int2 pr = pairs[Pl];
                live = !spheres_apart(pos[pr.x], pos[pr.y]);
                if (!live && a.collision) a.collision[Pl] = 0;
            }
            unsigned m = g.ballot(live);
            while (__any_sync(0xffffffffu, m != 0)) {
                const int l = __ffs(m) - 1;
                narrow_pairs<LPP, MODE>(a, base + l, m != 0, g, em, hA, hB);
                m &= m - 1;
                __syncwarp();
            }
        }
    } else {
        for (int64_t base = (int64_t)blockIdx.x * GPB; base < n; base += (int64_t)gridDim.x * GPB) {
            narrow_pairs<LPP, MODE>(a, base + grp, base + grp < n, g, em, hA, hB);
            __syncwarp();
        }
    }
}

// ------------------------------------------------------------------ two-pass narrow phase (table mode)
//
// Pass 1 (gjk_pass_kernel) runs the sphere pre-test and GJK on every candidate pair with the hulls
// read straight from the world-vertex table (no shared memory, few registers, many resident warps);
// separated and undecided pairs are finished there.  Pairs GJK finds in contact append the simplex
// it stopped on to a compact list.  Pass 2 (epa_pass_kernel) continues exactly where pass 1
// stopped -- CorrectFlat, EPA, force -- for the listed pairs only, a warp each.
// The operation sequence per pair is the single-pass kernel's.

// The outcome of GJK on pair P: its contact flag, and for a pair in contact its simplex in the EPA list
__device__ __forceinline__ void gjk_outcome(const NarrowArgs& a, int64_t P, bool ok, int out, const GjkState& g,
                                            int queries, int verts)
{
    if (!ok) {
        set_status(a.status, MWD_ST_BAD_SHAPE);
        if (a.collision) a.collision[P] = -1;
    } else if (out == 1) {
        const int slot = atomicAdd(a.epa_count, 1);
        if (slot < a.epa_cap) {
            SimplexRec rec;
            gjk_record(g, rec);
            rec.P = P;
            reinterpret_cast<SimplexRec*>(a.epa_rec)[slot] = rec;
        } else {
            set_status(a.status, MWD_ST_PAIR_OVERFLOW);
        }
        if (a.collision) a.collision[P] = 1;
    } else {
        // undecided pairs add zero force in the reference (.cu:1304-1319): nothing to add
        if (out == -1) set_status(a.status, MWD_ST_GJK_NOCONV);
        if (a.collision) a.collision[P] = out;
    }
    if (a.work_counters) {
        atomicAdd(a.work_counters + 0, (unsigned long long)queries * (unsigned long long)verts);
        atomicAdd(a.work_counters + 2, (unsigned long long)queries);
    }
}

// a pair's hulls and centres in the tables
struct TablePair {
    const float4 *hA, *hB;
    int nA, nB;
    f3 cA, cB;
    bool ok;
    __device__ __forceinline__ void load(const NarrowArgs& a, int64_t P)
    {
        const double4* pos = reinterpret_cast<const double4*>(a.st.pos);
        const float4* wv = reinterpret_cast<const float4*>(a.st.world_verts);
        const int2 pr = reinterpret_cast<const int2*>(a.pairs)[P];
        const double4 pa = pos[pr.x], pb = pos[pr.y];
        cA = mk3((float)pa.x, (float)pa.y, (float)pa.z);
        cB = mk3((float)pb.x, (float)pb.y, (float)pb.z);
        const int oa = a.st.vert_off[pr.x], ob = a.st.vert_off[pr.y];
        nA = a.st.vert_off[pr.x + 1] - oa;
        nB = a.st.vert_off[pr.y + 1] - ob;
        hA = wv + oa;
        hB = wv + ob;
        ok = nA <= a.hull_cap && nB <= a.hull_cap;
    }
};

// GJK on pair P (if any: on) by each group: one lane by itself, a group of a warp in lockstep, or a warp,
// which holds the hulls in registers
template <int LPP>
__device__ __forceinline__ void gjk_pair(const NarrowArgs& a, int64_t P, bool on)
{
    TablePair p;
    p.hA = p.hB = nullptr;
    p.nA = p.nB = 0;
    p.cA = p.cB = mk3(0.f, 0.f, 0.f);
    p.ok = false;
    if (on) p.load(a, P);
    GjkState g;
    int out = 0, queries = 0;
    if constexpr (LPP == 32) {
        if (p.ok) {
            WarpHulls h;
            h.load(p.hA, p.nA, p.hB, p.nB);
            out = gjk_start(h, p.cA, p.cB, g, queries);
            if (out == GJK_OPEN) out = gjk_search<32>(h, g, 0, GJK_TESTS, queries);
            if (out == GJK_OPEN) out = -1;
        }
    } else if constexpr (LPP == 1) {
        if (p.ok) {
            const LaneHulls h = {p.hA, p.hB, p.nA, p.nB};
            out = gjk_start(h, p.cA, p.cB, g, queries);
            if (out == GJK_OPEN) out = gjk_search<1>(h, g, 0, GJK_TESTS, queries);
            if (out == GJK_OPEN) out = -1;
        }
    } else {
        out = gjk_lockstep<LPP>(LockHulls<LPP>{p.hA, p.hB, p.nA, p.nB}, p.ok, p.cA, p.cB, g, queries);
    }
    if (on && (threadIdx.x & (LPP - 1)) == 0) gjk_outcome(a, P, p.ok, out, g, queries, p.nA + p.nB);
    if (LPP > 1) __syncwarp();
}

// The pair list over the grid's warps, 32 / LPP pairs each at a time.  Where the broad phase has not dropped
// the pairs whose spheres are apart (a.pre_culled), they are tested here first, a lane per candidate:
// 32 candidates per warp when there are that many, else as many as the warp has groups.
template <int LPP, int BT>
__device__ __forceinline__ void gjk_stride(const NarrowArgs& a, int64_t n)
{
    if constexpr (LPP == 1) {
        // every lane at its own pace (meeting the others at each pair, and handing its slow pairs to the warp,
        // a 256-scene batch's pass took 170 us instead of 152)
        const int64_t step = (int64_t)gridDim.x * BT;
        for (int64_t P = (int64_t)blockIdx.x * BT + threadIdx.x; P < n; P += step) {
            bool live = true;
            if (!a.pre_culled) {
                const double4* pos = reinterpret_cast<const double4*>(a.st.pos);
                const int2 pr = reinterpret_cast<const int2*>(a.pairs)[P];
                live = !spheres_apart(pos[pr.x], pos[pr.y]);
                if (!live && a.collision) a.collision[P] = 0;
            }
            if (live) gjk_pair<1>(a, P, true);
        }
        return;
    }
    constexpr int G = 32 / LPP;
    const int lane = threadIdx.x & 31, grp = lane / LPP;
    const int64_t warps = (int64_t)gridDim.x * (BT / 32);
    const int chunk = !a.pre_culled && n > warps * G ? 32 : G;
    for (int64_t base = ((int64_t)blockIdx.x * (BT / 32) + threadIdx.x / 32) * chunk; base < n; base += warps * chunk) {
        bool live = lane < chunk && base + lane < n;
        if (live && !a.pre_culled) {
            const double4* pos = reinterpret_cast<const double4*>(a.st.pos);
            const int2 pr = reinterpret_cast<const int2*>(a.pairs)[base + lane];
            live = !spheres_apart(pos[pr.x], pos[pr.y]);
            if (!live && a.collision) a.collision[base + lane] = 0;
        }
        unsigned m = __ballot_sync(0xffffffffu, live);
        while (m) {
            // the next G survivors, one per group
            unsigned mine = m;
            for (int k = 0; k < grp; ++k) mine &= mine - 1;
            gjk_pair<LPP>(a, base + (mine ? __ffs(mine) - 1 : 0), mine != 0);
            for (int k = 0; k < G; ++k) m &= m - 1;
        }
    }
}

// BT threads per block (64, 128 or 256: the autotuner's block-size knob), registers capped so that
// 896 threads per SM stay resident with one lane per pair (the 256-scene step measured 0.716 ms at
// 7 blocks of 128, 0.720 at 8 and 0.726 at 6) and 768 with lane groups
template <int LPP, int BT>
__global__ void __launch_bounds__(BT, (LPP == 1 ? 896 : 768) / BT) gjk_pass_kernel(NarrowArgs a)
{
    pdl_wait();
    pdl_launch_dependents();
    const int64_t m = *a.n_pairs_dev;
    const int64_t n = m < a.pair_cap ? m : a.pair_cap;
    // as many warps as pairs: a warp for each, whatever LPP (both passes on 4,200 random pairs 59 us and on 5,000,
    // past the line of one lane per pair, 87; groups of eight 64 and 67)
    if (LPP < 32 && n <= (int64_t)gridDim.x * (BT / 32)) gjk_stride<32, BT>(a, n);
    else gjk_stride<LPP, BT>(a, n);
}

// ------------------------------------------------------------------ persistent tangential history
// Open-addressing table keyed by the unordered pair (lower id << 32 | higher id; 0 = empty), linear
// probing, the MurmurHash3 64-bit finaliser as the hash.  Values are stored in the (lower, higher)
// orientation: a pair listed the other way round reads and writes the negated displacement.
__device__ __forceinline__ unsigned long long hist_key(int a, int b)
{
    const unsigned lo = (unsigned)(a < b ? a : b), hi = (unsigned)(a < b ? b : a);
    return ((unsigned long long)lo << 32) | hi;
}
__device__ __forceinline__ unsigned long long hist_hash(unsigned long long k)
{
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}
__device__ __forceinline__ f3 hist_get(const NarrowArgs& a, int A, int B)
{
    const int par = *a.hist_parity & 1;
    const unsigned long long* K = a.hist_keys + (size_t)par * a.hist_cap;
    const float4* V = a.hist_vals + (size_t)par * a.hist_cap;
    const unsigned long long key = hist_key(A, B);
    const unsigned long long m = (unsigned long long)a.hist_cap - 1;
    unsigned long long slot = hist_hash(key) & m;
    for (int64_t probe = 0; probe < a.hist_cap; ++probe) {
        const unsigned long long k = K[slot];
        if (k == key) {
            const f3 v = xyz(V[slot]);
            return A < B ? v : v * (-1.f);
        }
        if (k == 0ull) break;
        slot = (slot + 1) & m;
    }
    return mk3(0.f, 0.f, 0.f);
}
__device__ __forceinline__ void hist_put(const NarrowArgs& a, int A, int B, f3 dt)
{
    const int par = (*a.hist_parity & 1) ^ 1;
    unsigned long long* K = a.hist_keys + (size_t)par * a.hist_cap;
    float4* V = a.hist_vals + (size_t)par * a.hist_cap;
    const unsigned long long key = hist_key(A, B);
    const unsigned long long m = (unsigned long long)a.hist_cap - 1;
    unsigned long long slot = hist_hash(key) & m;
    for (int64_t probe = 0; probe < a.hist_cap; ++probe) {
        const unsigned long long prev = atomicCAS(K + slot, 0ull, key);
        if (prev == 0ull || prev == key) {
            V[slot] = f4(A < B ? dt : dt * (-1.f), 0.f);
            return;
        }
        slot = (slot + 1) & m;
    }
    set_status(a.status, MWD_ST_HIST_OVERFLOW);
}

// empties the table this narrow phase writes
__global__ void hist_clear_kernel(NarrowArgs a)
{
    pdl_wait();
    pdl_launch_dependents();
    const int par = (*a.hist_parity & 1) ^ 1;
    unsigned long long* K = a.hist_keys + (size_t)par * a.hist_cap;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.hist_cap; i += (int64_t)gridDim.x * blockDim.x)
        K[i] = 0ull;
}

// the table just written is read by the next narrow phase
__global__ void hist_flip_kernel(NarrowArgs a)
{
    pdl_wait();
    pdl_launch_dependents();
    if (threadIdx.x == 0 && blockIdx.x == 0) *a.hist_parity ^= 1;
}

// the EPA queue's smallest claim, and the fraction of the remaining records per group a claim takes
constexpr int EPA_CLAIM = 2;
constexpr int EPA_GUIDE = 4;

// A finished EPA whose force is still to be evaluated: the final face's normal and depth, its three
// polytope vertices with their support indices, and the record
struct EpaDone {
    float4 nd;       // normal, depth
    float4 a, b, c;  // vertices; w: support indices of a and b, of c and the status bits, the record
};

// The forces of up to 32 finished records, one per lane
__device__ __noinline__ void epa_flush(const NarrowArgs& a, const EpaDone* done, int n)
{
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (lane < n) {
        const EpaDone e = done[lane];
        const uint32_t pab = __float_as_uint(e.a.w), pcs = __float_as_uint(e.b.w);
        const int64_t i = (int64_t)__float_as_uint(e.c.w);
        const int64_t P = reinterpret_cast<const SimplexRec*>(a.epa_rec)[i].P;
        PairView p;
        load_pair<1, 0>(a, P, p, nullptr, nullptr, 0);
        const float4* wv = reinterpret_cast<const float4*>(a.st.world_verts);
        EpaResult er;
        er.depth = e.nd.w;
        epa_contact(xyz(e.a), xyz(e.b), xyz(e.c), (int)(pab & 0xffffu), (int)(pab >> 16), (int)(pcs & 0xffffu),
                    wv + a.st.vert_off[p.idA], wv + a.st.vert_off[p.idB], xyz(e.nd), er);
        if (a.hist_keys) {
            p.dt = hist_get(a, p.idA, p.idB);
            p.dtn = sqrtf(p.dt.x * p.dt.x + p.dt.y * p.dt.y + p.dt.z * p.dt.z);
        }
        const mwd_material& M = a.scenes[a.st.info[p.idA] >> 1].mat[p.wall];
        ForceResult fo;
        float imA, imB;
        pair_inv_mass<1>(a, p, M, imA, imB);
        contact_force(p.cA, p.cB, er.depth, er.n, er.cpA, er.cpB, M, p.vA, p.vB, p.wA, p.wB, p.dt, p.qA, p.dtn,
                      p.IsA, p.IsB, imA, imB, fo);
        set_status(a.status, pcs >> 16);
        if (a.hist_keys) hist_put(a, p.idA, p.idB, fo.dt);
        if (a.det_out) {
            float4* o = a.det_out + 3 * i;
            o[0] = f4(fo.F, 0.f);
            o[1] = f4(fo.TA, 0.f);
            o[2] = f4(fo.TB, 0.f);
        } else {
            accumulate<1>(a, p, fo);
        }
        if (a.face_ids) {
            int* fid = a.face_ids + 6 * P;
            for (int k = 0; k < 3; ++k) {
                fid[k] = er.fa[k];
                fid[3 + k] = er.fb[k];
            }
        }
    }
    __syncwarp();
}

// BT threads per block, registers capped so that 640 threads per SM stay resident (5 blocks of 128)
template <int BT>
__global__ void __launch_bounds__(BT, 640 / BT) epa_pass_kernel(const __grid_constant__ NarrowArgs a)
{
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ float4 smem[];
    constexpr int W = BT / 32;
    const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    WarpEpaMem& em = reinterpret_cast<WarpEpaMem*>(smem)[warp];
    EpaDone* done = reinterpret_cast<EpaDone*>(reinterpret_cast<WarpEpaMem*>(smem) + W) + 32 * warp;
    const float4* wv = reinterpret_cast<const float4*>(a.st.world_verts);
    const SimplexRec* recs = reinterpret_cast<const SimplexRec*>(a.epa_rec);
    const int cnt = *a.epa_count;
    const int m = (int64_t)cnt < a.epa_cap ? cnt : (int)a.epa_cap;
    // Persistent over a work queue (guided self-scheduling): every warp first takes a fixed share of
    // the records, interleaved with the others' (all of them when there are no more records than
    // warps: no atomic at all); the rest are claimed from the queue in pieces of a quarter of what is
    // left per warp, so that the warps that finish early take over the work of the others and the
    // pass ends with its last record rather than with the unluckiest fixed share.  (Record counts are
    // int32.)
    const int G = (int)gridDim.x * W;
    const int share = m <= G ? 1 : (m / (2 * G) > 1 ? m / (2 * G) : 1);
    const int fixed = m <= G ? m : G * share;
    unsigned long long* next = epa_queue(a);
    // records i, i + step, ... below e: first the fixed share (step G), then each claimed piece (step 1)
    int i = (int)blockIdx.x * W + warp, step = G, e = fixed;
    int seen = 0;  // queue position after this warp's last claim
    int nd = 0;    // finished records whose forces are still to be evaluated
    Work3 wk = {0u, 0u, 0u};
    unsigned long long dots = 0;
    for (;;) {
        if (i >= e) {
            if (fixed >= m) break;
            int size = (m - fixed - seen) / (EPA_GUIDE * G);
            if (size < EPA_CLAIM) size = EPA_CLAIM;
            const int64_t b = (int64_t)fixed + claim(next, size);
            if (b >= m) break;
            i = (int)b;
            step = 1;
            e = b + size < m ? (int)b + size : m;
            seen = i - fixed + size;
        }
        const SimplexRec rec = recs[i];
        const int2 pr = reinterpret_cast<const int2*>(a.pairs)[rec.P];
        const int oa = a.st.vert_off[pr.x], ob = a.st.vert_off[pr.y];
        WarpHulls h;
        h.load(wv + oa, a.st.vert_off[pr.x + 1] - oa, wv + ob, a.st.vert_off[pr.y + 1] - ob);
        WarpEpaOut o;
        epa_from_simplex(em, h, xyz(rec.S[0]), xyz(rec.S[1]), xyz(rec.S[2]), xyz(rec.S[3]), rec.ia, rec.ib, o);
        wk.queries += (uint32_t)o.queries;
        wk.faces += (uint32_t)o.faces;
        dots += (unsigned long long)o.queries * (unsigned)(h.nA + h.nB);
        if (lane == 0) {
            const int ta = ft_v(o.t, 0), tb = ft_v(o.t, 1), tc = ft_v(o.t, 2);
            EpaDone& d = done[nd];
            d.nd = o.face;
            d.a = f4(xyz(em.pv[ta]), __uint_as_float((uint32_t)em.pab[ta] | ((uint32_t)em.pab[tb] << 16)));
            d.b = f4(xyz(em.pv[tb]), __uint_as_float((uint32_t)em.pab[tc] | (o.status << 16)));
            d.c = f4(xyz(em.pv[tc]), __uint_as_float((uint32_t)i));
        }
        if (++nd == 32) {
            epa_flush(a, done, nd);
            nd = 0;
        }
        i += step;
    }
    if (nd) epa_flush(a, done, nd);
    if (a.work_counters && lane == 0 && wk.queries) {
        atomicAdd(a.work_counters + 0, dots);
        atomicAdd(a.work_counters + 1, (unsigned long long)wk.faces);
        atomicAdd(a.work_counters + 2, (unsigned long long)wk.queries);
    }
}

template <int BT>
int launch_epa_bt(const NarrowArgs& a, cudaStream_t s)
{
    constexpr int W = BT / 32;
    static LaunchSetup setup;
    int per_sm = 0;
    const size_t shm = (size_t)W * (sizeof(WarpEpaMem) + 32 * sizeof(EpaDone));
    int rc = launch_setup(setup, epa_pass_kernel<BT>, BT, shm, 200 * 1024, &per_sm);
    if (rc) return rc;
    MWD_CUDA(launch_pdl(epa_pass_kernel<BT>, (unsigned)(num_sms() * per_sm), BT, shm, s, a));
    return MWD_OK;
}

template <int LPP, int BT>
int launch_gjk_bt(const NarrowArgs& a, cudaStream_t s)
{
    static LaunchSetup setup;
    int per_sm = 0;
    int rc = launch_setup(setup, gjk_pass_kernel<LPP, BT>, BT, 0, 0, &per_sm);
    if (rc) return rc;
    MWD_CUDA(launch_pdl(gjk_pass_kernel<LPP, BT>, (unsigned)(num_sms() * per_sm), BT, 0, s, a));
    return MWD_OK;
}

template <int LPP>
int launch_gjk(const NarrowArgs& a, int code, cudaStream_t s)
{
    if (code == 1) return launch_gjk_bt<LPP, 64>(a, s);
    if (code == 2) return launch_gjk_bt<LPP, 256>(a, s);
    return launch_gjk_bt<LPP, 128>(a, s);
}

int launch_epa(const NarrowArgs& a, int code, cudaStream_t s)
{
    if (code == 1) return launch_epa_bt<64>(a, s);
    if (code == 2) return launch_epa_bt<256>(a, s);
    return launch_epa_bt<128>(a, s);
}

// Resolve the reference's overlapping stride-1 history writes (.cu:1018-1021, :1158-1161): the
// value left at hist[k] is the one written by the highest pair index P' in [k-3, k] that wrote.
__global__ void hist_resolve_kernel(float* hist, const float4* stage, const uint8_t* wrote, int64_t n)
{
    int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n + 3) return;
    for (int64_t P = (k < n - 1 ? k : n - 1); P >= 0 && P >= k - 3; --P) {
        if (wrote[P]) {
            float4 v = stage[P];
            int j = (int)(k - P);
            hist[k] = j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
            return;
        }
    }
}

template <int LPP, int MODE>
int launch_lpp(const NarrowArgs& a, int64_t n_hint, cudaStream_t s)
{
    constexpr int GPB = NARROW_THREADS / LPP;
    size_t shm = (size_t)(NARROW_THREADS / 32) * sizeof(WarpEpaMem) + (size_t)GPB * 2 * a.hull_cap * sizeof(float4);
    static LaunchSetup setup;
    int per_sm = 0;
    int rc = launch_setup(setup, narrow_kernel<LPP, MODE>, NARROW_THREADS, shm, 200 * 1024, &per_sm);
    if (rc) return rc;
    int64_t grid = (int64_t)num_sms() * per_sm;
    int64_t need = (n_hint + GPB - 1) / GPB;
    if (n_hint >= 0 && need < grid) grid = need > 0 ? need : 1;
    narrow_kernel<LPP, MODE><<<(unsigned)grid, NARROW_THREADS, shm, s>>>(a);
    MWD_CUDA(cudaGetLastError());
    return MWD_OK;
}

}  // namespace

int launch_narrow(const NarrowArgs& a, int mode, int lanes, int64_t n_hint, cudaStream_t s)
{
    if (mode == 0) {
        switch (lanes) {
            case 4: return launch_lpp<4, 0>(a, n_hint, s);
            case 8: return launch_lpp<8, 0>(a, n_hint, s);
            case 16: return launch_lpp<16, 0>(a, n_hint, s);
            case 32: return launch_lpp<32, 0>(a, n_hint, s);
        }
    } else {
        switch (lanes) {
            case 4: return launch_lpp<4, 1>(a, n_hint, s);
            case 8: return launch_lpp<8, 1>(a, n_hint, s);
            case 16: return launch_lpp<16, 1>(a, n_hint, s);
            case 32: return launch_lpp<32, 1>(a, n_hint, s);
        }
    }
    set_error("lanes per pair must be 4, 8, 16 or 32 (got %d)", lanes);
    return MWD_ERR_INVALID;
}

// lanes = GJK-pass lanes per pair | EPA-pass lanes per pair << 8 (checked; the EPA pass gives each pair
// a warp) | the two passes' block-size codes (MWD_LANES_*_BLOCK_SHIFT)
int launch_narrow_two_pass(const NarrowArgs& a, int lanes, cudaStream_t s)
{
    const int gl = lanes & 0xff;
    int el = (lanes >> 8) & 0xff;
    if (!el) el = gl;
    const int gb = (lanes >> MWD_LANES_GJK_BLOCK_SHIFT) & 3, eb = (lanes >> MWD_LANES_EPA_BLOCK_SHIFT) & 3;
    const bool gl_ok = gl == 1 || gl == 4 || gl == 8 || gl == 16 || gl == 32;
    const bool el_ok = el == 4 || el == 8 || el == 16 || el == 32;
    if (!gl_ok || !el_ok) {
        set_error("lanes per pair must be 1 (GJK pass only), 4, 8, 16 or 32 (got GJK %d, EPA %d)", gl, el);
        return MWD_ERR_INVALID;
    }
    if (gb == 3 || eb == 3) {
        set_error("block-size code must be 0 (128 threads), 1 (64) or 2 (256) (got GJK %d, EPA %d)", gb, eb);
        return MWD_ERR_INVALID;
    }
    if (!a.epa_zeroed) MWD_CUDA(cudaMemsetAsync(a.epa_count, 0, 8 * sizeof(int32_t), s));
    if (a.hist_keys) MWD_CUDA(launch_pdl(hist_clear_kernel, (unsigned)(num_sms() * 4), 256, 0, s, a));
    int rc = MWD_OK;
    switch (gl) {
        case 1: rc = launch_gjk<1>(a, gb, s); break;
        case 4: rc = launch_gjk<4>(a, gb, s); break;
        case 8: rc = launch_gjk<8>(a, gb, s); break;
        case 16: rc = launch_gjk<16>(a, gb, s); break;
        default: rc = launch_gjk<32>(a, gb, s); break;
    }
    if (rc) return rc;
    rc = launch_epa(a, eb, s);
    if (rc) return rc;
    if (a.hist_keys) MWD_CUDA(launch_pdl(hist_flip_kernel, 1, 32, 0, s, a));
    return MWD_OK;
}

int launch_hist_resolve(float* hist, const float* stage, const uint8_t* wrote, int64_t n, cudaStream_t s)
{
    if (n <= 0) return MWD_OK;
    int64_t total = n + 3;
    unsigned grid = (unsigned)((total + 255) / 256);
    hist_resolve_kernel<<<grid, 256, 0, s>>>(hist, reinterpret_cast<const float4*>(stage), wrote, n);
    MWD_CUDA(cudaGetLastError());
    return MWD_OK;
}

}  // namespace mwd
