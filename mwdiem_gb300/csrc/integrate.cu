// Quaternion leapfrog integrator (gpu_Verlet.cu:85-431), two variants:
//
//  * verlet_ref_kernel -- FP64 over the reference's own arrays (the drop-in for gpu_Verlet.Verlet_GPU).
//    The reference's formulas with products and sums fused; the per-vertex rotation of the world-frame
//    vertex table (gpu_Verlet.cu:279-323) is done by all lanes of the rows' warp, so the (N,V,3) array is
//    read and written with coalesced accesses instead of one thread walking V vertices.
//
//  * integrate_kernel -- FP32 state in float4 structure-of-arrays with FP64 centres (the
//    device-resident step).  Instead of rotating every world vertex by q each step (which compounds
//    the rotation, gpu_Verlet.cu:279-305), it keeps q_acc = q_k (x) q_acc, the product of those
//    rotations, and regenerates world = pos + R(q_acc) r0 from the body-frame table: the same
//    vertices, without accumulating rounding in the vertex coordinates.  Walls are not integrated
//    (rows below num_part_min, gpu_Verlet.cu:110).  The force/torque accumulators are consumed and
//    zeroed for the next step.
#include "common.cuh"
#include "integrate.cuh"

namespace mwd {

namespace {

struct d3 {
    double x, y, z;
};
__device__ __forceinline__ d3 dm(double x, double y, double z)
{
    d3 r;
    r.x = x;
    r.y = y;
    r.z = z;
    return r;
}
__device__ __forceinline__ d3 operator+(d3 a, d3 b) { return dm(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return dm(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ d3 operator*(d3 a, double s) { return dm(a.x * s, a.y * s, a.z * s); }
// a s + b
__device__ __forceinline__ d3 dfma(d3 a, double s, d3 b) { return dm(fma(a.x, s, b.x), fma(a.y, s, b.y), fma(a.z, s, b.z)); }
__device__ __forceinline__ double ddot(d3 a, d3 b) { return fma(a.x, b.x, fma(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ d3 dcross(d3 a, d3 b)
{
    return dm(fma(a.y, b.z, -(a.z * b.y)), fma(a.z, b.x, -(a.x * b.z)), fma(a.x, b.y, -(a.y * b.x)));
}
__device__ __forceinline__ d3 dld(const double* p) { return dm(p[0], p[1], p[2]); }
__device__ __forceinline__ void dst(double* p, d3 v) { p[0] = v.x; p[1] = v.y; p[2] = v.z; }

struct dq {
    double w, x, y, z;
};
// Hamilton product (gpu_Verlet.cu:43-54)
__device__ __forceinline__ dq dqmul(dq a, dq b)
{
    dq r;
    r.w = fma(a.w, b.w, -ddot(dm(a.x, a.y, a.z), dm(b.x, b.y, b.z)));
    r.x = fma(a.w, b.x, fma(a.x, b.w, fma(a.y, b.z, -(a.z * b.y))));
    r.y = fma(a.w, b.y, fma(a.y, b.w, fma(a.z, b.x, -(a.x * b.z))));
    r.z = fma(a.w, b.z, fma(a.z, b.w, fma(a.x, b.y, -(a.y * b.x))));
    return r;
}
// vector part of q (0, v) q* (sign 1) or q* (0, v) q (sign -1), q of any length:
// (w^2 - u.u) v + 2 (u.v) u + sign 2 w (u x v)
__device__ __forceinline__ d3 dqturn(dq q, d3 v, double sign)
{
    const d3 u = dm(q.x, q.y, q.z);
    const d3 r = dfma(u, 2 * ddot(u, v), v * fma(q.w, q.w, -ddot(u, u)));
    return dfma(dcross(u, v), sign * 2 * q.w, r);
}
__device__ __forceinline__ dq dqld(const double* p)
{
    dq q;
    q.w = p[0];
    q.x = p[1];
    q.y = p[2];
    q.z = p[3];
    return q;
}
__device__ __forceinline__ void dqst(double* p, dq q)
{
    p[0] = q.w;
    p[1] = q.x;
    p[2] = q.y;
    p[3] = q.z;
}
__device__ __forceinline__ d3 matvec(const double* M, d3 v)
{
    return dm(ddot(dld(M), v), ddot(dld(M + 3), v), ddot(dld(M + 6), v));
}
// [cos(|w| s), sin(|w| s) w / |w|]
__device__ __forceinline__ dq dqincrement(d3 w, double s)
{
    const double wn = sqrt(ddot(w, w));
    double sn, cs;
    sincos(wn * s, &sn, &cs);
    const double k = wn != 0 ? sn / wn : 0.0;
    dq r;
    r.w = cs;
    r.x = w.x * k;
    r.y = w.y * k;
    r.z = w.z * k;
    return r;
}

// One warp per block, `rows` of its lanes with a row each; then all lanes turn the rows' vertices.  Bound
// by FP64 instructions, each of which holds its scheduler for 64 cycles on this GPU however many of its
// lanes work: so products and sums are fused, the turn of a vertex is a product with a matrix that its
// row's lane forms (15 instructions with the shifts; the quaternion products were 65), and the host picks `rows` so that
// the warps fill whole rounds of the schedulers.  20,005 rows of 32 vertices: 189 us before.
constexpr int VR = 32;
__global__ void __launch_bounds__(VR) verlet_ref_kernel(VerletRefArgs a, int rows)
{
    __shared__ double s_m[VR][9];  // turn about the old centre
    __shared__ d3 s_c[VR], s_t[VR];  // old centre, and where it goes (a reset row: its undone shift)
    __shared__ int s_mode[VR];       // 0 inactive, 1 active, 2 active with a fly-away reset
    const int lane = threadIdx.x;
    const int p0 = blockIdx.x * rows;
    const int P = p0 + lane;
    const double dt = a.p.dt;
    const bool on = lane < rows && P < a.N && P >= a.p.n_min && P < a.p.n_max;
    if (on) {
        d3 vel12 = dld(a.v12 + 3 * P), om12bf = dld(a.w12bf + 3 * P), ombf = dld(a.wbf + 3 * P);
        d3 om = dld(a.w + 3 * P), c = dld(a.com + 3 * P);
        const d3 f = dld(a.F + 3 * P), t = dld(a.T + 3 * P);
        const double m = a.mass[P];
        dq qq = dqld(a.q + 4 * P), qh = dqld(a.q12 + 4 * P);
        d3 dxa = dld(a.dxall + 3 * P);

        // F / m, each quotient corrected by its exact remainder (Markstein, IBM J. Res. Dev. 34, 1990; extreme
        // operands divide)
        const double im = 1 / m;
        const bool plain = fabs(m) > 1e-150 && fabs(m) < 1e150;
        auto over_m = [&](double x) {
            const double y = x * im;
            if (plain && (x == 0 || (fabs(x) > 1e-120 && fabs(x) < 1e150))) return x == 0 ? y : fma(fma(-m, y, x), im, y);
            return x / m;
        };
        const d3 acc = dm(over_m(f.x), over_m(f.y), over_m(f.z));
        const d3 tbf = dqturn(qq, t, -1);
        const d3 p1 = matvec(a.I + 9 * P, ombf);
        const d3 p2 = tbf - dcross(ombf, p1);
        const d3 alpha = matvec(a.Iinv + 9 * P, p2);
        vel12 = dfma(acc, dt, vel12);
        qh = dqmul(dqincrement(om, dt / 2), qh);
        om12bf = dfma(alpha, dt, om12bf);
        const d3 dx = vel12 * dt;
        dxa = dxa + dx;
        const d3 om34 = dqturn(qh, dfma(alpha, dt / 4, om12bf), 1);
        const dq qold = qq;
        qq = dqmul(dqincrement(om34, dt / 4), qh);
        const dq qa = dqmul(qq, qold);
        ombf = dfma(alpha, dt / 2, om12bf);
        om = dqturn(qq, ombf, 1);
        d3 vel = dfma(acc, dt, vel12);
        const d3 c_old = c;
        c = c + dx;
        d3 to = c;
        int mode = 1;
        const double* box = a.p.box;
        if (c.x > box[0] || c.x < box[1] || c.y > box[2] || c.y < box[3] || c.z > box[4] || c.z < box[5]) {
            // fly-away reset (gpu_Verlet.cu:338-352): stop the particle, undo the move
            vel = dm(0, 0, 0);
            vel12 = vel;
            om12bf = vel;
            ombf = vel;
            om = vel;
            c = c + dx * (-1);
            to = dx;
            mode = 2;
            if (a.n_reset) atomicAdd(a.n_reset, 1);
        }
        dst(a.v + 3 * P, vel);
        dst(a.v12 + 3 * P, vel12);
        dst(a.w12bf + 3 * P, om12bf);
        dst(a.com + 3 * P, c);
        dst(a.dxall + 3 * P, dxa);
        dst(a.wbf + 3 * P, ombf);
        dst(a.w + 3 * P, om);
        dqst(a.q12 + 4 * P, qh);
        dqst(a.q + 4 * P, qq);
        dqst(a.qall + 4 * P, qa);
        // the matrix of v -> vector part of q (0, v) q*
        const double ww = qq.w * qq.w, xx = qq.x * qq.x, yy = qq.y * qq.y, zz = qq.z * qq.z;
        double* M = s_m[lane];
        M[0] = (ww + xx) - (yy + zz);
        M[4] = (ww + yy) - (xx + zz);
        M[8] = (ww + zz) - (xx + yy);
        M[1] = 2 * fma(qq.x, qq.y, -(qq.w * qq.z));
        M[3] = 2 * fma(qq.x, qq.y, qq.w * qq.z);
        M[2] = 2 * fma(qq.x, qq.z, qq.w * qq.y);
        M[6] = 2 * fma(qq.x, qq.z, -(qq.w * qq.y));
        M[5] = 2 * fma(qq.y, qq.z, -(qq.w * qq.x));
        M[7] = 2 * fma(qq.y, qq.z, qq.w * qq.x);
        s_c[lane] = c_old;
        s_t[lane] = to;
        s_mode[lane] = mode;
    } else {
        s_mode[lane] = 0;
    }
    __syncwarp();
    // vertices of the warp's rows: turned about the old centre, then moved (gpu_Verlet.cu:279-352)
    const int V = a.p.V;
    const int total = min(rows, a.N - p0) * V;
    double* vp = a.verts + (size_t)p0 * V * 3;
    constexpr int U = 4;  // vertices in flight per lane
    for (int j0 = lane; j0 < total; j0 += U * VR) {
        d3 v[U];
        int r[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int j = j0 + k * VR;
            r[k] = j < total ? j / V : 0;
            if (j < total && s_mode[r[k]]) v[k] = dld(vp + 3 * (size_t)j);
            else r[k] = -1;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (r[k] < 0) continue;
            const d3 c = s_c[r[k]], t = s_t[r[k]];
            const double* M = s_m[r[k]];
            const d3 d = v[k] - c;
            // the turned offset first: rounded at its own size, not at the coordinates'
            const d3 o = dm(ddot(dld(M), d), ddot(dld(M + 3), d), ddot(dld(M + 6), d));
            // a reset undoes the vertices' shift as it does the centre's (:338-352), with the same rounding
            d3 w = o + t;
            if (s_mode[r[k]] == 2) w = ((o + c) + t) + t * (-1);
            dst(vp + 3 * (size_t)(j0 + k * VR), w);
        }
    }
}

constexpr int RB = 128;  // rows per block

// ------------------------------------------------------------------ FP32 device-resident step

__device__ __forceinline__ float4 ld4(const float* p, int i) { return reinterpret_cast<const float4*>(p)[i]; }
__device__ __forceinline__ void st4(float* p, int i, float4 v) { reinterpret_cast<float4*>(p)[i] = v; }

struct alignas(32) dpos {
    double x, y, z, w;
};

// rotation increment [cos(|w| s), sin(|w| s) w/|w|]
__device__ __forceinline__ float4 rot_increment(f3 w, float s)
{
    float wn = sqrtf(w.x * w.x + w.y * w.y + w.z * w.z);
    float sn, cs;
    sincosf(wn * s, &sn, &cs);
    f3 h = mk3(0.f, 0.f, 0.f);
    if (wn != 0.f) h = (w / wn) * sn;
    return make_float4(cs, h.x, h.y, h.z);
}

// one row's update (walls: unchanged); returns the centre and q_acc the vertex pass uses
// MIRROR: every state array written here is also written `mirror` bytes further on, into a copy of the
// state block that lives in host memory the GPU can reach (the force/torque accumulators excepted)
template <bool MIRROR = false>
__device__ __forceinline__ void row_update(const mwd_state& st, const mwd_scene* __restrict__ scenes, int P,
                                           dpos& pos_out, float4& qacc_out, int64_t mirror = 0)
{
    const int info = st.info[P];
    dpos pos = reinterpret_cast<const dpos*>(st.pos)[P];
    float4 qacc = ld4(st.q_acc, P);
    if (!(info & (1 | MWD_INFO_INACTIVE))) {  // walls and rows waiting at an inlet stay as they are
        const mwd_scene& sc = scenes[info >> 1];
        const float dt = (float)sc.dt;
        float4 Fa = ld4(st.force, P), Ta = ld4(st.torque, P);
        float4 Fe = ld4(st.ext_force, P), Te = ld4(st.ext_torque, P);
        f3 F = mk3(Fa.x + Fe.x, Fa.y + Fe.y, Fa.z + Fe.z);
        f3 T = mk3(Ta.x + Te.x, Ta.y + Te.y, Ta.z + Te.z);
        float4 I = ld4(st.inertia, P), Ii = ld4(st.inv_inertia, P);
        const float invm = Ii.w;
        f3 vh = xyz(ld4(st.vel_half, P));
        f3 whbf = xyz(ld4(st.w_half_bf, P));
        f3 wbf = xyz(ld4(st.w_bf, P));
        f3 w = xyz(ld4(st.w, P));
        float4 q = ld4(st.q, P), qh = ld4(st.q_half, P), qall = ld4(st.q_all, P);
        dpos dxall = reinterpret_cast<const dpos*>(st.dx_all)[P];

        f3 v32 = vh + F * (invm * dt);
        f3 tbf = qtrip(qconj(q), T, q);
        f3 p1 = mk3(I.x * wbf.x, I.y * wbf.y, I.z * wbf.z);
        f3 p2 = tbf - cross(wbf, p1);
        f3 alpha = mk3(Ii.x * p2.x, Ii.y * p2.y, Ii.z * p2.z);
        f3 w32bf = whbf + alpha * dt;
        float4 q32 = qmul(rot_increment(w, dt * 0.5f), qh);
        vh = v32;
        qh = q32;
        whbf = w32bf;
        f3 dx = vh * dt;
        dxall.x += (double)dx.x;
        dxall.y += (double)dx.y;
        dxall.z += (double)dx.z;
        f3 w34bf = whbf + alpha * (dt * 0.25f);
        f3 w34 = qtrip(qh, w34bf, qconj(qh));
        float4 qold = q;
        q = qmul(rot_increment(w34, dt * 0.25f), qh);
        qall = qmul(q, qold);
        wbf = whbf + alpha * (dt * 0.5f);
        w = qtrip(q, wbf, qconj(q));
        f3 v = vh + F * (invm * dt);
        // vertices compound the rotation q every step (gpu_Verlet.cu:279-305): q_acc <- q q_acc;
        // under the physical law the vertices follow the orientation itself: q_acc <- q
        qacc = sc.mat[0].physical ? q : qmul(q, qacc);
        float qn = rsqrtf(qacc.x * qacc.x + qacc.y * qacc.y + qacc.z * qacc.z + qacc.w * qacc.w);
        qacc = make_float4(qacc.x * qn, qacc.y * qn, qacc.z * qn, qacc.w * qn);
        dpos np;
        np.x = pos.x + (double)dx.x;
        np.y = pos.y + (double)dx.y;
        np.z = pos.z + (double)dx.z;
        np.w = pos.w;
        if (np.x > sc.box[0] || np.x < sc.box[1] || np.y > sc.box[2] || np.y < sc.box[3] || np.z > sc.box[4] ||
            np.z < sc.box[5]) {
            // fly-away reset (gpu_Verlet.cu:338-352): stop the particle, undo the move
            v = vh = whbf = wbf = w = mk3(0.f, 0.f, 0.f);
            np = pos;
        }
        pos = np;
        auto putd = [&](double* a, const dpos& x) {
            reinterpret_cast<dpos*>(a)[P] = x;
            if (MIRROR) reinterpret_cast<dpos*>(reinterpret_cast<char*>(a) + mirror)[P] = x;
        };
        auto put4 = [&](float* a, float4 x) {
            st4(a, P, x);
            if (MIRROR) st4(reinterpret_cast<float*>(reinterpret_cast<char*>(a) + mirror), P, x);
        };
        putd(st.pos, pos);
        putd(st.dx_all, dxall);
        put4(st.vel, f4(v, 0.f));
        put4(st.vel_half, f4(vh, 0.f));
        put4(st.w_half_bf, f4(whbf, 0.f));
        put4(st.w_bf, f4(wbf, 0.f));
        put4(st.w, f4(w, 0.f));
        put4(st.q, q);
        put4(st.q_half, qh);
        put4(st.q_all, qall);
        put4(st.q_acc, qacc);
        st4(st.force, P, make_float4(0.f, 0.f, 0.f, 0.f));
        st4(st.torque, P, make_float4(0.f, 0.f, 0.f, 0.f));
    }
    pos_out = pos;
    qacc_out = qacc;
}

// R(q_acc) row-major and the centre as hi + lo floats per axis
__device__ __forceinline__ void row_xform(float4 qacc, dpos pos, float* R, float* c)
{
    const float qw = qacc.x, qx = qacc.y, qy = qacc.z, qz = qacc.w;
    R[0] = 1.f - 2.f * (qy * qy + qz * qz); R[1] = 2.f * (qx * qy - qw * qz); R[2] = 2.f * (qx * qz + qw * qy);
    R[3] = 2.f * (qx * qy + qw * qz); R[4] = 1.f - 2.f * (qx * qx + qz * qz); R[5] = 2.f * (qy * qz - qw * qx);
    R[6] = 2.f * (qx * qz - qw * qy); R[7] = 2.f * (qy * qz + qw * qx); R[8] = 1.f - 2.f * (qx * qx + qy * qy);
    const float hx = (float)pos.x, hy = (float)pos.y, hz = (float)pos.z;
    c[0] = hx; c[1] = (float)(pos.x - (double)hx);
    c[2] = hy; c[3] = (float)(pos.y - (double)hy);
    c[4] = hz; c[5] = (float)(pos.z - (double)hz);
}

__device__ __forceinline__ float4 world_vertex(const float* R, const float* c, float4 r0)
{
    const float rx = R[0] * r0.x + R[1] * r0.y + R[2] * r0.z;
    const float ry = R[3] * r0.x + R[4] * r0.y + R[5] * r0.z;
    const float rz = R[6] * r0.x + R[7] * r0.y + R[8] * r0.z;
    return make_float4(c[0] + (rx + c[1]), c[2] + (ry + c[3]), c[4] + (rz + c[5]), 0.f);
}

__global__ void __launch_bounds__(RB) integrate_kernel(mwd_state st, const mwd_scene* __restrict__ scenes,
                                                       uint32_t* status)
{
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float s_R[RB][9];
    __shared__ float s_c[RB][6];  // centre split hi/lo per axis
    __shared__ int s_off[RB + 1];
    const int P = blockIdx.x * RB + threadIdx.x;
    const int p0 = blockIdx.x * RB;
    const int rows = min(RB, st.n - p0);
    if (P < st.n) {
        dpos pos;
        float4 qacc;
        row_update(st, scenes, P, pos, qacc);
        row_xform(qacc, pos, s_R[threadIdx.x], s_c[threadIdx.x]);
        s_off[threadIdx.x] = st.vert_off[P];
    }
    if (threadIdx.x == 0) s_off[rows] = st.vert_off[p0 + rows];
    __syncthreads();
    const int v0 = s_off[0], v1 = s_off[rows];
    const float4* bv = reinterpret_cast<const float4*>(st.body_verts);
    float4* wv = reinterpret_cast<float4*>(st.world_verts);
    constexpr int U = 4;  // vertices in flight per thread: loads first, then the stores
    for (int j0 = v0 + threadIdx.x; j0 < v1; j0 += U * RB) {
        float4 r0[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int j = j0 + k * RB;
            r0[k] = j < v1 ? __ldg(bv + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int j = j0 + k * RB;
            if (j >= v1) break;
            // owner row: last r with s_off[r] <= j
            int lo = 0, hi = rows - 1;
            while (lo < hi) {
                int mid = (lo + hi + 1) >> 1;
                if (s_off[mid] <= j) lo = mid; else hi = mid - 1;
            }
            wv[j] = world_vertex(s_R[lo], s_c[lo], r0[k]);
        }
    }
}

// the row pass of the split integrator: one thread per row, the transform to st.xform (MIRROR: the
// state also written into its copy in GPU-reachable host memory, `mirror` bytes further on)
template <bool MIRROR>
__global__ void __launch_bounds__(RB) integrate_rows_kernel(mwd_state st, const mwd_scene* __restrict__ scenes,
                                                            uint32_t* status, int64_t mirror)
{
    pdl_wait();
    pdl_launch_dependents();
    const int P = blockIdx.x * RB + threadIdx.x;
    if (P >= st.n) return;
    dpos pos;
    float4 qacc;
    row_update<MIRROR>(st, scenes, P, pos, qacc, mirror);
    float x[16];
    row_xform(qacc, pos, x, x + 9);
    x[15] = 0.f;
    float4* o = reinterpret_cast<float4*>(st.xform) + 4 * (size_t)P;
    o[0] = make_float4(x[0], x[1], x[2], x[3]);
    o[1] = make_float4(x[4], x[5], x[6], x[7]);
    o[2] = make_float4(x[8], x[9], x[10], x[11]);
    o[3] = make_float4(x[12], x[13], x[14], x[15]);
}

// the row transforms alone, from the current centres and orientations (no integration)
__global__ void __launch_bounds__(RB) xform_rows_kernel(mwd_state st)
{
    pdl_wait();
    pdl_launch_dependents();
    const int P = blockIdx.x * RB + threadIdx.x;
    if (P >= st.n) return;
    const dpos pos = reinterpret_cast<const dpos*>(st.pos)[P];
    float x[16];
    row_xform(ld4(st.q_acc, P), pos, x, x + 9);
    x[15] = 0.f;
    float4* o = reinterpret_cast<float4*>(st.xform) + 4 * (size_t)P;
    o[0] = make_float4(x[0], x[1], x[2], x[3]);
    o[1] = make_float4(x[4], x[5], x[6], x[7]);
    o[2] = make_float4(x[8], x[9], x[10], x[11]);
    o[3] = make_float4(x[12], x[13], x[14], x[15]);
}

// the vertex pass of the split integrator: one thread per vertex
__global__ void __launch_bounds__(256) world_verts_kernel(mwd_state st)
{
    pdl_wait();
    pdl_launch_dependents();
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= st.n_verts) return;
    const int o = st.vert_owner[j];
    const float4* xf = reinterpret_cast<const float4*>(st.xform) + 4 * (size_t)o;
    const float4 a = xf[0], b = xf[1], c = xf[2], d = xf[3];
    const float R[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x};
    const float cc[6] = {c.y, c.z, c.w, d.x, d.y, d.z};
    const float4 r0 = __ldg(reinterpret_cast<const float4*>(st.body_verts) + j);
    reinterpret_cast<float4*>(st.world_verts)[j] = world_vertex(R, cc, r0);
}
}  // namespace

int launch_verlet_ref(const VerletRefArgs& a, cudaStream_t s)
{
    if (a.N <= 0) return MWD_OK;
    // whole rounds of one warp per scheduler (four per SM), with the fewest rows per warp that need no
    // further round: a row's own arithmetic takes a warp as long for 1 row as for 32, its vertices do not
    const int schedulers = 4 * num_sms();
    const int rounds = (a.N + VR * schedulers - 1) / (VR * schedulers);
    const int rows = (a.N + rounds * schedulers - 1) / (rounds * schedulers);
    verlet_ref_kernel<<<(a.N + rows - 1) / rows, VR, 0, s>>>(a, rows);
    MWD_CUDA(cudaGetLastError());
    return MWD_OK;
}

int launch_world_verts(const mwd_state& st, cudaStream_t s)
{
    if (st.n_verts <= 0) return MWD_OK;
    MWD_CUDA(launch_pdl(world_verts_kernel, (st.n_verts + 255) / 256, 256, 0, s, st));
    return MWD_OK;
}

int launch_refresh_vertices(const mwd_state& st, cudaStream_t s)
{
    if (st.n <= 0) return MWD_OK;
    MWD_CUDA(launch_pdl(xform_rows_kernel, (st.n + RB - 1) / RB, RB, 0, s, st));
    return launch_world_verts(st, s);
}

int launch_integrate_rows_mirror(const mwd_state& st, const mwd_scene* scenes, uint32_t* status, int64_t mirror,
                                 cudaStream_t s)
{
    if (st.n <= 0) return MWD_OK;
    MWD_CUDA(launch_pdl(integrate_rows_kernel<true>, (st.n + RB - 1) / RB, RB, 0, s, st, scenes, status, mirror));
    MWD_CUDA(cudaGetLastError());
    return MWD_OK;
}

// Rows and vertices in one kernel (integrate_kernel: each block's rows, then their vertices) once its
// grid spans at least two full waves of the GPU; below that the row pass and the one-thread-per-vertex
// pass spread the vertex work better.  On 256 batched scenes (2.0M rows) one kernel per step measured
// 0.676 ms per step against 0.699 ms for the two passes with the vertex pass overlapped with the next
// step's broad phase: it moves neither the row transforms nor the vertex owners through memory.
bool integrate_in_one_kernel(int64_t n)
{
    static LaunchSetup setup;
    int per_sm = 0;
    if (launch_setup(setup, integrate_kernel, RB, 0, 0, &per_sm) != MWD_OK || per_sm <= 0) return false;
    return (n + RB - 1) / RB >= 2 * (int64_t)num_sms() * per_sm;
}

int launch_integrate(const mwd_state& st, const mwd_scene* scenes, uint32_t* status, cudaStream_t s,
                     bool with_verts)
{
    if (st.n <= 0) return MWD_OK;
    if (st.vert_owner && st.xform && !(with_verts && integrate_in_one_kernel(st.n))) {
        MWD_CUDA(launch_pdl(integrate_rows_kernel<false>, (st.n + RB - 1) / RB, RB, 0, s, st, scenes, status,
                            (int64_t)0));
        if (with_verts && st.n_verts > 0)
            MWD_CUDA(launch_pdl(world_verts_kernel, (st.n_verts + 255) / 256, 256, 0, s, st));
    } else {
        MWD_CUDA(launch_pdl(integrate_kernel, (st.n + RB - 1) / RB, RB, 0, s, st, scenes, status));
    }
    MWD_CUDA(cudaGetLastError());
    return MWD_OK;
}

}  // namespace mwd
