// pk_plastic.cu -- ElastoplasticityModule and FractureModule
// (Dynamics/ParticleSystem/ElastoplasticityModule.cu, FractureModule.cu) on
// the context's peridynamics rest shape.  Every kernel updates only the bonds
// of its own particle, so the rest shape can be rewritten in place.  Bond
// walks split a particle's bonds over kPlG lanes; the double-precision
// eigen-decompositions run one thread per particle.
//
// The reference's SVDs come from svd3_cuda.h (McAdams et al. 2011: U and V
// rotations, the sign of det A on the smallest singular value).  What the
// modules use from them is unique: the clamped inverse V D^-1 U^T of a
// symmetric positive semi-definite matrix (its eigen-decomposition) and the
// polar rotation U V^T.  Both are formed in double from a Jacobi
// eigen-decomposition (jacobi3), with the same sign convention.
#include "pk_kernels.cuh"
#include "pk_pd_common.cuh"

namespace pk {

struct RestView {
    const int* index;
    int cap;
    long long total;
    int n;
    const int* ridx;
    float* rpos;
};
// The same shape as the projection's compact bonds (pk_pd_adj.cu): rest_j -
// rest_i and j (~j for a broken bond, which plasticity moves like any other) in
// one 16-byte load, in ascending order of j; positions packed to 16 bytes.  The
// rotation's sums walk these (82 -> 56 us at 65,536 particles with 113 bonds).
// The kernels after it read and write the rest shape in its own order: writing
// it bond by bond in the compact order took 235-250 us (partly written sectors)
// against 38 and 70.
struct BondView {
    const float4* bond;
    const float4* x;
};
// Bonds a lane has in flight.
constexpr int kPlU = 4;
__device__ __forceinline__ int bond_j(const float4& b)
{
    const int j = __float_as_int(b.w);
    return j >= 0 ? j : ~j;
}
// Calls f(place in the row, bond, x_j) on the lane's bonds, in order.
template <class F>
__device__ __forceinline__ void walk_bonds(const BondView& V, long long a0, int m, int sub, int i, const F& f)
{
    for (int e0 = sub; e0 < m; e0 += 8 * kPlU) {
        float4 b[kPlU], xj[kPlU];
#pragma unroll
        for (int u = 0; u < kPlU; ++u)
            b[u] = e0 + 8 * u < m ? V.bond[a0 + e0 + 8 * u] : make_float4(0.f, 0.f, 0.f, __int_as_float(i));
#pragma unroll
        for (int u = 0; u < kPlU; ++u) xj[u] = __ldg(V.x + bond_j(b[u]));
#pragma unroll
        for (int u = 0; u < kPlU; ++u)
            if (e0 + 8 * u < m) f(e0 + 8 * u, b[u], xj[u]);
    }
}

__device__ __forceinline__ float len3(float x, float y, float z) { return sqrtf((x * x + y * y) + z * z); }

// kPlG lanes per particle: lane `sub` walks bonds sub, sub + kPlG, ...; the
// group's partial sums are combined with xor shuffles in a fixed order.  The
// idle lanes of the last group mirror particle n - 1 and write nothing.
constexpr int kPlG = 8;
constexpr int kPlBlock = 128;
struct PlLane {
    int i, sub;
    bool valid;
};
__device__ __forceinline__ PlLane pl_lane(int n)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    PlLane L;
    L.i = (int)(gid / kPlG);
    L.sub = (int)(gid % kPlG);
    L.valid = L.i < n;
    if (!L.valid) L.i = n - 1;
    return L;
}
__device__ __forceinline__ float gsum8(float v)
{
#pragma unroll
    for (int o = kPlG / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ void gsum8(float (&M)[3][3])
{
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) M[a][b] = gsum8(M[a][b]);
}

// Eigenpairs by decreasing eigenvalue.
__device__ inline void eig_sorted(double A[3][3], double Q[3][3], double w[3])
{
    jacobi3(A, Q, w);
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2 - a; ++b)
            if (w[b] < w[b + 1]) {
                double t = w[b];
                w[b] = w[b + 1];
                w[b + 1] = t;
                for (int k = 0; k < 3; ++k) {
                    t = Q[k][b];
                    Q[k][b] = Q[k][b + 1];
                    Q[k][b + 1] = t;
                }
            }
}

__device__ inline double det3d(const double M[3][3])
{
    return M[0][0] * (M[1][1] * M[2][2] - M[1][2] * M[2][1]) - M[0][1] * (M[1][0] * M[2][2] - M[1][2] * M[2][0]) +
           M[0][2] * (M[1][0] * M[2][1] - M[1][1] * M[2][0]);
}

__device__ inline void unit3d(double u[3])
{
    const double l = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    if (l > 0) {
        u[0] /= l;
        u[1] /= l;
        u[2] /= l;
    }
}

__device__ inline void cross3d(const double a[3], const double b[3], double c[3])
{
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

// polarDecomposition's R (MatrixFunc.inl:81-98): V from the eigenvectors of
// A^T A (v_2 flipped so det V = 1), u_0, u_1 = A v_0, A v_1 normalised,
// u_2 = u_0 x u_1; R = U V^T.  Zero matrix: identity.
__device__ inline void polar_rotation(const double A[3][3], double R[3][3])
{
    double S[3][3], V[3][3], w[3], u[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) S[a][b] = A[0][a] * A[0][b] + A[1][a] * A[1][b] + A[2][a] * A[2][b];
    eig_sorted(S, V, w);
    if (!(w[0] > 0)) {
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) R[a][b] = (a == b) ? 1.0 : 0.0;
        return;
    }
    if (det3d(V) < 0)
        for (int a = 0; a < 3; ++a) V[a][2] = -V[a][2];
    for (int k = 0; k < 2; ++k)
        for (int a = 0; a < 3; ++a) u[k][a] = A[a][0] * V[0][k] + A[a][1] * V[1][k] + A[a][2] * V[2][k];
    unit3d(u[0]);
    if (w[1] > 1e-24 * w[0]) {
        const double d = u[1][0] * u[0][0] + u[1][1] * u[0][1] + u[1][2] * u[0][2];
        for (int a = 0; a < 3; ++a) u[1][a] -= d * u[0][a];
        unit3d(u[1]);
    } else {
        double e[3] = {0, 0, 0};
        const int m = fabs(u[0][0]) <= fabs(u[0][1]) ? (fabs(u[0][0]) <= fabs(u[0][2]) ? 0 : 2)
                                                      : (fabs(u[0][1]) <= fabs(u[0][2]) ? 1 : 2);
        e[m] = 1.0;
        cross3d(u[0], e, u[1]);
        unit3d(u[1]);
    }
    cross3d(u[0], u[1], u[2]);
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) R[a][b] = u[0][a] * V[b][0] + u[1][a] * V[b][1] + u[2][a] * V[b][2];
}

// V D' U^T of a symmetric positive semi-definite M: D' = 1/s above thr, fill below.
__device__ inline void clamped_inverse(const float M[3][3], double thr, double fill, float out[3][3])
{
    double A[3][3], Q[3][3], w[3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) A[a][b] = (double)M[a][b];
    jacobi3(A, Q, w);
    for (int a = 0; a < 3; ++a) {
        const double sv = fabs(w[a]);
        w[a] = sv > thr ? 1.0 / sv : fill;
    }
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b)
            out[a][b] = (float)(Q[a][0] * w[0] * Q[b][0] + Q[a][1] * w[1] * Q[b][1] + Q[a][2] * w[2] * Q[b][2]);
}

__device__ inline void mat_mul(const float A[3][3], const float B[3][3], float C[3][3])
{
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) C[a][b] = (A[a][0] * B[0][b] + A[a][1] * B[1][b]) + A[a][2] * B[2][b];
}

__device__ inline float det3f(const float M[3][3])
{
    return +M[0][0] * (M[1][1] * M[2][2] - M[1][2] * M[2][1]) - M[0][1] * (M[1][0] * M[2][2] - M[1][2] * M[2][0]) +
           M[0][2] * (M[1][0] * M[2][1] - M[1][1] * M[2][0]);
}

// EM_RotateRestShape (ElastoplasticityModule.cu:568-644) in three kernels:
// kPlG lanes per particle sum the deformation moment and the rest-shape
// moment over the bonds (coalesced walks), one thread per particle forms the
// rotation (two double-precision eigen-decompositions, every lane of a warp
// busy with its own particle), and kPlG lanes per particle rotate the bonds.
// Scratch per particle (kPlMk floats): mat (9), K (9), tw; then R (9).
__global__ void __launch_bounds__(kPlBlock) k_pl_rot_sums(RestView R, BondView V, float h, float* __restrict__ mk)
{
    const PlLane L = pl_lane(R.n);
    const int i = L.i;
    const long long a0 = pd_at(R.index, R.cap, i, 0);
    const int m = pd_size(R.index, R.cap, R.total, R.n, i);
    const float4 xi = __ldg(V.x + i);
    float tw = 0.f, mat[3][3] = {}, K[3][3] = {};
    walk_bonds(V, a0, m, L.sub, i, [&](int, const float4& d, const float4& xj) {
        const float r = len3(d.x, d.y, d.z);
        if (r > kEpsilon) {
            const float wt = smooth_w(r, h);
            const float p[3] = {(xj.x - xi.x) / h, (xj.y - xi.y) / h, (xj.z - xi.z) / h};
            const float q[3] = {d.x / h, d.y / h, d.z / h};
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    mat[a][b] += p[a] * q[b] * wt;
                    K[a][b] += q[a] * q[b] * wt;
                }
            tw += wt;
        }
    });
    gsum8(mat);
    gsum8(K);
    tw = gsum8(tw);
    if (!L.valid || L.sub != 0) return;
    float* o = mk + (long long)kPlMk * i;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            o[3 * a + b] = mat[a][b];
            o[9 + 3 * a + b] = K[a][b];
        }
    o[18] = tw;
}

__global__ void __launch_bounds__(128) k_pl_rot_solve(int n, float h, float* __restrict__ mk)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float* o = mk + (long long)kPlMk * i;
    float mat[3][3], K[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            mat[a][b] = o[3 * a + b];
            K[a][b] = o[9 + 3 * a + b];
        }
    const float tw = o[18];
    if (tw > kEpsilon) {
        const float s = 1.0f / tw;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) {
                mat[a][b] *= s;
                K[a][b] *= s;
            }
    }
    float Ki[3][3], M2[3][3];
    clamped_inverse(K, (double)(0.0001f * h), 1.0, Ki);
    mat_mul(mat, Ki, M2);
    double Md[3][3], Rd[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) Md[a][b] = (double)M2[a][b];
    polar_rotation(Md, Rd);
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) o[3 * a + b] = (float)Rd[a][b];
}

__global__ void __launch_bounds__(kPlBlock) k_pl_rot_apply(RestView R, const float* __restrict__ mk)
{
    const PlLane L = pl_lane(R.n);
    const int i = L.i;
    const long long a0 = pd_at(R.index, R.cap, i, 0);
    const float ri[3] = {R.rpos[3 * a0], R.rpos[3 * a0 + 1], R.rpos[3 * a0 + 2]};
    const int m = pd_size(R.index, R.cap, R.total, R.n, i);
    float Rf[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) Rf[a][b] = mk[(long long)kPlMk * i + 3 * a + b];
    __syncwarp();  // every lane holds rest_i before bond 0 (rest_i itself) is rewritten
    if (!L.valid) return;
    for (int e = L.sub; e < m; e += kPlG) {
        float* rj = R.rpos + 3 * pd_at(R.index, R.cap, i, e);
        const float d[3] = {rj[0] - ri[0], rj[1] - ri[1], rj[2] - ri[2]};
        for (int a = 0; a < 3; ++a) rj[a] = ri[a] + ((Rf[a][0] * d[0] + Rf[a][1] * d[1]) + Rf[a][2] * d[2]);
    }
}

// I1 and the reference's J2 (PM_ComputeInvariants, ElastoplasticityModule.cu:43-128;
// the J2 loop assigns, so only the last bond over 0.01 h of the list counts),
// by the particle's lane group on the packed positions x, kPlU bonds in flight:
// the I1 sums are combined, and J2 is the term of the last qualifying bond,
// looked for from the end of the row.
__device__ inline void invariants(const RestView& R, const float4* __restrict__ x, float h, int i, int sub, float& I1,
                                  float& J2)
{
    const long long a0 = pd_at(R.index, R.cap, i, 0);
    const float ri[3] = {R.rpos[3 * a0], R.rpos[3 * a0 + 1], R.rpos[3 * a0 + 2]};
    const int m = pd_size(R.index, R.cap, R.total, R.n, i);
    const float4 xi = __ldg(x + i);
    const double lim = 0.01 * (double)h;
    auto length = [&](float4 xj) { return len3(xj.x - xi.x, xj.y - xi.y, xj.z - xi.z); };
    float s1 = 0.f, tw = 0.f;
    for (int e0 = 1 + sub; e0 < m; e0 += kPlG * kPlU) {
        float r[kPlU];
        float4 xj[kPlU];
#pragma unroll
        for (int u = 0; u < kPlU; ++u) {
            const int e = e0 + u * kPlG;
            const bool in = e < m;
            const float* rj = R.rpos + 3 * (in ? a0 + e : a0);
            r[u] = in ? len3(ri[0] - rj[0], ri[1] - rj[1], ri[2] - rj[2]) : 0.f;
            xj[u] = __ldg(x + (in ? R.ridx[a0 + e] : i));
        }
#pragma unroll
        for (int u = 0; u < kPlU; ++u)
            if ((double)r[u] > lim) {
                const float wt = corr_w(r[u], h);
                s1 += wt * (length(xj[u]) / r[u]);
                tw += wt;
            }
    }
    s1 = gsum8(s1);
    tw = gsum8(tw);
    s1 = tw > kEpsilon ? s1 / tw : 1.0f;
    int last = -1;
    float j2 = 0.f;
    for (int top = m - 1; __any_sync(0xffffffffu, last < 0 && top >= 1); top -= kPlG) {
        const int e = top - sub;
        if (last < 0 && e >= 1) {
            const long long at = a0 + e;
            const float* rj = R.rpos + 3 * at;
            const float r = len3(ri[0] - rj[0], ri[1] - rj[1], ri[2] - rj[2]);
            if ((double)r > lim) {
                const float ratio = length(__ldg(x + R.ridx[at])) / r;
                j2 = (ratio - s1) * (ratio - s1) * corr_w(r, h);
                last = e;
            }
        }
#pragma unroll
        for (int o = kPlG / 2; o >= 1; o >>= 1) {
            const int ol = __shfl_xor_sync(0xffffffffu, last, o);
            const float oj = __shfl_xor_sync(0xffffffffu, j2, o);
            if (ol > last) {
                last = ol;
                j2 = oj;
            }
        }
    }
    I1 = s1;
    J2 = tw > kEpsilon ? sqrtf(j2 / tw) : 0.0f;
}

// PM_ComputeInvariants: Drucker-Prager yield (a yielding particle keeps its flag).
// Bound by the gathers of positions: 60 us at 65,536 particles with 113 bonds, 94
// on 12-byte positions with a second walk for the last bond.
__global__ void __launch_bounds__(kPlBlock)
    k_pl_invariants(RestView R, const float4* __restrict__ x, const float* __restrict__ bulk, float h, float A,
                    float B, float mu, float lambda, float* __restrict__ y1, float* __restrict__ y2, float* __restrict__ i1,
                    unsigned char* __restrict__ byield, float4* __restrict__ y4)
{
    const PlLane L = pl_lane(R.n);
    const int i = L.i;
    float I1, J2;
    invariants(R, x, h, i, L.sub, I1, J2);
    if (!L.valid || L.sub != 0) return;
    const float sJ2 = J2 * mu * bulk[i];
    const float sD1 = (1.0f - I1) * lambda * bulk[i];
    const float lim = A + B * sD1;
    float a = 0.f, b = 0.f;
    if (sJ2 <= lim) {
        byield[i] = 0;
    } else if (lim > 0.f) {
        b = (sJ2 - lim) / sJ2;
    } else {
        a = lim < -kEpsilon ? lim / (B * sD1) : 1.0f;
        b = 1.0f;
    }
    y1[i] = a;
    y2[i] = b;
    i1[i] = I1;
    y4[i] = make_float4(a, b, I1, 0.f);  // gathered together by k_pl_yield
}

// v.norm() > EPSILON ? v.normalize() : 0 (normalize gives 0 below FLT_EPSILON).
__device__ inline void unit_or_zero3(float v[3])
{
    const float l = len3(v[0], v[1], v[2]);
    if (l > kEpsilon && l > 1.1920928955078125e-7f) {
        const float is = 1.0f / l;
        v[0] *= is;
        v[1] *= is;
        v[2] *= is;
    } else {
        v[0] = v[1] = v[2] = 0.f;
    }
}

// PM_ApplyYielding (ElastoplasticityModule.cu:165-226).  59 us at 65,536 particles
// with 113 bonds on packed positions, 71 on 12-byte ones.
__global__ void __launch_bounds__(kPlBlock)
    k_pl_yield(RestView R, const float4* __restrict__ x, const float4* __restrict__ y4)
{
    const PlLane L = pl_lane(R.n);
    const int i = L.i;
    const long long a0 = pd_at(R.index, R.cap, i, 0);
    const float ri[3] = {R.rpos[3 * a0], R.rpos[3 * a0 + 1], R.rpos[3 * a0 + 2]};
    const int m = pd_size(R.index, R.cap, R.total, R.n, i);
    const float4 xi = __ldg(x + i), yi = __ldg(y4 + i);
    __syncwarp();  // every lane has read slot 0 before lane 0 of the group rewrites it
    if (!L.valid) return;
    for (int e0 = L.sub; e0 < m; e0 += kPlG * 2) {
        float4 xj[2], yj[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int j = e0 + u * kPlG < m ? R.ridx[a0 + e0 + u * kPlG] : i;
            xj[u] = __ldg(x + j);
            yj[u] = __ldg(y4 + j);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (e0 + u * kPlG >= m) break;
            float* rj = R.rpos + 3 * (a0 + e0 + u * kPlG);
            const float s = yi.z + yj[u].z;
            const float ya = (yi.x + yj[u].x) / 2, yb = (yi.y + yj[u].y) / 2;
            float q[3], nq[3], iso[3], dq[3];
            for (int a = 0; a < 3; ++a) {
                q[a] = rj[a] - ri[a];
                nq[a] = q[a] * s / 2;
                iso[a] = nq[a] - q[a];
                dq[a] = q[a];
            }
            unit_or_zero3(dq);
            const float pl = len3(xj[u].x - xi.x, xj[u].y - xi.y, xj[u].z - xi.z);
            for (int a = 0; a < 3; ++a) rj[a] = (rj[a] + ya * iso[a]) + yb * (pl * dq[a] - nq[a]);
        }
    }
}

// PM_ComputeInverseDeformation (ElastoplasticityModule.cu:389-471).
__global__ void __launch_bounds__(128)
    k_pl_invF(RestView R, const float* __restrict__ x, float h, float* __restrict__ invF)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= R.n) return;
    const long long a0 = pd_at(R.index, R.cap, i, 0);
    const float ri[3] = {R.rpos[3 * a0], R.rpos[3 * a0 + 1], R.rpos[3 * a0 + 2]};
    const int m = pd_size(R.index, R.cap, R.total, R.n, i);
    float tw = 0.f, cur[3][3] = {}, ref[3][3] = {};
    for (int e = 0; e < m; ++e) {
        const long long at = pd_at(R.index, R.cap, i, e);
        const int j = R.ridx[at];
        const float* rj = R.rpos + 3 * at;
        const float r = len3(rj[0] - ri[0], rj[1] - ri[1], rj[2] - ri[2]);
        if (r > kEpsilon) {
            const float wt = corr_w(r, h);
            float p[3], q[3];
            for (int a = 0; a < 3; ++a) {
                p[a] = (x[3 * j + a] - x[3 * i + a]) / h;
                q[a] = (rj[a] - ri[a]) / h;
            }
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    cur[a][b] += p[a] * p[b] * wt;
                    ref[a][b] += q[a] * p[b] * wt;
                }
            tw += wt;
        }
    }
    if (tw < kEpsilon) tw = 1.0f;
    const float s = 1.0f / tw;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            ref[a][b] *= s;
            cur[a][b] *= s;
        }
    float Ci[3][3], out[3][3];
    clamped_inverse(cur, (double)0.00001f, 1.0 / (double)0.00001f, Ci);
    mat_mul(ref, Ci, out);
    if (det3f(out) < kEpsilon)
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) out[a][b] = (a == b) ? 1.0f : 0.0f;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) invF[9LL * i + 3 * a + b] = out[a][b];
}

// PM_ReconfigureRestShape (ElastoplasticityModule.cu:373-387).
__global__ void __launch_bounds__(256)
    k_pl_recon_sizes(RestView R, const unsigned char* __restrict__ byield, const int* __restrict__ nindex, int ncap,
                     long long ntotal, int* __restrict__ sizes)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= R.n) return;
    sizes[i] = byield[i] ? pd_size(nindex, ncap, ntotal, R.n, i) : pd_size(R.index, R.cap, R.total, R.n, i);
}

// PM_ReconstructRestShape (ElastoplasticityModule.cu:309-371) into CSR `off`.
__global__ void __launch_bounds__(128)
    k_pl_recon_fill(RestView R, const float* __restrict__ x, unsigned char* __restrict__ byield,
                    const float* __restrict__ invF, const int* __restrict__ nindex,
                    const int* __restrict__ nelements, int ncap, long long ntotal, const int* __restrict__ off,
                    int* __restrict__ new_idx, float* __restrict__ new_pos)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= R.n) return;
    const long long o = off[i];
    if (!byield[i]) {
        const int m = pd_size(R.index, R.cap, R.total, R.n, i);
        for (int e = 0; e < m; ++e) {
            const long long at = pd_at(R.index, R.cap, i, e);
            new_idx[o + e] = R.ridx[at];
            for (int a = 0; a < 3; ++a) new_pos[3 * (o + e) + a] = R.rpos[3 * at + a];
        }
    } else {
        const int m = pd_size(nindex, ncap, ntotal, R.n, i);
        const float* Fi = invF + 9LL * i;
        for (int e = 0; e < m; ++e) {
            const int j = nelements[pd_at(nindex, ncap, i, e)];
            const float* Fj = invF + 9LL * j;
            float M[3][3], d[3], np[3];
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) M[a][b] = 0.5f * (Fi[3 * a + b] + Fj[3 * a + b]);
            for (int a = 0; a < 3; ++a) d[a] = x[3 * j + a] - x[3 * i + a];
            for (int a = 0; a < 3; ++a) np[a] = x[3 * i + a] + ((M[a][0] * d[0] + M[a][1] * d[1]) + M[a][2] * d[2]);
            if (i != j || e == 0) {
                new_idx[o + e] = j;
                for (int a = 0; a < 3; ++a) new_pos[3 * (o + e) + a] = np[a];
            } else {
                new_idx[o + e] = new_idx[o];
                for (int a = 0; a < 3; ++a) new_pos[3 * (o + e) + a] = new_pos[3 * o + a];
                new_idx[o] = j;
                for (int a = 0; a < 3; ++a) new_pos[3 * o + a] = np[a];
            }
        }
    }
    byield[i] = 0;
}

// FractureModule's PM_ComputeInvariants (FractureModule.cu:15-105).
__global__ void __launch_bounds__(kPlBlock)
    k_pl_fracture(RestView R, const float4* __restrict__ x, float* __restrict__ bulk, float h, float A, float B,
                  float mu, float lambda)
{
    const PlLane L = pl_lane(R.n);
    const int i = L.i;
    float I1, J2;
    invariants(R, x, h, i, L.sub, I1, J2);
    if (!L.valid || L.sub != 0) return;
    const float sJ2 = J2 * mu * bulk[i];
    const float sD1 = (1.0f - I1) * lambda * bulk[i];
    if (sJ2 > A + B * sD1) bulk[i] = 0.0f;
}

__global__ void __launch_bounds__(256) k_pl_fill_u8(unsigned char* __restrict__ p, long long m, unsigned char v)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) p[t] = v;
}

static RestView rest_view(pk_ctx* c)
{
    return RestView{c->pd_index, c->pd_cap, c->pd_total, c->pd_n, c->pd_rest_idx, c->pd_rest_pos};
}

static unsigned blocks(long long m, int b) { return (unsigned)((m + b - 1) / b); }

int pl_rotate(pk_ctx* c, const float* x, float h, cudaStream_t st)
{
    if (c->pd_n <= 0) return 0;
    const RestView R = rest_view(c);
    int l = 0;
    const float4* x4 = pd_pack(c, x, true, l, st);
    if (!x4) return -1;
    const BondView V{c->pd_bond, x4};
    const unsigned g = blocks((long long)c->pd_n * kPlG, kPlBlock);
    k_pl_rot_sums<<<g, kPlBlock, 0, st>>>(R, V, h, c->pl_mk);
    k_pl_rot_solve<<<blocks(c->pd_n, 128), 128, 0, st>>>(c->pd_n, h, c->pl_mk);
    k_pl_rot_apply<<<g, kPlBlock, 0, st>>>(R, c->pl_mk);
    return l + 3;
}

int pl_yield(pk_ctx* c, const float* x, const pk_plastic_params* p, cudaStream_t st)
{
    const int n = c->pd_n;
    if (n <= 0) return 0;
    const RestView R = rest_view(c);
    int l = 0;
    const float4* x4 = pd_pack(c, x, false, l, st);
    if (!x4) return -1;
    const unsigned g = blocks((long long)n * kPlG, kPlBlock);
    float4* const y4 = reinterpret_cast<float4*>(c->pl_mk);  // the rotation's scratch
    k_pl_invariants<<<g, kPlBlock, 0, st>>>(R, x4, c->pd_bulk, p->horizon, p->A, p->B, p->mu, p->lambda, c->pl_y1,
                                            c->pl_y2, c->pl_i1, c->pl_yield, y4);
    k_pl_yield<<<g, kPlBlock, 0, st>>>(R, x4, y4);
    return l + 2;
}

int pl_fracture(pk_ctx* c, const float* x, const pk_plastic_params* p, cudaStream_t st)
{
    if (c->pd_n <= 0) return 0;
    int l = 0;
    const float4* x4 = pd_pack(c, x, false, l, st);
    if (!x4) return -1;
    k_pl_fracture<<<blocks((long long)c->pd_n * kPlG, kPlBlock), kPlBlock, 0, st>>>(rest_view(c), x4, c->pd_bulk,
                                                                                    p->horizon, p->A, p->B, p->mu,
                                                                                    p->lambda);
    return l + 1;
}

int pl_enable_all(pk_ctx* c, cudaStream_t st)
{
    if (c->pd_n <= 0) return 0;
    k_pl_fill_u8<<<blocks(c->pd_n, 256), 256, 0, st>>>(c->pl_yield, c->pd_n, 1);
    return 1;
}

int pl_recon_begin(pk_ctx* c, const float* x, const int* nindex, int ncap, long long ntotal, float h,
                   cudaStream_t st)
{
    const int n = c->pd_n;
    if (n <= 0) return 0;
    const RestView R = rest_view(c);
    k_pl_recon_sizes<<<blocks(n, 256), 256, 0, st>>>(R, c->pl_yield, nindex, ncap, ntotal, c->pl_sizes);
    exclusive_scan(c->pl_sizes, n, c->pl_off, c->scan_part, st);
    k_pl_invF<<<blocks(n, 128), 128, 0, st>>>(R, x, h, c->pl_invF);
    return 2 + scan_launches();
}

int pl_recon_fill(pk_ctx* c, const float* x, const int* nindex, const int* nelements, int ncap, long long ntotal,
                  cudaStream_t st)
{
    const int n = c->pd_n;
    if (n <= 0) return 0;
    k_pl_recon_fill<<<blocks(n, 128), 128, 0, st>>>(rest_view(c), x, c->pl_yield, c->pl_invF, nindex, nelements,
                                                   ncap, ntotal, c->pl_off, c->pl_rest_idx2, c->pl_rest_pos2);
    return 1;
}

int pl_fill_alive(pk_ctx* c, long long bonds, cudaStream_t st)
{
    if (bonds <= 0) return 0;
    k_pl_fill_u8<<<blocks(bonds, 256), 256, 0, st>>>(c->pd_alive, bonds, 1);
    return 1;
}

}  // namespace pk
