// pk_pd_adj.cu -- the peridynamics projection as gathers, its adjoint, and
// checkpointed rollouts (float forward with a double reverse pass, and an
// all-double rollout for reference gradients).
//
// Forward: one projection iteration of ElasticityModule::solveElasticity
// (EM_EnforceElasticity, ElasticityModule.cu:123-242, + K_UpdatePosition
// :281-292) is
//     x'_i = (x_old,i + D_i(x)) / (1 + W_i)
// with, over the alive bonds i->j of i's frozen rest shape (r_ij = |rest_i -
// rest_j| > 0.01 h) and the alive bonds k->i that name i (the incoming list,
// built once because the bonds are frozen):
//     D_i = sum_{i->j} mu_ij (x_j + r n(F_i e_ij)) + la_ij (x_j + r n(x_i - x_j))
//         + sum_{k->i} mu_ki (x_k - r n(F_k e_ki)) + la_ki (x_k - r n(x_k - x_i))
//     W_i = sum_{i->j} (mu_ij + la_ij) + sum_{k->i} (mu_ki + la_ki)
// mu_ij = mu bulk_i wrr(r), la_ij = lambda bulk_i wrr(r), e_ij = rest_i -
// rest_j, n(u) = u/|u| (0 below epsilon), and F_i the deformation gradient of
// EM_EnforceElasticity's first loop (identity when det F < -0.001).  The
// reference scatters the k->i terms with atomics; here every particle gathers
// them, so the sums have a fixed order and a recomputed trajectory repeats the
// forward bit for bit, which the adjoint relies on.
//
// Adjoint of one iteration, given g = dL/dx':  a_i = g_i/(1 + W_i) (the
// adjoint of D_i and of x_old,i); then
//   kernel B (per source i): Fbar_i = sum_{i->j} mu_ij r J_n(F_i e)^T (a_i - a_j) e^T,
//     the bulk_i gradient (a bond's weight w adds w*target to D and w to W at
//     both ends: d x'/d w = (target - x')/(1 + W)),
//     and G_i = dL/dFraw_i / (tw_i h), Fraw being the unscaled first-loop sum;
//   kernel C (per particle): dL/dx_i from the linear parts, the n(x_i - x_j)
//     terms (J_n(u) = (I - n n^T)/|u|) and F (x_j enters F_i through
//     (x_j - x_i)/h: + G_i q_j at j, - G_i q_j at i).
#include "pk_kernels.cuh"
#include "pk_pd_common.cuh"

namespace pk {

// Four values as one 16-byte (float) or 32-byte (double) group, loaded and
// stored with 16-byte accesses: positions and adjoint vectors are gathered by
// bond, and a group costs one load where three scalars cost three.
template <class R>
struct alignas(16) Q4 {
    R x, y, z, w;
};
__device__ __forceinline__ Q4<float> ldq(const Q4<float>* p)
{
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    return Q4<float>{q.x, q.y, q.z, q.w};
}
__device__ __forceinline__ Q4<double> ldq(const Q4<double>* p)
{
    const double2 a = __ldg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldg(reinterpret_cast<const double2*>(p) + 1);
    return Q4<double>{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void stq(Q4<float>* p, float x, float y, float z, float w)
{
    *reinterpret_cast<float4*>(p) = make_float4(x, y, z, w);
}
__device__ __forceinline__ void stq(Q4<double>* p, double x, double y, double z, double w)
{
    reinterpret_cast<double2*>(p)[0] = make_double2(x, y);
    reinterpret_cast<double2*>(p)[1] = make_double2(z, w);
}

template <class R>
struct V3 {
    R x, y, z;
};
// The first three values of a group in the precision R.
template <class R, class RX>
__device__ __forceinline__ V3<R> ld3q(const Q4<RX>* p)
{
    const Q4<RX> q = ldq(p);
    return V3<R>{(R)q.x, (R)q.y, (R)q.z};
}
template <class R>
__device__ __forceinline__ R dot3(V3<R> a, V3<R> b)
{
    return a.x * b.x + a.y * b.y + a.z * b.z;
}

// 1/sqrt of a normal number.
__device__ __forceinline__ float rsq(float v)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ double rsq(double v) { return rsqrt(v); }

// 1/|u| from |u|^2, or 0 where v.norm() > EPSILON fails and the reference
// takes the zero vector for the unit vector (ElasticityModule.cu:211-212).
template <class R>
__device__ __forceinline__ R inv_len(R l2)
{
    return l2 > (R)(kEpsilon * kEpsilon) ? rsq(l2) : (R)0;
}

struct PdBonds {
    const int* index;
    int cap;
    long long total;
    int n;
    // Compact bonds: (rest_j - rest_i, j, or ~j for a broken bond), 16 bytes
    // read with one load where the rest shape's index, position and alive byte
    // took five.  A particle's bonds take the rest shape's places in ascending
    // order of j (k_pd_order): the lanes of a warp then gather positions from
    // runs of neighbours instead of from the list's order.  alive, the bond
    // slots and the incoming lists are in this order.
    float4* bond;
    unsigned char* alive;
    const float* invK;
    const int* in_off;   // incoming bonds k->i of particle i: in_list[in_off[i] .. in_off[i+1])
    const int2* in_list; // (source k, bond slot)
    const int* in_slot;  // the bond slots of in_list alone
    float h, mu, lambda;
    float inv_h;         // 1/h: the kernels multiply where the reference divides
};

// Bond geometry: the squared rest length, the rest length, and CorrectedKernel
// Weight and WeightRR (Kernel.h:99-142) with q = r / h.  Every rounding is
// explicit, so each kernel gets the same bits whatever the compiler's
// contraction choices at its call site: the reverse pass must see the
// forward's r (a one-ulp difference in r between the forward's F and the
// reverse's recomputation moved the double adjoint of a 2,000-iteration
// rollout by 1.4e-4).
__device__ __forceinline__ float bond_r2(const float4& b)
{
    return __fmaf_rn(b.z, b.z, __fmaf_rn(b.x, b.x, __fmul_rn(b.y, b.y)));
}
__device__ __forceinline__ float bond_len(float r2) { return __fmul_rn(r2, rsq(fmaxf(r2, 1e-30f))); }
__device__ __forceinline__ float corr_w_f(float r, float inv_h)
{
    const float q = __fmul_rn(r, inv_h);
    const float qq = __fmul_rn(q, q);
    return __fmul_rn(__fmul_rn(qq, q), fmaxf(__fsub_rn(1.0f, qq), 0.0f));
}
__device__ __forceinline__ float corr_wrr_f(float r, float inv_h)
{
    const float q = __fmul_rn(r, inv_h);
    return __fmul_rn(__fmul_rn(q, fmaxf(__fsub_rn(1.0f, __fmul_rn(q, q)), 0.0f)), __fmul_rn(inv_h, inv_h));
}

// Every particle is handled by a group of kPdG lanes of one warp: lane `sub`
// takes bonds sub, sub + kPdG, ... and the group's partial sums are combined
// with xor shuffles in a fixed order (deterministic, so a replayed rollout
// repeats the forward bit for bit).
constexpr int kPdG = 8;
constexpr int kPdBlock = 128;
constexpr unsigned kPdAll = 0xffffffffu;

template <class R>
__device__ __forceinline__ R gsum(R v)
{
#pragma unroll
    for (int o = kPdG / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(kPdAll, v, o);
    return v;
}

struct PdLane {
    int i, sub;
    bool valid;
};
__device__ __forceinline__ PdLane pd_lane(int n)
{
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    PdLane L;
    L.i = gid / kPdG;
    L.sub = gid % kPdG;
    L.valid = L.i < n;
    if (!L.valid) L.i = n - 1;  // idle lanes of the last group mirror a valid particle, write nothing
    return L;
}

// The compact bonds of the current rest shape (after every change of it).
__global__ void __launch_bounds__(kPdBlock)
    k_pd_bonds(PdBonds B, const int* __restrict__ raw, const int* __restrict__ ridx, const float* __restrict__ rpos)
{
    const PdLane L = pd_lane(B.n);
    if (!L.valid) return;
    const long long a0 = pd_at(B.index, B.cap, L.i, 0);
    const int m = pd_size(B.index, B.cap, B.total, B.n, L.i);
    if (m <= 0) return;
    const float r0 = rpos[3 * a0], r1 = rpos[3 * a0 + 1], r2 = rpos[3 * a0 + 2];
    for (int e = L.sub; e < m; e += kPdG) {
        const long long at = raw[a0 + e];
        const int j = ridx[at];
        B.bond[a0 + e] = make_float4(rpos[3 * at] - r0, rpos[3 * at + 1] - r1, rpos[3 * at + 2] - r2,
                                     __int_as_float(B.alive[a0 + e] ? j : ~j));
    }
}

// W_i (the denominator of K_UpdatePosition) for the reverse pass: constant
// while bulk and the bonds are.
template <class R, class RB>
__global__ void __launch_bounds__(kPdBlock) k_pd_W(PdBonds B, const RB* __restrict__ bulk, R* __restrict__ W)
{
    const PdLane L = pd_lane(B.n);
    const int i = L.i;
    const long long a0 = pd_at(B.index, B.cap, i, 0);
    const int m = pd_size(B.index, B.cap, B.total, B.n, i);
    const R ml = (R)B.mu + (R)B.lambda;
    R w = 0;
    auto weight = [&](const float4& b, int src) {
        const float r = bond_len(bond_r2(b));
        if (__float_as_int(b.w) >= 0 && r > 0.01f * B.h) w += ml * (R)bulk[src] * (R)corr_wrr_f(r, B.inv_h);
    };
    for (int e = L.sub; e < m; e += kPdG) weight(__ldg(B.bond + a0 + e), i);
    for (int t = B.in_off[i] + L.sub; t < B.in_off[i + 1]; t += kPdG) {
        const int2 kb = B.in_list[t];
        weight(__ldg(B.bond + kb.y), kb.x);
    }
    w = gsum(w);
    if (L.valid && L.sub == 0) W[i] = w;
}

// One projection iteration with each bond's term formed once.  A bond i->j's
// term in D_j (the incoming sum above, seen from j) uses F_i, x_i, x_j and
// the rest vector of i's shape, exactly like its term in D_i with the sign
// flipped: mu (x_i - x_j - r n(F_i e)) + la (x_i - x_j - r n(x_i - x_j)) =
// -t_ij.  So k_pd_FP computes F_i and every outgoing t_ij of particle i, keeps
// the sum in own[i] and each t_ij in its bond slot (0 for a dead or too-short
// bond), and k_pd_gather sums -t over the incoming slots: no neighbour F is
// gathered and no bond is evaluated twice.
//
// F_i (first loop of EM_EnforceElasticity): sum p q^T / tw K^-1 with
// p = (x_j - x_i)/h, q = e wt / h, e = rest_j - rest_i, the identity when
// det F < -0.001.  Both walks load kPdBatch bonds, then their neighbours'
// positions, before the first is used; the second finds the bonds in L1.  With
// d = x_j - x_i and e the rest vector, a bond's term is
//   t = w (mu + la (1 - r/|d|)) d - w mu r/|F e| F e,   w = bulk_i wrr(r),
// two multiply-adds per component.
//
// Bound by L1 (75% of its throughput: 16-byte gathers of positions) at 2.6 TB/s
// of DRAM.  524,288 particles with 80 bonds, per launch: 271 us (498 before the
// compact bonds, their order and the batches).  Of the variants on the same
// box: bonds in list order 385-509 us; one bond ahead 329 us, batches of 2
// 293 us, of 5 271 us; with the first walk's bonds kept in shared memory
// instead of L1 295 us (batches of 5); 4 lanes per particle 281 us, 16 lanes
// 364 us (batches of 2).
// kBreak (the first iteration of a solve with a stretch limit): a bond dies
// for good once |x_i - x_j| > (1 + s) |rest_i - rest_j|, lengths rounded as
// Vector3f::norm compiles (no reference counterpart).
constexpr int kPdBatch = 5;  // bonds a lane has in flight (cap 80 over 8 lanes: two batches)
template <class R, bool kBreak>
__global__ void __launch_bounds__(kPdBlock)
    k_pd_FP(PdBonds B, const Q4<R>* __restrict__ x, const R* __restrict__ bulk, R* __restrict__ Fout,
            float* __restrict__ twout, Q4<R>* __restrict__ own, Q4<R>* __restrict__ tslot, float stretch)
{
    const PdLane L = pd_lane(B.n);
    const int i = L.i;
    const long long a0 = pd_at(B.index, B.cap, i, 0);
    const int m = pd_size(B.index, B.cap, B.total, B.n, i);
    float4* const bond = B.bond + a0;
    const V3<R> ci = ld3q<R>(x + i);
    R F[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    float tw = 0.f;
    constexpr int U = sizeof(R) == 4 ? kPdBatch : 1;
    const float4 none = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    for (int e0 = L.sub; e0 < m; e0 += kPdG * U) {
        float4 b[U];
        V3<R> xj[U];
#pragma unroll
        for (int u = 0; u < U; ++u) b[u] = e0 + u * kPdG < m ? bond[e0 + u * kPdG] : none;
#pragma unroll
        for (int u = 0; u < U; ++u) xj[u] = ld3q<R>(x + (__float_as_int(b[u].w) >= 0 ? __float_as_int(b[u].w) : i));
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = e0 + u * kPdG;
            V3<R> d{xj[u].x - ci.x, xj[u].y - ci.y, xj[u].z - ci.z};
            const float r2 = bond_r2(b[u]);
            if (kBreak && __float_as_int(b[u].w) >= 0) {
                const float c0 = (float)d.x, c1 = (float)d.y, c2 = (float)d.z;
                const float lr = __fsqrt_rn(r2);
                const float lc = __fsqrt_rn(__fmaf_rn(c2, c2, __fmaf_rn(c0, c0, __fmul_rn(c1, c1))));
                if (lc > __fmul_rn(__fadd_rn(1.0f, stretch), lr)) {
                    b[u].w = __int_as_float(~__float_as_int(b[u].w));
                    d = V3<R>{0, 0, 0};
                    if (L.valid) {
                        bond[e].w = b[u].w;
                        B.alive[a0 + e] = 0;
                    }
                }
            }
            const float wt = __float_as_int(b[u].w) >= 0 && r2 > kEpsilon * kEpsilon
                                 ? corr_w_f(bond_len(r2), B.inv_h) : 0.0f;
            const R g0 = (R)__fmul_rn(b[u].x, wt), g1 = (R)__fmul_rn(b[u].y, wt), g2 = (R)__fmul_rn(b[u].z, wt);
            F[0][0] += d.x * g0;
            F[0][1] += d.x * g1;
            F[0][2] += d.x * g2;
            F[1][0] += d.y * g0;
            F[1][1] += d.y * g1;
            F[1][2] += d.y * g2;
            F[2][0] += d.z * g0;
            F[2][1] += d.z * g1;
            F[2][2] += d.z * g2;
            tw += wt;
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) F[a][b] = gsum(F[a][b]);
    tw = gsum(tw);
    R s = (R)B.inv_h * (R)B.inv_h;
    if (tw > kEpsilon) {
        s = s / (R)tw;
        const float* K = B.invK + 9LL * i;
        R G[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)
                G[a][b] = F[a][0] * (R)K[b] + F[a][1] * (R)K[3 + b] + F[a][2] * (R)K[6 + b];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) F[a][b] = G[a][b];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) F[a][b] *= s;
    const R det = F[0][0] * (F[1][1] * F[2][2] - F[1][2] * F[2][1]) -
                  F[0][1] * (F[1][0] * F[2][2] - F[1][2] * F[2][0]) +
                  F[0][2] * (F[1][0] * F[2][1] - F[1][1] * F[2][0]);
    const bool ident = det < (R)-0.001;
    if (ident) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) F[a][b] = (a == b) ? (R)1 : (R)0;
    }
    if (Fout != nullptr && L.valid && L.sub == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) Fout[9LL * i + 3 * a + b] = F[a][b];
        twout[i] = ident ? -1.0f - tw : tw;
    }
    V3<R> acc{0, 0, 0};
    R accw = 0;  // the particle's own bond weights (W, the target's share is in the slots)
    const R bulk_i = bulk[i];
    const R mu = (R)B.mu, la = (R)B.lambda, ml = mu + la;
    for (int e0 = L.sub; e0 < m; e0 += kPdG * U) {
        float4 b[U];
        V3<R> xj[U];
#pragma unroll
        for (int u = 0; u < U; ++u) b[u] = e0 + u * kPdG < m ? bond[e0 + u * kPdG] : none;
#pragma unroll
        for (int u = 0; u < U; ++u) xj[u] = ld3q<R>(x + (__float_as_int(b[u].w) >= 0 ? __float_as_int(b[u].w) : i));
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = e0 + u * kPdG;
            const float r = bond_len(bond_r2(b[u]));
            const V3<R> d{xj[u].x - ci.x, xj[u].y - ci.y, xj[u].z - ci.z};
            const R b0 = (R)b[u].x, b1 = (R)b[u].y, b2 = (R)b[u].z;
            const V3<R> f{F[0][0] * b0 + F[0][1] * b1 + F[0][2] * b2, F[1][0] * b0 + F[1][1] * b1 + F[1][2] * b2,
                          F[2][0] * b0 + F[2][1] * b1 + F[2][2] * b2};
            const R w = __float_as_int(b[u].w) >= 0 && r > 0.01f * B.h ? bulk_i * (R)corr_wrr_f(r, B.inv_h) : (R)0;
            const R wr = w * (R)r;
            const R ca = w * ml - wr * la * inv_len(dot3(d, d));
            const R cb = wr * mu * inv_len(dot3(f, f));
            // f = F (rest_j - rest_i): the reference's F e_ij is -f
            const V3<R> t{ca * d.x - cb * f.x, ca * d.y - cb * f.y, ca * d.z - cb * f.z};
            const R wb = ml * w;
            acc.x += t.x;
            acc.y += t.y;
            acc.z += t.z;
            accw += wb;
            if (L.valid && e < m) stq(tslot + a0 + e, t.x, t.y, t.z, wb);
        }
    }
    acc.x = gsum(acc.x);
    acc.y = gsum(acc.y);
    acc.z = gsum(acc.z);
    accw = gsum(accw);
    if (L.valid && L.sub == 0) stq(own + i, acc.x, acc.y, acc.z, accw);
}

// Sum of the slots of i's incoming bonds over the lane group, kPdU loads in
// flight per lane.
constexpr int kPdU = 4;
template <class R>
__device__ __forceinline__ Q4<R> gather_slots(const PdBonds& B, const Q4<R>* __restrict__ slot, int i, int sub)
{
    Q4<R> in{0, 0, 0, 0};
    const int t1 = B.in_off[i + 1];
    for (int t = B.in_off[i] + sub; t < t1; t += kPdG * kPdU) {
        int at[kPdU];
#pragma unroll
        for (int u = 0; u < kPdU; ++u) at[u] = t + u * kPdG < t1 ? __ldg(B.in_slot + t + u * kPdG) : -1;
        Q4<R> q[kPdU];
#pragma unroll
        for (int u = 0; u < kPdU; ++u) q[u] = at[u] >= 0 ? ldq(slot + at[u]) : Q4<R>{0, 0, 0, 0};
#pragma unroll
        for (int u = 0; u < kPdU; ++u) {
            in.x += q[u].x;
            in.y += q[u].y;
            in.z += q[u].z;
            in.w += q[u].w;
        }
    }
    in.x = gsum(in.x);
    in.y = gsum(in.y);
    in.z = gsum(in.z);
    in.w = gsum(in.w);
    return in;
}

// xn = (xold + own - sum of the incoming bond terms) / (1 + W), written about
// x_i: the bond targets enter as offsets from x_i, which keeps float accuracy
// at the scale of the bonds instead of the scale of the coordinates.  W = the
// particle's own bond weights + those of the bonds naming it (each bond's
// weight rides in its slot's fourth value, so W follows broken bonds and
// changed stiffness without a pass of its own).  kLast writes the caller's x
// (3 per particle) and, with v, v += (xn - xold)/dt (K_UpdateVelocity,
// ElasticityModule.cu:295-306) instead of the next iterate.  Bound by the
// scattered 16-byte slots; four in flight per lane: 154 us per launch at 524,288
// particles with 80 bonds, one ahead 184.
template <class R, bool kLast>
__global__ void __launch_bounds__(kPdBlock)
    k_pd_gather(PdBonds B, const Q4<R>* __restrict__ x, const Q4<R>* __restrict__ xold,
                const Q4<R>* __restrict__ own, const Q4<R>* __restrict__ tslot, Q4<R>* __restrict__ xn,
                R* __restrict__ xout, R* __restrict__ v, R dt)
{
    const PdLane L = pd_lane(B.n);
    const int i = L.i;
    const Q4<R> in = gather_slots(B, tslot, i, L.sub);
    if (!L.valid || L.sub != 0) return;
    const V3<R> ci = ld3q<R>(x + i), xo = ld3q<R>(xold + i);
    const Q4<R> oi = ldq(own + i);
    const R den = (R)1 + (oi.w + in.w);
    const R y0 = ci.x + ((xo.x - ci.x) + (oi.x - in.x)) / den;
    const R y1 = ci.y + ((xo.y - ci.y) + (oi.y - in.y)) / den;
    const R y2 = ci.z + ((xo.z - ci.z) + (oi.z - in.z)) / den;
    if (!kLast) {
        stq(xn + i, y0, y1, y2, (R)0);
        return;
    }
    const long long o = 3LL * i;
    xout[o] = y0;
    xout[o + 1] = y1;
    xout[o + 2] = y2;
    if (v != nullptr) {
        v[o] += (y0 - xo.x) / dt;
        v[o + 1] += (y1 - xo.y) / dt;
        v[o + 2] += (y2 - xo.z) / dt;
    }
}

// ---- adjoint of one iteration

// Reverse pass of one projection iteration, per source particle i (8 lanes):
// the first walk over i's bonds forms F-bar_i (through the normalisation
// Jacobian of n(F e)), the stiffness gradient of bulk_i and the terms of
// dL/dx that do not go through F; every lane of the group then forms G_i =
// dL/dF_raw / (tw h^2) (0 when the identity was taken); the second walk adds
// F's share.  A bond k->i contributes to dL/dx_i through F_k and the
// n(x_k - x_i) term, and that contribution is formed by the source k, which
// holds G_k, x_k, a_k and the bond's rest vector: G_k q + dw a_k - u, u the
// normalisation adjoint of n(x_k - x_i), the same u as in k's own term.  k
// keeps its own sum in gown[k] and the partner terms in the bond slots, which
// k_pd_adjC_gather adds.  The second walk reads back its own bond slots, so it
// gathers nothing and takes no square root; G never goes through global
// memory.  Bound by double arithmetic and the gathers of x, x', a in turn: 123
// us per launch at 65,536 particles with 80 bonds, 184 before the compact
// bonds, the direct terms in the first walk and one reciprocal square root in
// place of each square root and division.  On the same box: the partner terms
// in shared memory 137 us, one bond at a time 142, 3 blocks per SM with two
// bonds 144, 5 blocks 135.
constexpr int kAdjBatch = 2;  // bonds a lane has in flight
template <class R, class RX>
__global__ void __launch_bounds__(kPdBlock, 4)
    k_pd_adjBC(PdBonds B, const Q4<RX>* __restrict__ x, const Q4<RX>* __restrict__ xn, const RX* __restrict__ bulk,
               const RX* __restrict__ Fst, const float* __restrict__ twst, const Q4<R>* __restrict__ a,
               double* __restrict__ bulkbar, Q4<R>* __restrict__ gown, Q4<R>* __restrict__ slot)
{
    const PdLane L = pd_lane(B.n);
    const int i = L.i;
    const long long a0 = pd_at(B.index, B.cap, i, 0);
    const V3<R> ci = ld3q<R>(x + i), ai = ld3q<R>(a + i);
    const R bulk_i = (R)bulk[i];
    const int m = pd_size(B.index, B.cap, B.total, B.n, i);
    const R mu = (R)B.mu, la = (R)B.lambda, ml = mu + la;
    R G[3][3];
    V3<R> out{0, 0, 0};
    // terms of one bond that do not go through F: dL/dx_i in out, the
    // target's share returned
    auto direct = [&](const V3<R>& xj, const V3<R>& aj, const V3<R>& da, R w, R rr, R& dnc) {
        const V3<R> c{ci.x - xj.x, ci.y - xj.y, ci.z - xj.z};
        const R ic = inv_len(dot3(c, c));
        const V3<R> nc{c.x * ic, c.y * ic, c.z * ic};
        dnc = dot3(nc, da);
        const R lr = la * w * rr * ic, dw = ml * w;
        const V3<R> u{lr * (da.x - nc.x * dnc), lr * (da.y - nc.y * dnc), lr * (da.z - nc.z * dnc)};
        out.x += dw * aj.x + u.x;
        out.y += dw * aj.y + u.y;
        out.z += dw * aj.z + u.z;
        return V3<R>{dw * ai.x - u.x, dw * ai.y - u.y, dw * ai.z - u.z};
    };
    {
        // the forward's F of this iterate, and its tw (negated: identity taken)
        R F[3][3];
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int q = 0; q < 3; ++q) F[p][q] = (R)Fst[9LL * i + 3 * p + q];
        const V3<R> yi = ld3q<R>(xn + i);
        R Fb[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        R gb = 0;  // d L / d bulk_i
        constexpr int U = kAdjBatch;
        for (int e0 = L.sub; e0 < m; e0 += kPdG * U) {
            float4 bb[U];
            V3<R> xu[U], au[U], yu[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                bb[u] = e0 + u * kPdG < m ? __ldg(B.bond + a0 + e0 + u * kPdG)
                                          : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = __float_as_int(bb[u].w) >= 0 ? __float_as_int(bb[u].w) : i;
                xu[u] = ld3q<R>(x + j);
                au[u] = ld3q<R>(a + j);
                yu[u] = ld3q<R>(xn + j);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + u * kPdG;
                if (e >= m) break;
                const float4 b = bb[u];
                const float r = bond_len(bond_r2(b));
                V3<R> pt{0, 0, 0};
                if (__float_as_int(b.w) >= 0 && r > 0.01f * B.h) {
                    const V3<R> xj = xu[u], aj = au[u], yj = yu[u];
                    const R b0 = (R)b.x, b1 = (R)b.y, b2 = (R)b.z;
                    // n(F e_ij) with e_ij = -(b0, b1, b2)
                    const V3<R> f{-(F[0][0] * b0 + F[0][1] * b1 + F[0][2] * b2),
                                  -(F[1][0] * b0 + F[1][1] * b1 + F[1][2] * b2),
                                  -(F[2][0] * b0 + F[2][1] * b1 + F[2][2] * b2)};
                    const R fi = inv_len(dot3(f, f));
                    const V3<R> nf{f.x * fi, f.y * fi, f.z * fi};
                    const V3<R> da{ai.x - aj.x, ai.y - aj.y, ai.z - aj.z};
                    const R rr = (R)r, wrr = (R)corr_wrr_f(r, B.inv_h), w = bulk_i * wrr;
                    const R dnf = dot3(nf, da);
                    const R mr = mu * w * rr * fi;
                    const V3<R> ub{mr * (da.x - nf.x * dnf), mr * (da.y - nf.y * dnf), mr * (da.z - nf.z * dnf)};
                    Fb[0][0] -= ub.x * b0;
                    Fb[0][1] -= ub.x * b1;
                    Fb[0][2] -= ub.x * b2;
                    Fb[1][0] -= ub.y * b0;
                    Fb[1][1] -= ub.y * b1;
                    Fb[1][2] -= ub.y * b2;
                    Fb[2][0] -= ub.z * b0;
                    Fb[2][1] -= ub.z * b1;
                    Fb[2][2] -= ub.z * b2;
                    R dnc;
                    pt = direct(xj, aj, da, w, rr, dnc);
                    // the bond's weight w adds w target to D and w to W at both
                    // ends: a . (target - x') summed over them
                    const R base = dot3(ai, V3<R>{xj.x - yi.x, xj.y - yi.y, xj.z - yi.z}) +
                                   dot3(aj, V3<R>{ci.x - yj.x, ci.y - yj.y, ci.z - yj.z});
                    gb += wrr * (mu * (base + rr * dnf) + la * (base + rr * dnc));
                }
                if (L.valid) stq(slot + a0 + e, pt.x, pt.y, pt.z, (R)0);  // completed by the second walk
            }
        }
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int q = 0; q < 3; ++q) Fb[p][q] = gsum(Fb[p][q]);
        gb = gsum(gb);
        if (L.valid && L.sub == 0) bulkbar[i] += (double)gb;
        // G = dL/dF_raw / (tw h^2): F = (F_raw / (tw h^2)) K, so dL/dF_raw = F-bar K^T / (tw h^2)
        const float tws = twst[i];
        const bool ident = tws < 0.f;
        const float tw = ident ? -1.0f - tws : tws;
        R sc = ident ? (R)0 : (R)B.inv_h * (R)B.inv_h;
        if (tw > kEpsilon) {
            sc = sc / (R)tw;
            const float* K = B.invK + 9LL * i;
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    G[p][c] = (Fb[p][0] * (R)K[3 * c] + Fb[p][1] * (R)K[3 * c + 1] + Fb[p][2] * (R)K[3 * c + 2]) * sc;
        } else {
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int c = 0; c < 3; ++c) G[p][c] = Fb[p][c] * sc;
        }
    }
    for (int e = L.sub; e < m; e += kPdG) {
        const float4 b = __ldg(B.bond + a0 + e);
        const Q4<R> q = slot[a0 + e];  // this lane's own store of the first walk
        V3<R> pt{q.x, q.y, q.z};
        // F_i depends on x_i through -x_i g and on x_j through +x_j g, g = e wt
        const float r2 = bond_r2(b);
        if (__float_as_int(b.w) >= 0 && r2 > kEpsilon * kEpsilon) {
            const float wt = corr_w_f(bond_len(r2), B.inv_h);
            const R g0 = (R)__fmul_rn(b.x, wt), g1 = (R)__fmul_rn(b.y, wt), g2 = (R)__fmul_rn(b.z, wt);
            const V3<R> gq{G[0][0] * g0 + G[0][1] * g1 + G[0][2] * g2, G[1][0] * g0 + G[1][1] * g1 + G[1][2] * g2,
                           G[2][0] * g0 + G[2][1] * g1 + G[2][2] * g2};
            out.x -= gq.x;
            out.y -= gq.y;
            out.z -= gq.z;
            pt.x += gq.x;
            pt.y += gq.y;
            pt.z += gq.z;
        }
        if (L.valid) stq(slot + a0 + e, pt.x, pt.y, pt.z, (R)0);
    }
    out.x = gsum(out.x);
    out.y = gsum(out.y);
    out.z = gsum(out.z);
    if (L.valid && L.sub == 0) stq(gown + i, out.x, out.y, out.z, (R)0);
}

// g = dL/dx of the iterate.  Unless it is the step's first iterate, what the
// previous iteration's reverse needs comes with it: a = g/(1 + W) and
// xoldbar += a; the first iterate's g is kept for k_pd_adj_tail.  Bound by the
// scattered 32-byte slots; at 65,536 particles with 80 bonds 46 us per launch,
// 49 and 3.3 as two kernels.
template <class R>
__global__ void __launch_bounds__(kPdBlock)
    k_pd_adjC_gather(PdBonds B, const Q4<R>* __restrict__ gown, const Q4<R>* __restrict__ slot,
                     const R* __restrict__ W, bool first, Q4<R>* __restrict__ g, Q4<R>* __restrict__ a,
                     Q4<R>* __restrict__ xoldbar)
{
    const PdLane L = pd_lane(B.n);
    const int i = L.i;
    const Q4<R> in = gather_slots(B, slot, i, L.sub);
    if (!L.valid || L.sub != 0) return;
    const V3<R> o = ld3q<R>(gown + i);
    const V3<R> gi{o.x + in.x, o.y + in.y, o.z + in.z};
    if (first) {
        stq(g + i, gi.x, gi.y, gi.z, (R)0);
        return;
    }
    const R den = (R)1 + W[i];
    const V3<R> ai{gi.x / den, gi.y / den, gi.z / den};
    const Q4<R> xb = xoldbar[i];
    stq(a + i, ai.x, ai.y, ai.z, (R)0);
    stq(xoldbar + i, xb.x + ai.x, xb.y + ai.y, xb.z + ai.z, (R)0);
}

// ---- step pieces

// y = the caller's positions (3 per particle) as groups.
template <class R>
__global__ void __launch_bounds__(256) k_pd_pack(int n, const R* __restrict__ x, Q4<R>* __restrict__ y)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) stq(y + i, x[3LL * i], x[3LL * i + 1], x[3LL * i + 2], (R)0);
}

// The caller's layout of a group array.
template <class R>
__global__ void __launch_bounds__(256) k_pd_unpack(int n, const Q4<R>* __restrict__ y, R* __restrict__ x)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V3<R> q = ld3q<R>(y + i);
    x[3LL * i] = q.x;
    x[3LL * i + 1] = q.y;
    x[3LL * i + 2] = q.z;
}

// ParticleIntegrator without a force: v += dt g, y = x + dt v.  x: 3 per
// particle, or (xq given) the previous step's last iterate.
template <class R>
__global__ void __launch_bounds__(256)
    k_pd_integrate(int n, const R* __restrict__ x, const Q4<R>* __restrict__ xq, R* __restrict__ v, R gx, R gy, R gz,
                   R dt, Q4<R>* __restrict__ y)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const R g[3] = {gx, gy, gz};
    R p[3], out[3];
    if (xq != nullptr) {
        const V3<R> q = ld3q<R>(xq + i);
        p[0] = q.x;
        p[1] = q.y;
        p[2] = q.z;
    } else {
        for (int c = 0; c < 3; ++c) p[c] = x[3LL * i + c];
    }
    for (int c = 0; c < 3; ++c) {
        const R vv = v[3LL * i + c] + dt * g[c];
        v[3LL * i + c] = vv;
        out[c] = p[c] + dt * vv;
    }
    stq(y + i, out[0], out[1], out[2], (R)0);
}

// v += (x - xold)/dt, x 3 per particle or (xq given) groups.
template <class R>
__global__ void __launch_bounds__(256)
    k_pd_vel(int n, R* __restrict__ v, const R* __restrict__ x, const Q4<R>* __restrict__ xq,
             const Q4<R>* __restrict__ xold, R dt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long o = 3LL * i;
    const V3<R> xo = ld3q<R>(xold + i);
    const V3<R> p = xq != nullptr ? ld3q<R>(xq + i) : V3<R>{x[o], x[o + 1], x[o + 2]};
    v[o] += (p.x - xo.x) / dt;
    v[o + 1] += (p.y - xo.y) / dt;
    v[o + 2] += (p.z - xo.z) / dt;
}

// Start of a step's reverse: g = xbar + vbar/dt (x_new feeds v_new), xoldbar =
// -vbar/dt; then a = g/(1 + W), xoldbar += a for the last iteration (none:
// g is kept for the tail).
template <class R>
__global__ void __launch_bounds__(256)
    k_pd_adj_head(int n, const R* __restrict__ xbar, const R* __restrict__ vbar, R dt, const R* __restrict__ W,
                  bool none, Q4<R>* __restrict__ g, Q4<R>* __restrict__ a, Q4<R>* __restrict__ xoldbar)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const R den = (R)1 + W[i];
    R gi[3], ai[3], xo[3];
    for (int c = 0; c < 3; ++c) {
        const R vd = vbar[3LL * i + c] / dt;
        gi[c] = xbar[3LL * i + c] + vd;
        ai[c] = gi[c] / den;
        xo[c] = none ? -vd : -vd + ai[c];
    }
    stq(g + i, gi[0], gi[1], gi[2], (R)0);
    stq(a + i, ai[0], ai[1], ai[2], (R)0);
    stq(xoldbar + i, xo[0], xo[1], xo[2], (R)0);
}

// End of a step's reverse: xbar' = g + xoldbar (x' is both x_0 and x_old),
// then through x' = x + dt v', v' = v + dt gravity: vbar += dt xbar', xbar = xbar'.
template <class R>
__global__ void __launch_bounds__(256)
    k_pd_adj_tail(int n, const Q4<R>* __restrict__ g, const Q4<R>* __restrict__ xoldbar, R dt, R* __restrict__ xbar,
                  R* __restrict__ vbar)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V3<R> gi = ld3q<R>(g + i), xo = ld3q<R>(xoldbar + i);
    const R xb[3] = {gi.x + xo.x, gi.y + xo.y, gi.z + xo.z};
    for (int c = 0; c < 3; ++c) {
        xbar[3LL * i + c] = xb[c];
        vbar[3LL * i + c] += dt * xb[c];
    }
}

// ---- incoming bonds (transpose of the frozen rest shape)

// The place of every compact bond in the rest shape: a particle's bonds in
// ascending order of their neighbour (equal neighbours in list order).  A warp
// per particle: rows of up to 128 bonds are held 4 per lane and each bond goes
// to its rank; longer rows keep the list's order, which only costs locality.
constexpr int kInSortWarps = 8;
__global__ void __launch_bounds__(kInSortWarps * 32)
    k_pd_order(int n, const int* __restrict__ index, int cap, long long total, const int* __restrict__ ridx,
               int* __restrict__ raw)
{
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kInSortWarps + (threadIdx.x >> 5);
    if (i >= n) return;  // the whole warp leaves together
    const long long a0 = pd_at(index, cap, i, 0);
    const int m = pd_size(index, cap, total, n, i);
    if (m > 128) {
        for (int e = lane; e < m; e += 32) raw[a0 + e] = (int)(a0 + e);
        return;
    }
    int j[4], rank[4] = {0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < 4; ++q) j[q] = 32 * q + lane < m ? ridx[a0 + 32 * q + lane] : 0x7fffffff;
#pragma unroll
    for (int sq = 0; sq < 4; ++sq) {
        if (32 * sq >= m) break;
        for (int sl = 0; sl < 32; ++sl) {
            const int w = __shfl_sync(0xffffffffu, j[sq], sl);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                rank[q] += w < j[q] || (w == j[q] && 32 * sq + sl < 32 * q + lane) ? 1 : 0;
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (32 * q + lane < m) raw[a0 + rank[q]] = (int)(a0 + 32 * q + lane);
}

__global__ void __launch_bounds__(256)
    k_in_count(int n, const int* __restrict__ index, int cap, long long total, const int* __restrict__ ridx,
               int* __restrict__ cnt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int m = pd_size(index, cap, total, n, i);
    for (int e = 1; e < m; ++e) {  // slot 0 is the particle itself
        const int j = ridx[pd_at(index, cap, i, e)];
        if (j != i && j >= 0 && j < n) atomicAdd(cnt + j, 1);
    }
}

__global__ void __launch_bounds__(256)
    k_in_fill(int n, const int* __restrict__ index, int cap, long long total, const int* __restrict__ ridx,
              const int* __restrict__ raw, const int* __restrict__ off, int* __restrict__ fill,
              int2* __restrict__ list)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long a0 = pd_at(index, cap, i, 0);
    const int m = pd_size(index, cap, total, n, i);
    for (int e = 0; e < m; ++e) {
        const int at = raw[a0 + e];
        if (at == a0) continue;  // the rest shape's slot 0 is the particle itself
        const int j = ridx[at];
        if (j != i && j >= 0 && j < n) list[off[j] + atomicAdd(fill + j, 1)] = make_int2(i, (int)(a0 + e));
    }
}

// Each particle's incoming bonds in ascending bond slot (a fixed order).  A
// warp per particle: lists of up to 128 entries are held 4 per lane and each
// entry goes to its rank (slots are distinct within a list); longer lists are
// sorted by lane 0 in place.
__global__ void __launch_bounds__(kInSortWarps * 32)
    k_in_sort(int n, const int* __restrict__ off, int2* __restrict__ list)
{
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kInSortWarps + (threadIdx.x >> 5);
    if (i >= n) return;  // the whole warp leaves together
    const int o = off[i], m = off[i + 1] - o;
    if (m <= 128) {
        int2 v[4];
        int rank[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = 32 * q + lane < m ? list[o + 32 * q + lane] : make_int2(0, 0x7fffffff);
#pragma unroll
        for (int sq = 0; sq < 4; ++sq)
            for (int sl = 0; sl < 32; ++sl) {
                const int w = __shfl_sync(0xffffffffu, v[sq].y, sl);
#pragma unroll
                for (int q = 0; q < 4; ++q) rank[q] += w < v[q].y ? 1 : 0;
            }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (32 * q + lane < m) list[o + rank[q]] = v[q];
        return;
    }
    if (lane != 0) return;
    for (int a = o + 1; a < o + m; ++a) {
        const int2 v = list[a];
        int b = a - 1;
        while (b >= o && list[b].y > v.y) {
            list[b + 1] = list[b];
            --b;
        }
        list[b + 1] = v;
    }
}

// Precision conversions of the adjoint state (the adjoint runs in double).
template <class RO, class RI>
__global__ void __launch_bounds__(256) k_convert(long long m, const RI* __restrict__ in, RO* __restrict__ out)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) out[t] = in ? (RO)in[t] : (RO)0;
}

// ---------------------------------------------------------------- host side

static unsigned pd_groups_blocks(int n) { return (unsigned)(((long long)n * kPdG + kPdBlock - 1) / kPdBlock); }

// Forward state in R (float or double); the reverse state always in double:
// the adjoint differences neighbouring values (a_i - a_j, x_i - x_j) and
// sums over ~80 bonds per particle, 10 iterations per step, which float
// arithmetic does not carry over a long rollout.
template <class R>
struct PdWork {
    int cap_n = 0;
    Q4<R> *xold = nullptr, *xa = nullptr, *xb = nullptr;  // x_old (the first iterate) and two iterates
    R *xr = nullptr, *vr = nullptr, *bulk = nullptr;      // replayed state (3 per particle), stiffness
    Q4<R>* own = nullptr;     // the sum of a particle's outgoing bond terms and of their weights
    Q4<R>* tslot = nullptr;   // per bond slot: the bond's term and weight
    long long tslot_cap = 0;
    Q4<double>* gown = nullptr;   // reverse pass
    Q4<double>* aslot = nullptr;  // reverse pass: per bond slot
    long long aslot_cap = 0;
    Q4<double> *a = nullptr, *g = nullptr, *xoldbar = nullptr;
    double *xbar = nullptr, *vbar = nullptr, *Wa = nullptr, *bulkbar = nullptr;
    int cap_rev = 0;
    // rollout record
    int steps = 0, every = 0, n = 0;
    R gravity[3] = {0, 0, 0};
    float dt = 0.f;
    int iterations = 0;
    R* ckpt = nullptr;  // (x, v) at the start of every segment
    long long ckpt_cap = 0;
    Q4<R>* seg = nullptr;   // iterates of one segment: every * (iterations + 1) * n
    long long seg_cap = 0;
    R* segF = nullptr;  // F of every iterate of a segment: every * iterations * 9n
    long long segF_cap = 0;
    float* segT = nullptr;  // tw of every iterate (negated: identity taken)
    long long segT_cap = 0;
};

template <class R>
static bool grow(R*& p, long long& cap, long long want)
{
    if (want <= cap) return true;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    if (cudaMalloc((void**)&p, sizeof(R) * (size_t)std::max(want, 1LL)) != cudaSuccess) return false;
    cap = want;
    return true;
}

template <class T>
static bool realloc_n(T*& p, size_t count)
{
    if (p) cudaFree(p);
    p = nullptr;
    return cudaMalloc((void**)&p, sizeof(T) * std::max(count, (size_t)1)) == cudaSuccess;
}

template <class R>
static bool work_alloc(PdWork<R>& w, int n)
{
    if (n <= w.cap_n) return true;
    const size_t m = (size_t)n;
    const bool ok = realloc_n(w.xold, m) && realloc_n(w.xa, m) && realloc_n(w.xb, m) && realloc_n(w.own, m);
    w.cap_n = ok ? n : 0;
    return ok;
}

// The reverse pass's and the replay's arrays, allocated with the first
// checkpointed rollout.
template <class R>
static bool reverse_alloc(PdWork<R>& w, int n, long long bonds)
{
    if (n > w.cap_rev) {
        const size_t m = (size_t)n;
        const bool ok = realloc_n(w.xr, 3 * m) && realloc_n(w.vr, 3 * m) && realloc_n(w.bulk, m) &&
                        realloc_n(w.gown, m) && realloc_n(w.a, m) && realloc_n(w.g, m) && realloc_n(w.xoldbar, m) &&
                        realloc_n(w.xbar, 3 * m) && realloc_n(w.vbar, 3 * m) && realloc_n(w.Wa, m) &&
                        realloc_n(w.bulkbar, m);
        w.cap_rev = ok ? n : 0;
        if (!ok) return false;
    }
    return grow(w.aslot, w.aslot_cap, std::max(bonds, 1LL));
}

template <class R>
static void work_free(PdWork<R>* w)
{
    if (!w) return;
    void* ps[] = {w->xold, w->xa,   w->xb,   w->xr,   w->vr,      w->bulk, w->own,  w->tslot, w->gown, w->aslot,
                  w->a,    w->g,    w->xoldbar, w->xbar, w->vbar, w->Wa,   w->bulkbar, w->ckpt, w->seg, w->segF,
                  w->segT};
    for (void* p : ps)
        if (p) cudaFree(p);
    delete w;
}

static PdBonds bonds_of(pk_ctx* c, float horizon, float mu, float lambda)
{
    PdBonds B;
    B.index = c->pd_index;
    B.cap = c->pd_cap;
    B.total = c->pd_total;
    B.n = c->pd_n;
    B.bond = c->pd_bond;
    B.alive = c->pd_alive;
    B.invK = c->pd_invK;
    B.in_off = c->pd_in_off;
    B.in_list = c->pd_in;
    B.in_slot = c->pd_in_slot;
    B.h = horizon;
    B.mu = mu;
    B.lambda = lambda;
    B.inv_h = 1.0f / horizon;
    return B;
}

template <class R>
static PdWork<R>*& work_of(pk_ctx* c);
template <>
PdWork<float>*& work_of<float>(pk_ctx* c)
{
    return reinterpret_cast<PdWork<float>*&>(c->pd_work32);
}
template <>
PdWork<double>*& work_of<double>(pk_ctx* c)
{
    return reinterpret_cast<PdWork<double>*&>(c->pd_work64);
}

void pd_work_release(pk_ctx* c)
{
    work_free(reinterpret_cast<PdWork<float>*>(c->pd_work32));
    work_free(reinterpret_cast<PdWork<double>*>(c->pd_work64));
    c->pd_work32 = c->pd_work64 = nullptr;
}

// The projection's workspace, and the compact bonds brought up to date with
// the rest shape (one launch after the shape changed, none otherwise).
// Returns null when memory runs out; launches counts what was enqueued.
template <class R>
static PdWork<R>* ensure_work(pk_ctx* c, int n, cudaStream_t st, int& launches)
{
    PdWork<R>*& w = work_of<R>(c);
    if (!w) w = new PdWork<R>();
    if (!work_alloc(*w, n)) return nullptr;
    const long long bonds = std::max(c->pd_total, 1LL);
    if (!grow(w->tslot, w->tslot_cap, bonds)) return nullptr;
    if (c->pd_bond_rev != c->pd_shape_rev || bonds > c->pd_bond_cap) {
        if (!grow(c->pd_bond, c->pd_bond_cap, bonds)) return nullptr;
        const PdBonds B = bonds_of(c, c->pd_horizon, 0.f, 0.f);
        if (n > 0) {
            k_pd_bonds<<<pd_groups_blocks(n), kPdBlock, 0, st>>>(B, c->pd_raw, c->pd_rest_idx, c->pd_rest_pos);
            ++launches;
        }
        c->pd_bond_rev = c->pd_shape_rev;
    }
    return w;
}

// The slots of the incoming lists as their own array: the gathers read 4
// bytes per incoming bond instead of the 8-byte (source, slot) pair.
__global__ void __launch_bounds__(256) k_in_slots(const int* __restrict__ total, const int2* __restrict__ list,
                                                  int* __restrict__ slots)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < *total) slots[t] = list[t].y;
}

// Orders the bonds of the frozen rest shape and builds its incoming-bond lists
// (once per pd_init or reconstruction).
int pd_build_incoming(pk_ctx* c, cudaStream_t st)
{
    const int n = c->pd_n;
    const unsigned nb = (unsigned)((n + 255) / 256);
    cudaMemsetAsync(c->pd_in_cnt, 0, sizeof(int) * (size_t)(n + 1), st);
    k_in_count<<<nb, 256, 0, st>>>(n, c->pd_index, c->pd_cap, c->pd_total, c->pd_rest_idx, c->pd_in_cnt);
    exclusive_scan(c->pd_in_cnt, n, c->pd_in_off, c->scan_part, st);
    cudaMemsetAsync(c->pd_in_cnt, 0, sizeof(int) * (size_t)(n + 1), st);
    const unsigned nw = (unsigned)((n + kInSortWarps - 1) / kInSortWarps);
    k_pd_order<<<nw, kInSortWarps * 32, 0, st>>>(n, c->pd_index, c->pd_cap, c->pd_total, c->pd_rest_idx, c->pd_raw);
    k_in_fill<<<nb, 256, 0, st>>>(n, c->pd_index, c->pd_cap, c->pd_total, c->pd_rest_idx, c->pd_raw, c->pd_in_off,
                                  c->pd_in_cnt, c->pd_in);
    k_in_sort<<<nw, kInSortWarps * 32, 0, st>>>(n, c->pd_in_off, c->pd_in);
    const long long nin = std::max(c->pd_total, 1LL);
    k_in_slots<<<(unsigned)((nin + 255) / 256), 256, 0, st>>>(c->pd_in_off + n, c->pd_in, c->pd_in_slot);
    return 6 + scan_launches();
}

// One projection solve from y_0 in w.xold (x_old and the first iterate): the
// last iteration writes x (3 per particle) and, with v, updates it.  With a
// stretch limit the first iteration breaks bonds (also when none follows).
template <class R>
static int project(PdWork<R>& w, const PdBonds& B, R* x, R* v, const R* bulk, int iterations, R dt, float stretch,
                   cudaStream_t st)
{
    const unsigned nb = pd_groups_blocks(B.n);
    const Q4<R>* cur = w.xold;
    int l = 0;
    for (int it = 0; it < iterations || (it == 0 && stretch > 0.f); ++it) {
        if (it == 0 && stretch > 0.f)
            k_pd_FP<R, true><<<nb, kPdBlock, 0, st>>>(B, cur, bulk, nullptr, nullptr, w.own, w.tslot, stretch);
        else
            k_pd_FP<R, false><<<nb, kPdBlock, 0, st>>>(B, cur, bulk, nullptr, nullptr, w.own, w.tslot, 0.f);
        ++l;
        if (it >= iterations) break;
        Q4<R>* nxt = it % 2 == 0 ? w.xa : w.xb;
        if (it == iterations - 1)
            k_pd_gather<R, true><<<nb, kPdBlock, 0, st>>>(B, cur, w.xold, w.own, w.tslot, nullptr, x, v, dt);
        else
            k_pd_gather<R, false><<<nb, kPdBlock, 0, st>>>(B, cur, w.xold, w.own, w.tslot, nxt, nullptr, nullptr,
                                                           dt);
        ++l;
        cur = nxt;
    }
    return l;
}

// pk_pd_solve's projection on the gather form (float, alive mask honoured).
int pd_project_solve(pk_ctx* c, float* x, float* v, int n, float horizon, float mu, float lambda, int iterations,
                     float dt, float stretch, cudaStream_t st)
{
    int l = 0;
    PdWork<float>* w = ensure_work<float>(c, n, st, l);
    if (!w) return -1;
    const PdBonds B = bonds_of(c, horizon, mu, lambda);
    k_pd_pack<float><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x, w->xold);
    return l + 1 + project<float>(*w, B, x, v, c->pd_bulk, iterations, dt, stretch, st);
}

// The caller's positions packed to 16 bytes (in scratch the next projection
// overwrites), with the compact bonds brought up to date where they are asked
// for; null when memory runs out.
const float4* pd_pack(pk_ctx* c, const float* x, bool bonds, int& launches, cudaStream_t st)
{
    const int n = c->pd_n;
    PdWork<float>*& w = work_of<float>(c);
    if (!w) w = new PdWork<float>();
    if (bonds ? !ensure_work<float>(c, n, st, launches) : !work_alloc(*w, n)) return nullptr;
    k_pd_pack<float><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x, w->xa);
    ++launches;
    return reinterpret_cast<const float4*>(w->xa);
}

// The projection one step at a time (pk_pd_begin / pk_pd_enforce /
// pk_pd_update_velocity): x_old is kept in the float workspace between the
// calls (the bond weights come with every iteration's bond terms).
int pd_begin(pk_ctx* c, const float* x, int n, float /*horizon*/, float /*mu*/, float /*lambda*/, cudaStream_t st)
{
    int l = 0;
    PdWork<float>* w = ensure_work<float>(c, n, st, l);
    if (!w) return -1;
    if (n <= 0) return 0;
    k_pd_pack<float><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x, w->xold);
    return l + 1;
}

int pd_enforce(pk_ctx* c, float* x, int n, float horizon, float mu, float lambda, cudaStream_t st)
{
    PdWork<float>* w = work_of<float>(c);
    if (!w || w->cap_n < n) return -1;
    if (n <= 0) return 0;
    int l = 0;
    if (!ensure_work<float>(c, n, st, l)) return -1;  // the rest shape may have changed since pk_pd_begin
    const PdBonds B = bonds_of(c, horizon, mu, lambda);
    const unsigned nb128 = pd_groups_blocks(n);
    k_pd_pack<float><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x, w->xa);
    k_pd_FP<float, false><<<nb128, kPdBlock, 0, st>>>(B, w->xa, c->pd_bulk, nullptr, nullptr, w->own, w->tslot, 0.f);
    k_pd_gather<float, true><<<nb128, kPdBlock, 0, st>>>(B, w->xa, w->xold, w->own, w->tslot, nullptr, x, nullptr,
                                                         1.f);
    return l + 3;
}

int pd_update_velocity(pk_ctx* c, const float* x, float* v, int n, float dt, cudaStream_t st)
{
    PdWork<float>* w = work_of<float>(c);
    if (!w || w->cap_n < n) return -1;
    if (n <= 0) return 0;
    k_pd_vel<float><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, v, x, nullptr, w->xold, dt);
    return 1;
}

template <class R>
static int rollout(pk_ctx* c, R* x, R* v, const R* bulk_in, int n, const R g[3], const pk_pd_params* p, int steps,
                   int every, cudaStream_t st)
{
    if (n <= 0) return 0;
    int l = 0;
    PdWork<R>* w = ensure_work<R>(c, n, st, l);
    if (!w || !reverse_alloc(*w, n, every > 0 ? c->pd_total : 0)) return -1;
    const PdBonds B = bonds_of(c, p->horizon, p->mu, p->lambda);
    const size_t bytes = sizeof(R) * 3 * (size_t)n;
    cudaMemcpyAsync(w->bulk, bulk_in, sizeof(R) * (size_t)n, cudaMemcpyDeviceToDevice, st);
    const int nseg = every > 0 ? (steps + every - 1) / every : 0;
    if (every > 0) {
        if (!grow(w->ckpt, w->ckpt_cap, 6LL * n * std::max(nseg, 1))) return -1;
        if (!grow(w->seg, w->seg_cap, 1LL * n * (p->iterations + 1) * every)) return -1;
        if (!grow(w->segF, w->segF_cap, 9LL * n * std::max(p->iterations, 1) * every)) return -1;
        if (!grow(w->segT, w->segT_cap, 1LL * n * std::max(p->iterations, 1) * every)) return -1;
    }
    w->steps = steps;
    w->every = every;
    w->n = n;
    w->dt = p->dt;
    w->iterations = p->iterations;
    for (int a = 0; a < 3; ++a) w->gravity[a] = g[a];
    const unsigned nb = (unsigned)((n + 255) / 256);
    for (int s = 0; s < steps; ++s) {
        if (every > 0 && s % every == 0) {
            R* ck = w->ckpt + 6LL * n * (s / every);
            cudaMemcpyAsync(ck, x, bytes, cudaMemcpyDeviceToDevice, st);
            cudaMemcpyAsync(ck + 3LL * n, v, bytes, cudaMemcpyDeviceToDevice, st);
        }
        k_pd_integrate<R><<<nb, 256, 0, st>>>(n, x, nullptr, v, g[0], g[1], g[2], (R)p->dt, w->xold);
        ++l;
        if (p->iterations > 0) {
            l += project<R>(*w, B, x, v, w->bulk, p->iterations, (R)p->dt, 0.f, st);
        } else {
            k_pd_unpack<R><<<nb, 256, 0, st>>>(n, w->xold, x);  // x' itself
            ++l;
        }
    }
    return l;
}

template <class R>
static int rollout_backward(pk_ctx* c, const R* xbar, const R* vbar, R* gx, R* gv, double* gbulk, cudaStream_t st)
{
    if (c->pd_n == 0) return 0;
    PdWork<R>* w = work_of<R>(c);
    if (!w || w->every <= 0 || w->n != c->pd_n) return -1;
    int l = 0;
    if (!ensure_work<R>(c, c->pd_n, st, l) || !reverse_alloc(*w, c->pd_n, c->pd_total)) return -2;
    const int n = w->n, iters = w->iterations;
    const PdBonds B = bonds_of(c, c->pd_horizon_last, c->pd_mu_last, c->pd_lambda_last);
    const size_t bytes = sizeof(R) * 3 * (size_t)n;
    const long long m3 = 3LL * n;
    const unsigned nb = (unsigned)((n + 255) / 256), nb128 = pd_groups_blocks(n),
                   nb3 = (unsigned)((m3 + 255) / 256);
    const R dt = (R)w->dt;
    k_convert<double, R><<<nb3, 256, 0, st>>>(m3, xbar, w->xbar);
    k_convert<double, R><<<nb3, 256, 0, st>>>(m3, vbar, w->vbar);
    cudaMemsetAsync(w->bulkbar, 0, sizeof(double) * (size_t)n, st);
    k_pd_W<double, R><<<nb128, kPdBlock, 0, st>>>(B, w->bulk, w->Wa);
    l += 3;
    const int nseg = (w->steps + w->every - 1) / w->every;
    for (int sg = nseg - 1; sg >= 0; --sg) {
        const int s0 = sg * w->every, s1 = std::min(w->steps, s0 + w->every);
        const R* ck = w->ckpt + 6LL * n * sg;
        R* vr = w->vr;
        cudaMemcpyAsync(w->xr, ck, bytes, cudaMemcpyDeviceToDevice, st);
        cudaMemcpyAsync(vr, ck + 3LL * n, bytes, cudaMemcpyDeviceToDevice, st);
        // replay the segment, keeping every iterate x_0 .. x_iters (x_0 = x' = x_old)
        const Q4<R>* prev = nullptr;  // the previous step's last iterate
        for (int s = s0; s < s1; ++s) {
            Q4<R>* it = w->seg + 1LL * n * (iters + 1) * (s - s0);
            k_pd_integrate<R><<<nb, 256, 0, st>>>(n, w->xr, prev, vr, w->gravity[0], w->gravity[1], w->gravity[2],
                                                  dt, it);
            for (int k = 0; k < iters; ++k) {
                const long long slot = (long long)(s - s0) * iters + k;
                k_pd_FP<R, false><<<nb128, kPdBlock, 0, st>>>(B, it + 1LL * n * k, w->bulk, w->segF + 9LL * n * slot,
                                                              w->segT + 1LL * n * slot, w->own, w->tslot, 0.f);
                k_pd_gather<R, false><<<nb128, kPdBlock, 0, st>>>(B, it + 1LL * n * k, it, w->own, w->tslot,
                                                                  it + 1LL * n * (k + 1), nullptr, nullptr, dt);
            }
            prev = it + 1LL * n * iters;
            k_pd_vel<R><<<nb, 256, 0, st>>>(n, vr, nullptr, prev, it, dt);
            l += 2 + 2 * iters;
        }
        for (int s = s1 - 1; s >= s0; --s) {
            const Q4<R>* it = w->seg + 1LL * n * (iters + 1) * (s - s0);
            k_pd_adj_head<double><<<nb, 256, 0, st>>>(n, w->xbar, w->vbar, (double)dt, w->Wa, iters == 0, w->g, w->a,
                                                      w->xoldbar);
            for (int k = iters - 1; k >= 0; --k) {
                const long long slot = (long long)(s - s0) * iters + k;
                k_pd_adjBC<double, R><<<nb128, kPdBlock, 0, st>>>(
                    B, it + 1LL * n * k, it + 1LL * n * (k + 1), w->bulk, w->segF + 9LL * n * slot,
                    w->segT + 1LL * n * slot, w->a, w->bulkbar, w->gown, w->aslot);
                k_pd_adjC_gather<double><<<nb128, kPdBlock, 0, st>>>(B, w->gown, w->aslot, w->Wa, k == 0, w->g, w->a,
                                                                     w->xoldbar);
            }
            k_pd_adj_tail<double><<<nb, 256, 0, st>>>(n, w->g, w->xoldbar, (double)dt, w->xbar, w->vbar);
            l += 2 + 2 * iters;
        }
    }
    k_convert<R, double><<<nb3, 256, 0, st>>>(m3, w->xbar, gx);
    k_convert<R, double><<<nb3, 256, 0, st>>>(m3, w->vbar, gv);
    cudaMemcpyAsync(gbulk, w->bulkbar, sizeof(double) * (size_t)n, cudaMemcpyDeviceToDevice, st);
    return l + 2;
}

int pd_rollout_f32(pk_ctx* c, float* x, float* v, int n, const float g[3], const pk_pd_params* p, int steps,
                   int every, cudaStream_t st)
{
    return rollout<float>(c, x, v, c->pd_bulk, n, g, p, steps, every, st);
}
int pd_rollout_f64(pk_ctx* c, double* x, double* v, const double* bulk, int n, const double g[3],
                   const pk_pd_params* p, int steps, int every, cudaStream_t st)
{
    return rollout<double>(c, x, v, bulk, n, g, p, steps, every, st);
}
int pd_backward_f32(pk_ctx* c, const float* xbar, const float* vbar, float* gx, float* gv, double* gbulk,
                    cudaStream_t st)
{
    return rollout_backward<float>(c, xbar, vbar, gx, gv, gbulk, st);
}
int pd_backward_f64(pk_ctx* c, const double* xbar, const double* vbar, double* gx, double* gv, double* gbulk,
                    cudaStream_t st)
{
    return rollout_backward<double>(c, xbar, vbar, gx, gv, gbulk, st);
}

}  // namespace pk
