// pk_pbd.cu -- DensityPBD (with SummationDensity) and ParticleIntegrator.
//
// Fast path: the rows built by pk_nbr.cu in sorted space.  One Jacobi
// iteration of the reference (DensityPBD::takeOneIteration,
// DensityPBD.cu:305-365: density, lambdas, displacement with atomics,
// position update) is two gather passes here:
//   pass A: rho_i and lambda_i over N(i) (K_ComputeDensity
//           SummationDensity.cu:13-36 + K_ComputeLambdas DensityPBD.cu:46-90),
//   pass B: x_i' = x_i + sum over the row of m_ij * dp_ij, m_ij = [j in N(i)]
//           + [i in N(j)] -- the same sum the reference's scatter
//           (+dp_ij to i, -dp_ij to j, DensityPBD.cu:134-179) accumulates,
//           since dp_ji = -dp_ij bit for bit.
// One thread per particle walks its solver row; rows are interleaved by
// blocks of 32 particles (row_slot), so a warp's row reads are one line per
// entry and its gathers at one entry index touch a few neighbour cells.
// Jacobi: pass A reads x, writes (x, lambda) to xl; pass B reads xl only and
// writes x'.
#include <algorithm>

#include "pk_kernels.cuh"

namespace pk {

// Constants of the two passes (Spiky kernel, Kernel.h SpikyKernel); all but
// inv_h multiply a finished sum, so no pair spends an instruction on them.
struct PassK {
    float inv_h, cwm, cg, c10g;
};
__host__ __device__ inline PassK pass_k(const Spiky& k, float mass)
{
    return PassK{k.inv_h, mass * k.cw, k.cg, 10.0f * k.cg};
}
constexpr float kEps2 = kEpsilon * kEpsilon;  // r > EPSILON  <=>  r^2 > EPSILON^2

// 1/sqrt of a normal number (the callers clamp from below): one instruction,
// where rsqrtf also handles denormals.
__device__ __forceinline__ float rsq(float v)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// Pair geometry shared by both passes: r from one reciprocal square root
// (r = d2 / sqrt(d2); d2 = 0 gives r = 0), 1/r, and d = 1 - r/h clamped at 0,
// so w = cw d^3 and |grad| = cg d^2 vanish beyond h as in SpikyKernel.
__device__ __forceinline__ void pair_geom(float dx, float dy, float dz, float inv_h, float& d2, float& ir,
                                          float& dd)
{
    d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    ir = rsq(fmaxf(d2, 1e-30f));
    dd = fmaxf(fmaf(-(d2 * ir), inv_h, 1.0f), 0.0f);
}

// One quad of row entries (16 bytes, streaming: the rows are read once per
// pass and outgrow L2).
__device__ __forceinline__ int4 row_quad(const int4* p) { return __ldcs(p); }

// Entries of a solver row past the row capacity: the particle's spill
// segment (rows that long exist only where more particles than the capacity
// sit inside one radius).
struct Tail {
    const int* rpool;
    const int* ovf;
    __device__ __forceinline__ int entry(int s, int k) const { return __ldg(rpool + __ldg(ovf + s) + k); }
};

// Entry v's position: the flag bits leave with the shift, and the 32-bit byte
// offset needs no 64-bit arithmetic (rows of 2^28 particles would not fit any
// memory).
__device__ __forceinline__ float4 row_pos(const float4* __restrict__ x, int v)
{
    return __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const char*>(x) + ((unsigned)v << 4)));
}

// Both passes, one thread per particle walking its interleaved row, two row
// entries per packed FP32x2 instruction (sm_100 FFMA2/FADD2/FMUL2): the full
// quads as two entry pairs, then the last partial quad one entry at a time.
// The sums run as two interleaved partial sums (even and odd entries of each
// pair).  d is taken as x_j - x_i (the exact negation of x_i - x_j), so the
// accumulated gradients and displacements carry the opposite sign and are
// negated at the end.
struct Geom2 {
    float2 dx, dy, dz, d2, ir, dd;
};

__device__ __forceinline__ void pair_geom2(const float4& a, const float4& b, const float4& xi, float inv_h, Geom2& g)
{
    g.dx = make_float2(a.x - xi.x, b.x - xi.x);
    g.dy = make_float2(a.y - xi.y, b.y - xi.y);
    g.dz = make_float2(a.z - xi.z, b.z - xi.z);
    g.d2 = __ffma2_rn(g.dz, g.dz, __ffma2_rn(g.dy, g.dy, __fmul2_rn(g.dx, g.dx)));
    g.ir = make_float2(rsq(fmaxf(g.d2.x, 1e-30f)), rsq(fmaxf(g.d2.y, 1e-30f)));
    const float2 t = __ffma2_rn(__fmul2_rn(g.d2, g.ir), make_float2(-inv_h, -inv_h), make_float2(1.0f, 1.0f));
    g.dd = make_float2(fmaxf(t.x, 0.0f), fmaxf(t.y, 0.0f));
}

// Pass A: rho_i and lambda_i over N(i).  sum |grad_j|^2 is taken as sum g_j^2
// (|x_ij / r| = 1).
struct DensPass {
    using Acc = struct {
        float2 rho, sg, gx, gy, gz;
    };
    static __device__ __forceinline__ int entries(const int2& c) { return c.x; }
    static __device__ __forceinline__ void pair(const float4& a, const float4& b, int, int, const float4& xi,
                                                const PassK& k_, Acc& s)
    {
        Geom2 g;
        pair_geom2(a, b, xi, k_.inv_h, g);
        const float2 dd2 = __fmul2_rn(g.dd, g.dd);
        s.rho = __ffma2_rn(dd2, g.dd, s.rho);
        const float2 w = make_float2(g.d2.x > kEps2 ? dd2.x : 0.0f, g.d2.y > kEps2 ? dd2.y : 0.0f);
        const float2 gi = __fmul2_rn(w, g.ir);
        s.gx = __ffma2_rn(gi, g.dx, s.gx);
        s.gy = __ffma2_rn(gi, g.dy, s.gy);
        s.gz = __ffma2_rn(gi, g.dz, s.gz);
        s.sg = __ffma2_rn(w, w, s.sg);
    }
    // One entry into the .x partial sums (the tail of a row).
    static __device__ __forceinline__ void one(const float4& a, int, const float4& xi, const PassK& k_, Acc& s)
    {
        const float dx = a.x - xi.x, dy = a.y - xi.y, dz = a.z - xi.z;
        float d2, ir, dd;
        pair_geom(dx, dy, dz, k_.inv_h, d2, ir, dd);
        const float dd2 = dd * dd;
        s.rho.x = fmaf(dd2, dd, s.rho.x);
        const float w = d2 > kEps2 ? dd2 : 0.0f;
        const float gi = w * ir;
        s.gx.x = fmaf(gi, dx, s.gx.x);
        s.gy.x = fmaf(gi, dy, s.gy.x);
        s.gz.x = fmaf(gi, dz, s.gz.x);
        s.sg.x = fmaf(w, w, s.sg.x);
    }
    // (x_i, lambda_i), so pass B gathers a neighbour's position and lambda in
    // one 16-byte load.
    static __device__ __forceinline__ float4 finish(const float4& xi, const PassK& k_, const Acc& a, float* rho_out,
                                                    int s)
    {
        const float rho = k_.cwm * (a.rho.x + a.rho.y), sg = k_.cg * k_.cg * (a.sg.x + a.sg.y);
        const float gx = k_.cg * (a.gx.x + a.gx.y), gy = k_.cg * (a.gy.x + a.gy.y), gz = k_.cg * (a.gz.x + a.gz.y);
        // (explicit, so that every instance of the pass rounds alike)
        float l = fmaf(gz, gz, fmaf(gy, gy, fmaf(gx, gx, sg)));
        l = -(rho - 1000.0f) / (l + 0.1f);  // rest density hard-coded (DensityPBD.cu:87)
        if (rho_out != nullptr) rho_out[s] = rho;
        return make_float4(xi.x, xi.y, xi.z, l > 0.0f ? 0.0f : l);
    }
};

// Pass B: x_i' = x_i + sum over U(i) of m_ij * 10 (x_i - x_j)(lambda_i +
// lambda_j) grad(r) / r (DensityPBD.cu:158), m_ij the number of flag bits set
// (1 or 2: 2 exactly when v >= 0xc0000000).
struct DispPass {
    using Acc = struct {
        float2 ax, ay, az;
    };
    static __device__ __forceinline__ int entries(const int2& c) { return c.y; }
    static __device__ __forceinline__ float mult(int v) { return (unsigned)v >= 0xc0000000u ? 2.0f : 1.0f; }
    static __device__ __forceinline__ void pair(const float4& a, const float4& b, int va, int vb, const float4& xi,
                                                const PassK& k_, Acc& s)
    {
        Geom2 g;
        pair_geom2(a, b, xi, k_.inv_h, g);
        const float2 lw = make_float2(xi.w + a.w, xi.w + b.w);
        const float2 c = __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(mult(va), mult(vb)), lw),
                                               __fmul2_rn(g.dd, g.dd)), g.ir);
        const float2 cc = make_float2(g.d2.x > kEps2 ? c.x : 0.0f, g.d2.y > kEps2 ? c.y : 0.0f);
        s.ax = __ffma2_rn(cc, g.dx, s.ax);
        s.ay = __ffma2_rn(cc, g.dy, s.ay);
        s.az = __ffma2_rn(cc, g.dz, s.az);
    }
    static __device__ __forceinline__ void one(const float4& a, int v, const float4& xi, const PassK& k_, Acc& s)
    {
        const float dx = a.x - xi.x, dy = a.y - xi.y, dz = a.z - xi.z;
        float d2, ir, dd;
        pair_geom(dx, dy, dz, k_.inv_h, d2, ir, dd);
        const float c = d2 > kEps2 ? mult(v) * (xi.w + a.w) * (dd * dd) * ir : 0.0f;
        s.ax.x = fmaf(c, dx, s.ax.x);
        s.ay.x = fmaf(c, dy, s.ay.x);
        s.az.x = fmaf(c, dz, s.az.x);
    }
    static __device__ __forceinline__ float4 finish(const float4& xi, const PassK& k_, const Acc& a, float*, int)
    {
        // the sums hold -(displacement): d was x_j - x_i
        return make_float4(fmaf(-k_.c10g, a.ax.x + a.ax.y, xi.x), fmaf(-k_.c10g, a.ay.x + a.ay.y, xi.y),
                           fmaf(-k_.c10g, a.az.x + a.az.y, xi.z), 0.f);
    }
};

// One particle of a pass.  NQ row quads are loaded together and their
// neighbours gathered together (4 NQ gathers in flight), with the next NQ quads
// already on their way; the additions run in row order whatever NQ is.
template <class Pass, int NQ>
__device__ __forceinline__ void pass_particle(int s, const float4* __restrict__ xin, const int* __restrict__ rows,
                                              const int2* __restrict__ rcnt, int row_cap, const PassK& k_,
                                              float4* __restrict__ xout, float* __restrict__ rho_out, const Tail& tl)
{
    const float4 xi = xin[s];
    const int m_all = Pass::entries(rcnt[s]), m = min(m_all, row_cap);
    const int4* rq = reinterpret_cast<const int4*>(rows + row_slot(s, 0, row_cap));
    typename Pass::Acc a{};
    const int nfull = m >> 2, nq = (m + 3) >> 2;
    int4 last;  // the row's partial quad
    if (NQ == 1) {
        // two quads ahead of the one worked on
        int4 r0 = nq > 0 ? row_quad(rq) : make_int4(0, 0, 0, 0);
        int4 r1 = nq > 1 ? row_quad(rq + 32) : make_int4(0, 0, 0, 0);
        for (int q = 0; q < nfull; ++q) {
            const int4 cur = r0;
            r0 = r1;
            if (q + 2 < nq) r1 = row_quad(rq + 32LL * (q + 2));
            const float4 x0 = row_pos(xin, cur.x), x1 = row_pos(xin, cur.y);
            const float4 x2 = row_pos(xin, cur.z), x3 = row_pos(xin, cur.w);
            Pass::pair(x0, x1, cur.x, cur.y, xi, k_, a);
            Pass::pair(x2, x3, cur.z, cur.w, xi, k_, a);
        }
        last = r0;
    } else {
        last = nq > nfull ? row_quad(rq + 32LL * nfull) : make_int4(0, 0, 0, 0);
        int4 nxt[NQ];
#pragma unroll
        for (int k = 0; k < NQ; ++k) nxt[k] = k < nfull ? row_quad(rq + 32LL * k) : make_int4(0, 0, 0, 0);
        for (int q = 0; q < nfull; q += NQ) {
            int4 cur[NQ];
            float4 x[4 * NQ];
#pragma unroll
            for (int k = 0; k < NQ; ++k) cur[k] = nxt[k];
#pragma unroll
            for (int k = 0; k < NQ; ++k) {  // entries past the row's end read particle 0, unused
                x[4 * k] = row_pos(xin, cur[k].x);
                x[4 * k + 1] = row_pos(xin, cur[k].y);
                x[4 * k + 2] = row_pos(xin, cur[k].z);
                x[4 * k + 3] = row_pos(xin, cur[k].w);
            }
#pragma unroll
            for (int k = 0; k < NQ; ++k)
                nxt[k] = q + NQ + k < nfull ? row_quad(rq + 32LL * (q + NQ + k)) : make_int4(0, 0, 0, 0);
#pragma unroll
            for (int k = 0; k < NQ; ++k) {
                if (q + k < nfull) {
                    Pass::pair(x[4 * k], x[4 * k + 1], cur[k].x, cur[k].y, xi, k_, a);
                    Pass::pair(x[4 * k + 2], x[4 * k + 3], cur[k].z, cur[k].w, xi, k_, a);
                }
            }
        }
    }
    const int rest = m - 4 * nfull;
    if (rest > 0) {
        const int ent[3] = {last.x, last.y, last.z};
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (k < rest) Pass::one(row_pos(xin, ent[k]), ent[k], xi, k_, a);
    }
    for (int e = m; e < m_all; ++e) {
        const int v = tl.entry(s, e - m);
        Pass::one(row_pos(xin, v), v, xi, k_, a);
    }
    xout[s] = Pass::finish(xi, k_, a, rho_out, s);
}

// Tiles of the persistent passes: each scene's sorted range (and the range of
// the particles outside every grid) cut into tiles of one block's threads, so
// no tile holds two scenes.  Null tiles: one scene, tile t = [t B, (t+1) B).
struct SceneTiles {
    const int2* tile;
    const int* count;  // device: number of tiles
};

// Row quads per step of a pass: 1 (the most resident warps) where the
// particles fill the chip, 4 for the small scenes (kDeepMax).
template <class Pass, int BLOCK, int NQ>
__global__ void __launch_bounds__(BLOCK)
    k_pass(const float4* __restrict__ xin, const int* __restrict__ rows, const int2* __restrict__ rcnt, int row_cap,
           int n, PassK k_, float4* __restrict__ xout, float* __restrict__ rho_out, Tail tl)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) pass_particle<Pass, NQ>(s, xin, rows, rcnt, row_cap, k_, xout, rho_out, tl);
}

// Persistent form: a grid of resident blocks walks the scene tiles.
// (32 resident warps per SM asked of the register allocator: the tile loop
// would otherwise take the kernel past 64 registers and a quarter of them)
template <class Pass, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK)
    k_pass_t(const float4* __restrict__ xin, const int* __restrict__ rows, const int2* __restrict__ rcnt, int row_cap,
             int n, PassK k_, float4* __restrict__ xout, float* __restrict__ rho_out, Tail tl, SceneTiles T)
{
    const int nt = T.tile ? *T.count : (n + BLOCK - 1) / BLOCK;
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const int2 r = T.tile ? T.tile[t] : make_int2(t * BLOCK, min((t + 1) * BLOCK, n));
        const int s = r.x + (int)threadIdx.x;
        if (s < r.y) pass_particle<Pass, 1>(s, xin, rows, rcnt, row_cap, k_, xout, rho_out, tl);
    }
}

// Scene tiles from the starts of the 64-cell blocks (K of them per scene):
// scene q holds the sorted range [start[q K], start[(q+1) K]), the particles
// outside every grid the block past the last.  One thread per scene.
__device__ __forceinline__ int2 scene_range(const int* start, long long scene_blocks, int nscenes, int q)
{
    const long long b = (long long)q * scene_blocks;
    return make_int2(start[b], start[q < nscenes ? b + scene_blocks : b + 1]);
}
__global__ void __launch_bounds__(256) k_tile_count(const int* __restrict__ start, long long scene_blocks,
                                                    int nscenes, int tile, int* __restrict__ cnt)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q > nscenes) return;
    const int2 r = scene_range(start, scene_blocks, nscenes, q);
    cnt[q] = (r.y - r.x + tile - 1) / tile;
}

__global__ void __launch_bounds__(256) k_tile_fill(const int* __restrict__ start, long long scene_blocks,
                                                   int nscenes, int tile, const int* __restrict__ off,
                                                   int2* __restrict__ tiles)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q > nscenes) return;
    const int2 r = scene_range(start, scene_blocks, nscenes, q);
    int o = off[q];
    for (int a = r.x; a < r.y; a += tile) tiles[o++] = make_int2(a, min(a + tile, r.y));
}

// Sorted -> caller order: x, v += (x - x_old)/dt (DP_UpdateVelocity,
// DensityPBD.cu:367-378), outDensity.  One thread per caller particle i
// (s = inv[i]): the 16-byte sorted values are gathered, the caller's AoS
// arrays written contiguously.
__global__ void __launch_bounds__(256)
    k_finish(const float4* __restrict__ xf, const float4* __restrict__ x0, const float4* __restrict__ vs,
             const float* __restrict__ rho_s, const int* __restrict__ inv, int n, float dt,
             float* __restrict__ x, float* __restrict__ v, float* __restrict__ rho_out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int s = inv[i];
    float4 p = xf[s], q = x0[s], u = vs[s];
    x[3 * i] = p.x;
    x[3 * i + 1] = p.y;
    x[3 * i + 2] = p.z;
    v[3 * i] = u.x + (p.x - q.x) / dt;
    v[3 * i + 1] = u.y + (p.y - q.y) / dt;
    v[3 * i + 2] = u.z + (p.z - q.z) / dt;
    if (rho_out != nullptr) rho_out[i] = rho_s[s];
}

// ---- ImplicitViscosity (ImplicitViscosity.cu:8-128)

// VB_VisWeight: 45/(13 pi h^3) (1 - r/h) for r <= h.
struct ViscK {
    float inv_h, cw, b;  // b = dt * viscosity / h
};

// DP_UpdateVelocity in sorted space: v = v_integrated + (x - x_old)/dt, kept
// as the viscosity's v_old and first iterate.
__global__ void __launch_bounds__(256)
    k_vel_sorted(const float4* __restrict__ xf, const float4* __restrict__ x0, float4* __restrict__ vs,
                 float4* __restrict__ vcur, int n, float dt)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float4 p = xf[s], q = x0[s], u = vs[s];
    const float4 v = make_float4(u.x + (p.x - q.x) / dt, u.y + (p.y - q.y) / dt, u.z + (p.z - q.z) / dt, 0.f);
    vs[s] = v;
    vcur[s] = v;
}

// One K_ApplyViscosity sweep over N(i) (the rows' first |N(i)| entries):
// v_i = v_old,i/(1+b) + (sum w v_j / sum w) b/(1+b); b = 0 and sum w = 1 when
// sum w < EPSILON.  The weights depend on the positions alone, which no sweep
// moves: the first sweep (kFirst) forms them, keeps them in wrow, laid out as
// the rows, and their sum in vold's fourth value; the others read them, 4
// bytes per entry in place of a 16-byte gather and the pair's geometry.  NQ as
// in the Jacobi passes.  Bound by L1 as they are: 152k particles, 22 us a sweep
// after a first of 35, where forming the weights in each took 36.
__device__ __forceinline__ float4 visc_mix(const float4& vo, float sx, float sy, float sz, float b, float t)
{
    // every rounding explicit: the sweeps over rows and over lists agree
    const float d = 1.0f + b;
    return make_float4(__fadd_rn(__fdiv_rn(vo.x, d), __fdiv_rn(__fmul_rn(__fdiv_rn(sx, t), b), d)),
                       __fadd_rn(__fdiv_rn(vo.y, d), __fdiv_rn(__fmul_rn(__fdiv_rn(sy, t), b), d)),
                       __fadd_rn(__fdiv_rn(vo.z, d), __fdiv_rn(__fmul_rn(__fdiv_rn(sz, t), b), d)), 0.f);
}
template <int BLOCK, int NQ, bool kFirst>
__global__ void __launch_bounds__(BLOCK)
    k_pass_visc(const float4* __restrict__ xs, const float4* __restrict__ vin, float4* __restrict__ vold,
                const int* __restrict__ rows, float* __restrict__ wrow, const int2* __restrict__ rcnt, int row_cap,
                int n, ViscK k_, float4* __restrict__ vout, Tail tl)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float4 xi = xs[s];
    const int na_all = rcnt[s].x, na = min(na_all, row_cap);
    const int4* rq = reinterpret_cast<const int4*>(rows + row_slot(s, 0, row_cap));
    float4* wq = reinterpret_cast<float4*>(wrow + row_slot(s, 0, row_cap));
    float4 vo = vold[s];
    // one partial sum per place in a quad, as pk_viscosity sums a caller's
    // list over 4 lanes: both give the same velocities for the same list
    float tw4[4] = {0.f, 0.f, 0.f, 0.f}, az[4] = {0.f, 0.f, 0.f, 0.f};
    float2 axy[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    auto weight = [&](const float4& xj) {
        float d2, ir, dd;
        pair_geom(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, k_.inv_h, d2, ir, dd);
        return d2 > kEps2 ? k_.cw * dd : 0.0f;
    };
    auto add = [&](int k, float w, const float4& vj) {
        if (kFirst) tw4[k] += w;
        axy[k] = __ffma2_rn(make_float2(w, w), make_float2(vj.x, vj.y), axy[k]);
        az[k] = fmaf(w, vj.z, az[k]);
    };
    const int nq = (na + 3) >> 2, nfull = na >> 2;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    int4 nxt[NQ];
    float4 wn[NQ];
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        nxt[k] = k < nq ? row_quad(rq + 32LL * k) : make_int4(0, 0, 0, 0);
        wn[k] = !kFirst && k < nq ? __ldcs(wq + 32LL * k) : zero;
    }
    int q = 0;
    for (; q + NQ <= nfull; q += NQ) {
        int4 cur[NQ];
        float4 w[NQ], v[4 * NQ], x[kFirst ? 4 * NQ : 1];
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            cur[k] = nxt[k];
            w[k] = wn[k];
            v[4 * k] = row_pos(vin, cur[k].x);
            v[4 * k + 1] = row_pos(vin, cur[k].y);
            v[4 * k + 2] = row_pos(vin, cur[k].z);
            v[4 * k + 3] = row_pos(vin, cur[k].w);
            if (kFirst) {
                x[4 * k] = row_pos(xs, cur[k].x);
                x[4 * k + 1] = row_pos(xs, cur[k].y);
                x[4 * k + 2] = row_pos(xs, cur[k].z);
                x[4 * k + 3] = row_pos(xs, cur[k].w);
            }
        }
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            const int qn = q + NQ + k;
            nxt[k] = qn < nq ? row_quad(rq + 32LL * qn) : make_int4(0, 0, 0, 0);
            if (!kFirst) wn[k] = qn < nq ? __ldcs(wq + 32LL * qn) : zero;
        }
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            if (kFirst) {
                w[k] = make_float4(weight(x[4 * k]), weight(x[4 * k + 1]), weight(x[4 * k + 2]), weight(x[4 * k + 3]));
                __stcs(wq + 32LL * (q + k), w[k]);
            }
            add(0, w[k].x, v[4 * k]);
            add(1, w[k].y, v[4 * k + 1]);
            add(2, w[k].z, v[4 * k + 2]);
            add(3, w[k].w, v[4 * k + 3]);
        }
    }
#pragma unroll
    for (int k = 0; k < NQ; ++k) {  // the quads left, the last of them partial
        const int left = na - 4 * (q + k);
        if (left <= 0) break;
        const int ent[4] = {nxt[k].x, nxt[k].y, nxt[k].z, nxt[k].w};
        float w[4] = {wn[k].x, wn[k].y, wn[k].z, wn[k].w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (kFirst) w[u] = u < left ? weight(row_pos(xs, ent[u])) : 0.f;
            if (u < left) add(u, w[u], row_pos(vin, ent[u]));
        }
        if (kFirst) __stcs(wq + 32LL * (q + k), make_float4(w[0], w[1], w[2], w[3]));
    }
    for (int e = na; e < na_all; ++e) {
        // entry e's place in its quad, without indexing the sums
        const int v = tl.entry(s, e - na);
        const float w = weight(row_pos(xs, v));
        const float4 vj = row_pos(vin, v);
        const int place = e & 3;
        if (place == 0) add(0, w, vj);
        if (place == 1) add(1, w, vj);
        if (place == 2) add(2, w, vj);
        if (place == 3) add(3, w, vj);
    }
    auto four = [](float a, float b, float c, float d) { return (a + c) + (b + d); };
    const float sx = four(axy[0].x, axy[1].x, axy[2].x, axy[3].x), sy = four(axy[0].y, axy[1].y, axy[2].y, axy[3].y);
    const float sz = four(az[0], az[1], az[2], az[3]);
    float tw = vo.w;
    if (kFirst) {
        tw = four(tw4[0], tw4[1], tw4[2], tw4[3]);
        vold[s].w = tw;
    }
    const float b = tw < kEpsilon ? 0.0f : k_.b;
    const float t = tw < kEpsilon ? 1.0f : tw;
    vout[s] = visc_mix(vo, sx, sy, sz, b, t);
}

// Sorted -> caller order with the velocity given: x, v, outDensity (one
// thread per caller particle, as k_finish).
__global__ void __launch_bounds__(256)
    k_finish_v(const float4* __restrict__ xf, const float4* __restrict__ vf, const float* __restrict__ rho_s,
               const int* __restrict__ inv, int n, float* __restrict__ x, float* __restrict__ v,
               float* __restrict__ rho_out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int s = inv[i];
    const float4 p = xf[s], u = vf[s];
    x[3 * i] = p.x;
    x[3 * i + 1] = p.y;
    x[3 * i + 2] = p.z;
    v[3 * i] = u.x;
    v[3 * i + 1] = u.y;
    v[3 * i + 2] = u.z;
    if (rho_out != nullptr) rho_out[i] = rho_s[s];
}

ViscK visc_k(float vis, float h, float dt)
{
    return ViscK{1.0f / h, 45.0f / (13.0f * (float)M_PI * h * h * h), dt * vis / h};
}

// Caller order -> sorted: the solver's starting state.
__global__ void __launch_bounds__(256)
    k_gather_state(const float* __restrict__ x, const float* __restrict__ v, const int* __restrict__ perm,
                   int n, float4* __restrict__ xs0, float4* __restrict__ vs)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    int i = perm[s];
    xs0[s] = make_float4(x[3 * i], x[3 * i + 1], x[3 * i + 2], 0.f);
    vs[s] = make_float4(v[3 * i], v[3 * i + 1], v[3 * i + 2], 0.f);
}

// The Jacobi passes at the block size the context's autotuner chose (128,
// 256 or 512 threads; one thread per particle, so the results do not depend
// on it).
template <template <int> class Launch, class... Args>
static void by_block(int block, Args&&... args)
{
    if (block == 128)
        Launch<128>::run(args...);
    else if (block == 512)
        Launch<512>::run(args...);
    else
        Launch<256>::run(args...);
}
template <class Pass>
struct LaunchPass {
    template <int B>
    struct At {
        static void run(unsigned nb, cudaStream_t st, const float4* cur, const int* rows, const int2* rcnt,
                        int row_cap, int n, PassK pk, float4* out, float* rho, Tail tl)
        {
            if (n <= kDeepMax)
                k_pass<Pass, 64, 4><<<(unsigned)((n + 63) / 64), 64, 0, st>>>(cur, rows, rcnt, row_cap, n, pk, out,
                                                                            rho, tl);
            else
                k_pass<Pass, B, 1><<<nb, B, 0, st>>>(cur, rows, rcnt, row_cap, n, pk, out, rho, tl);
        }
    };
};
// Resident blocks per SM of a persistent pass kernel (one query per shape).
template <class K>
static int resident_blocks(K kernel, int block)
{
    int per_sm = 0, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0);
    return std::max(1, per_sm) * std::max(1, sms);
}
template <class Pass>
struct LaunchPassT {
    template <int B>
    struct At {
        static void run(unsigned, cudaStream_t st, const float4* cur, const int* rows, const int2* rcnt, int row_cap,
                        int n, PassK pk, float4* out, float* rho, Tail tl, SceneTiles T)
        {
            static const int grid = resident_blocks(k_pass_t<Pass, B>, B);
            k_pass_t<Pass, B><<<grid, B, 0, st>>>(cur, rows, rcnt, row_cap, n, pk, out, rho, tl, T);
        }
    };
};
template <int B>
struct LaunchVisc {
    static void run(unsigned nb, cudaStream_t st, bool first, const float4* xs, const float4* vin, float4* vold,
                    const int* rows, float* wrow, const int2* rcnt, int row_cap, int n, ViscK vk, float4* vout, Tail tl)
    {
        const unsigned nd = (unsigned)((n + 63) / 64);
        if (n <= kDeepMax && first)
            k_pass_visc<64, 2, true><<<nd, 64, 0, st>>>(xs, vin, vold, rows, wrow, rcnt, row_cap, n, vk, vout, tl);
        else if (n <= kDeepMax)
            k_pass_visc<64, 4, false><<<nd, 64, 0, st>>>(xs, vin, vold, rows, wrow, rcnt, row_cap, n, vk, vout, tl);
        else if (first)
            k_pass_visc<B, 1, true><<<nb, B, 0, st>>>(xs, vin, vold, rows, wrow, rcnt, row_cap, n, vk, vout, tl);
        else
            k_pass_visc<B, 2, false><<<nb, B, 0, st>>>(xs, vin, vold, rows, wrow, rcnt, row_cap, n, vk, vout, tl);
    }
};

int pbd_fast_solve(pk_ctx* c, int n, const Spiky& k, float mass, int iterations, float dt,
                   float* x, float* v, float* rho_out, cudaStream_t st, float viscosity, int vis_iterations)
{
    if (n <= 0) return 0;
    const int pb = c->tune.pass_block;
    const unsigned nb1 = (unsigned)((n + 255) / 256), nbp = (unsigned)((n + pb - 1) / pb);
    if (c->tune.on) cudaEventRecord(c->tune.ev[2], st);
    int launches = 0;
    const float4* cur = c->xs0;
    const PassK pk = pass_k(k, mass);
    const Tail tl{c->rpool, c->ovf};
    // resident-grid passes (an autotuner shape): scene tiles of batched frames
    // from the cell table
    const bool persist = c->tune.persist;
    SceneTiles T{nullptr, nullptr};
    if (persist && c->grid.nscenes > 1) {
        const int ns = c->grid.nscenes;
        const unsigned nb = (unsigned)((ns + 1 + 255) / 256);
        k_tile_count<<<nb, 256, 0, st>>>(c->blk_start, c->grid.scene_keys >> 6, ns, pb, c->tile_cnt);
        exclusive_scan(c->tile_cnt, ns + 1, c->tile_off, c->scan_part, st);
        k_tile_fill<<<nb, 256, 0, st>>>(c->blk_start, c->grid.scene_keys >> 6, ns, pb, c->tile_off, c->tiles);
        T = SceneTiles{c->tiles, c->tile_off + ns + 1};
        launches += 2 + scan_launches();
    }
    // pass B reads only xl, so it may overwrite the positions pass A read
    // (except xs0, which the velocity update needs)
    for (int it = 0; it < iterations; ++it) {
        const bool last = it == iterations - 1;
        prof_begin(c, PK_PROF_DENSITY, st);
        float* const rho = last ? c->rho : nullptr;
        if (persist)
            by_block<LaunchPassT<DensPass>::At>(pb, nbp, st, cur, c->rows, c->rcnt, c->row_cap, n, pk, c->xb, rho, tl,
                                                T);
        else
            by_block<LaunchPass<DensPass>::At>(pb, nbp, st, cur, c->rows, c->rcnt, c->row_cap, n, pk, c->xb, rho, tl);
        prof_end(c, PK_PROF_DENSITY, st);
        prof_begin(c, PK_PROF_DISP, st);
        if (persist)
            by_block<LaunchPassT<DispPass>::At>(pb, nbp, st, c->xb, c->rows, c->rcnt, c->row_cap, n, pk, c->xa,
                                                (float*)nullptr, tl, T);
        else
            by_block<LaunchPass<DispPass>::At>(pb, nbp, st, c->xb, c->rows, c->rcnt, c->row_cap, n, pk, c->xa,
                                               (float*)nullptr, tl);
        prof_end(c, PK_PROF_DISP, st);
        cur = c->xa;
        launches += 2;
    }
    float* rho = (rho_out != nullptr && iterations > 0) ? rho_out : nullptr;
    prof_begin(c, PK_PROF_FINISH, st);
    if (viscosity > 0.f && vis_iterations > 0) {
        // ImplicitViscosity after the solve (PositionBasedFluidModel.cpp:98), on
        // the same rows; velocities ping-pong between vv and xb
        k_vel_sorted<<<nb1, 256, 0, st>>>(cur, c->xs0, c->vs, c->vv, n, dt);
        const ViscK vk = visc_k(viscosity, k.h, dt);
        float4* vin = c->vv;
        float4* vout = c->xb;
        for (int t = 0; t < vis_iterations; ++t) {
            // the hit rows are not needed any more: their place holds the weights
            by_block<LaunchVisc>(pb, nbp, st, t == 0, cur, vin, c->vs, c->rows, reinterpret_cast<float*>(c->hits),
                                 c->rcnt, c->row_cap, n, vk, vout, tl);
            float4* tmp = vin;
            vin = vout;
            vout = tmp;
        }
        k_finish_v<<<nb1, 256, 0, st>>>(cur, vin, c->rho, c->inv, n, x, v, rho);
        launches += 2 + vis_iterations;
    } else {
        k_finish<<<nb1, 256, 0, st>>>(cur, c->xs0, c->vs, c->rho, c->inv, n, dt, x, v, rho);
        ++launches;
    }
    prof_end(c, PK_PROF_FINISH, st);
    if (c->tune.on) cudaEventRecord(c->tune.ev[3], st);
    return launches;
}

// pbd_fast_solve without viscosity, keeping every Jacobi iterate for a
// reverse pass: ys[0..n) holds y_0 (the integrated positions, as sorted by
// the frame's build), iteration t reads ys[t n ..) and writes ys[(t+1) n ..)
// with the same kernels and arithmetic, so the iterates are those of the
// fused frame bit for bit.  Then x, v in caller order as k_finish writes them.
int pbd_replay_solve(pk_ctx* c, int n, const Spiky& k, float mass, int iterations, float dt, float4* ys,
                     float* x, float* v, cudaStream_t st)
{
    if (n <= 0) return 0;
    const int pb = c->tune.pass_block;
    const unsigned nb1 = (unsigned)((n + 255) / 256), nbp = (unsigned)((n + pb - 1) / pb);
    const PassK pk = pass_k(k, mass);
    const Tail tl{c->rpool, c->ovf};  // unused: the rollout's rows fit their capacity
    for (int it = 0; it < iterations; ++it) {
        by_block<LaunchPass<DensPass>::At>(pb, nbp, st, ys + (size_t)it * n, c->rows, c->rcnt, c->row_cap, n, pk, c->xb,
                                           (float*)nullptr, tl);
        by_block<LaunchPass<DispPass>::At>(pb, nbp, st, c->xb, c->rows, c->rcnt, c->row_cap, n, pk,
                                           ys + (size_t)(it + 1) * n, (float*)nullptr, tl);
    }
    k_finish<<<nb1, 256, 0, st>>>(ys + (size_t)iterations * n, ys, c->vs, c->rho, c->inv, n, dt, x, v, nullptr);
    return 2 * iterations + 1;
}

int gather_state(pk_ctx* c, const float* x, const float* v, int n, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_gather_state<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, v, c->perm, n, c->xs0, c->vs);
    return 1;
}

// ------------------------------------------------------------------------
// Generic path: any NeighborList<int> in caller order (a list that did not
// come from this context's pk_nq_build).  One thread per particle, the
// displacement scattered with atomics as in the reference.

__device__ __forceinline__ int nb_size(const int* index, int cap, long long total, int n, int i)
{
    // NeighborList::getNeighborSize (NeighborList.h:27-41)
    if (cap > 0) return index[i];
    if (i >= n - 1) return (int)(total - index[i]);
    return index[i + 1] - index[i];
}
__device__ __forceinline__ long long nb_at(const int* index, int cap, int i, int k)
{
    return cap > 0 ? (long long)cap * i + k : (long long)index[i] + k;
}

// A neighbour id of a caller's list outside [0, n) is skipped (never read or
// scattered to) and latched as kErrBadIndex where the caller gave a flag word.
__device__ __forceinline__ bool valid_id(int j, int n, int* err)
{
    if (j >= 0 && j < n) return true;
    if (err) atomicOr(err, kErrBadIndex);
    return false;
}

// Sums over a caller's list: G lanes per particle read G consecutive entries
// where a lane per particle read one entry of each of 32 rows.
struct ListLane {
    int i, sub, m;
    long long at;
    bool valid;
};
template <int G>
__device__ __forceinline__ ListLane list_lane(const int* index, int cap, long long total, int n)
{
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    ListLane L;
    L.i = (int)(gid / G);
    L.sub = (int)(gid % G);
    L.valid = L.i < n;
    if (!L.valid) L.i = n - 1;
    L.m = L.valid ? nb_size(index, cap, total, n, L.i) : 0;
    L.at = nb_at(index, cap, L.i, 0);
    return L;
}
template <int G>
__device__ __forceinline__ float lane_sum(float v)
{
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
constexpr int kDensG = 8, kViscG = 4;
static unsigned list_blocks(int n, int lanes) { return (unsigned)(((long long)n * lanes + 255) / 256); }

// 8 lanes per particle read the list's entries together; a thread per particle
// took 47 us at 99k particles with a dynamic list, this 24.
__global__ void __launch_bounds__(256)
    k_g_density(const float* __restrict__ x, int n, const int* __restrict__ index,
                const int* __restrict__ elements, int cap, long long total, Spiky k, float mass,
                float* __restrict__ rho, int* __restrict__ err)
{
    const ListLane L = list_lane<kDensG>(index, cap, total, n);
    const int i = L.i;
    const float xi = x[3 * i], yi = x[3 * i + 1], zi = x[3 * i + 2];
    float acc = 0.f;
#pragma unroll 2
    for (int e = L.sub; e < L.m; e += kDensG) {
        const int j = elements[L.at + e];
        if (!valid_id(j, n, err)) continue;
        const float dx = xi - x[3 * j], dy = yi - x[3 * j + 1], dz = zi - x[3 * j + 2];
        float w, g;
        spiky_wg(k, sqrtf(dx * dx + dy * dy + dz * dz), w, g);
        acc += mass * w;
    }
    acc = lane_sum<kDensG>(acc);
    if (L.valid && L.sub == 0) rho[i] = acc;
}

__global__ void __launch_bounds__(256)
    k_g_lambda(const float* __restrict__ x, const float* __restrict__ rho, int n,
               const int* __restrict__ index, const int* __restrict__ elements, int cap,
               long long total, Spiky k, float* __restrict__ lam, float* __restrict__ dpos,
               int* __restrict__ err)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float xi = x[3 * i], yi = x[3 * i + 1], zi = x[3 * i + 2];
    float sg = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
    int m = nb_size(index, cap, total, n, i);
    for (int e = 0; e < m; ++e) {
        int j = elements[nb_at(index, cap, i, e)];
        if (!valid_id(j, n, err)) continue;
        float dx = xi - x[3 * j], dy = yi - x[3 * j + 1], dz = zi - x[3 * j + 2];
        float r = sqrtf(dx * dx + dy * dy + dz * dz);
        if (r > kEpsilon) {
            float w, g;
            spiky_wg(k, r, w, g);
            float ir = 1.0f / r;
            float g0 = g * dx * ir, g1 = g * dy * ir, g2 = g * dz * ir;
            gx += g0; gy += g1; gz += g2;
            sg += g0 * g0 + g1 * g1 + g2 * g2;
        }
    }
    float l = sg + (gx * gx + gy * gy + gz * gz);
    l = -(rho[i] - 1000.0f) / (l + 0.1f);
    lam[i] = l > 0.0f ? 0.0f : l;
    dpos[3 * i] = 0.f;  // m_deltaPos.reset() (DensityPBD.cu:315)
    dpos[3 * i + 1] = 0.f;
    dpos[3 * i + 2] = 0.f;
}

__global__ void __launch_bounds__(256)
    k_g_disp(const float* __restrict__ x, const float* __restrict__ lam, int n,
             const int* __restrict__ index, const int* __restrict__ elements, int cap,
             long long total, Spiky k, float* __restrict__ dpos, int* __restrict__ err)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float xi = x[3 * i], yi = x[3 * i + 1], zi = x[3 * i + 2], li = lam[i];
    int m = nb_size(index, cap, total, n, i);
    for (int e = 0; e < m; ++e) {
        int j = elements[nb_at(index, cap, i, e)];
        if (!valid_id(j, n, err)) continue;
        float dx = xi - x[3 * j], dy = yi - x[3 * j + 1], dz = zi - x[3 * j + 2];
        float r = sqrtf(dx * dx + dy * dy + dz * dz);
        if (r > kEpsilon) {
            float w, g;
            spiky_wg(k, r, w, g);
            float sl = li + lam[j], ir = 1.0f / r;
            float p0 = 10.0f * dx * sl * g * ir, p1 = 10.0f * dy * sl * g * ir,
                  p2 = 10.0f * dz * sl * g * ir;
            atomicAdd(dpos + 3 * i, p0);
            atomicAdd(dpos + 3 * j, -p0);
            atomicAdd(dpos + 3 * i + 1, p1);
            atomicAdd(dpos + 3 * j + 1, -p1);
            atomicAdd(dpos + 3 * i + 2, p2);
            atomicAdd(dpos + 3 * j + 2, -p2);
        }
    }
}

__global__ void __launch_bounds__(256) k_g_add(float* __restrict__ x, const float* __restrict__ d, long long m)
{
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) x[t] += d[t];
}

__global__ void __launch_bounds__(256)
    k_g_velocity(float* __restrict__ v, const float* __restrict__ x, const float* __restrict__ xold,
                 long long m, float dt)
{
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) v[t] += (x[t] - xold[t]) / dt;
}

int density_generic(const float* x, int n, const int* index, const int* elements, int cap,
                    long long total, const Spiky& k, float mass, float* rho, int* err, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_g_density<<<list_blocks(n, kDensG), 256, 0, st>>>(x, n, index, elements, cap, total, k, mass, rho, err);
    return 1;
}

int pbd_generic_solve(pk_ctx* c, float* x, float* v, int n, const int* index, const int* elements,
                      int cap, long long total, const Spiky& k, float mass, int iterations,
                      float dt, float* rho_out, cudaStream_t st)
{
    return pbd_generic_solve_scratch(x, v, n, index, elements, cap, total, k, mass, iterations, dt, rho_out,
                                     c->g_rho, c->g_lam, c->g_dpos, c->g_xold, c->d_err, st);
}

// The generic solve on caller-supplied scratch (rho_s, lam: n floats; dpos,
// xold: 3n floats): a context's arrays, or the allocation-free entry point's
// fixed array. err (nullable) receives kErrBadIndex for list ids outside [0, n).
int pbd_generic_solve_scratch(float* x, float* v, int n, const int* index, const int* elements,
                              int cap, long long total, const Spiky& k, float mass, int iterations,
                              float dt, float* rho_out, float* rho_s, float* lam, float* dpos,
                              float* xold, int* err, cudaStream_t st)
{
    if (n <= 0) return 0;
    const unsigned nb = (unsigned)((n + 255) / 256);
    const long long m3 = 3LL * n;
    const unsigned nb3 = (unsigned)((m3 + 255) / 256);
    int launches = 0;
    cudaMemcpyAsync(xold, x, sizeof(float) * (size_t)m3, cudaMemcpyDeviceToDevice, st);
    float* rho = rho_out != nullptr ? rho_out : rho_s;
    for (int it = 0; it < iterations; ++it) {
        k_g_density<<<list_blocks(n, kDensG), 256, 0, st>>>(x, n, index, elements, cap, total, k, mass, rho, err);
        k_g_lambda<<<nb, 256, 0, st>>>(x, rho, n, index, elements, cap, total, k, lam, dpos, err);
        k_g_disp<<<nb, 256, 0, st>>>(x, lam, n, index, elements, cap, total, k, dpos, err);
        k_g_add<<<nb3, 256, 0, st>>>(x, dpos, m3);
        launches += 4;
    }
    k_g_velocity<<<nb3, 256, 0, st>>>(v, x, xold, m3, dt);
    return launches + 1;
}

// ------------------------------------------------ integrator and boundary

__global__ void __launch_bounds__(256)
    k_integrate(float* __restrict__ x, float* __restrict__ v, const float* __restrict__ f, int n,
                float gx, float gy, float gz, float dt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float g[3] = {gx, gy, gz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float fa = f != nullptr ? f[3 * i + a] : 0.f;
        float va = v[3 * i + a] + dt * (fa + g[a]);  // K_UpdateVelocity (ParticleIntegrator.cu:69)
        v[3 * i + a] = va;
        if (x != nullptr) x[3 * i + a] += dt * va;  // K_UpdatePosition (ParticleIntegrator.cu:111)
    }
}

int integrate_aos(float* x, float* v, const float* f, int n, const float g[3], float dt, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_integrate<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, v, f, n, g[0], g[1], g[2], dt);
    return 1;
}

__global__ void __launch_bounds__(256) k_advect(float* __restrict__ x, const float* __restrict__ v,
                                                long long m, float dt)
{
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) x[t] += dt * v[t];
}

int advect_aos(float* x, const float* v, int n, float dt, cudaStream_t st)
{
    if (n <= 0) return 0;
    long long m = 3LL * n;
    k_advect<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(x, v, m, dt);
    return 1;
}

int velocity_from_positions(float* v, const float* x, const float* xold, int n, float dt, cudaStream_t st)
{
    if (n <= 0) return 0;
    long long m = 3LL * n;
    k_g_velocity<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(v, x, xold, m, dt);
    return 1;
}

__global__ void __launch_bounds__(256)
    k_boundary(float* __restrict__ x, float* __restrict__ v, int n, SdfView s, float nfric,
               float tfric, float dt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float3 p = make_float3(x[3 * i], x[3 * i + 1], x[3 * i + 2]);
    float3 u = make_float3(v[3 * i], v[3 * i + 1], v[3 * i + 2]);
    if (sdf_constrain(s, i, p, u, nfric, tfric, dt)) {
        x[3 * i] = p.x; x[3 * i + 1] = p.y; x[3 * i + 2] = p.z;
        v[3 * i] = u.x; v[3 * i + 1] = u.y; v[3 * i + 2] = u.z;
    }
}

int boundary_aos(float* x, float* v, int n, const SdfView& s, float nfric, float tfric, float dt,
                 cudaStream_t st)
{
    if (n <= 0) return 0;
    k_boundary<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, v, n, s, nfric, tfric, dt);
    return 1;
}

__global__ void __launch_bounds__(256) k_jitter(float* __restrict__ out, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    curandState st;
    curand_init((unsigned long long)i, 0ull, 0ull, &st);
    out[i] = curand_uniform(&st);
}

int boundary_jitter(float* out, int n, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_jitter<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, n);
    return 1;
}

SdfView sdf_view(const pk_ctx* c)
{
    SdfView s{};
    s.data = c->sdf;
    float mh = 0.f;
    for (int a = 0; a < 3; ++a) {
        s.left[a] = c->sdf_left[a];
        s.inv_h[a] = (float)(1.0 / (double)c->sdf_h[a]);
        s.box_lo[a] = c->sdf_box_lo[a];
        s.box_hi[a] = c->sdf_box_hi[a];
        mh = fmaxf(mh, c->sdf_h[a]);
    }
    s.margin = 2.0f * mh + 1e-6f;
    s.nx = c->sdf_dims[0];
    s.ny = c->sdf_dims[1];
    s.nz = c->sdf_dims[2];
    s.inverted = c->sdf_inverted;
    return s;
}


// ImplicitViscosity on any NeighborList<int> in caller order, 4 lanes per
// particle on positions and velocities packed to 16 bytes.  The weights do not
// change between the sweeps: where w is given, the first sweep keeps them in
// the list's layout and their sums in vold's fourth value, and the others read
// them (kMode 0: form, 1: form and keep, 2: read).  A thread per particle read a
// sector for each entry and for each coordinate: 103 us a sweep at 262k
// particles, now 60 after a first of 129 (which writes the weights).
template <int kMode>
__global__ void __launch_bounds__(256)
    k_g_visc(const float4* __restrict__ x, const float4* __restrict__ vin, float4* __restrict__ vold,
             float4* __restrict__ vout, float* __restrict__ v_last, int n, const int* __restrict__ index,
             const int* __restrict__ elements, int cap, long long total, ViscK k_, float* __restrict__ w_list,
             int* __restrict__ err)
{
    const ListLane L = list_lane<kViscG>(index, cap, total, n);
    const int i = L.i;
    const float4 xi = __ldg(x + i);
    float tw = 0.f, d0 = 0.f, d1 = 0.f, d2v = 0.f;
#pragma unroll 4
    for (int e = L.sub; e < L.m; e += kViscG) {
        const int j = elements[L.at + e];
        float w = 0.0f;
        if (kMode == 2) w = __ldg(w_list + L.at + e);
        if (!valid_id(j, n, err)) continue;
        if (kMode != 2) {
            const float4 xj = __ldg(x + j);
            float d2, ir, dd;
            pair_geom(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, k_.inv_h, d2, ir, dd);
            w = d2 > kEps2 ? k_.cw * dd : 0.0f;
            if (kMode == 1) w_list[L.at + e] = w;
            tw += w;
        }
        const float4 vj = __ldg(vin + j);
        d0 = fmaf(w, vj.x, d0);
        d1 = fmaf(w, vj.y, d1);
        d2v = fmaf(w, vj.z, d2v);
    }
    d0 = lane_sum<kViscG>(d0);
    d1 = lane_sum<kViscG>(d1);
    d2v = lane_sum<kViscG>(d2v);
    if (kMode != 2) tw = lane_sum<kViscG>(tw);
    if (!L.valid || L.sub != 0) return;
    const float4 vo = vold[i];
    if (kMode == 2) tw = vo.w;
    if (kMode == 1) vold[i].w = tw;
    const float b = tw < kEpsilon ? 0.0f : k_.b;
    const float t = tw < kEpsilon ? 1.0f : tw;
    const float4 r = visc_mix(vo, d0, d1, d2v, b, t);
    if (v_last != nullptr) {
        v_last[3LL * i] = r.x;
        v_last[3LL * i + 1] = r.y;
        v_last[3LL * i + 2] = r.z;
    } else {
        vout[i] = r;
    }
}

__global__ void __launch_bounds__(256)
    k_g_pack(const float* __restrict__ x, const float* __restrict__ v, int n, float4* __restrict__ x4,
             float4* __restrict__ v4, float4* __restrict__ vold)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long o = 3LL * i;
    x4[i] = make_float4(x[o], x[o + 1], x[o + 2], 0.f);
    const float4 u = make_float4(v[o], v[o + 1], v[o + 2], 0.f);
    v4[i] = u;
    vold[i] = u;
}

int viscosity_generic(pk_ctx* c, const float* x, float* v, int n, const int* index, const int* elements, int cap,
                      long long total, float vis, float h, int iterations, float dt, cudaStream_t st)
{
    if (n <= 0 || iterations <= 0) return 0;
    const ViscK vk = visc_k(vis, h, dt);
    float4 *x4 = c->g_quads, *vold = x4 + n, *va = vold + n, *vb = va + n;
    // no room for the weights, or a single sweep: every sweep forms them
    float* const w = iterations > 1 && c->g_w_cap >= (cap > 0 ? (long long)n * cap : total) ? c->g_w : nullptr;
    k_g_pack<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, v, n, x4, va, vold);
    for (int t = 0; t < iterations; ++t) {
        float* const last = t == iterations - 1 ? v : nullptr;
        if (w == nullptr)
            k_g_visc<0><<<list_blocks(n, kViscG), 256, 0, st>>>(x4, va, vold, vb, last, n, index, elements, cap, total, vk, w,
                                                        c->d_err);
        else if (t == 0)
            k_g_visc<1><<<list_blocks(n, kViscG), 256, 0, st>>>(x4, va, vold, vb, last, n, index, elements, cap, total, vk, w,
                                                        c->d_err);
        else
            k_g_visc<2><<<list_blocks(n, kViscG), 256, 0, st>>>(x4, va, vold, vb, last, n, index, elements, cap, total, vk, w,
                                                        c->d_err);
        std::swap(va, vb);
    }
    return 1 + iterations;
}

}  // namespace pk
