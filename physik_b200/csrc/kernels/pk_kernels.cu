// pk_kernels.cu -- sm_100a kernels of PhysiK's implicit soft-body step.
//
//   tet_kernel   per tet: F = Ds * DmInv, polar rotation R, corotated stress; stores the
//                corners' P = sqrt(V mu) R g, from which blocks are built, and their part of the
//                right-hand side, or the explicit step's forces (TetView::rec).
//                (FEMModel::ComputeCorotationalElasticForces, FEMModel.cpp:635-679;
//                 ExtractRotationPolar :115-163; ComputeElasticForcesAndStiffness :377-424)
//   block_list_kernel, block_rows_kernel
//                after a pattern change, per stored block its tets and corner pairs; then each
//                step a thread per off-diagonal block and four lanes per row: the upper blocks
//                dt^2 * sum R Ke_ab R^T (+ m I on the diagonal), the right-hand side
//                dt*(f + m g) - dt^2 * sum K_ab v_b, and the block-Jacobi inverse of the
//                diagonal block.  Deterministic: fixed orders, no atomics.
//                (TetMeshPhysicsComponent::UpdateSystem, TetMeshPhysicsComponent.cpp:293-354;
//                 SolverData::AssembleImplicitMatrixAndRhs, SolverData.cpp:308-465;
//                 SolverData::BuildInversePreconditioner, SolverData.cpp:260-306)
//   row_kernel   the same with one thread per row over its tets, where there are no lists.
//   extra_rows_kernel
//                connections and host-emitted contributions added to the rows.
//   explicit_row_kernel
//                the explicit step from the tets' forces (World::IntegrateExplicitEuler).
//   spmv_kernel  y = A x for the upper-stored symmetric BSR (SparseBlockMatrix::Multiply,
//                SparseBlockMatrix.cpp:209-268).
// The PCG kernels live in pk_pcg*.cu.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "pk_device.cuh"

namespace pk {

namespace {

// ------------------------------------------------------------------ SpMV row
// q_r = sum over the row's upper blocks B x_c plus its transposed lower blocks B^T x_c,
// where x = s + beta*d (d omitted when use_d is false).  W lanes share one row; the
// result is reduced over those lanes (fixed tree) and valid in all of them.
// r < 0 marks an idle row slot that still joins the shuffles.
template <class Real, int W>
__device__ __forceinline__ V3<Real> row_spmv(const BsrView<Real>& A, int r, int hl, const Real* s, const Real* d,
                                             Real beta, bool use_d)
{
    V3<Real> acc{Real(0), Real(0), Real(0)};
    if (r >= 0) {
        const int ks = __ldg(A.row_start + r), ke = __ldg(A.row_start + r + 1);
        const int ls = __ldg(A.lt_start + r), le = __ldg(A.lt_start + r + 1);
        const int nu = ke - ks, tot = nu + (le - ls);
        for (int j = hl; j < tot; j += W) {
            int k, c;
            const bool tr = j >= nu;
            if (!tr) {
                k = ks + j;
                c = __ldg(A.col + k);
            } else {
                const int idx = ls + (j - nu);
                k = __ldg(A.lt_block + idx);
                c = __ldg(A.lt_row + idx);
            }
            const M3<Real> B = ld9(A.values, (size_t)k);
            V3<Real> xc = ldcg3(s, c);
            if (use_d) xc = xc + ldcg3(d, c) * beta;
            acc = acc + (tr ? mul_t(B, xc) : mul(B, xc));
        }
    }
#pragma unroll
    for (int off = W / 2; off > 0; off >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
        acc.z += __shfl_xor_sync(0xffffffffu, acc.z, off);
    }
    return acc;
}

// ------------------------------------------------------------------ element stiffness block
// K_ab = V (lambda P_a P_b^T + mu P_b P_a^T + mu (g_a.g_b) R R^T), P = R g, written with
// explicit roundings (products and fused multiply-adds in one fixed order) so that every
// kernel that builds a block produces the same bits, whatever the compiler contracts.
__device__ __forceinline__ float kfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double kfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float kmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double kmul(double a, double b) { return __dmul_rn(a, b); }

__device__ __forceinline__ float kadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double kadd(double a, double b) { return __dadd_rn(a, b); }
template <class Real>
__device__ __forceinline__ V3<Real> kadd3(const V3<Real>& a, const V3<Real>& b)
{
    return V3<Real>{kadd(a.x, b.x), kadd(a.y, b.y), kadd(a.z, b.z)};
}
template <class Real>
__device__ __forceinline__ V3<Real> kscale3(const V3<Real>& a, Real s)
{
    return V3<Real>{kmul(a.x, s), kmul(a.y, s), kmul(a.z, s)};
}
template <class Real>
__device__ __forceinline__ Real kdot(const V3<Real>& a, const V3<Real>& b)
{
    return kfma(a.z, b.z, kfma(a.y, b.y, kmul(a.x, b.x)));
}
// R g for column-major R (R.c[j] is column j).
template <class Real>
__device__ __forceinline__ V3<Real> krot(const M3<Real>& R, const V3<Real>& g)
{
    return V3<Real>{kfma(R.c[2].x, g.z, kfma(R.c[1].x, g.y, kmul(R.c[0].x, g.x))),
                    kfma(R.c[2].y, g.z, kfma(R.c[1].y, g.y, kmul(R.c[0].y, g.x))),
                    kfma(R.c[2].z, g.z, kfma(R.c[1].z, g.y, kmul(R.c[0].z, g.x)))};
}
// R R^T: column j holds the rows' dot products with row j.
template <class Real>
__device__ __forceinline__ M3<Real> krrt(const M3<Real>& R)
{
    const V3<Real> r0{R.c[0].x, R.c[1].x, R.c[2].x}, r1{R.c[0].y, R.c[1].y, R.c[2].y},
        r2{R.c[0].z, R.c[1].z, R.c[2].z};
    M3<Real> m;
    m.c[0] = V3<Real>{kdot(r0, r0), kdot(r1, r0), kdot(r2, r0)};
    m.c[1] = V3<Real>{kdot(r0, r1), kdot(r1, r1), kdot(r2, r1)};
    m.c[2] = V3<Real>{kdot(r0, r2), kdot(r1, r2), kdot(r2, r2)};
    return m;
}
template <class Real>
__device__ __forceinline__ M3<Real> kblock(const V3<Real>& pa, const V3<Real>& pb, const V3<Real>& ga,
                                           const V3<Real>& gb, const M3<Real>& rrt, Real vol, Real lam, Real mu)
{
    const Real l = kmul(vol, lam), m = kmul(vol, mu), md = kmul(m, kdot(ga, gb));
    const Real lp[3] = {kmul(l, pb.x), kmul(l, pb.y), kmul(l, pb.z)};
    const Real mp[3] = {kmul(m, pa.x), kmul(m, pa.y), kmul(m, pa.z)};
    M3<Real> K;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const V3<Real>& rc = rrt.c[j];
        K.c[j] = V3<Real>{kfma(rc.x, md, kfma(pb.x, mp[j], kmul(pa.x, lp[j]))),
                          kfma(rc.y, md, kfma(pb.y, mp[j], kmul(pa.y, lp[j]))),
                          kfma(rc.z, md, kfma(pb.z, mp[j], kmul(pa.z, lp[j])))};
    }
    return K;
}

// K_ab from a record's P = sqrt(V mu) R g and ratio lambda / mu:
//   ratio P_a P_b^T + P_b P_a^T + V mu (g_a.g_b) R R^T,
// whose last term is (P_a.P_b) I to FP32 rounding where the rotation converged (FP32), and
// taken from the record's products (FP64).
__device__ __forceinline__ M3<float> kblock_p(const V3<float>& a, const V3<float>& b, float ratio)
{
    const float s = kdot(a, b);
    const float t[3] = {kmul(ratio, b.x), kmul(ratio, b.y), kmul(ratio, b.z)};
    M3<float> K;
    K.c[0] = V3<float>{kfma(a.x, t[0], kfma(b.x, a.x, s)), kfma(a.y, t[0], kmul(b.y, a.x)),
                       kfma(a.z, t[0], kmul(b.z, a.x))};
    K.c[1] = V3<float>{kfma(a.x, t[1], kmul(b.x, a.y)), kfma(a.y, t[1], kfma(b.y, a.y, s)),
                       kfma(a.z, t[1], kmul(b.z, a.y))};
    K.c[2] = V3<float>{kfma(a.x, t[2], kmul(b.x, a.z)), kfma(a.y, t[2], kmul(b.y, a.z)),
                       kfma(a.z, t[2], kfma(b.z, a.z, s))};
    return K;
}
__device__ __forceinline__ M3<double> kblock_p(const V3<double>& a, const V3<double>& b, double ratio, double gram,
                                               const M3<double>& rrt)
{
    const double t[3] = {kmul(ratio, b.x), kmul(ratio, b.y), kmul(ratio, b.z)}, p[3] = {a.x, a.y, a.z};
    M3<double> K;
#pragma unroll
    for (int j = 0; j < 3; ++j)
        K.c[j] = V3<double>{kfma(rrt.c[j].x, gram, kfma(a.x, t[j], kmul(b.x, p[j]))),
                            kfma(rrt.c[j].y, gram, kfma(a.y, t[j], kmul(b.y, p[j]))),
                            kfma(rrt.c[j].z, gram, kfma(a.z, t[j], kmul(b.z, p[j])))};
    return K;
}

// ------------------------------------------------------------------ tet records
// A corner of a record: three values and a fourth (TetView::rec).
template <class Real>
struct Corner {
    V3<Real> v;
    Real w;
};
__device__ __forceinline__ Corner<float> ld_corner(const float* p)
{
    const float4 c = __ldg(reinterpret_cast<const float4*>(p));
    return {V3<float>{c.x, c.y, c.z}, c.w};
}
__device__ __forceinline__ Corner<double> ld_corner(const double* p)
{
    const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
    return {V3<double>{a.x, a.y, b.x}, b.y};
}
// g_a.g_b's place among the record's ten (FP64).
__device__ __forceinline__ int gram_at(int a, int b)
{
    const int lo = min(a, b), hi = max(a, b);
    return lo * (7 - lo) / 2 + hi;
}
// Block K_ab of a record whose corners hold P.
__device__ __forceinline__ M3<float> record_block(const float*, int, int, V3<float> pa, V3<float> pb, float ratio)
{
    return kblock_p(pa, pb, ratio);
}
__device__ __forceinline__ M3<double> record_block(const double* rec, int a, int b, V3<double> pa, V3<double> pb,
                                                   double ratio)
{
    const double2* q = reinterpret_cast<const double2*>(rec + 42);
    const double2 r0 = __ldg(q), r1 = __ldg(q + 1), r2 = __ldg(q + 2);  // xx xy xz yy yz zz
    M3<double> rrt;
    rrt.c[0] = V3<double>{r0.x, r0.y, r1.x};
    rrt.c[1] = V3<double>{r0.y, r1.y, r2.x};
    rrt.c[2] = V3<double>{r1.x, r2.x, r2.y};
    return kblock_p(pa, pb, ratio, __ldg(rec + 32 + gram_at(a, b)), rrt);
}
// Block K_ab of a record that holds R and S (kFormPlain).
template <class Real>
__device__ __forceinline__ M3<Real> plain_block(const AssemblyArgs<Real>& A, int t, int a, int b)
{
    const Real* rec = A.tets.rec + tet_rec<Real>() * (size_t)t;
    M3<Real> R;
#pragma unroll
    for (int j = 0; j < 3; ++j) R.c[j] = ld_corner(rec + 4 * j).v;
    V3<Real> gr[4], ga, gb;
    shape_gradients(ld9(A.tets.dm_inv, (size_t)t), gr);
    ga = gb = gr[0];
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        if (a == q) ga = gr[q];
        if (b == q) gb = gr[q];
    }
    const Real* prm = A.tets.params + 4 * (size_t)t;
    return kblock(krot(R, ga), krot(R, gb), ga, gb, krrt(R), __ldg(prm), __ldg(prm + 1), __ldg(prm + 2));
}
// Corner a's elastic force -S g_a of such a record.
template <class Real>
__device__ __forceinline__ V3<Real> plain_force(const AssemblyArgs<Real>& A, int t, int a)
{
    const Real* rec = A.tets.rec + tet_rec<Real>() * (size_t)t;
    M3<Real> S;
    S.c[0] = ld_corner(rec + 12).v;
    S.c[1] = ld_corner(rec + 16).v;
    S.c[2] = ld_corner(rec + 20).v;
    V3<Real> gr[4], ga;
    shape_gradients(ld9(A.tets.dm_inv, (size_t)t), gr);
    ga = gr[0];
#pragma unroll
    for (int q = 1; q < 4; ++q)
        if (a == q) ga = gr[q];
    return -krot(S, ga);
}

// The long way, for a tet that is not folded (P_0's fourth value is NaN).
template <class Real>
__device__ __noinline__ M3<Real> unfolded_block(const AssemblyArgs<Real>& A, int t, int a, int b)
{
    const Real* rec = A.tets.rec + tet_rec<Real>() * (size_t)t;
    const Real form = __ldg(rec + 19);
    M3<Real> K;
    K.c[0] = K.c[1] = K.c[2] = V3<Real>{Real(0), Real(0), Real(0)};
    if (form == Real(kFormForces))
        K = record_block(rec, a, b, ld_corner(rec + 4 * a).v, ld_corner(rec + 4 * b).v, __ldg(rec + 23));
    else if (form == Real(kFormPlain))
        K = plain_block(A, t, a, b);
    return K;
}
// Its force on corner a (elastic and damping) into fsum, and its sum_b K_ab v_b into kv;
// true when a block or a velocity is not finite.
template <class Real>
__device__ __noinline__ bool unfolded_rhs(const AssemblyArgs<Real>& A, int t, int a, const V3<Real>& vr, V3<Real>& fsum,
                                          V3<Real>& kv)
{
    const Real* rec = A.tets.rec + tet_rec<Real>() * (size_t)t;
    const Real form = __ldg(rec + 19);
    if (form == Real(kFormSkip)) return false;
    const V3<Real> f = form == Real(kFormForces) ? ld_corner(rec + 16 + 4 * a).v : plain_force(A, t, a);
    const V3<Real> fa = kadd3(f, kscale3(vr, -__ldg(A.tets.params + 4 * (size_t)t + 3)));
    if (finite3(fa)) fsum = kadd3(fsum, fa);
    const int4 tn = __ldg(A.tets.nodes + t);
    bool bad = false;
    for (int b = 0; b < 4; ++b) {
        const M3<Real> K = unfolded_block(A, t, a, b);
        const V3<Real> vb = ld3(A.v, b == 0 ? tn.x : b == 1 ? tn.y : b == 2 ? tn.z : tn.w);
        bad |= !finite9(K) || !finite3(vb);
        kv = kv + mul(K, vb);
    }
    return bad;
}

// ------------------------------------------------------------------ tet kernel
// The part of a tet that does not change between steps: DmInv, volume, lambda, mu.
constexpr int kTetRest = 12;
template <class Real>
__global__ void tet_pack_kernel(const Real* __restrict__ dm_inv, const Real* __restrict__ params, Real* rest,
                                int tet_count)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tet_count) return;
    for (int e = 0; e < 9; ++e) rest[kTetRest * (size_t)t + e] = dm_inv[9 * (size_t)t + e];
    for (int e = 0; e < 3; ++e) rest[kTetRest * (size_t)t + 9 + e] = params[4 * (size_t)t + e];
}
__device__ __forceinline__ void ld_rest(const float* p, float (&w)[kTetRest])
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p) + i);
        w[4 * i] = v.x;
        w[4 * i + 1] = v.y;
        w[4 * i + 2] = v.z;
        w[4 * i + 3] = v.w;
    }
}
__device__ __forceinline__ void ld_rest(const double* p, double (&w)[kTetRest])
{
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(p) + i);
        w[2 * i] = v.x;
        w[2 * i + 1] = v.y;
    }
}

// Tet t's record, corner by corner: put(c, v, w) its corner c, extra(i, x, y) its values 32 +
// 2 i and 33 + 2 i (FP64).
template <class Real, bool kFp64Polar, bool kExplicit, class Put, class Extra>
__device__ __forceinline__ void make_record(const AssemblyArgs<Real>& A, int t, Put put, Extra extra)
{
    Real w[kTetRest];
    ld_rest(A.tets.rest + kTetRest * (size_t)t, w);
    const Real vol = w[9], lam = w[10], mu = w[11], damp = __ldg(A.tets.params + 4 * (size_t)t + 3);
    const unsigned char en = __ldg(A.tets.enabled + t);
    const int4 n = __ldg(A.tets.nodes + t);
    M3<Real> dmi;
#pragma unroll
    for (int j = 0; j < 3; ++j) dmi.c[j] = V3<Real>{w[3 * j], w[3 * j + 1], w[3 * j + 2]};
    M3<Real> f = dmi;
    bool skip = !(en & 1u) || !(vol > Real(0));
    if (!skip) {
        const V3<Real> x0 = ld3(A.x, n.x), x1 = ld3(A.x, n.y), x2 = ld3(A.x, n.z), x3 = ld3(A.x, n.w);
        f = mul(mcols(x1 - x0, x2 - x0, x3 - x0), dmi);
        skip = !finite9(f);
    }
    if (skip) {  // no part in this step (explicit: none of the four forces is finite)
        const V3<Real> none{qnan<Real>(), qnan<Real>(), qnan<Real>()};
#pragma unroll
        for (int k = 0; k < 4; ++k) put(k, none, qnan<Real>());
        if (!kExplicit) put(4, none, Real(kFormSkip));
        return;
    }
    const bool linear = A.linear || (en & 2u);
    M3<Real> R = mident<Real>();
    bool converged = true;
    if (!linear) {
        int iters = 0;
        bool fallback = false;
        if (kFp64Polar && det(f) <= Real(0.25)) {
            // Near-inverted element: the Newton iteration in double precision.
            R = cast<Real>(polar_rotation<double>(cast<double>(f), &iters, &fallback, &converged));
            atomicOr(A.flags, kFlagPolarFp64);
            atomicAdd(&A.stats->polar_fp64_count, 1);
        } else {
            R = polar_rotation<Real>(f, &iters, &fallback, &converged);
        }
        if (fallback) {
            atomicOr(A.flags, kFlagPolarIdentity);
            atomicAdd(&A.stats->polar_identity_count, 1);
        }
    }
    const M3<Real> S = corotated_stress(f, R, linear, vol, lam, mu);
    V3<Real> gr[4];
    shape_gradients(dmi, gr);
    if (kExplicit) {
        // The explicit step needs only the corners' elastic forces -S g_a, with the damping.
#pragma unroll
        for (int k = 0; k < 4; ++k) put(k, -krot(S, gr[k]), damp);
        return;
    }
    // |K_ab entries| <= V (|lambda| + 2 |mu|) |g_a| |g_b|
    Real g2 = Real(0);
#pragma unroll
    for (int k = 0; k < 4; ++k) g2 = fmax(g2, dot(gr[k], gr[k]));
    const bool small = vol * (fabs(lam) + Real(2) * fabs(mu)) * g2 < Real(sizeof(Real) == 4 ? 1.0e37 : 1.0e306);
    // The blocks come from P = sqrt(V mu) R g and lambda / mu; in FP32 only where R R^T is I to
    // rounding.
    const Real m = kmul(vol, mu), root = sqrt(m), ratio = lam / mu;
    const bool regular = small && m > Real(1.0e-30) && fabs(ratio) < Real(1.0e6) && (sizeof(Real) == 8 || converged);
    if (!regular) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            put(j, R.c[j], qnan<Real>());
            put(3 + j, S.c[j], j == 1 ? Real(kFormPlain) : qnan<Real>());
        }
        return;
    }
    // The tet's stiffness times the velocities, folded: with K_ab = R Ke_ab R^T and
    // Ke_ab = V (lambda g_a g_b^T + mu g_b g_a^T + mu (g_a.g_b) I),
    //   sum_b K_ab v_b = Q g_a,  Q = V R (lambda tr(G) I + mu (G + G^T)),
    //   G = R^T sum_b v_b g_b^T = R^T [v1 - v0, v2 - v0, v3 - v0] DmInv,
    // so the row kernel adds T g_a - dt c v_a with T = -(dt S + dt^2 Q) instead of
    // building all 16 blocks.  Used only when every corner force -S g_k - c v_k (the
    // row kernel's force term) and T are finite and no block can overflow; otherwise
    // the row kernel takes the long way with S, which applies the reference's rules
    // for non-finite forces and blocks.
    bool folded = false;
    M3<Real> T = S;
    V3<Real> vk[4] = {S.c[0], S.c[0], S.c[0], S.c[0]};
    if (A.fold) {
        vk[0] = ld3(A.v, n.x);
        vk[1] = ld3(A.v, n.y);
        vk[2] = ld3(A.v, n.z);
        vk[3] = ld3(A.v, n.w);
        const M3<Real> Q = folded_stiffness(R, dmi, vk, linear, vol, lam, mu);
        const Real dt = A.dt, dt2 = dt * dt;
#pragma unroll
        for (int j = 0; j < 3; ++j) T.c[j] = -(S.c[j] * dt + Q.c[j] * dt2);
        folded = finite9(T);
        // Every corner force is finite when S, the gradients and the damping stay small (NaN
        // entries show in T); otherwise each is looked at.
        Real s1 = Real(0), v1 = Real(0);
#pragma unroll
        for (int j = 0; j < 3; ++j) s1 = fmax(s1, fmax(fabs(S.c[j].x), fmax(fabs(S.c[j].y), fabs(S.c[j].z))));
#pragma unroll
        for (int k = 0; k < 4; ++k) v1 = fmax(v1, fmax(fabs(vk[k].x), fmax(fabs(vk[k].y), fabs(vk[k].z))));
        const Real big = sizeof(Real) == 4 ? Real(1.0e18) : Real(1.0e150);
        if (!(s1 < big && g2 < big && v1 < big && fabs(damp) < big))
#pragma unroll
            for (int k = 0; k < 4; ++k) folded = folded && finite3((-mul(S, gr[k])) + vk[k] * (-damp));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        put(k, kscale3(krot(R, gr[k]), root), folded ? ratio : qnan<Real>());
        if (folded)
            put(4 + k, kadd3(krot(T, gr[k]), kscale3(vk[k], -kmul(A.dt, damp))), Real(0));
        else
            put(4 + k, -krot(S, gr[k]), k == 0 ? Real(kFormForces) : ratio);
    }
    if constexpr (sizeof(Real) == 8) {
        const M3<Real> rrt = krrt(R);
        extra(0, kmul(m, kdot(gr[0], gr[0])), kmul(m, kdot(gr[0], gr[1])));
        extra(1, kmul(m, kdot(gr[0], gr[2])), kmul(m, kdot(gr[0], gr[3])));
        extra(2, kmul(m, kdot(gr[1], gr[1])), kmul(m, kdot(gr[1], gr[2])));
        extra(3, kmul(m, kdot(gr[1], gr[3])), kmul(m, kdot(gr[2], gr[2])));
        extra(4, kmul(m, kdot(gr[2], gr[3])), kmul(m, kdot(gr[3], gr[3])));
        extra(5, rrt.c[0].x, rrt.c[0].y);
        extra(6, rrt.c[0].z, rrt.c[1].y);
        extra(7, rrt.c[1].z, rrt.c[2].z);
    }
}

// One thread per tet.  A warp's records leave through shared memory, 16 bytes a lane and
// consecutive lanes on consecutive words: stored by their own threads, 128 bytes apart, they
// took half the L1 data pipe's wavefronts (66 % of its peak).  A record's 16-byte words are
// permuted within each eight (explicit: four) by its lane, so that neither side has bank
// conflicts: 240 -> 183 us with 3.1 M FP32 tets, 602 -> 381 FP64.  Bound now by the polar
// iterations' latency at the registers' occupancy.
template <class Real>
constexpr int kTetThreads = sizeof(Real) == 4 ? 128 : 64;
template <class Real, bool kFp64Polar, bool kExplicit>
__global__ void __launch_bounds__(kTetThreads<Real>, 7)
    tet_kernel(const __grid_constant__ AssemblyArgs<Real> A)
{
    constexpr int kValues = kExplicit ? kTetForces : tet_rec<Real>();
    constexpr int kWords = kValues * int(sizeof(Real)) / 16;  // 16-byte words of a record
    constexpr int kVec = 16 / int(sizeof(Real));
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, t = blockIdx.x * blockDim.x + threadIdx.x;
    Real* const mine = reinterpret_cast<Real*>(smem_raw) + (size_t)(threadIdx.x - lane) * kValues;
    auto word = [&](int q, int c) {  // word c of lane q's record
        return mine + (size_t)(q * kWords + (kWords % 8 == 0 ? c ^ (q & 7) : c ^ ((q >> 1) & 3))) * kVec;
    };
    if (t < A.tets.tet_count) {
        make_record<Real, kFp64Polar, kExplicit>(
            A, t,
            [&](int c, V3<Real> v, Real w) {
                if constexpr (sizeof(Real) == 4) {
                    *reinterpret_cast<float4*>(word(lane, c)) = make_float4(v.x, v.y, v.z, w);
                } else {
                    *reinterpret_cast<double2*>(word(lane, 2 * c)) = make_double2(v.x, v.y);
                    *reinterpret_cast<double2*>(word(lane, 2 * c + 1)) = make_double2(v.z, w);
                }
            },
            [&](int i, Real x, Real y) {
                if constexpr (sizeof(Real) == 8) *reinterpret_cast<double2*>(word(lane, 16 + i)) = make_double2(x, y);
            });
    }
    __syncwarp();
    float4* const out = reinterpret_cast<float4*>(A.tets.rec + (size_t)kValues * (t - lane));
    const int words = kWords * min(32, A.tets.tet_count - (t - lane));
#pragma unroll
    for (int j = 0; j < kWords; ++j) {
        const int i = lane + 32 * j;
        if (i < words) out[i] = *reinterpret_cast<const float4*>(word(i / kWords, i % kWords));
    }
}

// ------------------------------------------------------------------ rows
// The block-Jacobi inverse of a diagonal block (identity without the preconditioner).
template <class Real>
__device__ __forceinline__ M3<Real> row_inverse(const AssemblyArgs<Real>& A, const M3<Real>& diag)
{
    M3<Real> mi = mident<Real>();
    if (A.use_jacobi) {
        const Real d = det(diag);
        if (!finite9(diag) || !isfinite(d) || fabs(d) <= Real(1.0e-8)) {
            atomicOr(A.flags, kFlagSingularDiag);
        } else {
            mi = inverse(diag);
            if (!finite9(mi)) atomicOr(A.flags, kFlagSingularDiag);
        }
    }
    return mi;
}
// Connections or host-emitted contributions follow (extra_rows_kernel): the diagonals are not
// complete yet.
template <class Real>
__host__ __device__ __forceinline__ bool has_extras(const AssemblyArgs<Real>& A)
{
    return A.conn_inc_start || A.ext_rhs_start || A.ext_force;
}
// A row's right-hand side (folded terms, forces and gravity, -dt^2 K v) and inverse.
template <class Real>
__device__ __forceinline__ void finish_row(const AssemblyArgs<Real>& A, int r, Real m, const M3<Real>& diag,
                                           V3<Real> bsum, V3<Real> fsum, V3<Real> kv, bool bad)
{
    const Real dt = A.dt, dt2 = kmul(dt, dt);
    const V3<Real> grav{A.gravity[0], A.gravity[1], A.gravity[2]};
    fsum = kadd3(fsum, kscale3(grav, m));
    const V3<Real> b = kadd3(bsum, kadd3(kscale3(kv, -dt2), kscale3(fsum, dt)));
    bad |= !finite3(kv) || !finite3(b);
    st3(A.rhs, r, b);
    if (bad) atomicOr(A.flags, kFlagPrecomputeFailed);
    if (!has_extras(A)) st9(A.minv, (size_t)r, row_inverse(A, diag));
}

// ------------------------------------------------------------------ assembly by block lists
// Per stored block (r, c) the tets that couple its nodes, as 16 t + 4 a + b (corners a at r, b
// at c) in tet order: block k's list is range[k] = {start, end} of `list`, a row's lists one
// after another from 4 inc_start[r]; ~start marks a diagonal block.  Eight lanes per row, a
// block each.  *missing counts the rows whose tets couple a block the pattern lacks.
__global__ void __launch_bounds__(128)
    block_list_kernel(int n, const int* __restrict__ row_start, const int* __restrict__ col,
                      const int* __restrict__ inc_start, const int* __restrict__ inc_list,
                      const int4* __restrict__ tet_nodes, const int* __restrict__ node_to_dyn, int2* __restrict__ range,
                      unsigned* __restrict__ list, int* __restrict__ missing)
{
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) / 8, lj = threadIdx.x % 8;
    const int ks = r < n ? __ldg(row_start + r) : 0, ke = r < n ? __ldg(row_start + r + 1) : 0;
    const int i0 = r < n ? __ldg(inc_start + r) : 0, i1 = r < n ? __ldg(inc_start + r + 1) : 0;
    int at = 4 * i0, coupled = 0;
    for (int k0 = ks; __any_sync(0xffffffffu, k0 < ke); k0 += 8) {
        const int k = k0 + lj, c = k < ke ? __ldg(col + k) : -2;
        int count = 0;
        for (int pass = 0; pass < 2; ++pass) {
            int start = count;
            if (pass == 1) {
#pragma unroll
                for (int off = 1; off < 8; off <<= 1) {
                    const int o = __shfl_up_sync(0xffffffffu, start, off, 8);
                    if (lj >= off) start += o;
                }
                const int total = __shfl_sync(0xffffffffu, start, 7, 8);
                start += at - count;
                at += total;
                if (k < ke) range[k] = make_int2(c == r ? ~start : start, start + count);
            }
            int found = 0;
            for (int i = i0; i < i1; ++i) {
                const int code = __ldg(inc_list + i);
                const int4 tn = __ldg(tet_nodes + (code >> 2));
                const int nb[4] = {tn.x, tn.y, tn.z, tn.w};
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int cb = __ldg(node_to_dyn + nb[b]);
                    if (pass == 0 && k0 == ks && lj == 0 && cb >= r) ++coupled;
                    if (cb != c) continue;
                    if (pass == 1) list[start + found] = 16u * (unsigned)(code >> 2) + 4u * (unsigned)(code & 3) + (unsigned)b;
                    ++found;
                }
            }
            count = found;
        }
    }
    if (r < n && lj == 0 && coupled != at - 4 * i0) atomicAdd(missing, 1);
}

// The implicit step's rows from the block lists.  The first blocks of the launch take a
// thread per off-diagonal block, K_ab summed over its tets in tet order; the others four
// lanes per row for its diagonal block, right-hand side and block-Jacobi inverse: lane q sums
// the row's tets q, q + 4, ..., joined as (0 + 1) + (2 + 3).  A thread reads P_a and P_b (or
// P_a and B_a), one 16-byte load each, the next tet's while it adds this one's.  Blocks leave
// through shared memory, so that a warp writes one run of the matrix.
//
// Against four lanes per row that staged every tet's record through shared memory and added
// into slots there (bound by the L1 data pipe, 75 wavefronts per warp and incidence, two of
// three lanes idle), the whole assembly went from 872 to 724 us with 3.1 M tets and 541 k rows
// in FP32 (this kernel 423), 1,600 to 1,412 in FP64, 53 to 35 with 98 k tets and 18 k rows, and
// 38 to 16 with 3,072 tets.  Bound now by the latency of the records' gathers.
constexpr int kBlockThreads = 128;
template <class Real>
__global__ void __launch_bounds__(kBlockThreads, sizeof(Real) == 4 ? 7 : 4)
    block_rows_kernel(const __grid_constant__ AssemblyArgs<Real> A, int off_blocks)
{
    __shared__ Real out[kBlockThreads / 32][32 * 9];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Real* const mine = &out[warp][0];
    const Real dt = A.dt, dt2 = kmul(dt, dt);
    M3<Real> sum;
    sum.c[0] = sum.c[1] = sum.c[2] = V3<Real>{Real(0), Real(0), Real(0)};
    if ((int)blockIdx.x < off_blocks) {
        const int k = blockIdx.x * kBlockThreads + threadIdx.x;
        int2 se = make_int2(-1, 0);
        if (k < A.nnz) se = __ldg(A.blk_range + k);
        const bool diagonal = se.x < 0;  // (or beyond the last block)
        int i = diagonal ? 0 : se.x;
        const int end = diagonal ? 0 : se.y;
        unsigned code = i < end ? __ldg(A.blk_list + i) : 0u;
        unsigned next = i + 1 < end ? __ldg(A.blk_list + i + 1) : 0u;
        Corner<Real> pa, pb;
        auto fetch = [&](unsigned x, Corner<Real>& p, Corner<Real>& q) {
            const Real* rec = A.tets.rec + tet_rec<Real>() * (size_t)(x >> 4);
            p = ld_corner(rec + 4 * ((x >> 2) & 3u));
            q = ld_corner(rec + 4 * (x & 3u));
        };
        if (i < end) fetch(code, pa, pb);
        while (i < end) {
            Corner<Real> na, nb;
            if (i + 1 < end) fetch(next, na, nb);
            const unsigned after = i + 2 < end ? __ldg(A.blk_list + i + 2) : 0u;
            const int t = (int)(code >> 4), a = (int)((code >> 2) & 3u), b = (int)(code & 3u);
            M3<Real> K;
            if (!isnan(pa.w))
                K = record_block(A.tets.rec + tet_rec<Real>() * (size_t)t, a, b, pa.v, pb.v, pa.w);
            else
                K = unfolded_block(A, t, a, b);
            sum.c[0] = kadd3(sum.c[0], K.c[0]);
            sum.c[1] = kadd3(sum.c[1], K.c[1]);
            sum.c[2] = kadd3(sum.c[2], K.c[2]);
            code = next;
            next = after;
            pa = na;
            pb = nb;
            ++i;
        }
        if (!finite9(sum)) atomicOr(A.flags, kFlagPrecomputeFailed);
        sum.c[0] = kscale3(sum.c[0], dt2);
        sum.c[1] = kscale3(sum.c[1], dt2);
        sum.c[2] = kscale3(sum.c[2], dt2);
        st9(mine, (size_t)lane, sum);
        const unsigned skip = __ballot_sync(0xffffffffu, diagonal);
        __syncwarp();  // (a vote orders no memory; the lanes leave lists of different lengths)
        Real* dst = A.values + 9 * (size_t)(k - lane);
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const int e = lane + 32 * j;
            if (!((skip >> (e / 9)) & 1u)) dst[e] = mine[e];
        }
        return;
    }
    const int r = ((int)(blockIdx.x - off_blocks) * kBlockThreads + (int)threadIdx.x) / 4, lq = lane & 3;
    const bool valid = r < A.a.n;
    if (blockIdx.x == (unsigned)off_blocks && threadIdx.x == 0 && *A.blk_missing)
        atomicOr(A.flags, kFlagPrecomputeFailed);  // host/device pattern mismatch
    int node = 0, ks = 0;
    int2 se = make_int2(~0, 0);
    if (valid) {
        node = __ldg(A.dyn_to_node + r);
        ks = __ldg(A.a.row_start + r);
        se = __ldg(A.blk_range + ks);
    }
    bool bad = valid && se.x >= 0;  // a row without its diagonal: the host never builds one
    const V3<Real> vr = valid ? ld3(A.v, node) : V3<Real>{Real(0), Real(0), Real(0)};
    const Real m = valid ? __ldg(A.mass + node) : Real(0);
    V3<Real> bsum{Real(0), Real(0), Real(0)}, fsum = bsum, kv = bsum;
    int i = (se.x < 0 ? ~se.x : 0) + lq;
    const int end = se.x < 0 ? se.y : 0;
    unsigned code = i < end ? __ldg(A.blk_list + i) : 0u;
    unsigned next = i + 4 < end ? __ldg(A.blk_list + i + 4) : 0u;
    Corner<Real> pa, ba;
    auto fetch = [&](unsigned x, Corner<Real>& p, Corner<Real>& q) {
        const Real* rec = A.tets.rec + tet_rec<Real>() * (size_t)(x >> 4) + 4 * ((x >> 2) & 3u);
        p = ld_corner(rec);
        q = ld_corner(rec + 16);
    };
    if (i < end) fetch(code, pa, ba);
    while (i < end) {
        Corner<Real> na, nb;
        if (i + 4 < end) fetch(next, na, nb);
        const unsigned after = i + 8 < end ? __ldg(A.blk_list + i + 8) : 0u;
        const int t = (int)(code >> 4), a = (int)((code >> 2) & 3u);
        M3<Real> K;
        if (!isnan(pa.w)) {
            K = record_block(A.tets.rec + tet_rec<Real>() * (size_t)t, a, a, pa.v, pa.v, pa.w);
            bsum = kadd3(bsum, ba.v);
        } else {
            K = unfolded_block(A, t, a, a);
            bad |= unfolded_rhs(A, t, a, vr, fsum, kv);
        }
        sum.c[0] = kadd3(sum.c[0], K.c[0]);
        sum.c[1] = kadd3(sum.c[1], K.c[1]);
        sum.c[2] = kadd3(sum.c[2], K.c[2]);
        code = next;
        next = after;
        pa = na;
        ba = nb;
        i += 4;
    }
    __syncwarp();
    auto join = [&](V3<Real>& v) {
#pragma unroll
        for (int off = 1; off < 4; off <<= 1) {
            v.x = kadd(v.x, __shfl_xor_sync(0xffffffffu, v.x, off));
            v.y = kadd(v.y, __shfl_xor_sync(0xffffffffu, v.y, off));
            v.z = kadd(v.z, __shfl_xor_sync(0xffffffffu, v.z, off));
        }
    };
    join(sum.c[0]);
    join(sum.c[1]);
    join(sum.c[2]);
    join(bsum);
    join(fsum);
    join(kv);
    bad = ((__ballot_sync(0xffffffffu, bad) >> (lane & 28)) & 15u) != 0u;
    if (!valid || lq != 0) return;
    bad |= !finite9(sum);
    M3<Real> diag;
    diag.c[0] = kscale3(sum.c[0], dt2);
    diag.c[1] = kscale3(sum.c[1], dt2);
    diag.c[2] = kscale3(sum.c[2], dt2);
    diag.c[0].x = kadd(m, diag.c[0].x);
    diag.c[1].y = kadd(m, diag.c[1].y);
    diag.c[2].z = kadd(m, diag.c[2].z);
    st9(A.values, (size_t)ks, diag);
    finish_row(A, r, m, diag, bsum, fsum, kv, bad);
}

// Host-emitted contributions and transient point connections, onto assembled rows (PointConnection::UpdateSystem, PointConnection.cpp:55-140: the connection's
// force times the corner's weight, and for stiffness > 0 the blocks k w_a w_b I to every
// corner b with a non-zero weight -- K v_b into the rhs for every b, and into the matrix where
// the column is a dynamic row c >= r; SolverData::AddStiffnessBlock / AddNodeForce).  One
// thread per row, after the rows kernel; then the rows' inverses.
template <class Real>
__global__ void __launch_bounds__(64) extra_rows_kernel(AssemblyArgs<Real> A)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.a.n) return;
    const int j0 = A.conn_inc_start ? __ldg(A.conn_inc_start + r) : 0;
    const int j1 = A.conn_inc_start ? __ldg(A.conn_inc_start + r + 1) : 0;
    int b0 = 0, b1 = 0, m0 = 0, m1 = 0;
    if (A.ext_rhs_start) {
        b0 = __ldg(A.ext_rhs_start + r);
        b1 = __ldg(A.ext_rhs_start + r + 1);
        m0 = __ldg(A.ext_mat_start + r);
        m1 = __ldg(A.ext_mat_start + r + 1);
    }
    const int ks = __ldg(A.a.row_start + r), nu = __ldg(A.a.row_start + r + 1) - ks;
    const Real dt = A.dt, dt2 = kmul(dt, dt);
    V3<Real> fsum{Real(0), Real(0), Real(0)}, kv = fsum;
    bool bad = false;
    auto find_slot = [&](int c) {
        int slot = 0;
        while (slot < nu && __ldg(A.a.col + ks + slot) != c) ++slot;
        return slot;
    };
    auto add = [&](int slot, const M3<Real>& B) {
        Real* q = A.values + 9 * (size_t)(ks + slot);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            q[3 * j] += kmul(dt2, B.c[j].x);
            q[3 * j + 1] += kmul(dt2, B.c[j].y);
            q[3 * j + 2] += kmul(dt2, B.c[j].z);
        }
    };
    for (int i = j0; i < j1; ++i) {
        const int cc = __ldg(A.conn_inc_list + i);
        const int ci = cc >> 2, ca = cc & 3;
        if ((unsigned)ci >= (unsigned)A.conn_count) {
            bad = true;
            continue;
        }
        const Real* ev = A.conn_eval + 4 * (size_t)ci;
        if (!(ev[3] != Real(0))) continue;  // point, velocity or target not finite: nothing
        const int4 cn = __ldg(A.conn_nodes + ci);
        const Real* q = A.conn_params + kConnParams * (size_t)ci;
        const Real wa = __ldg(q + ca);
        fsum = fsum + V3<Real>{ev[0], ev[1], ev[2]} * wa;
        const Real kk = __ldg(q + 7);
        if (!(kk > Real(0))) continue;
        for (int b = 0; b < 4; ++b) {
            const Real wb = __ldg(q + b);
            if (wb == Real(0)) continue;
            const int nb = b == 0 ? cn.x : b == 1 ? cn.y : b == 2 ? cn.z : cn.w;
            const Real kab = kk * wa * wb;
            bad |= !isfinite(kab);
            kv = kv + ld3(A.v, nb) * kab;
            const int c = __ldg(A.node_to_dyn + nb);
            if (c < r) continue;
            const int slot = find_slot(c);
            if (slot >= nu) {
                bad = true;  // pattern does not hold the block: host/device mismatch
                continue;
            }
            add(slot, scale(mident<Real>(), kab));
        }
    }
    for (int i = b0; i < b1; ++i) {
        const int kq = __ldg(A.ext_rhs_list + i);
        const M3<Real> B = ld9(A.ext_blocks, (size_t)kq);
        const V3<Real> vb = ld3(A.v, __ldg(A.ext_nodes + kq).y);
        bad |= !finite3(vb) || !finite9(B);
        kv = kv + mul(B, vb);
    }
    for (int i = m0; i < m1; ++i) {
        const unsigned cq = (unsigned)__ldg(A.ext_mat_list + i);
        const int kq = (int)(cq & 0x7fffffffu);
        const bool tr = (cq & 0x80000000u) != 0;
        M3<Real> B = ld9(A.ext_blocks, (size_t)kq);
        if (tr) B = transpose(B);
        const int2 nd = __ldg(A.ext_nodes + kq);
        const int c = __ldg(A.node_to_dyn + (tr ? nd.x : nd.y));
        const int slot = find_slot(c);
        if (c < r || slot >= nu) {
            bad = true;
            continue;
        }
        add(slot, B);
    }
    if (A.ext_force) fsum = kadd3(fsum, ld3(A.ext_force, r));
    M3<Real> diag;
    for (int k = nu - 1; k >= 0; --k) {  // the diagonal block last
        const Real* q = A.values + 9 * (size_t)(ks + k);
        diag.c[0] = V3<Real>{q[0], q[1], q[2]};
        diag.c[1] = V3<Real>{q[3], q[4], q[5]};
        diag.c[2] = V3<Real>{q[6], q[7], q[8]};
        bad |= !finite9(diag);
    }
    Real* rhs = A.rhs + 3 * (size_t)r;
    const V3<Real> b = kadd3(V3<Real>{rhs[0], rhs[1], rhs[2]}, kadd3(kscale3(kv, -dt2), kscale3(fsum, dt)));
    bad |= !finite3(kv) || !finite3(b);
    st3(A.rhs, r, b);
    if (bad) atomicOr(A.flags, kFlagPrecomputeFailed);
    st9(A.minv, (size_t)r, row_inverse(A, diag));
}

// ------------------------------------------------------------------ sphere contacts
// CollisionSphereComponent::UpdateSystem (CollisionSphereComponent.cpp:112-190): a tet
// whose centroid p = ((x0 w + x1 w) + x2 w) + x3 w (w = 1/4) lies strictly inside the
// sphere, |p - c| < radius, becomes a contact.  The arithmetic rounds each operation once,
// as the reference's Vec3 code does (no contraction into fused multiply-adds).  Only tets
// marked active (flag bit 2) count.  Contacts are appended in any order; the host sorts
// them by tet.
__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double rn_add(double a, double b) { return __dadd_rn(a, b); }

template <class Real>
__global__ void sphere_contact_kernel(const int4* __restrict__ nodes, const unsigned char* __restrict__ flags,
                                      const Real* __restrict__ x, int tet_count, Real cx, Real cy, Real cz,
                                      Real radius, int max_out, int* count, int* out_tet, Real* out_point)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tet_count || !(__ldg(flags + t) & 4u)) return;
    const int4 n = __ldg(nodes + t);
    const int nd[4] = {n.x, n.y, n.z, n.w};
    const Real w = Real(0.25);
    Real p[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        Real acc = rn_mul(__ldg(x + 3 * (size_t)nd[0] + a), w);
#pragma unroll
        for (int k = 1; k < 4; ++k) acc = rn_add(acc, rn_mul(__ldg(x + 3 * (size_t)nd[k] + a), w));
        p[a] = acc;
    }
    const Real dx = rn_add(p[0], -cx), dy = rn_add(p[1], -cy), dz = rn_add(p[2], -cz);
    const Real d2 = rn_add(rn_add(rn_mul(dx, dx), rn_mul(dy, dy)), rn_mul(dz, dz));
    if (!(sqrt(d2) < radius)) return;
    const int slot = atomicAdd(count, 1);
    if (slot >= max_out) return;
    out_tet[slot] = t;
    out_point[3 * (size_t)slot] = p[0];
    out_point[3 * (size_t)slot + 1] = p[1];
    out_point[3 * (size_t)slot + 2] = p[2];
}

// ------------------------------------------------------------------ post-step geometry
// Surface triangles (SurfaceVisualComponent::UpdateVisualSurfaceGeometry,
// SurfaceVisualComponent.cpp:150-213): each triangle's three node positions become its three
// visual vertices and its flat normal Cross(p1 - p0, p2 - p0) / length (0, 1, 0 when the
// length is at most 1e-6) their normals.  Embedded vertices (VisualMeshComponent::
// UpdateDeformedVertices, VisualMeshComponent.cpp:257-333): ((x0 w0 + x1 w1) + x2 w2) + x3 w3
// for the vertices marked live, the others keep their last value.  The positions these read
// are the float copies the components hold (a double state is rounded to float first), and
// every operation is a float operation rounded once, as the reference's Vec3 code does.
template <class Real>
__global__ void surface_triangle_kernel(const int* __restrict__ nodes, int count, const Real* __restrict__ x,
                                        float* __restrict__ verts, float* __restrict__ normals)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    float p[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int n = __ldg(nodes + 3 * t + k);
#pragma unroll
        for (int a = 0; a < 3; ++a) p[k][a] = static_cast<float>(__ldg(x + 3 * (size_t)n + a));
    }
    float e1[3], e2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        e1[a] = __fsub_rn(p[1][a], p[0][a]);
        e2[a] = __fsub_rn(p[2][a], p[0][a]);
    }
    const float cx = __fsub_rn(__fmul_rn(e1[1], e2[2]), __fmul_rn(e1[2], e2[1]));
    const float cy = __fsub_rn(__fmul_rn(e1[2], e2[0]), __fmul_rn(e1[0], e2[2]));
    const float cz = __fsub_rn(__fmul_rn(e1[0], e2[1]), __fmul_rn(e1[1], e2[0]));
    const float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy)), __fmul_rn(cz, cz)));
    float nrm[3] = {0.0f, 1.0f, 0.0f};
    if (len > 0.000001f) {
        nrm[0] = __fdiv_rn(cx, len);
        nrm[1] = __fdiv_rn(cy, len);
        nrm[2] = __fdiv_rn(cz, len);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            verts[9 * (size_t)t + 3 * k + a] = p[k][a];
            normals[9 * (size_t)t + 3 * k + a] = nrm[a];
        }
}

template <class Real>
__global__ void embedded_vertex_kernel(const int* __restrict__ nodes, const float* __restrict__ weights,
                                       const unsigned char* __restrict__ live, int count, const Real* __restrict__ x,
                                       float* __restrict__ verts)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= count || !__ldg(live + v)) return;
    int n[4];
    float w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        n[k] = __ldg(nodes + 4 * v + k);
        w[k] = __ldg(weights + 4 * v + k);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float acc = __fmul_rn(static_cast<float>(__ldg(x + 3 * (size_t)n[0] + a)), w[0]);
#pragma unroll
        for (int k = 1; k < 4; ++k)
            acc = __fadd_rn(acc, __fmul_rn(static_cast<float>(__ldg(x + 3 * (size_t)n[k] + a)), w[k]));
        verts[3 * (size_t)v + a] = acc;
    }
}

// ------------------------------------------------------------------ row kernel
// The rows without block lists (which found no room or do not apply): one thread per row over its tets.
// MAXU > 0: accumulate the row's upper blocks in shared memory (MAXU slots per thread and the
// diagonal's other three partial sums, joined as the block-list kernel joins them); MAXU == 0:
// accumulate in place in the values array (rows of any length).
template <class Real, int MAXU>
__global__ void __launch_bounds__(128) row_kernel(const __grid_constant__ AssemblyArgs<Real> A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Real* acc = reinterpret_cast<Real*>(smem_raw);
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.a.n) return;
    const int T = blockDim.x, tid = threadIdx.x;
    const int node = __ldg(A.dyn_to_node + r);
    const int ks = __ldg(A.a.row_start + r), ke = __ldg(A.a.row_start + r + 1);
    const int nu = ke - ks;
    if (MAXU > 0 && nu > MAXU) {
        atomicOr(A.flags, kFlagRowTooLong | kFlagPrecomputeFailed);
        return;
    }
    Real* gacc = A.values + 9 * (size_t)ks;
#define PK_ACC(slot, e) (MAXU > 0 ? acc[((slot) * 9 + (e)) * T + tid] : gacc[(slot) * 9 + (e)])
    for (int j = 0; j < nu; ++j)
        for (int e = 0; e < 9; ++e) PK_ACC(j, e) = Real(0);
    if (MAXU > 0)
        for (int j = MAXU; j < MAXU + 3; ++j)
            for (int e = 0; e < 9; ++e) PK_ACC(j, e) = Real(0);
    const V3<Real> zero{Real(0), Real(0), Real(0)}, vr = ld3(A.v, node);
    V3<Real> fsum = zero, kv = zero, bsum[4] = {zero, zero, zero, zero};
    bool bad = false;
    const int i0 = __ldg(A.inc_start + r), i1 = __ldg(A.inc_start + r + 1);
    for (int i = i0; i < i1; ++i) {
        const int code = __ldg(A.inc_list + i);
        const int t = code >> 2, a = code & 3, part = (i - i0) & 3;
        const Real* rec = A.tets.rec + tet_rec<Real>() * (size_t)t;
        const Corner<Real> pa = ld_corner(rec + 4 * a);
        const bool folded = !isnan(pa.w);
        if (folded) {
            const V3<Real> ba = ld_corner(rec + 16 + 4 * a).v;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (part == q) bsum[q] = kadd3(bsum[q], ba);
        } else {
            if (__ldg(rec + 19) == Real(kFormSkip)) continue;
            bad |= unfolded_rhs(A, t, a, vr, fsum, kv);
        }
        const int4 tn = __ldg(A.tets.nodes + t);
        for (int b = 0; b < 4; ++b) {
            const int c = __ldg(A.node_to_dyn + (b == 0 ? tn.x : b == 1 ? tn.y : b == 2 ? tn.z : tn.w));
            if (c < r) continue;
            int slot = 0;
            while (slot < nu && __ldg(A.a.col + ks + slot) != c) ++slot;
            if (slot >= nu) {
                bad = true;  // pattern does not hold the block: host/device mismatch
                continue;
            }
            const M3<Real> K = folded ? record_block(rec, a, b, pa.v, ld_corner(rec + 4 * b).v, pa.w)
                                      : unfolded_block(A, t, a, b);
            if (MAXU > 0 && slot == 0 && part > 0) slot = MAXU + part - 1;
            PK_ACC(slot, 0) = kadd(PK_ACC(slot, 0), K.c[0].x);
            PK_ACC(slot, 1) = kadd(PK_ACC(slot, 1), K.c[0].y);
            PK_ACC(slot, 2) = kadd(PK_ACC(slot, 2), K.c[0].z);
            PK_ACC(slot, 3) = kadd(PK_ACC(slot, 3), K.c[1].x);
            PK_ACC(slot, 4) = kadd(PK_ACC(slot, 4), K.c[1].y);
            PK_ACC(slot, 5) = kadd(PK_ACC(slot, 5), K.c[1].z);
            PK_ACC(slot, 6) = kadd(PK_ACC(slot, 6), K.c[2].x);
            PK_ACC(slot, 7) = kadd(PK_ACC(slot, 7), K.c[2].y);
            PK_ACC(slot, 8) = kadd(PK_ACC(slot, 8), K.c[2].z);
        }
    }
    if (MAXU > 0)
        for (int e = 0; e < 9; ++e)
            PK_ACC(0, e) = kadd(kadd(PK_ACC(0, e), PK_ACC(MAXU, e)), kadd(PK_ACC(MAXU + 1, e), PK_ACC(MAXU + 2, e)));
    const Real m = __ldg(A.mass + node), dt2 = kmul(A.dt, A.dt);
    M3<Real> diag = mident<Real>();
    for (int j = 0; j < nu; ++j) {
        M3<Real> blk;
        blk.c[0] = v3<Real>(PK_ACC(j, 0), PK_ACC(j, 1), PK_ACC(j, 2));
        blk.c[1] = v3<Real>(PK_ACC(j, 3), PK_ACC(j, 4), PK_ACC(j, 5));
        blk.c[2] = v3<Real>(PK_ACC(j, 6), PK_ACC(j, 7), PK_ACC(j, 8));
        bad |= !finite9(blk);
        blk.c[0] = kscale3(blk.c[0], dt2);
        blk.c[1] = kscale3(blk.c[1], dt2);
        blk.c[2] = kscale3(blk.c[2], dt2);
        if (j == 0) {
            blk.c[0].x = kadd(m, blk.c[0].x);
            blk.c[1].y = kadd(m, blk.c[1].y);
            blk.c[2].z = kadd(m, blk.c[2].z);
            diag = blk;
        }
        st9(A.values, (size_t)(ks + j), blk);
    }
#undef PK_ACC
    finish_row(A, r, m, diag, kadd3(kadd3(bsum[0], bsum[1]), kadd3(bsum[2], bsum[3])), fsum, kv, bad);
}

// ------------------------------------------------------------------ explicit step
// World::IntegrateExplicitEuler (World.cpp:697-725): a = f / m, v += a dt, x += v dt.  One
// thread per row sums its tets' corner forces (written by the tet kernel, 16 bytes each in
// FP32) in tet order; a force that is not finite is left out, as the reference does.  Bound
// by the latency of dependent loads at the sizes explicit steps run at, so kBatch forces are
// in flight at a time and blocks are small.  On the 64x16x16 beam 27 -> 6 us against the
// general row kernel, which gathered the whole 128-byte record and multiplied S g_a again
// for every corner.
__device__ __forceinline__ void ld_force(const float* p, V3<float>& f, float& damp)
{
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    f = V3<float>{v.x, v.y, v.z};
    damp = v.w;
}
__device__ __forceinline__ void ld_force(const double* p, V3<double>& f, double& damp)
{
    const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
    f = V3<double>{a.x, a.y, b.x};
    damp = b.y;
}
constexpr int kExplicitThreads = 64;
template <class Real>
__global__ void __launch_bounds__(kExplicitThreads) explicit_row_kernel(AssemblyArgs<Real> A)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.a.n) return;
    constexpr int kBatch = sizeof(Real) == 4 ? 12 : 8;
    const int node = __ldg(A.dyn_to_node + r);
    const int i0 = __ldg(A.inc_start + r), i1 = __ldg(A.inc_start + r + 1);
    const V3<Real> vr = ld3(A.v, node), xr = ld3(A.x, node);
    V3<Real> fsum{Real(0), Real(0), Real(0)};
    for (int i = i0; i < i1; i += kBatch) {
        int code[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) code[q] = i + q < i1 ? __ldg(A.inc_list + i + q) : -1;
        V3<Real> f[kBatch];
        Real damp[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
            if (code[q] >= 0) ld_force(A.tets.rec + kTetForces * (size_t)(code[q] >> 2) + 4 * (code[q] & 3), f[q], damp[q]);
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
            if (code[q] >= 0) {
                const V3<Real> fa = kadd3(f[q], kscale3(vr, -damp[q]));
                if (finite3(fa)) fsum = kadd3(fsum, fa);
            }
    }
    if (A.conn_inc_start) {
        const int j0 = __ldg(A.conn_inc_start + r), j1 = __ldg(A.conn_inc_start + r + 1);
        for (int i = j0; i < j1; ++i) {
            const int cc = __ldg(A.conn_inc_list + i);
            const int ci = cc >> 2;
            if ((unsigned)ci >= (unsigned)A.conn_count) continue;
            const Real* ev = A.conn_eval + 4 * (size_t)ci;
            if (!(ev[3] != Real(0))) continue;
            const Real wa = __ldg(A.conn_params + kConnParams * (size_t)ci + (cc & 3));
            fsum = fsum + V3<Real>{ev[0], ev[1], ev[2]} * wa;
        }
    }
    if (A.ext_force) fsum = kadd3(fsum, ld3(A.ext_force, r));
    const Real m = __ldg(A.mass + node);
    const V3<Real> grav{A.gravity[0], A.gravity[1], A.gravity[2]};
    fsum = kadd3(fsum, kscale3(grav, m));
    const V3<Real> acc{fsum.x / m, fsum.y / m, fsum.z / m};
    const V3<Real> nv = vr + acc * A.dt;
    const V3<Real> nx = xr + nv * A.dt;
    st3(A.v, node, nv);
    st3(A.x_out, node, nx);
}

// ------------------------------------------------------------------ point connections
// One thread per connection (PointConnection::UpdateSystem, PointConnection.cpp:55-108):
// the weighted point and velocity of its four nodes, left to right; if they and the
// target are finite, the force k (target - point) - c velocity, else the connection
// contributes nothing this step.  Evaluated before the row kernel, which in explicit mode
// overwrites the nodes' state.
template <class Real>
__global__ void conn_kernel(AssemblyArgs<Real> A)
{
    const int ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci >= A.conn_count) return;
    const int4 cn = __ldg(A.conn_nodes + ci);
    const int nb[4] = {cn.x, cn.y, cn.z, cn.w};
    const Real* q = A.conn_params + kConnParams * (size_t)ci;
    V3<Real> p = ld3(A.x, nb[0]) * __ldg(q);
    V3<Real> u = ld3(A.v, nb[0]) * __ldg(q);
#pragma unroll
    for (int b = 1; b < 4; ++b) {
        p = p + ld3(A.x, nb[b]) * __ldg(q + b);
        u = u + ld3(A.v, nb[b]) * __ldg(q + b);
    }
    const V3<Real> target{__ldg(q + 4), __ldg(q + 5), __ldg(q + 6)};
    Real* ev = A.conn_eval + 4 * (size_t)ci;
    if (!finite3(p) || !finite3(u) || !finite3(target)) {
        ev[0] = ev[1] = ev[2] = Real(0);
        ev[3] = Real(0);
        return;
    }
    const Real k = __ldg(q + 7), damp = __ldg(q + 8);
    const V3<Real> f = (target - p) * k + u * (-damp);
    ev[0] = f.x;
    ev[1] = f.y;
    ev[2] = f.z;
    ev[3] = Real(1);
}

// ------------------------------------------------------------------ SpMV kernel
template <class Real>
__global__ void __launch_bounds__(256) spmv_kernel(BsrView<Real> A, const Real* x, Real* y)
{
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int r = 2 * warp + (lane >> 4);
    const bool valid = r < A.n;
    const V3<Real> q = row_spmv<Real, 16>(A, valid ? r : -1, lane & 15, x, nullptr, Real(0), false);
    if (valid && (lane & 15) == 0) st3(y, r, q);
}

}  // namespace

// ------------------------------------------------------------------ launchers
template <class Real>
cudaError_t launch_tet_kernel(const AssemblyArgs<Real>& args, bool fp64_polar_fallback, cudaStream_t stream)
{
    const int t = args.tets.tet_count;
    if (t <= 0) return cudaSuccess;
    constexpr int T = kTetThreads<Real>;
    const int blocks = (t + T - 1) / T;
    const size_t smem = (size_t)T * (args.explicit_mode ? kTetForces : tet_rec<Real>()) * sizeof(Real);
    if (args.explicit_mode) {
        if (fp64_polar_fallback)
            tet_kernel<Real, true, true><<<blocks, T, smem, stream>>>(args);
        else
            tet_kernel<Real, false, true><<<blocks, T, smem, stream>>>(args);
    } else if (fp64_polar_fallback) {
        tet_kernel<Real, true, false><<<blocks, T, smem, stream>>>(args);
    } else {
        tet_kernel<Real, false, false><<<blocks, T, smem, stream>>>(args);
    }
    return cudaGetLastError();
}

template <class Real>
cudaError_t launch_sphere_contacts(const int* nodes, const unsigned char* flags, const Real* x, int tet_count,
                                   const Real* center, Real radius, int max_out, int* count, int* out_tet,
                                   Real* out_point, cudaStream_t stream)
{
    if (tet_count <= 0) return cudaSuccess;
    sphere_contact_kernel<Real><<<(tet_count + 255) / 256, 256, 0, stream>>>(
        reinterpret_cast<const int4*>(nodes), flags, x, tet_count, center[0], center[1], center[2], radius, max_out,
        count, out_tet, out_point);
    return cudaGetLastError();
}

template <class Real>
cudaError_t launch_visual_kernel(int kind, const int* nodes, const float* weights, const unsigned char* live, int count,
                                 const Real* x, float* verts, float* normals, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    if (kind == 0)
        surface_triangle_kernel<Real><<<(count + 127) / 128, 128, 0, stream>>>(nodes, count, x, verts, normals);
    else
        embedded_vertex_kernel<Real><<<(count + 127) / 128, 128, 0, stream>>>(nodes, weights, live, count, x, verts);
    return cudaGetLastError();
}

template <class Real>
cudaError_t launch_tet_pack(const Real* dm_inv, const Real* params, Real* rest, int tet_count, cudaStream_t stream)
{
    if (tet_count <= 0) return cudaSuccess;
    tet_pack_kernel<Real><<<(tet_count + 255) / 256, 256, 0, stream>>>(dm_inv, params, rest, tet_count);
    return cudaGetLastError();
}

cudaError_t launch_block_list_kernel(int n, const int* row_start, const int* col, const int* inc_start,
                                     const int* inc_list, const int4* tet_nodes, const int* node_to_dyn, int2* range,
                                     unsigned* list, int* missing, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    block_list_kernel<<<(n + 15) / 16, 128, 0, stream>>>(n, row_start, col, inc_start, inc_list, tet_nodes, node_to_dyn,
                                                         range, list, missing);
    return cudaGetLastError();
}

template <class Real>
cudaError_t launch_conn_kernel(const AssemblyArgs<Real>& args, cudaStream_t stream)
{
    if (args.conn_count <= 0) return cudaSuccess;
    conn_kernel<Real><<<(args.conn_count + 127) / 128, 128, 0, stream>>>(args);
    return cudaGetLastError();
}

template <class Real, int MAXU>
static cudaError_t launch_rows(const AssemblyArgs<Real>& args, cudaStream_t stream)
{
    const int n = args.a.n;
    int threads = 128;
    size_t smem = 0;
    if (MAXU > 0) {
        while (threads > 32 && (size_t)(MAXU + 3) * 9 * sizeof(Real) * threads > 48 * 1024) threads >>= 1;
        smem = (size_t)(MAXU + 3) * 9 * sizeof(Real) * threads;
    }
    const int blocks = (n + threads - 1) / threads;
    row_kernel<Real, MAXU><<<blocks, threads, smem, stream>>>(args);
    return cudaGetLastError();
}

template <class Real>
cudaError_t launch_row_kernel(const AssemblyArgs<Real>& args, int max_row_blocks, cudaStream_t stream)
{
    if (args.a.n <= 0) return cudaSuccess;
    if (args.explicit_mode) {
        explicit_row_kernel<Real>
            <<<(args.a.n + kExplicitThreads - 1) / kExplicitThreads, kExplicitThreads, 0, stream>>>(args);
        return cudaGetLastError();
    }
    cudaError_t e;
    if (args.blk_range) {
        const int off = (args.nnz + kBlockThreads - 1) / kBlockThreads;
        const int rows = (int)((4ll * args.a.n + kBlockThreads - 1) / kBlockThreads);
        block_rows_kernel<Real><<<off + rows, kBlockThreads, 0, stream>>>(args, off);
        e = cudaGetLastError();
    } else {
        e = max_row_blocks <= 8    ? launch_rows<Real, 8>(args, stream)
            : max_row_blocks <= 16 ? launch_rows<Real, 16>(args, stream)
                                   : launch_rows<Real, 0>(args, stream);
    }
    if (e != cudaSuccess || !has_extras(args)) return e;
    extra_rows_kernel<Real><<<(args.a.n + 63) / 64, 64, 0, stream>>>(args);
    return cudaGetLastError();
}

template <class Real>
cudaError_t launch_spmv_kernel(const BsrView<Real>& a, const Real* x, Real* y, cudaStream_t stream)
{
    if (a.n <= 0) return cudaSuccess;
    const int threads = 256;
    const int rows_per_block = threads / 16;
    const int blocks = (a.n + rows_per_block - 1) / rows_per_block;
    spmv_kernel<Real><<<blocks, threads, 0, stream>>>(a, x, y);
    return cudaGetLastError();
}

template cudaError_t launch_tet_kernel<float>(const AssemblyArgs<float>&, bool, cudaStream_t);
template cudaError_t launch_tet_kernel<double>(const AssemblyArgs<double>&, bool, cudaStream_t);
template cudaError_t launch_tet_pack<float>(const float*, const float*, float*, int, cudaStream_t);
template cudaError_t launch_tet_pack<double>(const double*, const double*, double*, int, cudaStream_t);
template cudaError_t launch_conn_kernel<float>(const AssemblyArgs<float>&, cudaStream_t);
template cudaError_t launch_conn_kernel<double>(const AssemblyArgs<double>&, cudaStream_t);
template cudaError_t launch_visual_kernel<float>(int, const int*, const float*, const unsigned char*, int,
                                                 const float*, float*, float*, cudaStream_t);
template cudaError_t launch_visual_kernel<double>(int, const int*, const float*, const unsigned char*, int,
                                                  const double*, float*, float*, cudaStream_t);
template cudaError_t launch_sphere_contacts<float>(const int*, const unsigned char*, const float*, int, const float*,
                                                   float, int, int*, int*, float*, cudaStream_t);
template cudaError_t launch_sphere_contacts<double>(const int*, const unsigned char*, const double*, int,
                                                    const double*, double, int, int*, int*, double*, cudaStream_t);
template cudaError_t launch_row_kernel<float>(const AssemblyArgs<float>&, int, cudaStream_t);
template cudaError_t launch_row_kernel<double>(const AssemblyArgs<double>&, int, cudaStream_t);
template cudaError_t launch_spmv_kernel<float>(const BsrView<float>&, const float*, float*, cudaStream_t);
template cudaError_t launch_spmv_kernel<double>(const BsrView<double>&, const double*, double*, cudaStream_t);

}  // namespace pk
