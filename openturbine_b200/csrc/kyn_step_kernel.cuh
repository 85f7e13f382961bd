// kyn_step_kernel.cuh -- fused per-beam time-step kernel for sm_100a.
//
// One CTA owns one beam element for a whole time step: predictor, every
// Newton iteration (tangent operator, quadrature-point physics, node-pair
// integration, assembly of the bordered constraint system, linear solve,
// convergence test, update) and the post-step update.  The beam system lives
// in shared memory for the whole step; HBM is touched only to read the beam's
// constant data and to read/write its resident state.  The beams of one model
// form a thread-block cluster and sum the model's convergence error through
// distributed shared memory, so every beam of a model takes the same Newton
// iterations as the reference's model-wide loop (src/step/step.hpp:54-83).
// Models without beam elements whose constraints are more than single-node
// BCs run in dense_kernel (the bordered system with a pivoted LU).
//
// Linear solve: the reference factors the whole bordered system with a
// sparse direct solver (src/step/solve_system.hpp:27-31).  Here the
// single-node boundary conditions are eliminated exactly: their gradient
// B = grad*T and transpose grad^T are block-diagonal with an identity
// translational block (src/constraints/calculate_fixed_bc_constraint.hpp,
// calculate_prescribed_bc_constraint.hpp), so the constrained node's
// correction follows from a 3x3 solve, the free-node block is eliminated in
// shared memory (FP64 form: by 8x8 blocks; FP32 form: panel LU), and the
// multipliers follow from the constrained rows.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/kynema_b200.h"
#include "kyn_types.h"

namespace kyn {

namespace cg = cooperative_groups;

// ---- small math (src/math/quaternion_operations.hpp, vector_operations.hpp) --
__device__ __forceinline__ void quat_compose(const double* a, const double* b, double* o) {
    o[0] = a[0] * b[0] - a[1] * b[1] - a[2] * b[2] - a[3] * b[3];
    o[1] = a[0] * b[1] + a[1] * b[0] + a[2] * b[3] - a[3] * b[2];
    o[2] = a[0] * b[2] - a[1] * b[3] + a[2] * b[0] + a[3] * b[1];
    o[3] = a[0] * b[3] + a[1] * b[2] - a[2] * b[1] + a[3] * b[0];
}

// Entry (i,j) of the rotation matrix of unit quaternion q.
__host__ __device__ __forceinline__ double rot_entry(const double* q, int i, int j) {
    const double w = q[0], x = q[1], y = q[2], z = q[3];
    switch (i * 3 + j) {
        case 0: return w * w + x * x - y * y - z * z;
        case 1: return 2. * (x * y - w * z);
        case 2: return 2. * (x * z + w * y);
        case 3: return 2. * (x * y + w * z);
        case 4: return w * w - x * x + y * y - z * z;
        case 5: return 2. * (y * z - w * x);
        case 6: return 2. * (x * z - w * y);
        case 7: return 2. * (y * z + w * x);
        default: return w * w - x * x - y * y + z * z;
    }
}

// Entry (i,j) of tilde(v) (VecTilde).
__device__ __forceinline__ double tilde_e(const double* v, int i, int j) {
    if (i == j) return 0.;
    const int k = 3 - i - j;
    const double s = ((i + 1) % 3 == j) ? -1. : 1.;
    return s * v[k];
}

__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

// Exponential map: rotation vector -> quaternion (RotationVectorToQuaternion,
// device form with factor 0 below 1e-12).
static __device__ __noinline__ void rotvec_to_quat(const double* phi, double* q) {
    const double angle = sqrt(phi[0] * phi[0] + phi[1] * phi[1] + phi[2] * phi[2]);
    double s, c;
    sincos(angle / 2., &s, &c);
    const double f = (fabs(angle) < 1.e-12) ? 0. : s / angle;
    q[0] = c;
    q[1] = phi[0] * f;
    q[2] = phi[1] * f;
    q[3] = phi[2] * f;
}

// Solve the 3x3 system M y = r (row-major M) by Cramer's rule; the matrices
// solved here (rotational blocks of the boundary-condition gradient) are
// close to rotations, so the determinant is far from zero.
__device__ inline bool solve3(const double* M, const double* r, double* y) {
    const double c00 = M[4] * M[8] - M[5] * M[7];
    const double c01 = M[5] * M[6] - M[3] * M[8];
    const double c02 = M[3] * M[7] - M[4] * M[6];
    const double det = M[0] * c00 + M[1] * c01 + M[2] * c02;
    if (!(fabs(det) > 0.)) return false;
    const double id = 1. / det;
    y[0] = (r[0] * c00 + M[1] * (M[5] * r[2] - r[1] * M[8]) + M[2] * (r[1] * M[7] - M[4] * r[2])) * id;
    y[1] = (M[0] * (r[1] * M[8] - M[5] * r[2]) + r[0] * c01 + M[2] * (M[3] * r[2] - r[1] * M[6])) * id;
    y[2] = (M[0] * (M[4] * r[2] - r[1] * M[7]) + M[1] * (r[1] * M[6] - M[3] * r[2]) + r[0] * c02) * id;
    return true;
}

// FP64 tensor-core product D += A B for one 8x8x4 tile (mma.sync m8n8k4 .f64).
// Fragment layout per lane l: a = A[l/4][l%4], b = B[l%4][l/4],
// d0/d1 = D[l/4][2(l%4)] / D[l/4][2(l%4)+1].
__device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// ---- bulk copies into shared memory (cp.async.bulk, completion on an mbarrier) --
// One thread arms the barrier with the byte count and issues the copy; every
// thread that reads the data waits on the barrier's phase parity.  The copy
// is a plain (non-multicast) global -> own-CTA shared-memory transfer.
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
// src, dst 16-byte aligned, bytes a multiple of 16.  Every thread that
// accessed the destination through ordinary loads and stores runs
// proxy_fence_async_smem() before the CTA barrier that precedes this call.
__device__ __forceinline__ void proxy_fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// Waits for phase `parity` of the barrier, at most kBulkWaitTries polls;
// false when it gave up.
constexpr int kBulkWaitTries = 1 << 22;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t b = smem_u32(bar);
    for (int i = 0; i < kBulkWaitTries; ++i) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(b), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Doubles of one beam system's per-point section data as it lies in the slab
// from x0' on: x0' [Q][3] (padded to even), r0 [Q][4], M* [Q][36], C* [Q][36]
// (SlabLayout keeps them contiguous); staged per Newton iteration.
__host__ __device__ inline int sec_doubles(int Q) { return ((3 * Q + 1) & ~1) + 76 * Q; }

// ---- shared-memory plan of one CTA --------------------------------------------
// The kernel runs with NT = 128, 256 or 512 threads (up to four, two or one
// CTAs per SM within the 128-register budget); four quadrature points per warp
// are processed at a time and NT/32 warps share the GEMM-shaped phases.  More
// resident CTAs overlap more beams' serial sections (the chain of diagonal
// blocks); more warps per CTA shorten the parallel phases of one beam.
constexpr int kConStride = 96;          // doubles per constraint record in smem
constexpr int kQpInterp = 24;           // doubles of interpolated values per quadrature point (qpi)
constexpr int kHubSmem = 208;           // doubles of the hub record (hubsm)
constexpr int kDriveSmem = 600;         // doubles of the hub record of a drive train

struct Smem {
    int A;              // TR [n6][ldA]; aliased by the interpolated values
    int G;              // weighted quadrature blocks (node-pair integration): FP64 form double
                        // [Q][kGPoint], FP32 form float [4 (Q rounded up to even)][kGCols32]
    int Fc, Fdig;       // double [Q][6]
    int phi, dphi;      // double [Q][N]
    int dphiJ;          // double [Q][N]
    int qpw;            // double [Q][4]
    int q, q_prev, v, vd, a, qd;  // node state
    int T;              // double [N][9]
    int resid;          // double [N][6]
    int b;              // double [n6]  permuted rhs
    int xs;             // double [n6]  permuted solution
    int droot;          // double [n6]  drive train: root corrections per unit shaft rotation
    int con;            // double [nc][kConStride]
    int red;            // double [2][NT/32 + 8]  (offset 0: cluster exchange)
    int hub;            // double [kHubSmem or kDriveSmem] hub state and records, or -1
    int pos;            // int [2][N] row block of each node, node of each row block
    int sec;            // double [sec_doubles(Q)] staged sections, inside A's region after
                        // the interpolated values (quadrature phase only)
    int bar;            // uint64 mbarrier of the section copies
    int bytes;
    int ldA;
};

// Position of entry (row, column) of the beam system: inside its group of eight
// columns an entry's pair moves by the row's place in its group of eight rows,
// which spreads the node-pair stores (rows 6 apart times an even pitch) and the
// column reads of the elimination over four times as many banks; pairs stay
// adjacent.  ldA is a multiple of 8.  The FP32 form keeps its rows as they are,
// an odd number of values apart.
template <typename TR = double>
__host__ __device__ __forceinline__ int sys_at(int ldA, int r, int c) {
    return r * ldA + (sizeof(TR) == 4 ? c : c ^ (r & 6));
}

// Weighted quadrature blocks G [Q][6 rows][kGRow]: what a node pair's 6x6 block
// takes from one point, row r, three columns each.  XI = beta' Muu + gamma' Guu,
// P, C, O, K the stiffness blocks; L / R the left / right three columns; the
// pitches keep the four points and two rows of a quarter-warp's loads in
// different banks.
namespace gblk {
constexpr int XIL = 0, PL = 3, CL = 6;                      // left: w J XI, w P, (w / J) C
constexpr int K = 9, PR = 12, XIR = 15, CR = 18, O = 21;    // right: w J K, w P, w J XI, (w / J) C, w O
}  // namespace gblk
constexpr int kGRow = 26;
constexpr int kGPoint = 6 * kGRow;

// FP32 form: the weighted blocks of a point are four rows of 54 quantities of a
// node pair (56 columns), one row per product of shape factors (phi_i phi_j,
// phi_i phi'_j, phi'_i phi'_j, phi'_i phi_j): L[r][c] (left 6x3 block, logical
// r*3+c), RS[r][k] (right block before the tangent, 18 + r*3+k) and RI[r][c]
// (right inertia block, 36 + r*3+c).  The tensor instruction leaves column
// 8*nt + 2*s + e of a tile row in lane s = lane%4, slot 2*nt + e; the layout
// puts the six values of two right-block rows (RS and RI) in one lane, so
// SM_ij = C_RS T_j + C_RI is formed from registers: lanes 0..2 own rows
// {2s, 2s+1} in slots 0..11 and two L values in slots 12..13 (lane 2: padding),
// lane 3 owns L[0..13].
constexpr int kGCols32 = 56;
__host__ __device__ constexpr int gcol_slot(int s, int t) { return 8 * (t >> 1) + 2 * s + (t & 1); }
__host__ __device__ constexpr int gcol(int logical) {
    return logical < 14   ? gcol_slot(3, logical)
           : logical < 16 ? gcol_slot(0, 12 + logical - 14)
           : logical < 18 ? gcol_slot(1, 12 + logical - 16)
                          : gcol_slot((logical - 18) % 18 / 6,
                                      (logical - 18) % 18 / 3 % 2 * 6 + (logical >= 36 ? 3 : 0) + logical % 3);
}

// Entries of one slot of the Gauss-Jordan pivot buffers for (storage bytes,
// threads): 2 (RT * NT/16 + CT * 16) with the tile sizes GJTile below (the
// pivot pair's column and row entries).
__host__ __device__ constexpr int gj_slot_entries(int real_bytes, int nt) {
    return 2 * (real_bytes == 8 ? (nt == 128 ? 7 * 8 + 4 * 16 : nt == 256 ? 6 * 16 + 6 * 16 : 4 * 32 + 8 * 16)
                                : (nt == 128 ? 8 * 8 + 5 * 16 : nt == 256 ? 8 * 16 + 8 * 16 : 4 * 32 + 8 * 16));
}

// Bytes of the solve-phase scratch that lives in the G region (dead after the
// integration): the two pivot-buffer slots, then FP64 vectors of n6 entries
// (residual, second right-hand side, its solution, correction) and 4 * 16
// doubles of reductions.
__host__ __device__ inline int gj_vec_offset(int real_bytes, int nt) {
    return (2 * gj_slot_entries(real_bytes, nt) * real_bytes + 15) & ~15;
}
// The block elimination keeps its diagonal-block inverses (64 doubles per 8
// rows) in the place of the pivot buffers, the FP32 form's LU its reciprocal
// pivots and a staged tile; beside them only a drive train (hub = 2) needs the
// vectors.  gj_rows: the most rows a Gauss-Jordan grid holds.
__host__ __device__ constexpr int gj_rows(int real_bytes, int nt) {
    return real_bytes == 8 ? (nt == 128 ? 56 : nt == 256 ? 96 : 128) : (nt == 128 ? 64 : 128);
}
__host__ __device__ inline int factor_scratch_bytes(int N, int nc, int real_bytes) {
    return real_bytes == 4 ? 6 * N * 8 + 64 * 8 : ((6 * (N - nc) + 7) / 8) * 64 * 8;
}
__host__ __device__ inline bool solve_vectors(int N, int nc, int real_bytes, int nt, int hub) {
    return hub > 1 || 6 * (N - nc) <= gj_rows(real_bytes, nt);
}
__host__ __device__ inline int solve_vec_offset(int N, int nc, int real_bytes, int nt, int hub) {
    const int gj = 6 * (N - nc) <= gj_rows(real_bytes, nt) ? gj_vec_offset(real_bytes, nt) : 0;
    const int lu = hub > 1 ? factor_scratch_bytes(N, nc, real_bytes) : 0;
    return lu > gj ? lu : gj;
}
__host__ __device__ inline int solve_scratch_bytes(int N, int nc, int real_bytes, int nt, int hub) {
    const int vec = solve_vectors(N, nc, real_bytes, nt, hub)
                        ? solve_vec_offset(N, nc, real_bytes, nt, hub) + 4 * 6 * N * 8 + 64 * 8 : 0;
    const int lu = factor_scratch_bytes(N, nc, real_bytes);
    return vec > lu ? vec : lu;
}

// The system matrix and the quadrature scratch never live at the same time:
// A is assembled after the quadrature phase and consumed by the solve, so the
// two share one region; so do the sections staged for the next quadrature
// phase, copied in once the solve has read A for the last time.
// hub: 0 none, 1 a hub node, 2 a drive train (hub chain of 2 or 3 nodes).
__host__ __device__ inline Smem plan_smem(int N, int Q, int real_bytes, int nt, int nc, int hub, int ldA) {
    Smem S{};
    int o = 0;
    auto take = [&](int bytes) {
        const int r = o;
        o += (bytes + 15) & ~15;
        return r;
    };
    const int n6 = 6 * N;
    S.ldA = ldA;
    // The cluster exchange areas come first, so that every CTA of a model's
    // cluster finds them at the same offset whatever its beam's size.
    S.red = take(2 * (nt / 32 + 8) * 8);
    S.hub = hub ? take((hub > 1 ? kDriveSmem : kHubSmem) * 8) : -1;
    {
        const int a_bytes = n6 * S.ldA * real_bytes;
        const int g_bytes = Q * kQpInterp * 8;
        const int q_bytes = g_bytes + sec_doubles(Q) * 8;
        S.A = take(a_bytes > q_bytes ? a_bytes : q_bytes);
        S.sec = S.A + g_bytes;
    }
    {
        // FP32 form: k-steps of two points, so an odd Q gets one zero pad point
        const int g_bytes = real_bytes == 4 ? 4 * ((Q + 1) & ~1) * kGCols32 * 4 : Q * kGPoint * 8;
        const int s_bytes = solve_scratch_bytes(N, nc, real_bytes, nt, hub);
        S.G = take(g_bytes > s_bytes ? g_bytes : s_bytes);
    }
    S.Fc = take(Q * 6 * 8);
    S.Fdig = take(Q * 6 * 8);
    S.phi = take(Q * N * 8);
    S.dphi = take(Q * N * 8);
    S.dphiJ = take(Q * N * 8);
    S.qpw = take(Q * 4 * 8);
    S.q = take(N * 7 * 8);
    S.q_prev = take(N * 7 * 8);
    S.v = take(N * 6 * 8);
    S.vd = take(N * 6 * 8);
    S.a = take(N * 6 * 8);
    S.qd = take(N * 6 * 8);
    S.T = take(N * 9 * 8);
    S.resid = take(N * 6 * 8);
    S.b = take(n6 * 8);
    S.xs = take(n6 * 8);
    S.droot = hub > 1 ? take(n6 * 8) : -1;
    S.con = take((nc > 0 ? nc : 1) * kConStride * 8);
    S.pos = take(2 * N * 4);
    S.bar = take(8);
    S.bytes = o;
    return S;
}

// Leading dimension of the system: n6 columns and one more where every node is
// free (the right-hand side is column m, a drive train's second one m + 1 with
// m <= n6 - 6), in whole tiles of eight.  Rows 8 values (mod 16) apart put the
// two rows of a quarter-warp's pair loads into different halves of the banks;
// where that padding would cost a resident CTA, or the fit, a row is the next
// multiple of 8.  The FP32 form's rows are n6 + 1 values.
constexpr int kSmemPerSM = 233472;          // 228 KB per SM, 1 KB of it taken per resident CTA
constexpr int kMaxDynSmem = 232448 - 1024;  // 227 KB per CTA on sm_100, minus static use
__host__ __device__ inline Smem make_smem(int N, int Q, int nc, int real_bytes, int nt, int hub = 0) {
    const int n6 = 6 * N, tight = (n6 + 8) & ~7;
    if (real_bytes == 4) return plan_smem(N, Q, real_bytes, nt, nc, hub, n6 + 1);
    const Smem P = plan_smem(N, Q, real_bytes, nt, nc, hub, ((n6 + 8) & ~15) + 8);
    const Smem T = plan_smem(N, Q, real_bytes, nt, nc, hub, tight);
    const int most = 512 / nt;  // resident CTAs that the register budget allows
    const int cp = kSmemPerSM / (P.bytes + 1024), ct = kSmemPerSM / (T.bytes + 1024);
    return P.bytes <= kMaxDynSmem && (cp < most ? cp : most) >= (ct < most ? ct : most) ? P : T;
}

// Constraint record layout inside Smem::con (doubles).
namespace conrec {
constexpr int Phi = 0;     // [6] residual
constexpr int Brot = 6;    // [9] rotational block of B = grad*T (row-major)
constexpr int AX = 15;     // [9] rotational block of grad^T  (= AX(C))
constexpr int Gl = 24;     // [6] grad^T lambda
constexpr int xl = 30;     // [6] multiplier correction
constexpr int lam = 36;    // [6] lambda
constexpr int inp = 42;    // [7] prescribed input
constexpr int yr = 49;     // [6] constrained-row residual b_r - A_r x
constexpr int R1X0 = 55;   // [3] rigid joint: R(hub) X0
constexpr int Btr = 58;    // [9] rigid joint: base block tilde(R1 X0) T_hub
constexpr int Brr = 67;    // [9] rigid joint: base block -AX(C) T_hub
constexpr int dr = 76;     // [6] drive train: root correction per unit shaft rotation
constexpr int wr = 82;     // [6] drive train: root test vector (G w = 0)
constexpr int s2 = 88;     // [6] drive train: A_r x2 of the second right-hand side
}  // namespace conrec

// Shared-memory record of a model's hub (doubles): the hub state in the slab
// layout (hubrec), the hub BC's constraint record, the hub correction, the
// hub multiplier correction, and the per-beam contributions exchanged over
// the cluster (double-buffered by iteration parity).
namespace hubsm {
constexpr int bc = 88;     // [kConStride] constraint record of the hub BC
constexpr int xh = 184;    // [6] hub correction
constexpr int xlh = 190;   // [6] hub multiplier correction (unconditioned)
constexpr int pub = 196;   // [2][6] sum over this beam's joints of G_base^T (lambda + x_lambda)
// drive train (records 1 and 2 of the hub chain, the revolute and rigid joints
// between them, and the vectors of the shaft-rotation elimination)
constexpr int n1 = 208;    // [kHubDoubles] chain record 1 (azimuth node)
constexpr int n2 = 296;    // [kHubDoubles] chain record 2 (hub node), if any
constexpr int rev = 384;   // [64] revolute joint record (revrec)
constexpr int ah = 448;    // [kConStride] rigid joint record 1 -> 2
constexpr int cA = 544;    // [6] record-1 correction at zero shaft rotation
constexpr int nA = 550;    // [6] record-1 correction per unit shaft rotation
constexpr int cH = 556;    // [6] record-2 correction at zero shaft rotation
constexpr int dH = 562;    // [6] record-2 correction per unit shaft rotation
constexpr int wA = 568;    // [6] record-1 test vector
constexpr int wH = 574;    // [6] record-2 test vector
constexpr int theta = 580; // shaft rotation of the Newton correction
constexpr int xt = 584;    // [2][8] this beam's part of the shaft equation (num, den,
                           // G_base^T lambda of its joints), exchanged over the cluster
}  // namespace hubsm

// Revolute joint record (doubles, at hubsm::rev).
namespace revrec {
constexpr int Phi = 0;     // [5] residual
constexpr int x = 5;       // [3] R(base) x0: joint axis
constexpr int y = 8;       // [3] R(target) y0
constexpr int z = 11;      // [3] R(target) z0
constexpr int xcz = 14;    // [3] x cross z
constexpr int xcy = 17;    // [3] x cross y
constexpr int Bt = 20;     // [2][3] rotational rows of G_target T_target
constexpr int Bb = 26;     // [2][3] rotational rows of G_base T_base
constexpr int sys = 32;    // [3] torque about R(target) x0
constexpr int lam = 35;    // [6] multipliers (5 used)
constexpr int xl = 41;     // [6] multiplier correction (unconditioned)
constexpr int GtL = 47;    // [6] G_target^T lambda
constexpr int GbL = 53;    // [6] G_base^T lambda
}  // namespace revrec

// Two adjacent values (even position, 16- or 8-byte aligned).
__device__ __forceinline__ double2 load_pair(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void store_pair(double* p, double a, double b) {
    *reinterpret_cast<double2*>(p) = make_double2(a, b);
}

// Node-pair blocks SM_ij = S_ij T_j + I_ij (integrate_stiffness_matrix.hpp,
// integrate_inertia_matrix.hpp, calculate_system_matrix.hpp) of one beam, on the
// FP64 tensor cores (FP64 form and dense models).  With f = phi_i, g = phi'_i at a point,
//   SM_ij = sum_q f_q H_jq + g_q H'_jq,
//   H  = [phi_j XI_L + phi'_j P_L | (phi_j K + phi'_j P_R) T_j + phi_j XI_R],
//   H' = [phi'_j C_L              | (phi'_j C_R + phi_j O) T_j],
// so the sum over points is a product [N x 2Q][2Q x 36 N] whose second operand
// a lane forms in registers, and the result needs no further step.  A unit of
// work is eight (j, row) lines and one half of the columns: a lane forms its
// line's three columns of H and H' at its point (line lane / 4, point lane % 4
// of a step of four) and holds three column tiles by up to three tiles of nodes
// i.  store(j, row, half) gives put(i, v0, v1, v2), which takes three
// adjacent columns.
//
// The former product over node pairs [N^2 x 4Q][4Q x 56] took N^2 Q 448
// multiply-adds where this takes 144, and was bound by the tensor pipe (36k of
// 55k cycles per iteration at 21 nodes).
template <int NT, typename Tangent, typename Store>
__device__ __forceinline__ void integrate_node_pairs(int N, int Q, const double* phi, const double* dphi,
                                                     const double* G, Tangent tangent, Store store) {
    constexpr int NW = NT / 32, MT = 3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g8 = lane >> 2, t = lane & 3;
    const int lines = 6 * N, blocks = (lines + 7) >> 3;
#pragma unroll 1
    for (int u = warp; u < 2 * blocks; u += NW) {
        const bool right = u < blocks;  // the longer halves first
        const int l0 = 8 * (right ? u : u - blocks);
        const int line = min(l0 + g8, lines - 1);
        const int j = line / 6, r = line - 6 * j;
        const double* gr = G + r * kGRow;
        double T[9];
        if (right) {
            const double* Tj = tangent(j);
#pragma unroll
            for (int k = 0; k < 9; ++k) T[k] = Tj[k];
        }
#pragma unroll 1
        for (int i0 = 0; i0 < N; i0 += 8 * MT) {
            double acc[MT][3][2];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[mt][c][0] = acc[mt][c][1] = 0.;
            const double* g = gr + min(t, Q - 1) * kGPoint;
            const double *pq = phi + min(t, Q - 1) * N, *dq = dphi + min(t, Q - 1) * N;
#pragma unroll 1
            for (int q = t; q - t < Q; q += 4) {
                // past the last point the line's factors are zero; rows i >= N are not stored
                const double pj = q < Q ? pq[j] : 0., dj = q < Q ? dq[j] : 0.;
                double h[3], hp[3];
                if (right) {
                    const double2 g8v = load_pair(g + 8), ga = load_pair(g + 10), gb = load_pair(g + 12),
                                  gc = load_pair(g + 14), gd = load_pair(g + 16), ge = load_pair(g + 18),
                                  gf = load_pair(g + 20), gg = load_pair(g + 22);
                    const double s0 = fma(g8v.y, pj, gb.x * dj), s1 = fma(ga.x, pj, gb.y * dj),
                                 s2 = fma(ga.y, pj, gc.x * dj);
                    const double p0 = fma(ge.x, dj, gf.y * pj), p1 = fma(ge.y, dj, gg.x * pj),
                                 p2 = fma(gf.x, dj, gg.y * pj);
                    const double xi[3] = {gc.y, gd.x, gd.y};
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        h[c] = fma(xi[c], pj, fma(s0, T[c], fma(s1, T[3 + c], s2 * T[6 + c])));
                        hp[c] = fma(p0, T[c], fma(p1, T[3 + c], p2 * T[6 + c]));
                    }
                } else {
                    const double2 ga = load_pair(g), gb = load_pair(g + 2), gc = load_pair(g + 4),
                                  gd = load_pair(g + 6), ge = load_pair(g + 8);
                    h[0] = fma(ga.x, pj, gb.y * dj);
                    h[1] = fma(ga.y, pj, gc.x * dj);
                    h[2] = fma(gb.x, pj, gc.y * dj);
                    hp[0] = gd.x * dj;
                    hp[1] = gd.y * dj;
                    hp[2] = ge.x * dj;
                }
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    if (i0 + 8 * mt < N) {  // uniform
                        const double f = pq[i0 + 8 * mt + g8], fp = dq[i0 + 8 * mt + g8];
#pragma unroll
                        for (int c = 0; c < 3; ++c) dmma884(acc[mt][c][0], acc[mt][c][1], f, h[c]);
#pragma unroll
                        for (int c = 0; c < 3; ++c) dmma884(acc[mt][c][0], acc[mt][c][1], fp, hp[c]);
                    }
                }
                const int step = q + 4 < Q ? 4 : 0;  // past the last point: any, with a zero factor
                g += step * kGPoint;
                pq += step * N;
                dq += step * N;
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int lo = l0 + 2 * t + e;
                if (lo < lines) {
                    const int jo = lo / 6;
                    auto put = store(jo, lo - 6 * jo, right ? 1 : 0);
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
                        if (i0 + 8 * mt + g8 < N)
                            put(i0 + 8 * mt + g8, acc[mt][0][e], acc[mt][1][e], acc[mt][2][e]);
                }
            }
        }
    }
}

// TF32 tensor-core product D += A B for one 16x8x8 tile (mma.sync m16n8k8).
// Fragment layout per lane l (g = l/4, t = l%4): a = {A[g][t], A[g+8][t],
// A[g][t+4], A[g+8][t+4]}, b = {B[t][g], B[t+4][g]}, d = {D[g][2t], D[g][2t+1],
// D[g+8][2t], D[g+8][2t+1]}.
__device__ __forceinline__ void mma_tf32(float* d, const unsigned* a, const unsigned* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// x = hi + lo with hi, lo representable in TF32 (round to nearest, ties away).
__device__ __forceinline__ void split_tf32(float x, unsigned& hi, unsigned& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    const float r = x - __uint_as_float(hi);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(r));
}

// Writes SM_ij = [C_L | C_RS T_j + C_RI] of node pair (i, j), scaled by the
// conditioner, into the system matrix from one lane's integration-GEMM slots
// (column layout: gcol; slot(t) returns the lane's slot t).
template <typename Slot>
__device__ __forceinline__ void store_pair_block(float* A, int ldA, const int* pos, const double* sT,
                                                 int i, int jn, int s4, double cond, Slot slot) {
    float* Arow = A + (6 * pos[i]) * ldA + 6 * pos[jn];
    if (s4 < 3) {
        const double* Tj = sT + jn * 9;
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int r = 2 * s4 + rr;
            // slots 6rr..6rr+2: RS[r][0..2]; 6rr+3..6rr+5: RI[r][0..2]
            double rs[3], ri[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                rs[k] = slot(6 * rr + k);
                ri[k] = slot(6 * rr + 3 + k);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double val = ri[c];
#pragma unroll
                for (int k = 0; k < 3; ++k) val += rs[k] * Tj[k * 3 + c];
                Arow[r * ldA + 3 + c] = static_cast<float>(val * cond);
            }
        }
        if (s4 < 2) {
            // slots 12, 13: L[14 + 2 s4 + e]
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int l = 14 + 2 * s4 + e;
                Arow[(l / 3) * ldA + l % 3] = static_cast<float>(slot(12 + e) * cond);
            }
        }
    } else {
        // slots 0..13: L[0..13]
#pragma unroll
        for (int t = 0; t < 14; ++t) Arow[(t / 3) * ldA + t % 3] = static_cast<float>(slot(t) * cond);
    }
}

// Node-pair blocks of the FP32 form.  For node pair (i, j):
//   C_ij = sum_q sum_m coef_m(i, j, q) G[4q + m]
// with coef = (phi_i phi_j, phi_i phi'_j, phi'_i phi'_j, phi'_i phi_j) and G the
// weighted blocks of the quadrature phase (K / inertia, P, C, O terms); then
// SM_ij = [C_L | C_RS T_j + C_RI], times the conditioner.  TF32 tensor cores with
// the 3-term split (hi*hi + hi*lo + lo*hi, FP32 accumulation), m16n8k8: 16 pairs
// per tile, two points per k-step (an odd Q reads the zero pad point).
//
// The form's states follow its roundings: a closing correction contracts by
// only 1e-3 on the worst beams, so another order of the integration or the
// factorisation moves the positions (by up to 6e-8 m in three steps, on some
// ensembles several times further from the 64-bit step).  Both therefore keep
// their order of operations, although the FP64 tensor cores' product
// (integrate_node_pairs) and the block elimination take less time: 4096 beams of
// 5 to 21 nodes step in 4313 us for 2617.  This takes 42k cycles an iteration at
// 13 nodes (four CTAs to an SM), 69k at 21, factor_fp32 53k and 100k.
template <int NT>
__device__ __forceinline__ void integrate_node_pairs_fp32(int N, int Q, const double* phi, const double* dphi,
                                                          const float* G, float* A, int ldA, const int* pos,
                                                          const double* sT, double cond) {
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int P2 = N * N, s4 = lane & 3, g8 = lane >> 2, QK = (Q + 1) >> 1;
    const double* fi_tab = (s4 < 2) ? phi : dphi;
    const double* fj_tab = (s4 == 0 || s4 == 3) ? phi : dphi;
#pragma unroll 1
    for (int p0 = 16 * warp; p0 < P2; p0 += 16 * NW) {
        const int pa = p0 + g8, pb = p0 + g8 + 8;
        const bool va = pa < P2, vb = pb < P2;
        const int ia = va ? pa / N : 0, ja = va ? pa % N : 0;
        const int ib = vb ? pb / N : 0, jb = vb ? pb % N : 0;
        float acc[7][4];
#pragma unroll
        for (int nt = 0; nt < 7; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll 1
        for (int ks = 0; ks < QK; ++ks) {
            const int q0 = 2 * ks, q1 = 2 * ks + 1;
            const bool q1ok = q1 < Q;
            const int q1c = q1ok ? q1 : q0;
            float av[4];
            av[0] = va ? static_cast<float>(fi_tab[q0 * N + ia] * fj_tab[q0 * N + ja]) : 0.f;
            av[1] = vb ? static_cast<float>(fi_tab[q0 * N + ib] * fj_tab[q0 * N + jb]) : 0.f;
            av[2] = (va && q1ok) ? static_cast<float>(fi_tab[q1c * N + ia] * fj_tab[q1c * N + ja]) : 0.f;
            av[3] = (vb && q1ok) ? static_cast<float>(fi_tab[q1c * N + ib] * fj_tab[q1c * N + jb]) : 0.f;
            unsigned ah[4], al[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) split_tf32(av[r], ah[r], al[r]);
            const float* g0 = G + (4 * q0 + s4) * kGCols32 + g8;
            const float* g1 = G + (4 * q1 + s4) * kGCols32 + g8;
#pragma unroll
            for (int nt = 0; nt < 7; ++nt) {
                unsigned bh[2], bl[2];
                split_tf32(g0[nt * 8], bh[0], bl[0]);
                split_tf32(g1[nt * 8], bh[1], bl[1]);
                mma_tf32(acc[nt], al, bh);
                mma_tf32(acc[nt], ah, bl);
                mma_tf32(acc[nt], ah, bh);
            }
        }
        if (va)
            store_pair_block(A, ldA, pos, sT, ia, ja, s4, cond,
                             [&](int t) { return static_cast<double>(acc[t >> 1][t & 1]); });
        if (vb)
            store_pair_block(A, ldA, pos, sT, ib, jb, s4, cond,
                             [&](int t) { return static_cast<double>(acc[t >> 1][2 + (t & 1)]); });
    }
}

// ---- block elimination of the free block in shared memory (FP64 form) --------------
// Right-looking elimination in 8-row panels on the FP64 tensor cores.  Panel k
// multiplies its rows by the inverse of its 8x8 diagonal
// block, U_kj = D_k^-1 A_kj, in registers, and subtracts A_ik U_kj from the
// rows below; A_kj and A_ik stay as they are, so no panel of L is solved and
// nothing but trailing tiles is stored.  Fragments use the k order
// (0,2,4,6 | 1,3,5,7): a lane's accumulator pair of U^T is then its B operand
// of the update, and every A operand is one two-value load.

// Reciprocal of a pivot: hardware approximation refined by Newton-Raphson
// steps r <- r + r (1 - d r) (each step squares the relative error): two in
// FP64 (exact to the last bit on all tested inputs), one in FP32.
__device__ __forceinline__ double pivot_rcp(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(r, fma(-d, r, 1.), r);
    r = fma(r, fma(-d, r, 1.), r);
    return r;
}
__device__ __forceinline__ float pivot_rcp(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-d, r, 1.f), r);
}

// Reciprocal by one third-order step from the hardware's approximation, a product
// shorter than two Newton steps.  The approximation takes the operand's and gives
// the result's upper 32 bits, 20 of them mantissa: a relative error below 2^-18,
// cubed below 2^-54, half of the rounding.
__device__ __forceinline__ double block_rcp(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d, r, 1.);
    return fma(r, fma(e, e, e), r);
}

// Inverse of an 8x8 block held by one warp in accumulator layout (lane l: row
// l/4, columns 2(l%4) and +1), into buf (row-major, 64 doubles of shared
// memory, also the exchange between the steps: a store and five pair loads
// take half the time of the twenty shuffles they stand for).  Gauss-Jordan over
// four 2x2 pivot blocks D, each inverted through its determinant.  With s the
// row's pivot entries times adj(D) and u the pivot rows' entries of the lane's
// columns, every entry becomes base - (s u) / det; pivot rows (whose pivot
// entries count as -1 in their own place) and columns (u the identity) differ
// only in the operands and a zero base, so the four steps are free of branches
// and hold one reciprocal each.  Bound by the latency of that chain: 966 cycles
// with shuffles, two Newton steps and a test per step, alone on an SM.  A zero
// or non-finite determinant sets bit 2 of *flag; three entries are multiplied
// before the reciprocal comes in, so that a system whose entries lie outside
// 1e-100 .. 1e100 counts as singular.
__device__ __forceinline__ void invert_block8(double v0, double v1, double* buf, int lane, int* flag) {
    const int r = lane >> 2, t = lane & 3;
    bool bad = false;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        store_pair(buf + 2 * lane, v0, v1);
        __syncwarp();
        const double2 ab = load_pair(buf + 18 * p), cd = load_pair(buf + 18 * p + 8);
        const double2 x = load_pair(buf + 8 * r + 2 * p);
        const double2 w0 = load_pair(buf + 16 * p + 2 * t), w1 = load_pair(buf + 16 * p + 8 + 2 * t);
        const double det = fma(ab.x, cd.y, -(ab.y * cd.x));
        const double rd = block_rcp(det);
        bad |= !(fabs(det) > 0.) || !isfinite(rd);
        const bool row0 = r == 2 * p, row1 = r == 2 * p + 1, col = t == p;
        const double x0 = row0 ? -1. : row1 ? 0. : x.x, x1 = row1 ? -1. : row0 ? 0. : x.y;
        const double s0 = fma(x0, cd.y, -(x1 * cd.x)), s1 = fma(x1, ab.x, -(x0 * ab.y));
        const double e0 = fma(s0, w0.x, s1 * w1.x), e1 = fma(s0, w0.y, s1 * w1.y);
        const bool clear = row0 || row1 || col;
        v0 = fma(-rd, col ? s0 : e0, clear ? 0. : v0);
        v1 = fma(-rd, col ? s1 : e1, clear ? 0. : v1);
        __syncwarp();
    }
    store_pair(buf + 2 * lane, v0, v1);
    if (bad && lane == 0) atomicOr(flag, 2);
}

// B operands of the update by panel k in column tile c0, the lane's pair of
// -U^T = -(A_kj^T D_k^-T): the panel's rows are read as they stand.
__device__ __forceinline__ double2 panel_multiplier(const double* A, int ldA, int k0, int c0, double2 dinv, int lane) {
    const int t2 = 2 * (lane & 3);
    const double* a = A + sys_at(ldA, k0 + t2, c0 + (lane >> 2));  // rows t2, t2 + 1 share their column shift
    double u0 = 0., u1 = 0.;
    dmma884(u0, u1, a[0], dinv.x);
    dmma884(u0, u1, a[ldA], dinv.y);
    return make_double2(-u0, -u1);
}

// Inverts diagonal block k0 (rows and columns from m on count as identity)
// after subtracting, for k0 > 0, the update of the panel before it, and
// writes the inverse (row-major 8x8) to dinv_out.  A last block of fewer than
// eight columns shares its tile with right-hand sides, whose update is stored.
// One warp.
__device__ __forceinline__ void factor_diag_block(double* A, int ldA, int m, int k0, const double* dinv_prev,
                                                  double* dinv_out, int lane, int* flag) {
    const int r = k0 + (lane >> 2), c = k0 + 2 * (lane & 3);
    double* at = A + sys_at(ldA, r, c);
    double2 d = load_pair(at);
    if (k0 > 0) {
        const double2 dp = load_pair(dinv_prev + 2 * lane);
        const double2 l = load_pair(at - 8);
        const double2 u = panel_multiplier(A, ldA, k0 - 8, k0, dp, lane);
        dmma884(d.x, d.y, l.x, u.x);
        dmma884(d.x, d.y, l.y, u.y);
    }
    if (k0 + 8 > m) {
        if (r < m && c >= m) store_pair(at, d.x, d.y);
        if (r >= m || c >= m) d.x = (r == c) ? 1. : 0.;
        if (r >= m || c + 1 >= m) d.y = (r == c + 1) ? 1. : 0.;
    }
    invert_block8(d.x, d.y, dinv_out, lane, flag);
}

// Replaces tile c0 of panel k0's rows (those below m) by U = D^-1 A.  One warp;
// no other reads those rows any more.
__device__ __forceinline__ void normalise_tile(double* A, int ldA, int m, int k0, int c0, const double* dinv, int lane) {
    const int t2 = 2 * (lane & 3);
    const bool in = k0 + t2 < m;  // m is even
    double* a = A + sys_at(ldA, k0 + t2, c0 + (lane >> 2));
    const double2 d = load_pair(dinv + 2 * lane);
    double u0 = 0., u1 = 0.;
    dmma884(u0, u1, in ? a[0] : 0., d.x);
    dmma884(u0, u1, in ? a[ldA] : 0., d.y);
    if (in) {
        a[0] = u0;
        a[ldA] = u1;
    }
}

// Eliminates the leading m unknowns of a system with leading dimension ldA (a
// multiple of 8 no smaller than the tiles' extent): nrt row tiles, of which the
// first ceil(m / 8) hold the m pivots (rows from m on are not touched where
// those are all), and nct column tiles with the right-hand sides behind the
// unknowns (columns past them are scratch).  With more row tiles than pivots m
// is a multiple of 8 and the rows below are left with the Schur complement.
// The pivot rows end as U = D^-1 A.  dinv: the inverses of the diagonal blocks,
// 64 doubles each.
//
// Warp 0 runs the serial chain (the next panel's diagonal block: update,
// inversion) while the other warps share the trailing tiles of panel k and the
// rows of panel k - 1, which become U = D^-1 A for the back substitution; one
// barrier per panel.  The former
// form (two barriers per panel, an unblocked 8x8 factorisation and a panel of
// L solved by all threads) spent 62k of 126k cycles per Newton iteration on a
// 13-node beam and 102k of 187k on a 21-node beam, two thirds of them in warp
// 0's chain.
template <int NT>
__device__ __forceinline__ void eliminate_blocks(double* A, int ldA, int m, int nrt, int nct, double* dinv, int* flag) {
    constexpr int NWK = NT / 32 - 1;  // warps on the trailing tiles
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = (m + 7) >> 3;
    const bool schur = nrt > nb;
    const int fr = lane >> 2, fc = (2 * (lane & 3)) ^ (fr & 6);
    const bool past = !schur && 8 * (nb - 1) + fr >= m;  // the lane's row of the last row tile
    if (warp == 0) factor_diag_block(A, ldA, m, 0, dinv, dinv, lane, flag);
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k + (schur ? 0 : 1) < nb; ++k) {
        const int k0 = 8 * k;
        const int next = k + 1 < nb ? 1 : 0;
        if (warp == 0) {
            if (next) factor_diag_block(A, ldA, m, k0 + 8, dinv + 64 * k, dinv + 64 * (k + 1), lane, flag);
        } else {
            // equal runs down the columns of the trailing tiles without the first
            // (warp 0's), then of the tiles of the panel before
            const int ni = nrt - k - 1, total = ni * (nct - k - 1) - next, both = total + (k > 0 ? nct - k : 0);
            const int lo = both * (warp - 1) / NWK, hi = both * warp / NWK;
            const double2 dk = load_pair(dinv + 64 * k + 2 * lane);
            int j = static_cast<int>(__fdividef(static_cast<float>(lo + next) + 0.5f, static_cast<float>(ni)));
            int i = lo + next - j * ni;
#pragma unroll 1
            for (int left = min(hi, total) - lo; left > 0;) {
                const int c0 = 8 * (k + 1 + j), cnt = min(ni - i, left);
                const double2 u = panel_multiplier(A, ldA, k0, c0, dk, lane);
                const double* lp = A + (8 * (k + 1 + i) + fr) * ldA + k0 + fc;
                double* cp = A + (8 * (k + 1 + i) + fr) * ldA + c0 + fc;
                const bool last = i + cnt == ni;  // rows from m on are not stored
#pragma unroll 1
                for (int e = 0; e < cnt; e += 2) {  // two tiles' loads ahead of their stores
                    const bool two = e + 1 < cnt;
                    const int o = two ? 8 * ldA : 0;
                    const double2 l0 = load_pair(lp), l1 = load_pair(lp + o);
                    double2 d0 = load_pair(cp), d1 = load_pair(cp + o);
                    dmma884(d0.x, d0.y, l0.x, u.x);
                    if (two) dmma884(d1.x, d1.y, l1.x, u.x);
                    dmma884(d0.x, d0.y, l0.y, u.y);
                    if (two) dmma884(d1.x, d1.y, l1.y, u.y);
                    if (!(last && past && e + 1 >= cnt)) store_pair(cp, d0.x, d0.y);
                    if (two && !(last && past && e + 2 >= cnt)) store_pair(cp + o, d1.x, d1.y);
                    lp += 16 * ldA;
                    cp += 16 * ldA;
                }
                left -= cnt;
                ++j;
                i = 0;
            }
#pragma unroll 1
            for (int e = max(lo, total); e < hi; ++e)
                normalise_tile(A, ldA, m, k0 - 8, 8 * (k + e - total), dinv + 64 * (k - 1), lane);
        }
        __syncthreads();
    }
    // the panels whose rows are still A: the last but one (none below a Schur
    // complement) and the last, where the columns behind the pivots count: at
    // most three tiles, or with a Schur complement as many as the boundary
    // unknowns and the right-hand side take, in turns
    if (schur) {
#pragma unroll 1
        for (int j = nb + warp; j < nct; j += NT / 32)
            normalise_tile(A, ldA, m, 8 * (nb - 1), 8 * j, dinv + 64 * (nb - 1), lane);
    } else {
        const int n2 = nb > 1 ? nct - nb + 1 : 0;
        if (warp < n2) normalise_tile(A, ldA, m, 8 * (nb - 2), 8 * (nb - 1 + warp), dinv + 64 * (nb - 2), lane);
        else if (warp < n2 + 1)
            normalise_tile(A, ldA, m, 8 * (nb - 1), 8 * (nct - 1 + warp - n2), dinv + 64 * (nb - 1), lane);
    }
    __syncthreads();
}

// Back substitution x_k = y_k - sum_{j>k} U_kj x_j by the CTA, y in xs[0:m] on
// entry (a barrier behind its last write) and x on exit, two blocks of rows per step and barrier.  Warp 0 finds the
// two blocks' x (the pair found before still to be subtracted, then the lower
// block's from the upper rows), while the other warps subtract the pair found
// before from all rows above.  All products run on the tensor cores with x
// spread to the lanes by shuffles: a lane's accumulators are its row's value in
// every column, so sums need no reduction.  One warp alone took 550 to 830
// cycles a block (9.3k at 13 nodes, 14.4k at 21): the sums over the older blocks
// were on its path.
template <int NT>
__device__ __forceinline__ void back_substitute(const double* A, int ldA, int m, double* xs) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = (m + 7) >> 3;
    const int fr = lane >> 2, t2 = 2 * (lane & 3), col = t2 ^ (fr & 6);
    auto tile = [&](int i, int b) {  // the lane's pair of -U_ib; columns past m count as zero
        const double2 a = load_pair(A + (8 * i + fr) * ldA + 8 * b + col);
        const bool in = 8 * b + t2 < m;
        return make_double2(in ? -a.x : 0., in ? -a.y : 0.);
    };
    double2 xh = make_double2(0., 0.), xl = xh;  // warp 0: pairs of the blocks found before
#pragma unroll 1
    for (int kh = nb - 1; kh >= 0; kh -= 2) {
        const bool prev = kh + 2 < nb;  // blocks kh + 1, kh + 2
        const int kl = kh - 1;
        if (warp == 0) {
            const int rh = 8 * kh + fr, rl = 8 * kl + fr;
            double d0 = rh < m ? xs[rh] : 0., d1 = d0;
            double e0 = kl >= 0 ? xs[rl] : 0., e1 = e0;
            double2 c = make_double2(0., 0.);
            if (kl >= 0) c = tile(kl, kh);
            if (prev) {
                const double2 a = tile(kh, kh + 1), b = tile(kh, kh + 2);
                dmma884(d0, d1, a.x, xl.x);
                dmma884(d0, d1, a.y, xl.y);
                dmma884(d0, d1, b.x, xh.x);
                dmma884(d0, d1, b.y, xh.y);
                if (kl >= 0) {
                    const double2 g = tile(kl, kh + 1), h = tile(kl, kh + 2);
                    dmma884(e0, e1, g.x, xl.x);
                    dmma884(e0, e1, g.y, xl.y);
                    dmma884(e0, e1, h.x, xh.x);
                    dmma884(e0, e1, h.y, xh.y);
                }
            }
            xh = make_double2(__shfl_sync(kAll, d0, 4 * t2), __shfl_sync(kAll, d0, 4 * t2 + 4));
            dmma884(e0, e1, c.x, xh.x);
            dmma884(e0, e1, c.y, xh.y);
            xl = make_double2(__shfl_sync(kAll, e0, 4 * t2), __shfl_sync(kAll, e0, 4 * t2 + 4));
            if (t2 == 0) {
                if (rh < m) xs[rh] = d0;
                if (kl >= 0) xs[rl] = e0;
            }
        } else if (prev) {
            const double2 pl = load_pair(xs + 8 * (kh + 1) + t2);
            const int ch = 8 * (kh + 2) + t2;  // the last block may be short
            const double2 ph = ch < m ? load_pair(xs + ch) : make_double2(0., 0.);
#pragma unroll 1
            for (int i = warp - 1; i < kl; i += NW - 1) {
                const double2 a = tile(i, kh + 1), b = tile(i, kh + 2);
                double d0 = xs[8 * i + fr], d1 = d0;
                dmma884(d0, d1, a.x, pl.x);
                dmma884(d0, d1, a.y, pl.y);
                dmma884(d0, d1, b.x, ph.x);
                dmma884(d0, d1, b.y, ph.y);
                if (t2 == 0) xs[8 * i + fr] = d0;
            }
        }
        __syncthreads();
    }
}

// ---- panel LU of the FP32 form's free block in shared memory -----------------------
// The pivot chains (diagonal blocks, panel solves, block back substitution)
// compute in FP32.  Trailing updates run on the FP64 tensor cores (FP32
// operands are exact in FP64; the result is rounded once to FP32 on store).
constexpr int kPanel = 8;  // panel width

// Warp-level factorisation of the kb x kb diagonal block of the panel of
// columns [p0, p0+kb): lane r holds row p0+r; pivots broadcast by shuffles.
__device__ __forceinline__ void factor_diag(float* A, int ldA, int m, int p0, double* rpiv, int lane,
                                            int* flag) {
    const int kb = min(kPanel, m - p0);
    float v[kPanel];
#pragma unroll
    for (int c = 0; c < kPanel; ++c) v[c] = (lane < kb && c < kb) ? A[(p0 + lane) * ldA + p0 + c] : float(0);
#pragma unroll
    for (int j = 0; j < kPanel; ++j) {
        if (j < kb) {
            const float d = __shfl_sync(0xffffffffu, v[j], j);
            float u[kPanel];
#pragma unroll
            for (int c = j + 1; c < kPanel; ++c) u[c] = __shfl_sync(0xffffffffu, v[c], j);
            const float rp = pivot_rcp(d);
            if (lane == 0) {
                rpiv[p0 + j] = static_cast<double>(rp);
                if (!(fabs(d) > float(0)) || !isfinite(rp)) *flag |= 2;
            }
            if (lane > j) {
                const float l = v[j] * rp;
                v[j] = l;
#pragma unroll
                for (int c = j + 1; c < kPanel; ++c) v[c] -= l * u[c];
            }
        }
    }
    if (lane < kb) {
#pragma unroll
        for (int c = 0; c < kPanel; ++c)
            if (c < kb) A[(p0 + lane) * ldA + p0 + c] = v[c];
    }
}

// L21 = A21 U11^{-1} for rows [r_begin, m) of the panel [p0, p0+kb), rows
// strided by `stride` starting at r_begin + idx.
__device__ __forceinline__ void solve_l21(float* A, int ldA, int m, int p0, const double* rpiv,
                                          int r_begin, int idx, int stride) {
    const int kb = min(kPanel, m - p0);
#pragma unroll 2
    for (int r = r_begin + idx; r < m; r += stride) {
        float u[kPanel];
#pragma unroll
        for (int c = 0; c < kPanel; ++c) u[c] = (c < kb) ? A[r * ldA + p0 + c] : float(0);
#pragma unroll
        for (int j = 0; j < kPanel; ++j) {
            if (j < kb) {
                u[j] *= static_cast<float>(rpiv[p0 + j]);
#pragma unroll
                for (int k = j + 1; k < kPanel; ++k)
                    if (k < kb) u[k] -= u[j] * A[(p0 + j) * ldA + p0 + k];
            }
        }
#pragma unroll
        for (int c = 0; c < kPanel; ++c)
            if (c < kb) A[r * ldA + p0 + c] = u[c];
    }
}

// One warp applies panel [k0, k0+kb) to the column tile [c0, c0+8) (columns
// beyond m masked) for rows [rb0, rb1): U12 = L11^{-1} A12 for the tile, then
// A22 -= L21 U12 on the FP64 tensor cores (8x8x4 tiles, two k-steps).
// Where U12 goes:
//   kU12InPlace  - lanes 0..7 solve one column each and overwrite A12 (the
//                  tile of U12 is part of the factorisation);
//   kU12ToStage  - same, but into stage[8][8]; the caller copies it into A once
//                  no other warp reads that A12 tile any more;
//   kU12InRegs   - every lane solves column c0 + lane/4 in registers and
//                  nothing is written (a helper warp on rows of a tile whose
//                  U12 another warp stores).
enum U12Mode { kU12InPlace = 0, kU12ToStage = 1, kU12InRegs = 2 };

template <int kMode>
__device__ __forceinline__ void update_tile(float* A, int ldA, int m, int k0, int kb, int c0, int rb0,
                                            int rb1, double* stage, int lane) {
    const int r0 = k0 + kb;
    const int s4 = lane & 3;
    const int kk0 = k0 + s4, kk1 = k0 + 4 + s4;
    double b0, b1;
    if (kMode != kU12InRegs) {
        if (lane < 8 && c0 + lane <= m) {
            const int c = c0 + lane;
            float u[kPanel];
#pragma unroll
            for (int j = 0; j < kPanel; ++j) u[j] = (j < kb) ? A[(k0 + j) * ldA + c] : float(0);
#pragma unroll
            for (int q = 0; q < kPanel - 1; ++q) {
#pragma unroll
                for (int j = q + 1; j < kPanel; ++j)
                    if (j < kb) u[j] -= A[(k0 + j) * ldA + k0 + q] * u[q];
            }
            if (kMode == kU12InPlace) {
#pragma unroll
                for (int j = 1; j < kPanel; ++j)
                    if (j < kb) A[(k0 + j) * ldA + c] = u[j];
            } else {
#pragma unroll
                for (int j = 0; j < kPanel; ++j) stage[j * 8 + lane] = static_cast<double>(u[j]);
            }
        }
        __syncwarp();
        const int bcol = c0 + (lane >> 2);
        const bool bok = bcol <= m;
        if (kMode == kU12InPlace) {
            b0 = (kk0 < r0 && bok) ? static_cast<double>(A[kk0 * ldA + bcol]) : 0.;
            b1 = (kk1 < r0 && bok) ? static_cast<double>(A[kk1 * ldA + bcol]) : 0.;
        } else {
            b0 = (kk0 < r0 && bok) ? stage[s4 * 8 + (lane >> 2)] : 0.;
            b1 = (kk1 < r0 && bok) ? stage[(4 + s4) * 8 + (lane >> 2)] : 0.;
        }
    } else {
        const int col = c0 + (lane >> 2);
        const bool cok = col <= m;
        float u[kPanel];
#pragma unroll
        for (int j = 0; j < kPanel; ++j) u[j] = (j < kb && cok) ? A[(k0 + j) * ldA + (cok ? col : c0)] : float(0);
#pragma unroll
        for (int q = 0; q < kPanel - 1; ++q) {
#pragma unroll
            for (int j = q + 1; j < kPanel; ++j)
                if (j < kb) u[j] -= A[(k0 + j) * ldA + k0 + q] * u[q];
        }
        b0 = u[0];
        b1 = u[4];
#pragma unroll
        for (int t = 1; t < 4; ++t) {
            b0 = (s4 == t) ? u[t] : b0;
            b1 = (s4 == t) ? u[4 + t] : b1;
        }
        if (kk0 >= r0) b0 = 0.;
        if (kk1 >= r0) b1 = 0.;
    }
    const int dcol = c0 + 2 * s4;
    const bool c0ok = dcol <= m, c1ok = dcol + 1 <= m;
#pragma unroll 2
    for (int rb = rb0; rb < rb1; rb += 8) {
        const int row = rb + (lane >> 2);
        const bool rv = row < rb1;
        const double a0 = (rv && kk0 < r0) ? -static_cast<double>(A[row * ldA + kk0]) : 0.;
        const double a1 = (rv && kk1 < r0) ? -static_cast<double>(A[row * ldA + kk1]) : 0.;
        double d0 = (rv && c0ok) ? static_cast<double>(A[row * ldA + dcol]) : 0.;
        double d1 = (rv && c1ok) ? static_cast<double>(A[row * ldA + dcol + 1]) : 0.;
        dmma884(d0, d1, a0, b0);
        dmma884(d0, d1, a1, b1);
        if (rv && c0ok) A[row * ldA + dcol] = static_cast<float>(d0);
        if (rv && c1ok) A[row * ldA + dcol + 1] = static_cast<float>(d1);
    }
}

// Solves L U y = r for the right-hand side in column rc (rows [0, m)) by one
// warp, in place, with the factors as the LU leaves them (unit L below the
// diagonal, U with its pivots on it, reciprocal pivots in rpiv): forward then
// back substitution, one column per step.
__device__ inline void solve_factored_column(float* A, int ldA, int m, int rc, const double* rpiv, int lane) {
    for (int j = 0; j < m; ++j) {
        const double yj = static_cast<double>(A[j * ldA + rc]);
        for (int i = j + 1 + lane; i < m; i += 32)
            A[i * ldA + rc] = static_cast<float>(static_cast<double>(A[i * ldA + rc]) -
                                              static_cast<double>(A[i * ldA + j]) * yj);
        __syncwarp();
    }
    for (int j = m - 1; j >= 0; --j) {
        const double yj = static_cast<double>(A[j * ldA + rc]) * rpiv[j];
        __syncwarp();
        if (lane == 0) A[j * ldA + rc] = static_cast<float>(yj);
        for (int i = lane; i < j; i += 32)
            A[i * ldA + rc] = static_cast<float>(static_cast<double>(A[i * ldA + rc]) -
                                              static_cast<double>(A[i * ldA + j]) * yj);
        __syncwarp();
    }
}

// Replaces the kb x kb upper-triangular diagonal block of panel p0 (pivots in
// rpiv) by its inverse; lane j < kb computes column j by back substitution
// (lanes >= kb compute on padding and store nothing).
__device__ __forceinline__ void invert_diag_block(float* A, int ldA, int m, int p0, const double* rpiv,
                                                  int lane) {
    const int kb = min(kPanel, m - p0);
    const int jc = lane & 7;
    float x[kPanel];
#pragma unroll
    for (int i = 0; i < kPanel; ++i) x[i] = (i == jc) ? float(1) : float(0);
#pragma unroll
    for (int c = kPanel - 1; c >= 0; --c) {
        if (c < kb) {  // warp-uniform; x[c] = 0 for c > jc, so no lane test is needed
            x[c] *= static_cast<float>(rpiv[p0 + c]);
#pragma unroll
            for (int i = 0; i < c; ++i) x[i] -= A[(p0 + i) * ldA + p0 + c] * x[c];
        }
    }
    __syncwarp();
    if (lane < kb) {
#pragma unroll
        for (int i = 0; i < kPanel; ++i)
            if (i <= lane) A[(p0 + i) * ldA + p0 + lane] = x[i];
    }
}

// Block back substitution U x = y by one warp (y in column m), with the
// diagonal blocks already inverted: x_b = U_bb^{-1} y_b, then the rows above
// the block take y_i -= U_i,b x_b.  Arithmetic in FP32; the solution is written
// to xs in FP64.
__device__ __forceinline__ void back_substitute_blocked(const float* A, int ldA, int m, double* xs, int lane) {
    for (int i = lane; i < m; i += 32) xs[i] = static_cast<double>(A[i * ldA + m]);
    __syncwarp();
    const int nblk = (m + kPanel - 1) / kPanel;
    for (int b = nblk - 1; b >= 0; --b) {
        const int k0 = b * kPanel, kb = min(kPanel, m - k0);
        float xv = float(0);
        if (lane < kb) {
#pragma unroll
            for (int c = 0; c < kPanel; ++c)
                if (c >= lane && c < kb) xv += A[(k0 + lane) * ldA + k0 + c] * static_cast<float>(xs[k0 + c]);
        }
        __syncwarp();
        if (lane < kb) xs[k0 + lane] = static_cast<double>(xv);
        __syncwarp();
        float xb[kPanel];
#pragma unroll
        for (int c = 0; c < kPanel; ++c) xb[c] = (c < kb) ? static_cast<float>(xs[k0 + c]) : float(0);
#pragma unroll 2
        for (int i = lane; i < k0; i += 32) {
            float acc = static_cast<float>(xs[i]);
#pragma unroll
            for (int c = 0; c < kPanel; ++c)
                if (c < kb) acc -= A[i * ldA + k0 + c] * xb[c];
            xs[i] = static_cast<double>(acc);
        }
        __syncwarp();
    }
}

// Factors the leading m unknowns of A (right-hand side in column m): warp 0 takes
// the next diagonal block (update, factorisation) while the others share the
// trailing tiles; then all threads form the next panel's L21.  rpiv: m reciprocal
// pivots; stage: 64 doubles.
template <int NT>
__device__ __forceinline__ void factor_fp32(float* A, int ldA, int m, double* rpiv, double* stage, int* flag) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp == 0) factor_diag(A, ldA, m, 0, rpiv, lane, flag);
    __syncthreads();
    solve_l21(A, ldA, m, 0, rpiv, min(kPanel, m), tid, NT);
    __syncthreads();
#pragma unroll 1
    for (int k0 = 0; k0 < m; k0 += kPanel) {
        const int kb = min(kPanel, m - k0);
        const int r0 = k0 + kb;
        const int nct = (m + 1 - r0 + 7) / 8;  // column tiles of [r0, m], rhs included
        const int top = min(r0 + kPanel, m);   // rows of the next diagonal block
        if (warp == 0) {
            update_tile<kU12ToStage>(A, ldA, m, k0, kb, r0, r0, top, stage, lane);
            if (r0 < m) {
                __syncwarp();
                factor_diag(A, ldA, m, r0, rpiv, lane, flag);
            }
        } else {
            // unit 0: tile 0 below the next diagonal block; unit u >= 1: tile u
#pragma unroll 1
            for (int u = warp - 1; u < nct; u += NW - 1) {
                if (u == 0) {
                    if (top < m) update_tile<kU12InRegs>(A, ldA, m, k0, kb, r0, top, m, nullptr, lane);
                } else {
                    update_tile<kU12InPlace>(A, ldA, m, k0, kb, r0 + 8 * u, r0, m, nullptr, lane);
                }
            }
        }
        __syncthreads();
        if (tid < 64) {  // tile 0 of U12 (rows k0+1 .. k0+kb-1) from the stage
            const int j = tid >> 3, c = r0 + (tid & 7);
            if (j >= 1 && j < kb && c <= m) A[(k0 + j) * ldA + c] = static_cast<float>(stage[tid]);
        }
        if (top < m) solve_l21(A, ldA, m, r0, rpiv, top, tid, NT);
        __syncthreads();
    }
}

// ---- register-resident Gauss-Jordan solve of the free block ----------------------
// The free block A[0:m][0:m] and its right-hand-side columns are spread over a
// (NT/16) x 16 grid of threads: thread (ri, cj) = (tid / 16, tid % 16) keeps the
// entries (ri + a*(NT/16), cj + 16*b), a < RT, b < CT, in registers (cyclic in
// both directions, so every thread keeps work until the last pivot).  Each
// pivot step is one CTA barrier: every thread reads the pivot column and row
// from a double-buffered shared-memory slot, forms the reciprocal pivot itself
// and updates its entries; the owners of the next pivot's column and row
// publish them into the other slot.  No single warp runs a serial panel, and
// the triangular solves of an LU disappear (Gauss-Jordan eliminates above the
// pivot as well), so the chain is m steps of ~one barrier each.
// Tile sizes per (type, threads): the registers a thread can spend on the block
// within its launch budget.  Blocks that do not fit are eliminated in shared memory.
template <typename TR, int NT>
struct GJTile;
template <> struct GJTile<double, 128> { static constexpr int RT = 7, CT = 4; };
template <> struct GJTile<double, 256> { static constexpr int RT = 6, CT = 6; };
template <> struct GJTile<double, 512> { static constexpr int RT = 4, CT = 8; };
template <> struct GJTile<float, 128> { static constexpr int RT = 8, CT = 5; };
template <> struct GJTile<float, 256> { static constexpr int RT = 8, CT = 8; };
template <> struct GJTile<float, 512> { static constexpr int RT = 4, CT = 8; };

constexpr int kGJCols = 16;  // column groups of the register grid
// Largest backward error an FP64 Gauss-Jordan solve may leave (rounding gives
// ~n eps); above it the unpivoted elimination has lost accuracy to growth.
constexpr double kGJBackwardErrorMax = 1e-10;

template <typename TR, int NT>
__host__ __device__ constexpr int gj_slot() {
    return 2 * (GJTile<TR, NT>::RT * (NT / kGJCols) + GJTile<TR, NT>::CT * kGJCols);
}
static_assert(gj_rows(8, 128) == GJTile<double, 128>::RT * 8 && gj_rows(8, 256) == GJTile<double, 256>::RT * 16 &&
                  gj_rows(8, 512) == GJTile<double, 512>::RT * 32 && gj_rows(4, 128) == GJTile<float, 128>::RT * 8 &&
                  gj_rows(4, 256) == GJTile<float, 256>::RT * 16 && gj_rows(4, 512) == GJTile<float, 512>::RT * 32,
              "gj_rows must follow GJTile");
static_assert(gj_slot<double, 128>() == gj_slot_entries(8, 128) &&
                  gj_slot<double, 256>() == gj_slot_entries(8, 256) &&
                  gj_slot<double, 512>() == gj_slot_entries(8, 512) &&
                  gj_slot<float, 128>() == gj_slot_entries(4, 128) &&
                  gj_slot<float, 256>() == gj_slot_entries(4, 256) &&
                  gj_slot<float, 512>() == gj_slot_entries(4, 512),
              "gj_slot_entries must follow GJTile");

// Whether the free block (m rows, m + nrhs columns; INV: m x m) fits the grid.
template <typename TR, int NT>
__host__ __device__ inline bool gj_fits(int m, int ncols) {
    return m <= GJTile<TR, NT>::RT * (NT / kGJCols) && ncols <= GJTile<TR, NT>::CT * kGJCols;
}

// Pair of TR values for vectorised shared-memory access.
template <typename TR> struct Pair2;
template <> struct Pair2<double> { using type = double2; };
template <> struct Pair2<float> { using type = float2; };

// Rank-2 update R[a][b] -= x0[a] u0[b] + x1[a] u1[b] of the column blocks
// b >= b0 (one uniform test per column block, none per entry: padding rows and
// columns hold zeros, so their updates change nothing).  (u0, u1) of column
// block b is read from the pivot pair's row buffer `rp` (pairs per column).
template <int B, typename TR, int RT, int CT>
__device__ __forceinline__ void gj_rank2_from(TR (&R)[RT][CT], const TR (&x0)[RT], const TR (&x1)[RT],
                                              const TR* rp, int b0) {
    using P2 = typename Pair2<TR>::type;
    if constexpr (B < CT) {
        if (B >= b0) {
            const P2 w = *reinterpret_cast<const P2*>(rp + 2 * B * kGJCols);
#pragma unroll
            for (int a = 0; a < RT; ++a) R[a][B] = fma(-x1[a], w.y, fma(-x0[a], w.x, R[a][B]));
        }
        gj_rank2_from<B + 1>(R, x0, x1, rp, b0);
    }
}

// Row a of R (a chosen at run time, the same in the whole warp) becomes
// p u0 + q u1 in the column blocks b >= b0, (u0, u1) from the row buffer `rp`.
template <typename TR, int RT, int CT>
__device__ __forceinline__ void gj_set_row(TR (&R)[RT][CT], int a_sel, TR p, TR q, const TR* rp, int b0) {
    using P2 = typename Pair2<TR>::type;
#pragma unroll
    for (int a = 0; a < RT; ++a)
        if (a == a_sel) {
#pragma unroll
            for (int b = 0; b < CT; ++b)
                if (b >= b0) {
                    const P2 w = *reinterpret_cast<const P2*>(rp + 2 * b * kGJCols);
                    R[a][b] = fma(p, w.x, q * w.y);
                }
        }
}

// Gauss-Jordan elimination without pivoting of the free block, held in R, two
// pivots per step (2x2 pivot blocks D, inverted through their determinant), so
// one CTA barrier serves two pivots.  Rows of a pivot pair are normalised
// (D^-1 applied), so on exit the block is the identity:
//   INV = false (solve): columns [0, m + nrhs) are loaded (only column blocks
//     that still hold a column right of the pair are updated); on exit column
//     m + r of row i holds x_i.
//   INV = true (inverse): columns [0, m) are loaded and replaced in place by
//     the inverse (pivot rows D^-1 A_K, pivot columns -A_iK D^-1, pivot block
//     D^-1).
// m must be even (free blocks are 6 per node).  buf: 2 slots of
// gj_slot<TR, NT>() entries in shared memory: the pivot pair's two columns,
// paired per row, then its two rows, paired per column; D is the pair of the
// pivot rows.  Every thread forms D^-1 and its rows' multipliers itself; the
// pivot rows' own update (multipliers ~ identity) is overwritten by their
// normalisation.  The pivot pair's block indices are the same in every
// thread, so the owners of the pivot rows and columns branch on them
// (warp-uniform) instead of selecting among their registers.  A zero or
// non-finite determinant sets bit 2 of *flag.
template <typename TR, int NT, bool INV>
__device__ __forceinline__ void gj_eliminate(const TR* A, int ldA, int m, int nrhs, TR* buf, int* flag,
                                             TR (&R)[GJTile<TR, NT>::RT][GJTile<TR, NT>::CT]) {
    using P2 = typename Pair2<TR>::type;
    constexpr int RT = GJTile<TR, NT>::RT, CT = GJTile<TR, NT>::CT;
    constexpr int PR = NT / kGJCols, PC = kGJCols;
    constexpr int SLOT = gj_slot<TR, NT>();
    constexpr int ROWS = 2 * RT * PR;
    const int tid = threadIdx.x, ri = tid / PC, cj = tid % PC;
    const int ncols = INV ? m : m + nrhs;
#pragma unroll
    for (int a = 0; a < RT; ++a) {
        const int i = ri + a * PR;
#pragma unroll
        for (int b = 0; b < CT; ++b) {
            const int j = cj + b * PC;
            R[a][b] = (i < m && j < ncols) ? A[sys_at<TR>(ldA, i, j)] : TR(0);
        }
    }
    // slot 0: columns 0, 1 and rows 0, 1; padding of both slots stays zero
    for (int t = tid; t < 2 * SLOT; t += NT) {
        const int e = t % SLOT;
        TR v = TR(0);
        if (t < SLOT) {
            if (e < ROWS) {
                const int i = e >> 1, h = e & 1;
                v = (i < m) ? A[sys_at<TR>(ldA, i, h)] : TR(0);
            } else {
                const int j = (e - ROWS) >> 1, h = (e - ROWS) & 1;
                v = (j < ncols) ? A[sys_at<TR>(ldA, h, j)] : TR(0);
            }
        }
        buf[t] = v;
    }
    __syncthreads();
    for (int k = 0; k < m; k += 2) {
        const TR* cb = buf + ((k >> 1) & 1) * SLOT;
        TR* nb = buf + (((k >> 1) + 1) & 1) * SLOT;
        const P2 dA = *reinterpret_cast<const P2*>(cb + 2 * k);
        const P2 dB = *reinterpret_cast<const P2*>(cb + 2 * k + 2);
        const TR det = fma(dA.x, dB.y, -(dA.y * dB.x));
        const TR rd = pivot_rcp(det);
        if (tid == 0 && (!(fabs(det) > TR(0)) || !isfinite(rd))) atomicOr(flag, 2);
        const TR i00 = dB.y * rd, i01 = -dA.y * rd, i10 = -dB.x * rd, i11 = dA.x * rd;
        TR x0[RT], x1[RT];
#pragma unroll
        for (int a = 0; a < RT; ++a) {
            const P2 c = *reinterpret_cast<const P2*>(cb + 2 * (ri + a * PR));
            x0[a] = fma(c.x, i00, c.y * i10);
            x1[a] = fma(c.x, i01, c.y * i11);
        }
        const TR* rp = cb + ROWS + 2 * cj;  // this thread's columns in the row pair
        // solve form: column blocks left of b0 hold only eliminated columns
        const int b0 = INV ? 0 : (k + 2) / PC;
        gj_rank2_from<0>(R, x0, x1, rp, b0);
        // the pivot rows: D^-1 [row k; row k+1]
        const int ak = k / PR;
        const bool r0 = ri == k % PR, r1 = ri == (k + 1) % PR;
        if (r0 || r1) gj_set_row(R, ak, r0 ? i00 : i10, r0 ? i01 : i11, rp, b0);
        if (INV) {  // the pivot columns: -A_iK D^-1, and D^-1 in the pivot rows
            const int bk = k / PC;
            const bool c0 = cj == k % PC, c1 = cj == (k + 1) % PC;
            if (c0 || c1) {
#pragma unroll
                for (int b = 0; b < CT; ++b)
                    if (b == bk) {
#pragma unroll
                        for (int a = 0; a < RT; ++a) {
                            TR v = c0 ? -x0[a] : -x1[a];
                            if (a == ak && r0) v = c0 ? i00 : i01;
                            if (a == ak && r1) v = c0 ? i10 : i11;
                            R[a][b] = v;
                        }
                    }
            }
        }
        // publish the next pair's columns and rows
        const int kn = k + 2;
        if (kn < m) {
            const int an = kn / PR, bn = kn / PC;
            const bool c0 = cj == kn % PC, c1 = cj == (kn + 1) % PC;
            if (c0 || c1) {
                TR* dst = nb + 2 * ri + (c0 ? 0 : 1);
#pragma unroll
                for (int b = 0; b < CT; ++b)
                    if (b == bn) {
#pragma unroll
                        for (int a = 0; a < RT; ++a) dst[2 * a * PR] = R[a][b];
                    }
            }
            const bool w0 = ri == kn % PR, w1 = ri == (kn + 1) % PR;
            if (w0 || w1) {
                TR* dst = nb + ROWS + 2 * cj + (w0 ? 0 : 1);
#pragma unroll
                for (int a = 0; a < RT; ++a)
                    if (a == an) {
#pragma unroll
                        for (int b = 0; b < CT; ++b) dst[2 * b * PC] = R[a][b];
                    }
            }
        }
        __syncthreads();
    }
}

// Gauss-Jordan with row pivoting on the same grid, one right-hand side in
// column m: the solve of a block whose unpivoted elimination lost accuracy to
// element growth (seen in steps that do not converge, so its three barriers per
// pivot matter little).  Rows stay in place; the pivot of column k is the
// largest entry of the rows not yet used.  x to out[0:m].  buf: two rows of the
// grid's extent and two of its integers.
template <typename TR, int NT>
__device__ __noinline__ void gj_solve_pivoted(const TR* A, int ldA, int m, TR* buf, double* out, int* flag) {
    constexpr int RT = GJTile<TR, NT>::RT, CT = GJTile<TR, NT>::CT;
    constexpr int PR = NT / kGJCols, PC = kGJCols;
    const int tid = threadIdx.x, lane = tid & 31, ri = tid / PC, cj = tid % PC;
    TR* col = buf;                   // [RT * PR]
    TR* row = col + RT * PR;         // [CT * PC]
    int* used = reinterpret_cast<int*>(row + CT * PC);  // [RT * PR]
    int* pivot = used + RT * PR;     // [RT * PR] row that solved column k
    TR R[RT][CT];
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
        for (int b = 0; b < CT; ++b) {
            const int i = ri + a * PR, j = cj + b * PC;
            R[a][b] = (i < m && j <= m) ? A[sys_at<TR>(ldA, i, j)] : TR(0);
        }
    for (int i = tid; i < RT * PR; i += NT) used[i] = i < m ? 0 : 1;
    for (int k = 0; k < m; ++k) {
        if (cj == k % PC) {
#pragma unroll
            for (int b = 0; b < CT; ++b)
                if (b == k / PC) {
#pragma unroll
                    for (int a = 0; a < RT; ++a) col[ri + a * PR] = R[a][b];
                }
        }
        __syncthreads();
        TR best = TR(-1);
        int p = 0;
        for (int i = lane; i < m; i += 32)
            if (!used[i] && fabs(col[i]) > best) {
                best = fabs(col[i]);
                p = i;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const TR ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int op = __shfl_xor_sync(0xffffffffu, p, o);
            if (ob > best || (ob == best && op < p)) {
                best = ob;
                p = op;
            }
        }
        if (ri == p % PR) {
#pragma unroll
            for (int a = 0; a < RT; ++a)
                if (a == p / PR) {
#pragma unroll
                    for (int b = 0; b < CT; ++b) row[cj + b * PC] = R[a][b];
                }
        }
        if (tid == 0 && !(best > TR(0))) atomicOr(flag, 2);
        __syncthreads();
        const TR rd = TR(1) / row[k];
        if (tid == 0) {
            used[p] = 1;
            pivot[k] = p;
        }
#pragma unroll
        for (int a = 0; a < RT; ++a) {
            const int i = ri + a * PR;
            const TR l = col[i] * rd;
#pragma unroll
            for (int b = 0; b < CT; ++b) {
                const TR w = row[cj + b * PC];
                R[a][b] = i == p ? w * rd : R[a][b] - l * w;
            }
        }
        __syncthreads();
    }
    if (cj == m % PC) {
#pragma unroll
        for (int b = 0; b < CT; ++b)
            if (b == m / PC) {
#pragma unroll
                for (int a = 0; a < RT; ++a) col[ri + a * PR] = R[a][b];
            }
    }
    __syncthreads();
    for (int k = tid; k < m; k += NT) out[k] = static_cast<double>(col[pivot[k]]);
    __syncthreads();
}

// Column `col` (col >= m) of the register grid after the solve form: the
// solution for that right-hand side, into out[0:m].
template <typename TR, int NT, typename Out>
__device__ __forceinline__ void gj_extract(const TR (&R)[GJTile<TR, NT>::RT][GJTile<TR, NT>::CT], int m,
                                           int col, Out* out) {
    constexpr int RT = GJTile<TR, NT>::RT, CT = GJTile<TR, NT>::CT;
    constexpr int PR = NT / kGJCols, PC = kGJCols;
    const int tid = threadIdx.x, ri = tid / PC, cj = tid % PC;
    if (cj != col % PC) return;
    const int bc = col / PC;
#pragma unroll
    for (int b = 0; b < CT; ++b)
        if (b == bc) {
#pragma unroll
            for (int a = 0; a < RT; ++a) {
                const int i = ri + a * PR;
                if (i < m) out[i] = static_cast<Out>(R[a][b]);
            }
        }
}

// y = M v for the free block, with M either the register grid (from_regs) or
// the block in shared memory (A, FP64 accumulation in both); v, y in FP64
// shared memory.  With `bvec`, y = bvec - M v and amax gets max |y| (lane 0 of
// each row group, reduced by the caller).  The 16 threads of a row group sit
// in one half-warp and sum their columns by shuffles.
template <typename TR, int NT, bool from_regs>
__device__ __forceinline__ void gj_matvec(const TR (&R)[GJTile<TR, NT>::RT][GJTile<TR, NT>::CT], const TR* A,
                                          int ldA, int m, const double* v, const double* bvec, double* y,
                                          double& amax) {
    constexpr int RT = GJTile<TR, NT>::RT, CT = GJTile<TR, NT>::CT;
    constexpr int PR = NT / kGJCols, PC = kGJCols;
    const int tid = threadIdx.x, ri = tid / PC, cj = tid % PC;
    amax = 0.;
#pragma unroll
    for (int a = 0; a < RT; ++a) {
        const int i = ri + a * PR;
        if (a * PR >= m) break;  // uniform: no row of this block is in range
        double acc = 0.;
#pragma unroll
        for (int b = 0; b < CT; ++b) {
            const int j = cj + b * PC;
            if (j < m && i < m) {
                const double mij = from_regs ? static_cast<double>(R[a][b])
                                             : static_cast<double>(A[sys_at<TR>(ldA, i, j)]);
                acc = fma(mij, v[j], acc);
            }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (cj == 0 && i < m) {
            const double val = bvec ? bvec[i] - acc : acc;
            y[i] = val;
            amax = fmax(amax, fabs(val));
        }
    }
}

// Residual, gradient blocks and G^T lambda of one constraint on node q `nu`
// (calculate_constraint_residual_gradient.hpp:60-320 and :468-540 with
// calculate_{fixed,prescribed}_bc_constraint.hpp,
// calculate_rigid_joint_constraint.hpp:17-113 and
// calculate_rotation_control_constraint.hpp:17-144).  FixedBC: R1 = I, u1 = 0;
// PrescribedBC: (u1, R1) = the record's input; joints: (u1, R1) = the hub
// node's q `hq`, X0 = target x0 - hub x0, and the base-node blocks
// tilde(R1 X0) T_hub and -AX(C) T_hub are kept for the hub elimination.
// RotationControl puts the commanded rotation Rc = exp(angle * axis) (angle =
// input[0]) between the target and the hub: C = R(R2 Rc^-1 R1^-1).
static __device__ __noinline__ void constraint_record(double* cr, int type, const double* nu, const double* X0,
                                         const double* Rt, const double* hq, const double* RtHub,
                                         const double* axis) {
    double u1[3] = {0., 0., 0.}, R1[4] = {1., 0., 0., 0.};
    if (type == KYN_CONSTRAINT_PRESCRIBED_BC) {
        for (int k = 0; k < 3; ++k) u1[k] = cr[conrec::inp + k];
        for (int k = 0; k < 4; ++k) R1[k] = cr[conrec::inp + 3 + k];
    } else if (is_hub_joint(type)) {
        for (int k = 0; k < 3; ++k) u1[k] = hq[k];
        for (int k = 0; k < 4; ++k) R1[k] = hq[3 + k];
    }
    const double len = sqrt(R1[0] * R1[0] + R1[1] * R1[1] + R1[2] * R1[2] + R1[3] * R1[3]);
    const double R1t[4] = {R1[0] / len, -R1[1] / len, -R1[2] / len, -R1[3] / len};
    double R1X0[3];
    for (int i = 0; i < 3; ++i) {
        R1X0[i] = 0.;
        for (int j = 0; j < 3; ++j) R1X0[i] += rot_entry(R1, i, j) * X0[j];
    }
    for (int i = 0; i < 3; ++i) cr[conrec::Phi + i] = nu[i] + X0[i] - u1[i] - R1X0[i];
    double R2R1t[4];
    if (type == KYN_CONSTRAINT_ROTATION_CONTROL) {
        // quaternion of the rotation vector axis*angle (quaternion_operations.hpp:231-242)
        const double ang = cr[conrec::inp];
        const double rv[3] = {axis[0] * ang, axis[1] * ang, axis[2] * ang};
        const double th = sqrt(rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
        const double fac = (fabs(th) < 1e-12) ? 0. : sin(th / 2.) / th;
        const double Rc[4] = {cos(th / 2.), rv[0] * fac, rv[1] * fac, rv[2] * fac};
        const double lc = sqrt(Rc[0] * Rc[0] + Rc[1] * Rc[1] + Rc[2] * Rc[2] + Rc[3] * Rc[3]);
        const double Rct[4] = {Rc[0] / lc, -Rc[1] / lc, -Rc[2] / lc, -Rc[3] / lc};
        double R2Rct[4];
        quat_compose(nu + 3, Rct, R2Rct);
        quat_compose(R2Rct, R1t, R2R1t);
    } else {
        quat_compose(nu + 3, R1t, R2R1t);
    }
    double C[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) C[e] = rot_entry(R2R1t, e / 3, e % 3);
    cr[conrec::Phi + 3] = (C[7] - C[5]) / 2.;
    cr[conrec::Phi + 4] = (C[2] - C[6]) / 2.;
    cr[conrec::Phi + 5] = (C[3] - C[1]) / 2.;
    // AX(C) = tr(C)/2 I - C/2 ; grad rotational block = AX^T ; grad^T block = AX
    const double tr = (C[0] + C[4] + C[8]) / 2.;
    double AXm[9];
    for (int e = 0; e < 9; ++e) AXm[e] = -C[e] / 2. + ((e % 4 == 0) ? tr : 0.);
    for (int e = 0; e < 9; ++e) cr[conrec::AX + e] = AXm[e];
    // B rotational block = AX^T * Rt  (Rt = stored tangent block of the node)
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            double acc = 0.;
            for (int k = 0; k < 3; ++k) acc += AXm[k * 3 + i] * Rt[k * 3 + j];
            cr[conrec::Brot + i * 3 + j] = acc;
        }
    // grad^T lambda
    for (int i = 0; i < 3; ++i) cr[conrec::Gl + i] = cr[conrec::lam + i];
    for (int i = 0; i < 3; ++i) {
        double acc = 0.;
        for (int k = 0; k < 3; ++k) acc += AXm[i * 3 + k] * cr[conrec::lam + 3 + k];
        cr[conrec::Gl + 3 + i] = acc;
    }
    if (is_hub_joint(type)) {
        for (int i = 0; i < 3; ++i) cr[conrec::R1X0 + i] = R1X0[i];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                double bt = 0., br = 0.;
                for (int k = 0; k < 3; ++k) {
                    bt += tilde_e(R1X0, i, k) * RtHub[k * 3 + j];
                    br -= AXm[i * 3 + k] * RtHub[k * 3 + j];
                }
                cr[conrec::Btr + i * 3 + j] = bt;
                cr[conrec::Brr + i * 3 + j] = br;
            }
    }
}

// G_base^T w of a rigid joint (base gradient [-I, tilde(R1 X0); 0, -AX]):
// [-w_t; tilde(R1 X0)^T w_t - AX^T w_r], accumulated into out.
__device__ inline void joint_base_transpose_add(const double* cr, const double* w, double* out) {
    const double* r = cr + conrec::R1X0;
    const double* AX = cr + conrec::AX;
    for (int i = 0; i < 3; ++i) out[i] -= w[i];
    for (int i = 0; i < 3; ++i) {
        double acc = 0.;
        for (int k = 0; k < 3; ++k) acc += tilde_e(r, k, i) * w[k] - AX[k * 3 + i] * w[3 + k];
        out[3 + i] += acc;
    }
}

// ---- drive train: revolute joint between hub-chain records 0 and 1 -------------------
// Residual, gradient rows and G^T lambda of the revolute joint
// (calculate_revolute_joint_constraint.hpp:19-113, calculate_revolute_joint_force.hpp:19-45,
// branch :388-465 of calculate_constraint_residual_gradient.hpp).  Rows 0-2:
// u2 + X0 - u1 - R1 X0 with gradients I (target) and -I (base); rows 3-4:
// (R2 z0).(R1 x0) and (R2 y0).(R1 x0) with gradients -(x cross z), -(x cross y)
// on the target's rotation and +(x cross z), +(x cross y) on the base's.
// `b` and `t` are hub-chain records (state at hubrec offsets).
__device__ inline void revolute_record(double* rr, const double* b, const double* t) {
    const double* X0 = t + hubrec::X0;
    const double* ax = t + hubrec::axes;
    const double* bq = b + hubrec::q;
    const double* tq = t + hubrec::q;
    double R1X0[3], x[3], y[3], z[3], ta[3];
    for (int i = 0; i < 3; ++i) {
        R1X0[i] = x[i] = y[i] = z[i] = ta[i] = 0.;
        for (int j = 0; j < 3; ++j) {
            R1X0[i] += rot_entry(bq + 3, i, j) * X0[j];
            x[i] += rot_entry(bq + 3, i, j) * ax[j];
            y[i] += rot_entry(tq + 3, i, j) * ax[3 + j];
            z[i] += rot_entry(tq + 3, i, j) * ax[6 + j];
            ta[i] += rot_entry(tq + 3, i, j) * ax[j];
        }
    }
    for (int i = 0; i < 3; ++i) rr[revrec::Phi + i] = tq[i] + X0[i] - bq[i] - R1X0[i];
    rr[revrec::Phi + 3] = z[0] * x[0] + z[1] * x[1] + z[2] * x[2];
    rr[revrec::Phi + 4] = y[0] * x[0] + y[1] * x[1] + y[2] * x[2];
    const double xcz[3] = {x[1] * z[2] - x[2] * z[1], x[2] * z[0] - x[0] * z[2], x[0] * z[1] - x[1] * z[0]};
    const double xcy[3] = {x[1] * y[2] - x[2] * y[1], x[2] * y[0] - x[0] * y[2], x[0] * y[1] - x[1] * y[0]};
    for (int i = 0; i < 3; ++i) {
        rr[revrec::x + i] = x[i];
        rr[revrec::y + i] = y[i];
        rr[revrec::z + i] = z[i];
        rr[revrec::xcz + i] = xcz[i];
        rr[revrec::xcy + i] = xcy[i];
        rr[revrec::sys + i] = ta[i] * t[hubrec::input];
    }
    // B = G T on the rotational columns (stored tangent blocks, row-major)
    const double* Tt = t + hubrec::tangent;
    const double* Tb = b + hubrec::tangent;
    for (int j = 0; j < 3; ++j) {
        double a0 = 0., a1 = 0., b0 = 0., b1 = 0.;
        for (int k = 0; k < 3; ++k) {
            a0 -= xcz[k] * Tt[k * 3 + j];
            a1 -= xcy[k] * Tt[k * 3 + j];
            b0 += xcz[k] * Tb[k * 3 + j];
            b1 += xcy[k] * Tb[k * 3 + j];
        }
        rr[revrec::Bt + j] = a0;
        rr[revrec::Bt + 3 + j] = a1;
        rr[revrec::Bb + j] = b0;
        rr[revrec::Bb + 3 + j] = b1;
    }
    const double* l = rr + revrec::lam;
    for (int i = 0; i < 3; ++i) {
        rr[revrec::GtL + i] = l[i];
        rr[revrec::GbL + i] = -l[i];
        rr[revrec::GtL + 3 + i] = -xcz[i] * l[3] - xcy[i] * l[4];
        rr[revrec::GbL + 3 + i] = xcz[i] * l[3] + xcy[i] * l[4];
    }
}

// Target correction of a six-row joint (constraint record cr, base blocks
// Btr/Brr, target block Brot) from its base correction xb: B_t x = -s Phi -
// B_base xb, with s = 1 for the correction and 0 for its part per unit shaft
// rotation.
__device__ inline bool joint_target_correction(const double* cr, const double* xb, double s, double* x) {
    double rr[3];
    for (int i = 0; i < 3; ++i) {
        x[i] = -s * cr[conrec::Phi + i] + xb[i];
        rr[i] = -s * cr[conrec::Phi + 3 + i];
        for (int k = 0; k < 3; ++k) {
            x[i] -= cr[conrec::Btr + i * 3 + k] * xb[3 + k];
            rr[i] -= cr[conrec::Brr + i * 3 + k] * xb[3 + k];
        }
    }
    return solve3(cr + conrec::Brot, rr, x + 3);
}

// Target test vector of a six-row joint from its base test vector: G_t w =
// -G_base wb with the gradients (not B = G T): G_t = [I 0; 0 AX^T],
// G_base = [-I tilde(R1 X0); 0 -AX].
__device__ inline bool joint_target_test(const double* cr, const double* wb, double* w) {
    const double* r = cr + conrec::R1X0;
    const double* AX = cr + conrec::AX;
    double rhs[3], AXt[9];
    for (int i = 0; i < 3; ++i) {
        w[i] = wb[i];
        rhs[i] = 0.;
        for (int k = 0; k < 3; ++k) {
            w[i] -= tilde_e(r, i, k) * wb[3 + k];
            rhs[i] += AX[i * 3 + k] * wb[3 + k];
            AXt[i * 3 + k] = AX[k * 3 + i];
        }
    }
    return solve3(AXt, rhs, w + 3);
}

// ---- point masses and springs at the nodes of one CTA's system ---------------------
// Adds, for local node n, the terms of every point mass at n
// (src/system/masses/calculate_quadrature_point_values.hpp:40-152: residual
// Fi - Fg, block b'Muu + g'Guu + Kuu T) and of every spring with an end at n
// (src/system/springs/calculate_quadrature_point_values.hpp:27-92: residual
// +-f, translational blocks +-a) to resid[n] and to node n's block row of A
// (scaled by the conditioner).  One thread per node: each writes only its own
// rows, and takes its elements in element order.
// Node n's rows and columns start at pos_mul * pos[n] (6 x the node's position
// in a beam system; the first-DOF map itself in a dense model).
template <typename At>
__device__ void add_lumped_terms(int n, const double* __restrict__ rec, int n_mass, int n_spring,
                                 const double* sq, const double* sv, const double* svd,
                                 const double* sT, const double* grav, double bprime,
                                 double gprime, double cond, const int* pos, At at,
                                 double* resid, int pos_mul = 6) {
    const int cn = pos_mul * pos[n];
    auto add = [&](int r, int c, double val) {
        auto& a = at(cn + r, c);
        a = static_cast<std::remove_reference_t<decltype(a)>>(static_cast<double>(a) + val);
    };
    for (int e = 0; e < n_mass; ++e) {
        const double* mr = rec + e * kMassRec;
        if (static_cast<int>(mr[0]) != n) continue;
        const double* ms = mr + 1;
        // Muu = diag(R, R) M* diag(R, R)^T, R = R(r o r0)
        double xr[4], R[9];
        quat_compose(sq + n * 7 + 3, mr + 37, xr);
        for (int e9 = 0; e9 < 9; ++e9) R[e9] = rot_entry(xr, e9 / 3, e9 % 3);
        double Mu[36];
        for (int bi = 0; bi < 2; ++bi)
            for (int bj = 0; bj < 2; ++bj)
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; j < 3; ++j) {
                        double acc = 0.;
                        for (int k = 0; k < 3; ++k) {
                            double t = 0.;
                            for (int l = 0; l < 3; ++l) t += ms[(3 * bi + k) * 6 + 3 * bj + l] * R[j * 3 + l];
                            acc += R[i * 3 + k] * t;
                        }
                        Mu[(3 * bi + i) * 6 + 3 * bj + j] = acc;
                    }
        const double mass = Mu[0];
        const double eta[3] = {Mu[5 * 6 + 1] / mass, -Mu[5 * 6 + 0] / mass, Mu[4 * 6 + 0] / mass};
        double rho[9];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) rho[i * 3 + j] = Mu[(3 + i) * 6 + 3 + j];
        const double* ud = svd + n * 6;       // u_ddot = vd[0:3], omega_dot = vd[3:6]
        const double* od = svd + n * 6 + 3;
        const double* om = sv + n * 6 + 3;
        const double me[3] = {mass * eta[0], mass * eta[1], mass * eta[2]};
        auto mat3 = [](const double* a, const double* b, int i, int j) {
            return a[i * 3] * b[j] + a[i * 3 + 1] * b[3 + j] + a[i * 3 + 2] * b[6 + j];
        };
        double omt[9], odt[9], met[9], udt[9];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                omt[i * 3 + j] = tilde_e(om, i, j);
                odt[i * 3 + j] = tilde_e(od, i, j);
                met[i * 3 + j] = tilde_e(me, i, j);
                udt[i * 3 + j] = tilde_e(ud, i, j);
            }
        double oo[9], orho[9];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                oo[i * 3 + j] = mat3(omt, omt, i, j);
                orho[i * 3 + j] = mat3(omt, rho, i, j);
            }
        // inertial force (calculate_inertial_force.hpp) minus gravity (calculate_gravity_force.hpp)
        double r6[6];
        for (int i = 0; i < 3; ++i) {
            double acc = 0.;
            for (int k = 0; k < 3; ++k) acc += (mass * oo[i * 3 + k] + mass * odt[i * 3 + k]) * eta[k];
            r6[i] = acc + mass * ud[i] - mass * grav[i];
        }
        for (int i = 0; i < 3; ++i) {
            double acc = 0.;
            for (int k = 0; k < 3; ++k)
                acc += tilde_e(eta, i, k) * (mass * ud[k]) + rho[i * 3 + k] * od[k] + orho[i * 3 + k] * om[k] -
                       tilde_e(eta, i, k) * (mass * grav[k]);
            r6[3 + i] = acc;
        }
        for (int c = 0; c < 6; ++c) resid[n * 6 + c] += r6[c];
        // Guu (calculate_gyroscopic_matrix.hpp) and Kuu (calculate_inertia_stiffness_matrix.hpp):
        // both are zero outside the columns 3..5
        double wm[3], rw[3], rwd[3];
        for (int i = 0; i < 3; ++i) {
            wm[i] = omt[i * 3] * me[0] + omt[i * 3 + 1] * me[1] + omt[i * 3 + 2] * me[2];
            rw[i] = rho[i * 3] * om[0] + rho[i * 3 + 1] * om[1] + rho[i * 3 + 2] * om[2];
            rwd[i] = rho[i * 3] * od[0] + rho[i * 3 + 1] * od[1] + rho[i * 3 + 2] * od[2];
        }
        double G12[9], G22[9], K12[9], K22[9], M1[9];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) M1[i * 3 + j] = mat3(rho, omt, i, j) - tilde_e(rw, i, j);
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                double a12 = tilde_e(wm, j, i), k12 = 0., k22 = 0.;
                for (int k = 0; k < 3; ++k) {
                    a12 += omt[i * 3 + k] * met[j * 3 + k];
                    k12 += (odt[i * 3 + k] + oo[i * 3 + k]) * met[j * 3 + k];
                    k22 += rho[i * 3 + k] * odt[k * 3 + j] + udt[i * 3 + k] * met[k * 3 + j] +
                           omt[i * 3 + k] * M1[k * 3 + j];
                }
                G12[i * 3 + j] = a12;
                G22[i * 3 + j] = orho[i * 3 + j] - tilde_e(rw, i, j);
                K12[i * 3 + j] = k12;
                K22[i * 3 + j] = k22 - tilde_e(rwd, i, j);
            }
        // block b'Muu + g'Guu + Kuu T (T = I on the translational block)
        const double* Tn = sT + n * 9;
        for (int r = 0; r < 6; ++r) {
            for (int c = 0; c < 6; ++c) {
                double val = bprime * Mu[r * 6 + c];
                if (c >= 3) {
                    const int cc = c - 3;
                    const double* G = r < 3 ? G12 + r * 3 : G22 + (r - 3) * 3;
                    const double* K = r < 3 ? K12 + r * 3 : K22 + (r - 3) * 3;
                    val += gprime * G[cc];
                    val += K[0] * Tn[cc] + K[1] * Tn[3 + cc] + K[2] * Tn[6 + cc];
                }
                add(r, cn + c, val * cond);
            }
        }
    }
    const double* srec = rec + n_mass * kMassRec;
    for (int e = 0; e < n_spring; ++e) {
        const double* sp = srec + e * kSpringRec;
        const int n1 = static_cast<int>(sp[0]), n2 = static_cast<int>(sp[1]);
        if (n1 != n && n2 != n) continue;
        double r[3];
        for (int c = 0; c < 3; ++c) r[c] = sp[2 + c] + sq[n2 * 7 + c] - sq[n1 * 7 + c];
        const double l = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
        const double lref = sp[5], k = sp[6];
        const double c1 = k * (lref / l - 1.);
        const double c2 = k * lref / (l * l * l);
        const double sgn = (n == n1) ? 1. : -1.;
        for (int c = 0; c < 3; ++c) resid[n * 6 + c] += sgn * (c1 * r[c]);
        const int other = (n == n1) ? n2 : n1;
        const int co = pos_mul * pos[other];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                double rr = 0.;
                for (int t = 0; t < 3; ++t) rr += tilde_e(r, i, t) * tilde_e(r, t, j);
                const double a = ((i == j) ? c1 - c2 * l * l : 0.) - c2 * rr;
                add(i, cn + j, a * cond);
                add(i, co + j, -a * cond);
            }
    }
}

// ---- dense models: masses, springs and constraints of any row count ---------------
// A model without beam elements whose constraints are not all single-node
// six-DOF BCs (three-row constraints on position-only nodes, joints between
// its nodes) runs the reference's own bordered system in one CTA: nodes carry
// the DOFs of their freedom signature (six, or three for position-only nodes),
// constraint rows follow, and the system is solved by LU with partial
// pivoting (src/step/step.hpp:42-124 with solve_system.hpp; the order of
// operations of the dense solve follows the row-pivoting Doolittle LU).  FP64
// in both precision forms: these systems have at most kDenseModelMaxDofs unknowns.

struct DenseSmem {
    int M, b, x, q, qp, v, vd, a, qd, T, resid, con, act, fmap, red, bord;
    // beam components (dense models with beams): shape tables, weights and
    // node state of one component at a time, its quadrature-point outputs and
    // the interpolated values
    int cphi, cdphi, cdphiJ, cqpw, cq, cv, cvd, cG, cFc, cFd, cgs;
    // condensed models: interior solution [6N], interior DOF map [N], the
    // bordered system's right-hand-side corrections [nd], the components'
    // orders (CompOrder) and one component's solution; M is -1 when the
    // bordered system lives in device memory (KBeam::cond_md)
    int xi, imap, bc, order, cx;
    int cW;  // condensed models: one component's system (inside M's region when M is shared)
    int chunk;  // condensed models: quadrature points per pass of a component's assembly,
    bool tight;  // and whether its rows are as short as whole tiles allow (cond_ld)
    int bytes;
};
// Row length of a bordered system of nd unknowns: the right-hand side is column
// nd, rows of even length.
KYN_HD inline int bord_ld(int nd) { return (nd + 2) & ~1; }
constexpr int kBordScratch = 1024;  // bytes of a BordScratch
// cN, cQ: nodes and points of the largest beam component (0: none);
// cond_nd > 0: a condensed model whose bordered system has cond_nd unknowns
// (md_global: kept in device memory instead of shared memory).
__host__ __device__ inline DenseSmem plan_dense_smem(int N, int nd, int cN, int cQ, int cond_nd,
                                                     bool md_global, int chunk, bool tight) {
    DenseSmem S{};
    int o = 0;
    auto take = [&](int bytes) {
        const int r = o;
        o += (bytes + 15) & ~15;
        return r;
    };
    if (cond_nd > 0) nd = cond_nd;
    // condensed models: the bordered system's region also holds, before the
    // system is assembled, one component's system [cond_rows][cond_ld], G and
    // the interpolated values of one chunk of its quadrature points (then the
    // inverse diagonal blocks, of which eight points hold twenty), and the
    // component's tables and node state
    auto r16 = [](int b) { return (b + 15) & ~15; };
    const int w_bytes = cond_nd > 0 ? cond_rows(cN) * cond_ld(cN, tight) * 8 : 0;
    const int t_bytes = cond_nd > 0 ? 3 * r16(cQ * cN * 8) + r16(cQ * 4 * 8) + r16(cN * 7 * 8) +
                                          2 * r16(cN * 6 * 8) + 2 * r16(cQ * 6 * 8) : 0;
    const int c_bytes = cond_nd > 0 ? w_bytes + chunk * (kGPoint + kQpInterp) * 8 + t_bytes : 0;
    const int m_bytes = md_global ? 0 : nd * bord_ld(nd) * 8;
    S.chunk = chunk;
    S.tight = tight;
    const int region = take(m_bytes > c_bytes ? m_bytes : c_bytes);
    S.M = md_global ? -1 : region;
    S.cW = cond_nd > 0 ? region : -1;
    S.b = take(nd * 8);
    S.x = take(nd * 8);
    S.q = take(N * 7 * 8);
    S.qp = take(N * 7 * 8);
    S.v = take(N * 6 * 8);
    S.vd = take(N * 6 * 8);
    S.a = take(N * 6 * 8);
    S.qd = take(N * 6 * 8);
    S.T = take(N * 9 * 8);
    S.resid = take(N * 6 * 8);
    S.con = take(kMaxBeamConstraints * kConStride * 8);
    S.act = take(N * 4);
    S.fmap = take(N * 4);
    S.red = take(64 * 8);  // per-warp partial sums of the error
    S.bord = take(kBordScratch);
    S.cphi = S.cdphi = S.cdphiJ = S.cqpw = S.cq = S.cv = S.cvd = S.cG = S.cFc = S.cFd = S.cgs = -1;
    if (cN > 0 && cond_nd > 0) {  // inside the bordered system's region, after the component's system
        int t = region + w_bytes;
        auto at = [&](int bytes) {
            const int r = t;
            t += r16(bytes);
            return r;
        };
        S.cG = at(S.chunk * kGPoint * 8);
        S.cgs = at(S.chunk * kQpInterp * 8);
        S.cphi = at(cQ * cN * 8);
        S.cdphi = at(cQ * cN * 8);
        S.cdphiJ = at(cQ * cN * 8);
        S.cqpw = at(cQ * 4 * 8);
        S.cq = at(cN * 7 * 8);
        S.cv = at(cN * 6 * 8);
        S.cvd = at(cN * 6 * 8);
        S.cFc = at(cQ * 6 * 8);
        S.cFd = at(cQ * 6 * 8);
    } else if (cN > 0) {
        S.cphi = take(cQ * cN * 8);
        S.cdphi = take(cQ * cN * 8);
        S.cdphiJ = take(cQ * cN * 8);
        S.cqpw = take(cQ * 4 * 8);
        S.cq = take(cN * 7 * 8);
        S.cv = take(cN * 6 * 8);
        S.cvd = take(cN * 6 * 8);
        S.cG = take(cQ * kGPoint * 8);
        S.cFc = take(cQ * 6 * 8);
        S.cFd = take(cQ * 6 * 8);
        S.cgs = take(cQ * kQpInterp * 8);
    }
    S.xi = S.imap = S.bc = S.order = S.cx = -1;
    if (cond_nd > 0) {
        S.xi = take(N * 6 * 8);
        S.imap = take(N * 4);
        S.bc = take(nd * 8);
        S.order = take(kMaxDenseComps * 164);
        S.cx = take((cN * 6 + 8) * 8);
    }
    S.bytes = o;
    return S;
}
// A condensed component's points are taken in one pass with the rows of its
// system on different banks where that fits, otherwise in smaller passes, at
// last with the rows packed.
__host__ __device__ inline DenseSmem make_dense_smem(int N, int nd, int cN = 0, int cQ = 0, int cond_nd = 0,
                                                     bool md_global = false) {
    DenseSmem S = plan_dense_smem(N, nd, cN, cQ, cond_nd, md_global, cQ > 8 ? cQ : 8, false);
    for (int chunk = 16; cond_nd > 0 && S.bytes > kMaxDynSmem && chunk >= 4; chunk /= 2)
        S = plan_dense_smem(N, nd, cN, cQ, cond_nd, md_global, chunk < 8 ? 8 : chunk, chunk < 8);
    return S;
}


// ---- quadrature-point physics -----------------------------------------------------
// Rows of x times tilde(w): each row crossed with w.
__device__ __forceinline__ void rows_cross(const double (&x)[9], const double (&w)[3], double (&o)[9]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        o[3 * i] = fma(x[3 * i + 1], w[2], -(x[3 * i + 2] * w[1]));
        o[3 * i + 1] = fma(x[3 * i + 2], w[0], -(x[3 * i] * w[2]));
        o[3 * i + 2] = fma(x[3 * i], w[1], -(x[3 * i + 1] * w[0]));
    }
}
// tilde(w) times x: w crossed with each column.
__device__ __forceinline__ void cols_cross(const double (&w)[3], const double (&x)[9], double (&o)[9]) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        o[j] = fma(w[1], x[6 + j], -(w[2] * x[3 + j]));
        o[3 + j] = fma(w[2], x[j], -(w[0] * x[6 + j]));
        o[6 + j] = fma(w[0], x[3 + j], -(w[1] * x[j]));
    }
}
// o += tilde(w)
__device__ __forceinline__ void add_tilde(double (&o)[9], const double (&w)[3]) {
    o[1] -= w[2];
    o[2] += w[1];
    o[3] += w[2];
    o[5] -= w[0];
    o[6] -= w[1];
    o[7] += w[0];
}
__device__ __forceinline__ void mul3(const double (&x)[9], const double (&w)[3], double (&o)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = fma(x[3 * i + 2], w[2], fma(x[3 * i + 1], w[1], x[3 * i] * w[0]));
}

// Interpolated values of one point in shared memory (doubles): r, u_ddot, omega,
// omega_dot by the shape values, u' and r' by the shape derivatives.
namespace qpi {
constexpr int r = 0, udd = 4, om = 7, omd = 10, up = 16, rp = 19;
}  // namespace qpi

// Quadrature-point physics of one beam system (calculate_quadrature_point_values.hpp:
// a6-a10 of the step path).  Inputs: shape tables phi / dphiJ [Q][N], weights
// qpw [Q][4], node state q [N][7], v, vd [N][6] (shared memory), the system's
// slab for the sections and reference frames (layout L), or sec: the sections
// already staged in shared memory (sec_doubles(Q), slab order from x0').
// Outputs: Fc, Fd + Fi - Fg [Q][6] and the weighted blocks of the integration, in
// FP64 G [Q][kGPoint] (gblk), the conditioner cond included, in FP32 G [4 Q][kGCols32]
// (gcol) without it.  itp: kQpInterp doubles of scratch per point.  Run by warps
// 0 .. NW - 1; ALL: they are the whole CTA (else they meet at barrier 1).
//
// The 20 interpolations are products [Q x N][N x 13] and [Q x N][N x 7] on the
// FP64 tensor cores.  Then eight lanes take a point, one rotated 3x3 block each
// (C11, C12, C21, C22, M11, M12, M21, M22), with the point's kinematics computed
// alike in all eight.  Every further matrix is such a block with its rows or
// columns crossed with a vector, or a dyad, so that one sequence of operations
// in registers serves all lanes, the operands selected by block:
//   O12 = C11 S - N~, O22 = C21 S - M~, P21 = S^T C11 + N~, P22 = S^T C12,
//   Q22 = S^T O12, G22 = w~ rho - (rho w)~,
//   K22 = rho w'~ - (rho w')~ + u''~ m~ + w~ (rho w~ - (rho w)~),
//   a~ b~ = b a^T - (a.b) I for G12, K12 and u''~ m~.
// The former form spent 16 lanes on a point, each entry by index arithmetic on
// shared memory with the six kinds of lanes one after the other: 23k cycles per
// iteration at 13 and at 21 nodes.
template <typename TG, int NW, bool ALL = true>
__device__ __forceinline__ void qp_phase(int N, int Q, const double* phi, const double* dphiJ,
                                         const double* qpw, const double* sq, const double* sv,
                                         const double* svd, const double* __restrict__ slab,
                                         const SlabLayout& L, const double* gravity, double beta_prime,
                                         double gamma_prime, double cond, double* itp, TG* G, double* Fc, double* Fdig,
                                         const double* sec = nullptr) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        const int g8 = lane >> 2, t = lane & 3;
        const int qt = (Q + 7) >> 3;
#pragma unroll 1
        for (int u = warp; u < 3 * qt; u += NW) {  // (tile of points, tile of columns)
            const int ct = u / qt, q0 = 8 * (u - ct * qt);
            const double* tab = (ct < 2 ? phi : dphiJ) + min(q0 + g8, Q - 1) * N;
            const double* src;
            int pitch = 6;
            if (ct == 0) {
                src = g8 < 4 ? sq + 3 + g8 : g8 < 7 ? svd + g8 - 4 : sv + 3;
                if (g8 < 4) pitch = 7;
            } else if (ct == 1) {
                src = g8 < 2 ? sv + 4 + g8 : svd + min(g8 + 1, 5);
            } else {
                src = sq + min(g8, 6);
                pitch = 7;
            }
            double d0 = 0., d1 = 0.;
#pragma unroll 2
            for (int n0 = 0; n0 < N; n0 += 4) {
                const int n = n0 + t, nc = min(n, N - 1);
                dmma884(d0, d1, n < N ? tab[nc] : 0., src[nc * pitch]);
            }
            if (q0 + g8 < Q) store_pair(itp + (q0 + g8) * kQpInterp + 8 * ct + 2 * t, d0, d1);
        }
    }
    if constexpr (ALL) __syncthreads();
    else asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
    const int role = lane & 7, bi = (role >> 1) & 1, bj = role & 1;
    const bool mass_block = role >= 4;
#pragma unroll 1
    for (int p0 = 4 * warp; p0 < Q; p0 += 4 * NW) {
        const int qp = p0 + (lane >> 3), qc = min(qp, Q - 1);
        const double *sx0, *sr0, *sblk;
        if (sec) {
            const int o = (3 * Q + 1) & ~1;
            sx0 = sec + qc * 3;
            sr0 = sec + o + qc * 4;
            sblk = sec + o + 4 * Q + (mass_block ? 0 : 36 * Q) + qc * 36;
        } else {
            sx0 = slab + L.x0p + qc * 3;
            sr0 = slab + L.r0 + qc * 4;
            sblk = slab + (mass_block ? L.mstar : L.cstar) + qc * 36;
        }
        sblk += 18 * bi + 3 * bj;
        const double* it = itp + qc * kQpInterp;
        double X[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) X[e] = sblk[(e / 3) * 6 + e % 3];
        double s[3], et[3], er[3];
        {
            double r[4], R[9], T[9];
#pragma unroll
            for (int e = 0; e < 4; ++e) r[e] = it[qpi::r + e];
            const double nr = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3]), inv = 1. / nr;
#pragma unroll
            for (int e = 0; e < 4; ++e) {  // r / nr, its residual put right
                const double v = r[e] * inv;
                r[e] = fma(fma(-v, nr, r[e]), inv, v);
            }
            // strain x0' + u' - R(r) x0', 2 E(r) r' (calculate_strain.hpp:27-46)
            const double x0[3] = {sx0[0], sx0[1], sx0[2]};
            double rx[3];
#pragma unroll
            for (int e = 0; e < 9; ++e) R[e] = rot_entry(r, e / 3, e % 3);
            mul3(R, x0, rx);
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                s[e] = x0[e] + it[qpi::up + e];
                et[e] = s[e] - rx[e];
            }
            const double rp[4] = {it[qpi::rp], it[qpi::rp + 1], it[qpi::rp + 2], it[qpi::rp + 3]};
            er[0] = 2. * (-r[1] * rp[0] + r[0] * rp[1] - r[3] * rp[2] + r[2] * rp[3]);
            er[1] = 2. * (-r[2] * rp[0] + r[3] * rp[1] + r[0] * rp[2] - r[1] * rp[3]);
            er[2] = 2. * (-r[3] * rp[0] - r[2] * rp[1] + r[1] * rp[2] + r[0] * rp[3]);
            // the block in the current frame, R(r o r0) X R^T
            double xr[4];
            const double r0[4] = {sr0[0], sr0[1], sr0[2], sr0[3]};
            quat_compose(r, r0, xr);
#pragma unroll
            for (int e = 0; e < 9; ++e) R[e] = rot_entry(xr, e / 3, e % 3);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    T[3 * i + j] = fma(X[3 * i], R[3 * j],
                                       fma(X[3 * i + 1], R[3 * j + 1], X[3 * i + 2] * R[3 * j + 2]));
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    X[3 * i + j] = fma(R[3 * i], T[j], fma(R[3 * i + 1], T[3 + j], R[3 * i + 2] * T[6 + j]));
        }
        // FC = Cuu eps (calculate_force_FC.hpp); rho omega, rho omega'; mass and
        // mass * eta from the rotated mass matrix
        double y[3], yd[3], ft[3], fr[3], me[3];
        {
            double a[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) a[e] = mass_block ? it[qpi::om + e] : bj ? er[e] : et[e];
            mul3(X, a, y);
#pragma unroll
            for (int e = 0; e < 3; ++e) a[e] = it[qpi::omd + e];
            mul3(X, a, yd);
        }
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const double f = y[e] + __shfl_xor_sync(kAll, y[e], 1);
            ft[e] = __shfl_sync(kAll, f, 0, 8);
            fr[e] = __shfl_sync(kAll, f, 2, 8);
        }
        const double m = __shfl_sync(kAll, X[0], 4, 8);
        me[0] = __shfl_sync(kAll, X[7], 6, 8);
        me[1] = -__shfl_sync(kAll, X[6], 6, 8);
        me[2] = __shfl_sync(kAll, X[3], 6, 8);
        // a section without mass has no centre of mass (eta = M/m): its step is refused
        if (m == 0.) me[0] = __longlong_as_double(0x7ff8000000000000ll);
        const bool on = qp < Q;
        constexpr bool wide = sizeof(TG) == 8;
        const double cw = wide ? cond : 1.;
        const double w = cw * qpw[qc * 4], wJ = cw * qpw[qc * 4 + 2];
        TG* Gq = G + qc * (wide ? kGPoint : 4 * kGCols32);
        if constexpr (!wide) {  // structural zeros, padding; the pad point of an odd Q
            if (on)
                for (int k = role; k < kGCols32 * ((Q & 1) && qp == Q - 1 ? 2 : 1); k += 8)
                    reinterpret_cast<float4*>(Gq)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            __syncwarp();
        }
        // blocks crossed with s (stiffness) or omega (mass): columns first
        double c[3], om[3], V[9];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            om[e] = it[qpi::om + e];
            c[e] = mass_block ? om[e] : -s[e];
        }
        double wme[3];  // omega x mass eta
        cross3(om, me, wme);
        const double wdm = om[0] * me[0] + om[1] * me[1] + om[2] * me[2];
        {
            double Z[9], tz[3];
            cols_cross(c, X, Z);
            if (role == 5) {  // G12 (calculate_gyroscopic_matrix.hpp)
#pragma unroll
                for (int e = 0; e < 9; ++e) Z[e] = (e % 4 == 0 ? wdm : 0.) - me[e / 3] * om[e % 3];
            }
#pragma unroll
            for (int e = 0; e < 3; ++e) tz[e] = role == 0 ? ft[e] : role == 7 ? -y[e] : role == 5 ? -wme[e] : 0.;
            add_tilde(Z, tz);  // P21, P22; G12, G22
            if (on && !wide) {
                // the same, XI by the sum that the form's rounding follows; left blocks at
                // 9 bi, right ones at 18 (C, K, O, P) or 36 (XI)
                TG* o = Gq + (mass_block ? 0 : 2 * kGCols32);
                const double wd = qpw[qc * 4 + 3];
#pragma unroll
                for (int e = 0; e < 9; ++e) {
                    const int l = bi ? gcol(9 + e) : gcol(e), rs = bi ? gcol(27 + e) : gcol(18 + e),
                              ri = bi ? gcol(45 + e) : gcol(36 + e);
                    const double xi = beta_prime * X[e] + gamma_prime * (bj ? Z[e] : 0.);
                    o[!bj ? l : mass_block ? ri : rs] = static_cast<TG>(mass_block ? wJ * xi : wd * X[e]);
                    if (role < 2) Gq[kGCols32 + (bj ? gcol(27 + e) : gcol(9 + e))] = static_cast<TG>(w * Z[e]);
                }
            } else if (on) {
                // C, XI = beta' Muu + gamma' Guu; P (no translational rows)
                TG* o = Gq + 3 * bi * kGRow + (mass_block ? (bj ? gblk::XIR : gblk::XIL) : (bj ? gblk::CR : gblk::CL));
                const double sc = mass_block ? wJ * beta_prime : cond * qpw[qc * 4 + 3];
                const double sg = mass_block && bj ? wJ * gamma_prime : 0.;
#pragma unroll
                for (int e = 0; e < 9; ++e) o[(e / 3) * kGRow + e % 3] = static_cast<TG>(fma(sg, Z[e], sc * X[e]));
                if (role < 4) {
                    TG* pp = Gq + (role < 2 ? 3 * kGRow : 0) + (bj ? gblk::PR : gblk::PL);
                    const double wp = role < 2 ? w : 0.;
#pragma unroll
                    for (int e = 0; e < 9; ++e) pp[(e / 3) * kGRow + e % 3] = static_cast<TG>(wp * Z[e]);
                }
            }
        }
        {
            double Y[9], ty[3], a[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                a[e] = mass_block ? om[e] : s[e];
                ty[e] = -(role == 0 ? ft[e] : role == 2 ? fr[e] : y[e]);
            }
            rows_cross(X, a, Y);
            add_tilde(Y, ty);  // O12, O22; rho w~ - (rho w)~
            if (on && (role == 0 || role == 2)) {
                TG* oo = wide ? Gq + 3 * bi * kGRow + gblk::O : Gq + 3 * kGCols32;
#pragma unroll
                for (int e = 0; e < 9; ++e)
                    oo[wide ? (e / 3) * kGRow + e % 3 : bi ? gcol(27 + e) : gcol(18 + e)] = static_cast<TG>(w * Y[e]);
            }
            cols_cross(c, Y, V);  // Q22; w~ (rho w~ - (rho w)~)
        }
#pragma unroll
        for (int e = 0; e < 9; ++e) {
            const double q22 = __shfl_sync(kAll, V[e], 0, 8);
            if (role == 7) V[e] += q22;
        }
        double ff[3] = {0., 0., 0.};
        if (role == 7) {
            // K22 (calculate_inertia_stiffness_matrix.hpp) + Q22; rotational part
            // of Fd + Fi - Fg (calculate_force_FD.hpp, calculate_inertial_force.hpp,
            // calculate_gravity_force.hpp)
            double W[9], g3[3], t0[3], t1[3], t2[3], u3[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                u3[e] = it[qpi::udd + e];
                t0[e] = it[qpi::omd + e];
            }
            rows_cross(X, t0, W);
            const double um = u3[0] * me[0] + u3[1] * me[1] + u3[2] * me[2];
#pragma unroll
            for (int e = 0; e < 9; ++e) V[e] += fma(me[e / 3], u3[e % 3], W[e]) - (e % 4 == 0 ? um : 0.);
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                t0[e] = -yd[e];
                g3[e] = u3[e] - gravity[e];
            }
            add_tilde(V, t0);
            cross3(ft, s, t0);
            cross3(me, g3, t1);
            cross3(om, y, t2);
#pragma unroll
            for (int e = 0; e < 3; ++e) ff[e] = t0[e] + t1[e] + yd[e] + t2[e];
        } else if (role == 3) {  // K12
            const double wd3[3] = {it[qpi::omd], it[qpi::omd + 1], it[qpi::omd + 2]};
            const double wm = wd3[0] * me[0] + wd3[1] * me[1] + wd3[2] * me[2];
#pragma unroll
            for (int e = 0; e < 9; ++e)
                V[e] = (e % 4 == 0 ? wm : 0.) - fma(me[e / 3], wd3[e % 3], wme[e / 3] * om[e % 3]);
            const double t0[3] = {wdm * om[0], wdm * om[1], wdm * om[2]};
            add_tilde(V, t0);
        } else if (role == 6) {  // translational part of the forces
            const double wd3[3] = {it[qpi::omd], it[qpi::omd + 1], it[qpi::omd + 2]};
            double t0[3], t1[3];
            cross3(om, wme, t0);
            cross3(wd3, me, t1);
#pragma unroll
            for (int e = 0; e < 3; ++e) ff[e] = fma(m, it[qpi::udd + e] - gravity[e], t0[e] + t1[e]);
        }
        if (on) {
            if (role == 3 || role == 7) {
                TG* kk = wide ? Gq + (role == 7 ? 3 * kGRow : 0) + gblk::K : Gq;
#pragma unroll
                for (int e = 0; e < 9; ++e)
                    kk[wide ? (e / 3) * kGRow + e % 3 : role == 7 ? gcol(27 + e) : gcol(18 + e)] =
                        static_cast<TG>(wJ * V[e]);
            }
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                if (role == 0) Fc[qp * 6 + e] = ft[e];
                if (role == 2) Fc[qp * 6 + 3 + e] = fr[e];
                if (role >= 6) Fdig[qp * 6 + (role == 7 ? 3 : 0) + e] = ff[e];
            }
        }
    }
}

// Beam element terms of the components of a dense model (the step path's
// a5-a14 for elements whose nodes sit in a dense bordered system): for each
// component, the quadrature-point physics (qp_phase, on the component's local
// nodes), the residual (integrate_residual_vector.hpp:33-50) into resid of
// the model nodes, and SM_ij = S_ij T_j + I_ij (integrate_stiffness_matrix.hpp,
// integrate_inertia_matrix.hpp, calculate_system_matrix.hpp) times the
// conditioner added into the dense matrix Md at the nodes' DOF rows and
// columns (contribute_beams_to_sparse_matrix.hpp).  Components run one after
// the other, so shared nodes sum without races.
template <int NT>
__device__ void dense_beam_terms(const KBeam& KB, const StepCoeffs& P, const DenseSmem& S, unsigned char* smem_raw,
                                 const double* sq, const double* sv, const double* svd, const double* sT,
                                 const int* fmap, double* Md, int nd, double* resid) {
    const int tid = threadIdx.x;
    double* phi = reinterpret_cast<double*>(smem_raw + S.cphi);
    double* dphi = reinterpret_cast<double*>(smem_raw + S.cdphi);
    double* dphiJ = reinterpret_cast<double*>(smem_raw + S.cdphiJ);
    double* qpw = reinterpret_cast<double*>(smem_raw + S.cqpw);
    double* cq = reinterpret_cast<double*>(smem_raw + S.cq);
    double* cv = reinterpret_cast<double*>(smem_raw + S.cv);
    double* cvd = reinterpret_cast<double*>(smem_raw + S.cvd);
    double* G = reinterpret_cast<double*>(smem_raw + S.cG);
    double* Fc = reinterpret_cast<double*>(smem_raw + S.cFc);
    double* Fd = reinterpret_cast<double*>(smem_raw + S.cFd);
    double* gscr = reinterpret_cast<double*>(smem_raw + S.cgs);
    const double cond = P.conditioner;
    for (int ci = 0; ci < KB.n_comps; ++ci) {
        const double* hd = KB.comps + ci * kCompHead;
        const double* cs = KB.comps + static_cast<long>(hd[0]);
        const int N = static_cast<int>(hd[1]), Q = static_cast<int>(hd[2]);
        const double* node = hd + 3;  // model node of each local node
        const SlabLayout L = make_slab_layout(N, Q);
        for (int k = tid; k < Q * N; k += NT) {
            phi[k] = cs[L.phi + k];
            dphi[k] = cs[L.dphi + k];
            dphiJ[k] = cs[L.dphiJ + k];
        }
        for (int k = tid; k < Q * 4; k += NT) qpw[k] = cs[L.qpw + k];
        for (int k = tid; k < N * 7; k += NT) cq[k] = sq[static_cast<int>(node[k / 7]) * 7 + k % 7];
        for (int k = tid; k < N * 6; k += NT) {
            const int n = static_cast<int>(node[k / 6]);
            cv[k] = sv[n * 6 + k % 6];
            cvd[k] = svd[n * 6 + k % 6];
        }
        __syncthreads();
        qp_phase<double, NT / 32>(N, Q, phi, dphiJ, qpw, cq, cv, cvd, cs, L, KB.gravity, P.beta_prime, P.gamma_prime,
                             cond, gscr, G, Fc, Fd);
        __syncthreads();
        for (int t = tid; t < N * 6; t += NT) {
            const int n = t / 6, c = t % 6;
            double acc = 0.;
            for (int qp = 0; qp < Q; ++qp) {
                const double w = qpw[qp * 4], wJ = qpw[qp * 4 + 2];
                acc += (w * dphi[qp * N + n]) * Fc[qp * 6 + c] + (wJ * phi[qp * N + n]) * Fd[qp * 6 + c];
            }
            resid[static_cast<int>(node[n]) * 6 + c] += acc;
        }
        integrate_node_pairs<NT>(
            N, Q, phi, dphi, G, [&](int j) { return sT + static_cast<int>(node[j]) * 9; },
            [&](int j, int r, int half) {
                double* col = Md + r * nd + fmap[static_cast<int>(node[j])] + 3 * half;
                return [=](int i, double v0, double v1, double v2) {
                    double* row = col + fmap[static_cast<int>(node[i])] * nd;
                    row[0] += v0;
                    row[1] += v1;
                    row[2] += v2;
                };
            });
        __syncthreads();
    }
}

// Record of a revolute joint in a dense model (constraint record layout drev;
// multipliers at conrec::lam, torque at conrec::inp): residual, the gradient
// rows B = G T on both nodes' rotations, G^T lambda and the torque about the
// target's joint axis (calculate_revolute_joint_constraint.hpp:19-113,
// calculate_revolute_joint_force.hpp:19-45, branch :388-465 of
// calculate_constraint_residual_gradient.hpp), as revolute_record computes it
// for the drive train's hub chain.  frame: x0, y0, z0 of the joint (rows).
namespace drev {
constexpr int Phi = 0;    // [5]
constexpr int Bt = 5;     // [2][3] rows 3-4 of G_target T_target (rotation)
constexpr int Bb = 11;    // [2][3] rows 3-4 of G_base T_base (rotation)
constexpr int sys = 17;   // [3] torque about R(target) x0
constexpr int GtL = 20;   // [6] G_target^T lambda
constexpr int GbL = 26;   // [6] G_base^T lambda
constexpr int xcz = 50;   // [3] x cross z
constexpr int xcy = 53;   // [3] x cross y
}  // namespace drev
__device__ inline void revolute_dense_record(double* cr, const double* bq, const double* tq, const double* frame,
                                             const double* X0, const double* Tb, const double* Tt) {
    double R1X0[3], x[3], y[3], z[3], ta[3];
    for (int i = 0; i < 3; ++i) {
        R1X0[i] = x[i] = y[i] = z[i] = ta[i] = 0.;
        for (int j = 0; j < 3; ++j) {
            R1X0[i] += rot_entry(bq + 3, i, j) * X0[j];
            x[i] += rot_entry(bq + 3, i, j) * frame[j];
            y[i] += rot_entry(tq + 3, i, j) * frame[3 + j];
            z[i] += rot_entry(tq + 3, i, j) * frame[6 + j];
            ta[i] += rot_entry(tq + 3, i, j) * frame[j];
        }
    }
    for (int i = 0; i < 3; ++i) cr[drev::Phi + i] = tq[i] + X0[i] - bq[i] - R1X0[i];
    cr[drev::Phi + 3] = z[0] * x[0] + z[1] * x[1] + z[2] * x[2];
    cr[drev::Phi + 4] = y[0] * x[0] + y[1] * x[1] + y[2] * x[2];
    const double xcz[3] = {x[1] * z[2] - x[2] * z[1], x[2] * z[0] - x[0] * z[2], x[0] * z[1] - x[1] * z[0]};
    const double xcy[3] = {x[1] * y[2] - x[2] * y[1], x[2] * y[0] - x[0] * y[2], x[0] * y[1] - x[1] * y[0]};
    const double torque = cr[conrec::inp];
    for (int i = 0; i < 3; ++i) {
        cr[drev::xcz + i] = xcz[i];
        cr[drev::xcy + i] = xcy[i];
        cr[drev::sys + i] = ta[i] * torque;
    }
    for (int j = 0; j < 3; ++j) {
        double a0 = 0., a1 = 0., b0 = 0., b1 = 0.;
        for (int k = 0; k < 3; ++k) {
            a0 -= xcz[k] * Tt[k * 3 + j];
            a1 -= xcy[k] * Tt[k * 3 + j];
            b0 += xcz[k] * Tb[k * 3 + j];
            b1 += xcy[k] * Tb[k * 3 + j];
        }
        cr[drev::Bt + j] = a0;
        cr[drev::Bt + 3 + j] = a1;
        cr[drev::Bb + j] = b0;
        cr[drev::Bb + 3 + j] = b1;
    }
    const double* l = cr + conrec::lam;
    for (int i = 0; i < 3; ++i) {
        cr[drev::GtL + i] = l[i];
        cr[drev::GbL + i] = -l[i];
        cr[drev::GtL + 3 + i] = -xcz[i] * l[3] - xcy[i] * l[4];
        cr[drev::GbL + 3 + i] = xcz[i] * l[3] + xcy[i] * l[4];
    }
}

// A component's place in shared memory, worked out once per step: its nodes in
// the model, and their order in the component's own system, interior nodes
// first.  That system has its interior unknowns padded to a multiple of eight
// (ones on the diagonal), then the boundary unknowns, then the right-hand side:
// whole tiles for eliminate_blocks.
struct CompOrder {
    short node[32];        // model node of each local node
    short row[32];         // first row of each local node
    unsigned char at[32];  // local node at each place (interior first)
    short ni, nb;          // interior and boundary nodes
};
static_assert(sizeof(CompOrder) == 164, "DenseSmem::order");
__device__ __forceinline__ int comp_pivots(const CompOrder& C) { return (6 * C.ni + 7) & ~7; }

// One warp per component.
template <int NT>
__device__ __forceinline__ void cond_order(const KBeam& KB, const int* fmap, CompOrder* order) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int ci = warp; ci < KB.n_comps; ci += NT / 32) {
        const double* hd = KB.comps + ci * kCompHead;
        const int N = static_cast<int>(hd[1]);
        CompOrder& C = order[ci];
        const int node = lane < N ? static_cast<int>(hd[3 + lane]) : 0;
        const bool inner = lane < N && fmap[node] < 0;
        const unsigned in = __ballot_sync(kAll, inner), out = __ballot_sync(kAll, lane < N && !inner);
        const unsigned below = (1u << lane) - 1u;
        const int ni = __popc(in), place = inner ? __popc(in & below) : ni + __popc(out & below);
        if (lane < N) {
            C.node[lane] = static_cast<short>(node);
            C.row[lane] = static_cast<short>(6 * place + (inner ? 0 : ((6 * ni + 7) & ~7) - 6 * ni));
            C.at[place] = static_cast<unsigned char>(lane);
        }
        if (lane == 0) {
            C.ni = static_cast<short>(ni);
            C.nb = static_cast<short>(__popc(out));
        }
    }
}

// Each component's system over its own local nodes, with the element terms of
// dense_beam_terms (residual, S_ij T_j + I_ij times the conditioner), S.chunk
// quadrature points at a time.  The interior rows carry their complete
// right-hand side -conditioner (R - node_FX - f); the boundary nodes' residual
// goes to resid like the other nodes of the bordered system.  The beam systems'
// block elimination of the interior rows leaves in the boundary rows the Schur
// complement A_bb - A_bi A_ii^-1 A_ib and the right-hand-side correction
// -A_bi A_ii^-1 b_i, and U = D^-1 A in the interior rows.  The eliminated system
// is saved to the component's workspace for cond_add_schur and
// cond_back_substitute.  This is the static condensation of the element groups
// that the reference's sparse direct solve factors as one matrix
// (src/solver/compute_system_row_entries.hpp:83-97 gives their overlap).  Bound
// by latency with eight warps on the SM: per iteration of a turbine (four
// components of 11 nodes) the points take 43k cycles, the assembly 73k, the
// elimination 42k.  One pivot per barrier with a row update per warp took 332k,
// and node by node lookups in device memory with sixteen points a pass 190k.
template <int NT>
__device__ __forceinline__ void cond_component_terms(const KBeam& KB, const StepCoeffs& P, const DenseSmem& S,
                                                     const double* sq, const double* sv, const double* svd,
                                                     const double* sT, const double* mslab, const SlabLayout& ML,
                                                     double* resid, int* flag, unsigned long long* ph = nullptr) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    // optional sub-phase timers (thread 0): quadrature physics, assembly,
    // elimination, save, in the slots kPhaseQuadrature, kPhaseCompIntegrate,
    // kPhaseCompEliminate, kPhaseCompSave of ph
    long long pt = (ph && tid == 0) ? clock64() : 0;
    auto sub = [&](int slot) {
        if (ph && tid == 0) {
            const long long t = clock64();
            ph[slot] += static_cast<unsigned long long>(t - pt);
            pt = t;
        }
    };
    double* phi = reinterpret_cast<double*>(smem_raw + S.cphi);
    double* dphi = reinterpret_cast<double*>(smem_raw + S.cdphi);
    double* dphiJ = reinterpret_cast<double*>(smem_raw + S.cdphiJ);
    double* qpw = reinterpret_cast<double*>(smem_raw + S.cqpw);
    double* cq = reinterpret_cast<double*>(smem_raw + S.cq);
    double* cv = reinterpret_cast<double*>(smem_raw + S.cv);
    double* cvd = reinterpret_cast<double*>(smem_raw + S.cvd);
    double* G = reinterpret_cast<double*>(smem_raw + S.cG);
    double* Fc = reinterpret_cast<double*>(smem_raw + S.cFc);
    double* Fd = reinterpret_cast<double*>(smem_raw + S.cFd);
    double* itp = reinterpret_cast<double*>(smem_raw + S.cgs);
    double* W = reinterpret_cast<double*>(smem_raw + S.cW);
    const CompOrder* order = reinterpret_cast<const CompOrder*>(smem_raw + S.order);
    const double cond = P.conditioner;
#pragma unroll 1
    for (int ci = 0; ci < KB.n_comps; ++ci) {
        const double* hd = KB.comps + ci * kCompHead;
        const double* cs = KB.comps + static_cast<long>(hd[0]);
        double* work = const_cast<double*>(KB.comps) + static_cast<long>(hd[kCompWork]);
        const int N = static_cast<int>(hd[1]), Q = static_cast<int>(hd[2]);
        const CompOrder& C = order[ci];
        const SlabLayout L = make_slab_layout(N, Q);
        const int mi = 6 * C.ni, mp = comp_pivots(C), rhs = mp + 6 * C.nb;
        const int rows = (rhs + 7) & ~7, ldw = cond_ld(N, S.tight);
        for (int k = tid; k < Q * N; k += NT) {
            phi[k] = cs[L.phi + k];
            dphi[k] = cs[L.dphi + k];
            dphiJ[k] = cs[L.dphiJ + k];
        }
        for (int k = tid; k < Q * 4; k += NT) qpw[k] = cs[L.qpw + k];
        for (int k = tid; k < 8 * N; k += NT) {
            const int l = k >> 3, c = k & 7, n = C.node[l];
            if (c < 7) cq[l * 7 + c] = sq[n * 7 + c];
            if (c < 6) {
                cv[l * 6 + c] = sv[n * 6 + c];
                cvd[l * 6 + c] = svd[n * 6 + c];
            }
        }
#pragma unroll 4
        for (int k = 2 * tid; k < rows * ldw; k += 2 * NT) store_pair(W + k, 0., 0.);
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < mp; i += NT) {  // interior right-hand side before the element residual; ones on the padding
            if (i < mi) {
                const int n = C.node[C.at[i / 6]] * 6 + i % 6;
                W[sys_at(ldw, i, rhs)] = cond * (mslab[ML.fx + n] + mslab[ML.f + n]);
            } else {
                W[sys_at(ldw, i, i)] = 1.;
            }
        }
#pragma unroll 1
        for (int q0 = 0; q0 < Q; q0 += S.chunk) {
            const int qn = min(S.chunk, Q - q0);
            SlabLayout Lc = L;
            Lc.mstar += 36 * q0;
            Lc.cstar += 36 * q0;
            Lc.r0 += 4 * q0;
            Lc.x0p += 3 * q0;
            qp_phase<double, NT / 32>(N, qn, phi + q0 * N, dphiJ + q0 * N, qpw + q0 * 4, cq, cv, cvd, cs, Lc,
                                 KB.gravity, P.beta_prime, P.gamma_prime, cond, itp, G, Fc, Fd);
            __syncthreads();
            sub(kPhaseQuadrature);
            for (int t = NT - 1 - tid; t < N * 6; t += NT) {  // the last warps have fewer pair units
                const int n = t / 6, c = t % 6;
                double acc = 0.;
#pragma unroll 2
                for (int qp = 0; qp < qn; ++qp) {
                    const int qa = q0 + qp;
                    const double w = qpw[qa * 4], wJ = qpw[qa * 4 + 2];
                    acc += (w * dphi[qa * N + n]) * Fc[qp * 6 + c] + (wJ * phi[qa * N + n]) * Fd[qp * 6 + c];
                }
                if (C.row[n] < mp) W[sys_at(ldw, C.row[n] + c, rhs)] -= cond * acc;
                else resid[C.node[n] * 6 + c] += acc;
            }
            integrate_node_pairs<NT>(
                N, qn, phi + q0 * N, dphi + q0 * N, G, [&](int j) { return sT + C.node[j] * 9; },
                [&](int j, int r, int half) {
                    const short* first = C.row;
                    const int col = first[j] + 3 * half;
                    return [=](int i, double v0, double v1, double v2) {
                        const int row = first[i] + r, sh = row & 6;
                        double* a = W + row * ldw;
                        if (q0 > 0) {  // uniform: added to the passes before
                            v0 += a[col ^ sh];
                            v1 += a[(col + 1) ^ sh];
                            v2 += a[(col + 2) ^ sh];
                        }
                        a[col ^ sh] = v0;
                        a[(col + 1) ^ sh] = v1;
                        a[(col + 2) ^ sh] = v2;
                    };
                });
            __syncthreads();
            sub(kPhaseCompIntegrate);
        }
        if (mp > 0) eliminate_blocks<NT>(W, ldw, mp, rows >> 3, (rhs + 8) >> 3, G, flag);
        sub(kPhaseCompEliminate);
#pragma unroll 4
        for (int k = 2 * tid; k < rows * ldw; k += 2 * NT) {
            const double2 v = load_pair(W + k);
            store_pair(work + k, v.x, v.y);
        }
        __syncthreads();
        sub(kPhaseCompSave);
    }
}

// Adds each condensed component's Schur complement (its workspace rows and
// columns of the boundary nodes) into the bordered system Md and its
// right-hand-side correction into bc, at the boundary nodes' DOF rows.
template <int NT>
__device__ __forceinline__ void cond_add_schur(const KBeam& KB, const DenseSmem& S, const CompOrder* order, const int* fmap, double* Md, int ldm,
                               double* bc) {
    const int tid = threadIdx.x;
#pragma unroll 1
    for (int ci = 0; ci < KB.n_comps; ++ci) {
        const double* hd = KB.comps + ci * kCompHead;
        const double* work = KB.comps + static_cast<long>(hd[kCompWork]);
        const CompOrder& C = order[ci];
        const int mp = comp_pivots(C), mb = 6 * C.nb, ldw = cond_ld(static_cast<int>(hd[1]), S.tight);
        for (int e = tid; e < mb * (mb + 1); e += NT) {
            const int t = e / (mb + 1), u = e % (mb + 1);
            const int rt = fmap[C.node[C.at[C.ni + t / 6]]] + t % 6;
            const double v = work[sys_at(ldw, mp + t, mp + u)];
            if (u == mb) bc[rt] += v;
            else Md[rt * ldm + fmap[C.node[C.at[C.ni + u / 6]]] + u % 6] += v;
        }
        __syncthreads();
    }
}

// Interior corrections of each condensed component from the bordered system's
// solution x at its boundary nodes: x_i = y_i - U_ib x_b - U_ii x_i, the rows of
// the eliminated system staged back into shared memory; the corrections go to
// xi at the nodes' interior DOFs.
template <int NT>
__device__ __forceinline__ void cond_back_substitute(const KBeam& KB, const DenseSmem& S, const int* fmap,
                                                     const int* imap, const double* x, double* xi) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* W = reinterpret_cast<double*>(smem_raw + S.cW);
    double* cx = reinterpret_cast<double*>(smem_raw + S.cx);
    const CompOrder* order = reinterpret_cast<const CompOrder*>(smem_raw + S.order);
#pragma unroll 1
    for (int ci = 0; ci < KB.n_comps; ++ci) {
        const double* hd = KB.comps + ci * kCompHead;
        const double* work = KB.comps + static_cast<long>(hd[kCompWork]);
        const CompOrder& C = order[ci];
        const int mi = 6 * C.ni, mp = comp_pivots(C), mb = 6 * C.nb, ldw = cond_ld(static_cast<int>(hd[1]), S.tight);
#pragma unroll 4
        for (int k = 2 * tid; k < mp * ldw; k += 2 * NT) {
            const double2 v = load_pair(work + k);
            store_pair(W + k, v.x, v.y);
        }
        __syncthreads();
#pragma unroll 1
        for (int i0 = 4 * warp; i0 < mp; i0 += NT / 8) {  // eight lanes per row
            const int i = i0 + (lane >> 3);
            double y = 0.;
#pragma unroll 1
            for (int u = lane & 7; u < mb; u += 8)
                y -= W[sys_at(ldw, i, mp + u)] * x[fmap[C.node[C.at[C.ni + u / 6]]] + u % 6];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
            if ((lane & 7) == 0) cx[i] = W[sys_at(ldw, i, mp + mb)] + y;
        }
        __syncthreads();
        if (mp > 0) back_substitute<NT>(W, ldw, mp, cx);
        for (int p = tid; p < mi; p += NT) xi[imap[C.node[C.at[p / 6]]] + p % 6] = cx[p];
        __syncthreads();
    }
}

// ---- pivoted LU of a bordered system ------------------------------------------------
// Md [md][ld], ld even, the right-hand side in column md; partial pivoting
// (largest entry by its leading 32 bits, lowest row on a tie), eight columns per
// panel:
//   1. the first warps factor the panel, a row per thread in registers; a pivot
//      is found by two integer reductions per warp and an exchange of the warps'
//      finds, and its row reaches the threads through shared memory;
//   2. tiles of eight columns to a warp: the pivot rows to the top, the rows they
//      displace to the places they leave, and U = L^-1 A with a row to four
//      lanes and the pivot rows by shuffle;
//   3. all warps subtract L U from the rest on the FP64 tensor cores.
// The unblocked form (pivot search, swap and a rank-1 update of the whole rest
// per column) was bound by the traffic of those updates and by three barriers a
// column: 643k cycles for 137 unknowns, now 185k, of which step 1 takes 95k (660
// cycles a column, a chain of reductions, barriers and a division), step 2 29k
// (34k with a column to a thread, whose straight-line code was fetched once per
// panel) and step 3 48k.  Slower: the panel in one warp with five rows to a lane
// (1100 cycles a column); the next panel beside step 3, whose tensor
// instructions hold up the panel's chain on the same FP64 pipes.
struct BordScratch {
    double prow[2][8];  // the pivot row, from the pivot on (double-buffered by column)
    double rp[2];       // the pivot's reciprocal
    unsigned long long key[2][8];  // per warp: leading bits of its largest entry, row (complemented)
    double lower[64];   // unit lower triangle of the panel's pivot rows [8][8]
    int piv[8];         // row each panel column was pivoted on
    int back[8];        // row (of the panel's eight) that goes where piv[c] was, or -1
};
static_assert(sizeof(BordScratch) <= kBordScratch, "DenseSmem::bord");

// Step 1, by warps 0 .. PW - 1 (which meet at barrier 2), RT rows per thread.
template <int PW, int RT>
__device__ __forceinline__ void factor_pivoted_panel(double* Md, int ld, int md, int k0, double* rpiv,
                                                     BordScratch* W, int* flag) {
    constexpr unsigned kAll = 0xffffffffu;
    auto meet = [&]() {
        if constexpr (PW == 1) __syncwarp();
        else asm volatile("bar.sync 2, %0;" ::"n"(32 * PW) : "memory");
    };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kb = min(8, md - k0);
    double v[RT][8];
    bool live[RT];
    int row[RT];
#pragma unroll
    for (int e = 0; e < RT; ++e) {
        const int i = k0 + tid + 32 * PW * e;
        live[e] = i < md;
        row[e] = min(i, md - 1) * ld + k0;
#pragma unroll
        for (int c = 0; c < 8; c += 2) {  // rows of even length: pairs
            const double2 x = load_pair(Md + row[e] + (c < kb ? c : 0));
            v[e][c] = c < kb ? x.x : 0.;
            v[e][c + 1] = c + 1 < kb ? x.y : 0.;
        }
    }
#pragma unroll 1
    for (int c = 0; c < kb; ++c) {  // the pivot column is v[.][0]
        const int h = c & 1;
        unsigned hi = 0;
        int at = 0;
        double best = v[0][0];
#pragma unroll
        for (int e = 0; e < RT; ++e) {
            const unsigned ah = static_cast<unsigned>(__double2hiint(v[e][0])) & 0x7fffffffu;
            const unsigned he = live[e] && ah <= 0x7ff00000u ? ah : 0u;  // NaN: 0
            if (he > hi) {
                hi = he;
                at = e;
                best = v[e][0];
            }
        }
        const unsigned mh = __reduce_max_sync(kAll, hi);
        const double inv = 1. / best;  // every lane's candidate, while the reductions run
        const unsigned mr = __reduce_min_sync(kAll, hi == mh ? static_cast<unsigned>(tid + 32 * PW * at) : ~0u);
        unsigned long long key = static_cast<unsigned long long>(mh) << 32 | (~mr);
        if constexpr (PW > 1) {
            if (lane == 0) W->key[h][warp] = key;
            meet();
            key = W->key[h][0];
#pragma unroll
            for (int w = 1; w < PW; ++w) key = max(key, W->key[h][w]);
        }
        const bool found = key >> 32 != 0ull;
        const int r = found ? static_cast<int>(~static_cast<unsigned>(key)) : c;
#pragma unroll
        for (int e = 0; e < RT; ++e)
            if (r == tid + 32 * PW * e) {  // the pivot row's thread
                W->rp[h] = inv;
                rpiv[k0 + c] = inv;
                W->piv[c] = k0 + r;
                if (!found) atomicOr(flag, 2);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    W->prow[h][j] = v[e][j];
                    if (c + j < kb) Md[row[e] + c + j] = v[e][j];
                }
                live[e] = false;
            }
        meet();
        const double rd = W->rp[h];
        double u[8];
#pragma unroll
        for (int j = 1; j < 8; ++j) u[j] = W->prow[h][j];
#pragma unroll
        for (int e = 0; e < RT; ++e) {
            const double l = v[e][0] * rd;
            if (live[e]) Md[row[e] + c] = l;
#pragma unroll
            for (int j = 0; j < 7; ++j) v[e][j] = fma(-l, u[j + 1], v[e][j + 1]);
            v[e][7] = 0.;
        }
    }
    meet();
    if (warp > 0) return;
    // the pivot rows' multipliers, and where the rows they displace go
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int r = lane >> 2, c = 2 * (lane & 3) + x;
        W->lower[8 * r + c] = r < kb && c < r ? Md[W->piv[r] * ld + k0 + c] : 0.;
    }
    const int p = lane < kb ? W->piv[lane] : -1;
    const unsigned out = __ballot_sync(kAll, p >= k0 + kb);                      // columns pivoted from below
    unsigned stay = __reduce_or_sync(kAll, p >= k0 && p < k0 + kb ? 1u << (p - k0) : 0u);
    stay = ~stay & ((1u << kb) - 1u);                                            // panel rows displaced
    if (lane < 8) {
        int d = -1;
        if (out >> lane & 1u) d = __fns(stay, 0, __popc(out & ((1u << lane) - 1u)) + 1);
        W->back[lane] = d;
        if (lane >= kb) W->piv[lane] = k0;
    }
}

template <int NT, bool SHARED>
__device__ __forceinline__ void solve_bordered(double* Mg, int off, int ld, int md, double* x, double* rpiv,
                                               BordScratch* W, int* flag) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int NW = NT / 32, CS = kCondMaxDofs / 32, PW = NW < CS ? NW : CS;
    double* Md = SHARED ? reinterpret_cast<double*>(smem_raw + off) : Mg;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fr = lane >> 2, t = lane & 3, t2 = 2 * t;
    auto panel = [&](int k0) {
        // up to 64 rows one warp does it without barriers
        if (md - k0 > 64) {
            if (warp < PW) factor_pivoted_panel<PW, (CS + PW - 1) / PW>(Md, ld, md, k0, rpiv, W, flag);
        } else if (warp == 0) {
            factor_pivoted_panel<1, 2>(Md, ld, md, k0, rpiv, W, flag);
        }
    };
    // tiles lo .. hi - 1, counted down columns of ni tiles from column c0 on, less the panel at k0
    auto update = [&](int k0, int c0, int ni, int lo, int hi) {
        const int r0 = k0 + 8;
        int j = static_cast<int>(__fdividef(static_cast<float>(lo) + 0.5f, static_cast<float>(ni)));
        int i = lo - j * ni;
#pragma unroll 1
        for (int left = hi - lo; left > 0;) {
            const int cj = c0 + 8 * j, cnt = min(ni - i, left), cu = min(cj + fr, md), cd = cj + t2;
            // products in the order of the columns, as the unblocked elimination takes them
            const double u0 = -Md[(k0 + t) * ld + cu], u1 = -Md[(k0 + 4 + t) * ld + cu];
#pragma unroll 1
            for (int e = 0; e < cnt; e += 2) {  // two tiles' loads ahead of their stores
                const int ra = r0 + 8 * (i + e) + fr, rb = ra + 8;
                const bool two = e + 1 < cnt;
                double* pa = Md + min(ra, md - 1) * ld;
                double* pb = Md + min(two ? rb : ra, md - 1) * ld;
                const int c1 = min(cd, ld - 2);
                const double la0 = pa[k0 + t], la1 = pa[k0 + 4 + t], lb0 = pb[k0 + t], lb1 = pb[k0 + 4 + t];
                double2 da = load_pair(pa + c1), db = load_pair(pb + c1);
                dmma884(da.x, da.y, la0, u0);
                if (two) dmma884(db.x, db.y, lb0, u0);
                dmma884(da.x, da.y, la1, u1);
                if (two) dmma884(db.x, db.y, lb1, u1);
                if (ra < md && cd <= md) store_pair(pa + cd, da.x, da.y);
                if (two && rb < md && cd <= md) store_pair(pb + cd, db.x, db.y);
            }
            left -= cnt;
            ++j;
            i = 0;
        }
    };
    panel(0);
    __syncthreads();
#pragma unroll 1
    for (int k0 = 0;; k0 += 8) {
        // 2. rows to their places, U = L^-1 A: a warp takes tiles of eight columns,
        // the pivot row and the displaced row of panel column fr to a lane
        const int kb = min(8, md - k0), r0 = k0 + 8;
        const int piv = W->piv[fr] * ld, back = W->back[fr];
        double low[7];
#pragma unroll
        for (int c = 0; c < 7; ++c) low[c] = -W->lower[8 * fr + c];
#pragma unroll 1
        for (int j0 = k0 + 8 * warp; j0 <= md; j0 += 8 * NW) {
            const int j = min(j0 + t2, ld - 2);
            const bool in = j0 + t2 <= md;
            double2 a = load_pair(Md + piv + j);
            const double2 d = load_pair(Md + (k0 + max(back, 0)) * ld + j);
            if (j0 > k0 || kb < 8) {
#pragma unroll
                for (int c = 0; c < 7; ++c) {
                    const double px = __shfl_sync(kAll, a.x, 4 * c + t), py = __shfl_sync(kAll, a.y, 4 * c + t);
                    if (c < fr && j >= k0 + kb) a.x = fma(low[c], px, a.x);
                    if (c < fr && j + 1 >= k0 + kb) a.y = fma(low[c], py, a.y);
                }
            }
            __syncwarp();
            if (in && fr < kb) store_pair(Md + (k0 + fr) * ld + j, a.x, a.y);
            if (in && back >= 0) store_pair(Md + piv + j, d.x, d.y);
        }
        __syncthreads();
        if (r0 >= md) break;
        // 3. the rest, in equal runs of tiles down the columns
        const int ni = (md - r0 + 7) >> 3, total = ni * ((md + 1 - r0 + 7) >> 3);
        update(k0, r0, ni, total * warp / NW, total * (warp + 1) / NW);
        __syncthreads();
        panel(r0);
        __syncthreads();
    }
    if (warp == 0 && md <= 64) {
        // Back substitution by rows.  A moored platform's step is the rounding of
        // 40 m arms to 1e-9 of its velocities, so the sums keep the order that its
        // results had: lane l takes columns i + 1 + l and i + 33 + l of row i, the
        // lanes' sums meet in an xor tree, the quotient is correctly rounded.  Only
        // lane 0's first term waits for x[i + 1]; what it receives in the tree (R)
        // is formed a row ahead, beside the row before it: 270 cycles a row for 480
        // with the tree, the division and x in shared memory one after the other.
        double xa = 0., xb = 0., m1 = 0., m2 = 0., R[5] = {0., 0., 0., 0., 0.};
#pragma unroll 1
        for (int i = md - 1; i >= 0; --i) {
            const double d = Md[i * ld + i], rd = rpiv[i];
            double s2 = fma(m2, xb, fma(m1, xa, 0.));
            // row i - 1 but for its first term
            const double *row = Md + max(i - 1, 0) * ld, up = __shfl_sync(kAll, xa, 31);
            double na = __shfl_up_sync(kAll, xa, 1), nb = __shfl_up_sync(kAll, xb, 1), r[5];
            if (lane == 0) nb = up;
            m1 = i + lane < md ? row[i + lane] : 0.;
            m2 = i + 32 + lane < md ? row[i + 32 + lane] : 0.;
            double p = fma(m2, nb, fma(m1, na, 0.));
#pragma unroll
            for (int e = 0; e < 5; ++e) {
                r[e] = __shfl_xor_sync(kAll, p, 16 >> e);
                p += r[e];
            }
#pragma unroll
            for (int e = 0; e < 5; ++e) s2 += R[e];
            // the quotient by the correctly rounded reciprocal and two corrections
            // (Markstein, IBM J. Res. Dev. 34, 1990)
            const double n = Md[i * ld + md] - s2;
            double q = n * rd;
            q = fma(fma(-q, d, n), rd, q);
            q = fma(fma(-q, d, n), rd, q);
            if (lane == 0) x[i] = q;
            xa = lane == 0 ? q : na;
            xb = nb;
#pragma unroll
            for (int e = 0; e < 5; ++e) R[e] = r[e];
        }
    } else if (warp == 0) {  // by columns, the right-hand side in registers
        double y[CS], u[CS];
        int row[CS];
#pragma unroll
        for (int e = 0; e < CS; ++e) {
            const int i = lane + 32 * e;
            row[e] = min(i, md - 1) * ld;
            y[e] = Md[row[e] + md];
            u[e] = i < md - 1 ? Md[row[e] + md - 1] : 0.;
        }
#pragma unroll
        for (int ks = CS - 1; ks >= 0; --ks) {
#pragma unroll 1
            for (int k = min(md - 1, 32 * ks + 31); k >= 32 * ks; --k) {
                const double xk = __shfl_sync(kAll, y[ks] * rpiv[k], k & 31);
                if (lane == 0) x[k] = xk;
#pragma unroll
                for (int e = 0; e <= ks; ++e) {
                    const int i = lane + 32 * e;
                    if (i < k) y[e] = fma(-u[e], xk, y[e]);
                    if (i < k - 1) u[e] = Md[row[e] + k - 1];  // for the next column
                }
            }
        }
    }
    __syncthreads();
}

template <int NT>
__device__ __forceinline__ void dense_model_step(const KBeam& KB, const StepCoeffs& P, int record, int* status_out,
                                 int* iters_out, unsigned char* smem_raw) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = KB.N, nc = KB.nc;
    const SlabLayout L = make_slab_layout(N, 0);
    double* __restrict__ slab = KB.slab;
    const int nd = KB.model_dofs;                       // the reference's unknowns
    const bool cnd = KB.cond_nd > 0;                    // condensed beam components
    const int md = cnd ? KB.cond_nd : nd;               // unknowns of the bordered system
    const DenseSmem S = make_dense_smem(N, nd, KB.n_comps > 0 ? KB.comp_maxN : 0, KB.comp_maxQ, KB.cond_nd,
                                        KB.cond_md != nullptr);
    double* Md = KB.cond_md ? KB.cond_md : reinterpret_cast<double*>(smem_raw + S.M);
    double* b = reinterpret_cast<double*>(smem_raw + S.b);
    double* x = reinterpret_cast<double*>(smem_raw + S.x);
    double* sq = reinterpret_cast<double*>(smem_raw + S.q);
    double* sqp = reinterpret_cast<double*>(smem_raw + S.qp);
    double* sv = reinterpret_cast<double*>(smem_raw + S.v);
    double* svd = reinterpret_cast<double*>(smem_raw + S.vd);
    double* sa = reinterpret_cast<double*>(smem_raw + S.a);
    double* sqd = reinterpret_cast<double*>(smem_raw + S.qd);
    double* sT = reinterpret_cast<double*>(smem_raw + S.T);
    double* resid = reinterpret_cast<double*>(smem_raw + S.resid);
    double* con = reinterpret_cast<double*>(smem_raw + S.con);
    int* act = reinterpret_cast<int*>(smem_raw + S.act);
    int* fmap = reinterpret_cast<int*>(smem_raw + S.fmap);
    double* red = reinterpret_cast<double*>(smem_raw + S.red);
    CompOrder* order = cnd ? reinterpret_cast<CompOrder*>(smem_raw + S.order) : nullptr;
    BordScratch* bord = reinterpret_cast<BordScratch*>(smem_raw + S.bord);
    const int ldm = bord_ld(md);
    double* xi = cnd ? reinterpret_cast<double*>(smem_raw + S.xi) : nullptr;
    int* imap = cnd ? reinterpret_cast<int*>(smem_raw + S.imap) : nullptr;
    double* bc = cnd ? reinterpret_cast<double*>(smem_raw + S.bc) : nullptr;
    __shared__ int s_flag, s_nsys;
    __shared__ short4 s_con[kMaxBeamConstraints];  // first row, type, node and base node of each constraint
    // phase timers (KYN_OPT_PHASE_TIMING): one CTA's clock, thread 0
    __shared__ unsigned long long s_ph[kNumPhases];
    const bool timing = KB.prof != nullptr;
    long long ph_t = 0;
    if (timing && tid == 0) {
        for (int k = 0; k < kNumPhases; ++k) s_ph[k] = 0ull;
        ph_t = clock64();
    }
    auto mark = [&](int phase) {
        if (timing && tid == 0) {
            const long long t = clock64();
            s_ph[phase] += static_cast<unsigned long long>(t - ph_t);
            ph_t = t;
        }
    };
    const double h = P.h;

    // state, constraint inputs, multipliers reset (ResetConstraints)
    for (int k = tid; k < N * 7; k += NT) sq[k] = slab[L.q + k];
    for (int k = tid; k < N * 6; k += NT) {
        sv[k] = slab[L.v + k];
        svd[k] = slab[L.vd + k];
        sa[k] = slab[L.a + k];
    }
    if (tid < nc) {
        double* c = con + tid * kConStride;
        for (int k = 0; k < 7; ++k) c[conrec::inp + k] = slab[L.con_input + tid * 7 + k];
        for (int k = 0; k < 6; ++k) c[conrec::lam + k] = 0.;
    }
    if (tid == 0) {
        // FreedomSignature per node (assemble_node_freedom_allocation_table.hpp):
        // masses six, springs position only, constraint targets six or three,
        // joint bases six; DOF map = exclusive scan (compute_node_freedom_map_table.hpp)
        for (int n = 0; n < N; ++n) act[n] = 0;
        if (cnd)
            for (int n = 0; n < N; ++n) imap[n] = 0;
        const double* mrec = KB.lumped;
        for (int e = 0; e < KB.n_mass; ++e) act[static_cast<int>(mrec[e * kMassRec])] |= kSigAll;
        const double* srec = KB.lumped + KB.n_mass * kMassRec;
        for (int e = 0; e < KB.n_spring; ++e) {
            act[static_cast<int>(srec[e * kSpringRec])] |= kSigPosition;
            act[static_cast<int>(srec[e * kSpringRec + 1])] |= kSigPosition;
        }
        for (int c = 0; c < nc; ++c) {
            const int t = KB.con_type[c];
            act[KB.con_node[c]] |= (t >= KYN_CONSTRAINT_FIXED_BC_3DOF) ? kSigPosition : kSigAll;
            if (KB.con_base[c] >= 0) act[KB.con_base[c]] |= kSigAll;
        }
        // condensed models: a node of one component only, with no mass, spring
        // or constraint, is interior (fmap -1, imap its first interior DOF)
        if (cnd)
            for (int n = 0; n < N; ++n) fmap[n] = act[n];
        for (int ci = 0; ci < KB.n_comps; ++ci) {  // beam nodes: all six components
            const double* hd = KB.comps + ci * kCompHead;
            for (int k = 0; k < static_cast<int>(hd[1]); ++k) {
                act[static_cast<int>(hd[3 + k])] |= kSigAll;
                if (cnd) ++imap[static_cast<int>(hd[3 + k])];
            }
        }
        int o = 0, oi = 0;
        for (int n = 0; n < N; ++n) {
            act[n] = (act[n] == kSigAll) ? 6 : (act[n] == kSigPosition) ? 3 : 0;
            if (cnd && imap[n] == 1 && fmap[n] == 0) {
                fmap[n] = -1;
                imap[n] = oi;
                oi += act[n];
            } else {
                fmap[n] = o;
                if (cnd) imap[n] = -1;
                o += act[n];
            }
        }
        int rows = 0;
        for (int c = 0; c < nc; ++c) rows += constraint_rows(KB.con_type[c]);
        s_nsys = o;
        s_flag = cnd ? ((o + rows != md || o + oi + rows != nd) ? 2 : 0) : (o > nd) ? 2 : 0;
    }
    __syncthreads();
    if (cnd) cond_order<NT>(KB, fmap, order);  // read behind the barriers below
    if (tid < nc) {
        int rf = s_nsys;
        for (int e = 0; e < tid; ++e) rf += constraint_rows(KB.con_type[e]);
        s_con[tid] = make_short4(static_cast<short>(rf), static_cast<short>(KB.con_type[tid]),
                                 static_cast<short>(KB.con_node[tid]), static_cast<short>(KB.con_base[tid]));
    }
    const int nsys = s_nsys;
    // PredictNextState (src/step/predict_next_state.hpp:14-47)
    for (int k = tid; k < N * 7; k += NT) sqp[k] = sq[k];
    for (int k = tid; k < N * 6; k += NT) {
        const double v_p = sv[k], vd_p = svd[k], a_p = sa[k];
        svd[k] = 0.;
        const double an = (P.alpha_f * vd_p - P.alpha_m * a_p) / (1. - P.alpha_m);
        sa[k] = an;
        sv[k] = v_p + h * (1. - P.gamma) * a_p + P.gamma * h * an;
        sqd[k] = v_p + (0.5 - P.beta) * h * a_p + P.beta * h * an;
    }
    __syncthreads();
    auto displacement = [&]() {
        for (int n = tid; n < N; n += NT) {
            for (int c = 0; c < 3; ++c) sq[n * 7 + c] = sqp[n * 7 + c] + h * sqd[n * 6 + c];
            const double d[3] = {h * sqd[n * 6 + 3], h * sqd[n * 6 + 4], h * sqd[n * 6 + 5]};
            double qd4[4], qn[4];
            rotvec_to_quat(d, qd4);
            quat_compose(qd4, sqp + n * 7 + 3, qn);
            for (int c = 0; c < 4; ++c) sq[n * 7 + 3 + c] = qn[c];
        }
    };
    displacement();
    __syncthreads();

    int status = KYN_NOT_CONVERGED, iters = 0;
    const double cond = P.conditioner;
    for (int iter = 0; iter < P.max_iter && s_flag == 0; ++iter) {
        // tangent operator, rotational block (src/system/calculate_tangent_operator.hpp)
        for (int n = tid; n < N; n += NT) {
            const double rv[3] = {h * sqd[n * 6 + 3], h * sqd[n * 6 + 4], h * sqd[n * 6 + 5]};
            const double ph = sqrt(rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
            double sn, cs;
            sincos(ph, &sn, &cs);
            const double t1 = (ph > 1.e-16) ? (cs - 1.) / (ph * ph) : 0.;
            const double t2 = (ph > 1.e-16) ? (1. - sn / ph) / (ph * ph) : 0.;
            for (int i = 0; i < 3; ++i)
                for (int j = 0; j < 3; ++j) {
                    double rr = 0.;
                    for (int k = 0; k < 3; ++k) rr += tilde_e(rv, j, k) * tilde_e(rv, k, i);
                    sT[n * 9 + i * 3 + j] = (i == j ? 1. : 0.) + (t1 * tilde_e(rv, j, i) + t2 * rr);
                }
        }
        for (int k = tid; k < N * 6; k += NT) resid[k] = 0.;
        mark(kPhaseLoadPredict);
        if (cnd) {  // components first: their systems share the bordered system's region
            __syncthreads();
            cond_component_terms<NT>(KB, P, S, sq, sv, svd, sT, slab, L, resid, &s_flag,
                                     timing ? s_ph : nullptr);
        }
        mark(kPhaseIntegrate);
#pragma unroll 4
        for (int k = 2 * tid; k < md * ldm; k += 2 * NT) store_pair(Md + k, 0., 0.);
        for (int k = tid; k < md; k += NT) b[k] = 0.;
        if (cnd)
            for (int k = tid; k < md; k += NT) bc[k] = 0.;
        __syncthreads();
        // masses and springs (residual into resid, conditioned blocks into Md)
        for (int n = tid; n < N; n += NT)
            add_lumped_terms(n, KB.lumped, KB.n_mass, KB.n_spring, sq, sv, svd, sT, KB.gravity,
                             P.beta_prime, P.gamma_prime, cond, fmap,
                             [&](int r, int c) -> double& { return Md[r * ldm + c]; }, resid, 1);
        if (KB.n_comps > 0) {  // beam elements, then their node_FX (summed per node)
            __syncthreads();
            if (cnd) cond_add_schur<NT>(KB, S, order, fmap, Md, ldm, bc);
            else dense_beam_terms<NT>(KB, P, S, smem_raw, sq, sv, svd, sT, fmap, Md, ldm, resid);
            for (int t = tid; t < N * 6; t += NT) resid[t] -= slab[L.fx + t];
        }
        // constraints: residual, gradients and G^T lambda
        // (one lane each, over the warps behind the masses' first: their types branch apart)
        const int cc = lane * (NW - 1) + warp - 1;
        if (warp > 0 && cc < nc) {
            double* cr = con + cc * kConStride;
            const int t = s_con[cc].y, tn = s_con[cc].z, bn = s_con[cc].w;
            if (t >= KYN_CONSTRAINT_FIXED_BC_3DOF) {
                // three rows (calculate_*_3DOF_constraint.hpp): u2 + X0 - u1 - R1 X0
                double u1[3] = {0., 0., 0.}, R1[4] = {1., 0., 0., 0.};
                if (t == KYN_CONSTRAINT_PRESCRIBED_BC_3DOF) {
                    for (int k = 0; k < 3; ++k) u1[k] = cr[conrec::inp + k];
                    for (int k = 0; k < 4; ++k) R1[k] = cr[conrec::inp + 3 + k];
                } else if (t == KYN_CONSTRAINT_RIGID_JOINT_6DOF_TO_3DOF) {
                    for (int k = 0; k < 3; ++k) u1[k] = sq[bn * 7 + k];
                    for (int k = 0; k < 4; ++k) R1[k] = sq[bn * 7 + 3 + k];
                }
                const double* X0 = KB.con_X0[cc];
                double r1x0[3];
                for (int i = 0; i < 3; ++i) {
                    r1x0[i] = 0.;
                    for (int j = 0; j < 3; ++j) r1x0[i] += rot_entry(R1, i, j) * X0[j];
                }
                for (int i = 0; i < 3; ++i) {
                    cr[conrec::Phi + i] = sq[tn * 7 + i] + X0[i] - u1[i] - r1x0[i];
                    cr[conrec::Gl + i] = cr[conrec::lam + i];
                    cr[conrec::R1X0 + i] = r1x0[i];
                }
                if (t == KYN_CONSTRAINT_RIGID_JOINT_6DOF_TO_3DOF)  // base block tilde(R1 X0) T_base
                    for (int i = 0; i < 3; ++i)
                        for (int j = 0; j < 3; ++j) {
                            double bt = 0.;
                            for (int k = 0; k < 3; ++k) bt += tilde_e(r1x0, i, k) * sT[bn * 9 + k * 3 + j];
                            cr[conrec::Btr + i * 3 + j] = bt;
                        }
            } else if (t == KYN_CONSTRAINT_REVOLUTE_JOINT) {
                revolute_dense_record(cr, sq + bn * 7, sq + tn * 7, KB.con_frames + cc * 9, KB.con_X0[cc],
                                      sT + bn * 9, sT + tn * 9);
            } else {
                constraint_record(cr, t, sq + tn * 7, KB.con_X0[cc], sT + tn * 9,
                                  bn >= 0 ? sq + bn * 7 : nullptr, bn >= 0 ? sT + bn * 9 : nullptr,
                                  KB.con_axis[cc]);
            }
            if (bn >= 0 && t != KYN_CONSTRAINT_REVOLUTE_JOINT) {  // G_base^T lambda
                double* gb = cr + conrec::yr;
                const double* lam = cr + conrec::lam;
                for (int k = 0; k < 6; ++k) gb[k] = 0.;
                if (constraint_rows(t) == 3) {
                    for (int i = 0; i < 3; ++i) {
                        gb[i] = -lam[i];
                        for (int k = 0; k < 3; ++k) gb[3 + i] += tilde_e(cr + conrec::R1X0, k, i) * lam[k];
                    }
                } else {
                    joint_base_transpose_add(cr, lam, gb);
                }
            }
        }
        __syncthreads();
        // scatter: rows of B = G T, columns G^T, residuals (assemble_constraints_matrix.hpp,
        // assemble_constraints_residual.hpp, assemble_system_residual.hpp)
        // One thread per constraint: its rows and columns of Md are its own, zero so far.  The
        // nodes' forces, which constraints share, are summed per component in
        // the order of the constraints by six lanes of another warp.
        if (tid < nc) {
            const double* cr = con + tid * kConStride;
            const int rf = s_con[tid].x, t = s_con[tid].y, bn = s_con[tid].w;
            const int rows = constraint_rows(t), ft = fmap[s_con[tid].z];
            if (t == KYN_CONSTRAINT_REVOLUTE_JOINT) {  // five rows, gradients on both nodes
                const int fb = fmap[bn];
#pragma unroll 1
                for (int r = 0; r < 5; ++r) {
                    double* row = Md + (rf + r) * ldm;
                    if (r < 3) {
                        row[ft + r] = 1.;
                        Md[(ft + r) * ldm + rf + r] = 1.;
                        row[fb + r] = -1.;
                        Md[(fb + r) * ldm + rf + r] = -1.;
                    } else {
                        const double* v = cr + (r == 3 ? drev::xcz : drev::xcy);
                        for (int j = 0; j < 3; ++j) {
                            row[ft + 3 + j] = cr[drev::Bt + (r - 3) * 3 + j];
                            row[fb + 3 + j] = cr[drev::Bb + (r - 3) * 3 + j];
                            Md[(ft + 3 + j) * ldm + rf + r] = -v[j];
                            Md[(fb + 3 + j) * ldm + rf + r] = v[j];
                        }
                    }
                    b[rf + r] += cr[drev::Phi + r];
                }
            } else {
#pragma unroll 1
                for (int r = 0; r < rows; ++r) {
                    double* row = Md + (rf + r) * ldm;
                    if (r < 3) {
                        row[ft + r] = 1.;
                        Md[(ft + r) * ldm + rf + r] = 1.;
                    } else {
                        for (int j = 0; j < 3; ++j) {
                            row[ft + 3 + j] = cr[conrec::Brot + (r - 3) * 3 + j];
                            Md[(ft + 3 + j) * ldm + rf + r] = cr[conrec::AX + j * 3 + (r - 3)];
                        }
                    }
                    b[rf + r] += cr[conrec::Phi + r];
                }
                if (bn >= 0) {  // joint base blocks: B_b = [-I, Btr; 0, Brr], G_b = [-I, tilde; 0, -AX]
                    const int fb = fmap[bn];
#pragma unroll 1
                    for (int r = 0; r < rows; ++r) {
                        double* row = Md + (rf + r) * ldm;
                        if (r < 3) {
                            row[fb + r] = -1.;
                            Md[(fb + r) * ldm + rf + r] = -1.;
                            for (int j = 0; j < 3; ++j) {
                                row[fb + 3 + j] = cr[conrec::Btr + r * 3 + j];
                                Md[(fb + 3 + j) * ldm + rf + r] = tilde_e(cr + conrec::R1X0, r, j);
                            }
                        } else {
                            for (int j = 0; j < 3; ++j) {
                                row[fb + 3 + j] = cr[conrec::Brr + (r - 3) * 3 + j];
                                Md[(fb + 3 + j) * ldm + rf + r] = -cr[conrec::AX + (r - 3) * 3 + j];
                            }
                        }
                    }
                }
            }
        } else if (warp == 1 && lane < 6) {
            const int e = lane;
#pragma unroll 1
            for (int c = 0; c < nc; ++c) {
                const double* cr = con + c * kConStride;
                const int t = s_con[c].y, bn = s_con[c].w, ft = fmap[s_con[c].z];
                if (t == KYN_CONSTRAINT_REVOLUTE_JOINT) {
                    b[ft + e] += cr[drev::GtL + e] + (e >= 3 ? cr[drev::sys + e - 3] : 0.);
                    b[fmap[bn] + e] += cr[drev::GbL + e];
                } else {
                    if (e < (constraint_rows(t) == 3 ? 3 : 6)) b[ft + e] += cr[conrec::Gl + e];
                    if (bn >= 0) b[fmap[bn] + e] += cr[conrec::yr + e];
                }
            }
        }
        __syncthreads();
        // b = -(cond (R - f) on the system rows, Phi on the constraint rows)
        for (int n = tid; n < N; n += NT)  // position-only nodes: components 0..2
            if (fmap[n] >= 0)
                for (int c = 0; c < act[n]; ++c) b[fmap[n] + c] += resid[n * 6 + c] - slab[L.f + n * 6 + c];
        __syncthreads();
        for (int k = tid; k < md; k += NT)
            Md[k * ldm + md] = -(k < nsys ? b[k] * cond : b[k]) + (cnd ? bc[k] : 0.);
        __syncthreads();
        mark(kPhaseConstraints);
        // (apart, so that the shared system is read by shared-memory loads)
        if (KB.cond_md) solve_bordered<NT, false>(KB.cond_md, 0, ldm, md, x, b, bord, &s_flag);
        else solve_bordered<NT, true>(nullptr, S.M, ldm, md, x, b, bord, &s_flag);
        mark(kPhaseFactor);
        // multipliers unconditioned; convergence error (calculate_convergence_error.hpp)
        for (int k = nsys + tid; k < md; k += NT) x[k] /= cond;
        __syncthreads();
        if (cnd) cond_back_substitute<NT>(KB, S, fmap, imap, x, xi);
        mark(kPhaseSubstitute);
        // correction of component c of node n
        auto delta_of = [&](int n, int c) { return fmap[n] >= 0 ? x[fmap[n] + c] : xi[imap[n] + c]; };
        double part = 0.;
        for (int k = tid; k < N * 6; k += NT) {
            const int n = k / 6, c = k - 6 * n;
            if (c < act[n]) {
                const double e = delta_of(n, c) / (P.atol + P.rtol * fabs(sqd[k] * h));
                part += e * e;
            }
        }
        for (int k = NT - 1 - tid; k < nc * 6; k += NT) {
            const int n = k / 6, r = k - 6 * n;
            if (r < constraint_rows(s_con[n].y)) {
                const double e = x[s_con[n].x + r] / (P.atol + P.rtol * fabs(con[n * kConStride + conrec::lam + r]));
                part += e * e;
            }
        }
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) red[warp] = part;
        __syncthreads();
        double total = 0.;
        for (int w2 = 0; w2 < NW; ++w2) total += red[w2];
        const double err = sqrt(total / static_cast<double>(nd));
        if (tid == 0 && iter < kMaxNewtonIters) KB.conv[iter] = err;
        iters = iter + 1;
        // update (update_state_prediction.hpp, update_lambda_prediction.hpp)
        for (int k = tid; k < N * 6; k += NT) {
            const int n = k / 6, c = k - 6 * n;
            if (c < act[n]) {
                const double delta = delta_of(n, c);
                sqd[k] += delta / h;
                if (P.dynamic) {
                    sv[k] += P.gamma_prime * delta;
                    svd[k] += P.beta_prime * delta;
                }
            }
        }
        for (int k = NT - 1 - tid; k < nc * 6; k += NT) {
            const int n = k / 6, r = k - 6 * n;
            if (r < constraint_rows(s_con[n].y)) con[n * kConStride + conrec::lam + r] += x[s_con[n].x + r];
        }
        __syncthreads();
        displacement();
        __syncthreads();
        mark(kPhaseUpdate);
        if (s_flag != 0) {
            status = KYN_ERR_SINGULAR;
            break;
        }
        if (!(err == err) || isinf(err)) {
            status = KYN_ERR_NONFINITE;
            break;
        }
        if (err <= 1.) {
            status = KYN_OK;
            break;
        }
    }
    if (s_flag != 0 && status == KYN_NOT_CONVERGED) status = KYN_ERR_INVALID;
    // post-step (step.hpp:86-121) and the resident state
    if (status == KYN_OK) {
        const double fac = (1. - P.alpha_f) / (1. - P.alpha_m);
        for (int k = tid; k < N * 6; k += NT) sa[k] += fac * svd[k];
    }
    __syncthreads();
    for (int k = tid; k < N * 7; k += NT) {
        slab[L.q + k] = sq[k];
        slab[L.q_prev + k] = sqp[k];
    }
    for (int k = tid; k < N * 6; k += NT) {
        slab[L.v + k] = sv[k];
        slab[L.vd + k] = svd[k];
        slab[L.a + k] = sa[k];
        slab[L.q_delta + k] = sqd[k];
    }
    if (status == KYN_OK)
        for (int n = tid; n < N; n += NT) {
            const double* x0 = slab + L.x0 + n * 7;
            for (int c = 0; c < 3; ++c) slab[L.x + n * 7 + c] = x0[c] + sq[n * 7 + c];
            double r[4];
            quat_compose(sq + n * 7 + 3, x0 + 3, r);
            for (int c = 0; c < 4; ++c) slab[L.x + n * 7 + 3 + c] = r[c];
        }
    for (int k = tid; k < N * 9; k += NT) slab[L.tangent + k] = sT[k];
    if (tid < 6 * nc) slab[L.lambda + tid] = con[(tid / 6) * kConStride + conrec::lam + tid % 6];
    if (tid == 0) {
        status_out[KB.plan_model] = status;
        iters_out[KB.plan_model] = iters;
        if (timing)
            for (int k = 0; k < kNumPhases; ++k) atomicAdd(KB.prof + k, s_ph[k]);
    }
    (void)record;  // dense models keep no system dump (kyn_get_system refuses them)
}

// One CTA per dense model.
template <int NT>
__global__ void __launch_bounds__(NT) dense_kernel(const KBeam* __restrict__ beams, StepCoeffs P, int record,
                                                   int* __restrict__ status_out, int* __restrict__ iters_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    dense_model_step<NT>(beams[blockIdx.x], P, record, status_out, iters_out, smem_raw);
}

// ---- the kernel ------------------------------------------------------------------
// Resident CTAs per SM that each instance is compiled for (its register budget
// is 65536 / (NT * this), 128 registers per thread for all three).  Three
// 256-thread CTAs per SM in the FP32 form (80 registers) would fit its shared
// memory up to 16 nodes, but the spills land in the pivot loops and cost more
// than the third beam per SM hides.
__host__ __device__ constexpr int step_min_blocks(int real_bytes, int nt) {
    return (void)real_bytes, nt == 128 ? 4 : nt == 256 ? 2 : 1;
}

// LUMP: the instance that also adds point masses and springs (KBeam::lumped);
// beams without them run the instance compiled without that code, whose
// registers it would otherwise crowd.
// GJ: the instance that also carries the register Gauss-Jordan solve
// (KYN_SOLVER_GAUSS_JORDAN); the default instances carry only the
// elimination in shared memory, whose register allocation the Gauss-Jordan tile would otherwise crowd.
template <typename TR, int NT, bool LUMP, bool GJ = false>
__global__ void __launch_bounds__(NT, step_min_blocks(sizeof(TR), NT))
    step_kernel(const KBeam* __restrict__ beams, StepCoeffs P, int record,
                int* __restrict__ status_out, int* __restrict__ iters_out) {
    static_assert(NT == 128 || NT == 256 || NT == 512, "step kernel runs with 128, 256 or 512 threads");
    constexpr int NW = NT / 32;  // warps
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const KBeam& KB = beams[blockIdx.x];
    const int N = KB.N, Q = KB.Q, nc = KB.nc;
    const int n6 = 6 * N;
    const int m = 6 * (N - nc);   // free-node block size
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chain = KB.hub;  // hub chain length (0: no hub)
    const bool hub = chain != 0;
    const bool drive = LUMP && chain > 1;  // drive trains run in the LUMP instance only
    if (!LUMP && chain > 1) {  // launch-plan error: refuse rather than solve without the chain
        if (tid == 0 && KB.rank == 0) {
            status_out[KB.plan_model] = KYN_ERR_UNSUPPORTED;
            iters_out[KB.plan_model] = 0;
        }
        return;
    }
    const Smem S = make_smem(N, Q, nc, sizeof(TR), NT, drive ? 2 : (hub ? 1 : 0));
    const SlabLayout L = make_slab_layout(N, Q);
    double* __restrict__ slab = KB.slab;

    TR* A = reinterpret_cast<TR*>(smem_raw + S.A);
    const int ldA = S.ldA;
    using TG = TR;  // element type of G: FP64 form double, FP32 form float
    TG* G = reinterpret_cast<TG*>(smem_raw + S.G);
    double* Fc = reinterpret_cast<double*>(smem_raw + S.Fc);
    double* Fdig = reinterpret_cast<double*>(smem_raw + S.Fdig);
    double* phi = reinterpret_cast<double*>(smem_raw + S.phi);
    double* dphi = reinterpret_cast<double*>(smem_raw + S.dphi);
    double* dphiJ = reinterpret_cast<double*>(smem_raw + S.dphiJ);
    double* qpw = reinterpret_cast<double*>(smem_raw + S.qpw);
    double* sq = reinterpret_cast<double*>(smem_raw + S.q);
    double* sqp = reinterpret_cast<double*>(smem_raw + S.q_prev);
    double* sv = reinterpret_cast<double*>(smem_raw + S.v);
    double* svd = reinterpret_cast<double*>(smem_raw + S.vd);
    double* sa = reinterpret_cast<double*>(smem_raw + S.a);
    double* sqd = reinterpret_cast<double*>(smem_raw + S.qd);
    double* sT = reinterpret_cast<double*>(smem_raw + S.T);
    double* hb = hub ? reinterpret_cast<double*>(smem_raw + S.hub) : nullptr;  // hub record
    // drive train: chain records 1 (revolute target) and 2 (optional), and the
    // record the beam roots join (the last of the chain)
    double* hA = drive ? hb + hubsm::n1 : nullptr;
    double* hH = (drive && chain == 3) ? hb + hubsm::n2 : nullptr;
    double* hj = drive ? (hH ? hH : hA) : hb;
    double* resid = reinterpret_cast<double*>(smem_raw + S.resid);
    double* bp = reinterpret_cast<double*>(smem_raw + S.b);
    double* xs = reinterpret_cast<double*>(smem_raw + S.xs);
    double* droot = drive ? reinterpret_cast<double*>(smem_raw + S.droot) : nullptr;
    double* con = reinterpret_cast<double*>(smem_raw + S.con);
    double* itp = reinterpret_cast<double*>(smem_raw + S.A);  // quadrature phase only
    double* red = reinterpret_cast<double*>(smem_raw + S.red);
    int* pos = reinterpret_cast<int*>(smem_raw + S.pos);
    int* node_at = pos + N;
    __shared__ int s_flag;
    __shared__ unsigned long long s_ph[kNumPhases];
    // sections of the next quadrature phase: one bulk copy per Newton
    // iteration (slab from x0' on -> the A region after the interpolated values)
    uint64_t* sec_bar = reinterpret_cast<uint64_t*>(smem_raw + S.bar);
    double* sec = reinterpret_cast<double*>(smem_raw + S.sec);
    const uint32_t sec_bytes = static_cast<uint32_t>(sec_doubles(Q)) * 8u;
    uint32_t sec_issued = 0, sec_waited = 0;  // copies issued / completed (thread 0 issues)
    const bool bulk = P.bulk_sections != 0;
    auto sec_issue = [&]() {  // all threads, after a proxy fence and a barrier behind the region's last use
        if (!bulk) return;
        if (tid == 0) bulk_copy_g2s(sec, slab + L.x0p, sec_bytes, sec_bar);
        ++sec_issued;
    };
    auto sec_wait = [&]() {  // all threads
        if (!bulk) return;
        if (!mbar_wait(sec_bar, sec_waited & 1u) && tid == 0) atomicOr(&s_flag, 8);
        ++sec_waited;
    };

    const double h = P.h;
    // Optional phase timing: thread 0 reads the SM clock at phase boundaries
    // (after a CTA barrier) and adds the cycles to prof[phase] at the end.
    const bool timing = KB.prof != nullptr;
    long long ph_t = 0;
    if (timing && tid == 0) {
#pragma unroll 1
        for (int k = 0; k < kNumPhases; ++k) s_ph[k] = 0ull;
        ph_t = clock64();
    }
    auto mark = [&](int phase) {
        if (timing && tid == 0) {
            const long long t = clock64();
            s_ph[phase] += static_cast<unsigned long long>(t - ph_t);
            ph_t = t;
        }
    };

    // ---- load constants and state ------------------------------------------
#pragma unroll 1
    for (int k = tid; k < Q * N; k += NT) {
        phi[k] = slab[L.phi + k];
        dphi[k] = slab[L.dphi + k];
        dphiJ[k] = slab[L.dphiJ + k];
    }
#pragma unroll 1
    for (int k = tid; k < Q * 4; k += NT) qpw[k] = slab[L.qpw + k];

#pragma unroll 1
    for (int k = tid; k < N * 7; k += NT) sq[k] = slab[L.q + k];
#pragma unroll 1
    for (int k = tid; k < N * 6; k += NT) {
        sv[k] = slab[L.v + k];
        svd[k] = slab[L.vd + k];
        sa[k] = slab[L.a + k];
    }
    if (tid < nc) {
        double* c = con + tid * kConStride;
        for (int k = 0; k < 7; ++k) c[conrec::inp + k] = slab[L.con_input + tid * 7 + k];
        for (int k = 0; k < 6; ++k) c[conrec::lam + k] = 0.;  // ResetConstraints
    }
    if (hub) {
#pragma unroll 1
        for (int k = tid; k < kHubDoubles; k += NT) hb[k] = slab[L.hub + k];
        if (tid == 0) {
            double* br = hb + hubsm::bc;
            for (int k = 0; k < 7; ++k) br[conrec::inp + k] = slab[L.hub + hubrec::input + k];
            for (int k = 0; k < 6; ++k) br[conrec::lam + k] = 0.;  // ResetConstraints
        }
    }
    if (drive) {
#pragma unroll 1
        for (int k = tid; k < (chain - 1) * kHubDoubles; k += NT)
            hb[hubsm::n1 + (k / kHubDoubles) * (hubsm::n2 - hubsm::n1) + k % kHubDoubles] =
                slab[L.hub + kHubDoubles + k];
        if (tid == 0)
            for (int k = 0; k < 6; ++k) {  // ResetConstraints
                hb[hubsm::rev + revrec::lam + k] = 0.;
                hb[hubsm::ah + conrec::lam + k] = 0.;
            }
    }
    if (tid < N) {  // free nodes first, constrained nodes last (in constraint order)
        int before = 0, at = -1;
#pragma unroll 1
        for (int c = 0; c < nc; ++c) {
            const int n = KB.con_node[c];
            before += n < tid;
            if (n == tid) at = N - nc + c;
        }
        if (at < 0) at = tid - before;
        pos[tid] = at;
        node_at[at] = tid;
    }
    if (tid == 0) {
        s_flag = 0;
        mbar_init(sec_bar);
    }
    __syncthreads();
    sec_issue();

    // ---- PredictNextState (src/step/predict_next_state.hpp:14-47) ------------
#pragma unroll 1
    for (int k = tid; k < N * 7; k += NT) sqp[k] = sq[k];
#pragma unroll 1
    for (int k = tid; k < N * 6; k += NT) {
        const double v_p = sv[k], vd_p = svd[k], a_p = sa[k];
        svd[k] = 0.;
        const double an = (P.alpha_f * vd_p - P.alpha_m * a_p) / (1. - P.alpha_m);
        sa[k] = an;
        sv[k] = v_p + h * (1. - P.gamma) * a_p + P.gamma * h * an;
        sqd[k] = v_p + (0.5 - P.beta) * h * a_p + P.beta * h * an;
    }
    // hub-chain records: thread NT-1-r owns record r (evaluated where used, so
    // that the instances without a drive train keep no extra register live)
    auto chain_rec = [&]() -> double* {
        return tid == NT - 1 ? hb : (tid == NT - 2) ? hA : (tid == NT - 3) ? hH : nullptr;
    };
    if (hub && chain_rec()) {  // the hub node(s): same predictor
        double* r = chain_rec();
        for (int k = 0; k < 7; ++k) r[hubrec::q_prev + k] = r[hubrec::q + k];
        for (int k = 0; k < 6; ++k) {
            const double v_p = r[hubrec::v + k], vd_p = r[hubrec::vd + k], a_p = r[hubrec::a + k];
            r[hubrec::vd + k] = 0.;
            const double an = (P.alpha_f * vd_p - P.alpha_m * a_p) / (1. - P.alpha_m);
            r[hubrec::a + k] = an;
            r[hubrec::v + k] = v_p + h * (1. - P.gamma) * a_p + P.gamma * h * an;
            r[hubrec::q_delta + k] = v_p + (0.5 - P.beta) * h * a_p + P.beta * h * an;
        }
    }
    __syncthreads();
    // CalculateDisplacement (src/state/calculate_displacement.hpp:25-50)
    auto displaced_rotation = [&](const double* qp, const double* qd, double* qn) {
        const double d[3] = {h * qd[3], h * qd[4], h * qd[5]};
        double qd4[4];
        rotvec_to_quat(d, qd4);
        quat_compose(qd4, qp + 3, qn);
    };
    auto displace = [&](int n, int c) {  // component c of q of node n
        if (c < 3) {
            sq[n * 7 + c] = sqp[n * 7 + c] + h * sqd[n * 6 + c];
        } else {
            double qn[4];
            displaced_rotation(sqp + n * 7, sqd + n * 6, qn);
            sq[n * 7 + c] = c == 3 ? qn[0] : c == 4 ? qn[1] : c == 5 ? qn[2] : qn[3];
        }
    };
    auto displace_chain = [&](double* r) {  // hub-chain record
        for (int c = 0; c < 3; ++c) r[hubrec::q + c] = r[hubrec::q_prev + c] + h * r[hubrec::q_delta + c];
        double qn[4];
        displaced_rotation(r + hubrec::q_prev, r + hubrec::q_delta, qn);
        for (int c = 0; c < 4; ++c) r[hubrec::q + 3 + c] = qn[c];
    };
#pragma unroll 1
    for (int t = tid; t < 8 * N; t += NT)
        if ((t & 7) < 7) displace(t >> 3, t & 7);
    if (hub && chain_rec()) displace_chain(chain_rec());
    __syncthreads();
    mark(kPhaseLoadPredict);

    int status = KYN_NOT_CONVERGED;
    int iters = 0;
    const cg::cluster_group cluster = cg::this_cluster();
    const bool clustered = KB.model_beams > 1;

    int extra = 0;  // refinement corrections taken after convergence (FP32 form)
#pragma unroll 1
    for (int iter = 0; iter < P.max_iter + extra; ++iter) {
        // ---- tangent operator (src/system/calculate_tangent_operator.hpp:26-65)
        // Only the rotational 3x3 block of the stored (transposed) operator is kept.
        auto tangent_op = [&](const double* qd, double* T) {
            const double rv[3] = {h * qd[3], h * qd[4], h * qd[5]};
            const double ph = sqrt(rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
            double sn, cs;
            sincos(ph, &sn, &cs);
            const double t1 = (ph > 1.e-16) ? (cs - 1.) / (ph * ph) : 0.;
            const double t2 = (ph > 1.e-16) ? (1. - sn / ph) / (ph * ph) : 0.;
            for (int i = 0; i < 3; ++i) {
                for (int j = 0; j < 3; ++j) {
                    // m1 = t2*(rv~ rv~) + t1*rv~ ; T_rot = I + m1 ; stored transposed
                    double rr = 0.;
                    for (int k = 0; k < 3; ++k) rr += tilde_e(rv, j, k) * tilde_e(rv, k, i);
                    T[i * 3 + j] = (i == j ? 1. : 0.) + (t1 * tilde_e(rv, j, i) + t2 * rr);
                }
            }
        };
        // The last warp forms the tangent operators, the constraint records
        // (calculate_constraint_residual_gradient.hpp:60-320) and the constrained
        // nodes' corrections B x_r = -Phi while the others do the quadrature
        // points: none of it needs their values, and its few lanes took 10k
        // cycles per iteration when the whole CTA waited for them.
        if (warp == NW - 1) {
            if (lane < N) tangent_op(sqd + lane * 6, sT + lane * 9);
            if (hub && chain_rec()) tangent_op(chain_rec() + hubrec::q_delta, chain_rec() + hubrec::tangent);
            __syncwarp();
            if (lane < nc) {
                const int tn = KB.con_node[lane];
                constraint_record(con + lane * kConStride, KB.con_type[lane], sq + tn * 7, KB.con_X0[lane],
                                  sT + tn * 9, hub ? hj + hubrec::q : nullptr,
                                  hub ? hj + hubrec::tangent : nullptr, KB.con_axis[lane]);
            }
            if (hub && lane == nc)  // the hub's own boundary condition
                constraint_record(hb + hubsm::bc, KB.hub_con_type, hb + hubrec::q, hb + hubrec::X0,
                                  hb + hubrec::tangent, nullptr, nullptr, nullptr);
            if (drive && lane == nc + 1)  // revolute joint record 0 -> 1
                revolute_record(hb + hubsm::rev, hb, hA);
            if (drive && hH && lane == nc + 2)  // rigid joint record 1 -> 2
                constraint_record(hb + hubsm::ah, KYN_CONSTRAINT_RIGID_JOINT, hH + hubrec::q, hH + hubrec::X0,
                                  hH + hubrec::tangent, hA + hubrec::q, hA + hubrec::tangent, nullptr);
            __syncwarp();
            // With a hub, its correction comes first (its BC rows), then each rigid
            // joint gives the root correction: B_t x_root = -Phi - B_base x_hub.
            if (hub) {
                if (lane == 0) {
                    const double* br = hb + hubsm::bc;
                    double* xh = hb + hubsm::xh;
                    for (int k = 0; k < 3; ++k) xh[k] = -br[conrec::Phi + k];
                    const double rhs[3] = {-br[conrec::Phi + 3], -br[conrec::Phi + 4], -br[conrec::Phi + 5]};
                    double y[3] = {0., 0., 0.};
                    if (!solve3(br + conrec::Brot, rhs, y)) atomicOr(&s_flag, 2);
                    for (int k = 0; k < 3; ++k) xh[3 + k] = y[k];
                    if (drive) {
                        // Drive train: the revolute rows fix record 1's translation and
                        // two of its rotation components; the third, the shaft rotation
                        // theta, stays free.  x_1 = cA + theta nA, nA spanning the null
                        // space of B_t; the chain's later corrections are affine in
                        // theta as well (cH + theta dH).  Test vectors w (G w = 0 with
                        // the gradients G, not G T) project the equilibrium rows onto
                        // the free rotation: w_1 = [0, joint axis].
                        const double* rv = hb + hubsm::rev;
                        double* cA = hb + hubsm::cA;
                        double* nA = hb + hubsm::nA;
                        double* wA = hb + hubsm::wA;
                        for (int k = 0; k < 3; ++k) {
                            cA[k] = -rv[revrec::Phi + k] + xh[k];
                            nA[k] = 0.;
                            wA[k] = 0.;
                            wA[3 + k] = rv[revrec::x + k];
                        }
                        const double* b0 = rv + revrec::Bt;
                        const double* b1 = rv + revrec::Bt + 3;
                        double r2[2];
                        for (int i = 0; i < 2; ++i) {
                            r2[i] = -rv[revrec::Phi + 3 + i];
                            for (int k = 0; k < 3; ++k) r2[i] -= rv[revrec::Bb + i * 3 + k] * xh[3 + k];
                        }
                        // minimum-norm particular solution B_t^T (B_t B_t^T)^-1 r2
                        const double g00 = b0[0] * b0[0] + b0[1] * b0[1] + b0[2] * b0[2];
                        const double g01 = b0[0] * b1[0] + b0[1] * b1[1] + b0[2] * b1[2];
                        const double g11 = b1[0] * b1[0] + b1[1] * b1[1] + b1[2] * b1[2];
                        const double det = g00 * g11 - g01 * g01;
                        if (!(fabs(det) > 0.)) atomicOr(&s_flag, 2);
                        const double l0 = (g11 * r2[0] - g01 * r2[1]) / det;
                        const double l1 = (g00 * r2[1] - g01 * r2[0]) / det;
                        for (int k = 0; k < 3; ++k) cA[3 + k] = b0[k] * l0 + b1[k] * l1;
                        nA[3] = b0[1] * b1[2] - b0[2] * b1[1];
                        nA[4] = b0[2] * b1[0] - b0[0] * b1[2];
                        nA[5] = b0[0] * b1[1] - b0[1] * b1[0];
                        if (hH) {
                            const double* ah = hb + hubsm::ah;
                            bool ok = joint_target_correction(ah, cA, 1., hb + hubsm::cH);
                            ok &= joint_target_correction(ah, nA, 0., hb + hubsm::dH);
                            ok &= joint_target_test(ah, wA, hb + hubsm::wH);
                            if (!ok) atomicOr(&s_flag, 2);
                        }
                    }
                }
                __syncwarp();
            }
            if (drive && lane < nc) {
                // roots: x_root = c_r + theta d_r from the corrections of the record
                // they join; d_r waits in droot for the second right-hand side
                double* cr = con + lane * kConStride;
                const int pr = 6 * pos[KB.con_node[lane]];
                double c6[6], d6[6];
                if (is_hub_joint(KB.con_type[lane])) {
                    const double* cb = hb + (hH ? hubsm::cH : hubsm::cA);
                    const double* db = hb + (hH ? hubsm::dH : hubsm::nA);
                    bool ok = joint_target_correction(cr, cb, 1., c6);
                    ok &= joint_target_correction(cr, db, 0., d6);
                    ok &= joint_target_test(cr, hb + (hH ? hubsm::wH : hubsm::wA), cr + conrec::wr);
                    if (!ok) atomicOr(&s_flag, 2);
                } else {
                    for (int k = 0; k < 3; ++k) {
                        c6[k] = -cr[conrec::Phi + k];
                        d6[k] = d6[3 + k] = 0.;
                    }
                    const double rr[3] = {-cr[conrec::Phi + 3], -cr[conrec::Phi + 4], -cr[conrec::Phi + 5]};
                    if (!solve3(cr + conrec::Brot, rr, c6 + 3)) atomicOr(&s_flag, 2);
                    for (int k = 0; k < 6; ++k) cr[conrec::wr + k] = 0.;
                }
                for (int k = 0; k < 6; ++k) {
                    xs[pr + k] = c6[k];
                    droot[pr + k] = d6[k];
                    cr[conrec::dr + k] = d6[k];
                }
            } else if (lane < nc) {
                const double* cr = con + lane * kConStride;
                const int pr = 6 * pos[KB.con_node[lane]];
                double rt[3], rr[3];
                for (int k = 0; k < 3; ++k) {
                    rt[k] = -cr[conrec::Phi + k];
                    rr[k] = -cr[conrec::Phi + 3 + k];
                }
                if (is_hub_joint(KB.con_type[lane])) {
                    const double* xh = hb + hubsm::xh;
                    for (int i = 0; i < 3; ++i) {
                        rt[i] += xh[i];
                        for (int k = 0; k < 3; ++k) {
                            rt[i] -= cr[conrec::Btr + i * 3 + k] * xh[3 + k];
                            rr[i] -= cr[conrec::Brr + i * 3 + k] * xh[3 + k];
                        }
                    }
                }
                for (int k = 0; k < 3; ++k) xs[pr + k] = rt[k];
                double y[3] = {0., 0., 0.};
                if (!solve3(cr + conrec::Brot, rr, y)) atomicOr(&s_flag, 2);
                for (int k = 0; k < 3; ++k) xs[pr + 3 + k] = y[k];
            }
            sec_wait();
        } else {
            // ---- quadrature-point values (calculate_quadrature_point_values.hpp) ---
            sec_wait();
            qp_phase<TG, NW - 1, false>(N, Q, phi, dphiJ, qpw, sq, sv, svd, slab, L, KB.gravity, P.beta_prime,
                                        P.gamma_prime, P.conditioner, itp, G, Fc, Fdig, bulk ? sec : nullptr);
        }
        __syncthreads();
        mark(kPhaseQuadrature);

        // ---- residual integration (integrate_residual_vector.hpp:33-50) ----------
#pragma unroll 1
        for (int t = NT - 1 - tid; t < N * 6; t += NT) {  // the last warps have fewer pair units
            const int n = t / 6, c = t % 6;
            double acc = 0.;
#pragma unroll 1
            for (int qp = 0; qp < Q; ++qp) {
                const double w = qpw[qp * 4], wJ = qpw[qp * 4 + 2];
                acc += (w * dphi[qp * N + n]) * Fc[qp * 6 + c] +
                       (wJ * phi[qp * N + n]) * Fdig[qp * 6 + c];
            }
            resid[t] = acc - slab[L.fx + t];
        }

        // ---- stiffness + inertia integration and S T + I, scaled by the conditioner
        //      into A (the residual's inputs stay untouched)
        if constexpr (sizeof(TR) == 4)
            integrate_node_pairs_fp32<NT>(N, Q, phi, dphi, G, A, ldA, pos, sT, P.conditioner);
        else
            integrate_node_pairs<NT>(
                N, Q, phi, dphi, G, [&](int j) { return sT + j * 9; },
                [&](int j, int r, int half) {
                    return [=](int i, double v0, double v1, double v2) {
                        const int row = 6 * pos[i] + r, col = 6 * pos[j] + 3 * half, sh = row & 6;
                        double* a = A + row * ldA;
                        a[col ^ sh] = v0;
                        a[(col + 1) ^ sh] = v1;
                        a[(col + 2) ^ sh] = v2;
                    };
                });
        __syncthreads();
        if (LUMP && KB.n_mass + KB.n_spring > 0) {  // point masses and springs at this CTA's nodes
#pragma unroll 1
            for (int n = tid; n < N; n += NT)
                add_lumped_terms(n, KB.lumped, KB.n_mass, KB.n_spring, sq, sv, svd, sT, KB.gravity,
                                 P.beta_prime, P.gamma_prime, P.conditioner, pos,
                                 [&](int r, int c) -> TR& { return A[sys_at<TR>(ldA, r, c)]; }, resid);
            __syncthreads();
        }
        mark(kPhaseIntegrate);

        if (record && KB.dump) {
            // Dump of the assembled local system (natural node order, then constraints):
            // matrix [nl][nl], then rhs [nl], then solution [nl]; nl = n6 + 6 nc.
            const int nl = n6 + 6 * nc;
            double* D = KB.dump;
#pragma unroll 1
            for (int t = tid; t < nl * nl; t += NT) D[t] = 0.;
        }
        if (record) __syncthreads();
        if (record && KB.dump) {
            const int nl = n6 + 6 * nc;
            double* D = KB.dump;
#pragma unroll 1
            for (int t = tid; t < n6 * n6; t += NT) {
                const int r = t / n6, c = t % n6;
                D[r * nl + c] = static_cast<double>(
                    A[sys_at<TR>(ldA, 6 * pos[r / 6] + r % 6, 6 * pos[c / 6] + c % 6)]);
            }
            if (tid < nc) {
                const double* cr = con + tid * kConStride;
                const int tn = KB.con_node[tid];
                const int r0 = n6 + 6 * tid;
                for (int k = 0; k < 3; ++k) {
                    D[(r0 + k) * nl + 6 * tn + k] = 1.;            // B translational block
                    D[(6 * tn + k) * nl + r0 + k] = 1.;            // grad^T translational block
                }
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; j < 3; ++j) {
                        D[(r0 + 3 + i) * nl + 6 * tn + 3 + j] = cr[conrec::Brot + i * 3 + j];
                        D[(6 * tn + 3 + i) * nl + r0 + 3 + j] = cr[conrec::AX + i * 3 + j];
                    }
                for (int k = 0; k < 6; ++k) D[nl * nl + r0 + k] = -cr[conrec::Phi + k];
            }
        }

        mark(kPhaseConstraints);

        // ---- solve -----------------------------------------------------------------
        // ---- right-hand side b = -cond (-f + R + G^T lambda) (assemble_system_residual.hpp,
        //      solve_system.hpp:20-24) in permuted order; the free rows' part
        //      -A_fr x_r of the constrained corrections folded in, in column m of A
        //      (and in FP64 in bp[0:m]); a drive train adds the second right-hand
        //      side -A_fr d_r in column m + 1 (FP64 copy in rhs2)
        double* gjv = reinterpret_cast<double*>(smem_raw + S.G + solve_vec_offset(N, nc, sizeof(TR), NT, drive ? 2 : 0));
        double* r64 = gjv;                 // [n6] residual of the linear solve
        double* rhs2 = gjv + n6;           // [n6] second right-hand side (drive train)
        double* x2 = gjv + 2 * n6;         // [n6] its solution
        double* red4 = gjv + 4 * n6;       // [64] reductions of the refinement
        // (eight lanes per row: the rows start in only two different banks)
#pragma unroll 1
        for (int i0 = 4 * warp; i0 < n6; i0 += 4 * NW) {
            const int i = i0 + (lane >> 3), ic = min(i, n6 - 1);
            double r = 0., r2 = 0.;
            if (i0 < m) {
#pragma unroll 1
                for (int j = m + (lane & 7); j < n6; j += 8) {
                    const double aij = static_cast<double>(A[sys_at<TR>(ldA, ic, j)]);
                    r -= aij * xs[j];
                    if (drive) r2 -= aij * droot[j];
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) {
                    r += __shfl_xor_sync(0xffffffffu, r, o);
                    if (drive) r2 += __shfl_xor_sync(0xffffffffu, r2, o);
                }
            }
            if ((lane & 7) == 0 && i < n6) {
                const int t = 6 * node_at[i / 6] + i % 6;
                double val = -slab[L.f + t] + resid[t];
                if (i >= m) val += con[((i - m) / 6) * kConStride + conrec::Gl + i % 6];
                double b = -(val * P.conditioner);
                if (record && KB.dump) KB.dump[(n6 + 6 * nc) * (n6 + 6 * nc) + t] = b;
                if (i < m) {
                    b += r;
                    A[sys_at<TR>(ldA, i, m)] = static_cast<TR>(b);
                    if (drive) {
                        A[sys_at<TR>(ldA, i, m + 1)] = static_cast<TR>(r2);
                        rhs2[i] = r2;
                    }
                }
                bp[i] = b;
            }
        }
        __syncthreads();
        mark(kPhaseEliminate);
        // (S3) the free block: Gauss-Jordan in registers where it fits the grid
        //      (FP64 form: solve; FP32 form: inverse, then FP64-residual
        //      refinement), else the elimination in shared memory (FP64 form: by 8x8
        //      blocks; FP32 form: panel LU).  x1 -> xs[0:m], x2 -> x2[0:m].
        constexpr bool kInv = sizeof(TR) == 4;
        const int nrhs = drive ? 2 : 1;
        const bool use_gj = GJ && P.solver == KYN_SOLVER_GAUSS_JORDAN && m > 0 && (m & 1) == 0 &&
                            gj_fits<TR, NT>(m, kInv ? m : m + nrhs);
        if (use_gj) {
          if constexpr (GJ) {
            TR R[GJTile<TR, NT>::RT][GJTile<TR, NT>::CT];
            TR* pivots = reinterpret_cast<TR*>(smem_raw + S.G);
            gj_eliminate<TR, NT, kInv>(A, ldA, m, nrhs, pivots, &s_flag, R);
            mark(kPhaseFactor);
            // Backward error of a solve: max|b - A x| / (||A|| ||x|| + ||b||),
            // infinity norms, FP64, A as assembled (its FP32 rounding in the
            // FP32 form).  Returns the same value in every thread.
            auto backward_error = [&](const double* x, const double* b, double* res) -> double {
                double ra = 0., xa = 0., ba = 0., aa = 0.;
                constexpr int PR = NT / kGJCols;
                const int ri = tid / kGJCols, cj = tid % kGJCols;
#pragma unroll
                for (int a = 0; a < GJTile<TR, NT>::RT; ++a) {
                    const int i = ri + a * PR;
                    if (a * PR >= m) break;
                    double acc = 0., asum = 0.;
#pragma unroll
                    for (int bb = 0; bb < GJTile<TR, NT>::CT; ++bb) {
                        const int j = cj + bb * kGJCols;
                        if (j < m && i < m) {
                            const double aij = static_cast<double>(A[sys_at<TR>(ldA, i, j)]);
                            acc = fma(aij, x[j], acc);
                            asum += fabs(aij);
                            if (a == 0) xa = fmax(xa, fabs(x[j]));
                        }
                    }
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) {
                        acc += __shfl_xor_sync(0xffffffffu, acc, o);
                        asum += __shfl_xor_sync(0xffffffffu, asum, o);
                    }
                    if (i < m) {
                        const double rv = b[i] - acc;
                        if (cj == 0) res[i] = rv;
                        ra = fmax(ra, fabs(rv));
                        ba = fmax(ba, fabs(b[i]));
                        aa = fmax(aa, asum);
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    ra = fmax(ra, __shfl_xor_sync(0xffffffffu, ra, o));
                    xa = fmax(xa, __shfl_xor_sync(0xffffffffu, xa, o));
                    ba = fmax(ba, __shfl_xor_sync(0xffffffffu, ba, o));
                    aa = fmax(aa, __shfl_xor_sync(0xffffffffu, aa, o));
                }
                if (lane == 0) {
                    red4[4 * warp] = ra;
                    red4[4 * warp + 1] = xa;
                    red4[4 * warp + 2] = ba;
                    red4[4 * warp + 3] = aa;
                }
                __syncthreads();
                ra = xa = ba = aa = 0.;
#pragma unroll 1
                for (int w2 = 0; w2 < NW; ++w2) {
                    ra = fmax(ra, red4[4 * w2]);
                    xa = fmax(xa, red4[4 * w2 + 1]);
                    ba = fmax(ba, red4[4 * w2 + 2]);
                    aa = fmax(aa, red4[4 * w2 + 3]);
                }
                __syncthreads();  // red4 is reused by the next call
                const double den = aa * xa + ba;
                return den > 0. ? ra / den : 0.;
            };
            if constexpr (!kInv) {
                // guard of the unpivoted elimination: the backward error of the
                // solve; above kGJBackwardErrorMax (element growth) the block,
                // which shared memory still holds, is solved with row pivoting,
                // and its residual once more (Gauss-Jordan's residual grows with
                // the condition number even when pivoted).
                // (One right-hand side: a drive train runs the LUMP instance.)
                gj_extract<TR, NT>(R, m, m, xs);
                __syncthreads();
                double eta = backward_error(xs, bp, r64);
                if (eta > kGJBackwardErrorMax) {
                    double* dx = gjv + 3 * n6;
                    for (int pass = 0; pass < 2; ++pass) {
                        gj_solve_pivoted<TR, NT>(A, ldA, m, pivots, pass ? dx : xs, &s_flag);
#pragma unroll 1
                        for (int i = tid; pass && i < m; i += NT) xs[i] += dx[i];
                        __syncthreads();
                        eta = backward_error(xs, bp, r64);
#pragma unroll 1
                        for (int i = tid; i < m; i += NT) A[sys_at<TR>(ldA, i, m)] = r64[i];
                        __syncthreads();
                    }
                }
                // counted: checked, still above the limit, largest
                if (tid == 0 && P.diag) {
                    atomicAdd(P.diag + kDiagChecked, 1ull);
                    if (!(eta <= kGJBackwardErrorMax)) atomicAdd(P.diag + kDiagGuardTrips, 1ull);
                    if (eta == eta)
                        atomicMax(P.diag + kDiagMaxBackwardError,
                                  static_cast<unsigned long long>(__double_as_longlong(eta)));
                }
            } else {
                // FP32 inverse in R; x = R b, then sweeps x += R (b - A x) with
                // the residual in FP64 until its backward error is at most
                // refine_tol (or refine_sweeps sweeps)
#pragma unroll 1
                for (int rhs = 0; rhs < nrhs; ++rhs) {
                    double* x = rhs ? x2 : xs;
                    const double* b = rhs ? rhs2 : bp;
                    double amax;
                    gj_matvec<TR, NT, true>(R, A, ldA, m, b, nullptr, x, amax);
                    __syncthreads();
#pragma unroll 1
                    for (int sweep = 1;; ++sweep) {
                        const double eta = backward_error(x, b, r64);
                        const bool done = eta <= P.refine_tol;
                        if (tid == 0 && P.diag) {
                            if (done || sweep > P.refine_sweeps) {
                                atomicAdd(P.diag + kDiagChecked, 1ull);
                                if (eta == eta)
                                    atomicMax(P.diag + kDiagMaxBackwardError,
                                              static_cast<unsigned long long>(__double_as_longlong(eta)));
                            }
                            if (!done && sweep > P.refine_sweeps) atomicAdd(P.diag + kDiagRefineShort, 1ull);
                            if (!done && sweep <= P.refine_sweeps) atomicAdd(P.diag + kDiagRefineSweeps, 1ull);
                        }
                        if (done || sweep > P.refine_sweeps) break;
                        // x += R r: one row group's 16 threads sum their columns
                        constexpr int PR = NT / kGJCols;
                        const int ri = tid / kGJCols, cj = tid % kGJCols;
#pragma unroll
                        for (int a = 0; a < GJTile<TR, NT>::RT; ++a) {
                            const int i = ri + a * PR;
                            if (a * PR >= m) break;
                            double acc = 0.;
#pragma unroll
                            for (int bb = 0; bb < GJTile<TR, NT>::CT; ++bb) {
                                const int j = cj + bb * kGJCols;
                                if (j < m) acc = fma(static_cast<double>(R[a][bb]), r64[j], acc);
                            }
#pragma unroll
                            for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                            if (cj == 0 && i < m) x[i] += acc;
                        }
                        __syncthreads();
                    }
                }
                mark(kPhaseRefine);
            }
          }
        } else {
            if (m > 0) {
                if constexpr (sizeof(TR) == 4) {
                    // panel LU; the back substitution with the diagonal blocks of U inverted
                    // (every warp some of them), by warp 0 block by block; a drive train's
                    // second right-hand side before they are
                    double* rpiv = reinterpret_cast<double*>(smem_raw + S.G);
                    factor_fp32<NT>(A, ldA, m, rpiv, rpiv + n6, &s_flag);
                    mark(kPhaseFactor);
                    if (drive) {
                        if (warp == 0) solve_factored_column(A, ldA, m, m + 1, rpiv, lane);
                        __syncthreads();
                        for (int i = tid; i < m; i += NT) x2[i] = static_cast<double>(A[i * ldA + m + 1]);
                    }
                    for (int b = warp; b * kPanel < m; b += NW) invert_diag_block(A, ldA, m, b * kPanel, rpiv, lane);
                    __syncthreads();
                    if (warp == 0) back_substitute_blocked(A, ldA, m, xs, lane);
                    __syncthreads();
                } else {
                    // block elimination, then the back substitution of each right-hand side
                    double* dinv = reinterpret_cast<double*>(smem_raw + S.G);
                    eliminate_blocks<NT>(A, ldA, m, (m + 7) >> 3, (m + nrhs + 7) >> 3, dinv, &s_flag);
                    mark(kPhaseFactor);
                    for (int i = tid; i < m; i += NT) {
                        xs[i] = A[sys_at<TR>(ldA, i, m)];
                        if (drive) x2[i] = A[sys_at<TR>(ldA, i, m + 1)];
                    }
                    __syncthreads();
                    back_substitute<NT>(A, ldA, m, xs);
                    if (drive) back_substitute<NT>(A, ldA, m, x2);
                }
            }
            mark(kPhaseBackSubstitute);
        }
        if (drive) {
            // Shaft rotation theta: x = x1 + theta x2 (x1 = (y1, c_r), x2 = (y2, d_r)).
            // The equilibrium rows projected on the test vectors lose every
            // multiplier term (G w = 0 joint by joint), leaving
            //   sum_roots w_r.(b_r - A_r x) + sum_chain w_n.b_n = 0,
            // b_n = -cond (sum of G^T lambda at the node + torque); chain nodes
            // carry no element terms.
#pragma unroll 1
            for (int rowi = warp; rowi < 6 * nc; rowi += NW) {
                const int c = rowi / 6, k = rowi % 6;
                const int pr = 6 * pos[KB.con_node[c]];
                double a1 = 0., a2 = 0.;
#pragma unroll 1
                for (int j = lane; j < n6; j += 32) {
                    const double arj = static_cast<double>(A[sys_at<TR>(ldA, pr + k, j)]);
                    a1 += arj * xs[j];
                    a2 += arj * (j < m ? x2[j] : droot[j]);
                }
                for (int o = 16; o > 0; o >>= 1) {
                    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
                    a2 += __shfl_xor_sync(0xffffffffu, a2, o);
                }
                if (lane == 0) {
                    con[c * kConStride + conrec::yr + k] = bp[pr + k] - a1;
                    con[c * kConStride + conrec::s2 + k] = a2;
                }
            }
            __syncthreads();
            double* xt = hb + hubsm::xt + 8 * (iter & 1);
            if (tid == 0) {  // this beam's roots: w.s1, w.s2 and G_base^T lambda
                for (int k = 0; k < 8; ++k) xt[k] = 0.;
#pragma unroll 1
                for (int c = 0; c < nc; ++c) {
                    const double* cr = con + c * kConStride;
                    for (int k = 0; k < 6; ++k) {
                        xt[0] += cr[conrec::wr + k] * cr[conrec::yr + k];
                        xt[1] += cr[conrec::wr + k] * cr[conrec::s2 + k];
                    }
                    if (is_hub_joint(KB.con_type[c])) joint_base_transpose_add(cr, cr + conrec::lam, xt + 2);
                }
            }
            if (clustered) cluster.sync(); else __syncthreads();
            if (tid == 0) {
                // every CTA sums the beams' parts in rank order, so all find the same theta
                double num = 0., den = 0.;
                double gj[6] = {0., 0., 0., 0., 0., 0.};  // roots' G_base^T lambda
#pragma unroll 1
                for (int r = 0; r < KB.model_beams; ++r) {
                    const double* peer = clustered ? cluster.map_shared_rank(xt, r) : xt;
                    num += peer[0];
                    den += peer[1];
                    for (int k = 0; k < 6; ++k) gj[k] += peer[2 + k];
                }
                const double* rv = hb + hubsm::rev;
                double bA[6];
                for (int k = 0; k < 6; ++k) bA[k] = rv[revrec::GtL + k] + (k >= 3 ? rv[revrec::sys + k - 3] : 0.);
                if (hH) {
                    const double* ah = hb + hubsm::ah;
                    joint_base_transpose_add(ah, ah + conrec::lam, bA);
                    for (int k = 0; k < 6; ++k)
                        num -= hb[hubsm::wH + k] * P.conditioner * (ah[conrec::Gl + k] + gj[k]);
                } else {
                    for (int k = 0; k < 6; ++k) bA[k] += gj[k];
                }
                for (int k = 0; k < 6; ++k) num -= hb[hubsm::wA + k] * P.conditioner * bA[k];
                if (!(fabs(den) > 0.)) atomicOr(&s_flag, 2);
                hb[hubsm::theta] = num / den;
            }
            __syncthreads();
            const double th = hb[hubsm::theta];
#pragma unroll 1
            for (int i = tid; i < m; i += NT) xs[i] += th * x2[i];
#pragma unroll 1
            for (int t = tid; t < 6 * nc; t += NT) {
                const int pr = 6 * pos[KB.con_node[t / 6]];
                xs[pr + t % 6] += th * droot[pr + t % 6];
            }
            __syncthreads();
        }
        // (S5) The last warp: multipliers from the constrained rows, grad^T x_l =
        //      b_r - A_r x, and their part of the error.  The others: error and
        //      update of the nodes (calculate_error_sum_squares.hpp:33-79,
        //      update_dynamic_prediction.hpp, calculate_displacement.hpp), eight
        //      lanes to a node.
        double part = 0.;
        if (warp == NW - 1) {
#pragma unroll 1
            for (int c = 0; c < nc; ++c) {
                const int pr = m + 6 * c;
                double y[6] = {0., 0., 0., 0., 0., 0.};
#pragma unroll 1
                for (int j = lane; j < n6; j += 32) {
                    const double xj = xs[j];
#pragma unroll
                    for (int k = 0; k < 6; ++k) y[k] += static_cast<double>(A[sys_at<TR>(ldA, pr + k, j)]) * xj;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int k = 0; k < 6; ++k) y[k] += __shfl_xor_sync(0xffffffffu, y[k], o);
                double* cr = con + c * kConStride;
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    if (lane == k) cr[conrec::yr + k] = bp[pr + k] - y[k];
            }
            __syncwarp();
            if (lane < nc) {
                double* cr = con + lane * kConStride;
                const double* y = cr + conrec::yr;
                double yr[3] = {0., 0., 0.};
                if (!solve3(cr + conrec::AX, y + 3, yr)) atomicOr(&s_flag, 2);
                // UnconditionSolution (condition_system.hpp): x_lambda /= conditioner
                const double ic = 1. / P.conditioner;
                for (int k = 0; k < 3; ++k) {
                    cr[conrec::xl + k] = y[k] * ic;
                    cr[conrec::xl + 3 + k] = yr[k] * ic;
                }
            }
            __syncwarp();
            if (hub && lane == 0) {
                // this beam's part of the hub rows: sum over its joints of
                // G_base^T (lambda + x_lambda), exchanged over the cluster below
                double* pub = hb + hubsm::pub + 6 * (iter & 1);
                for (int k = 0; k < 6; ++k) pub[k] = 0.;
#pragma unroll 1
                for (int c = 0; c < nc; ++c) {
                    if (!is_hub_joint(KB.con_type[c])) continue;
                    const double* cr = con + c * kConStride;
                    double w[6];
                    for (int k = 0; k < 6; ++k) w[k] = cr[conrec::lam + k] + cr[conrec::xl + k];
                    joint_base_transpose_add(cr, w, pub);
                }
            }
            if (record && KB.dump) {
                const int nl = n6 + 6 * nc;
                double* D = KB.dump + nl * nl + nl;
#pragma unroll 1
                for (int t = lane; t < n6; t += 32) D[t] = xs[6 * pos[t / 6] + t % 6];
                if (lane < nc)
                    for (int k = 0; k < 6; ++k) D[n6 + 6 * lane + k] = con[lane * kConStride + conrec::xl + k];
            }
#pragma unroll 1
            for (int t = lane; t < 6 * nc; t += 32) {
                double* cr = con + (t / 6) * kConStride;
                const double lam = cr[conrec::lam + t % 6], xl = cr[conrec::xl + t % 6];
                const double e = xl / (P.atol + P.rtol * fabs(lam));
                part += e * e;
                if (!hub) cr[conrec::lam + t % 6] = lam + xl;  // update_lambda_prediction.hpp
            }
        } else {
#pragma unroll 1
            for (int n0 = 4 * warp; n0 < N; n0 += 4 * (NW - 1)) {
                const int n = n0 + (lane >> 3), c = lane & 7, t = 6 * n + c;
                if (n < N && c < 6) {
                    const double delta = xs[6 * pos[n] + c], qd = sqd[t];
                    const double e = delta / (P.atol + P.rtol * fabs(qd * h));
                    part += e * e;
                    sqd[t] = qd + delta / h;
                    if (P.dynamic) {
                        sv[t] += P.gamma_prime * delta;
                        svd[t] += P.beta_prime * delta;
                    }
                }
                __syncwarp();
                if (n < N && c < 7) displace(n, c);
            }
        }
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        // per warp its part, then the flags; each CTA of the model sums all of
        // them in the same order
        double* slot = red + (iter & 1) * (NW + 8);
        if (lane == 0) slot[warp] = part;
        if (tid == NT - 1) slot[NW] = static_cast<double>(*static_cast<volatile int*>(&s_flag));
        proxy_fence_async_smem();
        if (clustered) cluster.sync(); else __syncthreads();
        sec_issue();  // A is not read again in this iteration
        mark(kPhaseSubstitute);
        double total = 0., flags = 0.;
#pragma unroll 1
        for (int k = lane; k < KB.model_beams * (NW + 1); k += 32) {
            const int r = k / (NW + 1), w2 = k - r * (NW + 1);
            const double v = clustered ? *cluster.map_shared_rank(slot + w2, r) : slot[w2];
            if (w2 < NW) total += v;
            else flags = fmax(flags, v);
        }
        for (int o = 16; o > 0; o >>= 1) {
            total += __shfl_xor_sync(0xffffffffu, total, o);
            flags = fmax(flags, __shfl_xor_sync(0xffffffffu, flags, o));
        }
        double xlh[6] = {0., 0., 0., 0., 0., 0.};
        if (hub) {
            // Hub rows have no element terms: G_hub^T x_lh = -G_hub^T lambda_hub -
            // sum_j G_base,j^T (lambda_j + x_lj), summed over the beams in rank order.
            double sum[6] = {0., 0., 0., 0., 0., 0.};
#pragma unroll 1
            for (int r = 0; r < KB.model_beams; ++r) {
                const double* peer = clustered ? cluster.map_shared_rank(hb + hubsm::pub + 6 * (iter & 1), r)
                                               : hb + hubsm::pub + 6 * (iter & 1);
                for (int k = 0; k < 6; ++k) sum[k] += peer[k];
            }
            if (drive) {
                // Drive train, from the roots back to the BC: record 2's rows give
                // the rigid joint's multipliers, record 1's rows (with the torque)
                // the revolute's five (least squares on the three rotation rows,
                // consistent once theta balances them), and G_rev,base^T L_rev
                // is what record 0's BC carries.
                double sumA[6];
                if (hH) {
                    const double* ah = hb + hubsm::ah;
                    double L[6];
                    for (int k = 0; k < 3; ++k) L[k] = -sum[k];
                    const double rr[3] = {-sum[3], -sum[4], -sum[5]};
                    if (!solve3(ah + conrec::AX, rr, L + 3)) flags = 1.;
                    for (int k = 0; k < 6; ++k) sumA[k] = 0.;
                    joint_base_transpose_add(ah, L, sumA);
                    for (int k = 0; k < 6; ++k) {
                        const double xl = L[k] - ah[conrec::lam + k];
                        const double e = xl / (P.atol + P.rtol * fabs(ah[conrec::lam + k]));
                        total += e * e;
                        if (tid == NT - 3) hb[hubsm::ah + conrec::xl + k] = xl;
                    }
                } else {
                    for (int k = 0; k < 6; ++k) sumA[k] = sum[k];
                }
                const double* rv = hb + hubsm::rev;
                double g[6];
                for (int k = 0; k < 6; ++k) g[k] = -sumA[k] - (k >= 3 ? rv[revrec::sys + k - 3] : 0.);
                const double* u = rv + revrec::xcz;
                const double* w = rv + revrec::xcy;
                const double a00 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
                const double a01 = u[0] * w[0] + u[1] * w[1] + u[2] * w[2];
                const double a11 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
                const double r0 = -(u[0] * g[3] + u[1] * g[4] + u[2] * g[5]);
                const double r1 = -(w[0] * g[3] + w[1] * g[4] + w[2] * g[5]);
                const double det = a00 * a11 - a01 * a01;
                if (!(fabs(det) > 0.)) flags = 1.;
                const double L[5] = {g[0], g[1], g[2], (a11 * r0 - a01 * r1) / det, (a00 * r1 - a01 * r0) / det};
                for (int k = 0; k < 5; ++k) {
                    const double xl = L[k] - rv[revrec::lam + k];
                    const double e = xl / (P.atol + P.rtol * fabs(rv[revrec::lam + k]));
                    total += e * e;
                    if (tid == NT - 2) hb[hubsm::rev + revrec::xl + k] = xl;
                }
                for (int k = 0; k < 3; ++k) {
                    sum[k] = -L[k];
                    sum[3 + k] = u[k] * L[3] + w[k] * L[4];
                }
                // the chain nodes' terms of the error sum
                const double th = hb[hubsm::theta];
#pragma unroll 1
                for (int r = 1; r < chain; ++r) {
                    const double* rec = r == 1 ? hA : hH;
                    const double* c0 = hb + (r == 1 ? hubsm::cA : hubsm::cH);
                    const double* d0 = hb + (r == 1 ? hubsm::nA : hubsm::dH);
                    for (int k = 0; k < 6; ++k) {
                        const double e = (c0[k] + th * d0[k]) / (P.atol + P.rtol * fabs(rec[hubrec::q_delta + k] * h));
                        total += e * e;
                    }
                }
            }
            const double* br = hb + hubsm::bc;
            for (int k = 0; k < 3; ++k) xlh[k] = -br[conrec::lam + k] - sum[k];
            double yr[3] = {0., 0., 0.};
            if (!solve3(br + conrec::AX, sum + 3, yr)) flags = 1.;
            for (int k = 0; k < 3; ++k) xlh[3 + k] = -br[conrec::lam + 3 + k] - yr[k];
            // the hub's own terms of the error sum (every CTA adds the same values)
            const double* xh = hb + hubsm::xh;
            const double* hqd = hb + hubrec::q_delta;
            for (int k = 0; k < 6; ++k) {
                const double e1 = xh[k] / (P.atol + P.rtol * fabs(hqd[k] * h));
                const double e2 = xlh[k] / (P.atol + P.rtol * fabs(br[conrec::lam + k]));
                total += e1 * e1 + e2 * e2;
            }
            // Every thread formed these sums from this CTA's hub record, which the
            // last warp changes below and, in the next iteration, forms anew beside
            // the quadrature points: it waits until all have read it, else they could
            // find another error and leave the loop at another iteration.  (As a
            // branch of its own the barrier cost models without a hub 2 %.)
            __syncthreads();
        }
        const double err = sqrt(total / static_cast<double>(KB.model_dofs));
        if (KB.rank == 0 && tid == 0 && iter < kMaxNewtonIters) KB.conv[iter] = err;
        iters = iter + 1;

        // ---- update of the hub chain and, with a hub, of the multipliers (read by
        //      the peers' sums above only through pub)
        if (hub && warp == NW - 1)
#pragma unroll 1
            for (int t = lane; t < 6 * nc; t += 32) {
                double* cr = con + (t / 6) * kConStride;
                cr[conrec::lam + t % 6] += cr[conrec::xl + t % 6];
            }
        if (hub && tid == NT - 1) {
            const double* xh = hb + hubsm::xh;
            for (int k = 0; k < 6; ++k) {
                hb[hubrec::q_delta + k] += xh[k] / h;
                if (P.dynamic) {
                    hb[hubrec::v + k] += P.gamma_prime * xh[k];
                    hb[hubrec::vd + k] += P.beta_prime * xh[k];
                }
                hb[hubsm::bc + conrec::lam + k] += xlh[k];
            }
        }
        if (drive && (tid == NT - 2 || tid == NT - 3) && chain_rec()) {
            double* my_rec = chain_rec();
            const double th = hb[hubsm::theta];
            const double* c0 = hb + (tid == NT - 2 ? hubsm::cA : hubsm::cH);
            const double* d0 = hb + (tid == NT - 2 ? hubsm::nA : hubsm::dH);
            for (int k = 0; k < 6; ++k) {
                const double x = c0[k] + th * d0[k];
                my_rec[hubrec::q_delta + k] += x / h;
                if (P.dynamic) {
                    my_rec[hubrec::v + k] += P.gamma_prime * x;
                    my_rec[hubrec::vd + k] += P.beta_prime * x;
                }
            }
            if (tid == NT - 2)
                for (int k = 0; k < 5; ++k) hb[hubsm::rev + revrec::lam + k] += hb[hubsm::rev + revrec::xl + k];
            else
                for (int k = 0; k < 6; ++k) hb[hubsm::ah + conrec::lam + k] += hb[hubsm::ah + conrec::xl + k];
        }
        if (hub && chain_rec()) displace_chain(chain_rec());
        mark(kPhaseUpdate);

        if (flags != 0.) {
            status = KYN_ERR_SINGULAR;
            break;
        }
        if (!(err == err) || isinf(err)) {
            status = KYN_ERR_NONFINITE;
            break;
        }
        if (err <= 1.) {
            if (extra < P.refine_iters) {
                ++extra;  // one more correction from the FP64 residual
                continue;
            }
            status = KYN_OK;
            break;
        }
    }

    // the copy issued in the last iteration lands before the region is released
    while (sec_waited < sec_issued) sec_wait();
    __syncthreads();
    if (s_flag & 8) status = KYN_ERR_CUDA;  // a section copy did not complete in time

    // ---- post-step (step.hpp:86-121) ---------------------------------------------------
    if (status == KYN_OK) {
        const double fac = (1. - P.alpha_f) / (1. - P.alpha_m);
#pragma unroll 1
        for (int t = tid; t < n6; t += NT) sa[t] += fac * svd[t];
    }
    if (hub && chain_rec()) {
        double* r = chain_rec();
        if (status == KYN_OK) {
            const double fac = (1. - P.alpha_f) / (1. - P.alpha_m);
            for (int k = 0; k < 6; ++k) r[hubrec::a + k] += fac * r[hubrec::vd + k];
            const double* x0 = r + hubrec::x0;
            for (int c = 0; c < 3; ++c) r[hubrec::x + c] = x0[c] + r[hubrec::q + c];
            quat_compose(r + hubrec::q + 3, x0 + 3, r + hubrec::x + 3);
        }
        const double* lam = (tid == NT - 1) ? hb + hubsm::bc + conrec::lam
                           : (tid == NT - 2) ? hb + hubsm::rev + revrec::lam : hb + hubsm::ah + conrec::lam;
        for (int k = 0; k < 6; ++k) r[hubrec::lambda + k] = (tid == NT - 2 && k == 5) ? 0. : lam[k];
    }
    __syncthreads();
    if (hub)  // every beam keeps its copy of the hub state (the input is the caller's)
#pragma unroll 1
        for (int k = tid; k < (drive ? chain : 1) * kHubDoubles; k += NT) {
            const int r = k / kHubDoubles, e = k % kHubDoubles;
            const double* src = r == 0 ? hb : r == 1 ? hA : hH;
            if (e < hubrec::input || e >= hubrec::input + 7) slab[L.hub + k] = src[e];
        }
#pragma unroll 1
    for (int k = tid; k < N * 7; k += NT) {
        slab[L.q + k] = sq[k];
        slab[L.q_prev + k] = sqp[k];
    }
#pragma unroll 1
    for (int k = tid; k < N * 6; k += NT) {
        slab[L.v + k] = sv[k];
        slab[L.vd + k] = svd[k];
        slab[L.a + k] = sa[k];
        slab[L.q_delta + k] = sqd[k];
    }
    if (status == KYN_OK) {
#pragma unroll 1
        for (int n = tid; n < N; n += NT) {
            const double* x0 = slab + L.x0 + n * 7;
            for (int c = 0; c < 3; ++c) slab[L.x + n * 7 + c] = x0[c] + sq[n * 7 + c];
            double r[4];
            quat_compose(sq + n * 7 + 3, x0 + 3, r);
            for (int c = 0; c < 4; ++c) slab[L.x + n * 7 + 3 + c] = r[c];
        }
    }
#pragma unroll 1
    for (int k = tid; k < N * 9; k += NT) slab[L.tangent + k] = sT[k];
    if (tid < 6 * nc) {
        const double* cr = con + (tid / 6) * kConStride;
        slab[L.lambda + tid] = cr[conrec::lam + tid % 6];
    }
    if (KB.rank == 0 && tid == 0) {
        status_out[KB.plan_model] = status;
        iters_out[KB.plan_model] = iters;
    }
    __syncthreads();
    mark(kPhaseStore);
    if (timing && tid == 0)
#pragma unroll 1
        for (int k = 0; k < kNumPhases; ++k) atomicAdd(KB.prof + k, s_ph[k]);
    if (clustered) cluster.sync();  // peers may still read this CTA's slot
}

}  // namespace kyn
