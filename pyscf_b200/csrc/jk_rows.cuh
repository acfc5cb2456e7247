// jk_rows.cuh — the row family of the J/K build: the classes whose Cartesian
// block is too large for the registers of one lane, spread over the lanes of
// a group by its first index.
//
// A lane of the group owns the components (a, *, c in its share, *) of one
// quartet and keeps them in registers over all primitive quartets: NB (NC /
// CS) ND accumulators, NA CS lanes a group.  What bounds the alternative that
// keeps the block in shared memory is the shared-memory pipe: three gathered
// 2D integrals per component and root, and two gathered values per
// contraction multiply-add.  Here the offsets of a lane's components differ
// from each other by compile-time constants, so one load of a 2D integral
// serves all components that share it ((21|20): 18 loads instead of 54 per
// root for 18 components), and all of J and K is contracted from registers:
// K[a,c], K[a,d] and J[a,b] are complete in a lane, K[b,c], K[b,d] and
// J[c,d] are summed over the lanes through shared memory (over the dead 2D
// integrals) with the same number of atomics as before.  The density blocks
// a quartet contracts with arrive by cp.async while it is evaluated.
//
// Measured on the FP64 build of (H2O)16/cc-pVTZ against groups with the block
// in shared memory: (21|20) 25.6 -> 13.2 ms, (21|11) 17.1 -> 7.9, (21|21) 13.4 ->
// 5.8, (31|21) 10.7 -> 4.3, (22|21) 10.3 -> 5.7, (32|22) 4.5 -> 1.4 ms.  What
// bounds it now is still the L1 data pipe, 90 % busy in (21|20) on
// (H2O)9/cc-pVTZ (2.09 ms): shared memory takes 442 M wavefronts, 160 M of them
// bank conflicts, of the 2D slices and the sums over lanes; FP64 35 %.
//
// A warp walks a chunk of one bra pair's kets: its 32 lanes screen 32 kets at
// once and the groups take the survivors in turn, in step (every loop of the
// warp runs to the longest trip count of its groups, the others adding zero).
#pragma once
#include "jk_launch.h"

namespace b200jk {

// Shares of the third index (CS above); 0: the class has no row kernel.
template <int LA, int LB, int LC, int LD>
__host__ __device__ constexpr int row_split()
{
        using K = Class4<LA, LB, LC, LD>;
        for (int cs = 1; cs <= K::NC; cs++)
                if (K::NC % cs == 0 && K::NA * cs <= 32 && K::NB * (K::NC / cs) * K::ND <= B2_ROW_ACC) return cs;
        return 0;
}

template <int LA, int LB, int LC, int LD, int CS, typename R>
struct RowSmem {
        using K = Class4<LA, LB, LC, LD>;
        static constexpr int NL = K::NA * CS;
        static constexpr int NGRP = 32 / NL;
        static constexpr int NCD1 = (LC + 1) * (LD + 1);
        // one (root, direction) slice: untransferred bra index, transferred ket
        // indices; odd, so that the slices written at once start on different banks
        static constexpr int SU = (K::NE * NCD1) | 1;
        // rows of the sums over the lanes, padded to an odd length
        static constexpr int WA = K::NA | 1, WL = NL | 1;
        static constexpr int RJ = 0, RBC = RJ + K::NCD * WA, RBD = RBC + K::NB * K::NC * WA;
        static constexpr int RED = RBD + K::NB * K::ND * WL;
        static constexpr int H = (3 * K::NR * SU * (int)sizeof(R) + 7) / 8;
        static constexpr int DCD = H > RED ? H : RED;      // doubles from here
        static constexpr int DAB = DCD + K::NCD;
        static constexpr int XBC = DAB + K::NAB;
        static constexpr int XBD = XBC + K::NB * K::NC;
        static constexpr int XAC = XBD + K::NB * K::ND;
        static constexpr int XAD = XAC + K::NA * K::NC;
        static constexpr int END = XAD + K::NA * K::ND;
        // the groups continue the lanes' pattern over the banks: NL slices on
        static constexpr int SIZE = END + ((SU * NL - END) % 16 + 16) % 16;
        // per warp: its groups, the list of surviving kets (32 bytes), and the
        // groups' roots and weights
        static constexpr int LIST = SIZE * NGRP;
        static constexpr int ROOTS = (LIST + 4 + 1) & ~1;
        static constexpr int WARP = ROOTS + 2 * K::NR * NGRP;
        static_assert(NGRP * K::NR <= 32, "a lane for every root of the warp's groups");
        // the Rys table is staged beside them up to four roots
        static constexpr bool STAGE = stage_table<R>(K::NR);
        static constexpr int TABLE = STAGE ? (RysStaged<K::NR, R>::ELEMS * (int)sizeof(R) + 15) / 16 * 2 : 0;   // doubles
        // Warps per block, one block per SM: 12 (168 registers a thread) where a
        // lane keeps at most 27 accumulators, else 8 (255), less where shared
        // memory does not admit them.  Both hold everything in registers; with
        // 16 and 12 warps the spills (200 and 700 bytes a thread) missed the
        // small L1 the shared memory leaves: (21|20) 15.4 -> 13.2 ms and (21|21)
        // 8.6 -> 5.8 ms on (H2O)16/cc-pVTZ; 8 warps for the former is 14.3.
        static constexpr int FIT = (227 * 1024 / 8 - TABLE) / WARP;
        static constexpr int WANT = K::NB * (K::NC / CS) * K::ND <= 27 ? 12 : 8;
        static constexpr int WPB = FIT < WANT ? FIT : WANT;
        static_assert(WPB >= 1, "a warp of the row family fits an SM");
};

__device__ __forceinline__ void cp_async8(double *smem, const double *g)
{
        const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_wait()
{
        asm volatile("cp.async.wait_all;" ::: "memory");
}

// block [rows][cols] of a row-major matrix into shared memory by the lanes of
// a group
template <int ROWS, int COLS, int NL>
__device__ __forceinline__ void row_stage(double *dst, const double *src, size_t ld, int gl)
{
#pragma unroll
        for (int t0 = 0; t0 < ROWS * COLS; t0 += NL) {
                const int t = t0 + gl;
                if (t < ROWS * COLS) cp_async8(dst + t, src + (size_t)(t / COLS) * ld + t % COLS);
        }
}

// One (root, direction) slice of the 2D integrals, transferred on the ket side
// only: h[e][c][d], e <= LA + LB.  The lanes that assemble components finish
// the bra transfer in registers, which stores LA + LB + 1 rows instead of
// (LA + 1)(LB + 1) ((22|: 5 instead of 9).
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void row_slice(R *h, R g00, R c00, R c00p, R b10, R b01, R b00, R cd)
{
        using K = Class4<LA, LB, LC, LD>;
        R g[K::NE * K::NF];
        vrr2d<K::NE, K::NF, R>(g, g00, c00, c00p, b10, b01, b00);
        R cdp[LD + 1];
        cdp[0] = (R)1;
#pragma unroll
        for (int k = 1; k <= LD; k++) cdp[k] = cdp[k - 1] * cd;
#pragma unroll
        for (int e = 0; e < K::NE; e++)
#pragma unroll
        for (int c = 0; c <= LC; c++)
#pragma unroll
        for (int d = 0; d <= LD; d++) {
                R v = (R)0;
#pragma unroll
                for (int k = 0; k <= d; k++) v += (R)binom(d, k) * cdp[d - k] * g[e * K::NF + c + k];
                h[(e * (LC + 1) + c) * (LD + 1) + d] = v;
        }
}

// Rows a .. a + LB of one direction's slice -> the N values (b, cd) of a lane's
// first index; abp[k] = (A - B)^k
template <int LB, int NCD1, int N, typename R>
__device__ __forceinline__ void row_transfer(R *h, const R *u, const R *abp)
{
        R x[(LB + 1) * N];
#pragma unroll
        for (int k = 0; k <= LB; k++)
#pragma unroll
                for (int t = 0; t < N; t++) x[k * N + t] = u[k * NCD1 + t];
#pragma unroll
        for (int b = 0; b <= LB; b++)
#pragma unroll
                for (int t = 0; t < N; t++) {
                        R v = (R)0;
#pragma unroll
                        for (int k = 0; k <= b; k++) v += (R)binom(b, k) * abp[b - k] * x[k * N + t];
                        h[b * N + t] = v;
                }
}

template <int LA, int LB, int LC, int LD, int CS, typename R, bool MULTI>
__global__ void __launch_bounds__((32 * RowSmem<LA, LB, LC, LD, CS, R>::WPB), 1) jk_row_kernel(JKArgs a0, int chunk_q, const JKArgs *__restrict__ margs,
                                                                  const long long *__restrict__ mchunk, int nmol)
{
        using K = Class4<LA, LB, LC, LD>;
        using S = RowSmem<LA, LB, LC, LD, CS, R>;
        constexpr int NL = S::NL, NGRP = S::NGRP, NCS = K::NC / CS, NACC = K::NB * NCS * K::ND;
        constexpr int NA = K::NA, NB = K::NB, NC = K::NC, ND = K::ND, NR = K::NR, SU = S::SU, NCD1 = S::NCD1;
        extern __shared__ __align__(32) double smem_dyn[];
        ChunkLoop loop(a0.next, MULTI ? mchunk[0] : a0.chunk_off[0],
                       MULTI ? mchunk[nmol] : a0.chunk_off[a0.tiled ? a0.ntile : a0.bra.n * B2_NBUCKET]);
        // one block per chunk at most: few chunks spread over as many SMs
        if (loop.first + blockIdx.x >= loop.total) return;
        const int lane = threadIdx.x & 31;
        // lanes past the last group evaluate nothing and contract nothing
        const bool busy = lane < NL * NGRP;
        const int grp = busy ? lane / NL : 0, gl = busy ? lane - grp * NL : NL;
        const int av = busy ? gl / CS : 0, cs = busy ? gl % CS : 0;
        double *wsm = smem_dyn + S::TABLE + (size_t)(threadIdx.x >> 5) * S::WARP;
        double *sm = wsm + grp * S::SIZE;
        unsigned char *list = reinterpret_cast<unsigned char *>(wsm + S::LIST);
        double2 *roots = reinterpret_cast<double2 *>(wsm + S::ROOTS);
        // the root this lane evaluates for its warp: lane / NR's group, root lane % NR
        const bool rooter = lane < NGRP * NR;
        const int rsrc = rooter ? lane / NR * NL : 0, rroot = rooter ? lane % NR : 0;
        R *H = reinterpret_cast<R *>(sm);
        const R *table = table_of<R>(a0) + RysLayout<R>::offset(NR);
        // (a launch of few chunks reads its few rows from global memory: staging
        // 35-53 KB would take longer than they do)
        const bool staged = S::STAGE && loop.total - loop.first > 4 * S::WPB;
        if (staged) {
                stage_rys<NR, R>(reinterpret_cast<R *>(smem_dyn), table);
                table = reinterpret_cast<const R *>(smem_dyn);
        }
        // 2D slices: this lane's direction, its first root and the roots a round
        // of the group's lanes takes
        constexpr int NRL = NL / 3;
        const int dir = gl % 3, r0 = busy && gl < 3 * NRL ? gl / 3 : NR;
        // first of this lane's rows of the three directions' slices
        int oa[3] = {0, 0, 0};
#pragma unroll
        for (int x = 0; x < NA; x++)
                if (av == x) {
                        oa[0] = cart_lx(LA, x) * NCD1;
                        oa[1] = cart_ly(LA, x) * NCD1 + SU;
                        oa[2] = cart_lz(LA, x) * NCD1 + 2 * SU;
                }
        // offsets of its c components (compile-time where it owns all of them)
        int oc[CS > 1 ? 3 * NCS : 1];
        if constexpr (CS > 1) {
#pragma unroll
                for (int c = 0; c < NC; c++)
                        if (c / NCS == cs) {
                                oc[3 * (c % NCS) + 0] = cart_lx(LC, c) * (LD + 1);
                                oc[3 * (c % NCS) + 1] = cart_ly(LC, c) * (LD + 1);
                                oc[3 * (c % NCS) + 2] = cart_lz(LC, c) * (LD + 1);
                        }
        }
        unsigned long long nq = 0, npq = 0;
        long long chunk;
        while (loop.get(chunk)) {
              auto body = [&](const JKArgs &a) {
                const size_t n = (size_t)a.naoc, nn = n * n;
                int sgi, kc, lg;
                if (!map_chunk(a, chunk, chunk_q, 3, sgi, kc, lg)) return;
                const int cq = chunk_q >> lg;
                const int ij = sgi / B2_NBUCKET;
                const int kb = a.ket.boff[sgi % B2_NBUCKET] + a.kst[sgi];
                const int kl0 = kb + kc * cq;
                const int kl1 = kb + min(kc * cq + cq, a.nkl[sgi]);
                const int4 sb = a.bra.sh[ij];
                const int2 pb = a.bra.pr[ij];
                const double qij = a.bra.q[ij];
                const double4 Ab = a.bra.A[ij];
                const double4 ABb = a.bra.AB[ij];
                // this lane's direction of A
                const double Ad = dir == 0 ? Ab.x : (dir == 1 ? Ab.y : Ab.z);
                R abp[3][LB + 1];   // powers of A - B
#pragma unroll
                for (int x = 0; x < 3; x++) {
                        abp[x][0] = (R)1;
#pragma unroll
                        for (int k = 1; k <= LB; k++) abp[x][k] = abp[x][k - 1] * (R)(x == 0 ? ABb.x : (x == 1 ? ABb.y : ABb.z));
                }
                const int ia = sb.x, ib = sb.y;
                // bra-side J of one density: summed over the chunk
                const bool jab_sum = a.with_j && a.n_dm == 1;
                double jab[NB];
#pragma unroll
                for (int b = 0; b < NB; b++) jab[b] = 0.0;
                if (jab_sum && busy) row_stage<NA, NB, NL>(sm + S::DAB, a.Ds + ia * n + ib, n, gl);
                for (int base = kl0; base < kl1; base += 32) {
                        // 32 kets screened at once
                        bool pass = false;
                        if (base + lane < kl1) pass = quartet_passes(a, sb, qij, a.ket.sh[base + lane], a.ket.q[base + lane]);
                        const unsigned mask = __ballot_sync(0xffffffffu, pass);
                        if (pass) list[__popc(mask & ((1u << lane) - 1u))] = (unsigned char)lane;
                        __syncwarp();
                        const int npass = __popc(mask);
                        for (int i0 = 0; i0 < npass; i0 += NGRP) {
                                const bool has = busy && i0 + grp < npass;
                                const int kl = base + list[has ? i0 + grp : i0];
                                const int4 sk = a.ket.sh[kl];
                                const int2 pk = a.ket.pr[kl];
                                const double4 Ak = a.ket.A[kl];
                                const double4 CDk = a.ket.AB[kl];
                                const int ic = sk.x, id = sk.y;
                                // density blocks of density s, transpose tk
                                auto stage = [&](int s, int tk) {
                                        if (!has) return;
                                        if (a.with_j && tk == 0) {
                                                const double *Ds = a.Ds + s * nn;
                                                if (a.Dpk) row_stage<1, K::NCD, NL>(sm + S::DCD, a.Dpk + s * a.pk_stride + (long long)kl * K::NCD, 0, gl);
                                                else row_stage<NC, ND, NL>(sm + S::DCD, Ds + ic * n + id, n, gl);
                                                if (!jab_sum) row_stage<NA, NB, NL>(sm + S::DAB, Ds + ia * n + ib, n, gl);
                                        }
                                        if (a.with_k) {
                                                const double *X = a.Dk + (s * a.nk + tk) * nn;
                                                row_stage<NB, NC, NL>(sm + S::XBC, X + ib * n + ic, n, gl);
                                                row_stage<NB, ND, NL>(sm + S::XBD, X + ib * n + id, n, gl);
                                                row_stage<NA, NC, NL>(sm + S::XAC, X + ia * n + ic, n, gl);
                                                row_stage<NA, ND, NL>(sm + S::XAD, X + ia * n + id, n, gl);
                                        }
                                };
                                stage(0, 0);
                                R fac = (R)1;
                                if (Ab.w != 0.0) fac *= (R)0.5;
                                if (Ak.w != 0.0) fac *= (R)0.5;
                                if (a.same && ij == kl) fac *= (R)0.5;
                                const double Cd = dir == 0 ? Ak.x : (dir == 1 ? Ak.y : Ak.z);
                                const R CDd = (R)(dir == 0 ? CDk.x : (dir == 1 ? CDk.y : CDk.z));
                                const int own = has ? pb.y * pk.y : 0;
                                const int most = __reduce_max_sync(0xffffffffu, own);
                                if (has && gl == 0) {
                                        nq++;
                                        npq += (unsigned long long)own;
                                }
                                R acc[NACC];
#pragma unroll
                                for (int t = 0; t < NACC; t++) acc[t] = (R)0;
                                int ip = 0, kp = 0;
                                for (int t = 0; t < most; t++) {
                                        const double4 P = a.PP[pb.x + ip];
                                        const double2 KP = a.PK[pb.x + ip];
                                        const double4 Q = a.PP[pk.x + kp];
                                        const double2 KQ = a.PK[pk.x + kp];
                                        const R kk = t < own ? (R)KP.x * fac * (R)KQ.x : (R)0;
                                        // as prim_setup
                                        const R p = (R)P.w, q = (R)Q.w, i2p = (R)KP.y, i2q = (R)KQ.y;
                                        const R ipq = (R)1 / (p + q), qf0 = q * ipq, pf0 = p * ipq;
                                        const double Pd = dir == 0 ? P.x : (dir == 1 ? P.y : P.z);
                                        const double Qd = dir == 0 ? Q.x : (dir == 1 ? Q.y : Q.z);
                                        R dx, dy, dz, PA, QC, PQ;
                                        if constexpr (sizeof(R) == 4) {
                                                // rounded after the difference to the bra centre, as every
                                                // float32 kernel (the passes then differ in summation order only)
                                                dx = (R)(P.x - Ab.x) - (R)(Q.x - Ab.x);
                                                dy = (R)(P.y - Ab.y) - (R)(Q.y - Ab.y);
                                                dz = (R)(P.z - Ab.z) - (R)(Q.z - Ab.z);
                                                PA = (R)(Pd - Ad);
                                                QC = (R)(Qd - Ad) - (R)(Cd - Ad);
                                                PQ = dir == 0 ? dx : (dir == 1 ? dy : dz);
                                        } else {
                                                dx = P.x - Q.x;
                                                dy = P.y - Q.y;
                                                dz = P.z - Q.z;
                                                PA = Pd - Ad;
                                                QC = Qd - Cd;
                                                PQ = Pd - Qd;
                                        }
                                        R T = p * qf0 * (dx * dx + dy * dy + dz * dz);
                                        R pref = (R)34.98683665524972497 * kk * ((R)4 * i2p * i2q) * b2sqrt(ipq);
                                        R theta = (R)1;
                                        if (a.omega2 > 0.0) {
                                                theta = (R)a.omega2 / ((R)a.omega2 + p * qf0);
                                                T *= theta;
                                                pref *= b2sqrt(theta);
                                        }
                                        // every root once: the lanes of a group that share one read it back
                                        // (a lane per task would read its table rows three times over, four
                                        // wavefronts per 16-byte load, as much as the whole assembly)
                                        const R Tr = __shfl_sync(0xffffffffu, T, rsrc);
                                        if (rooter) {
                                                R ur, wr;
                                                if (staged) rys_root_one_staged<NR, R>(Tr, table, rroot, ur, wr);
                                                else rys_root_one<NR, R>(Tr, table, rroot, ur, wr);
                                                roots[lane] = make_double2((double)ur, (double)wr);
                                        }
                                        // (the 2D integrals of the previous primitive quartet are read, too)
                                        __syncwarp();
#pragma unroll 1
                                        for (int r = r0; r < NR; r += NRL) {
                                                const double2 uw = roots[grp * NR + r];
                                                const R ur = (R)uw.x * theta, wr = (R)uw.y;
                                                const R qf = qf0 * ur, pf = pf0 * ur;
                                                row_slice<LA, LB, LC, LD, R>(H + (3 * r + dir) * SU, dir == 2 ? pref * wr : (R)1,
                                                                             PA - qf * PQ, QC + pf * PQ, i2p * ((R)1 - qf),
                                                                             i2q * ((R)1 - pf), (R)0.5 * ur * ipq, CDd);
                                        }
                                        __syncwarp();
                                        // (float32: a primitive quartet's sum over roots apart, as the other kernels)
                                        R one[sizeof(R) == 4 ? NACC : 1];
                                        R *sum = sizeof(R) == 4 ? one : acc;
                                        if constexpr (sizeof(R) == 4) {
#pragma unroll
                                                for (int u = 0; u < NACC; u++) one[u] = (R)0;
                                        }
#pragma unroll 1
                                        for (int r = 0; r < NR; r++) {
                                                const R *ux = H + 3 * r * SU + oa[0];
                                                const R *uy = H + 3 * r * SU + oa[1];
                                                const R *uz = H + 3 * r * SU + oa[2];
                                                if constexpr (CS == 1) {
                                                        R hx[(LB + 1) * NCD1], hy[(LB + 1) * NCD1], hz[(LB + 1) * NCD1];
                                                        row_transfer<LB, NCD1, NCD1, R>(hx, ux, abp[0]);
                                                        row_transfer<LB, NCD1, NCD1, R>(hy, uy, abp[1]);
                                                        row_transfer<LB, NCD1, NCD1, R>(hz, uz, abp[2]);
                                                        for_parts([&](auto tag) {
                                                                constexpr int T = decltype(tag)::value;
                                                                constexpr int d = T % ND, c = T / ND % NCS, b = T / (ND * NCS);
                                                                constexpr int ox = K::hidx(0, cart_lx(LB, b), cart_lx(LC, c), cart_lx(LD, d));
                                                                constexpr int oy = K::hidx(0, cart_ly(LB, b), cart_ly(LC, c), cart_ly(LD, d));
                                                                constexpr int oz = K::hidx(0, cart_lz(LB, b), cart_lz(LC, c), cart_lz(LD, d));
                                                                sum[T] += hx[ox] * hy[oy] * hz[oz];
                                                        }, std::make_integer_sequence<int, NACC>{});
                                                } else {
#pragma unroll
                                                        for (int c = 0; c < NCS; c++) {
                                                                R hx[(LB + 1) * (LD + 1)], hy[(LB + 1) * (LD + 1)], hz[(LB + 1) * (LD + 1)];
                                                                row_transfer<LB, NCD1, LD + 1, R>(hx, ux + oc[3 * c], abp[0]);
                                                                row_transfer<LB, NCD1, LD + 1, R>(hy, uy + oc[3 * c + 1], abp[1]);
                                                                row_transfer<LB, NCD1, LD + 1, R>(hz, uz + oc[3 * c + 2], abp[2]);
                                                                for_parts([&](auto tag) {
                                                                        constexpr int T = decltype(tag)::value;
                                                                        constexpr int d = T % ND, b = T / ND;
                                                                        constexpr int ox = cart_lx(LB, b) * (LD + 1) + cart_lx(LD, d);
                                                                        constexpr int oy = cart_ly(LB, b) * (LD + 1) + cart_ly(LD, d);
                                                                        constexpr int oz = cart_lz(LB, b) * (LD + 1) + cart_lz(LD, d);
                                                                        sum[(b * NCS + c) * ND + d] += hx[ox] * hy[oy] * hz[oz];
                                                                }, std::make_integer_sequence<int, NB * ND>{});
                                                        }
                                                }
                                        }
                                        if constexpr (sizeof(R) == 4) {
#pragma unroll
                                                for (int u = 0; u < NACC; u++) acc[u] += one[u];
                                        }
                                        if (t + 1 < own && ++kp == pk.y) {
                                                kp = 0;
                                                ip++;
                                        }
                                }
                                // contraction: the 2D integrals are dead, their space holds the sums over lanes
                                for (int s = 0; s < a.n_dm; s++)
                                for (int tk = 0; tk < (a.with_k ? a.nk : 1); tk++) {
                                        const bool doj = a.with_j && tk == 0;
                                        if (s + tk > 0) stage(s, tk);
                                        cp_async_wait();
                                        __syncwarp();
                                        if (doj) {
                                                // element by element of the ket: J[a,b] of the lane, J[c,d] summed over a
                                                const double *dcd = sm + S::DCD + cs * NCS * ND;
                                                double *rj = sm + S::RJ + cs * NCS * ND * S::WA + av;
                                                double dab[NB], v[NB];
#pragma unroll
                                                for (int b = 0; b < NB; b++) {
                                                        dab[b] = sm[S::DAB + av * NB + b];
                                                        v[b] = 0.0;
                                                }
#pragma unroll
                                                for (int u = 0; u < NCS * ND; u++) {
                                                        const double du = dcd[u];
                                                        double w = 0.0;
#pragma unroll
                                                        for (int b = 0; b < NB; b++) {
                                                                v[b] += (double)acc[b * NCS * ND + u] * du;
                                                                w += (double)acc[b * NCS * ND + u] * dab[b];
                                                        }
                                                        if (has) rj[u * S::WA] = w;
                                                }
                                                if (has) {
#pragma unroll
                                                        for (int b = 0; b < NB; b++) {
                                                                if (jab_sum) jab[b] += v[b];
                                                                else atomicAdd(a.Jacc + s * nn + (ia + av) * n + ib + b, v[b]);
                                                        }
                                                }
                                        }
                                        double *Kt = a.with_k ? a.Kacc + (s * a.nk + tk) * nn : nullptr;
                                        if (a.with_k) {
                                                // one sweep over b: K[a,c] += G X[b,d] and K[a,d] += G X[b,c] in
                                                // the lane, K[b,c] += G X[a,d] and K[b,d] += G X[a,c] summed over a
                                                double kac[NCS], kad[ND], xad[ND];
#pragma unroll
                                                for (int c = 0; c < NCS; c++) kac[c] = 0.0;
#pragma unroll
                                                for (int d = 0; d < ND; d++) {
                                                        kad[d] = 0.0;
                                                        xad[d] = sm[S::XAD + av * ND + d];
                                                }
                                                double *rbc = sm + S::RBC + cs * NCS * S::WA + av, *rbd = sm + S::RBD + gl;
                                                const double *xac = sm + S::XAC + av * NC + cs * NCS;
#pragma unroll
                                                for (int b = 0; b < NB; b++) {
                                                        double xbd[ND], vbd[ND];
#pragma unroll
                                                        for (int d = 0; d < ND; d++) {
                                                                xbd[d] = sm[S::XBD + b * ND + d];
                                                                vbd[d] = 0.0;
                                                        }
#pragma unroll
                                                        for (int c = 0; c < NCS; c++) {
                                                                const double xbc = sm[S::XBC + b * NC + cs * NCS + c], xc = xac[c];
                                                                double vbc = 0.0;
#pragma unroll
                                                                for (int d = 0; d < ND; d++) {
                                                                        const double g = (double)acc[(b * NCS + c) * ND + d];
                                                                        kac[c] += g * xbd[d];
                                                                        kad[d] += g * xbc;
                                                                        vbc += g * xad[d];
                                                                        vbd[d] += g * xc;
                                                                }
                                                                if (has) rbc[(b * NC + c) * S::WA] = vbc;
                                                        }
                                                        if (has) {
#pragma unroll
                                                                for (int d = 0; d < ND; d++) rbd[(b * ND + d) * S::WL] = vbd[d];
                                                        }
                                                }
#pragma unroll
                                                for (int d = 0; d < ND; d++) {
                                                        double w = kad[d];
#pragma unroll
                                                        for (int k = 1; k < CS; k++) w += __shfl_down_sync(0xffffffffu, kad[d], k);
                                                        if (has && cs == 0) atomicAdd(Kt + (ia + av) * n + id + d, w);
                                                }
                                                if (has) {
#pragma unroll
                                                        for (int c = 0; c < NCS; c++) atomicAdd(Kt + (ia + av) * n + ic + cs * NCS + c, kac[c]);
                                                }
                                        }
                                        __syncwarp();
                                        if (has) {
                                                if (doj)
                                                        for (int u = gl; u < K::NCD; u += NL) {
                                                                double v = 0.0;
#pragma unroll
                                                                for (int x = 0; x < NA; x++) v += sm[S::RJ + u * S::WA + x];
                                                                if (a.Jpk) atomicAdd(a.Jpk + s * a.pk_stride + (long long)kl * K::NCD + u, v);
                                                                else atomicAdd(a.Jacc + s * nn + (ic + u / ND) * n + id + u % ND, v);
                                                        }
                                                if (a.with_k) {
                                                        for (int u = gl; u < NB * NC; u += NL) {
                                                                double v = 0.0;
#pragma unroll
                                                                for (int x = 0; x < NA; x++) v += sm[S::RBC + u * S::WA + x];
                                                                atomicAdd(Kt + (ib + u / NC) * n + ic + u % NC, v);
                                                        }
                                                        for (int u = gl; u < NB * ND; u += NL) {
                                                                double v = 0.0;
#pragma unroll
                                                                for (int x = 0; x < NL; x++) v += sm[S::RBD + u * S::WL + x];
                                                                atomicAdd(Kt + (ib + u / ND) * n + id + u % ND, v);
                                                        }
                                                }
                                        }
                                        __syncwarp();
                                }
                        }
                }
                if (jab_sum) {
                        // over the groups (and shares) of the warp: one atomic per element
                        if (busy)
#pragma unroll
                                for (int b = 0; b < NB; b++) sm[b * NL + gl] = jab[b];
                        cp_async_wait();
                        __syncwarp();
                        for (int u = lane; u < K::NAB; u += 32) {
                                const int x = u / NB, b = u % NB;
                                double v = 0.0;
                                for (int g = 0; g < NGRP; g++)
#pragma unroll
                                        for (int k = 0; k < CS; k++) v += wsm[g * S::SIZE + b * NL + x * CS + k];
                                if (v != 0.0) atomicAdd(a.Jacc + (ia + x) * n + ib + b, v);
                        }
                        __syncwarp();
                }
              };
                if constexpr (MULTI) body(margs[find_bra(mchunk, nmol, chunk)]);
                else body(a0);
        }
        if (a0.stats && busy && gl == 0 && nq) {
                atomicAdd(a0.stats + 0, nq);
                atomicAdd(a0.stats + 1, npq);
        }
}

} // namespace b200jk
