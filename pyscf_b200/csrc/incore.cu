// incore.cu — J and K from a stored two-electron integral tensor: the in-core
// path of the reference, _vhf.incore (pyscf/scf/_vhf.py:318-401) driving
// CVHFnrs8_incore_drv / CVHFnrs4_incore_drv with the contractions of
// pyscf/lib/vhf/nr_incore.c (CVHFics8_tridm_vj :389, CVHFics8_jk_s2il :422,
// CVHFics8_jk_s1il :413, CVHFics4_kl_s2ij :461, CVHFics4_il_s1jk :438).
//
// Tensor layouts (pair index ij = i(i+1)/2 + j, i >= j; npair pairs):
//   s8  entry (ij|kl), ij >= kl, at ij(ij+1)/2 + kl;
//   s4  entry (ij|kl) at ij * npair + kl.
// A stored entry v = (ij|kl) stands for its symmetry images (a,b,c,d); image
// (a,b,c,d) adds v D[b,c] to K[a,d] and v D[a,b] to J[c,d].  A pass
// accumulates, with weight w = 1/(number of images that coincide),
//   A[i,l] += w v D[j,k]   A[j,l] += w v D[i,k]
//   A[i,k] += w v D[j,l]   A[j,k] += w v D[i,l]
// (the images that keep the order of the two pairs) and packed J
//   Jp[kl] += v t[ij]      Jp[ij] += v t[kl]  (s8 only; weight 1/2 if ij == kl)
// with t[ij] = D[i,j] + D[j,i] (D[i,i] on the diagonal).  The pair-swapped
// images are then, for s8, A(D^T)^T (so K = A(D) + A(D)^T for symmetric D),
// and for s4 the swapped entries are stored themselves (K = A(D)).
//
// Work decomposition.  A thread block owns the packed rows ij of one pair of
// AO blocks (i in block I, j in block J, I >= J, 8 AOs a block) and a window
// of packed columns kl.  Each thread takes one column kl of a 256-column
// chunk and walks the block's rows, so every row's chunk is one coalesced
// 2 KB read and each entry is read from HBM once.  One launch of four
// variants: the interior of the packed matrix (blocks I > J, columns before
// the block's rows: no per-entry test or weight), the windows of such blocks
// that reach their rows (EDGE: q <= p tested per entry), and the same two for
// the diagonal blocks I == J (DIAG: rows j > i skipped, the K images of
// j == i halved).  The K images and J row sums of a lane's register sums go
// straight to the (L2-resident) accumulators with float64 reductions, after a
// warp reduction where all lanes share k.  The floor is HBM: 8 bytes per
// stored entry.
#include <vector>
#include "incore_launch.h"

namespace b200jk {

namespace {

constexpr int NT = 256;   // threads per block = packed columns per chunk

__device__ __forceinline__ void pair_of(long long q, int &k, int &l)
{
        // k = floor((sqrt(8q + 1) - 1) / 2), corrected for rounding
        int kk = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
        while ((long long)kk * (kk + 1) / 2 > q) kk--;
        while ((long long)(kk + 1) * (kk + 2) / 2 <= q) kk++;
        k = kk;
        l = (int)(q - (long long)kk * (kk + 1) / 2);
}

// N values a lane -> each value summed over the warp; lane gets the sum of
// value `row` (lanes that share `row` hold the same sum; the one with
// (lane & (32 / N - 1)) == 0 writes it)
template <int N>
__device__ __forceinline__ double reduce_scatter(double (&v)[N], int lane, int &row)
{
        int base = 0;
        int off = 16;
#pragma unroll
        for (int h = N / 2; h >= 1; h /= 2) {
                const bool up = (lane & off) != 0;
#pragma unroll
                for (int m = 0; m < h; m++) {
                        const double send = up ? v[m] : v[m + h];
                        const double keep = up ? v[m + h] : v[m];
                        v[m] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
                if (up) base += h;
                off >>= 1;
        }
        double s = v[0];
        for (; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        row = base;
        return s;
}

// stages of the kernel's ring of entries
constexpr int STAGES = 4;

// 8 bytes global -> shared without a register; zeros where !ok (nothing is read)
__device__ __forceinline__ void cp_async8z(double *smem, const double *g, bool ok)
{
        const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(g), "r"(ok ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit()
{
        asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait_group()
{
        asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The interior of the packed matrix: full AO blocks I > J (so i > j for
// every row) and, for s8, columns before the block's first row (so q < p for
// every entry).  No entry needs a validity test, rows follow each other by
// their length, and the only symmetry weight is the column's own k == l,
// applied once to the K sums of a lane.  The K images and the J row sums go
// straight to the (L2-resident) accumulators with fire-and-forget float64
// reductions, about one per four entries, so the block keeps only the two
// density slabs in shared memory and needs no flush.
// EDGE: the windows of such a block that reach its rows (s8): an entry is
// stored only for q <= p and counts half on the packed diagonal q == p.
// DIAG: a diagonal block I == J, whose rows are the pairs j <= i (the others
// are skipped, uniformly over the block) and count half for j == i.
// A partial last block row only has fewer rows i.
//
// What bounds it is the shared-memory and shuffle pipe, so a lane keeps the
// density rows of its column's k and l in registers for all rows of the block
// (2 x 8 doubles), reads the row weights T as 16-byte vectors and reduces its
// sums over l four rows at a time (12 shuffles instead of 40).
// Measured per call (s8, one symmetric density, HBM floor in brackets): nao
// 192 609 -> 541 us (207), nao 129 341 -> 197 us (42), nao 64 107 -> 73 us;
// s4, nao 117, two general densities 819 -> 352 us (115): bases whose size is
// no multiple of 8 spent their time in a general kernel for the last block row.
template <int B, bool S8, bool EDGE, bool DIAG>
__device__ __forceinline__ void incore_fast_body(const IncoreArgs &a, const int4 it)
{
        extern __shared__ __align__(16) double sm[];
        const int nao = a.nao;
        double *T = sm, *ring = T + B * B, *DI = ring + STAGES * B * NT, *DJ = DI + B * nao;
        const int i0 = it.x * B, j0 = it.y * B;
        const int nrow = min(B, nao - i0);
        const int tid = threadIdx.x, lane = tid & 31;
        const long long c0 = it.z, c1 = it.w;
        // the stages: row group fi of the chunk of columns at fq, slot fs
        int fi = 0, fs = 0;
        long long fq = c0;
        auto fetch = [&]() {
                if (fq < c1) {
                        const int i = i0 + fi;
                        const long long q = fq + tid;
                        const long long p0 = (long long)i * (i + 1) / 2 + j0;
                        // edge windows: rows before the chunk hold none of its columns
                        if (!EDGE || p0 + B - 1 >= fq) {
                                const double *row = a.eri + (S8 ? p0 * (p0 + 1) / 2 : p0 * a.npair) + q;
                                double *dst = ring + fs * (B * NT) + tid;
#pragma unroll
                                for (int jj = 0; jj < B; jj++) {
                                        // DIAG rows j > i do not exist; what is not stored reads as zero
                                        const bool ok = q < c1 && (!DIAG || jj <= fi) && (!EDGE || q <= p0 + jj);
                                        cp_async8z(dst + jj * NT, ok ? row : a.eri, ok);
                                        row += S8 ? p0 + jj + 1 : a.npair;   // next row: p + 1 entries on (s8)
                                }
                        }
                        fs = (fs + 1) % STAGES;
                        if (++fi == nrow) {
                                fi = 0;
                                fq += NT;
                        }
                }
                cp_async_commit();
        };
#pragma unroll
        for (int st = 0; st < STAGES - 1; st++) fetch();
        for (int e = tid; e < B * nao; e += NT) {
                const int r = e / nao, x = e % nao;
                DI[e] = i0 + r < nao ? a.D[(size_t)(i0 + r) * nao + x] : 0.0;
                DJ[e] = j0 + r < nao ? a.D[(size_t)(j0 + r) * nao + x] : 0.0;
        }
        for (int e = tid; e < B * B; e += NT) {
                // (diagonal blocks: rows j > i do not exist)
                const int i = i0 + e / B, j = j0 + e % B;
                T[e] = j <= i && i < nao ? a.t[(long long)i * (i + 1) / 2 + j] : 0.0;
        }
        __syncthreads();
        double *AI = a.A + (size_t)i0 * nao, *AJ = a.A + (size_t)j0 * nao;
        int slot = 0;
        for (long long qb = c0; qb < c1; qb += NT) {
                const long long q = qb + tid;
                const bool active = q < c1;
                int k = 0, l = 0;
                if (active) pair_of(q, k, l);
                const double tq = active ? a.t[q] : 0.0;
                const double wkl = k == l ? 0.5 : 1.0;
                const int k0 = __shfl_sync(0xffffffffu, k, 0);
                const bool kuni = __all_sync(0xffffffffu, !active || k == k0);
                double acc2[B], acc4[B], djk[B], djl[B];
#pragma unroll
                for (int jj = 0; jj < B; jj++) {
                        acc2[jj] = 0.0;
                        acc4[jj] = 0.0;
                        djk[jj] = DJ[jj * nao + k];
                        djl[jj] = DJ[jj * nao + l];
                }
                double colj = 0.0;
                for (int ib = 0; ib < nrow; ib += 4) {
                        double a3[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                                const int ii = ib + u;
                                a3[u] = 0.0;
                                if (ii >= nrow) continue;
                                fetch();
                                cp_async_wait_group<STAGES - 1>();
                                const double *src = ring + slot * (B * NT) + tid;
                                slot = (slot + 1) % STAGES;
                                const int i = i0 + ii;
                                const long long p0 = (long long)i * (i + 1) / 2 + j0;
                                if (EDGE && p0 + B - 1 < qb) continue;
                                const double dik = DI[ii * nao + k], dil = DI[ii * nao + l];
                                double acc1 = 0.0, acc3 = 0.0, rp[B];
#pragma unroll
                                for (int jj = 0; jj < B; jj += 2) {
                                        const double2 tw = *reinterpret_cast<const double2 *>(T + ii * B + jj);
#pragma unroll
                                        for (int h = 0; h < 2; h++) {
                                                const int j = jj + h;
                                                double v = src[j * NT];
                                                if (EDGE && q == p0 + j) v *= 0.5;   // the packed diagonal counts half
                                                // the K images of a row j == i count half (DIAG)
                                                const double vk = DIAG && j == ii ? 0.5 * v : v;
                                                acc1 += vk * djk[j];
                                                acc3 += vk * djl[j];
                                                acc2[j] += vk * dik;
                                                acc4[j] += vk * dil;
                                                colj += v * (h ? tw.y : tw.x);
                                                rp[j] = v * tq;
                                        }
                                }
                                a3[u] = wkl * acc3;
                                if (active && acc1 != 0.0) atomicAdd(AI + (size_t)ii * nao + l, wkl * acc1);
                                if (!kuni && active && acc3 != 0.0) atomicAdd(AI + (size_t)ii * nao + k, a3[u]);
                                if (S8 && a.Jp) {
                                        int rrow;
                                        const double s = reduce_scatter<B>(rp, lane, rrow);
                                        if ((lane & (32 / B - 1)) == 0 && (!DIAG || rrow <= ii) && s != 0.0)
                                                atomicAdd(a.Jp + p0 + rrow, s);
                                }
                        }
                        if (kuni) {
                                int rrow;
                                const double s = reduce_scatter<4>(a3, lane, rrow);
                                if ((lane & 7) == 0 && ib + rrow < nrow && s != 0.0)
                                        atomicAdd(AI + (size_t)(ib + rrow) * nao + k0, s);
                        }
                }
#pragma unroll
                for (int jj = 0; jj < B; jj++) {
                        acc2[jj] *= wkl;
                        acc4[jj] *= wkl;
                        if (active && (!DIAG || jj < nrow) && acc2[jj] != 0.0) atomicAdd(AJ + (size_t)jj * nao + l, acc2[jj]);
                }
                if (kuni) {
                        int rrow;
                        const double s = reduce_scatter<B>(acc4, lane, rrow);
                        if ((lane & (32 / B - 1)) == 0 && (!DIAG || rrow < nrow) && s != 0.0)
                                atomicAdd(AJ + (size_t)rrow * nao + k0, s);
                } else if (active) {
#pragma unroll
                        for (int jj = 0; jj < B; jj++)
                                if ((!DIAG || jj < nrow) && acc4[jj] != 0.0) atomicAdd(AJ + (size_t)jj * nao + k, acc4[jj]);
                }
                if (a.Jp && active && colj != 0.0) atomicAdd(a.Jp + q, colj);
        }
}

// One launch for the four variants: blocks take the items of variant 0
// (the bulk of the tensor) first, then those of 1, 2 and 3, which fill the
// tail of the launch.
template <int B, bool S8>
__global__ void __launch_bounds__(NT, 2) incore_fast_kernel(IncoreArgs a)
{
        // (the item lists are selected by constant indices: a run-time index
        // into the parameter array would copy it to local memory)
        int b = blockIdx.x;
        if (b < a.nf[0]) {
                incore_fast_body<B, S8, false, false>(a, a.fitems[0][b]);
                return;
        }
        b -= a.nf[0];
        if (b < a.nf[1]) {
                incore_fast_body<B, S8, true, false>(a, a.fitems[1][b]);
                return;
        }
        b -= a.nf[1];
        if (b < a.nf[2]) {
                incore_fast_body<B, S8, false, true>(a, a.fitems[2][b]);
                return;
        }
        b -= a.nf[2];
        incore_fast_body<B, S8, true, true>(a, a.fitems[3][b]);
}

__global__ void tridm_kernel(const double *__restrict__ D, int nao, double *__restrict__ t)
{
        const long long np = (long long)nao * (nao + 1) / 2;
        const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        if (p >= np) return;
        int i, j;
        pair_of(p, i, j);
        t[p] = i == j ? D[(size_t)i * nao + i] : D[(size_t)i * nao + j] + D[(size_t)j * nao + i];
}

__global__ void unpack_j_kernel(const double *__restrict__ Jp, int nao, double *__restrict__ vj)
{
        const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        if (e >= (long long)nao * nao) return;
        const int x = (int)(e / nao), y = (int)(e % nao);
        const int hi = x >= y ? x : y, lo = x >= y ? y : x;
        vj[e] = Jp[(long long)hi * (hi + 1) / 2 + lo];
}

__global__ void finish_k_kernel(const double *__restrict__ A1, const double *__restrict__ A2, int nao, int mode,
                                int hermi, double *__restrict__ vk)
{
        const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        if (e >= (long long)nao * nao) return;
        int x = (int)(e / nao), y = (int)(e % nao);
        double sign = 1.0;
        // hermi_triu: the upper triangle is the (negated) mirror of the lower
        if (hermi != 0 && x < y) {
                const int t = x; x = y; y = t;
                if (hermi == 2) sign = -1.0;
        }
        const size_t xy = (size_t)x * nao + y, yx = (size_t)y * nao + x;
        double v;
        switch (mode) {
        case 0: v = A1[xy] + A2[yx]; break;
        case 1: v = A1[xy] + A1[yx]; break;
        case 2: v = A1[xy] - A1[yx]; break;
        default: v = A1[xy]; break;
        }
        vk[e] = sign * v;
}

__global__ void transpose_kernel(const double *__restrict__ D, int nao, double *__restrict__ Dt)
{
        const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        if (e >= (long long)nao * nao) return;
        const int x = (int)(e / nao), y = (int)(e % nao);
        Dt[e] = D[(size_t)y * nao + x];
}

inline unsigned blocks_for(long long n, int b) { return (unsigned)((n + b - 1) / b); }

int check(const char *what, std::string &err)
{
        const cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) return 0;
        err = std::string(what) + ": " + cudaGetErrorString(e);
        return 1;
}

// shared memory of a block: two density slabs, the row weights, the ring
constexpr size_t pass_smem(int B, int nao)
{
        return sizeof(double) * (2 * (size_t)B * nao + B * B + (size_t)STAGES * B * NT);
}

template <int B, bool S8>
int launch_pass(const IncoreArgs &a, cudaStream_t s, std::string &err)
{
        const size_t smem = pass_smem(B, a.nao);
        cudaError_t e = cudaFuncSetAttribute(incore_fast_kernel<B, S8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) {
                err = std::string("in-core kernel configuration: ") + cudaGetErrorString(e);
                return 1;
        }
        const int n = a.nf[0] + a.nf[1] + a.nf[2] + a.nf[3];
        if (n > 0) {
                incore_fast_kernel<B, S8><<<n, NT, smem, s>>>(a);
                if (check("in-core kernel launch", err)) return 1;
        }
        return 0;
}

} // namespace

// 8 AO rows per block: a lane keeps 4 x B doubles in registers (its J-row
// image sums and density rows), which B = 8 keeps under the 128 registers of
// two resident blocks.  The entry point takes bases of up to 906 functions (a
// tensor of 675 GB in s8: memory ends earlier); their two density slabs fit a
// block beside the ring of entries.
static_assert(pass_smem(8, 906) <= 227 * 1024, "the largest basis fits a block");
int incore_block(int nao)
{
        return nao <= 906 ? 8 : 0;
}

void incore_items(int nao, int s8, int B, int nsm, std::vector<int4> (&items)[4])
{
        for (auto &v : items) v.clear();
        const long long npair = (long long)nao * (nao + 1) / 2;
        const int nb = (nao + B - 1) / B;
        // columns of a window: 2048, less where that leaves fewer than four
        // blocks per SM (nao 64: 107 us with 50 blocks)
        long long total = 0;   // columns of all block pairs
        for (int I = 0; I < nb; I++)
                for (int J = 0; J <= I; J++) {
                        const long long i1 = std::min(nao, (I + 1) * B) - 1;
                        total += s8 ? i1 * (i1 + 1) / 2 + 1 : npair;
                }
        const long long want = total / (4ll * nsm * NT) * NT;
        const long long window = std::min<long long>(2048, std::max<long long>(NT, want));
        auto split = [&](std::vector<int4> &v, int I, int J, long long c0, long long c1) {
                for (long long c = c0; c < c1; c += window)
                        v.push_back(make_int4(I, J, (int)c, (int)std::min(c1, c + window)));
        };
        for (int I = 0; I < nb; I++)
                for (int J = 0; J <= I; J++) {
                        const int imax = std::min(nao, (I + 1) * B) - 1;
                        const int jmax = std::min(std::min(nao, (J + 1) * B) - 1, imax);
                        const long long pmax = (long long)imax * (imax + 1) / 2 + jmax;
                        const int diag = I == J ? 2 : 0;
                        if (!s8) {
                                split(items[diag], I, J, 0, npair);
                        } else {
                                // the block's first row (i0, j0): columns
                                // before it are below the packed diagonal for
                                // every row of the block
                                const long long i0 = (long long)I * B;
                                const long long pmin = i0 * (i0 + 1) / 2 + (long long)J * B;
                                split(items[diag], I, J, 0, pmin);
                                split(items[diag + 1], I, J, pmin, pmax + 1);
                        }
                }
}

int launch_incore_pass(const IncoreArgs &a, cudaStream_t s, std::string &err)
{
        const int B = incore_block(a.nao);
        if (B == 8) return a.s8 ? launch_pass<8, true>(a, s, err) : launch_pass<8, false>(a, s, err);
        err = "in-core contraction: nao too large for the shared-memory slabs";
        return 1;
}

int launch_incore_tridm(const double *D, int nao, double *t, cudaStream_t s, std::string &err)
{
        const long long np = (long long)nao * (nao + 1) / 2;
        tridm_kernel<<<blocks_for(np, 256), 256, 0, s>>>(D, nao, t);
        return check("in-core pair density", err);
}

int launch_incore_unpack_j(const double *Jp, int nao, double *vj, cudaStream_t s, std::string &err)
{
        unpack_j_kernel<<<blocks_for((long long)nao * nao, 256), 256, 0, s>>>(Jp, nao, vj);
        return check("in-core J unpack", err);
}

int launch_incore_finish_k(const double *A1, const double *A2, int nao, int mode, int hermi, double *vk,
                           cudaStream_t s, std::string &err)
{
        finish_k_kernel<<<blocks_for((long long)nao * nao, 256), 256, 0, s>>>(A1, A2, nao, mode, hermi, vk);
        return check("in-core K finish", err);
}

int launch_incore_transpose(const double *D, int nao, double *Dt, cudaStream_t s, std::string &err)
{
        transpose_kernel<<<blocks_for((long long)nao * nao, 256), 256, 0, s>>>(D, nao, Dt);
        return check("in-core transpose", err);
}

} // namespace b200jk
