// Native-FP64 kernels: the DMMA gather-GEMM ("plain path" contraction layer) and the
// HBM-bound elementwise / reduction kernels of the iteration.
//
// The GEMM computes, for one planned block contraction,
//   C[Cm_v[m] + Cn_w[n]] += s_vw * alpha * sum_k A[Am[m]+Ak[k]] * B[Bk[k]+Bn[n]]
// i.e. a GEMM whose operands are gathered straight from the stored tensor blocks
// through per-dimension offset tables (no separate transpose pass), and whose
// epilogue scatters into the output block, once per antisymmetric image.
#include <atomic>
#include <cstdint>
#include <map>
#include <mutex>
#include <set>
#include <utility>
#include <algorithm>
#include <stdexcept>
#include <cuda_runtime.h>

#include "kernels.hpp"

namespace ccsd {
namespace kern {

std::atomic<int64_t> g_launches{0};
int64_t launch_count() { return g_launches.load(); }
void reset_launch_count() { g_launches = 0; }
#define COUNT_LAUNCH() (g_launches++)

// dynamic shared memory above 48 KiB must be opted into once per kernel and device;
// contexts on several host threads may launch the same kernel first
void set_smem_once(const void* kernel, int bytes) {
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (done.insert({kernel, dev}).second) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// ---------------------------------------------------------------------------
// FP64 DMMA gather-GEMM
// ---------------------------------------------------------------------------
namespace {

constexpr int BK = 16;                  // k per chunk
constexpr int TILE_THREADS = 128;       // 2 x 2 warps, each a quarter of the tile

// Tile shapes.  The FP64 tensor pipe (36.8 TFLOP/s measured for m8n8k4) bounds large
// products.  64 x 64 (32 x 32 per warp, 64 accumulator registers) leaves room for four CTAs
// of four warps per SM, whose barriers and copy latencies hide behind one another's
// products: 28.6 TFLOP/s at M=25600 N=400 K=4096, 29.9 at 2048^3, 31.2 at 2304 x 2304 x 16384 (pipe 84% busy),
// against 25.4 for 128 x 64 tiles with two CTAs per SM and 18.5-22.7 for 128 x 128 with one;
// the 128 x 64 kernel with one CTA per SM before it ran the ladder of o=20 v=160 at 13.5.
// With extents that leave every other pair misaligned (8-byte copies) it keeps 22.3, 28.5 at 2401 x 2401 x 16641.
// 32 x 32 (16 x 16 per warp) takes the products that would leave a 64 x 64 tile mostly empty.
template <int ROWS>
struct Tile {
    static constexpr int BM = ROWS, BN = ROWS, WM = ROWS / 2, WN = ROWS / 2, STAGES = 3;
    static constexpr int MT = WM / 8, NT = WN / 8;
    static constexpr int PER_SM = ROWS == 64 ? 4 : 8;
    static constexpr int LD = ROWS + 2;                 // [k][row] layout: 2 mod 8 doubles
    static constexpr int ELEMS = BM * BN;
};

template <class T, bool AK, bool BKc>
struct TileSmem {
    static constexpr int a_elems = AK ? T::BM * BK : BK * T::LD;
    static constexpr int b_elems = BKc ? T::BN * BK : BK * T::LD;
    static constexpr size_t bytes = (size_t)T::STAGES * (a_elems + b_elems) * sizeof(double) + 2 * 2 * BK * sizeof(int64_t);
};

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool valid) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    int sz = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// [row][k] tiles: 16 k = eight 16-byte units per row, unit XOR 4 on odd rows, so that the
// 16-byte fragment reads of a quarter warp (2 rows x 4 units) fall on different banks
__device__ __forceinline__ int tile_rk(int r, int k) { return r * BK + (k ^ ((r & 1) << 3)); }

// Copies one operand's rows x BK tiles into shared memory, two neighbours at a time (along
// k where the operand is contiguous there, else along the rows): one 16-byte copy where the
// two are adjacent and aligned, two 8-byte copies otherwise.  A thread's rows are the same
// for every chunk and stay in registers; the chunk's k offsets come from shared memory.
template <int ROWS, int LD, bool KC>
struct TileLoader {
    static constexpr int N = ROWS * BK / 2 / TILE_THREADS;   // pairs per thread
    static constexpr int NR = KC ? N : 2;
    int64_t row[NR];                                         // -1 past the last row
    bool adj = true;                                         // the two rows of a pair are adjacent
    __device__ __forceinline__ void init(const int64_t* __restrict__ R, int r0, int nrows, int64_t parity) {
        const int tid = threadIdx.x;
        if (KC) {
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int r = r0 + tid / (BK / 2) + (TILE_THREADS / (BK / 2)) * i;
                row[i] = r < nrows ? __ldg(R + r) + parity : -1;
            }
        } else {
            const int r = r0 + 2 * (tid % (ROWS / 2));
            row[0] = r < nrows ? __ldg(R + r) + parity : -1;
            row[1] = r + 1 < nrows ? __ldg(R + r + 1) + parity : -1;
            adj = row[0] >= 0 && row[1] == row[0] + 1;
        }
    }
    // X is the operand moved down to a 16-byte boundary (the parity sits in the row
    // offsets); tab holds the chunk's BK offsets, -1 past K
    __device__ __forceinline__ void copy(double* dst, const double* __restrict__ X, const int64_t* tab) const {
        const int tid = threadIdx.x;
#pragma unroll
        for (int i = 0; i < N; i++) {
            int64_t o0, o1;
            bool v0, v1;
            double* d;
            if (KC) {
                const int k = 2 * (tid % (BK / 2)), r = tid / (BK / 2) + (TILE_THREADS / (BK / 2)) * i;
                const int64_t k0 = tab[k], k1 = tab[k + 1];
                o0 = row[i] + k0;
                o1 = row[i] + k1;
                v0 = (row[i] | k0) >= 0;
                v1 = (row[i] | k1) >= 0;
                d = dst + tile_rk(r, k);
            } else {
                const int k = tid / (ROWS / 2) + (TILE_THREADS / (ROWS / 2)) * i;
                const int64_t kk = tab[k];
                o0 = row[0] + kk;
                o1 = row[1] + kk;
                v0 = (row[0] | kk) >= 0;
                v1 = (row[1] | kk) >= 0;
                d = dst + k * LD + 2 * (tid % (ROWS / 2));
            }
            if (v0 && v1 && (KC ? o1 == o0 + 1 : adj) && !(o0 & 1)) {
                cp_async16(d, X + o0);
            } else {
                cp_async8(d, v0 ? X + o0 : X, v0);
                cp_async8(d + 1, v1 ? X + o1 : X, v1);
            }
        }
    }
};

template <class T>
struct TileAcc {
    double v[T::MT][T::NT][2];
};

// Row / column of the tile that accumulator (i, j, c) of this lane holds.  Operands stored
// [k][row] are read two neighbouring rows at a time, which interleaves the rows of two
// 8-row fragments.
template <class T, bool AK>
__device__ __forceinline__ int tile_row(int i) {
    const int warp = threadIdx.x >> 5, fr = (threadIdx.x & 31) >> 2;
    return (warp & 1) * T::WM + (AK ? 8 * i + fr : 16 * (i >> 1) + 2 * fr + (i & 1));
}
template <class T, bool BKc>
__device__ __forceinline__ int tile_col(int j, int c) {
    const int warp = threadIdx.x >> 5, fk = threadIdx.x & 3;
    return (warp >> 1) * T::WN + (BKc ? 8 * j + 2 * fk + c : 16 * (j >> 1) + 4 * fk + 2 * c + (j & 1));
}

// Chunks [kt0, kt0 + nkt) of the tile at (m0, n0) into acc.  Three stages of cp.async; the
// k offsets of a chunk are fetched to a register two chunks ahead of the chunk's copies and
// staged in shared memory one chunk ahead, so no copy waits on a table load.  Within an
// 8-k block a lane takes k = 2 (lane % 4) and the next one: 16-byte fragment reads, the
// same permutation of k for both operands.
template <class T, bool AK, bool BKc>
__device__ __forceinline__ void tile_product(const GemmArgs& g, int m0, int n0, int kt0, int nkt, TileAcc<T>& acc,
                                             unsigned char* smem_raw) {
    using S = TileSmem<T, AK, BKc>;
    constexpr int MT = T::MT, NT = T::NT, STAGES = T::STAGES;
    double* As = reinterpret_cast<double*>(smem_raw);
    double* Bs = As + STAGES * S::a_elems;
    int64_t* tab = reinterpret_cast<int64_t*>(Bs + STAGES * S::b_elems);   // [2][A | B][BK]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp & 1) * T::WM, wn = (warp >> 1) * T::WN;
    const int64_t pa = (reinterpret_cast<uintptr_t>(g.A) >> 3) & 1, pb = (reinterpret_cast<uintptr_t>(g.B) >> 3) & 1;
    const double* A = g.A - pa;
    const double* B = g.B - pb;
    TileLoader<T::BM, T::LD, AK> la;
    TileLoader<T::BN, T::LD, BKc> lb;
    la.init(g.Am, m0, g.M, pa);
    lb.init(g.Bn, n0, g.N, pb);
    const int64_t* kt_src = tid < BK ? g.Ak : g.Bk;
    const int K = g.K;
    auto fetch = [&](int c) -> int64_t {
        const int k = (kt0 + c) * BK + (tid & (BK - 1));
        return (tid < 2 * BK && k < K) ? __ldg(kt_src + k) : -1;
    };
    auto put = [&](int c, int64_t v) {
        if (tid < 2 * BK) tab[(c & 1) * 2 * BK + tid] = v;
    };
    auto load = [&](int c) {
        const int64_t* t = tab + (c & 1) * 2 * BK;
        la.copy(As + (c % STAGES) * S::a_elems, A, t);
        lb.copy(Bs + (c % STAGES) * S::b_elems, B, t + BK);
    };
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) acc.v[i][j][0] = acc.v[i][j][1] = 0.0;

    int64_t next = fetch(0);
#pragma unroll
    for (int c = 0; c < STAGES - 1; c++) {
        put(c, next);
        next = fetch(c + 1);
        __syncthreads();
        if (c < nkt) load(c);
        cp_commit();
    }
    put(STAGES - 1, next);
    next = fetch(STAGES);
    const int fr = lane >> 2, fk = lane & 3;
    for (int kt = 0; kt < nkt; kt++) {
        cp_wait<STAGES - 2>();
        __syncthreads();
        if (kt + STAGES - 1 < nkt) load(kt + STAGES - 1);
        cp_commit();
        put(kt + STAGES, next);
        next = fetch(kt + STAGES + 1);
        const double* as = As + (kt % STAGES) * S::a_elems;
        const double* bs = Bs + (kt % STAGES) * S::b_elems;
#pragma unroll
        for (int kb = 0; kb < BK; kb += 8) {
            double af[2][MT], bf[2][NT];     // [k of the lane's pair][fragment]
            if (AK) {
#pragma unroll
                for (int i = 0; i < MT; i++) {
                    const double2 v = *reinterpret_cast<const double2*>(as + tile_rk(wm + 8 * i + fr, kb + 2 * fk));
                    af[0][i] = v.x;
                    af[1][i] = v.y;
                }
            } else {
#pragma unroll
                for (int s = 0; s < 2; s++)
#pragma unroll
                    for (int i = 0; i < MT; i += 2) {
                        const double2 v = *reinterpret_cast<const double2*>(as + (kb + 2 * fk + s) * T::LD + wm + 8 * i + 2 * fr);
                        af[s][i] = v.x;
                        af[s][i + 1] = v.y;
                    }
            }
            if (BKc) {
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    const double2 v = *reinterpret_cast<const double2*>(bs + tile_rk(wn + 8 * j + fr, kb + 2 * fk));
                    bf[0][j] = v.x;
                    bf[1][j] = v.y;
                }
            } else {
#pragma unroll
                for (int s = 0; s < 2; s++)
#pragma unroll
                    for (int j = 0; j < NT; j += 2) {
                        const double2 v = *reinterpret_cast<const double2*>(bs + (kb + 2 * fk + s) * T::LD + wn + 8 * j + 2 * fr);
                        bf[s][j] = v.x;
                        bf[s][j + 1] = v.y;
                    }
            }
#pragma unroll
            for (int s = 0; s < 2; s++)
#pragma unroll
                for (int i = 0; i < MT; i++)
#pragma unroll
                    for (int j = 0; j < NT; j++) dmma(acc.v[i][j][0], acc.v[i][j][1], af[s][i], bf[s][j]);
        }
    }
    cp_wait<0>();
}

// one row of fragments of a finished tile: raw to a dense product, or scattered into C
template <class T, bool AK, bool BKc>
__device__ __forceinline__ void tile_write_row(const GemmArgs& g, int m0, int n0, int i, const double (&v)[T::NT][2],
                                               double* dense) {
    constexpr int NT = T::NT;
    const int m = m0 + tile_row<T, AK>(i);
    if (m >= g.M) return;
    if (dense) {
        double* w = dense + (int64_t)m * g.N;
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int n = n0 + tile_col<T, BKc>(j, c);
                if (n < g.N) w[n] = v[j][c];
            }
        return;
    }
    if (g.nvm == 1 && g.nvn == 1) {
        // one destination per element: the reads of the row first, then its writes, so that
        // the read-modify-writes of a thread overlap instead of running one by one
        const int64_t cm = __ldg(g.Cm[0] + m);
        const double sc = g.alpha * g.vsign[0];
        int64_t off[2 * NT];
        double old[2 * NT];
#pragma unroll
        for (int t = 0; t < 2 * NT; t++) {
            const int n = n0 + tile_col<T, BKc>(t >> 1, t & 1);
            off[t] = n < g.N ? cm + __ldg(g.Cn[0] + n) : -1;
        }
#pragma unroll
        for (int t = 0; t < 2 * NT; t++) old[t] = off[t] >= 0 ? g.C[off[t]] : 0.0;
#pragma unroll
        for (int t = 0; t < 2 * NT; t++)
            if (off[t] >= 0) g.C[off[t]] = old[t] + sc * v[t >> 1][t & 1];
        return;
    }
    // every destination variant in turn
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int n = n0 + tile_col<T, BKc>(j, c);
            if (n >= g.N) continue;
            const double x = g.alpha * v[j][c];
            for (int a = 0; a < g.nvm; a++)
                for (int b = 0; b < g.nvn; b++) g.C[g.Cm[a][m] + g.Cn[b][n]] += g.vsign[a * g.nvn + b] * x;
        }
}

// One problem, one CTA per output tile (the integral build's products; a statement's share
// grouped launches).  The shorter side of the tile grid runs fastest, so that the CTAs in flight
// share the panels of the longer operand.
template <class T, bool AK, bool BKc>
__global__ void __launch_bounds__(TILE_THREADS, T::PER_SM) gemm_fp64_kernel(GemmArgs g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tm = (g.M + T::BM - 1) / T::BM, tn = (g.N + T::BN - 1) / T::BN;
    const int t = blockIdx.x;
    const int m0 = (tm <= tn ? t % tm : t / tn) * T::BM, n0 = (tm <= tn ? t / tm : t % tn) * T::BN;
    TileAcc<T> acc;
    tile_product<T, AK, BKc>(g, m0, n0, 0, (g.K + BK - 1) / BK, acc, smem_raw);
#pragma unroll
    for (int i = 0; i < T::MT; i++) tile_write_row<T, AK, BKc>(g, m0, n0, i, acc.v[i], nullptr);
}

// Many problems with pairwise disjoint outputs: each CTA walks its segments (a tile and a
// range of its chunks, laid out by plan_tile_work).  A segment that covers its tile writes
// the output; one that shares its tile with other CTAs leaves its accumulators in slot
// seg.slot of ws, in register order.
template <class T, bool AK, bool BKc>
__global__ void __launch_bounds__(TILE_THREADS, T::PER_SM)
    gemm_fp64_grouped_kernel(const GemmArgs* __restrict__ probs, const TileSeg* __restrict__ segs,
                             const int* __restrict__ seg_start, double* __restrict__ ws) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int s1 = seg_start[blockIdx.x + 1];
    for (int s = seg_start[blockIdx.x]; s < s1; s++) {
        const TileSeg seg = segs[s];
        const GemmArgs& g = probs[seg.prob];
        TileAcc<T> acc;
        tile_product<T, AK, BKc>(g, seg.m0, seg.n0, seg.kt0, seg.nkt, acc, smem_raw);
        if (seg.slot >= 0) {
            double* w = ws + (int64_t)seg.slot * T::ELEMS + threadIdx.x;
#pragma unroll
            for (int i = 0; i < T::MT; i++)
#pragma unroll
                for (int j = 0; j < T::NT; j++)
#pragma unroll
                    for (int c = 0; c < 2; c++) w[((i * T::NT + j) * 2 + c) * TILE_THREADS] = acc.v[i][j][c];
        } else {
            double* dense = g.partial_out ? g.ws : nullptr;
#pragma unroll
            for (int i = 0; i < T::MT; i++) tile_write_row<T, AK, BKc>(g, seg.m0, seg.n0, i, acc.v[i], dense);
        }
        __syncthreads();   // the stages and the offset table are free for the next segment
    }
}

// The tiles that several CTAs share: blockIdx.y's row of fragments of tile blockIdx.x, its
// parts added in order of k
template <class T, bool AK, bool BKc>
__global__ void __launch_bounds__(TILE_THREADS)
    tile_fold_kernel(const GemmArgs* __restrict__ probs, const TileFold* __restrict__ folds, const double* __restrict__ ws) {
    const TileFold f = folds[blockIdx.x];
    const GemmArgs& g = probs[f.prob];
    const int i = blockIdx.y;
    const double* w = ws + (int64_t)f.slot0 * T::ELEMS + (int64_t)i * T::NT * 2 * TILE_THREADS + threadIdx.x;
    double v[T::NT][2];
#pragma unroll
    for (int j = 0; j < T::NT; j++) v[j][0] = v[j][1] = 0.0;
#pragma unroll 4
    for (int p = 0; p < f.parts; p++, w += T::ELEMS)
#pragma unroll
        for (int j = 0; j < T::NT; j++)
#pragma unroll
            for (int c = 0; c < 2; c++) v[j][c] += w[(j * 2 + c) * TILE_THREADS];
    tile_write_row<T, AK, BKc>(g, f.m0, f.n0, i, v, g.partial_out ? g.ws : nullptr);
}

// Shared-output groups.  Latency bounds this kernel (a few KB to a few MB of partials): a
// thread adds all terms of its element, their loads in flight together, and writes once.
// The terms of a node are added in plan order, the nodes of an item one after the other.
__global__ void __launch_bounds__(256) fold_groups_kernel(const FoldItem* __restrict__ items, const FoldNode* __restrict__ nodes,
                                                          const FoldTerm* __restrict__ terms) {
    const FoldItem it = items[blockIdx.x];
    for (int q = it.n0; q < it.n1; q++) {
        const FoldNode& f = nodes[q];
        const int mn = f.M * f.N, hi = min(it.l1, mn), t1 = f.term0 + f.nterms;
        for (int l = it.l0 + threadIdx.x; l < hi; l += blockDim.x) {
            double v = 0.0;
            for (int t = f.term0; t < t1; t++) {
                const double* p = terms[t].part + l;
                const int ks = terms[t].ks;
                double s = 0.0;
#pragma unroll 8
                for (int z = 0; z < ks; z++) s += p[(int64_t)z * mn];
                v += terms[t].scale * s;
            }
            const int m = l / f.N, n = l % f.N;
            for (int a = 0; a < f.nvm; a++)
                for (int b = 0; b < f.nvn; b++) f.C[f.Cm[a][m] + f.Cn[b][n]] += f.vsign[a * f.nvn + b] * v;
        }
        if (q + 1 < it.n1) __syncthreads();   // the next node may write the same elements
    }
}

// ---------------------------------------------------------------------------
// Skinny FP64 product: one small extent (<= 32) against a long operand.
//   C[Cr_v[r] + Cs_w[s]] += sign_vw * alpha * sum_k L[Lr[r] + Lk[k]] * S[Sk[k] + Sn[s]]
// HBM (the long operand, read once) bounds large products, latency small ones.  Each warp
// takes 32 rows and walks k in steps of 16, loading its m8n8k4 fragments straight from global
// memory: a lane reads L at row lane/4 + 8i and k = 4u + lane%4, 64-byte runs along the rows or
// 32-byte runs along k, whole sectors either way; the k offsets of the next step are fetched
// while the step's loads are in flight.  The small operand comes through L1, which the warps
// of a CTA share.  VAMEF t(fm) over 33856 rows x 4416 k (1.2 GB) takes 184 us, 6.5 TB/s, 310 us
// with the long operand staged in shared memory and two CTAs per SM; VAMEF t(fi) of o=24
// v=184 2.68 ms, 3.14 before.  No shared-memory stages, so 12 (NS > 16) to 20 (NS <= 8) warps per SM hide one
// another's latencies and a product of few k costs few round trips.  The four warps of a CTA
// are 4 / wk slots of 32 rows times wk parts of the k range, the parts added in shared memory;
// a long K over few rows is also cut over nz CTAs into ws[z][r][s], folded in order of z.
// ---------------------------------------------------------------------------
constexpr int SK_THREADS = 128, SK_STEP = 16, SK_ROWS = 32;
constexpr int SK_RED = SK_ROWS + 2;           // pitch of a warp's [s][r] fragments: 2 mod 16 doubles
constexpr int skinny_per_sm(int nt) { return nt == 1 ? 5 : nt == 2 ? 4 : 3; }

// one CTA: row tile `rtile` (SK_ROWS * 4 / wk rows) over K range z of nz
template <int NT>
__device__ __forceinline__ void skinny_body(const SkinnyArgs& g, int rtile, int z, int nz) {
    constexpr int MT = SK_ROWS / 8, U = SK_STEP / 4;
    __shared__ double red[SK_THREADS / 32][8 * NT * SK_RED];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int fr = lane >> 2, fk = lane & 3;
    const int wk = g.wk;
    const int r0 = (rtile * (SK_THREADS / 32 / wk) + warp / wk) * SK_ROWS;

    // steps of the CTA's range, and this warp's part of them
    const int steps = (g.K + SK_STEP - 1) / SK_STEP, per = (steps + nz - 1) / nz;
    const int z0 = min(steps, z * per), z1 = min(steps, z0 + per);
    const int pw = (z1 - z0 + wk - 1) / wk;
    const int kb = min(z1, z0 + (warp % wk) * pw) * SK_STEP, ke = min(g.K, min(z1, z0 + (warp % wk + 1) * pw) * SK_STEP);

    double acc[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

    if (r0 < g.R && kb < ke) {
        int64_t lr[MT], sn[NT];               // -1 past the last row / column
#pragma unroll
        for (int i = 0; i < MT; i++) lr[i] = r0 + 8 * i + fr < g.R ? __ldg(g.Lr + r0 + 8 * i + fr) : -1;
#pragma unroll
        for (int j = 0; j < NT; j++) sn[j] = 8 * j + fr < g.NS ? __ldg(g.Sn + 8 * j + fr) : -1;
        auto offsets = [&](int k0, int64_t* lk, int64_t* sk) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int k = k0 + 4 * u + fk;
                const bool ok = k < ke;
                lk[u] = !ok ? -1 : (g.lk_affine ? g.lk0 + g.lk_step * k : __ldg(g.Lk + k));
                sk[u] = !ok ? -1 : (g.sk_affine ? g.sk0 + g.sk_step * k : __ldg(g.Sk + k));
            }
        };
        int64_t lk[U], sk[U];
        offsets(kb, lk, sk);
        for (int k0 = kb; k0 < ke; k0 += SK_STEP) {
            double a[U][MT], b[U][NT];
#pragma unroll
            for (int u = 0; u < U; u++) {
#pragma unroll
                for (int i = 0; i < MT; i++) a[u][i] = (lk[u] | lr[i]) >= 0 ? __ldg(g.L + lr[i] + lk[u]) : 0.0;
#pragma unroll
                for (int j = 0; j < NT; j++) b[u][j] = (sk[u] | sn[j]) >= 0 ? __ldg(g.S + sk[u] + sn[j]) : 0.0;
            }
            if (k0 + SK_STEP < ke) offsets(k0 + SK_STEP, lk, sk);
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int i = 0; i < MT; i++)
#pragma unroll
                    for (int j = 0; j < NT; j++) dmma(acc[i][j][0], acc[i][j][1], a[u][i], b[u][j]);
        }
    }

    // lane holds rows r0 + 8i + fr, columns 8j + 2 fk + {0, 1}
    const bool raw = nz > 1 || g.partial;
    double* wz = raw ? g.ws + (int64_t)z * g.R * g.NS : nullptr;
    if (wk > 1) {
        // the parts of k through shared memory, then one thread per element: lanes along the
        // rows of C, along the columns of a partial
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) red[warp][(8 * j + 2 * fk + h) * SK_RED + 8 * i + fr] = acc[i][j][h];
        __syncthreads();
        const int rows = SK_ROWS * (SK_THREADS / 32 / wk), rb = rtile * rows;
        for (int e = threadIdx.x; e < rows * g.NS; e += SK_THREADS) {
            const int r = raw ? e / g.NS : e % rows, s = raw ? e % g.NS : e / rows;
            if (rb + r >= g.R) continue;
            double v = 0.0;
            for (int w = 0; w < wk; w++) v += red[r / SK_ROWS * wk + w][s * SK_RED + r % SK_ROWS];
            if (raw) {
                wz[(int64_t)(rb + r) * g.NS + s] = v;
                continue;
            }
            v *= g.alpha;
            for (int a = 0; a < g.nvr; a++)
                for (int b = 0; b < g.nvs; b++) g.C[g.Cr[a][rb + r] + g.Cs[b][s]] += g.vsign[a * g.nvs + b] * v;
        }
        return;
    }
    if (raw) {
#pragma unroll
        for (int i = 0; i < MT; i++) {
            const int r = r0 + 8 * i + fr;
            if (r >= g.R) continue;
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int s = 8 * j + 2 * fk + h;
                    if (s < g.NS) wz[(int64_t)r * g.NS + s] = acc[i][j][h];
                }
        }
        return;
    }
    if (g.nvr == 1 && g.nvs == 1) {
        // one destination per element: the reads of a row first, then its writes
        const double sc = g.alpha * g.vsign[0];
#pragma unroll
        for (int i = 0; i < MT; i++) {
            const int r = r0 + 8 * i + fr;
            if (r >= g.R) continue;
            const int64_t cr = __ldg(g.Cr[0] + r);
            int64_t off[2 * NT];
            double old[2 * NT];
#pragma unroll
            for (int q = 0; q < 2 * NT; q++) {
                const int s = 8 * (q >> 1) + 2 * fk + (q & 1);
                off[q] = s < g.NS ? cr + __ldg(g.Cs[0] + s) : -1;
            }
#pragma unroll
            for (int q = 0; q < 2 * NT; q++) old[q] = off[q] >= 0 ? g.C[off[q]] : 0.0;
#pragma unroll
            for (int q = 0; q < 2 * NT; q++)
                if (off[q] >= 0) g.C[off[q]] = old[q] + sc * acc[i][q >> 1][q & 1];
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < MT; i++) {
        const int r = r0 + 8 * i + fr;
        if (r >= g.R) continue;
        int64_t cr[2];
        cr[0] = g.Cr[0][r];
        cr[1] = g.nvr > 1 ? g.Cr[1][r] : 0;
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int s = 8 * j + 2 * fk + h;
                if (s >= g.NS) continue;
                const double v = g.alpha * acc[i][j][h];
                for (int a = 0; a < g.nvr; a++)
                    for (int b = 0; b < g.nvs; b++) g.C[cr[a] + g.Cs[b][s]] += g.vsign[a * g.nvs + b] * v;
            }
    }
}

template <int NT>
__global__ void __launch_bounds__(SK_THREADS, skinny_per_sm(NT)) skinny_kernel(SkinnyArgs g) {
    skinny_body<NT>(g, blockIdx.x, blockIdx.y, gridDim.y);
}

// Grouped launch: ctas[t] = (problem, row tile + tiles * K range) of CTA t
template <int NT>
__global__ void __launch_bounds__(SK_THREADS, skinny_per_sm(NT))
    skinny_grouped_kernel(const SkinnyArgs* __restrict__ probs, const int2* __restrict__ ctas) {
    const int2 c = ctas[blockIdx.x];
    const SkinnyArgs& g = probs[c.x];
    const int tiles = skinny_tiles(g);
    skinny_body<NT>(g, c.y % tiles, c.y / tiles, g.nz);
}

// The K ranges of a product added in order: eight threads per element take contiguous
// ranges of z each and their sums are added in order, so that a product of many ranges and
// few elements keeps many loads in flight (T1 residual of o=20 v=160, 3200 elements x 296
// ranges: 53 us with one thread walking all ranges).
__global__ void __launch_bounds__(256) skinny_fold_kernel(SkinnyArgs g, int ks) {
    __shared__ double part[8][33];
    const int64_t rs = (int64_t)g.R * g.NS;
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int per = (ks + 7) / 8, z0 = min(ks, grp * per), z1 = min(ks, z0 + per);
    for (int64_t l0 = blockIdx.x * 32ll; l0 < rs; l0 += gridDim.x * 32ll) {
        const int64_t l = l0 + lane;
        double sum = 0.0;
        if (l < rs) {
#pragma unroll 8
            for (int z = z0; z < z1; z++) sum += g.ws[z * rs + l];
        }
        part[grp][lane] = sum;
        __syncthreads();
        if (grp == 0 && l < rs) {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < 8; q++) v += part[q][lane];
            v *= g.alpha;
            const int r = (int)(l / g.NS), s = (int)(l % g.NS);
            for (int a = 0; a < g.nvr; a++)
                for (int b = 0; b < g.nvs; b++) g.C[g.Cr[a][r] + g.Cs[b][s]] += g.vsign[a * g.nvs + b] * v;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Short products: M, N <= 64, long K.  Each warp of a CTA walks its own part of the CTA's
// K range, 16 k per step (8 for the widest shapes), loading the m8n8k4 fragments straight
// from global memory (a lane reads A[m = lane/4 + 8i][k] and B[k][n = lane/4 + 8j] for
// k = 4u + lane%4: 32-byte runs along k, or 64-byte runs along m / n, both whole
// sectors); the k offsets of the next step are fetched while the current step's data
// loads are in flight.  The eight warps' fragments are added in warp order in shared
// memory and the CTA writes one partial M x N product.
// ---------------------------------------------------------------------------
constexpr int SH_THREADS = 256;
constexpr int SH_KGRAN = 16 * (SH_THREADS / 32);   // kper is a multiple of this (128)

template <int MT, int NT>
__global__ void __launch_bounds__(SH_THREADS, MT * NT > 8 ? 1 : 2)
    short_grouped_kernel(const ShortDesc* __restrict__ descs, const int* __restrict__ cta_start, int nprob) {
    // steps of 16 k (8 for the widest shapes, whose loads of a step would not fit the registers)
    constexpr int SH_U = MT + NT <= 6 ? 4 : 2, SH_KSTEP = 4 * SH_U;
    __shared__ ShortDesc sd;
    __shared__ int sp;
    // the warps' fragments for the reduction (dynamic: 64 KB for 16 fragments)
    extern __shared__ __align__(16) unsigned char short_smem[];
    auto red = reinterpret_cast<double(*)[MT * 8 * NT * 8]>(short_smem);
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        int lo = 0, hi = nprob - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (cta_start[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        sp = lo;
        sd = descs[lo];
    }
    __syncthreads();
    const ShortDesc& g = sd;
    const int local = t - cta_start[sp];
    const int fr = lane >> 2, fk = lane & 3;
    int64_t am[MT], bn[NT];
#pragma unroll
    for (int i = 0; i < MT; i++) am[i] = (8 * i + fr < g.M) ? __ldg(g.Am + 8 * i + fr) : -1;
#pragma unroll
    for (int j = 0; j < NT; j++) bn[j] = (8 * j + fr < g.N) ? __ldg(g.Bn + 8 * j + fr) : -1;

    const int kw = g.kper / (SH_THREADS / 32);               // k per warp (a multiple of 16)
    const int kb = local * g.kper + warp * kw;
    const int ke = min(g.K, kb + kw);
    double acc[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

    auto offsets = [&](int k0, int64_t* ak, int64_t* bk) {
#pragma unroll
        for (int u = 0; u < SH_U; u++) {
            const int k = k0 + 4 * u + fk;
            const bool ok = k < ke;
            ak[u] = !ok ? -1 : (g.ak_affine ? g.ak0 + g.ak_step * k : __ldg(g.Ak + k));
            bk[u] = !ok ? -1 : (g.bk_affine ? g.bk0 + g.bk_step * k : __ldg(g.Bk + k));
        }
    };
    int64_t ak[SH_U], bk[SH_U];
    if (kb < ke) offsets(kb, ak, bk);
    for (int k0 = kb; k0 < ke; k0 += SH_KSTEP) {
        double a[SH_U][MT], b[SH_U][NT];
#pragma unroll
        for (int u = 0; u < SH_U; u++) {
#pragma unroll
            for (int i = 0; i < MT; i++) a[u][i] = (ak[u] >= 0 && am[i] >= 0) ? __ldg(g.A + am[i] + ak[u]) : 0.0;
#pragma unroll
            for (int j = 0; j < NT; j++) b[u][j] = (bk[u] >= 0 && bn[j] >= 0) ? __ldg(g.B + bk[u] + bn[j]) : 0.0;
        }
        if (k0 + SH_KSTEP < ke) offsets(k0 + SH_KSTEP, ak, bk);
#pragma unroll
        for (int u = 0; u < SH_U; u++)
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < NT; j++) dmma(acc[i][j][0], acc[i][j][1], a[u][i], b[u][j]);
    }
    // lane holds rows 8i + fr, columns 8j + 2 fk + {0, 1}
    constexpr int LDR = NT * 8;
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) red[warp][(8 * i + fr) * LDR + 8 * j + 2 * fk + h] = acc[i][j][h];
    __syncthreads();
    double* out = g.part + (int64_t)local * g.M * g.N;
    for (int e = tid; e < g.M * g.N; e += SH_THREADS) {
        const int m = e / g.N, n = e % g.N;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < SH_THREADS / 32; w++) s += red[w][m * LDR + n];
        out[e] = s;
    }
}

template <int MT, int NT>
void launch_short_t(const ShortDesc* d, const int* cta_start, int nprob, int total, cudaStream_t s) {
    constexpr int bytes = (SH_THREADS / 32) * MT * 8 * NT * 8 * (int)sizeof(double);
    set_smem_once((const void*)short_grouped_kernel<MT, NT>, bytes);
    short_grouped_kernel<MT, NT><<<total, SH_THREADS, bytes, s>>>(d, cta_start, nprob);
}

}  // namespace

// n-groups of 8 for a small extent (0: not a skinny product)
int skinny_groups(int M, int N) {
    const int small = std::min(M, N);
    return small > 32 ? 0 : (small + 7) / 8;
}

// Warps that share a row slot (wk), and CTAs (nz) that share a row tile.  wk keeps the 4 / wk
// slots of 32 rows of a tile full (R=184: 3 tiles of 64 rows, not 2 of 128 with two warps of
// the second idle), then splits k inside the CTA, which needs no fold, when the tiles are too
// few and K is short; nz then balances the waves of CTAs against their prologues (about 6
// steps) and the fold, a warp keeping 64 k or more.
SkinnySplit skinny_split(int R, int K, int nt) {
    SkinnySplit s;
    auto tiles = [&](int w) { return ((int64_t)R + SK_ROWS * (4 / w) - 1) / (SK_ROWS * (4 / w)); };
    for (int w : {2, 4})
        if (tiles(w) * (4 / w) * 10 < tiles(s.wk) * (4 / s.wk) * 9) s.wk = w;
    while (s.wk < 4 && K < 4096 && tiles(s.wk) < 2 * 148 && K >= s.wk * 128) s.wk *= 2;
    const int64_t t = tiles(s.wk), slots = 148 * skinny_per_sm(nt), steps = (K + SK_STEP - 1) / SK_STEP;
    const int64_t most = std::min<int64_t>(1024, K / (64 * s.wk));
    if (t >= 4 * slots || most < 2) return s;
    int64_t best = -1;
    for (int64_t nz = 1; nz <= most; nz += std::max<int64_t>(1, nz / 8)) {
        const int64_t per = (steps + nz - 1) / nz;
        const int64_t cost = (t * nz + slots - 1) / slots * ((per + s.wk - 1) / s.wk + 6) + (nz > 1 ? 12 : 0);
        if (best < 0 || cost < best) {
            best = cost;
            s.nz = (int)nz;
        }
    }
    return s;
}

namespace {

template <int NT>
void launch_skinny_t(const SkinnyArgs& a, int ks, cudaStream_t s) {
    skinny_kernel<NT><<<dim3(skinny_tiles(a), ks), SK_THREADS, 0, s>>>(a);
}

void launch_skinny(const GemmArgs& g, int nt, cudaStream_t s) {
    SkinnyArgs a = skinny_args(g);
    int ks = skinny_split(a.R, a.K, nt).nz;
    if (!g.ws || (int64_t)ks * a.R * a.NS > g.ws_elems) ks = 1;
    a.ws = g.ws;
    switch (nt) {
        case 1: launch_skinny_t<1>(a, ks, s); break;
        case 2: launch_skinny_t<2>(a, ks, s); break;
        case 3: launch_skinny_t<3>(a, ks, s); break;
        default: launch_skinny_t<4>(a, ks, s); break;
    }
    COUNT_LAUNCH();
    if (ks > 1) {
        const int64_t rs = (int64_t)a.R * a.NS;
        const int nb = (int)std::min<int64_t>((rs + 31) / 32, 148 * 16);
        skinny_fold_kernel<<<nb, 256, 0, s>>>(a, ks);
        COUNT_LAUNCH();
    }
}

}  // namespace

SkinnyArgs skinny_args(const GemmArgs& g) {
    SkinnyArgs a;
    const bool long_a = g.M >= g.N;
    a.C = g.C;
    a.alpha = g.alpha;
    a.K = g.K;
    if (long_a) {
        a.L = g.A; a.Lr = g.Am; a.Lk = g.Ak; a.S = g.B; a.Sk = g.Bk; a.Sn = g.Bn;
        a.R = g.M; a.NS = g.N; a.nvr = g.nvm; a.nvs = g.nvn;
        for (int v = 0; v < 2; v++) { a.Cr[v] = g.Cm[v]; a.Cs[v] = g.Cn[v]; }
        for (int i = 0; i < 4; i++) a.vsign[i] = g.vsign[i];
        a.lk_affine = g.ak_affine; a.lk0 = g.ak0; a.lk_step = g.ak_step;
        a.sk_affine = g.bk_affine; a.sk0 = g.bk0; a.sk_step = g.bk_step;
    } else {
        a.L = g.B; a.Lr = g.Bn; a.Lk = g.Bk; a.S = g.A; a.Sk = g.Ak; a.Sn = g.Am;
        a.R = g.N; a.NS = g.M; a.nvr = g.nvn; a.nvs = g.nvm;
        for (int v = 0; v < 2; v++) { a.Cr[v] = g.Cn[v]; a.Cs[v] = g.Cm[v]; }
        for (int r = 0; r < g.nvn; r++)
            for (int c = 0; c < g.nvm; c++) a.vsign[r * g.nvm + c] = g.vsign[c * g.nvn + r];
        a.lk_affine = g.bk_affine; a.lk0 = g.bk0; a.lk_step = g.bk_step;
        a.sk_affine = g.ak_affine; a.sk0 = g.ak0; a.sk_step = g.ak_step;
    }
    a.wk = skinny_split(a.R, a.K, skinny_groups(g.M, g.N)).wk;
    return a;
}

void skinny_grouped(const SkinnyArgs* d, const int2* ctas, int nctas, int nt, cudaStream_t s) {
    if (nctas <= 0) return;
    switch (nt) {
        case 1: skinny_grouped_kernel<1><<<nctas, SK_THREADS, 0, s>>>(d, ctas); break;
        case 2: skinny_grouped_kernel<2><<<nctas, SK_THREADS, 0, s>>>(d, ctas); break;
        case 3: skinny_grouped_kernel<3><<<nctas, SK_THREADS, 0, s>>>(d, ctas); break;
        default: skinny_grouped_kernel<4><<<nctas, SK_THREADS, 0, s>>>(d, ctas); break;
    }
    COUNT_LAUNCH();
}

namespace {

template <bool AK, bool BKc>
void launch_fp64(const GemmArgs& g, cudaStream_t s) {
    using T = Tile<64>;
    constexpr size_t bytes = TileSmem<T, AK, BKc>::bytes;
    set_smem_once((const void*)gemm_fp64_kernel<T, AK, BKc>, (int)bytes);
    const int64_t tiles = (int64_t)((g.M + T::BM - 1) / T::BM) * ((g.N + T::BN - 1) / T::BN);
    if (tiles > INT32_MAX) throw std::runtime_error("FP64 GEMM: too many output tiles for the grid");
    gemm_fp64_kernel<T, AK, BKc><<<(unsigned)tiles, TILE_THREADS, bytes, s>>>(g);
    COUNT_LAUNCH();
}

}  // namespace

int skinny_ksplit(int M, int N, int K) {
    const int nt = skinny_groups(M, N);
    return nt ? skinny_split(std::max(M, N), K, nt).nz : 1;
}

void gemm_fp64(const GemmArgs& g, cudaStream_t s) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0) return;
    if (const int nt = g.skinny_ok ? skinny_groups(g.M, g.N) : 0) {
        launch_skinny(g, nt, s);
        return;
    }
    if (g.a_kcontig) {
        if (g.b_kcontig) launch_fp64<true, true>(g, s);
        else launch_fp64<true, false>(g, s);
    } else {
        if (g.b_kcontig) launch_fp64<false, true>(g, s);
        else launch_fp64<false, false>(g, s);
    }
}

int fp64_tile_rows(int M, int N) {
    // 64 unless 32 x 32 tiles cover the product with at most three fifths of the area
    auto area = [&](int64_t r) { return ((M + r - 1) / r) * ((N + r - 1) / r) * r * r; };
    return 5 * area(32) <= 3 * area(64) ? 32 : 64;
}

// Tiles of longer K first.  The tiles of the last full waves run one per CTA; the tiles
// before them (up to two waves, and every tile whose K is more than half of a CTA's share)
// form one range of chunks that is cut into equal pieces, one per CTA of a wave, so that
// neither a last wave that is nearly empty nor a tile of long K keeps the rest waiting.  A
// cut closer to a tile's end than TILE_MIN_CHUNKS / 2 moves there: a short piece would cost
// more in its prologue and its partial tile than it balances.  (597 tiles of K=12720 on 592
// CTA slots ran at 22.5 TFLOP/s one per CTA; with the cuts the three ladder products of o=20
// v=160, 597 + 2800 + 597 tiles, take 21.8 ms at 29.7 TFLOP/s, 47.8 ms before.)
TileWork plan_tile_work(const std::vector<TileProblem>& probs, int rows, bool split) {
    constexpr int TILE_MIN_CHUNKS = 16;
    TileWork w;
    const int64_t slots = 148 * (rows == 64 ? Tile<64>::PER_SM : Tile<32>::PER_SM);
    auto tiles_of = [&](const TileProblem& p) { return (int64_t)((p.M + rows - 1) / rows) * ((p.N + rows - 1) / rows); };
    auto chunks_of = [&](const TileProblem& p) { return (int64_t)(p.K + BK - 1) / BK; };
    std::vector<int> order(probs.size());
    int64_t T = 0, U = 0;
    for (size_t i = 0; i < probs.size(); i++) {
        order[i] = (int)i;
        T += tiles_of(probs[i]);
        U += tiles_of(probs[i]) * chunks_of(probs[i]);
    }
    if (T == 0) return w;
    if (U > INT32_MAX || T > INT32_MAX / 2) split = false;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return probs[a].K > probs[b].K; });
    // the range of chunks that is cut: its tiles, chunks and pieces
    int64_t R = 0, UR = 0, P = 0;
    if (split) {
        const int64_t whole = T >= 2 * slots ? (T / slots - 1) * slots : 0;
        const double share = (double)U / slots;
        int64_t seen = 0, longest = 0;
        for (int i : order) {
            const int64_t nt = tiles_of(probs[i]), c = chunks_of(probs[i]);
            longest = std::max(longest, c);
            int64_t take = std::max<int64_t>(0, std::min(nt, T - whole - seen));
            if (c > std::max(0.5 * share, (double)TILE_MIN_CHUNKS)) take = nt;
            if (take == 0) break;
            R += take;
            UR += take * c;
            seen += nt;
            if (take < nt) break;
        }
        P = std::min(slots, UR / TILE_MIN_CHUNKS);
        // not worth cutting: no tile is long enough for two pieces, or the pieces would be no
        // shorter than the longest tile by a third
        if (P <= 0 || longest < TILE_MIN_CHUNKS || (R <= slots && 3 * UR > 2 * P * longest)) R = UR = P = 0;
    }
    constexpr int64_t h = TILE_MIN_CHUNKS / 2;
    int64_t ts = 0, b = 1, left = R;       // first chunk of the tile in the range, next cut, tiles left in it
    w.seg_start.push_back(0);
    auto next_cta = [&] {
        if ((int)w.segs.size() > w.seg_start.back()) w.seg_start.push_back((int)w.segs.size());
    };
    for (int i : order) {
        const TileProblem& p = probs[i];
        const int tm = (p.M + rows - 1) / rows, tn = (p.N + rows - 1) / rows;
        const int64_t c = chunks_of(p), nt = tiles_of(p);
        for (int64_t t = 0; t < nt; t++) {
            TileSeg s;
            s.prob = i;
            s.m0 = (int)(tm <= tn ? t % tm : t / tn) * rows;
            s.n0 = (int)(tm <= tn ? t / tm : t % tn) * rows;
            auto add = [&](int64_t from, int64_t to, int slot) {
                s.kt0 = (int)from;
                s.nkt = (int)(to - from);
                s.slot = slot;
                w.segs.push_back(s);
            };
            if (left == 0) {
                next_cta();
                add(0, c, -1);
                continue;
            }
            left--;
            int64_t at = 0;
            int parts = 0;
            bool after = false;
            for (; b < P && b * UR / P < ts + c; b++) {
                const int64_t x = b * UR / P - ts;
                if (x < h) {
                    next_cta();
                } else if (c - x < h) {
                    after = true;
                } else {
                    add(at, x, w.slots + parts++);
                    at = x;
                    next_cta();
                }
            }
            add(at, c, parts ? w.slots + parts++ : -1);
            if (after) next_cta();
            if (parts) {
                w.folds.push_back({i, s.m0, s.n0, w.slots, parts});
                w.slots += parts;
            }
            ts += c;
        }
    }
    next_cta();
    return w;
}

namespace {
template <class T, bool AK, bool BKc>
void launch_tiles_t(const GemmArgs* probs, const TileSeg* segs, const int* seg_start, int nctas, const TileFold* folds,
                    int nfolds, double* ws, cudaStream_t s) {
    constexpr size_t bytes = TileSmem<T, AK, BKc>::bytes;
    set_smem_once((const void*)gemm_fp64_grouped_kernel<T, AK, BKc>, (int)bytes);
    gemm_fp64_grouped_kernel<T, AK, BKc><<<nctas, TILE_THREADS, bytes, s>>>(probs, segs, seg_start, ws);
    COUNT_LAUNCH();
    if (nfolds > 0) {
        tile_fold_kernel<T, AK, BKc><<<dim3(nfolds, T::MT), TILE_THREADS, 0, s>>>(probs, folds, ws);
        COUNT_LAUNCH();
    }
}
template <class T>
void launch_tiles(bool ak, bool bk, const GemmArgs* probs, const TileSeg* segs, const int* seg_start, int nctas,
                  const TileFold* folds, int nfolds, double* ws, cudaStream_t s) {
    if (ak) {
        if (bk) launch_tiles_t<T, true, true>(probs, segs, seg_start, nctas, folds, nfolds, ws, s);
        else launch_tiles_t<T, true, false>(probs, segs, seg_start, nctas, folds, nfolds, ws, s);
    } else {
        if (bk) launch_tiles_t<T, false, true>(probs, segs, seg_start, nctas, folds, nfolds, ws, s);
        else launch_tiles_t<T, false, false>(probs, segs, seg_start, nctas, folds, nfolds, ws, s);
    }
}
}  // namespace

int64_t tile_ws_elems(int slots, int rows) { return (int64_t)slots * rows * rows; }

void gemm_fp64_grouped(const GemmArgs* probs, const TileSeg* segs, const int* seg_start, int nctas,
                       const TileFold* folds, int nfolds, double* ws, int rows, bool a_kcontig, bool b_kcontig,
                       cudaStream_t s) {
    if (nctas <= 0) return;
    if (rows == 64) launch_tiles<Tile<64>>(a_kcontig, b_kcontig, probs, segs, seg_start, nctas, folds, nfolds, ws, s);
    else launch_tiles<Tile<32>>(a_kcontig, b_kcontig, probs, segs, seg_start, nctas, folds, nfolds, ws, s);
}

std::pair<int, int> short_shape(int M, int N) {
    if (M <= 0 || N <= 0 || M > 64 || N > 64) return {0, 0};
    auto frag = [](int x) { return x <= 8 ? 1 : (x <= 16 ? 2 : (x <= 32 ? 4 : 8)); };
    const int mt = frag(M), nt = frag(N);
    if (mt * nt > 16) return {0, 0};
    return {mt, nt};
}

int short_ctas(int K, int* kper) {
    // about 2048 k per CTA (eight warps, 16 steps of 16 k each), at most 512 CTAs
    int ctas = std::max(1, std::min(512, (K + 2047) / 2048));
    int per = (K + ctas - 1) / ctas;
    per = (per + SH_KGRAN - 1) / SH_KGRAN * SH_KGRAN;
    ctas = (K + per - 1) / per;
    *kper = per;
    return ctas;
}

void short_grouped(const ShortDesc* d, const int* cta_start, int nprob, int total_ctas, int mt, int nt,
                   cudaStream_t s) {
    if (nprob <= 0 || total_ctas <= 0) return;
    switch (mt * 16 + nt) {
        case 0x11: launch_short_t<1, 1>(d, cta_start, nprob, total_ctas, s); break;
        case 0x12: launch_short_t<1, 2>(d, cta_start, nprob, total_ctas, s); break;
        case 0x14: launch_short_t<1, 4>(d, cta_start, nprob, total_ctas, s); break;
        case 0x18: launch_short_t<1, 8>(d, cta_start, nprob, total_ctas, s); break;
        case 0x21: launch_short_t<2, 1>(d, cta_start, nprob, total_ctas, s); break;
        case 0x22: launch_short_t<2, 2>(d, cta_start, nprob, total_ctas, s); break;
        case 0x24: launch_short_t<2, 4>(d, cta_start, nprob, total_ctas, s); break;
        case 0x41: launch_short_t<4, 1>(d, cta_start, nprob, total_ctas, s); break;
        case 0x42: launch_short_t<4, 2>(d, cta_start, nprob, total_ctas, s); break;
        case 0x81: launch_short_t<8, 1>(d, cta_start, nprob, total_ctas, s); break;
        case 0x28: launch_short_t<2, 8>(d, cta_start, nprob, total_ctas, s); break;
        case 0x44: launch_short_t<4, 4>(d, cta_start, nprob, total_ctas, s); break;
        case 0x82: launch_short_t<8, 2>(d, cta_start, nprob, total_ctas, s); break;
        default: throw std::runtime_error("short product: unsupported fragment shape");
    }
    COUNT_LAUNCH();
}

void fold_groups(const FoldItem* items, int nitems, const FoldNode* nodes, const FoldTerm* terms, cudaStream_t s) {
    if (nitems <= 0) return;
    fold_groups_kernel<<<nitems, 256, 0, s>>>(items, nodes, terms);
    COUNT_LAUNCH();
}

// ---------------------------------------------------------------------------
// elementwise and reductions
// ---------------------------------------------------------------------------
namespace {

constexpr int EW_THREADS = 256;

inline int ew_blocks(int64_t n) {
    int64_t b = (n + EW_THREADS - 1) / EW_THREADS;
    if (b > 148 * 16) b = 148 * 16;
    if (b < 1) b = 1;
    return (int)b;
}

__global__ void sum_strided_kernel(const double* __restrict__ A, double* __restrict__ C, StridedArgs a,
                                   double alpha) {
    for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < a.total;
         l += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = l, oa = 0, oc = 0;
        for (int d = 0; d < a.ndim; d++) {
            int64_t x = r % a.len[d];
            r /= a.len[d];
            oa += x * a.sA[d];
            oc += x * a.sB[d];
        }
        C[oc] += alpha * A[oa];
    }
}

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    v = 0;
    if (threadIdx.x < (blockDim.x >> 5)) v = red[threadIdx.x];
    if (w == 0)
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double block_max(double v) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    v = 0;
    if (threadIdx.x < (blockDim.x >> 5)) v = red[threadIdx.x];
    if (w == 0)
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// deterministic two-pass reductions: blocks write partials, one block folds them
__global__ void dot_strided_kernel(const double* __restrict__ A, const double* __restrict__ B, StridedArgs a,
                                   double* partial) {
    double s = 0;
    for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < a.total;
         l += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = l, oa = 0, ob = 0;
        for (int d = 0; d < a.ndim; d++) {
            int64_t x = r % a.len[d];
            r /= a.len[d];
            oa += x * a.sA[d];
            ob += x * a.sB[d];
        }
        s += A[oa] * B[ob];
    }
    s = block_sum(s);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void fold_sum_kernel(const double* partial, int n, double alpha, double* out) {
    double s = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
    s = block_sum(s);
    if (threadIdx.x == 0) out[0] += alpha * s;
}

__global__ void norm_kernel(const double* __restrict__ X, int64_t n, int p, double* partial) {
    double s = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double x = X[i];
        if (p == 0) s = fmax(s, fabs(x));
        else if (p == 1) s += fabs(x);
        else s += x * x;
    }
    s = p == 0 ? block_max(s) : block_sum(s);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void fold_norm_kernel(const double* partial, int n, int p, double w, double* out) {
    double s = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s = p == 0 ? fmax(s, partial[i]) : s + partial[i];
    s = p == 0 ? block_max(s) : block_sum(s);
    if (threadIdx.x == 0) out[0] = p == 0 ? fmax(out[0], s) : out[0] + w * s;
}

__global__ void scale_kernel(double* X, int64_t n, double beta) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        X[i] = beta == 0.0 ? 0.0 : beta * X[i];
}

__global__ void fill_kernel(double* X, int64_t n, double v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        X[i] = v;
}

__global__ void axpby_kernel(const double* __restrict__ x, double* __restrict__ y, int64_t n, double a, double b) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = a * x[i] + (b == 0.0 ? 0.0 : b * y[i]);
}

// denominators of elements l[0..P) (past the end: any index below total), a position's factors
// read once for all of them
template <int P>
__device__ __forceinline__ void den_of(const WeightArgs& w, const int64_t (&l)[P], double (&den)[P]) {
#pragma unroll
    for (int q = 0; q < P; q++) den[q] = 0;
    if (w.fast) {
        uint32_t r[P];
#pragma unroll
        for (int q = 0; q < P; q++) r[q] = (uint32_t)l[q];
        for (int d = 0; d < w.ndim; d++) {
            const uint32_t mul = w.dmul[d], shr = w.dshr[d], len = (uint32_t)w.len[d];
            const double* e = w.d[d];
#pragma unroll
            for (int q = 0; q < P; q++) {
                const uint32_t t = (uint32_t)(((uint64_t)__umulhi(r[q], mul) + r[q]) >> shr);
                den[q] += __ldg(e + (r[q] - t * len));
                r[q] = t;
            }
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < P; q++) {
        int64_t r = l[q];
        for (int d = 0; d < w.ndim; d++) {
            int64_t x = r % w.len[d];
            r /= w.len[d];
            den[q] += w.d[d][x];
        }
    }
}

__global__ void weight_kernel(double* X, WeightArgs w, double shift) {
    for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < w.total;
         l += (int64_t)gridDim.x * blockDim.x) {
        double den[1];
        den_of<1>(w, {l}, den);
        X[l] = fabs(den[0] + shift) < 1e-4 ? 0.0 : X[l] / (den[0] + shift);
    }
}

__global__ void kv_write_kernel(double* X, const int64_t* keys, const double* vals, int64_t n, double a, double b) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double* p = X + keys[i];
        *p = (b == 0.0 ? 0.0 : b * *p) + a * vals[i];
    }
}

__global__ void kv_read_kernel(const double* X, const int64_t* keys, double* vals, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        vals[i] = X[keys[i]];
}

// out[j] = sum of partial[b * ny + j] over b, one CTA per j
__global__ void fold_batch_kernel(const double* partial, int nb, int ny, double* out) {
    const int j = blockIdx.x;
    double s = 0;
#pragma unroll 4
    for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b * ny + j];
    s = block_sum(s);
    if (threadIdx.x == 0) out[j] = s;
}

// sum_j c[j] xs[j][i] of two elements at a time, the vectors' loads in flight together (a
// vector with c[j] = 0 is not read).  HBM bounds it: T2 of o=20 v=144 with eight vectors (1.8 GB)
// took 310 us with one load in flight per thread and takes 265.
template <int N, class Out>
__device__ __forceinline__ void lincomb_body(int64_t n, const double* const* xs, int64_t off, const double* c, Out out) {
    __shared__ const double* sx[N];
    __shared__ double sc[N];
    if (threadIdx.x < N) {
        sx[threadIdx.x] = xs[threadIdx.x] + off;
        sc[threadIdx.x] = c[threadIdx.x];
    }
    __syncthreads();
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += 2 * step) {
        const int64_t i1 = i + step;
        const bool two = i1 < n;
        double v[2][N];
#pragma unroll
        for (int j = 0; j < N; j++) {
            const bool use = sc[j] != 0.0;
            v[0][j] = use ? __ldg(sx[j] + i) : 0.0;
            v[1][j] = use && two ? __ldg(sx[j] + i1) : 0.0;
        }
        double s0 = 0, s1 = 0;
#pragma unroll
        for (int j = 0; j < N; j++) {
            s0 += sc[j] * v[0][j];
            s1 += sc[j] * v[1][j];
        }
        out(i, s0);
        if (two) out(i1, s1);
    }
}

template <int N>
__global__ void __launch_bounds__(EW_THREADS) lincomb_kernel(double* __restrict__ out1, int64_t n1, double* __restrict__ out2,
                                                             int64_t n2, const double* const* xs, const double* c) {
    lincomb_body<N>(n1 + n2, xs, 0, c, [&](int64_t i, double v) {
        if (i < n1) out1[i] = v;
        else out2[i - n1] = v;
    });
}

// out[i] = sum_j c[j] * xs[j][off + i]
template <int N>
__global__ void __launch_bounds__(EW_THREADS) lincomb_segment_kernel(double* __restrict__ out, int64_t len,
                                                                     const double* const* xs, int64_t off,
                                                                     const double* c) {
    lincomb_body<N>(len, xs, off, c, [&](int64_t i, double v) { out[i] = v; });
}

// f(std::integral_constant<int, n>) for a ring of n vectors
template <class F>
void for_vectors(int n, F f) {
    switch (n) {
        case 1: f(std::integral_constant<int, 1>()); break;
        case 2: f(std::integral_constant<int, 2>()); break;
        case 3: f(std::integral_constant<int, 3>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 5: f(std::integral_constant<int, 5>()); break;
        case 6: f(std::integral_constant<int, 6>()); break;
        case 7: f(std::integral_constant<int, 7>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        case 9: f(std::integral_constant<int, 9>()); break;
        case 10: f(std::integral_constant<int, 10>()); break;
        case 11: f(std::integral_constant<int, 11>()); break;
        case 12: f(std::integral_constant<int, 12>()); break;
        case 13: f(std::integral_constant<int, 13>()); break;
        case 14: f(std::integral_constant<int, 14>()); break;
        case 15: f(std::integral_constant<int, 15>()); break;
        case 16: f(std::integral_constant<int, 16>()); break;
        default: throw std::runtime_error("a DIIS ring holds 1 to 16 vectors");
    }
}

// Scratch for the two-pass reductions, one buffer per stream: work on one stream is
// ordered, and each fold consumes its partials before the next reduction on that
// stream overwrites them.  Buffers live until process exit.
}  // namespace

namespace {
std::mutex g_partial_mu;
std::map<std::pair<int, cudaStream_t>, double*> g_partial;
}  // namespace

double* partial_buffer(cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(g_partial_mu);
    auto key = std::make_pair(dev, s);
    auto it = g_partial.find(key);
    if (it != g_partial.end()) return it->second;
    double* p = nullptr;
    cudaMalloc(&p, sizeof(double) * 148 * 16 * 16);
    g_partial[key] = p;
    return p;
}

namespace {

// the problem that chunk c belongs to (every thread gets it): a warp probes 32 first chunks at
// a time, so that thousands of blocks take three dependent loads instead of twelve
__device__ __forceinline__ int find_problem(const int64_t* __restrict__ cs, int n, int64_t c) {
    __shared__ int sp;
    if (threadIdx.x < 32) {
        int lo = 0, m = n;
        while (m > 1) {
            const int step = (m + 31) >> 5, i = lo + (int)threadIdx.x * step;
            const unsigned below = __ballot_sync(0xffffffffu, i < lo + m && cs[min(i, n - 1)] <= c);
            const int hit = __popc(below) - 1;
            m = min(step, m - hit * step);
            lo += hit * step;
        }
        if (threadIdx.x == 0) sp = lo;
    }
    __syncthreads();
    return sp;
}

// a descriptor into shared memory (its fields are read in every loop); sync before use
template <class D>
__device__ __forceinline__ void stage_desc(D* dst, const D* __restrict__ src) {
    static_assert(sizeof(D) % 8 == 0, "copied in 8-byte words");
    for (int i = threadIdx.x; i < (int)(sizeof(D) / 8); i += blockDim.x)
        reinterpret_cast<uint64_t*>(dst)[i] = __ldg(reinterpret_cast<const unsigned long long*>(src) + i);
}

// x / len[k] of a descriptor's position k
template <class D>
__device__ __forceinline__ int64_t div_pos(const D& d, int k, int64_t x) {
    if (d.fast) return (uint32_t)(((uint64_t)__umulhi((uint32_t)x, d.dmul[k]) + (uint32_t)x) >> d.dshr[k]);
    return x / d.len[k];
}

// Offsets of kPer elements of this thread in half h (of two) of chunk c, -1 past the end: of
// A and of the other operand (strides sX).  ROWS: a warp walks eight consecutive slots of 32
// neighbours and splits the row number only when the row changes.
constexpr int kPer = 4;
template <class D>
__device__ __forceinline__ void chunk_offsets(const D& d, const int64_t* sX, int64_t c, int h, int64_t (&oa)[kPer],
                                              int64_t (&ox)[kPer]) {
    if (d.mode == SumDesc::ROWS) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int64_t slot = c * kRowSlots + warp * (2 * kPer) + h * kPer;
        int64_t row = slot / d.spr;
        int seg = (int)(slot - row * d.spr);
        bool fresh = true;
        int64_t ra = 0, rx = 0;
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            if (fresh) {
                ra = rx = 0;
                int64_t r = row;
                for (int k = 1; k < d.ndim; k++) {
                    const int64_t t = div_pos(d, k, r), x = r - t * d.len[k];
                    ra += x * d.sA[k];
                    rx += x * sX[k];
                    r = t;
                }
                fresh = false;
            }
            const int64_t x = seg * 32 + lane;
            const bool ok = slot + q < d.units && x < d.len[0];
            oa[q] = ok ? ra + x : -1;
            ox[q] = ok ? rx + x : -1;
            if (++seg == d.spr) {
                seg = 0;
                row++;
                fresh = true;
            }
        }
        return;
    }
    const int64_t l0 = c * kBatchChunk + h * 256 * kPer + threadIdx.x;
#pragma unroll
    for (int q = 0; q < kPer; q++) oa[q] = ox[q] = l0 + q * 256 < d.total ? 0 : -1;
    if (d.fast) {
        uint32_t r[kPer];
#pragma unroll
        for (int q = 0; q < kPer; q++) r[q] = (uint32_t)(l0 + q * 256);
        for (int k = 0; k < d.ndim; k++) {
            const uint32_t mul = d.dmul[k], shr = d.dshr[k], len = (uint32_t)d.len[k];
            const int64_t sa = d.sA[k], sx = sX[k];
#pragma unroll
            for (int q = 0; q < kPer; q++) {
                const uint32_t t = (uint32_t)(((uint64_t)__umulhi(r[q], mul) + r[q]) >> shr), x = r[q] - t * len;
                if (oa[q] >= 0) {
                    oa[q] += x * sa;
                    ox[q] += x * sx;
                }
                r[q] = t;
            }
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        if (oa[q] < 0) continue;
        int64_t r = l0 + q * 256;
        for (int k = 0; k < d.ndim; k++) {
            const int64_t t = r / d.len[k], x = r - t * d.len[k];
            oa[q] += x * d.sA[k];
            ox[q] += x * sX[k];
            r = t;
        }
    }
}

// Tile t of a TILES descriptor (32 x 32 over the fastest positions p0 of A and pc of the other
// operand): its corner (past the extents where t is past the end) and the operands' offsets
template <class D>
__device__ __forceinline__ void tile_corner(const D& d, const int64_t* sX, int64_t t, int64_t& x0, int64_t& xc,
                                            int64_t& oa, int64_t& ox) {
    const int64_t l0 = d.len[d.p0], lc = d.len[d.pc];
    const int64_t t0n = (l0 + 31) / 32, tcn = (lc + 31) / 32;
    oa = ox = 0;
    x0 = l0;
    xc = lc;
    if (t >= d.units) return;
    int64_t r = t / t0n;
    x0 = (t - r * t0n) * 32;
    const int64_t u = r / tcn;
    xc = (r - u * tcn) * 32;
    r = u;
    for (int k = 0; k < d.ndim; k++) {
        if (k == d.p0 || k == d.pc) continue;
        const int64_t v = div_pos(d, k, r), x = r - v * d.len[k];
        oa += x * d.sA[k];
        ox += x * sX[k];
        r = v;
    }
}

// Permuted sums (antisymmetriser images, copies): HBM bounds them, 24 bytes per element (16
// where the sum assigns).  Copies and sums of equal layouts merge to one long row.  o=24 v=184: the
// copy of <am||ei> (117M elements) 860 us as a scaling and a sum that splits every index, 434
// as an assignment; images of the ring (39M elements) 247 -> 147.
__global__ void __launch_bounds__(256) sum_batched_kernel(const SumDesc* __restrict__ d, const int64_t* __restrict__ cs,
                                                          int n) {
    __shared__ SumDesc D;
    __shared__ double tile[2][32][33];
    const int p = find_problem(cs, n, blockIdx.x);
    stage_desc(&D, d + p);
    const int64_t c = blockIdx.x - cs[p];
    __syncthreads();
    if (D.mode == SumDesc::TILES) {
        // two 32 x 32 tiles over (p0, pc): read along p0 (A-contiguous), write along pc; the
        // reads of both tiles and of C are in flight together
        const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8 threads
        const int64_t l0 = D.len[D.p0], lc = D.len[D.pc];
        const int64_t sa0 = D.sA[D.p0], sac = D.sA[D.pc], sc0 = D.sC[D.p0], scc = D.sC[D.pc];
        double va[2][4], vc[2][4];
        int64_t oc[2], x0[2], xc[2];
#pragma unroll
        for (int tt = 0; tt < 2; tt++) {
            int64_t oa;
            tile_corner(D, D.sC, c * 2 + tt, x0[tt], xc[tt], oa, oc[tt]);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int64_t y0 = x0[tt] + tx, yc = xc[tt] + ty + 8 * q;
                va[tt][q] = y0 < l0 && yc < lc ? __ldg(D.A + oa + y0 * sa0 + yc * sac) : 0.0;
                const int64_t z0 = x0[tt] + ty + 8 * q, zc = xc[tt] + tx;
                vc[tt][q] = !D.assign && z0 < l0 && zc < lc ? D.C[oc[tt] + z0 * sc0 + zc * scc] : 0.0;
            }
        }
#pragma unroll
        for (int tt = 0; tt < 2; tt++)
#pragma unroll
            for (int q = 0; q < 4; q++) tile[tt][ty + 8 * q][tx] = va[tt][q];
        __syncthreads();
#pragma unroll
        for (int tt = 0; tt < 2; tt++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int64_t z0 = x0[tt] + ty + 8 * q, zc = xc[tt] + tx;
                if (z0 < l0 && zc < lc) D.C[oc[tt] + z0 * sc0 + zc * scc] = vc[tt][q] + D.alpha * tile[tt][tx][ty + 8 * q];
            }
        return;
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int64_t oa[kPer], oc[kPer];
        chunk_offsets(D, D.sC, c, h, oa, oc);
        double va[kPer], vc[kPer];
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            va[q] = oa[q] >= 0 ? __ldg(D.A + oa[q]) : 0.0;
            vc[q] = oa[q] >= 0 && !D.assign ? D.C[oc[q]] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kPer; q++)
            if (oa[q] >= 0) D.C[oc[q]] = vc[q] + D.alpha * va[q];
    }
}

__global__ void __launch_bounds__(256) scale_batched_kernel(const ScaleDesc* __restrict__ d,
                                                            const int64_t* __restrict__ cs, int n) {
    const int p = find_problem(cs, n, blockIdx.x);
    const ScaleDesc D = d[p];
    const int64_t base = (blockIdx.x - cs[p]) * kBatchChunk;
#pragma unroll 4
    for (int i = threadIdx.x; i < kBatchChunk; i += blockDim.x) {
        const int64_t l = base + i;
        if (l >= D.n) break;
        D.X[l] = D.beta == 0.0 ? 0.0 : D.beta * D.X[l];
    }
}

// Tau of one chunk of one block; HBM bounds it, 16 bytes per element
__global__ void __launch_bounds__(256) tau_batched_kernel(const TauArgs* __restrict__ d, const int64_t* __restrict__ cs,
                                                          int n) {
    __shared__ TauArgs a;
    const int p = find_problem(cs, n, blockIdx.x);
    stage_desc(&a, d + p);
    const int64_t base = (blockIdx.x - cs[p]) * kBatchChunk;
    __syncthreads();
    const int64_t la = a.len[0], lb = a.len[1], total = la * lb * a.len[2] * a.len[3];
    const double *ai = a.t1ai, *bj = a.t1bj, *aj = a.t1aj, *bi = a.t1bi;
    const bool fast = a.fast != 0;
    const uint32_t n0 = (uint32_t)la, n1 = (uint32_t)lb, n2 = (uint32_t)a.len[2];
    const uint32_t m0 = a.dmul[0], m1 = a.dmul[1], m2 = a.dmul[2], s0 = a.dshr[0], s1 = a.dshr[1], s2 = a.dshr[2];
    constexpr int P = kBatchChunk / 256;
    double v[P];
#pragma unroll
    for (int q = 0; q < P; q++) {
        const int64_t l = base + q * 256 + threadIdx.x;
        v[q] = l < total ? __ldg(a.t2 + l) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < P; q++) {
        const int64_t l = base + q * 256 + threadIdx.x;
        if (l >= total) continue;
        if (ai || aj) {
            int64_t x, y, i, j;
            if (fast) {
                uint32_t r = (uint32_t)l, t = (uint32_t)(((uint64_t)__umulhi(r, m0) + r) >> s0);
                x = r - t * n0;
                r = t;
                t = (uint32_t)(((uint64_t)__umulhi(r, m1) + r) >> s1);
                y = r - t * n1;
                r = t;
                t = (uint32_t)(((uint64_t)__umulhi(r, m2) + r) >> s2);
                i = r - t * n2;
                j = t;
            } else {
                x = l % la;
                y = l / la % lb;
                i = l / (la * lb) % a.len[2];
                j = l / (la * lb) / a.len[2];
            }
            if (ai) v[q] += __ldg(ai + x + la * i) * __ldg(bj + y + lb * j);
            if (aj) v[q] -= __ldg(aj + x + la * j) * __ldg(bi + y + lb * i);
        }
        a.tau[l] = v[q];
    }
}

// Jacobi update of one chunk of one block; the residual max goes to red_max through an
// atomic max on the bits of non-negative doubles (order-independent).  HBM bounds it, 32
// bytes per element.
__global__ void __launch_bounds__(256) update_batched_kernel(const UpdateDesc* __restrict__ d,
                                                             const int64_t* __restrict__ cs, int n, double* red_max) {
    __shared__ UpdateDesc D;
    const int p = find_problem(cs, n, blockIdx.x);
    stage_desc(&D, d + p);
    const int64_t base = (blockIdx.x - cs[p]) * kBatchChunk;
    __syncthreads();
    double mx = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        double z[kPer], t[kPer];
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int64_t l = base + (h * kPer + q) * 256 + threadIdx.x;
            z[q] = l < D.w.total ? D.Z[l] : 0.0;
            t[q] = l < D.w.total ? D.T[l] : 0.0;
        }
        int64_t l[kPer];
        double den[kPer];
#pragma unroll
        for (int q = 0; q < kPer; q++) l[q] = min(base + (h * kPer + q) * 256 + threadIdx.x, D.w.total - 1);
        den_of<kPer>(D.w, l, den);
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            if (base + (h * kPer + q) * 256 + threadIdx.x >= D.w.total) continue;
            const double x = fabs(den[q]) < 1e-4 ? 0.0 : z[q] / den[q];
            D.Z[l[q]] = x;
            D.T[l[q]] = t[q] + x;
            mx = fmax(mx, fabs(x));
        }
    }
    mx = block_max(mx);
    if (threadIdx.x == 0 && mx > 0.0)
        atomicMax(reinterpret_cast<unsigned long long*>(red_max), (unsigned long long)__double_as_longlong(mx));
}

// dot of one chunk of one block into part[c]; HBM bounds it, 16 bytes per element (the energy of
// o=24 v=184, 117M elements through a permuted view: 1060 us element by element, 446 by tiles)
__global__ void __launch_bounds__(256) dot_batched_kernel(const DotDesc* __restrict__ d, const int64_t* __restrict__ cs,
                                                          int n, double* part) {
    __shared__ DotDesc D;
    __shared__ double tile[2][32][33];
    const int p = find_problem(cs, n, blockIdx.x);
    stage_desc(&D, d + p);
    const int64_t c = blockIdx.x - cs[p];
    __syncthreads();
    double acc = 0;
    if (D.mode == SumDesc::TILES) {
        // as the sum's tiles: A read along p0, B along pc
        const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
        const int64_t l0 = D.len[D.p0], lc = D.len[D.pc];
        const int64_t sa0 = D.sA[D.p0], sac = D.sA[D.pc], sb0 = D.sB[D.p0], sbc = D.sB[D.pc];
        double va[2][4], vb[2][4];
#pragma unroll
        for (int tt = 0; tt < 2; tt++) {
            int64_t x0, xc, oa, ob;
            tile_corner(D, D.sB, c * 2 + tt, x0, xc, oa, ob);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int64_t y0 = x0 + tx, yc = xc + ty + 8 * q;
                va[tt][q] = y0 < l0 && yc < lc ? __ldg(D.A + oa + y0 * sa0 + yc * sac) : 0.0;
                const int64_t z0 = x0 + ty + 8 * q, zc = xc + tx;
                vb[tt][q] = z0 < l0 && zc < lc ? __ldg(D.B + ob + z0 * sb0 + zc * sbc) : 0.0;
            }
        }
#pragma unroll
        for (int tt = 0; tt < 2; tt++)
#pragma unroll
            for (int q = 0; q < 4; q++) tile[tt][ty + 8 * q][tx] = va[tt][q];
        __syncthreads();
#pragma unroll
        for (int tt = 0; tt < 2; tt++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc += vb[tt][q] * tile[tt][tx][ty + 8 * q];
    } else {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int64_t oa[kPer], ob[kPer];
        chunk_offsets(D, D.sB, c, h, oa, ob);
#pragma unroll
        for (int q = 0; q < kPer; q++)
            if (oa[q] >= 0) acc += __ldg(D.A + oa[q]) * __ldg(D.B + ob[q]);
    }
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = D.alpha * acc;
}

}  // namespace

// multiply-shift division by every extent (Granlund-Montgomery, round-up variant): for
// 1 <= len < 2^31, shr = ceil(log2 len), mul = floor(2^32 (2^shr - len) / len) + 1 gives
// x / len = (umulhi(x, mul) + x) >> shr for every x < 2^32
void plan_divisors(const int64_t* lens, int ndim, int64_t total, int& fast, uint32_t* dmul, uint32_t* dshr) {
    fast = total < ((int64_t)1 << 31) ? 1 : 0;
    for (int k = 0; k < ndim && fast; k++) {
        const uint64_t len = (uint64_t)lens[k];
        if (len < 1 || len >= ((uint64_t)1 << 31)) {
            fast = 0;
            break;
        }
        uint32_t l = 0;
        while (((uint64_t)1 << l) < len) l++;
        dshr[k] = l;
        dmul[k] = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << l) - len)) / len + 1);
    }
}

namespace {
// Positions in order of the stride sX, extents of 1 dropped, neighbours that run through both
// operands without a gap merged; ROWS where the fastest position is contiguous in both and a
// row fills half of a warp or more, TILES where the fastest positions differ and fill a
// quarter of a tile's side.
template <class D>
void plan_positions(D& d, int64_t* sX) {
    int n = 0;
    for (int k = 0; k < d.ndim; k++) {
        if (d.len[k] == 1) continue;
        const int64_t len = d.len[k], sa = d.sA[k], sx = sX[k];
        int at = n++;
        for (; at > 0 && sX[at - 1] > sx; at--) {
            d.len[at] = d.len[at - 1];
            d.sA[at] = d.sA[at - 1];
            sX[at] = sX[at - 1];
        }
        d.len[at] = len;
        d.sA[at] = sa;
        sX[at] = sx;
    }
    d.ndim = 0;
    for (int k = 0; k < n; k++) {
        const int j = d.ndim - 1;
        if (j >= 0 && d.sA[k] == d.sA[j] * d.len[j] && sX[k] == sX[j] * d.len[j]) {
            d.len[j] *= d.len[k];
            continue;
        }
        d.len[d.ndim] = d.len[k];
        d.sA[d.ndim] = d.sA[k];
        sX[d.ndim++] = sX[k];
    }
    plan_divisors(d.len, d.ndim, d.total, d.fast, d.dmul, d.dshr);
    d.mode = SumDesc::ELEMENTS;
    if (d.ndim > 0 && d.sA[0] == 1 && sX[0] == 1 && d.len[0] >= 16 && d.len[0] < ((int64_t)1 << 31)) {
        d.mode = SumDesc::ROWS;
        d.spr = (int)((d.len[0] + 31) / 32);
        d.units = d.total / d.len[0] * d.spr;
        return;
    }
    if (d.ndim < 2) return;
    int p0 = 0, pc = 0;
    for (int k = 1; k < d.ndim; k++) {
        if (d.sA[k] < d.sA[p0]) p0 = k;
        if (sX[k] < sX[pc]) pc = k;
    }
    if (p0 == pc || d.len[p0] < 8 || d.len[pc] < 8) return;
    d.mode = SumDesc::TILES;
    d.p0 = p0;
    d.pc = pc;
    d.units = ((d.len[p0] + 31) / 32) * ((d.len[pc] + 31) / 32);
    for (int k = 0; k < d.ndim; k++)
        if (k != p0 && k != pc) d.units *= d.len[k];
}
}  // namespace

void sum_plan(SumDesc& d) { plan_positions(d, d.sC); }

void dot_plan(DotDesc& d) { plan_positions(d, d.sB); }

void weight_plan(WeightArgs& w) { plan_divisors(w.len, w.ndim, w.total, w.fast, w.dmul, w.dshr); }

void tau_plan(TauArgs& a) {
    plan_divisors(a.len, 4, a.len[0] * a.len[1] * a.len[2] * a.len[3], a.fast, a.dmul, a.dshr);
}

void sum_batched(const SumDesc* d, const int64_t* chunk_start, int n, int64_t chunks, cudaStream_t s) {
    if (n <= 0 || chunks <= 0) return;
    sum_batched_kernel<<<(unsigned)chunks, 256, 0, s>>>(d, chunk_start, n);
    COUNT_LAUNCH();
}

void tau_batched(const TauArgs* d, const int64_t* chunk_start, int n, int64_t chunks, cudaStream_t s) {
    if (n <= 0 || chunks <= 0) return;
    tau_batched_kernel<<<(unsigned)chunks, 256, 0, s>>>(d, chunk_start, n);
    COUNT_LAUNCH();
}

void update_batched(const UpdateDesc* d, const int64_t* chunk_start, int n, int64_t chunks, double* red_max,
                    cudaStream_t s) {
    if (n <= 0 || chunks <= 0) return;
    update_batched_kernel<<<(unsigned)chunks, 256, 0, s>>>(d, chunk_start, n, red_max);
    COUNT_LAUNCH();
}

void dot_batched(const DotDesc* d, const int64_t* chunk_start, int n, int64_t chunks, double* part, double* out,
                 cudaStream_t s) {
    if (n <= 0 || chunks <= 0) return;
    dot_batched_kernel<<<(unsigned)chunks, 256, 0, s>>>(d, chunk_start, n, part);
    fold_sum_kernel<<<1, 1024, 0, s>>>(part, (int)chunks, 1.0, out);
    COUNT_LAUNCH();
    COUNT_LAUNCH();
}

void scale_batched(const ScaleDesc* d, const int64_t* chunk_start, int n, int64_t chunks, cudaStream_t s) {
    if (n <= 0 || chunks <= 0) return;
    scale_batched_kernel<<<(unsigned)chunks, 256, 0, s>>>(d, chunk_start, n);
    COUNT_LAUNCH();
}

void release_stream_buffers(cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(g_partial_mu);
    auto it = g_partial.find(std::make_pair(dev, s));
    if (it == g_partial.end()) return;
    cudaStreamSynchronize(s);
    cudaFree(it->second);
    g_partial.erase(it);
}

void sum_strided(const double* A, double* C, const StridedArgs& a, double alpha, cudaStream_t s) {
    if (a.total <= 0) return;
    sum_strided_kernel<<<ew_blocks(a.total), EW_THREADS, 0, s>>>(A, C, a, alpha);
    COUNT_LAUNCH();
}

void dot_strided(const double* A, const double* B, const StridedArgs& a, double alpha, double* out,
                 cudaStream_t s) {
    if (a.total <= 0) return;
    int nb = ew_blocks(a.total);
    double* part = partial_buffer(s);
    dot_strided_kernel<<<nb, EW_THREADS, 0, s>>>(A, B, a, part);
    fold_sum_kernel<<<1, 1024, 0, s>>>(part, nb, alpha, out);
    COUNT_LAUNCH();
    COUNT_LAUNCH();
}

void scale(double* X, int64_t n, double beta, cudaStream_t s) {
    if (n <= 0 || beta == 1.0) return;
    scale_kernel<<<ew_blocks(n), EW_THREADS, 0, s>>>(X, n, beta);
    COUNT_LAUNCH();
}

void fill(double* X, int64_t n, double val, cudaStream_t s) {
    if (n <= 0) return;
    fill_kernel<<<ew_blocks(n), EW_THREADS, 0, s>>>(X, n, val);
    COUNT_LAUNCH();
}

void norm_accum(const double* X, int64_t n, int p, double w, double* out, cudaStream_t s) {
    if (n <= 0) return;
    int nb = ew_blocks(n);
    double* part = partial_buffer(s);
    norm_kernel<<<nb, EW_THREADS, 0, s>>>(X, n, p, part);
    fold_norm_kernel<<<1, 1024, 0, s>>>(part, nb, p, w, out);
    COUNT_LAUNCH();
    COUNT_LAUNCH();
}

void axpby(const double* x, double* out, int64_t n, double alpha, double beta, cudaStream_t s) {
    if (n <= 0) return;
    axpby_kernel<<<ew_blocks(n), EW_THREADS, 0, s>>>(x, out, n, alpha, beta);
    COUNT_LAUNCH();
}

void weight_block(double* X, const WeightArgs& w, double shift, cudaStream_t s) {
    if (w.total <= 0) return;
    weight_kernel<<<ew_blocks(w.total), EW_THREADS, 0, s>>>(X, w, shift);
    COUNT_LAUNCH();
}

void kv_write(double* X, const int64_t* keys, const double* vals, int64_t n, double alpha, double beta,
              cudaStream_t s) {
    if (n <= 0) return;
    kv_write_kernel<<<ew_blocks(n), EW_THREADS, 0, s>>>(X, keys, vals, n, alpha, beta);
    COUNT_LAUNCH();
}

void kv_read(const double* X, const int64_t* keys, double* vals, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    kv_read_kernel<<<ew_blocks(n), EW_THREADS, 0, s>>>(X, keys, vals, n);
    COUNT_LAUNCH();
}

void lincomb(double* out1, int64_t n1, double* out2, int64_t n2, const double* const* xs, const double* c, int nx,
             cudaStream_t s) {
    if (n1 + n2 <= 0) return;
    for_vectors(nx, [&](auto N) {
        lincomb_kernel<decltype(N)::value><<<ew_blocks((n1 + n2 + 1) / 2), EW_THREADS, 0, s>>>(out1, n1, out2, n2, xs, c);
    });
    COUNT_LAUNCH();
}


// ---------------------------------------------------------------------------
// device-resident DIIS
// ---------------------------------------------------------------------------
namespace {

__global__ void diis_advance_kernel(int* st, int order) {
    st[0] = (st[0] + 1) % order;
    st[1] = min(st[1] + 1, order);
}

__global__ void diis_store_kernel(const int* st, const double* const* xs, const double* const* dxs,
                                  const double* __restrict__ t1, int64_t n1, const double* __restrict__ t2, int64_t n2,
                                  const double* __restrict__ z1, const double* __restrict__ z2) {
    const int h = st[0];
    double* x = const_cast<double*>(xs[h]);
    double* dx = const_cast<double*>(dxs[h]);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n1 + n2; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < n1) {
            x[i] = t1[i];
            dx[i] = z1[i];
        } else {
            x[i] = t2[i - n1];
            dx[i] = z2[i - n1];
        }
    }
}

// <dxs[head], dxs[j]> of every vector over all weighted segments, a partial per CTA.  HBM
// bounds it (each vector once); two elements of every vector are in flight per thread.
template <int N>
__global__ void __launch_bounds__(EW_THREADS) diis_dots_kernel(const int* st, const double* const* dxs,
                                                               const DiisSegment* __restrict__ segs, int nsegs,
                                                               double* partial) {
    __shared__ const double* sx[N];
    __shared__ const double* shead;
    if (threadIdx.x < N) sx[threadIdx.x] = dxs[threadIdx.x];
    if (threadIdx.x == 0) shead = dxs[st[0]];
    __syncthreads();
    double s[N];
#pragma unroll
    for (int j = 0; j < N; j++) s[j] = 0;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int q = 0; q < nsegs; q++) {
        const DiisSegment g = segs[q];
        const int64_t end = g.off + g.len;
        for (int64_t i = g.off + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < end; i += 2 * step) {
            const int64_t i1 = i + step;
            const bool two = i1 < end;
            double v[2][N];
            const double x0 = g.w * __ldg(shead + i), x1 = two ? g.w * __ldg(shead + i1) : 0.0;
#pragma unroll
            for (int j = 0; j < N; j++) {
                v[0][j] = __ldg(sx[j] + i);
                v[1][j] = two ? __ldg(sx[j] + i1) : 0.0;
            }
#pragma unroll
            for (int j = 0; j < N; j++) s[j] += x0 * v[0][j] + x1 * v[1][j];
        }
    }
#pragma unroll
    for (int j = 0; j < N; j++) {
        const double t = block_sum(s[j]);
        if (threadIdx.x == 0) partial[blockIdx.x * N + j] = t;
    }
}

// Gaussian elimination with partial pivoting on an m x m system (m <= 17); false if a
// pivot is exactly zero
__device__ bool small_solve(double (*A)[17], double* b, int m) {
    for (int k = 0; k < m; k++) {
        int p = k;
        for (int i = k + 1; i < m; i++)
            if (fabs(A[i][k]) > fabs(A[p][k])) p = i;
        if (A[p][k] == 0.0) return false;
        if (p != k) {
            for (int j = 0; j < m; j++) {
                double t = A[k][j];
                A[k][j] = A[p][j];
                A[p][j] = t;
            }
            double t = b[k];
            b[k] = b[p];
            b[p] = t;
        }
        for (int i = k + 1; i < m; i++) {
            double f = A[i][k] / A[k][k];
            for (int j = k; j < m; j++) A[i][j] -= f * A[k][j];
            b[i] -= f * b[k];
        }
    }
    for (int k = m - 1; k >= 0; k--) {
        double t = b[k];
        for (int j = k + 1; j < m; j++) t -= A[k][j] * b[j];
        b[k] = t / A[k][k];
    }
    return true;
}

__global__ void diis_solve_kernel(int* st, double* e, double* c, const double* dots, int order) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int ld = order + 1;
    const int head = st[0], cnt = st[1];
    for (int j = 0; j < order; j++) {
        e[head * ld + j] = dots[j];
        e[j * ld + head] = dots[j];
    }
    for (int j = 0; j <= order; j++) c[j] = 0.0;
    // diis.hpp:151: a single vector gives no extrapolation
    if (cnt == 1) {
        c[head] = 1.0;
        return;
    }
    // diis.hpp:153: --start > 1 delays the extrapolation
    int start = --st[2];
    if (start > 1) {
        c[head] = 1.0;
        return;
    }
    double A[17][17], b[17];
    auto slot = [&](int age) { return ((head - age) % order + order) % order; };
    auto fill = [&](double shift) {
        for (int i = 0; i < cnt; i++) {
            for (int j = 0; j < cnt; j++) A[i][j] = e[slot(i) * ld + slot(j)];
            A[i][i] += shift;
            A[i][cnt] = -1.0;
            A[cnt][i] = -1.0;
            b[i] = 0.0;
        }
        A[cnt][cnt] = 0.0;
        b[cnt] = -1.0;
    };
    fill(0.0);
    bool ok = small_solve(A, b, cnt + 1);
    if (!ok) {
        // diis.hpp:177-185: shift the diagonal by eps * e[n-1][n-1] and retry
        double eps = e[slot(cnt - 1) * ld + slot(cnt - 1)] * 2.220446049250313e-16;
        fill(eps);
        ok = small_solve(A, b, cnt + 1);
    }
    if (!ok) {
        st[3] = 1;
        c[head] = 1.0;
        return;
    }
    for (int i = 0; i < cnt; i++) c[slot(i)] = b[i];
}

// one piece of a caller's (x, dx) pair into the head slot at offset `off`
__global__ void diis_store_segment_kernel(const int* st, const double* const* xs, const double* const* dxs,
                                          int64_t off, const double* __restrict__ x, const double* __restrict__ dx,
                                          int64_t len) {
    const int h = st[0];
    double* rx = const_cast<double*>(xs[h]) + off;
    double* rdx = const_cast<double*>(dxs[h]) + off;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x) {
        rx[i] = x[i];
        rdx[i] = dx[i];
    }
}

// diis.hpp:155-161: while the start counter is above 1 (and two vectors are stored), the
// stored newest x becomes (damping - 1) x_0 + damping x_1
__global__ void diis_damp_kernel(const int* st, const double* const* xs, int order, int64_t len, double damping) {
    if (st[1] < 2 || st[2] <= 1) return;
    const int h = st[0], p = (st[0] - 1 + order) % order;
    double* x0 = const_cast<double*>(xs[h]);
    const double* x1 = xs[p];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x)
        x0[i] = (damping - 1.0) * x0[i] + damping * x1[i];
}

}  // namespace

namespace {

__device__ __forceinline__ void tri_decode(int64_t p, int64_t& x, int64_t& y) {
    // p = y(y-1)/2 + x with 0 <= x < y
    int64_t yy = (int64_t)((1.0 + sqrt(1.0 + 8.0 * (double)p)) * 0.5);
    while (yy * (yy - 1) / 2 > p) yy--;
    while ((yy + 1) * yy / 2 <= p) yy++;
    y = yy;
    x = p - yy * (yy - 1) / 2;
}

__global__ void pack_vvvv_kernel(double* V, int kab, int kcd, int n0, int n1, int n2, int n3, int64_t scd,
                                 const double* __restrict__ tJ, const double* __restrict__ tK, int a0, int a1,
                                 bool J, bool K) {
    const int ca = a1 - a0;
    const int64_t ncd = kcd == 1 ? (int64_t)n2 * (n2 - 1) / 2 : (int64_t)n2 * n3;
    const int64_t total = (int64_t)ca * n1 * ncd;
    for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < total; l += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = l;
        int a = (int)(r % ca) + a0;
        r /= ca;
        int b = (int)(r % n1);
        int64_t pcd = r / n1;
        if (kab == 1 && b <= a) continue;
        int64_t c, d;
        if (kcd == 1) tri_decode(pcd, c, d);
        else {
            c = pcd % n2;
            d = pcd / n2;
        }
        int64_t pab = kab == 1 ? (int64_t)b * (b - 1) / 2 + a : (int64_t)a + (int64_t)n0 * b;
        const int64_t ap = a - a0;
        double v = 0;
        if (J) v += tJ[ap + ca * (c + (int64_t)n2 * (b + (int64_t)n1 * d))];
        if (K) v -= tK[ap + ca * (d + (int64_t)n3 * (b + (int64_t)n1 * c))];
        V[pab + scd * pcd] = v;
    }
}

}  // namespace

namespace {
// 32 x 32 tiles of one matrix per blockIdx.z, 32 x 8 threads
__global__ void transpose_factor_kernel(const double* __restrict__ in, double* __restrict__ out, int n) {
    __shared__ double tile[32][33];
    const int64_t base = (int64_t)blockIdx.z * n * n;
    int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 32 + threadIdx.y;
    for (int j = 0; j < 32; j += 8)
        if (x < n && y + j < n) tile[threadIdx.y + j][threadIdx.x] = in[base + (int64_t)(y + j) * n + x];
    __syncthreads();
    x = blockIdx.y * 32 + threadIdx.x;
    y = blockIdx.x * 32 + threadIdx.y;
    for (int j = 0; j < 32; j += 8)
        if (x < n && y + j < n) out[base + (int64_t)(y + j) * n + x] = tile[threadIdx.x][threadIdx.y + j];
}
__global__ void eri_gather_kernel(EriGatherArgs a, const double* __restrict__ eri) {
    const int64_t total = (int64_t)a.len[0] * a.len[1] * a.len[2] * a.len[3];
    for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < total; l += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = l, dst = a.off;
        int64_t g[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int x = (int)(r % a.len[p]);
            r /= a.len[p];
            dst += a.st[p] * x;
            g[p] = a.g[p][x];
        }
        const int64_t src = ((g[a.pos[0]] * a.n + g[a.pos[1]]) * a.n + g[a.pos[2]]) * a.n + g[a.pos[3]];
        a.C[dst] += a.sign * eri[src];
    }
}

}  // namespace

void transpose_factor(const double* in, double* out, int naux, int n, cudaStream_t s) {
    const int t = (n + 31) / 32;
    for (int p = 0; p < naux; p += 65535) {
        const int64_t off = (int64_t)p * n * n;
        transpose_factor_kernel<<<dim3(t, t, std::min(naux - p, 65535)), dim3(32, 8), 0, s>>>(in + off, out + off, n);
        COUNT_LAUNCH();
    }
}

void eri_gather(const EriGatherArgs& a, const double* eri, cudaStream_t s) {
    const int64_t n = (int64_t)a.len[0] * a.len[1] * a.len[2] * a.len[3];
    if (n <= 0) return;
    eri_gather_kernel<<<ew_blocks(n), EW_THREADS, 0, s>>>(a, eri);
    COUNT_LAUNCH();
}

namespace {
__global__ void closed_shell_jk_kernel(const double* __restrict__ eri, int n, int nocc, double* __restrict__ F) {
    const int64_t pq = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (pq >= (int64_t)n * n) return;
    const int64_t p = pq / n, q = pq % n, n2 = (int64_t)n * n, n3 = n2 * n;
    double v = 0;
    for (int i = 0; i < nocc; i++) v += 2.0 * eri[p * n3 + q * n2 + (int64_t)i * n + i] - eri[p * n3 + (int64_t)i * n2 + (int64_t)i * n + q];
    F[pq] = v;
}
}  // namespace

void closed_shell_jk(const double* eri, int n, int nocc, double* F, cudaStream_t s) {
    const int64_t nn = (int64_t)n * n;
    if (nn <= 0) return;
    closed_shell_jk_kernel<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(eri, n, nocc, F);
    COUNT_LAUNCH();
}

void pack_vvvv(double* V, int kind_ab, int kind_cd, int n0, int n1, int n2, int n3, int64_t scd, const double* tJ,
               const double* tK, int a0, int a1, bool J, bool K, cudaStream_t s) {
    int64_t ncd = kind_cd == 1 ? (int64_t)n2 * (n2 - 1) / 2 : (int64_t)n2 * n3;
    int64_t total = (int64_t)(a1 - a0) * n1 * ncd;
    if (total <= 0) return;
    pack_vvvv_kernel<<<ew_blocks(total), EW_THREADS, 0, s>>>(V, kind_ab, kind_cd, n0, n1, n2, n3, scd, tJ, tK, a0,
                                                              a1, J, K);
    COUNT_LAUNCH();
}

void diis_advance(int* state, int order, cudaStream_t s) {
    diis_advance_kernel<<<1, 1, 0, s>>>(state, order);
    COUNT_LAUNCH();
}

void diis_store(const int* state, const double* const* xs, const double* const* dxs, const double* t1, int64_t n1,
                const double* t2, int64_t n2, const double* z1, const double* z2, cudaStream_t s) {
    diis_store_kernel<<<ew_blocks(n1 + n2), EW_THREADS, 0, s>>>(state, xs, dxs, t1, n1, t2, n2, z1, z2);
    COUNT_LAUNCH();
}

void diis_dots(const int* state, const double* const* dxs, int order, const DiisSegment* segs, int nsegs, int64_t total,
               double* dots, cudaStream_t s) {
    const int nb = std::min(ew_blocks((total + 1) / 2), 148 * 8);
    double* part = partial_buffer(s);
    for_vectors(order, [&](auto N) {
        diis_dots_kernel<decltype(N)::value><<<nb, EW_THREADS, 0, s>>>(state, dxs, segs, nsegs, part);
    });
    fold_batch_kernel<<<order, 256, 0, s>>>(part, nb, order, dots);
    COUNT_LAUNCH();
    COUNT_LAUNCH();
}

void diis_solve(int* state, double* e, double* c, const double* dots, int order, cudaStream_t s) {
    diis_solve_kernel<<<1, 32, 0, s>>>(state, e, c, dots, order);
    COUNT_LAUNCH();
}

void diis_store_segment(const int* state, const double* const* xs, const double* const* dxs, int64_t off,
                        const double* x, const double* dx, int64_t len, cudaStream_t s) {
    if (len <= 0) return;
    diis_store_segment_kernel<<<ew_blocks(len), EW_THREADS, 0, s>>>(state, xs, dxs, off, x, dx, len);
    COUNT_LAUNCH();
}

void lincomb_segment(double* out, int64_t len, const double* const* xs, int64_t off, const double* c, int nx,
                     cudaStream_t s) {
    if (len <= 0) return;
    for_vectors(nx, [&](auto N) {
        lincomb_segment_kernel<decltype(N)::value><<<ew_blocks((len + 1) / 2), EW_THREADS, 0, s>>>(out, len, xs, off, c);
    });
    COUNT_LAUNCH();
}

void diis_damp(const int* state, const double* const* xs, int order, int64_t len, double damping, cudaStream_t s) {
    if (len <= 0 || damping <= 0.0) return;
    diis_damp_kernel<<<ew_blocks(len), EW_THREADS, 0, s>>>(state, xs, order, len, damping);
    COUNT_LAUNCH();
}

}  // namespace kern
}  // namespace ccsd
