// resident.cu -- the whole Jacobi-PCG solve (krylov::cg_jacobi, include/femd/krylov/cg.hpp:296-350)
// in one launch, the matrix held in shared memory.
//
// A system whose matrix fits the SMs' shared memory (about 30 MB) is read from HBM once; an
// iteration then moves only the exchanged direction through L2, and what bounds it is latency:
// the two sums over the grid and the gather of the direction.  The three kernels an iteration of
// the streaming loop (krylov.cu) takes cost 14-18 us at these sizes, whatever the size.
//
// Layout.  Every block owns a contiguous range of rows of equal weight (10 B an entry + 40 B a
// row, about what a row takes here), one lane a row, or 2 to 8 where that leaves lanes idle.  Its
// shared memory holds the rows' entries in slices of one warp's rows, an entry of every lane side
// by side (32 consecutive values a load: over plain rows, a row length of 16 put all lanes on one
// bank and an SpMV of 10,000 entries took 13,600 cycles): the value and the 16-bit place of its column in the
// block's own list of the distinct columns it reads (the halo); the direction p at those places;
// and nothing else: r, x, D^-1 and z of a row live in registers of the row's first lane.  The list
// is made at the start of the solve from a bitmap of the columns (its ranks are the places, so the
// list is sorted and its gathers run along memory).
//
// One iteration has two sums over the grid.  p is never exchanged: every block forms
// p = z + beta p at its halo's places from the exchanged z (the same fused multiply-add of the
// same numbers everywhere), so the owner publishes z before the sum of r.z and nothing else waits.
//
// Sums.  A block's sum is a fixed tree; the blocks' sums are added in one fixed tree by every
// block, so all blocks take the same decisions and the bits depend on the system and the launch
// shape alone.
//   grid     every block stores its sum, adds one to a counter (release), waits for the counter to
//            reach the sum's number times the blocks (a bounded wait: past it the solve ends with
//            FEMD_ETIMEOUT) and reads all the sums.  1.9 us at 148 blocks; measured beside it: a
//            16-byte {sum, number} slot per block polled by every block 4.3 us (148 x 148 polls of
//            the same lines), the slots pushed into every block's own set 2.0-2.3 us, clusters
//            with one block each in the grid's sum 2.7-4.1 us.
//   cluster  up to 16 blocks of one cluster write their sums into each other's shared memory and
//            meet at the cluster's barrier; z is read from its owner's shared memory.
#include <algorithm>

#include "resident.h"

namespace femd {

static constexpr int RES_THREADS = 512, RES_WARPS = RES_THREADS / 32;
static_assert(RES_WARPS == 16, "a half-warp holds a value per warp, or per block of a cluster");
static constexpr int RES_SLOTS = 4;                   // rows a lane group holds in registers
static constexpr int RES_MAX_CLUSTER = 16;           // a half-warp
static constexpr long long RES_SPINS = 1ll << 24;     // polls of the counter (some 0.5 us each) before giving up
static constexpr int RES_ROW_WEIGHT = 40, RES_NNZ_WEIGHT = 10;

struct ResArgs {
    const int *indptr, *indices;
    const double *data, *inv, *b;
    double *x;
    double *zx;                 // grid: the exchanged vector
    double *part;               // grid: the blocks' sums, [set][value][block]
    unsigned long long *count;  // grid: blocks that have stored a sum, counted from the launch
    ResidentOut *out;
    double tol;
    int n, max_iter, smem;
};

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned map_to_cta(unsigned addr, int cta)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}

__device__ __forceinline__ void cluster_store(unsigned addr, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(addr), "d"(v) : "memory");
}

__device__ __forceinline__ double cluster_load(unsigned addr)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));   // ordered by the barriers (volatile)
    return v;
}

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the sum over a half-warp, in every lane of it
__device__ __forceinline__ double half_sum(double v)
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The first row i with weight(rows before i) >= goal, by one warp (32-way search).
__device__ __forceinline__ int weight_bound(const int *indptr, int n, long long goal)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;                               // the answer lies in [lo, hi]
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32;
        const int i = lo + lane * step;               // probes lo, lo + step, ...: true from some lane on
        const bool ge = i >= hi || (long long)RES_NNZ_WEIGHT * indptr[i] + (long long)RES_ROW_WEIGHT * i >= goal;
        const unsigned m = __ballot_sync(0xffffffffu, ge);
        const int f = m ? __ffs(m) - 1 : 32;          // the first true probe
        const int top = f < 32 ? min(lo + f * step, hi) : hi;
        if (f == 0) return lo;
        lo = lo + (f - 1) * step + 1;                 // the last false probe + 1
        hi = top;
    }
    return lo;
}

template <bool CL>
__global__ void __launch_bounds__(RES_THREADS, 1) k_cg_resident(const ResArgs A)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double s_red[2][3][RES_WARPS];
    __shared__ double s_tot[2][3][RES_MAX_BLOCKS / 32];
    __shared__ double s_cl[2][3][RES_MAX_CLUSTER];
    __shared__ int s_bound[RES_MAX_CLUSTER + 1];
    __shared__ int s_scan[RES_WARPS], s_slice[RES_SLOTS * RES_WARPS];
    __shared__ int s_fail;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int G = gridDim.x, me = blockIdx.x, n = A.n;
    unsigned long long number = 0;                    // of the next sum over the grid

    // The sums of v over the grid, in every thread; false when a wait ran out.
    auto grid_sum = [&](auto &v) -> bool {
        constexpr int NV = sizeof(v) / sizeof(double);
        ++number;
        const int set = (int)(number & 1);
        if (NV == 2) {
            // both values in five exchanges: the half-warps take one value each
            const bool up = lane >= 16;
            double t = up ? v[NV - 1] : v[0];
            t += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[NV - 1], 16);
            t = half_sum(t);
            if ((lane & 15) == 0) s_red[set][up][w] = t;
        } else {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const double t = warp_sum(v[k]);
                if (lane == 0) s_red[set][k][w] = t;
            }
        }
        __syncthreads();
        if (CL) {
            if (tid < NV * RES_MAX_CLUSTER && tid % RES_MAX_CLUSTER < G) {
                const int k = tid / RES_MAX_CLUSTER, to = tid % RES_MAX_CLUSTER;
                double t[RES_WARPS];
#pragma unroll
                for (int i = 0; i < RES_WARPS; ++i) t[i] = s_red[set][k][i];
#pragma unroll
                for (int o = RES_WARPS / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < o; ++i) t[i] += t[i + o];
                cluster_store(map_to_cta(smem_addr(&s_cl[set][k][me]), to), t[0]);
            }
            cluster_barrier();
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                v[k] = half_sum((lane & 15) < G ? s_cl[set][k][lane & 15] : 0.0);
            }
            return true;
        }
        double *const part = A.part + (size_t)set * 3 * RES_MAX_BLOCKS;
        if (w == 0) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const double t = half_sum(s_red[set][k][lane & 15]);
                if (lane == 0) __stcg(part + k * RES_MAX_BLOCKS + me, t);
            }
            if (lane == 0) {
                // release: the sums above and what the block published before the barrier above
                asm volatile("red.release.gpu.global.add.u64 [%0], %1;" :: "l"(A.count), "l"(1ull) : "memory");
                unsigned long long c;
                for (long long spin = 0;; ++spin) {
                    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(A.count) : "memory");
                    if (c >= number * (unsigned long long)G) break;
                    if (spin > RES_SPINS) { s_fail = 1; break; }
                }
            }
        }
        __syncthreads();
        if (tid < (G + 31) / 32 * 32) {
            double t[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) t[k] = tid < G ? __ldcg(part + k * RES_MAX_BLOCKS + tid) : 0.0;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                t[k] = warp_sum(t[k]);
                if (lane == 0) s_tot[set][k][w] = t[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double t = 0.0;
#pragma unroll
            for (int i = 0; i < RES_MAX_BLOCKS / 32; ++i) t += i < (G + 31) / 32 ? s_tot[set][k][i] : 0.0;
            v[k] = t;
        }
        return s_fail == 0;
    };

    // ---- this block's rows -------------------------------------------------------------------
    if (tid == 0) s_fail = 0;
    const long long weight = (long long)RES_NNZ_WEIGHT * A.indptr[n] + (long long)RES_ROW_WEIGHT * n;
    if (CL) {
        for (int t = w; t <= G; t += RES_WARPS) {
            const int i = t == 0 ? 0 : t == G ? n : weight_bound(A.indptr, n, weight * t / G);
            if (lane == 0) s_bound[t] = i;
        }
    } else if (w < 2) {
        const int t = me + w, i = t == 0 ? 0 : t == G ? n : weight_bound(A.indptr, n, weight * t / G);
        if (lane == 0) s_bound[w] = i;
    }
    __syncthreads();
    const int r0 = CL ? s_bound[me] : s_bound[0], rows = (CL ? s_bound[me + 1] : s_bound[1]) - r0;
    const int q0 = A.indptr[r0], nz = A.indptr[r0 + rows] - q0;
    const int words = (n + 31) >> 5;
    auto up16 = [](size_t v) { return (v + 15) & ~(size_t)15; };
    // TPR lanes a row: row s NG + grp (s < RES_SLOTS) is lane group grp's row s
    int sh = 0;
    while (sh < 3 && (rows << (sh + 1)) <= RES_THREADS) ++sh;
    const int TPR = 1 << sh, NG = RES_THREADS >> sh, grp = tid >> sh, sub = tid & (TPR - 1);
    bool fits = rows <= RES_SLOTS * NG;
    int len[RES_SLOTS], at[RES_SLOTS], src[RES_SLOTS];   // this lane's entries of row s, where they lie here and in the CSR
    if (fits) {
#pragma unroll
        for (int s = 0; s < RES_SLOTS; ++s) {
            const int lr = grp + s * NG;
            len[s] = src[s] = 0;
            if (lr < rows) {
                src[s] = A.indptr[r0 + lr] + sub;
                len[s] = max(0, (A.indptr[r0 + lr + 1] - src[s] + TPR - 1) >> sh);
            }
            const int width = __reduce_max_sync(0xffffffffu, len[s]);
            if (lane == 0) s_slice[s * RES_WARPS + w] = width;
        }
    }
    __syncthreads();
    int slots = 0;                                    // entries here, a slice's shorter rows filled up
    if (fits)
#pragma unroll
        for (int s = 0; s < RES_SLOTS; ++s)
            for (int i = 0; i < RES_WARPS; ++i) {
                if (i == w) at[s] = slots + lane;
                slots += 32 * s_slice[s * RES_WARPS + i];
            }
    // (cluster: zbuf), idx, hl, p, values; the bitmap and its ranks at the end, dead before p is written
    size_t off = CL ? up16((size_t)RES_SLOTS * RES_THREADS * sizeof(double)) : 0;
    double *const zbuf = reinterpret_cast<double *>(dyn);     // cluster: z of the own rows, the same place in every block
    unsigned short *const idx = reinterpret_cast<unsigned short *>(dyn + off);
    off = up16(off + (size_t)slots * sizeof(unsigned short));
    unsigned *const hl = reinterpret_cast<unsigned *>(dyn + off);
    const size_t tmp = ((size_t)A.smem - 2 * (size_t)words * sizeof(int)) & ~(size_t)15;
    unsigned *const bits = reinterpret_cast<unsigned *>(dyn + tmp);
    int *const rank = reinterpret_cast<int *>(dyn + tmp + (size_t)words * sizeof(int));
    fits = fits && 2 * (size_t)words * sizeof(int) + 16 <= (size_t)A.smem && off <= tmp;

    // ---- the halo: distinct columns in increasing order, every entry's place -----------------
    int H = 0;
    if (fits) {
        for (int i = tid; i < words; i += RES_THREADS) bits[i] = 0;
        __syncthreads();
        for (int i = tid; i < rows; i += RES_THREADS) atomicOr(&bits[(r0 + i) >> 5], 1u << ((r0 + i) & 31));
        for (int q = tid; q < nz; q += RES_THREADS) {
            const int c = A.indices[q0 + q];
            const unsigned bit = 1u << (c & 31);
            if (!(bits[c >> 5] & bit)) atomicOr(&bits[c >> 5], bit);
        }
        __syncthreads();
        // ranks: each thread a run of words
        const int per = (words + RES_THREADS - 1) / RES_THREADS, i0 = min(tid * per, words), i1 = min(i0 + per, words);
        int cnt = 0;
        for (int i = i0; i < i1; ++i) cnt += __popc(bits[i]);
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_scan[w] = inc;
        __syncthreads();
        int before = inc - cnt;
        for (int i = 0; i < RES_WARPS; ++i) {
            if (i < w) before += s_scan[i];
            H += s_scan[i];
        }
        const size_t o_p = up16(off + (size_t)H * sizeof(unsigned));
        fits = H <= 65536 && o_p <= tmp && o_p + ((size_t)H + slots) * sizeof(double) <= (size_t)A.smem;
        if (fits) {
            for (int i = i0; i < i1; ++i) {
                rank[i] = before;
                unsigned m = bits[i];
                while (m) {
                    hl[before++] = (unsigned)(i * 32 + __ffs(m) - 1);
                    m &= m - 1;
                }
            }
            __syncthreads();
#pragma unroll
            for (int s = 0; s < RES_SLOTS; ++s)
                for (int j = 0; j < len[s]; ++j) {
                    const int c = A.indices[src[s] + (j << sh)];
                    idx[at[s] + 32 * j] = (unsigned short)(rank[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1u)));
                }
        }
    }
    const bool first = sub == 0;
    double r[RES_SLOTS], x[RES_SLOTS], iv[RES_SLOTS], q[RES_SLOTS];
    int own[RES_SLOTS];                               // the row's place in the halo
#pragma unroll
    for (int s = 0; s < RES_SLOTS; ++s) {
        const int lr = grp + s * NG, i = r0 + lr;
        r[s] = x[s] = iv[s] = q[s] = 0.0;
        own[s] = -1;
        if (fits && first && lr < rows) {
            own[s] = rank[i >> 5] + __popc(bits[i >> 5] & ((1u << (i & 31)) - 1u));
            iv[s] = A.inv ? A.inv[i] : 1.0;
        }
    }
    {
        double v[1] = {fits ? 0.0 : 1.0};
        const bool ok = grid_sum(v);
        if (!ok || v[0] != 0.0) {
            if (me == 0 && tid == 0) { A.out->unfit = ok; A.out->timeout = !ok; }
            return;
        }
    }
    const size_t o_p = up16(off + (size_t)H * sizeof(unsigned));
    double *const p = reinterpret_cast<double *>(dyn + o_p);
    double *const vals = p + H;
#pragma unroll
    for (int s = 0; s < RES_SLOTS; ++s)
        for (int j = 0; j < len[s]; ++j) vals[at[s] + 32 * j] = A.data[src[s] + (j << sh)];

    // y = A p on the block's rows; every lane of a group holds its rows' sums
    auto spmv = [&]() {
#pragma unroll
        for (int s = 0; s < RES_SLOTS; ++s) {
            if (s * NG >= rows) break;
            double acc = 0.0;
            const double *const vs = vals + at[s];
            const unsigned short *const is = idx + at[s];
#pragma unroll 4
            for (int j = 0; j < len[s]; ++j) acc = fma(vs[32 * j], p[is[32 * j]], acc);
            for (int o = TPR >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            q[s] = acc;
        }
    };
    // publish a value of an own row / read the halo's places of the published vector
    auto publish = [&](int s, double v) {
        const int lr = grp + s * NG;
        if (CL) zbuf[lr] = v;
        else A.zx[r0 + lr] = v;
    };
    // p = beta p + the published vector at the halo's places; a round's loads are issued before its stores
    constexpr int GU = 8;
    auto gather = [&](double scale) {
        for (int u0 = tid; u0 < H; u0 += GU * RES_THREADS) {
            double t[GU];
#pragma unroll
            for (int g = 0; g < GU; ++g) {
                const int u = u0 + g * RES_THREADS;
                t[g] = 0.0;
                if (u < H) t[g] = CL ? cluster_load(hl[u]) : __ldcg(A.zx + hl[u]);
            }
#pragma unroll
            for (int g = 0; g < GU; ++g) {
                const int u = u0 + g * RES_THREADS;
                if (u < H) p[u] = fma(scale, p[u], t[g]);
            }
        }
        __syncthreads();
    };

    // ---- start: r = b - A x, z = D^-1 r (cg.hpp:305-324) --------------------------------------
    for (int u = tid; u < H; u += RES_THREADS) {
        const int c = (int)hl[u];
        p[u] = A.x[c];
        if (CL) {                                     // from now on: the place of the column's z in its owner
            int o = 0;
            while (c >= s_bound[o + 1]) ++o;
            hl[u] = map_to_cta(smem_addr(zbuf + (c - s_bound[o])), o);
        }
    }
    __syncthreads();
    spmv();
    double v3[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int s = 0; s < RES_SLOTS; ++s)
        if (own[s] >= 0) {
            const double bi = A.b[r0 + grp + s * NG];
            x[s] = p[own[s]];
            r[s] = bi - q[s];
            const double z = iv[s] * r[s];
            publish(s, z);
            v3[0] += bi * bi;
            v3[1] += r[s] * r[s];
            v3[2] += r[s] * z;
        }
    bool ok = grid_sum(v3);
    const double nb = sqrt(v3[0]), tol_nb = A.tol * nb;
    double rn = sqrt(v3[1]), rz = v3[2], beta = 0.0;
    int it = 0, breakdown = 0;
    bool done = !ok || nb == 0.0 || rn <= tol_nb;
    if (!done && !(rz > 0.0)) { breakdown = 1; done = true; }
    for (int u = tid; u < H; u += RES_THREADS) p[u] = 0.0;

    // ---- the loop (cg.hpp:323-346) ------------------------------------------------------------
    while (!done) {
        gather(beta);
        spmv();
        double v1[1] = {0.0};
#pragma unroll
        for (int s = 0; s < RES_SLOTS; ++s)
            if (own[s] >= 0) v1[0] += p[own[s]] * q[s];
        ok = grid_sum(v1);
        if (!ok) break;
        if (!(v1[0] > 0.0)) { breakdown = 1; break; }
        const double alpha = rz / v1[0];
        double v2[2] = {0.0, 0.0};
#pragma unroll
        for (int s = 0; s < RES_SLOTS; ++s)
            if (own[s] >= 0) {
                r[s] = r[s] - alpha * q[s];
                x[s] = x[s] + alpha * p[own[s]];
                const double z = iv[s] * r[s];
                publish(s, z);
                v2[0] += r[s] * r[s];
                v2[1] += r[s] * z;
            }
        ok = grid_sum(v2);
        if (!ok) break;
        ++it;
        rn = sqrt(v2[0]);
        if (rn <= tol_nb || it >= A.max_iter) break;
        beta = v2[1] / rz;
        rz = v2[1];
        if (!(rz > 0.0)) { breakdown = 1; break; }
    }

    // ---- finish: ||b - A x|| (cg.hpp:222-237) -------------------------------------------------
    double res = 0.0;
    if (ok) {
#pragma unroll
        for (int s = 0; s < RES_SLOTS; ++s)
            if (own[s] >= 0) publish(s, x[s]);
        double v0[1] = {0.0};
        ok = grid_sum(v0);
        if (ok) {
            for (int u = tid; u < H; u += RES_THREADS) p[u] = 0.0;
            gather(0.0);
            spmv();
            double v1[1] = {0.0};
#pragma unroll
            for (int s = 0; s < RES_SLOTS; ++s)
                if (own[s] >= 0) {
                    const double t = A.b[r0 + grp + s * NG] - q[s];
                    v1[0] += t * t;
                }
            ok = grid_sum(v1);
            res = sqrt(v1[0]);
        }
    }
#pragma unroll
    for (int s = 0; s < RES_SLOTS; ++s)
        if (own[s] >= 0) A.x[r0 + grp + s * NG] = nb == 0.0 ? 0.0 : x[s];
    if (me == 0 && tid == 0) {
        A.out->nb = nb;
        A.out->rn = rn;
        A.out->res64 = res;
        A.out->it = it;
        A.out->breakdown = breakdown;
        A.out->unfit = 0;
        A.out->timeout = !ok;
    }
    if (CL) cluster_barrier();                        // no block leaves while another reads its shared memory
}

// ---- host side -------------------------------------------------------------------------------
using ResKernel = void (*)(ResArgs);

// Where the line lies: at what fits, for every size below it is faster on chip.  Microseconds an
// iteration, the streaming loop / here (P2 unless said, one B200):
//     rows      1,521   9,025 (P3)   16,129    25,281    74,529   89,401 (P3)  159,201
//             14 / 3.2   15 / 4.5   15 / 4.4  15 / 5.5  17.9 / 6.0  20 / 7.0   24 / 7.2
// One cluster is taken as long as 16 blocks hold the system: its sums take 0.7 to 1.0 us against
// 2.0 us over the grid, more than the fewer SMs cost (16,129 rows: 4.4 us).
// A lane group holds RES_SLOTS rows, so a block at most RES_SLOTS RES_THREADS: a matrix of few entries a
// row goes to the grid where the cluster has room for its bytes but not for its rows.  Where a form did not
// fit after all (rows of very uneven length), the next one is tried, and then the streaming loop.
bool resident_plan(femd_ctx ctx, int n, long long nnz, int unfit, ResidentPlan &plan)
{
    // a block's share: 10 B an entry, 4 B a row, and 12 B for each of its distinct columns; on P1-P3
    // meshes of 20 to 400 squares a side the fullest block takes 1.3 to 1.6 times its entries' and
    // rows' bytes.  The kernel checks what it finds and says so where a block does not fit.
    const int smem = 220 * 1024;
    const double bytes = 1.6 * (10.0 * (double)nnz + 4.0 * n);
    plan.smem = smem;
    const long long rows = RES_SLOTS * RES_THREADS;
    plan.cluster = !(unfit & RES_UNFIT_CLUSTER) && bytes <= (double)RES_MAX_CLUSTER * (smem - 20 * 1024) && n <= RES_MAX_CLUSTER * rows;
    plan.blocks = plan.cluster ? RES_MAX_CLUSTER : std::min(ctx->sm_count, RES_MAX_BLOCKS);
    return plan.cluster || (!(unfit & RES_UNFIT_GRID) && bytes <= (double)plan.blocks * smem && n <= plan.blocks * rows);
}

cudaError_t resident_launch(const ResidentPlan &plan, const int *indptr, const int *indices, const double *data,
                            const double *inv, const double *b, double *x, int n, int max_iter, double tol, double *zx,
                            double *slots, ResidentOut *out, cudaStream_t s)
{
    ResArgs A{indptr, indices, data, inv, b, x, zx, slots, reinterpret_cast<unsigned long long *>(slots + RES_SUM_DOUBLES), out,
              tol, n, max_iter, plan.smem};
    ResKernel k = plan.cluster ? k_cg_resident<true> : k_cg_resident<false>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, plan.smem);
    if (e == cudaSuccess && plan.cluster) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess && !plan.cluster) e = cudaMemsetAsync(A.count, 0, sizeof(*A.count), s);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)plan.blocks);
    cfg.blockDim = dim3(RES_THREADS);
    cfg.dynamicSmemBytes = (size_t)plan.smem;
    cfg.stream = counted(s);
    cudaLaunchAttribute at[1];
    if (plan.cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)plan.blocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, A);
}

}  // namespace femd
