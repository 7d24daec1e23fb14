// precond.cu -- the reference's stronger preconditioners on the GPU: ILU(0) and SSOR on the natural
// ordering (include/femd/sparse/precond.hpp:105-213), for CG (krylov::cg, krylov/cg.hpp:245-290).
//
// Both are sequential sweeps over the rows: ILU(0)'s factorization (IKJ: row i is eliminated with
// the finished rows k < i of its lower part) and the triangular solves of every application.  Row
// i depends only on the rows its lower (forward) or upper (backward) part names, so the rows fall
// into levels -- level(i) = 1 + the largest level among them -- and the rows of one level are
// independent.  The level schedules are built once per pattern on the host.  The factorization and
// each application then run as ONE thread block that walks the levels in order with a block barrier
// between them: a thread takes a row and does that row's arithmetic exactly as the reference
// writes it (the same operations in the same order, no contraction), so the factors and every
// application are bit-identical to the reference's; only the order in which independent rows are
// done differs.  No block waits on another, so nothing can hang.
//
// The price is parallelism: one SM per application, latency-bound by the number of levels (about
// 4 N for P2 on an N x N rectangle, each way).  The reference's natural-order ILU(0) has no more
// parallelism to give; a faster preconditioner would be a different one (another ordering), with
// other iterates.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <limits>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "precond_host.h"

struct femd_precond_s : femd::HandleBase {
    femd_ctx ctx = nullptr;
    femd_pattern pattern = nullptr;
    unsigned long long id;               // of no other preconditioner of the process, before or after
    int pc_kind = 0;                     // FEMD_PC_ILU0 / FEMD_PC_SSOR
    double omega = 1.0, min_pivot = 0.0;
    int n = 0, levels_f = 0, levels_b = 0;
    int nlf = 0, nlb = 0;                // chunks: one a level, more where a level is very large
    // the sweeps' chunks, one per forward and backward level in order (k_pc_apply), their places and
    // sizes, and the launch
    femd::DevBuf<uint4> chunks;
    femd::DevBuf<int2> places;
    int threads = 0, slot = 0, zs = 0, ring = 0;
    // the bound of a wait for the ring's copies, and the word an application sets where one ran out
    int spins = 0;
    femd::DevBuf<int> late;
    size_t smem = 0;
    static unsigned long long next_id()
    {
        static std::atomic<unsigned long long> count{0};
        return ++count;
    }
    femd_precond_s() : HandleBase(femd::KIND_PRECOND), id(next_id()) {}
    ~femd_precond_s() override { femd::ctx_release(ctx); }
};

namespace femd {

static constexpr int PC_BLOCK = 1024;

// ILU(0) factorization, the reference's IKJ loop per row (precond.hpp:172-186): for each k in the
// lower part of row i (increasing), v_ik /= v_kk, then v_ij -= v_ik v_kj over the upper part of
// row k where (i, j) is in the pattern (found by a merge of the two sorted rows).
__global__ void __launch_bounds__(PC_BLOCK) k_ilu0_factor(const int *__restrict__ ip, const int *__restrict__ ix,
                                                         const int *__restrict__ diag, double *__restrict__ v, int nl,
                                                         const int *__restrict__ lptr, const int *__restrict__ rows,
                                                         int *__restrict__ status)
{
    for (int L = 0; L < nl; ++L) {
        for (int t = lptr[L] + (int)threadIdx.x; t < lptr[L + 1]; t += PC_BLOCK) {
            const int i = rows[t];
            const int hi = ip[i + 1], di = diag[i];
            for (int p = ip[i]; p < di; ++p) {
                const int k = ix[p];
                const double lik = __ddiv_rn(v[p], v[diag[k]]);
                v[p] = lik;
                int s = p + 1;                                   // columns of row i after k (sorted)
                for (int q = diag[k] + 1; q < ip[k + 1]; ++q) {
                    const int j = ix[q];
                    while (s < hi && ix[s] < j) ++s;
                    if (s < hi && ix[s] == j) v[s] = __dsub_rn(v[s], __dmul_rn(lik, v[q]));
                }
            }
            if (v[di] == 0.0) atomicMin(status, i);
        }
        __syncthreads();                                         // the level's rows are final
    }
}

// ---- an application: the forward and the backward sweep, level by level ------------------------
// What bounds it is the chain of one level, most of all the instructions one warp issues in it: the
// barrier, the gathers of z, the row's subtractions in order (and in the backward sweep a
// division), the store of z.  So everything that does not depend on z is brought near beforehand:
// the levels' rows are packed into chunks in the order of the sweeps, a warp of its own has
// them copied into a ring of shared memory 8 or 4 levels ahead (bulk copies; the block's barrier of a
// level also hands them over), a row's first entries are in registers before the barrier that
// frees it, and z itself lies in shared memory (ZS) while it fits; all of it at 32-bit places in
// shared memory with constant strides.  One application at P2 64 x 64 (16,129 rows, 254 + 254
// levels): 935 us with rows read from CSR through the level lists by two launches, 282 here; of
// that the division takes 6 %, the subtractions 20 %, loading the next level's rows 24 %.
//
// A chunk that no slot holds (the inner nodes of all cells at P3 are one level) is read where it lies.
//
// Chunk: int4 {its rows, the next chunk's rows, the next chunk's place (in 16 B) where it is read
// there or -1, 0};
// a PcRow per row; values double x E; columns int x E.  A chunk's rows are sorted by length and lie
// in slices of PC_SLICE rows, two values or four columns of a row side by side (16-byte loads, a
// slice's 128 B together).  The 32 rows of a warp are filled up to the same number of entries, a
// multiple of 4, with the value +0 on column n, whose z is +0: s - (+0 * +0) is s, bit for bit, so
// no lane needs a test in the chain.  With z in shared memory a column is its place there in bytes.
static constexpr int PC_AHEAD = 8;
static constexpr int PC_ROWS = 256, PC_COPY = 32;    // threads that take rows (at most), and that copy
static constexpr size_t PC_SMEM = 220 * 1024;

struct __align__(16) PcRow {
    int row, len, val, col;              // len: filled up; bytes from the chunk's start to the first value and column
    double diag, pad;
};

static_assert(sizeof(PcRow) == PC_RECORD && sizeof(int4) == PC_HEAD, "as the host lays the chunks out");

// Fill the chunks: one thread per row in level order (rows; lptr: the levels' first).
__global__ void k_pc_pack(const int *__restrict__ ip, const int *__restrict__ ix, const int *__restrict__ diag,
                          const double *__restrict__ v, const int *__restrict__ rows, const int *__restrict__ lptr, int nl,
                          const int *__restrict__ eoff, const int *__restrict__ etot, const int *__restrict__ place,
                          const int *__restrict__ next_m, int l0, int nchunk, int slot, int n, bool forward, bool zs, char *__restrict__ chunks)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        int lo = 0, hi = nl - 1;                             // the level of t
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (lptr[mid] <= t) lo = mid; else hi = mid - 1;
        }
        const int first = lptr[lo], m = lptr[lo + 1] - first, u = t - first, c = l0 + lo, E = etot[c];
        char *base = chunks + 16 * (size_t)place[c];
        if (u == 0)
            *reinterpret_cast<int4 *>(base) =
                make_int4(m, next_m[c], c + 1 < nchunk && 16ll * (place[c + 2] - place[c + 1]) > slot ? place[c + 1] : -1, 0);
        const int i = rows[t], d = diag[i];
        const int q0 = forward ? ip[i] : d + 1, len = forward ? d - q0 : ip[i + 1] - q0;
        PcRow rec;
        int most = 0;                                        // of the warp's rows
        for (int x = u & ~31; x < min(m, (u & ~31) + 32); ++x) {
            const int k = rows[first + x];
            most = max(most, forward ? diag[k] - ip[k] : ip[k + 1] - diag[k] - 1);
        }
        rec.row = i;
        rec.len = (most + 3) & ~3;
        rec.val = 16 + (int)sizeof(PcRow) * m + 8 * eoff[t] + 16 * (u % PC_SLICE);
        rec.col = 16 + (int)sizeof(PcRow) * m + 8 * E + 4 * eoff[t] + 16 * (u % PC_SLICE);
        rec.diag = v[d];
        rec.pad = 0.0;
        reinterpret_cast<PcRow *>(base + 16)[u] = rec;
        for (int j = 0; j < rec.len; ++j) {
            const int k = j < len ? ix[q0 + j] : n;
            *reinterpret_cast<double *>(base + rec.val + 16 * PC_SLICE * (j / 2) + 8 * (j % 2)) = j < len ? v[q0 + j] : 0.0;
            *reinterpret_cast<int *>(base + rec.col + 16 * PC_SLICE * (j / 4) + 4 * (j % 4)) = zs ? 8 * k : k;
        }
    }
}

// The ring's copies: one mbarrier a slot, waited on by the copying warp alone.  A wait is bounded: past
// it the block leaves at the next barrier, before anything is read from the slot, gives z back as NaN
// (so CG ends, by its breakdown test) and sets *late_out, which the solve reports.  The word that every
// thread reads for it takes 10 us of an application's 282 at P2 64 x 64; a barrier that carries it
// (__syncthreads_or) 14, a chunk of zeros in the slot's place 21.
static constexpr int PC_SPINS = 1 << 22;

__device__ __forceinline__ void pc_copy(char *dst, const uint4 *src, int n16, uint64_t *bar)
{
    const unsigned b = (unsigned)__cvta_generic_to_shared(bar), d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(b), "r"(16u * n16) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(d), "l"(src), "r"(16u * n16), "r"(b) : "memory");
}

__device__ __forceinline__ bool pc_wait(uint64_t *bar, unsigned parity, int spins)
{
    for (int spin = 0; spin < spins; ++spin) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"((unsigned)__cvta_generic_to_shared(bar)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// z = M^{-1} r.  ILU(0): z_i = r_i - sum_{p < d_i} v_p z_col, then z_i = (z_i - sum_{p > d_i} v_p
// z_col) / v_ii (precond.hpp:193-204).  SSOR: (r_i - sum) w / v_ii; z_i c v_ii / w with c = (2 -
// w) / w; (z_i - sum) w / v_ii (:127-142).  ZS: z in shared memory; RING: the ring's slots; places: the
// chunks' places and sizes in 16 B (size 0: read where it lies); spins: the bound of a wait.
template <bool SSOR, bool ZS, int RING>
__global__ void __launch_bounds__(PC_ROWS + PC_COPY) k_pc_apply(const uint4 *__restrict__ chunks, const int2 *__restrict__ places, int nlf,
                                                      int nl, int slot, int n, double w, const double *__restrict__ r,
                                                      double *z, const int *__restrict__ skip, int spins, int *late_out)
{
    extern __shared__ __align__(16) char dyn[];
    if (skip && *skip) return;
    // shared memory: z (ZS), then the ring; places are 32-bit
    const unsigned ring0 = ZS ? ((unsigned)n * 8u + 23u) / 16u * 16u : 0u;   // z and its +0
    const unsigned dyn0 = (unsigned)__cvta_generic_to_shared(dyn);
    auto z_at = [&](int i) -> double & { return ZS ? reinterpret_cast<double *>(dyn)[i] : z[i]; };
    const int tid = threadIdx.x, T = blockDim.x - PC_COPY;   // threads that take rows
    const double c = SSOR ? __ddiv_rn(__dsub_rn(2.0, w), w) : 0.0;
    if (ZS) {
        constexpr int U = 8;                                 // loads in flight
        for (int i0 = tid; i0 < n; i0 += U * blockDim.x) {
            double t[U];
#pragma unroll
            for (int u = 0; u < U; ++u) t[u] = i0 + u * blockDim.x < n ? r[i0 + u * blockDim.x] : 0.0;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i0 + u * blockDim.x < n) z_at(i0 + u * blockDim.x) = t[u];
        }
        if (tid == 0) z_at(n) = 0.0;
    }
    __shared__ uint64_t bar[RING];
    // the level whose barrier followed a wait that ran out (-1: the first barrier): a thread past the barrier
    // of level L leaves where that is L or before; a later barrier's word may already be there
    __shared__ volatile int s_late;
    if (tid >= T) {
        // the copying warp: chunk L + 2 is in when level L ends (its threads then load from it)
        const bool lead = tid == T;
        int issued = 0, arrived = 0;
        // chunk k into its slot; one that no slot holds only counts as arrived
        auto issue = [&](int2 c) {
            if (c.y) pc_copy(dyn + ring0 + issued % RING * slot, chunks + c.x, c.y, &bar[issued % RING]);
            else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"((unsigned)__cvta_generic_to_shared(&bar[issued % RING])) : "memory");
            ++issued;
        };
        int2 next = make_int2(0, 0);                         // the chunk issued after the next barrier
        if (lead) {
            s_late = nl;
            for (int k = 0; k < RING; ++k)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((unsigned)__cvta_generic_to_shared(&bar[k])) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            while (issued < RING && issued < nl) issue(places[issued]);
            if (issued < nl) next = places[issued];
        }
        for (int L = -1; L < nl; ++L) {
            if (lead)
                while (arrived < min(L + 3, issued)) {
                    if (!pc_wait(&bar[arrived % RING], (unsigned)(arrived / RING) & 1u, spins)) {
                        s_late = L;
                        break;
                    }
                    ++arrived;
                }
            __syncwarp();
            __syncthreads();                                 // the level's rows are final, its slot is free
            if (s_late <= L) break;
            if (lead && L >= 0 && issued < nl) {
                issue(next);
                if (issued < nl) next = places[issued];
            }
        }
        if (lead && s_late < nl)                                  // leave no copy in flight
            for (; arrived < issued; ++arrived) pc_wait(&bar[arrived % RING], (unsigned)(arrived / RING) & 1u, PC_SPINS);
        __syncwarp();
    } else {
        __syncthreads();
        unsigned place = dyn0 + ring0;                       // of the level's chunk in the ring
        const char *chunk = nullptr;                         // or where it lies (AT)
        auto get4 = [&](auto AT, int o) {
            int4 t;
            if (AT) t = *reinterpret_cast<const int4 *>(chunk + o);
            else asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(t.x), "=r"(t.y), "=r"(t.z), "=r"(t.w) : "r"(place + o));
            return t;
        };
        auto get2 = [&](auto AT, int o) {
            double2 t;
            if (AT) t = *reinterpret_cast<const double2 *>(chunk + o);
            else asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(t.x), "=d"(t.y) : "r"(place + o));
            return t;
        };
        auto z_get = [&](int col) {                          // col as the chunk has it
            double t;
            if (ZS) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(t) : "r"(dyn0 + col));
            else t = col < n ? z[col] : 0.0;
            return t;
        };
        // a row's record and first entries
        int4 me = make_int4(0, 0, 0, 0), col[PC_AHEAD / 4];
        double2 v[PC_AHEAD / 2];
        double dg = 1.0;
        bool have = false;
        auto load = [&](auto AT, int u, int m) {
            have = u < m;
            if (!have) return;
            me = get4(AT, 16 + 32 * u);
            dg = get2(AT, 32 + 32 * u).x;
#pragma unroll
            for (int h = 0; h < PC_AHEAD / 4; ++h)
                if (4 * h < me.y) {
                    col[h] = get4(AT, me.w + 16 * PC_SLICE * h);
                    v[2 * h] = get2(AT, me.z + 32 * PC_SLICE * h);
                    v[2 * h + 1] = get2(AT, me.z + 32 * PC_SLICE * h + 16 * PC_SLICE);
                }
        };
        auto subtract4 = [&](double s, const int4 &k, const double2 &a, const double2 &b) {
            const double g0 = z_get(k.x), g1 = z_get(k.y), g2 = z_get(k.z), g3 = z_get(k.w);
            s = __dsub_rn(s, __dmul_rn(a.x, g0));
            s = __dsub_rn(s, __dmul_rn(a.y, g1));
            s = __dsub_rn(s, __dmul_rn(b.x, g2));
            return __dsub_rn(s, __dmul_rn(b.y, g3));
        };
        auto row = [&](auto AT, auto forward) {
            if (!have) return;
            constexpr bool FWD = decltype(forward)::value;
            double s = !ZS && FWD ? r[me.x] : z_get(ZS ? 8 * me.x : me.x);
            if (SSOR && !FWD) s = __dmul_rn(s, __ddiv_rn(__dmul_rn(c, dg), w));
#pragma unroll
            for (int h = 0; h < PC_AHEAD / 4; ++h)
                if (4 * h < me.y) s = subtract4(s, col[h], v[2 * h], v[2 * h + 1]);
            if (PC_AHEAD < me.y) {
                // the rest: the next four are loaded while these are subtracted
                int ov = me.z + 8 * PC_SLICE * PC_AHEAD, oc = me.w + 4 * PC_SLICE * PC_AHEAD;
                int4 k = get4(AT, oc);
                double2 a = get2(AT, ov), b = get2(AT, ov + 16 * PC_SLICE);
                for (int left = me.y - PC_AHEAD - 4; left >= 0; left -= 4) {
                    const int4 kk = k;
                    const double2 aa = a, bb = b;
                    if (left > 0) {
                        oc += 16 * PC_SLICE;
                        ov += 32 * PC_SLICE;
                        k = get4(AT, oc);
                        a = get2(AT, ov);
                        b = get2(AT, ov + 16 * PC_SLICE);
                    }
                    s = subtract4(s, kk, aa, bb);
                }
            }
            if (SSOR) s = __ddiv_rn(__dmul_rn(s, w), dg);
            else if (!FWD) s = __ddiv_rn(s, dg);
            if (ZS) asm volatile("st.shared.f64 [%0], %1;" :: "r"(dyn0 + 8 * me.x), "d"(s) : "memory");
            else z[me.x] = s;
        };
        const std::true_type lies{};
        const std::false_type ringed{};
        // rows of this level and the next, and whether this level is read where it lies
        int4 head = make_int4(0, 0, -1, 0);
        bool at = places[0].y == 0;
        const bool none = s_late < 0;                        // the first chunks are not here
        if (none) at = false;
        else if (at) chunk = reinterpret_cast<const char *>(chunks + places[0].x);
        else {
            head = get4(ringed, 0);
            load(ringed, tid, head.x);
        }
        auto levels = [&](auto forward, int L0, int L1) {
            for (int L = L0; L < L1; ++L) {
                const int late = s_late;                     // covers the next level's chunk
                if (at) {
                    head = get4(lies, 0);
                    for (int u = tid; u < head.x; u += T) {
                        load(lies, u, head.x);
                        row(lies, forward);
                    }
                } else {
                    row(ringed, forward);
                    for (int u = tid + T; u < head.x; u += T) {
                        load(ringed, u, head.x);
                        row(ringed, forward);
                    }
                }
                if (late < L) return;
                // the next level's rows: its chunk was handed over by the last barrier
                place = (L + 1) % RING ? place + slot : dyn0 + ring0;
                at = head.z >= 0;
                if (at) chunk = reinterpret_cast<const char *>(chunks + head.z);
                else if (L + 1 < nl) {
                    load(ringed, tid, head.y);
                    head = get4(ringed, 0);
                }
                __syncthreads();                             // the level's rows are final
            }
        };
        if (!none) levels(std::true_type(), 0, nlf);
        if (s_late >= nlf) levels(std::false_type(), nlf, nl);
    }
    const bool left = s_late < nl;
    if (left) {                                              // every thread left at the same barrier
        __syncthreads();                                     // a last level's rows may just have been stored
        if (tid == 0) *late_out = 1;
    }
    if (ZS || left)
        for (int i = tid; i < n; i += blockDim.x) z[i] = left ? __longlong_as_double(0x7ff8000000000000ll) : z_at(i);
}

using PcKernel = void (*)(const uint4 *, const int2 *, int, int, int, int, double, const double *, double *, const int *, int, int *);

template <bool SSOR>
static PcKernel pc_kernel(bool zs, int ring)
{
    if (zs) return ring == 8 ? k_pc_apply<SSOR, true, 8> : k_pc_apply<SSOR, true, 4>;
    return ring == 8 ? k_pc_apply<SSOR, false, 8> : k_pc_apply<SSOR, false, 4>;
}

__global__ void k_pc_min_diag(int n, const int *__restrict__ diag, const double *__restrict__ v, double *out)
{
    __shared__ double sh[32];
    double m = INFINITY;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmin(m, v[diag[i]]);
    for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = INFINITY;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) r = fmin(r, sh[k]);
        *out = r;
    }
}

static femd_precond_s *as_precond(void *h)
{
    femd_precond_s *p = static_cast<femd_precond_s *>(h);
    return (p && p->kind == KIND_PRECOND) ? p : nullptr;
}

// z = M^{-1} r on the stream, every kernel skipped when *skip is set (a finished CG loop)
int precond_enqueue(femd_precond P, const double *r, double *z, const int *skip, cudaStream_t s)
{
    if (P->n == 0) return FEMD_OK;
    PcKernel k = P->pc_kind == FEMD_PC_ILU0 ? pc_kernel<false>(P->zs, P->ring) : pc_kernel<true>(P->zs, P->ring);
    FEMD_TRY_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PC_SMEM));
    k<<<1, P->threads, P->smem, counted(s)>>>(P->chunks.p, P->places.p, P->nlf, P->nlf + P->nlb, P->slot, P->n, P->omega, r, z, skip,
                                               P->spins, P->late.p);
    FEMD_TRY_CUDA(cudaGetLastError());
    return FEMD_OK;
}

unsigned long long precond_id(femd_precond P) { return P->id; }

// Whether a wait of an application on s ran out since the last call; waits for s.
int precond_take_late(femd_precond P, bool *late, cudaStream_t s)
{
    int word = 0;
    *late = false;
    if (P->n == 0) return FEMD_OK;
    FEMD_TRY_CUDA(cudaMemcpyAsync(&word, P->late.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    FEMD_TRY_CUDA(cudaMemsetAsync(P->late.p, 0, sizeof(int), s));
    FEMD_TRY_CUDA(cudaStreamSynchronize(s));
    *late = word != 0;
    return FEMD_OK;
}

int precond_rows(femd_precond P) { return P->n; }
femd_ctx precond_ctx(femd_precond P) { return P->ctx; }
femd_pattern precond_pattern(femd_precond P) { return P->pattern; }

}  // namespace femd

using namespace femd;

extern "C" {

int femd_cuda_precond_create(femd_ctx ctx, femd_matrix K, int kind, double omega, femd_precond *out)
{
    clear_error();
    FEMD_CHECK_ARG(ctx && K && K->kind == KIND_MATRIX && out, "preconditioner: NULL argument");
    FEMD_CHECK_ARG(kind == FEMD_PC_ILU0 || kind == FEMD_PC_SSOR, "preconditioner: kind is FEMD_PC_ILU0 or FEMD_PC_SSOR");
    const char *what = kind == FEMD_PC_ILU0 ? "ILU(0)" : "SSOR";
    FEMD_CHECK_ARG(K->pattern->nrows == K->pattern->ncols, std::string(what) + ": the matrix must be square");
    FEMD_CHECK_ARG(kind != FEMD_PC_SSOR || (omega > 0.0 && omega < 2.0), "SSOR: omega must lie in (0, 2)");
    *out = nullptr;
    FEMD_TRY_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    femd_pattern Q = K->pattern;
    const int n = Q->nrows;
    const long long nnz = Q->nnz;
    // the pattern and the diagonal positions on the host (precond.hpp:68-78: a missing or zero
    // diagonal entry is refused)
    std::vector<int> ip((size_t)n + 1), ix((size_t)std::max<long long>(nnz, 1)), dg((size_t)std::max(n, 1));
    std::vector<double> vals((size_t)std::max<long long>(nnz, 1));
    FEMD_TRY_CUDA(cudaMemcpyAsync(ip.data(), Q->indptr.p, ((size_t)n + 1) * sizeof(int), cudaMemcpyDeviceToHost, s));
    if (nnz) {
        FEMD_TRY_CUDA(cudaMemcpyAsync(ix.data(), Q->indices.p, (size_t)nnz * sizeof(int), cudaMemcpyDeviceToHost, s));
        FEMD_TRY_CUDA(cudaMemcpyAsync(vals.data(), K->data.p, (size_t)nnz * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    FEMD_TRY_CUDA(cudaStreamSynchronize(s));
    for (int i = 0; i < n; ++i) {
        const int *b = ix.data() + ip[i], *e = ix.data() + ip[i + 1];
        const int *f = std::lower_bound(b, e, i);
        dg[i] = (f != e && *f == i) ? (int)(f - ix.data()) : -1;
        FEMD_CHECK_ARG(dg[i] >= 0 && vals[dg[i]] != 0.0, std::string(what) + ": zero diagonal entry in row " + std::to_string(i));
    }
    auto P = new femd_precond_s();
    std::unique_ptr<femd_precond_s> guard(P);
    P->ctx = ctx;
    ctx_retain(ctx);
    P->pattern = Q;
    P->pc_kind = kind;
    P->omega = omega;
    P->n = n;
    std::vector<int> fr, fp, br, bp;
    level_schedule(n, ip, ix, dg, true, fr, fp);
    level_schedule(n, ip, ix, dg, false, br, bp);
    P->levels_f = (int)fp.size() - 1;
    P->levels_b = (int)bp.size() - 1;
    std::vector<int> feoff, beoff, etot, rtot;
    std::vector<long long> pl(1, 0);
    chunk_layout(ip, dg, true, PC_CHUNK_MAX, fr, fp, feoff, etot, rtot, pl);
    chunk_layout(ip, dg, false, PC_CHUNK_MAX, br, bp, beoff, etot, rtot, pl);
    P->nlf = (int)fp.size() - 1;
    P->nlb = (int)bp.size() - 1;
    bool large = pl.back() >= INT_MAX;
    for (size_t k = 0; k + 1 < pl.size(); ++k) large |= 16 * (pl[k + 1] - pl[k]) > INT_MAX;
    FEMD_CHECK_ARG(!large, std::string(what) + ": the matrix is too large");
    std::vector<int> place(pl.begin(), pl.end());
    const int nch = P->nlf + P->nlb;
    rtot.push_back(0);                   // the chunk after the last
    // A thread per row of most levels, in whole warps, at most PC_ROWS.  z in shared memory where it
    // fits beside four slots for nearly all chunks (P2: up to about 20,000 rows), else slots alone.
    std::vector<int> sizes((size_t)nch), widths(rtot.begin(), rtot.end() - 1);
    for (int k = 0; k < nch; ++k) sizes[k] = 16 * (place[k + 1] - place[k]);
    std::sort(sizes.begin(), sizes.end());
    std::sort(widths.begin(), widths.end());
    const int usual = nch ? sizes[(size_t)(nch - 1) * 49 / 50] : 16, width = nch ? widths[(size_t)(nch - 1) * 49 / 50] : 1;
    P->threads = std::min(PC_ROWS, std::max(64, (width + 31) / 32 * 32)) + PC_COPY;
    const size_t zbytes = ((size_t)n * sizeof(double) + 23) / 16 * 16;
    P->zs = zbytes + 4 * (size_t)usual <= PC_SMEM;
    const size_t room = PC_SMEM - (P->zs ? zbytes : 0);
    P->ring = 8 * (size_t)usual <= room ? 8 : 4;
    P->slot = 16;
    for (int b : sizes)
        if ((size_t)b * P->ring <= room) P->slot = std::max(P->slot, b);
    P->smem = (size_t)P->ring * P->slot + (P->zs ? zbytes : 0);
    std::vector<int2> first((size_t)std::max(nch, 1));
    for (int k = 0; k < nch; ++k) {
        const int size = place[k + 1] - place[k];
        first[k] = make_int2(place[k], 16ll * size <= P->slot ? size : 0);
    }
    DevBuf<double> v;                    // ILU(0): the factors L (unit, strict lower) and U; SSOR: the values
    DevBuf<int> diag, frows, fptr, brows, bptr, fe, be, et, rt, plc;
    int st;
    if ((st = v.alloc((size_t)std::max<long long>(nnz, 1))) || (st = diag.alloc((size_t)std::max(n, 1))) ||
        (st = frows.alloc((size_t)std::max(n, 1))) || (st = fptr.alloc(fp.size())) ||
        (st = brows.alloc((size_t)std::max(n, 1))) || (st = bptr.alloc(bp.size())) || (st = fe.alloc(feoff.size() + 1)) ||
        (st = be.alloc(beoff.size() + 1)) || (st = et.alloc(etot.size() + 1)) || (st = rt.alloc(rtot.size())) ||
        (st = plc.alloc(place.size())) || (st = P->chunks.alloc((size_t)pl.back() + 1)) || (st = P->places.alloc(first.size())) || (st = P->late.alloc(1)))
        return st;
    P->spins = PC_SPINS;
    FEMD_TRY_CUDA(cudaMemsetAsync(P->late.p, 0, sizeof(int), s));
    auto up = [&](void *d, const void *h, size_t bytes) { return bytes ? cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s) : cudaSuccess; };
    if (nnz) FEMD_TRY_CUDA(cudaMemcpyAsync(v.p, K->data.p, (size_t)nnz * sizeof(double), cudaMemcpyDeviceToDevice, s));
    FEMD_TRY_CUDA(up(diag.p, dg.data(), (size_t)n * sizeof(int)));
    FEMD_TRY_CUDA(up(frows.p, fr.data(), (size_t)n * sizeof(int)));
    FEMD_TRY_CUDA(up(brows.p, br.data(), (size_t)n * sizeof(int)));
    FEMD_TRY_CUDA(up(fptr.p, fp.data(), fp.size() * sizeof(int)));
    FEMD_TRY_CUDA(up(bptr.p, bp.data(), bp.size() * sizeof(int)));
    FEMD_TRY_CUDA(up(fe.p, feoff.data(), (size_t)n * sizeof(int)));
    FEMD_TRY_CUDA(up(be.p, beoff.data(), (size_t)n * sizeof(int)));
    FEMD_TRY_CUDA(up(et.p, etot.data(), etot.size() * sizeof(int)));
    FEMD_TRY_CUDA(up(rt.p, rtot.data(), rtot.size() * sizeof(int)));
    FEMD_TRY_CUDA(up(plc.p, place.data(), place.size() * sizeof(int)));
    FEMD_TRY_CUDA(up(P->places.p, first.data(), first.size() * sizeof(int2)));
    if (kind == FEMD_PC_ILU0 && n) {
        CtxLock status(ctx->shared);
        FEMD_TRY(reset_status(ctx));
        // status [1] holds the first row with a zero pivot (INT_MAX: none)
        k_ilu0_factor<<<1, PC_BLOCK, 0, counted(s)>>>(Q->indptr.p, Q->indices.p, diag.p, v.p, P->nlf, fptr.p, frows.p,
                                                       ctx->status_dev + 1);
        FEMD_TRY_CUDA(cudaGetLastError());
        int flags = 0, bad = 0;
        FEMD_TRY(read_status(ctx, &flags, &bad));
        if (bad != INT_MAX) {
            set_error("ILU(0): zero pivot in row " + std::to_string(bad));
            return FEMD_EPIVOT;
        }
        DevBuf<double> mp;
        FEMD_TRY(mp.alloc(1));
        k_pc_min_diag<<<1, 1024, 0, counted(s)>>>(n, diag.p, v.p, mp.p);
        FEMD_TRY_CUDA(cudaGetLastError());
        FEMD_TRY_CUDA(cudaMemcpyAsync(&P->min_pivot, mp.p, sizeof(double), cudaMemcpyDeviceToHost, s));
        FEMD_TRY_CUDA(cudaStreamSynchronize(s));   // mp is released here
    }
    if (n) {
        const unsigned grid = grid_for((size_t)n, 128, 1u << 16);
        char *dst = reinterpret_cast<char *>(P->chunks.p);
        k_pc_pack<<<grid, 128, 0, counted(s)>>>(Q->indptr.p, Q->indices.p, diag.p, v.p, frows.p, fptr.p, P->nlf, fe.p, et.p, plc.p,
                                                rt.p + 1, 0, nch, P->slot, n, true, P->zs, dst);
        k_pc_pack<<<grid, 128, 0, counted(s)>>>(Q->indptr.p, Q->indices.p, diag.p, v.p, brows.p, bptr.p, P->nlb, be.p, et.p, plc.p,
                                                rt.p + 1, P->nlf, nch, P->slot, n, false, P->zs, dst);
        FEMD_TRY_CUDA(cudaGetLastError());
    }
    FEMD_TRY_CUDA(cudaStreamSynchronize(s));   // the host vectors are released on return
    *out = reinterpret_cast<femd_precond>(guard.release());
    return FEMD_OK;
}

int femd_cuda_precond_info(femd_precond handle, int *kind, int *levels_forward, int *levels_backward, double *min_pivot)
{
    clear_error();
    femd_precond_s *P = as_precond(handle);
    FEMD_CHECK_ARG(P, "preconditioner: not a preconditioner handle");
    if (kind) *kind = P->pc_kind;
    if (levels_forward) *levels_forward = P->levels_f;
    if (levels_backward) *levels_backward = P->levels_b;
    if (min_pivot) *min_pivot = P->pc_kind == FEMD_PC_ILU0 ? P->min_pivot : 0.0;
    return FEMD_OK;
}

int femd_cuda_precond_debug(femd_precond handle, int spin_limit)
{
    clear_error();
    femd_precond_s *P = as_precond(handle);
    FEMD_CHECK_ARG(P, "preconditioner: not a preconditioner handle");
    P->spins = spin_limit >= 0 ? spin_limit : PC_SPINS;
    P->id = femd_precond_s::next_id();   // a chunk captured before has the old bound
    return FEMD_OK;
}

int femd_cuda_precond_apply(femd_ctx ctx, femd_precond handle, const double *r_dev, double *z_dev)
{
    clear_error();
    femd_precond_s *P = as_precond(handle);
    FEMD_CHECK_ARG(ctx && P && (P->n == 0 || (r_dev && z_dev)), "preconditioner: bad arguments");
    FEMD_CHECK_ARG(r_dev != z_dev || P->n == 0, "preconditioner: r and z must be separate vectors");
    FEMD_TRY_CUDA(cudaSetDevice(ctx->device));
    return precond_enqueue(P, r_dev, z_dev, nullptr, ctx->stream);
}

}  // extern "C"
