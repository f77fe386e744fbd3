// Resident PCG: every phase of a solve in one cooperative launch, with one
// block per SM and a fixed share of a system's rows per block. Included by
// cfem_solve.cu (it uses that file's SysDev, SysState, advance()).
//
// What bounds a CG iteration on the systems this runs is not traffic but
// the chain of dependent steps - gathers, block sums, the grid-wide sum and
// the scalars that follow from it - and the L1 throughput of 32-way
// scattered gathers. So a block keeps what it alone reads in shared memory
// for the whole solve: its rows' vectors, as many of its matrix slices as
// fit (the 148 SMs hold 33 MB between them; the rest streams from L2 or
// HBM), and the part of the direction that its rows' columns name (the
// halo). The product phase first loads the halo, every distinct column once
// and all of them in flight together, and then gathers from shared memory
// with 16-bit local columns.
//
// The grid meets twice per iteration in a sum that is its own barrier: every
// block writes its partial sums with an epoch in one 16-byte word, one warp
// of every block reads all the words, adds them in block order and advances
// the system's state for its own block. No atomics, and no second round trip
// to fetch the result. The words are kept in several copies, each read by
// its share of the blocks: 148 blocks polling one copy took 10.0 us for an
// iteration's two sums (measured without the CG arithmetic), 8 copies 6.7 us.
//
// A neighbour's z and its previous direction p, from which the new direction
// p = zeta z + beta p follows, are stored as pairs, so the halo is one load
// per entry. A pair is written by its row's block in the update phase and
// read in the product phase, with the grid's sum between them.
//
// Measured per iteration (residual replacements included), before on the
// launches over CSR or on the graph scheduler, and here: P1 box 20^3 in FP64
// 22 -> 7.2 us; Tet10 cantilever of 40 x 5 x 5 cells in FP64 41 -> 10.7 us
// (0.6 halo, 1.8 products, 3.2 sum, 0.4 update, 4.3 sum); Tet10 box of 27 x
// 15 x 13 cells, elasticity in FP32, 52 MB of blocks of which 60 % fit, 32
// -> 19 us; Tet10 heat of 44,415 rows in FP32 45 -> 10.0 us; P1 heat of
// 699,273 rows in FP64 (104 MB streamed per iteration) 60 -> 40 us.
//
// Sums depend on the system's own block count and lanes per row. There are
// two block counts, one for solves and a smaller one for solve slots
// (rs_blocks), which depend on the system alone: within either a result is
// bitwise the same alone and in any batch. Only a batch with dealt blocks
// (rs_plan) has others.

constexpr int RT = 512;              // threads per block
constexpr int RWARPS = RT / 32;
constexpr int RS_WINDOW = 256;       // rows sorted by length together
constexpr int RS_SMEM_MAX = 224 * 1024;
constexpr size_t RS_MAX_WAVES = 4;   // launches of one batch
constexpr int RS_HOLD = 150 * 1024;  // matrix bytes a block is meant to hold
constexpr int64_t RS_DEAL_BYTES = 2 << 20;   // matrix bytes per block when blocks are dealt out
constexpr int RS_COPIES = 8;         // copies of the partial sums, at most
constexpr int RM = 6;                // rigid-body modes of a piece (cfem_coarse.cuh)

template <typename T> struct PairOf;
template <> struct PairOf<float> { using type = float2; };
template <> struct PairOf<double> { using type = double2; };

struct RsShared {
    double red[4][RWARPS];
    SysState st;
    int quit;
    int nres;                        // leading slices held in shared memory
    int own;                         // place of the block's first row in its halo
};
// ... of the coarse correction: partial sums, products with the coarse
// inverse, the block's own coefficients y
struct RsCoarse {
    double red[RM][64], prod[2][RM], y[RM];
};

__host__ __device__ inline size_t rs_al(size_t v) { return (v + 15) & ~(size_t)15; }
__host__ __device__ inline int rs_slices(int rows, int lsh) {   // of 32 / L rows
    return (rows + (32 >> lsh) - 1) >> (5 - lsh);
}
// Shared-memory bytes of a block's slice offsets and row order, of its halo
// (column list and direction) and of its rows' vectors (q, r, the Jacobi
// inverse and the fixed mask).
__host__ __device__ inline size_t rs_meta_bytes(int rows, int lsh) {
    const size_t nsl = (size_t)rs_slices(rows, lsh);
    return rs_al((nsl + 1) * 4) + rs_al(nsl << (5 - lsh));
}
// Place of a halo entry, its low five bits mixed with the next five. A slice's
// lanes hold rows of one kind (sorted by length), whose k-th columns lie a
// fixed stride apart, 8 on a Tet10 mesh: 8 of 32 lanes met in each of 4 banks
// (a batch of 48 Tet10 meshes: 53.7 ms without, 49.2 with). Applied to the
// local columns when they are made, and to the halo's and the own rows' places.
__host__ __device__ inline int rs_swz(int i) { return i ^ ((i >> 5) & 31); }
__host__ __device__ inline size_t rs_halo_bytes(int u, int bs, size_t ts) {
    return rs_al((size_t)u * 4) + (size_t)((u + 31) & ~31) * bs * ts;
}
// ... of the coarse correction: the block's rows of the coarse inverse, the
// sums of all pieces, the rows' coordinates in their piece.
__host__ __device__ inline size_t rs_coarse_bytes(int rows, int ncta) {
    return (size_t)(RM + 1) * RM * ncta * 8 + rs_al((size_t)rows * 12);
}
__host__ __device__ inline size_t rs_vec_bytes(int rows, int bs, size_t ts) {
    const size_t nd = (size_t)rows * bs;
    return 3 * rs_al(nd * ts) + rs_al(nd);
}
// Copies of the words: contention grows with the blocks that poll one.
__host__ __device__ inline int rs_copies_of(int ncta) {
    return ncta > 24 ? RS_COPIES : (ncta > 4 ? 4 : 1);
}
__host__ __device__ inline size_t rs_mail_bytes(int ncta) {
    return (size_t)2 * 4 * rs_copies_of(ncta) * ncta * sizeof(ulonglong2);
}

__device__ __forceinline__ uint16_t ld_stream(const uint16_t *p) {
    uint16_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

// One block's partial sum of one quantity: the value and the epoch it
// belongs to in one 16-byte word that is written and read whole.
__device__ __forceinline__ void mail_put(ulonglong2 *p, double v, unsigned long long epoch) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\t"
                 "st.relaxed.gpu.global.b128 [%0], t;\n\t}"
                 :: "l"(p), "l"(__double_as_longlong(v)), "l"(epoch) : "memory");
}
__device__ __forceinline__ bool mail_get(const ulonglong2 *p, unsigned long long epoch, double &v) {
    long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\t"
                 "mov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    v = __longlong_as_double(lo);
    return (unsigned long long)hi == epoch;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Grid-wide sum of NV quantities over a system's blocks, then the state
// transition adv(totals), in every block for itself (one thread). PUB: what
// the block wrote to global memory before is visible to the system's other
// blocks after it, and theirs to this one (the product phase writes nothing
// others read and goes without). Returns false when a block gave up waiting
// (bounded: timeout_ns).
template <int NV, bool PUB, typename Shared, typename Adv>
__device__ __forceinline__ bool rs_sync(Shared &sh, ulonglong2 *mail, int nc, GridBar *bar, int cta,
                                        unsigned long long epoch, double part[4],
                                        unsigned long long timeout_ns, unsigned hold, Adv adv) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int v = 0; v < NV; ++v) part[v] = warp_sum(part[v]);
    if (lane == 0)
#pragma unroll
        for (int v = 0; v < NV; ++v) sh.red[v][w] = part[v];
    __syncthreads();
    if (w == 0) {
        double tot[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            double t = sh.red[v][lane & (RWARPS - 1)];
#pragma unroll
            for (int o = RWARPS / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            tot[v] = t;
        }
        bool ok = true;
        if (nc > 1 || hold) {
            const int R = rs_copies_of(nc);
            // two sets of words in turn: a block writes set e + 2 only after
            // every block has written, and so read past, set e
            ulonglong2 *box = mail + (size_t)(epoch & 1) * 4 * R * nc;
            if (PUB) fence_gpu();    // the block's writes before its words
            if (lane < R)
#pragma unroll
                for (int v = 0; v < NV; ++v)
                    mail_put(box + (size_t)(4 * lane + v) * nc + cta, tot[v], epoch);
            const ulonglong2 *in = box + (size_t)4 * (cta % R) * nc;
            constexpr int PER = (RS_MAX_CTAS + 31) / 32;
            double got[NV][PER];
            unsigned long long t0 = 0;
            for (unsigned spin = 0;; ++spin) {
                bool all = hold == 0;
#pragma unroll
                for (int v = 0; v < NV; ++v)
#pragma unroll
                    for (int k = 0; k < PER; ++k) {
                        const int c = lane + 32 * k;
                        got[v][k] = 0.0;
                        if (c < nc) all &= mail_get(in + v * nc + c, epoch, got[v][k]);
                    }
                if (__all_sync(0xffffffffu, all)) break;
                if ((spin & 63u) == 63u) {
                    const unsigned long long now = globaltimer();
                    if (t0 == 0) t0 = now;
                    int stop = 0;
                    if (lane == 0) {
                        if (now - t0 > timeout_ns) atomicExch(&bar->err, 1);
                        stop = *(volatile int *)&bar->err;
                    }
                    if (__shfl_sync(0xffffffffu, stop, 0)) {
                        ok = false;
                        break;
                    }
                }
            }
            if (PUB) fence_gpu();    // the other blocks' writes after their words
            if (ok)
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    double t = 0.0;
#pragma unroll
                    for (int k = 0; k < PER; ++k) t += got[v][k];
                    tot[v] = warp_sum(t);
                }
        }
        if (lane == 0) {
            if (ok) adv(tot);
            else sh.quit = 1;
        }
    }
    __syncthreads();
    return sh.quit == 0;
}

// FP32 scalar slices keep a lane's slots in groups of Q = 4, so that a lane
// loads a group's values in 16 bytes and its columns in 8: slot k of a lane
// sits at 32 Q (k / Q) + Q lane + k % Q of the slice (widths are whole
// groups). With one load per slot a streaming slice kept too little in flight:
// 100,000 entries took a block 22 us, now 16. FP64 slots are one 8-byte load
// each: pairs cost more in padding (P1 rows of 15) and registers than they gave.
template <typename T> struct SlotGroup;
template <> struct SlotGroup<float> {
    static constexpr int Q = 4;
    using V = float4;
    using C = ushort4;
};
template <> struct SlotGroup<double> {
    static constexpr int Q = 1;
    using V = double;
    using C = uint16_t;
};
// A warp's next slice: 2 RWARPS - 1 - w, 2 RWARPS + w, 4 RWARPS - 1 - w, ... after
// its first, w. A window's slices go from its longest rows to its shortest, so
// with equal steps the same warps had the longest ones each time (products of a
// block of 332,000 entries 80 -> 62 us).
__device__ __forceinline__ void rs_next(int &s, int &next) {
    const int after = s + 2 * RWARPS;
    s = next;
    next = after;
}
// Slots per group of a slice's layout.
__host__ __device__ inline int rs_group(int bs, size_t ts) { return bs == 1 && ts == 4 ? 4 : 1; }
__device__ __forceinline__ int rs_slot(int k, int lane, int q) {
    return 32 * q * (k / q) + q * lane + k % q;
}
__device__ __forceinline__ float4 ld_stream(const float4 *p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ ushort4 ld_stream(const ushort4 *p) {
    ushort4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u16 {%0, %1, %2, %3}, [%4];"
                 : "=h"(v.x), "=h"(v.y), "=h"(v.z), "=h"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void slots(const float4 &v, float o[4]) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
__device__ __forceinline__ void slots(double v, double o[1]) { o[0] = v; }
__device__ __forceinline__ void slots(const ushort4 &v, int o[4]) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
__device__ __forceinline__ void slots(uint16_t v, int o[1]) { o[0] = v; }

// Groups g .. g + U - 1 of a lane's slots, all loaded first; a group past the
// n-th repeats the last (its values are not used): branches around the loads
// instead cost the streaming FP64 rows a third of their rate.
template <typename T, int U, bool SM>
__device__ __forceinline__ void rs_load(const uint16_t *cp, const T *vp, int g, int n,
                                        typename SlotGroup<T>::C c[U], typename SlotGroup<T>::V a[U]) {
    using G = SlotGroup<T>;
#pragma unroll
    for (int j = 0; j < U; ++j) {
        const auto *p = (const typename G::C *)(cp + 32 * G::Q * (g + j < n ? g + j : n - 1));
        c[j] = SM ? *p : ld_stream(p);
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
        const auto *p = (const typename G::V *)(vp + 32 * G::Q * (g + j < n ? g + j : n - 1));
        a[j] = SM ? *p : ld_stream(p);
    }
}

// One lane's part of a row of a slice of 32 / L rows (L lanes per row, slot k
// of the row in lane k % L); the row's slot 0 (diag: this lane holds it) is
// the diagonal, or the row sum of the FP32 difference form (DIFF), whose
// other slots multiply p_j - p_i. cp, vp: the lane's first group; w: slots.
//
// FP32 slots are loaded 24 at a time of a streaming slice and 8 of a held one,
// and which slices are held depends on what else is in the launch. The sums must
// not: slot e of every group has a running sum of its own, which takes the
// groups in their order however many were loaded together (groups past the
// last add zero). FP64 slots are loaded 8 at a time either way, and every load
// has its own sum.
template <typename T, bool DIFF, bool SM, int U>
__device__ __forceinline__ void rs_groups1(const uint16_t *cp, const T *vp, int g, int n, bool diag,
                                           const T *halo, T pi, T acc[SlotGroup<T>::Q]) {
    constexpr int Q = SlotGroup<T>::Q;
    typename SlotGroup<T>::C c[U];
    typename SlotGroup<T>::V a[U];
    rs_load<T, U, SM>(cp, vp, g, n, c, a);
    T sum[Q];
#pragma unroll
    for (int e = 0; e < Q; ++e) sum[e] = Q == 1 ? (T)0 : acc[e];
#pragma unroll
    for (int j = 0; j < U; ++j) {
        int cj[Q];
        T aj[Q];
        slots(c[j], cj);
        slots(a[j], aj);
#pragma unroll
        for (int e = 0; e < Q; ++e) {
            T pj = halo[cj[e]];
            if (DIFF) pj = (diag && g + j == 0 && e == 0) ? pi : pj - pi;
            sum[e] += (g + j < n ? aj[e] : (T)0) * pj;
        }
    }
#pragma unroll
    for (int e = 0; e < Q; ++e) acc[e] = Q == 1 ? acc[e] + sum[e] : sum[e];
}
template <typename T, bool DIFF, bool SM, int SLOTS>
__device__ __forceinline__ T rs_row1(const uint16_t *cp, const T *vp, int w, bool diag,
                                     const T *halo, T pi) {
    constexpr int Q = SlotGroup<T>::Q, U = SLOTS / Q;
    const int n = w / Q;
    T acc[Q] = {};
    int g = 0;
    for (; n - g > U / 2; g += U) rs_groups1<T, DIFF, SM, U>(cp, vp, g, n, diag, halo, pi, acc);
    if (g < n) rs_groups1<T, DIFF, SM, U / 2>(cp, vp, g, n, diag, halo, pi, acc);
    if constexpr (Q == 4) return (acc[0] + acc[1]) + (acc[2] + acc[3]);
    else return acc[0];
}

// The same over 3x3 blocks: nine value planes of 32 lanes per step.
template <typename T, bool DIFF, bool SM>
__device__ __forceinline__ void rs_row3(const uint16_t *cp, const T *vp, int w, bool diag,
                                        const T *halo, const T pi[3], T acc[3]) {
    constexpr int U = !SM && sizeof(T) == 4 ? 4 : 2;
    for (int t = 0; t < w; t += U) {
        int c[U];
        T a[U][9];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int tt = t + j < w ? t + j : w - 1;
            c[j] = SM ? cp[32 * tt] : ld_stream(cp + 32 * tt);
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int tt = t + j < w ? t + j : w - 1;
#pragma unroll
            for (int e = 0; e < 9; ++e)
                a[j][e] = SM ? vp[32 * (9 * tt + e)] : ld_stream(vp + 32 * (9 * tt + e));
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
            T pj[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                pj[d] = halo[3 * c[j] + d];
                if (DIFF) pj[d] = (diag && t + j == 0) ? pi[d] : pj[d] - pi[d];
                if (t + j >= w) pj[d] = 0;
            }
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int d = 0; d < 3; ++d) acc[r] += a[j][r * 3 + d] * pj[d];
        }
    }
}

// Compensated sums of one lane's part of a row for the FP64 true residual
// (x in the halo), with the sum of magnitudes for its round-off floor.
template <bool SM>
__device__ __forceinline__ void rs_row_dd1(const uint16_t *cp, const double *vp, int w,
                                           const double *halo, double &hi, double &lo, double &ab) {
    constexpr int U = 4;
    for (int g = 0; g < w; g += U) {
        uint16_t c[U];
        double a[U];
        rs_load<double, U, SM>(cp, vp, g, w, c, a);
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (g + j >= w) continue;
            const double x0 = halo[c[j]];
            dd_fma(hi, lo, a[j], x0);
            ab += fabs(a[j] * x0);
        }
    }
}
template <bool SM>
__device__ __forceinline__ void rs_row_dd3(const uint16_t *cp, const double *vp, int w,
                                           const double *halo, double hi[3], double lo[3],
                                           double ab[3]) {
    for (int t = 0; t < w; ++t) {
        const int c = SM ? cp[32 * t] : ld_stream(cp + 32 * t);
        double a[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) a[e] = SM ? vp[32 * (9 * t + e)] : ld_stream(vp + 32 * (9 * t + e));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double xj = halo[3 * c + d];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                dd_fma(hi[r], lo[r], a[r * 3 + d], xj);
                ab[r] += fabs(a[r * 3 + d] * xj);
            }
        }
    }
}

// One lane's part of a CSR row for the FP64 true residual, entries k, k + LANES,
// ... as acc_R, a few loaded together: one at a time, each waiting for its column
// and then for x there, a residual of the Tet10 elastic box of 27 x 15 x 13 cells
// took 125 us, now 85. x comes through L1: the grid's last sum ordered its writes
// before these reads.
template <bool INIT, int BS>
__device__ __forceinline__ void rs_row_R(const SysDev &S, int32_t k, int32_t k1, int64_t row,
                                         double acc[BS], double alo[BS], double aab[BS],
                                         double accf[BS], double dg[BS * BS]) {
    constexpr int U = BS == 1 ? 4 : 2, B2 = BS * BS;
    const double *x = S.x;
    for (; k < k1; k += U * LANES) {
        int64_t j[U];
        double a[U][B2], xj[U][BS];
        bool fj[U][BS];
#pragma unroll
        for (int u = 0; u < U; ++u) j[u] = __ldg(S.ci + (k + u * LANES < k1 ? k + u * LANES : k));
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double *vk = S.v64 + (int64_t)(k + u * LANES < k1 ? k + u * LANES : k) * B2;
#pragma unroll
            for (int e = 0; e < B2; ++e) a[u][e] = __ldg(vk + e);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int d = 0; d < BS; ++d) {
                xj[u][d] = x[j[u] * BS + d];
                fj[u][d] = INIT && S.fixed ? __ldg(S.fixed + j[u] * BS + d) != 0 : false;
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + u * LANES >= k1) break;
#pragma unroll
            for (int c = 0; c < BS; ++c)
#pragma unroll
                for (int d = 0; d < BS; ++d) {
                    const double ax = a[u][c * BS + d] * xj[u][d];
                    dd_fma(acc[c], alo[c], a[u][c * BS + d], xj[u][d]);
                    aab[c] += fabs(ax);
                    if (INIT && fj[u][d]) accf[c] += ax;
                    if (INIT && j[u] == row) dg[c * BS + d] = a[u][c * BS + d];
                }
        }
    }
}

// list: (system, its block) of every block of the launch. A launch runs its
// systems to the end, or for max_iters iterations when they may go on in a
// later launch (keep: the residual and the Jacobi inverse then stay in
// global memory between the launches; the rest is there anyway).
// CO: with the coarse correction of cfem_coarse.cuh.
template <typename T, int BS, bool CO = false>
__global__ void __launch_bounds__(RT, 1)
k_resident(const SysDev *__restrict__ sys, SysState *gst, GridBar *bar,
           const int2 *__restrict__ list_, int nbytes, int max_steps, int max_iters, int keep,
           unsigned long long timeout_ns, unsigned hold) {
    extern __shared__ __align__(128) unsigned char rs_area[];
    __shared__ RsShared sh;
    __shared__ SysDev S;
    __shared__ typename std::conditional<CO, RsCoarse, int>::type co;
    using P2 = typename PairOf<T>::type;
    constexpr bool DIFF = sizeof(T) == 4;
    constexpr int B2 = BS * BS;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int2 place = __ldg(list_ + blockIdx.x);
    const int cta = place.y;
    for (int i = tid; i < (int)(sizeof(SysDev) / 4); i += RT)
        ((int *)&S)[i] = __ldcg((const int *)(sys + place.x) + i);
    for (int i = tid; i < (int)(sizeof(SysState) / 4); i += RT)
        ((int *)&sh.st)[i] = __ldcg((const int *)(gst + place.x) + i);
    if (tid == 0) {
        sh.quit = 0;
        sh.own = 0;
    }
    __syncthreads();
    int ph = sh.st.phase;
    if (ph == PH_DONE) return;
    const RsCta me = S.ctas[cta];
    const uint16_t *scol = S.rcol;
    const T *sval = (const T *)S.rval;
    const int lsh = S.lsh, L = 1 << lsh;
    const int nloc = me.rows, nd = nloc * BS, nsl = rs_slices(nloc, lsh);
    const int64_t r0 = me.row0, d0 = r0 * BS;
    P2 *pair = (P2 *)S.pair;
    const int nu = __ldg(&S.ucnt[cta].x);
    // the block's own arrays
    unsigned char *area = rs_area;
    int *so = (int *)area;                       // slice offsets, from the block's first
    area += rs_al((size_t)(nsl + 1) * 4);
    uint8_t *perm = area;
    area += rs_al((size_t)nsl << (5 - lsh));
    int32_t *list = (int32_t *)area;
    area += rs_al((size_t)nu * 4);
    T *halo = (T *)area;
    area += (size_t)((nu + 31) & ~31) * BS * sizeof(T);
    T *q, *r, *dinv;
    const uint8_t *fx;
    if (S.vsm) {
        const size_t one = rs_al((size_t)nd * sizeof(T));
        q = (T *)area;
        r = (T *)(area + one);
        dinv = (T *)(area + 2 * one);
        uint8_t *f = area + 3 * one;
        for (int i = tid; i < nd; i += RT) f[i] = S.fixed ? __ldg(S.fixed + d0 + i) : 0;
        if (ph != PH_INIT)
            for (int i = tid; i < nd; i += RT) {
                r[i] = __ldcg((const T *)S.r + d0 + i);
                dinv[i] = __ldcg((const T *)S.dinv + d0 + i);
            }
        fx = f;
        area += rs_vec_bytes(nloc, BS, sizeof(T));
    } else {
        q = (T *)S.q + d0;
        r = (T *)S.r + d0;
        dinv = (T *)S.dinv + d0;
        fx = S.fixed ? S.fixed + d0 : nullptr;
    }
    double *ainv = nullptr, *gall = nullptr;     // coarse inverse (own rows), all pieces' sums
    float *xl = nullptr;
    const int nm = RM * S.ncta;
    if constexpr (CO) {
        ainv = (double *)area;
        gall = ainv + RM * nm;
        xl = (float *)(gall + nm);
        area += rs_coarse_bytes(nloc, S.ncta);
        for (int i = tid; i < RM * nm; i += RT) ainv[i] = __ldg(S.ainv + (size_t)RM * cta * nm + i);
        for (int i = tid; i < 3 * nloc; i += RT) xl[i] = __ldg(S.xl + 3 * r0 + i);
    }
    const int64_t *gso = S.soff + me.sl0;
    const int64_t off0 = __ldg(gso);
    for (int i = tid; i <= nsl; i += RT) so[i] = (int)(__ldg(gso + i) - off0);
    for (int i = tid; i < nsl << (5 - lsh); i += RT)
        perm[i] = __ldg(S.sperm + me.sl0 * 32 + i);
    for (int i = tid; i < nu; i += RT) {
        const int32_t c = __ldg(S.ulist + (size_t)cta * S.umax + i);
        list[i] = c;
        if (c == (int32_t)r0) sh.own = i;        // own rows follow one another in the list
    }
    __syncthreads();
    // as many of the leading slices as fit
    const size_t cost = 2 + B2 * sizeof(T);
    const size_t room = (size_t)nbytes - (size_t)(area - rs_area);
    if (tid == 0) {
        int lo = 0, hi = nsl;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((size_t)so[mid] * cost <= room) lo = mid; else hi = mid - 1;
        }
        sh.nres = lo;
    }
    __syncthreads();
    const int nres = sh.nres;
    const int eres = so[nres];                   // entries held (a multiple of 32)
    T *mv = (T *)area;
    uint16_t *mc = (uint16_t *)(area + (size_t)eres * B2 * sizeof(T));
    const uint16_t *gc = scol + off0;
    const T *gv = sval + (size_t)B2 * off0;
    {
        const int n16 = (int)((size_t)eres * B2 * sizeof(T) / 16);
        for (int i = tid; i < n16; i += RT) ((int4 *)mv)[i] = __ldcs((const int4 *)gv + i);
        for (int i = tid; i < eres / 8; i += RT) ((int4 *)mc)[i] = __ldcs((const int4 *)gc + i);
    }
    const int own = sh.own;                      // the direction on the block's own rows
    auto hplace = [](int i) { return BS == 1 ? rs_swz(i) : 3 * rs_swz(i / 3) + i % 3; };
    __syncthreads();

    // the words of an earlier launch hold its epochs: go on from there
    unsigned long long epoch = (unsigned long long)(unsigned)sh.st.pad;
    const int iter0 = sh.st.iter;
    auto adv = [&](const double tot[4]) {
        // a bad diagonal: minus infinity among the magnitudes, or NaN where those
        // overflow as well (a NaN of their own makes the residual's sum one too)
        if (ph == PH_INIT && (tot[3] < 0.0 || (isnan(tot[3]) && isfinite(tot[0]))))
            sh.st.status = CFEM_ERR_BREAKDOWN;
        advance(S, &sh.st, bar, ph, tot, cta == 0);
    };
    // Coarse correction: w += R_i^T v for a row's vector v (0 at fixed DOFs);
    // the block's sums of w to its place among all pieces'; after the grid has
    // met, the block's six products with the coarse inverse in co.prod.
    auto mode_add = [&](double w[RM], int rl, const double v[3]) {
        const double x = xl[3 * rl], y = xl[3 * rl + 1], z = xl[3 * rl + 2];
        w[0] += v[0];
        w[1] += v[1];
        w[2] += v[2];
        w[3] += y * v[2] - z * v[1];
        w[4] += z * v[0] - x * v[2];
        w[5] += x * v[1] - y * v[0];
    };
    auto modes_out = [&](double w[RM]) {
        if constexpr (CO) {
#pragma unroll
            for (int k = 0; k < RM; ++k) {
#pragma unroll
                for (int o = 16; o > 2; o >>= 1) w[k] += __shfl_xor_sync(0xffffffffu, w[k], o);
                if (lane < 4) co.red[k][4 * wid + lane] = w[k];
            }
            __syncthreads();
            if (wid < RM) {
                const double t = warp_sum(co.red[wid][lane] + co.red[wid][lane + 32]);
                if (lane == 0) S.gall[RM * cta + wid] = t;
            }
        }
    };
    auto modes_in = [&]() {
        if constexpr (CO) {
            for (int i = tid; i < nm; i += RT) gall[i] = __ldcg(S.gall + i);
            __syncthreads();
            if (wid < 2 * RM) {
                const int k = wid % RM;
                double t = 0.0;
                for (int i = (wid / RM) * 32 + lane; i < nm; i += 64) t += ainv[k * nm + i] * gall[i];
                t = warp_sum(t);
                if (lane == 0) co.prod[wid / RM][k] = t;
            }
            __syncthreads();
        }
    };
    // (P y)_i of DOF c of a row
    auto coarse_at = [&](int rl, int c) -> double {
        if constexpr (CO) {
            const double x = xl[3 * rl], y = xl[3 * rl + 1], z = xl[3 * rl + 2];
            const double *a = co.y;
            return c == 0 ? a[0] + z * a[4] - y * a[5]
                          : (c == 1 ? a[1] - z * a[3] + x * a[5] : a[2] + y * a[3] - x * a[4]);
        }
        return 0.0;
    };
    // After a true residual: its coarse sums over the grid, the block's y, then
    // z and the direction's partner on its rows; returns r.z (ok: no wait
    // gave up).
    auto coarse_residual = [&](double w[RM], bool init, bool &ok) -> double {
        double rz = 0.0;
        if constexpr (CO) {
            modes_out(w);
            double none[4] = {0.0, 0.0, 0.0, 0.0};
            ok = rs_sync<1, true>(sh, S.mail, S.ncta, bar, cta, epoch, none, timeout_ns, hold,
                                  [](const double *) {});
            ++epoch;
            if (!ok) return 0.0;
            modes_in();
            if (tid < RM) co.y[tid] = co.prod[0][tid] + co.prod[1][tid];
            __syncthreads();
            for (int i = tid; i < nd; i += RT) {
                const int rl = i / 3;
                const bool fixed = fx && fx[i];
                const T rv = r[i];
                P2 g;
                g.x = fixed ? (T)0 : (T)((double)(dinv[i] * rv) + coarse_at(rl, i - 3 * rl));
                g.y = init ? (T)0 : pair[d0 + i].y;
                pair[d0 + i] = g;
                rz += (double)rv * (double)g.x;
            }
        }
        return rz;
    };
    for (int step = 0; step < max_steps; ++step) {
        double part[4] = {0.0, 0.0, 0.0, 0.0};
        double wm[RM] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        ++epoch;
        bool ok = true;
        if (ph == PH_A) {
            const T beta = (T)sh.st.beta, zeta = (T)sh.st.zeta;
            const int nh = nu * BS;
            for (int i0 = tid; i0 < nh; i0 += 4 * RT) {
                P2 g[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = i0 + k * RT < nh ? i0 + k * RT : i0;
                    const int e = BS == 1 ? i : i / 3;
                    g[k] = __ldcg(pair + (int64_t)BS * list[e] + (BS == 1 ? 0 : i - 3 * e));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i0 + k * RT < nh) halo[hplace(i0 + k * RT)] = zeta * g[k].x + beta * g[k].y;
            }
            __syncthreads();
            double pq = 0.0;
            const int grp = lane >> lsh;
            const bool first = (lane & (L - 1)) == 0;
            for (int s = wid, sn = 2 * RWARPS - 1 - wid; s < nsl; rs_next(s, sn)) {
                const int off = so[s], w = (so[s + 1] - off) >> 5;
                const int pos = s * (32 >> lsh) + grp;
                const int rl = (pos & ~(RS_WINDOW - 1)) + perm[pos];
                const bool valid = rl < nloc;
                const int ri = valid ? rl : 0;
                T pi[BS], acc[BS];
#pragma unroll
                for (int c = 0; c < BS; ++c) {
                    pi[c] = halo[BS * rs_swz(own + ri) + c];
                    acc[c] = 0;
                }
                if constexpr (BS == 1) {
                    const int at = off + SlotGroup<T>::Q * lane;
                    acc[0] = s < nres ? rs_row1<T, DIFF, true, 8>(mc + at, mv + at, w, first, halo, pi[0])
                                      : rs_row1<T, DIFF, false, sizeof(T) == 4 ? 24 : 8>(gc + at, gv + at, w, first, halo, pi[0]);
                } else {
                    if (s < nres)
                        rs_row3<T, DIFF, true>(mc + off + lane, mv + 9 * (size_t)off + lane, w, first,
                                               halo, pi, acc);
                    else
                        rs_row3<T, DIFF, false>(gc + off + lane, gv + 9 * (size_t)off + lane, w, first,
                                                halo, pi, acc);
                }
                for (int o = L >> 1; o > 0; o >>= 1)
#pragma unroll
                    for (int c = 0; c < BS; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
                if (valid && first) {
#pragma unroll
                    for (int c = 0; c < BS; ++c) {
                        q[rl * BS + c] = acc[c];
                        pq += (double)pi[c] * (double)acc[c];
                    }
                    if constexpr (CO) {
                        double v[3];
#pragma unroll
                        for (int c = 0; c < 3; ++c) v[c] = fx && fx[rl * 3 + c] ? 0.0 : (double)acc[c];
                        mode_add(wm, rl, v);
                    }
                }
            }
            part[0] = pq;
            if constexpr (CO) modes_out(wm);
            ok = rs_sync<1, CO>(sh, S.mail, S.ncta, bar, cta, epoch, part, timeout_ns, hold, adv);
            if (CO && ok && sh.st.phase == PH_B) {   // y follows the residual
                modes_in();
                if constexpr (CO)
                    if (tid < RM) co.y[tid] -= sh.st.alpha * (co.prod[0][tid] + co.prod[1][tid]);
                __syncthreads();
            }
        } else if (ph == PH_B) {
            const double alpha64 = sh.st.alpha;
            const T alpha = (T)alpha64;
            double rz = 0.0, rr = 0.0;
            double *x = S.x + d0;
            // (all loads of four rows first: one at a time, a block of 10,600
            // rows with its vectors in global memory took 20 us, now 7)
            for (int i0 = tid; i0 < nd; i0 += 4 * RT) {
                double xv[4];
                T pi[4], rv[4], qv[4], dv[4];
                bool fixed[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = i0 + k * RT < nd ? i0 + k * RT : i0;
                    fixed[k] = fx && fx[i];
                    xv[k] = x[i];
                    rv[k] = r[i];
                    qv[k] = q[i];
                    dv[k] = dinv[i];
                    pi[k] = halo[hplace(BS * own + i)];
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = i0 + k * RT;
                    if (i >= nd) break;
                    if (!fixed[k]) {
                        x[i] = xv[k] + alpha64 * (double)pi[k];
                        rv[k] -= alpha * qv[k];
                        r[i] = rv[k];
                    }
                    T zv = dv[k] * rv[k];
                    if constexpr (CO) zv = (T)((double)zv + coarse_at(i / 3, i % 3));
                    if (fixed[k]) zv = (T)0;
                    P2 g;
                    g.x = zv;
                    g.y = pi[k];
                    pair[d0 + i] = g;
                    rz += (double)rv[k] * (double)zv;
                    rr += (double)rv[k] * (double)rv[k];
                }
            }
            part[0] = rz;
            part[1] = rr;
            ok = rs_sync<2, true>(sh, S.mail, S.ncta, bar, cta, epoch, part, timeout_ns, hold, adv);
        } else if (ph == PH_R && sizeof(T) == 8) {
            // FP64 true residual from the slices, x in the halo's place
            double *hx = (double *)halo;
            const int nh = nu * BS;
            for (int i0 = tid; i0 < nh; i0 += 4 * RT) {
                double g[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = i0 + k * RT < nh ? i0 + k * RT : i0;
                    const int e = BS == 1 ? i : i / 3;
                    g[k] = __ldcg(S.x + (int64_t)BS * list[e] + (BS == 1 ? 0 : i - 3 * e));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i0 + k * RT < nh) hx[hplace(i0 + k * RT)] = g[k];
            }
            __syncthreads();
            double rr = 0.0, rp = 0.0, rz = 0.0, aa = 0.0;
            const int grp = lane >> lsh;
            const bool first = (lane & (L - 1)) == 0;
            for (int s = wid, sn = 2 * RWARPS - 1 - wid; s < nsl; rs_next(s, sn)) {
                const int off = so[s], w = (so[s + 1] - off) >> 5;
                const int pos = s * (32 >> lsh) + grp;
                const int rl = (pos & ~(RS_WINDOW - 1)) + perm[pos];
                double hi[BS], lo[BS], ab[BS];
#pragma unroll
                for (int c = 0; c < BS; ++c) hi[c] = lo[c] = ab[c] = 0.0;
                if constexpr (BS == 1) {
                    const int at = off + lane;
                    if (s < nres) rs_row_dd1<true>(mc + at, (const double *)mv + at, w, hx, hi[0], lo[0], ab[0]);
                    else rs_row_dd1<false>(gc + at, (const double *)gv + at, w, hx, hi[0], lo[0], ab[0]);
                } else {
                    const size_t at = 9 * (size_t)off + lane;
                    if (s < nres) rs_row_dd3<true>(mc + off + lane, (const double *)mv + at, w, hx, hi, lo, ab);
                    else rs_row_dd3<false>(gc + off + lane, (const double *)gv + at, w, hx, hi, lo, ab);
                }
                for (int o = L >> 1; o > 0; o >>= 1)
#pragma unroll
                    for (int c = 0; c < BS; ++c) {
                        const double h2 = __shfl_xor_sync(0xffffffffu, hi[c], o);
                        const double l2 = __shfl_xor_sync(0xffffffffu, lo[c], o);
                        dd_add(hi[c], lo[c], h2, l2);
                        ab[c] += __shfl_xor_sync(0xffffffffu, ab[c], o);
                    }
                if (rl < nloc && first) {
#pragma unroll
                    for (int c = 0; c < BS; ++c) {
                        const int i = rl * BS + c;
                        const bool fixed = fx && fx[i];
                        const double rt = fixed ? 0.0 : dd_residual(__ldg(S.b + d0 + i), hi[c], lo[c]);
                        rr += rt * rt;
                        if (!fixed) aa += ab[c] * ab[c];
                        const T rv = (T)rt;
                        r[i] = rv;
                        P2 g = pair[d0 + i];
                        rp += (double)rv * (double)g.y;
                        if (!CO) {
                            g.x = fixed ? (T)0 : dinv[i] * rv;
                            pair[d0 + i] = g;
                            rz += (double)rv * (double)g.x;
                        }
                    }
                    if constexpr (CO) {
                        const double v[3] = {(double)r[3 * rl], (double)r[3 * rl + 1], (double)r[3 * rl + 2]};
                        mode_add(wm, rl, v);
                    }
                }
            }
            if constexpr (CO) {
                rz = coarse_residual(wm, false, ok);
                if (!ok) return;
            }
            part[0] = rr;
            part[1] = rp;
            part[2] = rz;
            part[3] = aa;
            ok = rs_sync<4, true>(sh, S.mail, S.ncta, bar, cta, epoch, part, timeout_ns, hold, adv);
        } else if (ph == PH_INIT || ph == PH_R) {
            // FP64 true residual from the FP64 CSR, 8 lanes per row
            // (compensated sums); INIT also the Jacobi inverse and |b_lift|
            const bool init = ph == PH_INIT;
            const int sub = lane & (LANES - 1), grp = lane / LANES;
            double rr = 0.0, s1 = 0.0, rz = 0.0, aa = 0.0;
            bool bad = false;
            // Scalar rows: a row's bounds are loaded a pass ahead, and what follows
            // its sum before the sum (a time step of the 40 x 36 x 33 P1 box 190 -> 178
            // us); 3x3 rows have no registers left
            // for it (residuals of the Tet10 box of 27 x 15 x 13 cells 85 -> 125 us)
            constexpr bool AHEAD = BS == 1;
            int32_t kn = 0, kn1 = 0;
            if (AHEAD && wid * RPP + grp < nloc) {
                kn = __ldg(S.rp + r0 + wid * RPP + grp);
                kn1 = __ldg(S.rp + r0 + wid * RPP + grp + 1);
            }
            for (int base = wid * RPP; base < nloc; base += RWARPS * RPP) {
                const int rl = base + grp;
                const bool valid = rl < nloc;
                const int64_t row = r0 + (valid ? rl : 0);
                const int32_t k0 = AHEAD ? kn : __ldg(S.rp + row), k1 = AHEAD ? kn1 : __ldg(S.rp + row + 1);
                if (AHEAD && rl + RWARPS * RPP < nloc) {
                    kn = __ldg(S.rp + row + RWARPS * RPP);
                    kn1 = __ldg(S.rp + row + RWARPS * RPP + 1);
                }
                double b1 = 0.0;
                T py1 = (T)0;
                if (AHEAD && valid && sub == 0) {
                    b1 = __ldg(S.b + d0 + rl);
                    if (!init) py1 = pair[d0 + rl].y;
                }
                double acc[BS], alo[BS], accf[BS], aab[BS], dg[B2];
#pragma unroll
                for (int c = 0; c < BS; ++c) acc[c] = alo[c] = accf[c] = aab[c] = 0.0;
#pragma unroll
                for (int c = 0; c < B2; ++c) dg[c] = 0.0;
                if (valid) {
                    if (init) rs_row_R<true, BS>(S, k0 + sub, k1, row, acc, alo, aab, accf, dg);
                    else rs_row_R<false, BS>(S, k0 + sub, k1, row, acc, alo, aab, accf, dg);
                }
#pragma unroll
                for (int c = 0; c < BS; ++c) {
                    group_sum_dd<LANES>(acc[c], alo[c]);
                    aab[c] = group_sum<LANES>(aab[c]);
                    if (init) {
                        accf[c] = group_sum<LANES>(accf[c]);
                        dg[c * BS + c] = group_sum<LANES>(dg[c * BS + c]);
                    }
                }
                if (valid && sub == 0) {
#pragma unroll
                    for (int c = 0; c < BS; ++c) {
                        const int i = rl * BS + c;
                        const bool fixed = fx && fx[i];
                        const double bi = AHEAD ? b1 : __ldg(S.b + d0 + i);
                        const double rt = fixed ? 0.0 : dd_residual(bi, acc[c], alo[c]);
                        rr += rt * rt;
                        if (!fixed) aa += aab[c] * aab[c];
                        const T rv = (T)rt;
                        r[i] = rv;
                        T dv;
                        if (init) {
                            double iv = 0.0;
                            if (!fixed) {
                                const double d = dg[c * BS + c];
                                const double bl = bi - accf[c];
                                s1 += bl * bl;
                                if (!(d > 0.0) || !isfinite(d)) bad = true;
                                else iv = 1.0 / d;
                            }
                            dv = (T)iv;
                            dinv[i] = dv;
                        } else {
                            dv = dinv[i];
                        }
                        P2 g;
                        g.y = init ? (T)0 : (AHEAD ? py1 : pair[d0 + i].y);
                        if (!init) s1 += (double)rv * (double)g.y;
                        if (!CO) {
                            g.x = fixed ? (T)0 : dv * rv;
                            rz += (double)rv * (double)g.x;
                            pair[d0 + i] = g;
                        }
                    }
                    if constexpr (CO) {
                        const double v[3] = {(double)r[3 * rl], (double)r[3 * rl + 1], (double)r[3 * rl + 2]};
                        mode_add(wm, rl, v);
                    }
                }
            }
            if constexpr (CO) {
                rz = coarse_residual(wm, init, ok);
                if (!ok) return;
            }
            part[0] = rr;
            part[1] = s1;
            part[2] = rz;
            part[3] = bad ? -INFINITY : aa;
            ok = rs_sync<4, true>(sh, S.mail, S.ncta, bar, cta, epoch, part, timeout_ns, hold, adv);
        } else {                              // zero right-hand side
            for (int i = tid; i < nd; i += RT)
                if (!(fx && fx[i])) S.x[d0 + i] = 0.0;
            ok = rs_sync<1, false>(sh, S.mail, S.ncta, bar, cta, epoch, part, timeout_ns, hold, adv);
        }
        if (!ok) return;
        ph = sh.st.phase;
        // (the update phase needs the product phase's vectors: not between)
        if (ph == PH_DONE || (ph != PH_B && sh.st.iter - iter0 >= max_iters)) break;
    }
    if (keep && S.vsm && ph != PH_DONE)
        for (int i = tid; i < nd; i += RT) {
            ((T *)S.r)[d0 + i] = r[i];
            ((T *)S.dinv)[d0 + i] = dinv[i];
        }
    if (cta == 0 && tid == 0) {
        sh.st.pad = (int32_t)epoch;
        gst[place.x] = sh.st;
    }
}

// ------------------------------------------------------------------ set-up
// A block's columns as a bitmap over the system's rows in shared memory:
// marked from the block's rows (and the rows themselves: an absent diagonal
// still takes slot 0), counted, and ranked by 4-word groups.
__host__ __device__ inline int rs_words(int64_t n) { return (int)((n + 127) / 128) * 4; }

__device__ __forceinline__ void rs_mark(const SysDev &S, int64_t r0, int nloc, uint32_t *bits,
                                        int *len) {
    const int lane = threadIdx.x & 31, sub = lane & 7, wid = threadIdx.x >> 5;
    for (int base = wid * 4; base < nloc; base += RWARPS * 4) {
        const int i = base + (lane >> 3);
        const bool valid = i < nloc;
        const int64_t row = r0 + i;
        const int32_t kb = valid ? __ldg(S.rp + row) : 0, ke = valid ? __ldg(S.rp + row + 1) : 0;
        int diag = 0;
        for (int32_t k = kb + sub; k < ke; k += 8) {
            const int32_t c = __ldg(S.ci + k);
            diag |= c == (int32_t)row;
            if ((uint32_t)c < (uint32_t)S.n) atomicOr(bits + (c >> 5), 1u << (c & 31));
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) diag |= __shfl_xor_sync(0xffffffffu, diag, o);
        if (valid && sub == 0) {
            atomicOr(bits + (row >> 5), 1u << (row & 31));
            if (len) len[i] = ke - kb + (diag ? 0 : 1);
        }
    }
}

// The blocks' rows: bounds of equal work, a row counting its stored entries
// and `alpha` more (its share of the update and of the halo). With equal
// rows instead the blocks that hold a Tet10 mesh's vertex rows (65 entries
// against 28 on average, and numbered first) had twice the others' work.
__global__ void k_rs_split(const SysDev *__restrict__ sys, RsCta *ctas, int n, int alpha) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const SysDev &S = sys[ctas[i].sys];
    const int c = ctas[i].cta;
    const int64_t first = __ldg(S.rp), total = __ldg(S.rp + S.n) - first + (int64_t)alpha * S.n;
    auto bound = [&](int k) {   // first row with k / ncta of the work before it
        const int64_t want = total * k / S.ncta;
        int64_t lo = 0, hi = S.n;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (__ldg(S.rp + mid) - first + alpha * mid < want) lo = mid + 1; else hi = mid;
        }
        return (int32_t)lo;
    };
    const int32_t r0 = bound(c), r1 = c + 1 == S.ncta ? (int32_t)S.n : bound(c + 1);
    ctas[i].row0 = r0;
    ctas[i].rows = r1 - r0;
    // ceil(rows / RS) slices fit before the next block's first
    ctas[i].sl0 = S.sl0 + (r0 >> (5 - S.lsh)) + c;
}

// Row order, slice sizes and halo size of every block: windows of RS_WINDOW
// rows (the last one shorter) sorted by stored length, longest first, ties
// in row order; a slice is 32 / L positions, its size 32 x its longest
// row's slots rounded up to whole steps of L and whole groups of q.
__global__ void __launch_bounds__(RT)
k_rs_rank(const SysDev *__restrict__ sys, const RsCta *__restrict__ ctas, int64_t *sizes_all,
          int2 *ucnt, int q) {
    extern __shared__ __align__(16) uint32_t rs_bits[];
    __shared__ int total;
    const RsCta me = ctas[blockIdx.x];
    const SysDev &S = sys[me.sys];
    const int nw = rs_words(S.n), t = threadIdx.x, lsh = S.lsh, L = 1 << lsh, rs = 32 >> lsh;
    const int npos = rs_slices(me.rows, lsh) * rs;   // positions: the rows, then padding
    int *len = (int *)(rs_bits + nw);
    for (int i = t; i < nw; i += RT) rs_bits[i] = 0;
    for (int i = t; i < npos; i += RT) len[i] = 0;
    if (t == 0) total = 0;
    __syncthreads();
    rs_mark(S, me.row0, me.rows, rs_bits, len);
    __syncthreads();
    int cnt = 0;
    for (int i = t; i < nw; i += RT) cnt += __popc(rs_bits[i]);
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((t & 31) == 0) atomicAdd(&total, cnt);
    uint8_t *perm = (uint8_t *)S.sperm + me.sl0 * 32;
    for (int i = t; i < npos; i += RT) {
        const int w0 = i & ~(RS_WINDOW - 1), w1 = min(npos, w0 + RS_WINDOW);
        const int Li = len[i];
        int rank = 0;
        for (int u = w0; u < w1; ++u) rank += (len[u] > Li || (len[u] == Li && u < i)) ? 1 : 0;
        perm[w0 + rank] = (uint8_t)(i - w0);
        if (rank % rs == 0) sizes_all[me.sl0 + (w0 + rank) / rs] = 32 * (int64_t)((((Li + L - 1) >> lsh) + q - 1) / q * q);
    }
    __syncthreads();
    if (t == 0) ucnt[blockIdx.x] = make_int2(total, me.rows);
}

// Slot k of a row of `len` entries with its diagonal at dpos (INT_MAX: none):
// the entry there, or -1 (padding, or an absent diagonal).
__device__ __forceinline__ int rs_entry(int k, int len, int dpos) {
    const int e = k == 0 ? (dpos == INT32_MAX ? -1 : dpos) : (k - 1 < dpos ? k - 1 : k);
    return e < len ? e : -1;
}
__device__ __forceinline__ int rs_dpos(const int32_t *ci, int32_t kb, int len, int32_t row, int u, int L) {
    int dpos = INT32_MAX;
    for (int k = u; k < len; k += L)
        if (__ldg(ci + kb + k) == row) {
            dpos = k;
            break;
        }
    for (int o = L >> 1; o > 0; o >>= 1) dpos = min(dpos, __shfl_xor_sync(0xffffffffu, dpos, o));
    return dpos;
}

// Every block's halo list and the slices' local columns (places in that
// list). A row repeated in the CSR keeps its repeats as entries.
__global__ void __launch_bounds__(RT)
k_rs_cols(const SysDev *__restrict__ sys, const RsCta *__restrict__ ctas,
          uint16_t *__restrict__ scol, int q) {
    extern __shared__ __align__(16) uint32_t rs_bits[];
    __shared__ int wsum[RWARPS];
    const RsCta me = ctas[blockIdx.x];
    const SysDev &S = sys[me.sys];
    const int nw = rs_words(S.n), ng = nw / 4, t = threadIdx.x;
    const int lane = t & 31, wid = t >> 5;
    int *pre = (int *)(rs_bits + nw);
    for (int i = t; i < nw; i += RT) rs_bits[i] = 0;
    __syncthreads();
    const int64_t r0 = me.row0;
    rs_mark(S, r0, me.rows, rs_bits, nullptr);
    __syncthreads();
    // exclusive prefix of the groups' counts, one run of groups per thread
    const int per = (ng + RT - 1) / RT, g0 = min(ng, t * per), g1 = min(ng, g0 + per);
    int sum = 0;
    for (int g = g0; g < g1; ++g)
        for (int j = 0; j < 4; ++j) sum += __popc(rs_bits[4 * g + j]);
    int inc = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    int base = inc - sum;
    for (int k = 0; k < wid; ++k) base += wsum[k];
    int32_t *list = (int32_t *)S.ulist + (size_t)me.cta * S.umax;
    for (int g = g0; g < g1; ++g) {
        pre[g] = base;
        for (int j = 0; j < 4; ++j) {
            uint32_t m = rs_bits[4 * g + j];
            while (m) {
                const int b = __ffs(m) - 1;
                list[base++] = 32 * (4 * g + j) + b;
                m &= m - 1;
            }
        }
    }
    __syncthreads();
    const int lsh = S.lsh, L = 1 << lsh, rs = 32 >> lsh, u = lane & (L - 1);
    auto place = [&](int32_t c) {
        if ((uint32_t)c >= (uint32_t)S.n) return (uint16_t)rs_swz(0);   // not a column of this matrix
        const int w = c >> 5, g = w >> 2;
        int v = pre[g];
        for (int j = 4 * g; j < w; ++j) v += __popc(rs_bits[j]);
        return (uint16_t)rs_swz(v + __popc(rs_bits[w] & ((1u << (c & 31)) - 1u)));
    };
    const uint8_t *perm = S.sperm + me.sl0 * 32;
    for (int s = wid; s < rs_slices(me.rows, lsh); s += RWARPS) {
        const int64_t off = __ldg(S.soff + me.sl0 + s);
        const int w = (int)((__ldg(S.soff + me.sl0 + s + 1) - off) >> 5);
        if (w == 0) continue;
        const int pos = s * rs + (lane >> lsh);
        const int rl = (pos & ~(RS_WINDOW - 1)) + __ldg(perm + pos);
        const int64_t row = r0 + rl;
        const bool valid = rl < me.rows;
        const int32_t kb = valid ? __ldg(S.rp + row) : 0, len = valid ? __ldg(S.rp + row + 1) - kb : 0;
        const int dpos = rs_dpos(S.ci, kb, len, (int32_t)row, u, L);
        const uint16_t own = place((int32_t)(valid ? row : r0));
        for (int k = 0; k < w; ++k) {
            const int e = rs_entry(k * L + u, len, dpos);
            scol[off + rs_slot(k, lane, q)] = e >= 0 ? place(__ldg(S.ci + kb + e)) : own;
        }
    }
}

// The slices' values from the CSR, one warp per slice: the diagonal (0 if
// the pattern has none) in slot 0, the row's other entries in order, 0 as
// padding. Run again when the values change.
template <typename T, int BS>
__global__ void __launch_bounds__(256)
k_rs_vals(const SysDev *__restrict__ sys, const RsCta *__restrict__ ctas, T *__restrict__ sval, int q) {
    constexpr int B2 = BS * BS;
    const RsCta me = ctas[blockIdx.x];
    const SysDev &S = sys[me.sys];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwp = blockDim.x >> 5;
    const int lsh = S.lsh, L = 1 << lsh, rs = 32 >> lsh, u = lane & (L - 1);
    const T *v = MatVal<T>::get(S);
    const int64_t r0 = me.row0;
    const uint8_t *perm = S.sperm + me.sl0 * 32;
    for (int s = blockIdx.y * nwp + wid; s < rs_slices(me.rows, lsh); s += gridDim.y * nwp) {
        const int64_t off = __ldg(S.soff + me.sl0 + s);
        const int w = (int)((__ldg(S.soff + me.sl0 + s + 1) - off) >> 5);
        if (w == 0) continue;
        const int pos = s * rs + (lane >> lsh);
        const int rl = (pos & ~(RS_WINDOW - 1)) + __ldg(perm + pos);
        const int64_t row = r0 + rl;
        const bool valid = rl < me.rows;
        const int32_t kb = valid ? __ldg(S.rp + row) : 0, len = valid ? __ldg(S.rp + row + 1) - kb : 0;
        const int dpos = rs_dpos(S.ci, kb, len, (int32_t)row, u, L);
        for (int k = 0; k < w; ++k) {
            const int e = rs_entry(k * L + u, len, dpos);
            T *dst = BS == 1 ? sval + off + rs_slot(k, lane, q) : sval + B2 * (off + 32 * (int64_t)k) + lane;
#pragma unroll
            for (int c = 0; c < B2; ++c)
                dst[32 * c] = e >= 0 ? __ldg(v + ((int64_t)kb + e) * B2 + c) : T{};
        }
    }
}
