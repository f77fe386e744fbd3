// Coarse correction of the resident CG for elasticity (3x3 systems whose
// block rows are mesh nodes with known coordinates). Included by
// cfem_solve.cu after cfem_resident.cuh, whose kernel applies it.
//
// Point Jacobi needs thousands of iterations on a bending part: it cannot see
// the rigid motions of large pieces. The nodes are put in Morton order, so a
// block's rows are a compact piece of the part, and the six rigid-body modes
// of every piece (fixed DOFs set to zero) span a coarse space P. The
// preconditioner is
//     z = D^-1 r + P (P^T A P)^-1 P^T r,
// the additive two-level method (Bramble, Pasciak, Schatz 1986; rigid-body
// aggregates: Vanek, Mandel, Brezina 1996, without smoothing). With one piece
// per block it adds no grid-wide sum to an iteration: P^T q is six sums per
// block that travel with p.q, every block keeps its own six rows of the
// coarse inverse in shared memory, and its coefficients y = (P^T A P)^-1 P^T r
// follow r -= alpha q as y -= alpha (P^T A P)^-1 P^T q; every true-residual
// replacement computes them anew.
//
// Measured, iterations and time of a whole solve call, plain -> with it: Tet10
// cantilever of 40 x 5 x 5 cells in FP64 1,740 -> 191, 23.7 -> 5.2 ms; Tet10 box
// of 27 x 15 x 13 in mixed precision 1,814 -> 268, 39 -> 13.1 ms; P1 box of 31 x
// 17 x 14 in FP64 763 -> 176, 9.2 -> 5.0 ms. An iteration costs 15 us instead of
// 10.7 on the first: the six sums and their way through memory.
//
// Set-up, in this file: Morton order (cfem_order.cuh copies the system), the
// pieces' geometry, P^T A P by blocks of 6 x 6, and its inverse.

constexpr int RC_NB = 40;            // neighbour pieces accumulated at a time

// Bounding box of the nodes: doubles mapped to ordered integers, so that the
// atomics' result does not depend on their order.
__device__ __forceinline__ unsigned long long rc_key(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b >> 63 ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double rc_val(unsigned long long k) {
    return __longlong_as_double((long long)(k >> 63 ? k & 0x7fffffffffffffffull : ~k));
}
__global__ void k_rc_box(const double *__restrict__ nodes, int64_t n, unsigned long long *lo,
                         unsigned long long *hi) {
    unsigned long long a[3] = {~0ull, ~0ull, ~0ull}, b[3] = {0, 0, 0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const unsigned long long k = rc_key(nodes[3 * i + d]);
            a[d] = k < a[d] ? k : a[d];
            b[d] = k > b[d] ? k : b[d];
        }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long a2 = __shfl_xor_sync(0xffffffffu, a[d], o);
            const unsigned long long b2 = __shfl_xor_sync(0xffffffffu, b[d], o);
            a[d] = a2 < a[d] ? a2 : a[d];
            b[d] = b2 > b[d] ? b2 : b[d];
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(lo + d, a[d]);
            atomicMax(hi + d, b[d]);
        }
    }
}

__device__ __forceinline__ uint32_t rc_spread(uint32_t v) {   // 10 bits, two zeros between
    v &= 1023u;
    v = (v | v << 16) & 0x030000ffu;
    v = (v | v << 8) & 0x0300f00fu;
    v = (v | v << 4) & 0x030c30c3u;
    return (v | v << 2) & 0x09249249u;
}
// Morton keys on a grid of cubic cells, 1024 along the longest edge.
__global__ void k_rc_morton(const double *__restrict__ nodes, int64_t n,
                            const unsigned long long *__restrict__ lo,
                            const unsigned long long *__restrict__ hi, unsigned long long *__restrict__ key,
                            int32_t *__restrict__ id) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double ext = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) ext = fmax(ext, rc_val(hi[d]) - rc_val(lo[d]));
    const double sc = ext > 0.0 ? 1023.0 / ext : 0.0;
    uint32_t k = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double t = (nodes[3 * i + d] - rc_val(lo[d])) * sc;
        const uint32_t c = t > 0.0 ? (t < 1023.0 ? (uint32_t)t : 1023u) : 0u;
        k |= rc_spread(c) << d;
    }
    key[i] = k;
    id[i] = (int32_t)i;
}

// Coordinates of every block's nodes from their mean, in units of the piece's
// size, and every node's block.
__global__ void __launch_bounds__(256)
k_rc_geo(const RsCta *__restrict__ ctas, const double *__restrict__ nodes,
         const int32_t *__restrict__ ord, float *__restrict__ xl, uint8_t *__restrict__ own) {
    __shared__ double red[8][3];
    __shared__ double mean[3], size;
    const RsCta me = ctas[blockIdx.x];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    double s[3] = {0.0, 0.0, 0.0};
    for (int i = t; i < me.rows; i += 256) {
        const int64_t o = ord[me.row0 + i];
#pragma unroll
        for (int d = 0; d < 3; ++d) s[d] += nodes[3 * o + d];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        s[d] = warp_sum(s[d]);
        if (lane == 0) red[w][d] = s[d];
    }
    __syncthreads();
    if (t < 3) {
        double m = 0.0;
        for (int k = 0; k < 8; ++k) m += red[k][t];
        mean[t] = me.rows ? m / me.rows : 0.0;
    }
    __syncthreads();
    double h = 0.0;
    for (int i = t; i < me.rows; i += 256) {
        const int64_t o = ord[me.row0 + i];
#pragma unroll
        for (int d = 0; d < 3; ++d) h = fmax(h, fabs(nodes[3 * o + d] - mean[d]));
    }
    for (int o = 16; o > 0; o >>= 1) h = fmax(h, __shfl_xor_sync(0xffffffffu, h, o));
    if (lane == 0) red[w][0] = h;
    __syncthreads();
    if (t == 0) {
        for (int k = 0; k < 8; ++k) h = fmax(h, red[k][0]);
        size = h > 0.0 ? h : 1.0;
    }
    __syncthreads();
    for (int i = t; i < me.rows; i += 256) {
        const int64_t o = ord[me.row0 + i];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            xl[3 * ((int64_t)me.row0 + i) + d] = (float)((nodes[3 * o + d] - mean[d]) / size);
        own[me.row0 + i] = (uint8_t)me.cta;
    }
}

// Mode p of a node at (x, y, z) from its piece's mean: three translations, then
// the rotations about the axes.
__device__ __forceinline__ void rc_mode(int p, double x, double y, double z, double m[3]) {
    m[0] = p == 0 ? 1.0 : (p == 4 ? z : (p == 5 ? -y : 0.0));
    m[1] = p == 1 ? 1.0 : (p == 3 ? -z : (p == 5 ? x : 0.0));
    m[2] = p == 2 ? 1.0 : (p == 3 ? y : (p == 4 ? -x : 0.0));
}

// The block row of P^T A P that belongs to piece blockIdx.x. A warp walks its
// rows' entries one at a time, its lanes holding the 36 values of a 6 x 6
// block (the last four lanes two each), into accumulators of its own; the
// warps' sums are added in warp order, so the result is the same every time.
constexpr int RC_WARPS = 16;
__global__ void __launch_bounds__(32 * RC_WARPS)
k_rc_ac(const SysDev *__restrict__ sys, const float *__restrict__ xl, const uint8_t *__restrict__ own,
        double *__restrict__ ac) {
    extern __shared__ __align__(16) double rc_acc[];      // [RC_WARPS][RC_NB][36]
    __shared__ int slot[RS_MAX_CTAS], nbr[RS_MAX_CTAS], count;
    const SysDev &S = *sys;
    const RsCta me = S.ctas[blockIdx.x];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, nm = RM * S.ncta;
    for (int i = t; i < RS_MAX_CTAS; i += 32 * RC_WARPS) slot[i] = 0;
    __syncthreads();
    for (int i = w; i < me.rows; i += RC_WARPS) {
        const int64_t row = (int64_t)me.row0 + i;
        for (int32_t k = __ldg(S.rp + row) + lane; k < __ldg(S.rp + row + 1); k += 32)
            slot[__ldg(own + __ldg(S.ci + k))] = 1;
    }
    __syncthreads();
    if (t == 0) {
        count = 0;
        for (int b = 0; b < S.ncta; ++b) {
            if (slot[b]) nbr[count] = b;
            slot[b] = slot[b] ? count++ : -1;
        }
    }
    __syncthreads();
    const int p0 = lane / 6, q0 = lane % 6, p1 = (lane + 32) / 6, q1 = (lane + 32) % 6;
    const bool two = lane < 4;                            // values lane and lane + 32
    for (int first = 0; first < count; first += RC_NB) {
        const int nb = min(RC_NB, count - first);
        double *acc = rc_acc + (size_t)w * RC_NB * 36;
        for (int i = lane; i < nb * 36; i += 32) acc[i] = 0.0;
        __syncwarp();
        for (int i = w; i < me.rows; i += RC_WARPS) {
            const int64_t row = (int64_t)me.row0 + i;
            double rp0[3], rp1[3];
            const float *xi = xl + 3 * row;
            rc_mode(p0, xi[0], xi[1], xi[2], rp0);
            rc_mode(two ? p1 : 0, xi[0], xi[1], xi[2], rp1);
#pragma unroll
            for (int d = 0; d < 3; ++d)
                if (S.fixed && __ldg(S.fixed + 3 * row + d)) rp0[d] = rp1[d] = 0.0;
            const int32_t k1 = __ldg(S.rp + row + 1);
            for (int32_t k = __ldg(S.rp + row); k < k1; ++k) {
                const int64_t j = __ldg(S.ci + k);
                const int b = slot[__ldg(own + j)] - first;
                if (b < 0 || b >= nb) continue;           // uniform over the warp
                const float *xj = xl + 3 * j;
                const double x = xj[0], y = xj[1], z = xj[2];
                double a[9], c0[3], c1[3];
#pragma unroll
                for (int e = 0; e < 9; ++e) a[e] = __ldg(S.v64 + 9 * (int64_t)k + e);
                rc_mode(q0, x, y, z, c0);
                rc_mode(two ? q1 : 0, x, y, z, c1);
                double s0 = 0.0, s1 = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    if (S.fixed && __ldg(S.fixed + 3 * j + d)) continue;
                    s0 += (rp0[0] * a[d] + rp0[1] * a[3 + d] + rp0[2] * a[6 + d]) * c0[d];
                    s1 += (rp1[0] * a[d] + rp1[1] * a[3 + d] + rp1[2] * a[6 + d]) * c1[d];
                }
                acc[b * 36 + lane] += s0;
                if (two) acc[b * 36 + 32 + lane] += s1;
            }
        }
        __syncthreads();
        for (int i = t; i < nb * 36; i += 32 * RC_WARPS) {
            double s = 0.0;
            for (int v = 0; v < RC_WARPS; ++v) s += rc_acc[(size_t)v * RC_NB * 36 + i];
            const int b = nbr[first + i / 36], e = i % 36;
            ac[(size_t)(RM * blockIdx.x + e / 6) * nm + RM * b + e % 6] = s;
        }
        __syncthreads();
    }
}

// Inverse of the SPD matrix ac (nm x nm) by block Gauss-Jordan without
// pivoting, block k the six rows of piece k held by its block in shared
// memory. Step k needs only row block k: its owner scales and publishes it
// with a flag, the others wait for the flag, read it and update their rows. A
// pivot that has all but vanished (a mode that others span: a piece of
// nodes on a line, or all its DOFs fixed) leaves its unknown out: zero row and
// column. Waits are bounded; on expiry *err is set and every block returns.
__global__ void __launch_bounds__(RT, 1)
k_rc_inv(const double *__restrict__ ac, int nblk, double *rowbuf, unsigned *flag, double *__restrict__ out,
         int *err, unsigned long long timeout_ns) {
    extern __shared__ __align__(16) double rc_rows[];     // the block's own rows
    __shared__ double D[RM][RM], F[RM][RM], d0[RM];
    __shared__ int quit;
    const int t = threadIdx.x, lane = t & 31, me = blockIdx.x, nm = RM * nblk;
    double *mine = rc_rows;
    for (int i = t; i < RM * nm; i += RT) mine[i] = ac[(size_t)RM * me * nm + i];
    if (t == 0) quit = 0;
    __syncthreads();
    if (t < RM) d0[t] = mine[t * nm + RM * me + t];
    __syncthreads();
    for (int k = 0; k < nblk; ++k) {
        if (k == me) {
            if (t < 32) {                                  // D^-1, entries lane and lane + 32
                for (int e = lane; e < RM * RM; e += 32) D[e / RM][e % RM] = mine[(e / RM) * nm + RM * k + e % RM];
                __syncwarp();
                for (int p = 0; p < RM; ++p) {
                    const double d = D[p][p];
                    const bool take = d > 1e-10 * d0[p] && d0[p] > 0.0;
                    const double iv = take ? 1.0 / d : 0.0;
                    double v[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int e = lane + 32 * u;
                        if (e >= RM * RM) continue;
                        const int i = e / RM, j = e % RM;
                        if (i == p && j == p) v[u] = iv;
                        else if (i == p) v[u] = D[p][j] * iv;
                        else if (j == p) v[u] = -D[i][p] * iv;
                        else v[u] = D[i][j] - D[i][p] * D[p][j] * iv;
                    }
                    __syncwarp();
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (lane + 32 * u < RM * RM) D[(lane + 32 * u) / RM][(lane + 32 * u) % RM] = v[u];
                    __syncwarp();
                }
            }
            __syncthreads();
            for (int j = t; j < nm; j += RT) {
                double c[RM], r[RM];
#pragma unroll
                for (int i = 0; i < RM; ++i) c[i] = mine[i * nm + j];
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    r[i] = 0.0;
#pragma unroll
                    for (int p = 0; p < RM; ++p) r[i] += D[i][p] * c[p];
                }
                const bool diag = j / RM == k;
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    const double v = diag ? D[i][j - RM * k] : r[i];
                    mine[i * nm + j] = v;
                    rowbuf[(size_t)(RM * k + i) * nm + j] = v;
                }
            }
            __syncthreads();
            if (t == 0) {
                fence_gpu();
                for (int c = 0; c < RS_COPIES; ++c)
                    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(flag + c * nblk + k), "r"(1u) : "memory");
            }
        } else {
            if (t == 0) {
                const unsigned *f = flag + (me % RS_COPIES) * nblk + k;
                unsigned long long t0 = 0;
                for (unsigned spin = 0; ld_acquire(f) == 0; ++spin)
                    if ((spin & 63u) == 63u) {
                        const unsigned long long now = globaltimer();
                        if (t0 == 0) t0 = now;
                        if (now - t0 > timeout_ns) atomicExch(err, 1);
                        if (*(volatile int *)err) {
                            quit = 1;
                            break;
                        }
                    }
            }
            if (t >= 32 && t < 32 + RM * RM) F[(t - 32) / RM][(t - 32) % RM] = mine[((t - 32) / RM) * nm + RM * k + (t - 32) % RM];
            __syncthreads();
            if (quit) return;
            for (int j = t; j < nm; j += RT) {
                double r[RM];
#pragma unroll
                for (int p = 0; p < RM; ++p) r[p] = __ldcg(rowbuf + (size_t)(RM * k + p) * nm + j);
                const bool diag = j / RM == k;
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    double v = diag ? 0.0 : mine[i * nm + j];
#pragma unroll
                    for (int p = 0; p < RM; ++p) v -= F[i][p] * r[p];
                    mine[i * nm + j] = v;
                }
            }
            __syncthreads();
        }
    }
    for (int i = t; i < RM * nm; i += RT) out[(size_t)RM * me * nm + i] = mine[i];
}
