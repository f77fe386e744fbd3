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
// cantilever of 40 x 5 x 5 cells in FP64 1,740 -> 191, 23.7 -> 5.0 ms; Tet10 box
// of 27 x 15 x 13 in mixed precision 1,814 -> 268, 39 -> 11.0 ms; P1 box of 31 x
// 17 x 14 in FP64 763 -> 176, 9.2 -> 4.8 ms. An iteration costs 15 us instead of
// 10.7 on the first: the six sums and their way through memory.
//
// Set-up, in this file: Morton order (cfem_order.cuh copies the system), the
// pieces' geometry, P^T A P by blocks of 6 x 6, and its inverse.

constexpr int RC_NB = 40;            // neighbour pieces accumulated at a time
constexpr int RC_MIN_ITER = 1000;    // iterations a corrected solve may take at least

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

// The block row of P^T A P that belongs to piece blockIdx.x. A warp takes its
// rows' entries 32 at a time: each lane fetches one entry's column, piece and
// coordinates, then 18 lanes (d, q) go through the entries together and sum
// T[d][q] = (A_ij C_j)[d][q], C_j the column node's modes, as long as the piece
// stays the same (mostly: a row's columns are near it). R_i^T T, R_i the row
// node's modes, goes into the warp's own sums for that piece, which are added
// in warp order at the end, so the result is the same every time. (One entry
// after the other, each waiting for its column, piece and coordinates: 1,320 us
// on the Tet10 box of 27 x 15 x 13 cells, now 440.)
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
    const int d = lane < 18 ? lane / 6 : 0;               // T[d][q0]
    for (int first = 0; first < count; first += RC_NB) {
        const int nb = min(RC_NB, count - first);
        double *acc = rc_acc + (size_t)w * RC_NB * 36;
        for (int i = lane; i < nb * 36; i += 32) acc[i] = 0.0;
        __syncwarp();
        for (int i = w; i < me.rows; i += RC_WARPS) {
            const int64_t row = (int64_t)me.row0 + i;
            double r0[3], r1[3];
            const float *xi = xl + 3 * row;
            rc_mode(p0, xi[0], xi[1], xi[2], r0);
            rc_mode(two ? p1 : 0, xi[0], xi[1], xi[2], r1);
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (S.fixed && __ldg(S.fixed + 3 * row + c)) r0[c] = r1[c] = 0.0;
            const int32_t kb = __ldg(S.rp + row), ke = __ldg(S.rp + row + 1);
            double T = 0.0;
            int cur = -1;
            auto flush = [&]() {                          // acc[cur] += R^T T
                double s0 = 0.0, s1 = 0.0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    s0 += r0[c] * __shfl_sync(0xffffffffu, T, 6 * c + q0);
                    s1 += r1[c] * __shfl_sync(0xffffffffu, T, 6 * c + q1);
                }
                if (cur >= 0) {
                    acc[cur * 36 + lane] += s0;
                    if (two) acc[cur * 36 + 32 + lane] += s1;
                }
                T = 0.0;
            };
            for (int32_t k0 = kb; k0 < ke; k0 += 32) {
                const int32_t k = k0 + lane < ke ? k0 + lane : ke - 1;
                const int64_t j = __ldg(S.ci + k);
                const int bl = slot[__ldg(own + j)] - first;
                const float x = __ldg(xl + 3 * j), y = __ldg(xl + 3 * j + 1), z = __ldg(xl + 3 * j + 2);
                int fl = 0;
#pragma unroll
                for (int c = 0; c < 3; ++c) fl |= S.fixed && __ldg(S.fixed + 3 * j + c) ? 1 << c : 0;
                const int m = min(32, ke - k0);
#pragma unroll 4
                for (int e = 0; e < m; ++e) {
                    const int b = __shfl_sync(0xffffffffu, bl, e), f = __shfl_sync(0xffffffffu, fl, e);
                    const float xe = __shfl_sync(0xffffffffu, x, e), ye = __shfl_sync(0xffffffffu, y, e),
                                ze = __shfl_sync(0xffffffffu, z, e);
                    const double *v = S.v64 + 9 * (int64_t)(k0 + e) + 3 * d;
                    const double a0 = __ldg(v), a1 = __ldg(v + 1), a2 = __ldg(v + 2);
                    if (b != cur) {                       // uniform over the warp
                        flush();
                        cur = b >= 0 && b < nb ? b : -1;
                    }
                    double c[3];
                    rc_mode(q0, xe, ye, ze, c);
                    T += a0 * (f & 1 ? 0.0 : c[0]) + a1 * (f & 2 ? 0.0 : c[1]) + a2 * (f & 4 ? 0.0 : c[2]);
                }
            }
            flush();
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
// pivoting, pivot blocks of RC_RB rows, each held by one block in shared memory
// (the last padded with zero rows to nmp = nb RC_RB). Step k needs only the rows
// of block k: their owner scales and publishes them with a flag, the others
// wait for the flag, read them and update theirs; the next owner's first warp
// meanwhile inverts its pivot block. A pivot that has all but vanished (a mode
// that others span: a piece of nodes on a line, all its DOFs fixed, padding)
// leaves its unknown out: zero row and column. A chain of nb steps of a few us,
// mostly the way of flag and rows through L2: 148 pieces took 820 us with a
// pivot block per piece, 690 with two. Waits are bounded; on expiry *err is
// set and every block returns (hold: as if no flag came, CFEM_PARAM_BARRIER_HOLD).
constexpr int RC_RB = 2 * RM;
__global__ void __launch_bounds__(RT, 1)
k_rc_inv(const double *__restrict__ ac, int nm, int nb, double *rowbuf, unsigned *flag,
         double *__restrict__ out, int *err, unsigned long long timeout_ns, unsigned hold) {
    extern __shared__ __align__(16) double rc_rows[];     // the block's own rows
    __shared__ double D[RC_RB][RC_RB], d0[RC_RB];
    __shared__ __align__(16) double Dt[RC_RB][RC_RB], Ft[RC_RB][RC_RB];   // [column][row]
    __shared__ int quit;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, me = blockIdx.x, nmp = RC_RB * nb;
    double *mine = rc_rows;
    for (int i = t; i < RC_RB * nmp; i += RT) {
        const int r = RC_RB * me + i / nmp, c = i % nmp;
        mine[i] = r < nm && c < nm ? ac[(size_t)r * nm + c] : 0.0;
    }
    if (t == 0) quit = 0;
    __syncthreads();
    if (t < RC_RB) d0[t] = mine[t * nmp + RC_RB * me + t];
    __syncthreads();
    // first warp: D = D^-1 in place, and Dt; lane (i, h) holds half h of row i
    auto invert = [&]() {
        constexpr int H = RC_RB / 2;
        const int i = lane % RC_RB, h = lane / RC_RB;
        double a[H];
#pragma unroll
        for (int c = 0; c < H; ++c) a[c] = h < 2 ? D[i][H * h + c] : 0.0;
#pragma unroll
        for (int p = 0; p < RC_RB; ++p) {
            double r[H];
#pragma unroll
            for (int c = 0; c < H; ++c) r[c] = __shfl_sync(0xffffffffu, a[c], p + RC_RB * min(h, 1));
            const double f = __shfl_sync(0xffffffffu, a[p % H], i + RC_RB * (p / H));
            const double dp = __shfl_sync(0xffffffffu, a[p % H], p + RC_RB * (p / H));
            const bool take = dp > 1e-10 * d0[p] && d0[p] > 0.0;
            const double iv = take ? 1.0 / dp : 0.0, g = i == p ? iv : -f * iv;
#pragma unroll
            for (int c = 0; c < H; ++c) a[c] = i == p ? r[c] * iv : a[c] + r[c] * g;
            if (h == p / H) a[p % H] = g;
        }
        if (h < 2)
#pragma unroll
            for (int c = 0; c < H; ++c) {
                D[i][H * h + c] = a[c];
                Dt[H * h + c][i] = a[c];
            }
    };
    // v[i] += M[p][i] x[p] over p: M's column by column from shared memory, all
    // rows' sums side by side
    auto times = [&](const double (*M)[RC_RB], const double x[RC_RB], double v[RC_RB]) {
        asm volatile("" ::: "memory");    // (M again for each column: it would not fit registers)
#pragma unroll
        for (int p = 0; p < RC_RB; ++p)
#pragma unroll
            for (int i = 0; i < RC_RB; i += 2) {
                const double2 m = *(const double2 *)&M[p][i];
                v[i] += m.x * x[p];
                v[i + 1] += m.y * x[p];
            }
    };
    if (me == 0 && wid == 0) {
        for (int e = lane; e < RC_RB * RC_RB; e += 32) D[e / RC_RB][e % RC_RB] = mine[(e / RC_RB) * nmp + e % RC_RB];
        __syncwarp();
        invert();
    }
    __syncthreads();
    for (int k = 0; k < nb; ++k) {
        if (k == me) {
            for (int j = t; j < nmp; j += RT) {
                double c[RC_RB], v[RC_RB];
#pragma unroll
                for (int p = 0; p < RC_RB; ++p) {
                    c[p] = mine[p * nmp + j];
                    v[p] = 0.0;
                }
                times(Dt, c, v);
                const bool diag = j / RC_RB == k;
#pragma unroll
                for (int i = 0; i < RC_RB; ++i) {
                    if (diag) v[i] = D[i][j - RC_RB * k];
                    mine[i * nmp + j] = v[i];
                    rowbuf[(size_t)(RC_RB * k + i) * nmp + j] = v[i];
                }
            }
            __syncthreads();
            if (t == 0) {
                fence_gpu();
                for (int c = 0; c < RS_COPIES; ++c)
                    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(flag + c * nb + k), "r"(1u) : "memory");
            }
        } else {
            if (t == 0) {
                const unsigned *f = flag + (me % RS_COPIES) * nb + k;
                unsigned long long t0 = 0;
                for (unsigned spin = 0; ld_acquire(f) == 0 || hold; ++spin)
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
            for (int e = t - 32; e >= 0 && e < RC_RB * RC_RB; e += RT)
                Ft[e % RC_RB][e / RC_RB] = -mine[(e / RC_RB) * nmp + RC_RB * k + e % RC_RB];
            const bool next = k + 1 == me;
            if (next && wid == RWARPS - 1)                // the next pivot block, as it is now
                for (int e = lane; e < RC_RB * RC_RB; e += 32)
                    D[e / RC_RB][e % RC_RB] = mine[(e / RC_RB) * nmp + RC_RB * me + e % RC_RB];
            __syncthreads();
            if (quit) return;
            const double *rk = rowbuf + (size_t)RC_RB * k * nmp;
            if (next && wid == 0) {
                for (int e = lane; e < RC_RB * RC_RB; e += 32) {
                    const int i = e / RC_RB, j = e % RC_RB;
                    double v = D[i][j];
#pragma unroll
                    for (int p = 0; p < RC_RB; ++p) v += Ft[p][i] * __ldcg(rk + (size_t)p * nmp + RC_RB * me + j);
                    D[i][j] = v;
                }
                __syncwarp();
                invert();
            }
            const int lo = next ? 32 : 0;                 // threads that update
            for (int j = t - lo; j >= 0 && j < nmp; j += RT - lo) {
                double r[RC_RB], v[RC_RB];
                const bool diag = j / RC_RB == k;
#pragma unroll
                for (int p = 0; p < RC_RB; ++p) {
                    r[p] = __ldcg(rk + (size_t)p * nmp + j);
                    v[p] = diag ? 0.0 : mine[p * nmp + j];
                }
                times(Ft, r, v);
#pragma unroll
                for (int i = 0; i < RC_RB; ++i) mine[i * nmp + j] = v[i];
            }
            __syncthreads();
        }
    }
    for (int i = t; i < RC_RB * nmp; i += RT) {
        const int r = RC_RB * me + i / nmp, c = i % nmp;
        if (r < nm && c < nm) out[(size_t)r * nm + c] = mine[i];
    }
}
