// Another row order for the resident scheduler: a copy of the systems in an
// order that makes a block's rows a compact piece of the mesh, and the
// solution's way back. Included by cfem_solve.cu.
//
// A Tet10 mesh numbers its vertices before its edge nodes, so a block of
// vertex rows names edge nodes all over the part: of 7 blocks that share a 22^3
// mesh (79,507 rows) the first has 47,951 columns to fetch, which do not fit its
// shared memory. Sorted by the lowest column of their row (vertices and
// edges then go through the mesh together, and no coordinates are needed)
// a block fetches its own layers and the two next to them.

struct OrderDev {
    const int32_t *rp, *ci;
    const double *v64, *b;
    const float *v32;
    const uint8_t *fixed;
    double *x;
    int64_t n, base;                 // rows, and rows of the systems before
};

// Sort keys (system, lowest column), one row per 8 lanes; blockIdx.y: system.
__global__ void __launch_bounds__(256)
k_ro_mincol(const OrderDev *__restrict__ src, unsigned long long *__restrict__ key,
            int32_t *__restrict__ id) {
    const OrderDev S = src[blockIdx.y];
    const int sub = threadIdx.x & 7;
    const int64_t nr = ((int64_t)gridDim.x * blockDim.x) >> 3;
    // (whole warps stay in the loop: the shuffles name all lanes)
    for (int64_t r0 = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 4; r0 < S.n; r0 += nr) {
        const int64_t i = r0 + ((threadIdx.x & 31) >> 3);
        int32_t lo = INT32_MAX;
        if (i < S.n)
            for (int32_t k = S.rp[i] + sub; k < S.rp[i + 1]; k += 8) lo = min(lo, S.ci[k]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        if (i < S.n && sub == 0) {
            key[S.base + i] = (unsigned long long)blockIdx.y << 32 | (uint32_t)max(lo, 0);
            id[S.base + i] = (int32_t)i;
        }
    }
}
// Inverse of the order, and the row lengths in it.
__global__ void k_ro_rows(const OrderDev *__restrict__ src, const unsigned long long *__restrict__ key,
                          const int32_t *__restrict__ ord, int64_t rows, int32_t *__restrict__ inv,
                          int32_t *__restrict__ len) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g > rows) return;
    if (g == rows) {
        len[g] = 0;
        return;
    }
    const OrderDev *S = src + (key[g] >> 32);
    const int32_t o = ord[g];
    inv[S->base + o] = (int32_t)(g - S->base);
    len[g] = S->rp[o + 1] - S->rp[o];
}
// The systems in the new order, one warp per row; `what` is a sum of these.
constexpr int RO_COLS = 1, RO_V64 = 2, RO_V32 = 4, RO_VEC = 8;
template <int BS>
__global__ void __launch_bounds__(256)
k_ro_copy(const OrderDev *__restrict__ src, const int32_t *__restrict__ ord_all,
          const int32_t *__restrict__ inv_all, const int32_t *__restrict__ rp, int32_t *__restrict__ ci,
          double *__restrict__ v64, float *__restrict__ v32, double *__restrict__ b,
          double *__restrict__ x, uint8_t *__restrict__ fixed, int what) {
    constexpr int B2 = BS * BS;
    const OrderDev S = src[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < S.n; i += nw) {
        const int64_t g = S.base + i, o = ord_all[g];
        const int64_t k0 = S.rp[o], len = S.rp[o + 1] - k0, t0 = rp[g];
        if (what & RO_COLS)
            for (int64_t k = lane; k < len; k += 32) {
                const int32_t c = S.ci[k0 + k];
                ci[t0 + k] = (uint32_t)c < (uint32_t)S.n ? inv_all[S.base + c] : (int32_t)i;
            }
        if (what & RO_V64)
            for (int64_t k = lane; k < B2 * len; k += 32) v64[B2 * t0 + k] = S.v64[B2 * k0 + k];
        if (what & RO_V32)
            for (int64_t k = lane; k < B2 * len; k += 32) v32[B2 * t0 + k] = S.v32[B2 * k0 + k];
        if ((what & RO_VEC) && lane < BS) {
            b[BS * g + lane] = S.b[BS * o + lane];
            x[BS * g + lane] = S.x[BS * o + lane];
            fixed[BS * g + lane] = S.fixed ? S.fixed[BS * o + lane] : 0;
        }
    }
}
template <int BS>
__global__ void k_ro_back(const OrderDev *__restrict__ src, const int32_t *__restrict__ ord_all,
                          const double *__restrict__ xn) {
    const OrderDev S = src[blockIdx.y];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < BS * S.n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / BS;
        S.x[BS * (int64_t)ord_all[S.base + i] + (t - BS * i)] = xn[BS * S.base + t];
    }
}
