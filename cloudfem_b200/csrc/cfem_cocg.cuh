// Resident COCG: the phasor A-V system's Jacobi-preconditioned conjugate
// orthogonal CG (the unconjugated form x^T y) in one cooperative launch, on
// the resident scheduler's layout and grid-wide sums (cfem_resident.cuh,
// included before this file). Entries, halo and vectors are complex
// (double2); the iteration and its tests are those of the launches in
// cfem_complex.cu, which takes what this does not: patterns too scattered for
// the halo.
//
// Bounds: as for the resident CG the chain of an iteration, two grid-wide
// sums and the products between them. A Tet10 box of 7 x 6 x 6 cells (7,500
// unknowns, rows of 100 entries on 8 lanes): 10.5 us per iteration, against
// 29.7 us for the five launches per iteration and the host check every eight
// of cfem_complex.cu.

struct CocgState {
    double2 rho, alpha, beta;
    double rr, bb;
    int iter, status, done;
};

struct CocgShared {
    double red[4][RWARPS];
    CocgState st;
    int quit, nres, own;
};

// One lane's part of a row: sum of a_j v_j over its slots.
template <bool SM>
__device__ __forceinline__ double2 cocg_row(const uint16_t *cp, const double2 *vp, int w,
                                            const double2 *halo) {
    constexpr int U = 4;
    double2 acc = make_double2(0.0, 0.0);
    for (int t = 0; t < w; t += U) {
        int c[U];
        double2 a[U];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int tt = t + j < w ? t + j : w - 1;
            c[j] = SM ? cp[32 * tt] : ld_stream(cp + 32 * tt);
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int tt = t + j < w ? t + j : w - 1;
            a[j] = SM ? vp[32 * tt] : __ldcs(vp + 32 * tt);
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const double2 m = cmul(a[j], halo[c[j]]);
            acc.x += t + j < w ? m.x : 0.0;
            acc.y += t + j < w ? m.y : 0.0;
        }
    }
    return acc;
}

__global__ void __launch_bounds__(RT, 1)
k_resident_cocg(const SysDev *__restrict__ sys, CocgState *gst, GridBar *bar,
                const RsCta *__restrict__ ctas, int nbytes, double rtol2, int max_iter,
                unsigned long long timeout_ns, unsigned hold) {
    extern __shared__ __align__(128) unsigned char rs_area[];
    __shared__ CocgShared sh;
    const SysDev &S = *sys;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const RsCta me = ctas[blockIdx.x];
    const int cta = me.cta, nc = S.ncta, lsh = S.lsh, L = 1 << lsh;
    const int nloc = me.rows, nsl = rs_slices(nloc, lsh);
    const int64_t r0 = me.row0;
    const double2 *b = (const double2 *)S.b + r0;
    double2 *xg = (double2 *)S.x, *x = xg + r0;
    double2 *pair = (double2 *)S.pair;   // (z, previous p) of row i at 2 i, 2 i + 1
    ulonglong2 *mail = S.mail;
    const int nu = __ldg(&S.ucnt[blockIdx.x].x);
    if (tid == 0) {
        memset(&sh.st, 0, sizeof(CocgState));
        sh.quit = 0;
        sh.own = 0;
    }
    __syncthreads();
    unsigned char *area = rs_area;
    int *so = (int *)area;
    area += rs_al((size_t)(nsl + 1) * 4);
    uint8_t *perm = area;
    area += rs_al((size_t)nsl << (5 - lsh));
    int32_t *list = (int32_t *)area;
    area += rs_al((size_t)nu * 4);
    double2 *halo = (double2 *)area;
    area += (size_t)((nu + 31) & ~31) * 16;
    double2 *q, *r, *dinv;
    if (S.vsm) {
        q = (double2 *)area;
        r = q + nloc;
        dinv = r + nloc;
        area += rs_vec_bytes(nloc, 1, 16);
    } else {
        q = (double2 *)S.q + r0;
        r = (double2 *)S.r + r0;
        dinv = (double2 *)S.dinv + r0;
    }
    const int64_t off0 = __ldg(S.soff + me.sl0);
    for (int i = tid; i <= nsl; i += RT) so[i] = (int)(__ldg(S.soff + me.sl0 + i) - off0);
    for (int i = tid; i < nsl << (5 - lsh); i += RT) perm[i] = __ldg(S.sperm + me.sl0 * 32 + i);
    for (int i = tid; i < nu; i += RT) {
        const int32_t c = __ldg(S.ulist + (size_t)blockIdx.x * S.umax + i);
        list[i] = c;
        if (c == (int32_t)r0) sh.own = i;
    }
    __syncthreads();
    if (tid == 0) {   // the leading slices that fit
        const size_t room = (size_t)nbytes - (size_t)(area - rs_area);
        int lo = 0, hi = nsl;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((size_t)so[mid] * 18 <= room) lo = mid; else hi = mid - 1;
        }
        sh.nres = lo;
    }
    __syncthreads();
    const int nres = sh.nres, eres = so[nres];
    double2 *mv = (double2 *)area;
    uint16_t *mc = (uint16_t *)(area + (size_t)eres * 16);
    const uint16_t *gc = S.rcol + off0;
    const double2 *gv = (const double2 *)S.rval + off0;
    for (int i = tid; i < eres; i += RT) mv[i] = __ldcs(gv + i);
    for (int i = tid; i < eres / 8; i += RT) ((int4 *)mc)[i] = __ldcs((const int4 *)gc + i);
    const int own = sh.own;
    __syncthreads();

    // q = A (halo) on the block's rows; fin(row, value, diagonal entry)
    auto product = [&](auto fin) {
        const int grp = lane >> lsh;
        const bool first = (lane & (L - 1)) == 0;
        for (int s = wid, sn = 2 * RWARPS - 1 - wid; s < nsl; rs_next(s, sn)) {
            const int off = so[s], w = (so[s + 1] - off) >> 5;
            const int pos = s * (32 >> lsh) + grp;
            const int rl = (pos & ~(RS_WINDOW - 1)) + perm[pos];
            double2 acc = s < nres ? cocg_row<true>(mc + off + lane, mv + off + lane, w, halo)
                                   : cocg_row<false>(gc + off + lane, gv + off + lane, w, halo);
            for (int o = L >> 1; o > 0; o >>= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            }
            if (rl < nloc && first) fin(rl, acc, s < nres ? mv + off + lane : gv + off + lane);
        }
    };
    unsigned long long epoch = 1;
    // r = b - A x, the Jacobi inverse (slot 0 of a row is its diagonal), z
    for (int i = tid; i < nu; i += RT) halo[rs_swz(i)] = __ldcg(xg + list[i]);
    __syncthreads();
    double part[4] = {0.0, 0.0, 0.0, 0.0};
    bool bad = false;
    product([&](int rl, double2 ax, const double2 *diag) {
        const double2 dg = *diag, bi = b[rl];
        const double2 ri = make_double2(bi.x - ax.x, bi.y - ax.y);
        double2 di = make_double2(0.0, 0.0);
        if (dg.x != 0.0 || dg.y != 0.0) di = cdiv(make_double2(1.0, 0.0), dg);
        else bad = true;
        const double2 zi = cmul(di, ri), rz = cmul(ri, zi);
        r[rl] = ri;
        dinv[rl] = di;
        pair[2 * (r0 + rl)] = zi;
        pair[2 * (r0 + rl) + 1] = make_double2(0.0, 0.0);
        part[0] += rz.x;
        part[1] += rz.y;
        part[2] += ri.x * ri.x + ri.y * ri.y;
        part[3] += bi.x * bi.x + bi.y * bi.y;
    });
    // (a zero diagonal: told by the state in global memory, which the grid's sum
    // orders like the pairs)
    if (bad) atomicExch(&gst->status, (int)CFEM_ERR_BREAKDOWN);
    CocgState &st = sh.st;
    if (!rs_sync<4, true>(sh, mail, nc, bar, cta, epoch, part, timeout_ns, hold, [&](const double t[4]) {
            st.rho = make_double2(t[0], t[1]);
            st.rr = t[2];
            st.bb = t[3];
            st.status = *(volatile int *)&gst->status;
            if (st.status != CFEM_OK || !isfinite(t[2])) {
                st.done = 1;
                st.status = CFEM_ERR_BREAKDOWN;
            } else if (t[2] <= rtol2 * t[3]) {
                st.done = 1;
            }
        }))
        return;
    while (!st.done) {
        // halo: p = z + beta p_old
        const double2 be = st.beta;
        for (int i0 = tid; i0 < nu; i0 += 2 * RT) {
            double2 z[2], o[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i = i0 + k * RT < nu ? i0 + k * RT : i0;
                z[k] = __ldcg(pair + 2 * (int64_t)list[i]);
                o[k] = __ldcg(pair + 2 * (int64_t)list[i] + 1);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
                if (i0 + k * RT < nu) {
                    const double2 m = cmul(be, o[k]);
                    halo[rs_swz(i0 + k * RT)] = make_double2(z[k].x + m.x, z[k].y + m.y);
                }
        }
        __syncthreads();
        part[0] = part[1] = part[2] = part[3] = 0.0;
        product([&](int rl, double2 qi, const double2 *) {
            q[rl] = qi;
            const double2 pq = cmul(halo[rs_swz(own + rl)], qi);
            part[0] += pq.x;
            part[1] += pq.y;
        });
        ++epoch;
        if (!rs_sync<2, false>(sh, mail, nc, bar, cta, epoch, part, timeout_ns, hold, [&](const double t[4]) {
                const double2 mu = make_double2(t[0], t[1]);
                const double m2 = mu.x * mu.x + mu.y * mu.y;
                const double r2 = st.rho.x * st.rho.x + st.rho.y * st.rho.y;
                if (!(m2 > 1e-300 * (r2 + 1e-300)) || !isfinite(m2)) {
                    st.status = CFEM_ERR_BREAKDOWN;
                    st.done = 1;
                } else {
                    st.alpha = cdiv(st.rho, mu);
                }
            }))
            return;
        if (st.done) break;
        const double2 al = st.alpha;
        part[0] = part[1] = part[2] = part[3] = 0.0;
        for (int i = tid; i < nloc; i += RT) {
            const double2 pi = halo[rs_swz(own + i)], dx = cmul(al, pi), dr = cmul(al, q[i]);
            double2 xi = x[i], ri = r[i];
            xi.x += dx.x;
            xi.y += dx.y;
            ri.x -= dr.x;
            ri.y -= dr.y;
            const double2 zi = cmul(dinv[i], ri), rz = cmul(ri, zi);
            x[i] = xi;
            r[i] = ri;
            pair[2 * (r0 + i)] = zi;
            pair[2 * (r0 + i) + 1] = pi;
            part[0] += rz.x;
            part[1] += rz.y;
            part[2] += ri.x * ri.x + ri.y * ri.y;
        }
        ++epoch;
        if (!rs_sync<3, true>(sh, mail, nc, bar, cta, epoch, part, timeout_ns, hold, [&](const double t[4]) {
                const double2 rho = make_double2(t[0], t[1]);
                st.rr = t[2];
                st.iter += 1;
                if (!isfinite(t[2]) || !isfinite(t[0]) || !isfinite(t[1])) {
                    st.status = CFEM_ERR_BREAKDOWN;
                    st.done = 1;
                } else if (t[2] <= rtol2 * st.bb) {
                    st.done = 1;
                } else if (st.iter >= max_iter) {
                    st.status = CFEM_ERR_NOT_CONVERGED;
                    st.done = 1;
                } else {
                    st.beta = cdiv(rho, st.rho);
                    st.rho = rho;
                }
            }))
            return;
    }
    if (cta == 0 && tid == 0) *gst = st;
}
