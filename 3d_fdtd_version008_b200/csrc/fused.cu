// fused.cu -- device code of the fused step (fused.cuh).
#include "fused.cuh"

namespace fdtdk {

__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(unsigned(__cvta_generic_to_shared(b))), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(unsigned(__cvta_generic_to_shared(b))),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(unsigned(__cvta_generic_to_shared(b))) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(unsigned(__cvta_generic_to_shared(b))), "r"(parity), "r"(2000u)  // suspended for up to 2 us
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned ns_now() {
    unsigned t;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    return t;
}
// Bounded wait for a phase: false when `limit` ns (below 2^31) have passed, or when another wait of
// the block has failed (what this one waits for may then never come).
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity, unsigned limit, volatile unsigned* failed) {
    if (mbar_try(b, parity)) return true;
    const unsigned t0 = ns_now();
    do {
        if (mbar_try(b, parity)) return true;
    } while (*failed == 0u && ns_now() - t0 < limit);
    *failed = 1u;
    return false;
}
constexpr unsigned kDrainNs = 1000000000u;  // bound on waiting for copies in flight before a block gives up

__device__ __forceinline__ void tma_load4(void* dst, const CUtensorMap* m, int x, int y, int z, int c, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
            unsigned(__cvta_generic_to_shared(dst))),
        "l"(m), "r"(x), "r"(y), "r"(z), "r"(c), "r"(unsigned(__cvta_generic_to_shared(bar)))
        : "memory");
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// One material row of the table as one 16-byte (FP64: 16 + 8) load.
__device__ __forceinline__ void row_of(const float* tab, unsigned id, float& x, float& y, float& z) {
    float w;
    asm("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x), "=f"(y), "=f"(z), "=f"(w) : "l"(tab + 4 * id));
}
__device__ __forceinline__ void row_of(const double* tab, unsigned id, double& x, double& y, double& z) {
    table_row(tab, id, x, y, z);
}
// bE of the vector's cells, from the block's copy of the table (st) or, when it has too many rows
// for that, from memory; a warp whose cells all hold their vector's first row reads one row.
template <typename T>
__device__ __forceinline__ void row_at(const T* st, const T* tab, unsigned id, T& x, T& y, T& z) {
    if (st) {
        if constexpr (sizeof(T) == 4) {
            const float4 v = *reinterpret_cast<const float4*>(st + 4 * id);
            x = v.x; y = v.y; z = v.z;
        } else {
            const double2 v = *reinterpret_cast<const double2*>(st + 4 * id);
            x = v.x; y = v.y; z = st[4 * id + 2];
        }
    } else {
        row_of(tab, id, x, y, z);
    }
}
template <typename T>
__device__ __forceinline__ void rows_of(const T* st, const T* tab, const RowIds<Vec<T>::W>& ids, T (&bx)[Vec<T>::W],
                                        T (&by)[Vec<T>::W], T (&bz)[Vec<T>::W]) {
    constexpr int W = Vec<T>::W;
    bool same = (ids.w[0] >> 16) == (ids.w[0] & 0xffffu);
    if constexpr (W == 4) same = same && ids.w[1] == ids.w[0];
    row_at(st, tab, ids[0], bx[0], by[0], bz[0]);
    if (__all_sync(kFull, same)) {
#pragma unroll
        for (int e = 1; e < W; ++e) { bx[e] = bx[0]; by[e] = by[0]; bz[e] = bz[0]; }
    } else {
#pragma unroll
        for (int e = 1; e < W; ++e) row_at(st, tab, ids[e], bx[e], by[e], bz[e]);
    }
}

// The CPML recursion on one derivative of a vector: psi from po + q (where `ld`), back to pn + q
// (where `st`), and towards L2 what the next plane needs, `step` further.  Loaded where it is used:
// few registers are held, and the block is long enough to be branched around when not wanted.
// Uniform coefficients (y and z slabs): co[0] = b, co[1] = c, ik = 1/kappa ...
template <typename T>
__device__ __forceinline__ void psi_yz(T (&d)[Vec<T>::W], const T* po, T* pn, unsigned q, unsigned step, bool ld, bool st,
                                       const T* co, T ik, T psc) {
    constexpr int W = Vec<T>::W;
    T psi[W];
#pragma unroll
    for (int e = 0; e < W; ++e) psi[e] = T(0);
    if (ld) Vec<T>::ld(po + q, psi);
    const T b = co[0], c = co[1];
#pragma unroll
    for (int e = 0; e < W; ++e) {
        psi[e] = psi_rec(b, psi[e], c, d[e]);
        d[e] = psi_eff<T, T>(d[e], ik, psi[e], psc);
    }
    if (st) {
        Vec<T>::st(pn + q, psi);
        prefetch_l2(po + (q + step));
    }
}
// ... and per cell (x slabs), in the cells of mask m; b = c = 0 in the others, whose psi stays 0.
template <typename T>
__device__ __forceinline__ void psi_x(T (&d)[Vec<T>::W], T (&psi)[Vec<T>::W], const T* po, T* pn, unsigned q, unsigned step,
                                      bool st, const T* b, const T* c, const T* ik, unsigned m, T psc) {
    constexpr int W = Vec<T>::W;
    T v[W], t[W];
    Vec<T>::ld(c, v);
#pragma unroll
    for (int e = 0; e < W; ++e) t[e] = mul_rn(v[e], d[e]);
    Vec<T>::ld(b, v);
#pragma unroll
    for (int e = 0; e < W; ++e) psi[e] = fma_rn(v[e], psi[e], t[e]);  // psi_rec
    Vec<T>::ld(ik, v);
#pragma unroll
    for (int e = 0; e < W; ++e) {
        const T f = psi_eff<T, T>(d[e], v[e], psi[e], psc);
        d[e] = (m >> e) & 1u ? f : d[e];
    }
    if (st) {
        Vec<T>::st(pn + q, psi);
        prefetch_l2(po + (q + step));
    }
}
// v += b * c, rounded once, in the cells of mask m (all of them unless MASKED).
template <bool MASKED, typename T, int W>
__device__ __forceinline__ void update(T (&v)[W], const T (&b)[W], const T (&c)[W], unsigned m) {
    if constexpr (MASKED) vfma_in(v, b, c, m);
    else vfma(v, b, c);
}

// a: the arguments with the fields and psi_H of the copy being written.
template <typename T, bool SH>
__global__ void __launch_bounds__(FusedShape<T>::kThreads, 2)
k_step_fused(const __grid_constant__ CUtensorMap mapE, const __grid_constant__ CUtensorMap mapH, const StepArgs<T, T> a,
             const PsiOld<T> old, const FusedGeom g, const ESrc src, unsigned* status_w) {
    using F = FusedShape<T>;
    constexpr int W = F::W, TY = F::TY, NS = F::NS, LH = F::LH, XW = F::XW;
    constexpr int EC = (TY + 2) * XW, HC = (TY + 1) * XW;  // elements of one staged component
    extern __shared__ __align__(1024) unsigned char fsm[];
    // full: the stage's copies have arrived; freed: every warp has read it for the last time;
    // xfull: the row's new Hx and Hz are in the stage
    __shared__ uint64_t full[NS], freed[NS], xfull[NS][TY];
    __shared__ unsigned failed;  // a wait of this block has run out
    __shared__ int issued;       // the last ring position whose copies were asked for
    int lane, w;  // opaque, so that they stay in registers
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(lane));
    asm volatile("mov.u32 %0, %%tid.y;" : "=r"(w));
    w = __shfl_sync(kFull, w, 0);
    const int kb = int(blockIdx.z) * g.kc, ke = min(kb + g.kc, a.NzT);
    const int k0 = max(kb - 1, 0);  // H of plane kb - 1 is recomputed
    const int j0 = int(blockIdx.y) * TY, j = j0 - 1 + w;
    const int xt = (int(blockIdx.x) * g.u - LH) * W;
    const int x0 = xt + lane * W;
    auto stage = [&](int s) { return reinterpret_cast<T*>(fsm + s * int(F::STAGE)); };
    // plane k: E of k + 1 and H of k
    auto issue = [&](int k, int s) {
        mbar_expect(&full[s], F::EB + F::HB);
        tma_load4(stage(s), &mapE, xt, j0 - 1, k + 1, 0, &full[s]);
        tma_load4(stage(s) + 3 * EC, &mapH, xt, j0 - 1, k, 0, &full[s]);
    };
    const bool leader = lane == 0 && w == 0;
    bool stop = false;
    if (leader) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&freed[s], TY + 1);
            for (int r = 0; r < TY; ++r) mbar_init(&xfull[s][r], 1 + g.hold);
        }
        failed = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // the first planes' copies, unless a failed monitor step has stopped the solve (one thread
        // decides, so that no block leaves with copies in flight)
        stop = *a.status != 0u;
        if (!stop) {
            mbar_expect(&full[0], F::EB);
            tma_load4(stage(0), &mapE, xt, j0 - 1, k0, 0, &full[0]);
#pragma unroll
            for (int p = 1; p < NS; ++p)
                if (k0 + p - 1 < ke) issue(k0 + p - 1, p);
            issued = min(NS - 1, ke - k0);
        }
    }
    // The tile's coefficients, so that a plane waits for no global load of them: along x (1/dx and,
    // in the slabs, b and c of H and E, 1/kappa; 0 outside), y and z (the same six), the material rows.
    T* const xco = reinterpret_cast<T*>(fsm + NS * int(F::STAGE)) + lane * W;
    T* const yco = reinterpret_cast<T*>(fsm + NS * int(F::STAGE) + int(F::XCO));  // [row w][6]
    T* const zco = yco + 6 * (TY + 2);  // [plane k - k0][6]
    const T* const smat = g.nrow <= F::kRows ? zco + 6 * (F::kMaxKc + 1) : nullptr;
    if (w < 6) {  // warp w: coefficient w of every axis
        auto pick = [&](const T* q0, const T* q1, const T* q2, const T* q3, const T* q4, const T* q5) {
            return w == 0 ? q0 : w == 1 ? q1 : w == 2 ? q2 : w == 3 ? q3 : w == 4 ? q4 : q5;
        };
        const T* const fx = pick(a.idx, a.pbH[0], a.pcH[0], a.pbE[0], a.pcE[0], a.ik[0]);
        const T* const fy = pick(a.idy, a.pbH[1], a.pcH[1], a.pbE[1], a.pcE[1], a.ik[1]);
        const T* const fz = pick(a.idz, a.pbH[2], a.pcH[2], a.pbE[2], a.pcE[2], a.ik[2]);
#pragma unroll
        for (int e = 0; e < W; ++e) {
            const int i = x0 + e;
            xco[w * XW + e] = i >= 0 && i < a.NxT && (w == 0 || in_pml(i, a.NxT, a.np)) ? __ldg(fx + i) : T(0);
        }
        const int jj = j0 - 1 + lane;
        if (lane < TY + 1) yco[6 * lane + w] = jj >= 0 && jj < a.NyT ? __ldg(fy + jj) : T(0);
        for (int t = lane; t < ke - k0; t += 32) zco[6 * t + w] = __ldg(fz + k0 + t);
    } else if (smat) {
        for (int t = (w - 6) * 32 + lane; t < 4 * g.nrow; t += 64) const_cast<T*>(smat)[t] = __ldg(a.btab + t);
    }
    if (__syncthreads_or(stop)) return;
    if (lane == 0 && w < TY) mbar_arrive(&xfull[0][w]);  // ring position 0 has no H
    const int np = a.np, np2 = 2 * np;
    const bool in = x0 >= 0 && x0 < a.NxT;
    const bool row_in = j >= 0 && j < a.NyT;
    const bool own = w >= 1 && row_in && in && lane >= LH && lane < LH + g.u;
    const bool hrow = j >= 0 && j < a.NyT - 1;
    const bool erow = w >= 1 && j >= 1 && j < a.NyT;
    const bool ypml = row_in && in_pml(j, a.NyT, np);
    const int jy = ypml ? slab_index(j, a.NyT, np) : 0;
    // masks of the vector's cells: in an x slab; where H, E are updated
    unsigned mx = 0, mh = 0, me = 0;
    if (in) {
#pragma unroll
        for (int e = 0; e < W; ++e) {
            const int i = x0 + e;
            mx |= unsigned(i < a.NxT && in_pml(i, a.NxT, np)) << e;
            mh |= unsigned(i < a.NxT - 1) << e;
            me |= unsigned(i >= 1 && i < a.NxT) << e;
        }
    }
    const bool xpml = mx != 0;
    const bool xgen = __any_sync(kFull, xpml);
    const bool grow = own && a.gain && j >= a.gj0 && j < a.gj0 + a.gY && x0 >= a.gi0 && x0 < a.gi0 + a.gX;
    bool srow = false;  // some source may lie in this thread's column
    for (int s = 0; s < src.n; ++s) srow |= src.sj[s] == j && src.si[s] >= x0 && src.si[s] < x0 + W;
    if constexpr (SH) srow |= src.ns > 0;
    srow = srow && own;
    // A warp takes the plain update in every plane away from the z slabs and the gain box when none of
    // its vectors needs a mask, lies in a slab or may hold a source, and its row is updated.
    const bool gen_col = __any_sync(kFull, mx != 0 || mh != (1u << W) - 1 || me != (1u << W) - 1 || srow) || ypml || !hrow ||
                         (w >= 1 && !erow);
    const bool gain_col = __any_sync(kFull, grow);
    T nbH[W];
#pragma unroll
    for (int e = 0; e < W; ++e) nbH[e] = -a.bH;
    int row = j * a.NxP + x0;  // within a plane
    int lanev = lane * W, wv = w;  // this thread's place in a staged row, its row in the stage
    T* out = a.Ex + ((long long)k0 * a.plane + row);
    const uint16_t* bid = a.bidx + ((long long)kb * a.plane + row);
    const long long fs = a.Ey - a.Ex;  // the six arrays are equally spaced

    T hxm[W], hym[W];  // Hx, Hy at k-1
#pragma unroll
    for (int e = 0; e < W; ++e) hxm[e] = hym[e] = T(0);
    RowIds<W> ids{};
    if (own) ids.load(bid);

    const T* eprev = stage(0) + wv * XW + lanev;  // this thread's vector of E(k) and of E(k+1), H(k)
    int sp = 0, sc = 1;                             // stages of E(k) and of E(k+1), H(k)
    unsigned php = 0, ph = 0;                       // parities of their phases
    unsigned xq = unsigned(xpsi_at(a, k0, row_in ? j : 0, x0));  // the vector's x-slab psi, y-slab psi
    unsigned yq = unsigned(k0 * np2 + jy) * unsigned(a.NxP) + unsigned(x0);
    unsigned xstep = unsigned(a.NyT) * unsigned(XSlab(a.NxT, np, W).len), ystep = unsigned(np2) * unsigned(a.NxP);
    auto wait = [&](uint64_t* b, unsigned parity) { return mbar_wait(b, parity, g.wait_ns, &failed); };
    bool ok = wait(&full[0], 0);

    // G: with everything a plane may need; else the plain update.
    auto plane = [&](auto general, const int k) __attribute__((always_inline)) {
        constexpr bool G = decltype(general)::value;
        const bool mine = own && k >= kb;
        const bool zpml = G && in_pml(k + a.kz0, a.NzG, np);
        const unsigned zq = G && zpml ? unsigned(slab_index(k + a.kz0, a.NzG, np)) * unsigned(a.plane) + unsigned(row) : 0u;
        const unsigned zs = G && in_pml(k + 1 + a.kz0, a.NzG, np) && k + 1 < ke ? unsigned(a.plane) : 0u;
        const unsigned xs1 = k + 1 < ke ? xstep : 0u, ys1 = k + 1 < ke ? ystep : 0u;
        const T* const zc = zco + 6 * (k - k0);
        const T* const yc = yco + 6 * w;
        const T idz = zc[0], idy = yc[0];
        const bool hup = !G || (hrow && k + a.kz0 < a.NzG - 1);
        const bool eup = w >= 1 && k >= kb && (!G || (erow && k + a.kz0 >= 1));
        T ex[W], ey[W], ez[W], hx[W], hy[W], hz[W];
        T px0[W], px1[W];  // x-slab psi, issued before the wait
        if (G && xpml && hup) { Vec<T>::ld(old.p[3] + xq, px0); Vec<T>::ld(old.p[4] + xq, px1); }
        ok = ok && wait(&full[sc], ph);
        T* const ecur = stage(sc) + wv * XW + lanev;
        Vec<T>::ld(eprev, ex);
        Vec<T>::ld(eprev + EC, ey);
        Vec<T>::ld(eprev + 2 * EC, ez);
        Vec<T>::ld(ecur + 3 * EC, hx);
        Vec<T>::ld(ecur + 3 * EC + HC, hy);
        Vec<T>::ld(ecur + 3 * EC + 2 * HC, hz);
        if (hup) {  // uniform in the warp
            const T eyn = __shfl_down_sync(kFull, ey[0], 1);
            const T ezn = __shfl_down_sync(kFull, ez[0], 1);
            T t[W], da[W], db[W], idx[W];
            Vec<T>::ld(xco, idx);
            // Hx: dEz/dy - dEy/dz
            Vec<T>::ld(eprev + XW + 2 * EC, t);
            vdq(da, t, ez, idy);
            Vec<T>::ld(ecur + EC, t);
            vdq(db, t, ey, idz);
            if (G && ypml) psi_yz(da, old.p[0], a.psiH[0], yq, ys1, in, mine, yc + 1, yc[5], a.psc);
            if (G && zpml) psi_yz(db, old.p[1], a.psiH[1], zq, zs, in, mine, zc + 1, zc[5], a.psc);
            vsub(da, db);
            update<G>(hx, nbH, da, mh);
            // Hy: dEx/dz - dEz/dx
            Vec<T>::ld(ecur, t);
            vdq(da, t, ex, idz);
#pragma unroll
            for (int e = 0; e < W; ++e) db[e] = sub_rn((e < W - 1) ? ez[e + 1] : ezn, ez[e]);
            vmul(db, idx);
            if (G && zpml) psi_yz(da, old.p[2], a.psiH[2], zq, zs, in, mine, zc + 1, zc[5], a.psc);
            if (G && xgen) psi_x(db, px0, old.p[3], a.psiH[3], xq, xs1, xpml && mine, xco + XW, xco + 2 * XW, xco + 5 * XW, mx, a.psc);
            vsub(da, db);
            update<G>(hy, nbH, da, mh);
            // Hz: dEy/dx - dEx/dy
            Vec<T>::ld(eprev + XW, t);
#pragma unroll
            for (int e = 0; e < W; ++e) da[e] = sub_rn((e < W - 1) ? ey[e + 1] : eyn, ey[e]);
            vmul(da, idx);
            vdq(db, t, ex, idy);
            if (G && xgen) psi_x(da, px1, old.p[4], a.psiH[4], xq, xs1, xpml && mine, xco + XW, xco + 2 * XW, xco + 5 * XW, mx, a.psc);
            if (G && ypml) psi_yz(db, old.p[5], a.psiH[5], yq, ys1, in, mine, yc + 1, yc[5], a.psc);
            vsub(da, db);
            update<G>(hz, nbH, da, mh);
        }
        {
            // the next row's warp reads Hx and Hz from the stage, where they replace the old ones
            Vec<T>::st(ecur + 3 * EC, hx);
            Vec<T>::st(ecur + 3 * EC + 2 * HC, hz);
            if (mine) {
                Vec<T>::st(out + 3 * fs, hx);
                Vec<T>::st(out + 4 * fs, hy);
                Vec<T>::st(out + 5 * fs, hz);
            }
        }
        if (G && xpml && own && eup) { Vec<T>::ld(a.psiE[3] + xq, px0); Vec<T>::ld(a.psiE[4] + xq, px1); }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&freed[sp]);
            if (w < TY) mbar_arrive(&xfull[sc][w]);
        }
        if (w == 0) {
            // E(k) is read: its stage takes the next plane
            if (k + NS - 1 < ke) {
                ok = ok && wait(&freed[sp], php);
                if (leader && ok) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // H was written into the stage
                    issue(k + NS - 1, sp);
                    issued = k + NS - k0;
                }
            }
        } else if (k >= kb) {
            ok = ok && wait(&xfull[sc][w - 1], ph);
        }

        if (eup) {  // uniform in the warp
            const T* const xs = ecur + 3 * EC - XW;  // the row below
            const T hzp = __shfl_up_sync(kFull, hz[W - 1], 1), hyp = __shfl_up_sync(kFull, hy[W - 1], 1);
            const unsigned special = G && srow ? src_in_vector<SH>(src, x0, j, k, W) : 0u;
            T bx[W], by[W], bz[W];
            rows_of(smat, a.btab, ids, bx, by, bz);
            T t[W], da[W], db[W], idx[W];
            Vec<T>::ld(xco, idx);
            // Ex: dHz/dy - dHy/dz
            Vec<T>::ld(xs + 2 * HC, t);
            vdq(da, hz, t, idy);
            vdq(db, hy, hym, idz);
            if (G && ypml) psi_yz(da, a.psiE[0], a.psiE[0], yq, ys1, own, own, yc + 3, yc[5], a.psc);
            if (G && zpml) psi_yz(db, a.psiE[1], a.psiE[1], zq, zs, own, own, zc + 3, zc[5], a.psc);
            vsub(da, db);
            if (G && special) sub_J<SH>(src, special, 0, x0, j, k, da);
            update<G>(ex, bx, da, me);
            // Ey: dHx/dz - dHz/dx
            vdq(da, hx, hxm, idz);
#pragma unroll
            for (int e = 0; e < W; ++e) db[e] = sub_rn(hz[e], (e > 0) ? hz[e - 1] : hzp);
            vmul(db, idx);
            if (G && zpml) psi_yz(da, a.psiE[2], a.psiE[2], zq, zs, own, own, zc + 3, zc[5], a.psc);
            if (G && xgen) psi_x(db, px0, a.psiE[3], a.psiE[3], xq, xs1, xpml && own, xco + 3 * XW, xco + 4 * XW, xco + 5 * XW, mx, a.psc);
            vsub(da, db);
            if (G && special) sub_J<SH>(src, special, 1, x0, j, k, da);
            update<G>(ey, by, da, me);
            // Ez: dHy/dx - dHx/dy
            Vec<T>::ld(xs, t);
#pragma unroll
            for (int e = 0; e < W; ++e) da[e] = sub_rn(hy[e], (e > 0) ? hy[e - 1] : hyp);
            vmul(da, idx);
            vdq(db, hx, t, idy);
            if (G && xgen) psi_x(da, px1, a.psiE[4], a.psiE[4], xq, xs1, xpml && own, xco + 3 * XW, xco + 4 * XW, xco + 5 * XW, mx, a.psc);
            if (G && ypml) psi_yz(db, a.psiE[5], a.psiE[5], yq, ys1, own, own, yc + 3, yc[5], a.psc);
            vsub(da, db);
            if (G && special) sub_J<SH>(src, special, 2, x0, j, k, da);
            if (G && grow && k >= a.gk0 && k < a.gk0 + a.gZ) {
                gain_vector(a, src.parity, x0, j, k, me, da, bz, ez);
            } else {
                update<G>(ez, bz, da, me);
            }
        }
        if (mine) {
            Vec<T>::st(out, ex);
            Vec<T>::st(out + fs, ey);
            Vec<T>::st(out + 2 * fs, ez);
        }
#pragma unroll
        for (int e = 0; e < W; ++e) { hxm[e] = hx[e]; hym[e] = hy[e]; }
        eprev = ecur;
    };
    for (int k = k0; k < ke; ++k) {  // to the end after a failed wait too: a plane's shuffles take every lane
        const bool gen = gen_col || in_pml(k + a.kz0, a.NzG, np) || k + a.kz0 >= a.NzG - 1 || k + a.kz0 < 1 ||
                         (gain_col && k >= a.gk0 && k < a.gk0 + a.gZ);
        if (gen) plane(std::true_type{}, k);
        else plane(std::false_type{}, k);
        out += a.plane;
        if (k >= kb) {
            bid += a.plane;
            if (own && k + 1 < ke) {
                ids.load(bid);
                if (k + 2 < ke) prefetch_l2(bid + a.plane);
            }
        }
        xq += xstep;
        yq += ystep;
        sp = sc;
        php = ph;
        if (++sc == NS) { sc = 0; ph ^= 1u; }
    }
    if (!ok) {  // a wait ran out: flag it and leave
        atomicOr(status_w, kStatusTimeout);
        if (leader) {  // ... but not before the copies in flight, whose target is the block's shared memory
            const unsigned t0 = ns_now();
            for (int m = max(issued - NS + 1, 0); m <= issued; ++m)
                while (!mbar_try(&full[m % NS], unsigned(m / NS) & 1u) && ns_now() - t0 < kDrainNs) {}
        }
    }
}

template <typename T>
FusedKernel<T> fused_kernel(bool sheets) {
    return sheets ? k_step_fused<T, true> : k_step_fused<T, false>;
}
template FusedKernel<float> fused_kernel<float>(bool);
template FusedKernel<double> fused_kernel<double>(bool);

}  // namespace fdtdk
