// The resident kernel (included by engine.cu inside namespace afd, after the
// per-unit PML arithmetic and the boundary and source/receiver roles).
//
// All steps of a chunk in one cooperative launch, for grids whose levels stay
// in L2: per step every group of 256 threads takes its share of PML pressure
// units, boundary entries and interior columns (they write disjoint cells and
// read only finished levels), one group or a few more the sources and receivers; a
// grid barrier, the auxiliary PML units where there are any, and another barrier
// end the step.
//
// Latency sets the pace: the chunk's 200 steps as graph nodes cost 10 us each
// even for the smallest room (three to five dependent launches), while the
// barrier here is 1.5 us, the boundary role 2.2, an interior column 0.9 and the
// sources and receivers 3.0. So what does not change from step to step is kept
// in registers across them (the first boundary entry of a thread, the rotating
// indices) and the items are found without divisions. A step measured 3.9 us
// for 28x22x18 (13.5 as launches), 15.0 for 160x120x100 with one PML face (20)
// and 47.5 for 204x157x131 with six (62); 24.3 for 256 members of 28x22x18 with a
// source each and 6.5 for 16 with 1000 receivers (42 and 25).
#pragma once

constexpr int kGroup = 256;
constexpr int kResGroups = 3;  // groups of a resident block (80 registers a thread)
struct FastDiv {
    uint32_t d, mul, sh;
    // n / d for 0 <= n < 2^31: mul = ceil(2^(32 + sh) / d) - 2^32, sh = ceil(log2 d)
    __host__ void set(uint32_t v) {
        d = v;
        sh = 0;
        while ((1ull << sh) < v) ++sh;
        mul = (uint32_t)(((1ull << 32) * ((1ull << sh) - v)) / v + 1);
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return (__umulhi(n, mul) + n) >> sh; }
};
struct ResidentGroup {
    int32_t p0, p1, i0, i1, l0, l1;  // PML pressure units, interior items, boundary entries
};
// PML boxes as one run of 4-cell units (x, then rows, then planes; the boxes in
// turn; `total` a member).
struct ResidentBox {
    int32_t x0, y0, z0, axis;
    uint32_t first;
    FastDiv by_units, by_rows;
};
struct ResidentBoxes {
    int32_t n;
    uint32_t total;
    FastDiv by_total;
    ResidentBox box[kMaxPmlBoxes];
    // unit u: member, box and position
    __device__ __forceinline__ const ResidentBox& find(uint32_t u, int* b, int* x, int* y, int* z) const {
        *b = (int)by_total.div(u);
        uint32_t r = u - (uint32_t)*b * total;
        int k = 0;
        while (k + 1 < n && r >= box[k + 1].first) ++k;
        const ResidentBox& q = box[k];
        r -= q.first;
        const uint32_t row = q.by_units.div(r), pl = q.by_rows.div(row);
        *x = q.x0 + 4 * (int)(r - row * q.by_units.d);
        *y = q.y0 + (int)(row - pl * q.by_rows.d);
        *z = q.z0 + (int)pl;
        return q;
    }
};
struct ResidentDev {
    const ResidentGroup* groups;
    // interior items: columns of 4-cell units (nu a row), zc planes each,
    // per_member of them (whole warps) a member
    int32_t nu, ncol, zc, n_zc, per_member;
    FastDiv by_nu, by_ncol, by_member, by_lrs;
    ResidentBoxes press, aux;  // PML units of the pressure and of the auxiliary updates
    const int32_t* order;      // boundary entries by kind, so that few warps mix kinds
    const uint32_t* owned;     // cells of the other roles, pitch / 32 words per row
    int64_t owned_words;       // words from a member's mask to the next one's, 0: one for all
    int32_t sr_groups;         // groups of the sources and receivers
    FastDiv by_rcv;
    unsigned int* bar;
    int32_t steps;
};

// Values x..x+3 of a row as stored (FP16: decoded, unscaled).
template <typename T>
__device__ __forceinline__ void row4(const T* p, float r[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        r[0] = v.x;
        r[1] = v.y;
        r[2] = v.z;
        r[3] = v.w;
    } else {
        const uint2 w = *reinterpret_cast<const uint2*>(p);
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&w.x));
        const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
        r[0] = lo.x;
        r[1] = lo.y;
        r[2] = hi.x;
        r[3] = hi.y;
    }
}

// Interior items i0 + tid, i0 + tid + 256, ... of a group: every cell 1..n-2
// computed as in k_interior, the cells of `owned` not stored. FP16: the
// largest |p^n| of the items, per member, into the scale slot (through
// shared memory when the group's items are of one member).
template <typename T>
__device__ __forceinline__ void interior_role(const StepArgs& a, const StepIdx& I, const ResidentDev& R,
                                              const ResidentGroup& G, int tid, unsigned int* smax) {
    const int64_t pitch = a.g.pitch, plane = a.g.plane;
    const int nx = a.g.nx, nz = a.g.nz;
    T* const pn0 = level_ptr<T>(a, I.wn);
    const T* const pc0 = level_ptr<T>(a, I.wc);
    const T* const po0 = level_ptr<T>(a, I.wo);
    const int wpr = (int)(pitch >> 5);
    const bool one = G.i0 / R.per_member == (G.i1 - 1) / R.per_member;
    unsigned int amax = 0;
    float rc = 1.0f, ro = 1.0f, ic = 1.0f;
    int b_sc = -1;
    bool bad = false;
    for (int it = G.i0 + tid; it < G.i1; it += kGroup) {
        const int b = (int)R.by_member.div((uint32_t)it), r = it - b * R.per_member;
        const int zi = (int)R.by_ncol.div((uint32_t)r);
        const bool valid = zi < R.n_zc;  // items are padded to whole warps per member
        if constexpr (sizeof(T) == 2) {
            if (b != b_sc) {
                const StepScales sc = step_scales(a.f16, b, I.s5);
                rc = sc.s_new * sc.inv_cur;
                ro = sc.s_new * sc.inv_old;
                ic = sc.inv_cur;
                b_sc = b;
            }
        }
        unsigned int cmax = 0;
        if (valid) {
            const int col = r - zi * R.ncol;
            const int yi = (int)R.by_nu.div((uint32_t)col);
            const int x = 4 * (col - yi * R.nu), y = 1 + yi;
            const int z0 = 1 + zi * R.zc, z1 = min(z0 + R.zc, nz - 1);
            const int64_t at = (int64_t)b * a.g.vol + (int64_t)z0 * plane + (int64_t)y * pitch + x;
            const T* pc = pc0 + at;
            const T* po = po0 + at;
            T* pn = pn0 + at;
            const uint32_t* ow =
                R.owned ? R.owned + b * R.owned_words + ((int64_t)z0 * a.g.ny + y) * wpr + (x >> 5) : nullptr;
            unsigned in = 15u;  // cells of the unit inside 1..nx-2
            if (x == 0) in &= 14u;
            if (x + 3 > nx - 2) in &= (1u << (nx - 1 - x)) - 1u;
            const bool lo = x > 0, hi = x + 4 < pitch;
            float zm[4], c[4];
            row4(pc - plane, zm);
            row4(pc, c);
            for (int z = z0; z < z1; ++z, pc += plane, po += plane, pn += plane) {
                float zp[4], ym[4], yp[4], o[4];
                row4(pc + plane, zp);
                row4(pc - pitch, ym);
                row4(pc + pitch, yp);
                row4(po, o);
                const float xm = lo ? lvl<false>(pc - 1, 1.0f) : 0.0f;
                const float xp = hi ? lvl<false>(pc + 4, 1.0f) : 0.0f;
                unsigned st = in;
                if (ow) {
                    st &= ~(*ow >> (x & 31));
                    ow += (int64_t)a.g.ny * wpr;
                }
                float v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float l = q == 0 ? xm : c[q - 1], h = q == 3 ? xp : c[q + 1];
                    if constexpr (sizeof(T) == 4)
                        v[q] = slf_update(a.lambda2, a.cint, h, l, yp[q], ym[q], zp[q], zm[q], c[q], o[q]);
                    else
                        v[q] = slf_update_scaled(a.lambda2, rc, ro, h, l, yp[q], ym[q], zp[q], zm[q], c[q], o[q]);
                }
                if constexpr (sizeof(T) == 4) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) bad |= (in >> q & 1u) && !(fabsf(v[q]) < 1e30f);
                    store4(pn, v, st);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        bad |= (in >> q & 1u) && !f16_finite(v[q]);
                        if (in >> q & 1u) cmax = max(cmax, __float_as_uint(fabsf(c[q])));
                    }
                    store4t(pn, v, st, 1.0f);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    zm[q] = c[q];
                    c[q] = zp[q];
                }
            }
        }
        if constexpr (sizeof(T) == 2) {
            // stored magnitudes scaled to field values (power of two: exact)
            const unsigned int f = __float_as_uint(__uint_as_float(cmax) * ic);
            if (one) {
                amax = max(amax, f);
            } else {
                const unsigned int w = __reduce_max_sync(0xffffffffu, f);
                if (w && (tid & 31) == 0) atomicMax(a.f16.mx + (size_t)b * 5 + slot_back(I.s5, 1), w);
            }
        }
    }
    if constexpr (sizeof(T) == 2) {
        if (one) {
            const unsigned int w = __reduce_max_sync(0xffffffffu, amax);
            if (w && (tid & 31) == 0) atomicMax(smax, w);
        }
    }
    if (__any_sync(0xffffffffu, bad) && (tid & 31) == 0) atomicOr(a.flag, 1);
}

// One boundary entry of the resident kernel, K known at run time.
template <bool REF, typename T>
__device__ __forceinline__ void resident_lrs(const StepArgs& a, const StepIdx& I, int K, int b, int e, int64_t c,
                                             uint32_t info) {
    switch (K) {
        case 1: lrs_update<REF, 1, T, false>(a, I, b, e, c, info, true); break;
        case 2: lrs_update<REF, 2, T, false>(a, I, b, e, c, info, true); break;
        case 3: lrs_update<REF, 3, T, false>(a, I, b, e, c, info, true); break;
        case 4: lrs_update<REF, 4, T, false>(a, I, b, e, c, info, true); break;
        default: lrs_update<REF, 0, T, false>(a, I, b, e, c, info, true); break;
    }
}

// Sources and receivers of all members, item t, t + threads, ... of the source
// pairs (whole warps of them), then of the members' receivers (see src_rcv_role
// for `record`).
template <bool REF, typename T>
__device__ __forceinline__ void src_rcv_items(const StepArgs& a, const StepIdx& I, const ResidentDev& R, int t,
                                              int threads, bool record) {
    const int pairs = (a.sr.n + 31) & ~31, all = pairs + (record ? a.rcv.n * a.batch : 0);
    for (int u = t; u < all; u += threads) {
        if (u >= pairs) {
            const int r = u - pairs, b = (int)R.by_rcv.div((uint32_t)r);
            const float ic = level_scales<T>(a, b, I.s5).ic;
            record_receiver<T>(a, b, r - b * a.rcv.n, I.g - 1, level_ptr<T>(a, I.wc) + (size_t)b * a.g.vol, ic, 1.0f / ic);
        } else if (u < a.sr.n) {
            src_pair<REF, T, false>(a, I, __ldg(a.sr.member + u), u);
        }
    }
    if constexpr (sizeof(T) == 2)
        for (int b = t; b < a.batch; b += threads) a.f16.mx[(size_t)b * 5 + I.s5] = 0u;
}

// PML: 0 none, 1 without psi, 2 with psi.
template <bool REF, int PML, typename T>
__global__ void __launch_bounds__(kResGroups* kGroup, 1)
    k_resident(const __grid_constant__ StepArgs a, const __grid_constant__ ResidentDev R) {
    __shared__ unsigned int smax[kResGroups];
    const int group = (int)threadIdx.x / kGroup, tid = (int)threadIdx.x % kGroup;
    const ResidentGroup G = R.groups[blockIdx.x * kResGroups + group];
    // the last groups (group k: block k mod blocks) take the sources and receivers
    const int sr_at = (kResGroups - 1 - group) * (int)gridDim.x + (int)(gridDim.x - 1 - blockIdx.x);
    StepIdx I = step_at(a, 0);
    const int K = a.lrs.K;
    // the thread's first boundary entry, kept over the steps
    int lb = 0, le = 0, lc = 0;
    uint32_t linfo = 0;
    if (G.l0 + tid < G.l1) {
        lb = (int)R.by_lrs.div((uint32_t)(G.l0 + tid));
        le = __ldg(R.order + (G.l0 + tid - lb * a.lrs.n));
        lc = __ldg(a.lrs.cell + le);
        linfo = __ldg(a.lrs.info + le);
        if ((linfo & kSrcEntry) && !has_source(a, lb, lc)) linfo &= ~kSrcEntry;
    }
    if (threadIdx.x < kResGroups) smax[threadIdx.x] = 0u;
    __syncthreads();
    unsigned int raised = 0;  // the barrier's next target
    for (int s = 0; s < R.steps; ++s) {
        if constexpr (PML > 0) {
            for (int u = G.p0 + tid; u < G.p1; u += kGroup) {
                int b, x, y, z;
                R.press.find((uint32_t)u, &b, &x, &y, &z);
                pml_p_unit<PML == 2, T, false>(a, b, x, y, z, I, level_scales<T>(a, b, I.s5));
            }
        }
        for (int l = G.l0 + tid; l < G.l1; l += kGroup) {
            int b = lb, e = le, c = lc;
            uint32_t info = linfo;
            if (l >= G.l0 + kGroup) {
                b = (int)R.by_lrs.div((uint32_t)l);
                e = __ldg(R.order + (l - b * a.lrs.n));
                c = __ldg(a.lrs.cell + e);
                info = __ldg(a.lrs.info + e);
            }
            resident_lrs<REF, T>(a, I, K, b, e, c, info);
        }
        if (G.i1 > G.i0) interior_role<T>(a, I, R, G, tid, smax + group);
        if (sr_at < R.sr_groups)
            src_rcv_items<REF, T>(a, I, R, sr_at * kGroup + tid, R.sr_groups * kGroup, s > 0);
        if constexpr (sizeof(T) == 2) {
            __syncthreads();
            if (tid == 0 && G.i1 > G.i0 && smax[group]) {
                atomicMax(a.f16.mx + (size_t)(G.i0 / R.per_member) * 5 + slot_back(I.s5, 1), smax[group]);
                smax[group] = 0u;
            }
        }
        if constexpr (PML > 0) {
            raised += gridDim.x;
            if (!grid_barrier(R.bar, raised, a.flag)) return;
            const uint32_t all = R.aux.total * (uint32_t)a.batch;
            for (uint32_t u = blockIdx.x * (kResGroups * kGroup) + threadIdx.x; u < all;
                 u += gridDim.x * (kResGroups * kGroup)) {
                int b, x, y, z;
                const int ax = R.aux.find(u, &b, &x, &y, &z).axis;
                const LevelScales sc = level_scales<T>(a, b, I.s5);
                if (ax == 0) pml_aux_unit<0, PML == 2, T, false>(a, b, x, y, z, I, sc);
                else if (ax == 1) pml_aux_unit<1, PML == 2, T, false>(a, b, x, y, z, I, sc);
                else pml_aux_unit<2, PML == 2, T, false>(a, b, x, y, z, I, sc);
            }
        }
        raised += gridDim.x;
        if (s + 1 < R.steps && !grid_barrier(R.bar, raised, a.flag)) return;
        I = StepIdx{I.g + 1, I.wo, I.wn, I.wc, I.ix == 0 ? K - 1 : I.ix - 1, I.lv ^ 1, I.s5 == 4 ? 0 : I.s5 + 1};
    }
}
