// pcg_gtg_resident.cu -- the SM-resident form of the G^T G preconditioned PCG (pcg_gtg.cu): the same
// iteration, the same arithmetic on every row and the same order of every sum, for systems whose
// bands fit shared memory.
//
// One 512-thread CTA per SM owns a contiguous band of rows and keeps in shared memory the windows
// (band + bandwidth halo) of p', r' and t, and of its own rows z, Ap', the row sums and the FP64
// solution; what is left holds the slots of the band's first slices of A, G and G^T, and the other
// slices stream (A's through a register ring requested ahead of the barrier).  All gathers are from
// shared memory.  Each phase publishes one float per row that a neighbour's
// window covers, because a reader keeps its halo's p and r itself:
//   A   p' = z + beta p over the window (halo z read), Ap', p'.Ap', publish Ap'    -> grid barrier
//   BC  x += alpha p' (FP64), r' = r - alpha Ap' over the window (halo Ap' read), r'.r',
//       t = G r', publish t                                                        -> grid barrier
//   D   z = G^T t (halo t read), r'.z, publish z                                   -> grid barrier
// In the global-memory form each phase was two dependent L2 round trips (slots, then records of the
// own band too: the barrier's acquire empties L1).  us per iteration there -> here, FP32 values:
// 300^2 16.7 -> 11.7, 600^2 26.1 -> 17.3, 900^2 50.9 -> 32.9 (less and less of the matrix fits); 4.3 of
// the 11.7 us are the three grid barriers.
// Shared memory per CTA: 20 bytes a row of the band, 12 a row of the window, then matrix slots.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "../../include/xplus_b200.h"
#include "device_common.cuh"
#include "pcg_device.cuh"
#include "pcg_kernels.cuh"

namespace xplus {
namespace {

using namespace dev;

// The scalar state of one solve, in shared memory: one thread advances it, so that none of it
// occupies registers through the products.
struct GtgState {
    double rz, rr, true_rr, rr_at_replace, tau_true_rr, best, rz_old, pap, alpha, zap;
    float be;          // the next iteration's beta as the vectors use it
    int code;          // kGo, kReplace (refresh the residual, then go on) or kStop
    int status, iterations, replacements, stagnated, mode, stagnant, drop_replace;
    int jac, fell_back, restart;
};
constexpr int kGo = 0, kReplace = 1, kStop = 2;

// Rows of G or G^T times a window x (row w0 first): row_done(row, y) for each of the warp's rows in
// slice order, y = sum_j g_ij x_j in slot order.  Four slices at a time, both chunks of all of them
// requested before any gather (a ring like A's would hold registers through the barriers for rows
// of four slots or fewer).
struct GSlots {
    const float *val, *mval;
    const short *col, *mcol;
    const int2* table;
    int sb, se, sm_end, m0, lane, warp, wpb;
};
template <typename RowDone>
__device__ __forceinline__ void g_rows(const GSlots& m, const float* x, int w0, RowDone&& row_done) {
    constexpr int NB = 4;
    const int lane = m.lane, wpb = m.wpb;
    for (int s0 = m.sb + m.warp; s0 < m.se; s0 += NB * wpb) {
        int w[NB], wmax = 0;
        const float* vp[NB];
        const short* cp[NB];
        unsigned at[NB];
        float y[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            const int s = min(s0 + k * wpb, m.se - 1);  // beyond the band: the last slice again, unused
            const int2 sl = m.table[s - m.sb];
            const bool staged = s < m.sm_end;
            const int off = sl.x - (staged ? m.m0 : 0) + lane * 2;
            w[k] = sl.y;  // at least 2: a G or G^T with a slice without slots does not come here
            wmax = max(wmax, sl.y);
            vp[k] = (staged ? m.mval : m.val) + off;
            cp[k] = (staged ? m.mcol : m.col) + off;
            at[k] = static_cast<unsigned>(__cvta_generic_to_shared(x + (s * 32 + lane - w0)));
            y[k] = 0.0f;
        }
        for (int c = 0; c < wmax; c += 4) {
            float2 v[NB][2];
            unsigned cc[NB][2];
#pragma unroll
            for (int k = 0; k < NB; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int q = min(c + 2 * h, w[k] - 2) * 32;
                    v[k][h] = *reinterpret_cast<const float2*>(vp[k] + q);
                    cc[k][h] = *reinterpret_cast<const unsigned*>(cp[k] + q);
                }
#pragma unroll
            for (int k = 0; k < NB; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (c + 2 * h < w[k]) {
                        y[k] = fmaf(v[k][h].x, raw_gather<2>(at[k], cc[k][h], 0), y[k]);
                        y[k] = fmaf(v[k][h].y, raw_gather<2>(at[k], cc[k][h], 1), y[k]);
                    }
        }
#pragma unroll
        for (int k = 0; k < NB; ++k)
            if (s0 + k * wpb < m.se) row_done((s0 + k * wpb) * 32 + lane, y[k]);
    }
}

template <typename VT, int CHUNK>
__global__ void __launch_bounds__(512, 1) pcg_gtg_res_kernel(PcgArgs a) {
    constexpr int kHaloU = 2;  // halo float4 groups per thread loaded ahead
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double s_red[32 * 4];
    __shared__ double s_tot[4];
    __shared__ int s_flag;
    __shared__ int2 s_slice[3][kGtgResSlices];  // A, G, G^T: {first slot, width}
    __shared__ long long s_clk[6];
    __shared__ int s_exp[2];
    __shared__ GtgState st;
    __shared__ int4 s_stage[3];  // A, G, G^T: first slice not staged, the band's first slot, slots
                                 // staged, byte offset of the staged values
    GridBarrier bar{a.bar, a.err, a.timeout_ns, 0u, a.debug_skip_block};
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    const int per_block = (a.n_slices + gridDim.x - 1) / gridDim.x;
    const int sb = blockIdx.x * per_block;
    const int se = min(a.n_slices, sb + per_block);
    const int r0 = sb * 32;
    const int nb = max(0, se - sb) * 32;
    const int2 win = a.win[blockIdx.x];
    const int w0 = win.x, wn = win.y;  // multiples of 4
    double* xs = reinterpret_cast<double*>(smem_raw);
    float* pw = reinterpret_cast<float*>(xs + nb);
    float* rw = pw + wn;
    float* tw = rw + wn;
    float* zv = tw + wn;
    float* apv = zv + nb;
    float* rsv = apv + nb;
    const float* __restrict__ minv = static_cast<const float*>(a.minv);
    float* z_g = static_cast<float*>(a.z);
    float* ap_g = static_cast<float*>(a.ap);
    float* r_g = static_cast<float*>(a.r);
    float* t_g = static_cast<float*>(a.t);
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    const bool true_mode = a.tau_true_rr >= 0.0;
    for (int k = threadIdx.x; k < se - sb; k += blockDim.x) {
        const long long* sp[3] = {a.slice_ptr, a.g_slice_ptr, a.gt_slice_ptr};
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const long long b0 = sp[m][sb + k];
            s_slice[m][k] = make_int2(static_cast<int>(b0), static_cast<int>((sp[m][sb + k + 1] - b0) >> 5));
        }
    }
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        xs[t] = a.x64[r0 + t];
        rsv[t] = static_cast<const float*>(a.rowsum)[r0 + t];
        zv[t] = 0.0f;
        apv[t] = 0.0f;
    }
    for (int t = threadIdx.x; t < wn; t += blockDim.x) pw[t] = rw[t] = tw[t] = 0.0f;
    // the rows of this band that another CTA's window covers: [r0, exp_lo) and [exp_hi, r0 + nb)
    if (warp == 0) {
        int lo = r0, hi = r0 + nb;
        for (int c = lane; c < static_cast<int>(gridDim.x); c += 32) {
            const int2 wc = a.win[c];
            if (wc.y <= 0) continue;
            if (c < static_cast<int>(blockIdx.x)) lo = max(lo, wc.x + wc.y);
            else if (c > static_cast<int>(blockIdx.x)) hi = min(hi, wc.x);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = max(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = min(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            s_exp[0] = min(lo, r0 + nb);
            s_exp[1] = max(hi, r0);
        }
    }
    // slots of the first `staged` slices of A, G and G^T
    SlotRing<VT, CHUNK, 2> ring_a;
    // Where the slots are, made afresh at each use so that none of it is kept in registers.
    auto bind_a = [&]() {
        const int4 d = s_stage[0];
        const int tid = thread_index();
        const VT* mval = reinterpret_cast<const VT*>(smem_raw + d.w);
        ring_a.val = static_cast<const VT*>(a.val);
        ring_a.col = static_cast<const short*>(a.col);
        ring_a.mval = mval;
        ring_a.mcol = reinterpret_cast<const short*>(mval + d.z);
        ring_a.table = s_slice[0];
        ring_a.sb = sb;
        ring_a.se = se;
        ring_a.sm_end = d.x;
        ring_a.m0 = d.y;
        ring_a.wpb = static_cast<int>(blockDim.x >> 5);
        ring_a.lane = tid & 31;
        return tid >> 5;
    };
    auto prime_a = [&]() { ring_a.prime_all(bind_a()); };
    auto slots_of = [&](int m, const void* val, const short* col) {
        const int4 d = s_stage[m];
        const int tid = thread_index();
        const float* mval = reinterpret_cast<const float*>(smem_raw + d.w);
        return GSlots{static_cast<const float*>(val), mval, col, reinterpret_cast<const short*>(mval + d.z), s_slice[m], sb,
                      se, d.x, d.y, tid & 31, tid >> 5, static_cast<int>(blockDim.x >> 5)};
    };
    auto g_slots = [&]() { return slots_of(1, a.g_val, a.g_col16); };
    auto t_slots = [&]() { return slots_of(2, a.gt_val, a.gt_col16); };
    {
        const int ns = max(0, se - sb);
        auto slots = [&](const long long* sp, int k) { return ns > 0 ? sp[sb + k] - sp[sb] : 0LL; };
        auto bytes = [&](int k) {
            return slots(a.slice_ptr, k) * static_cast<long long>(sizeof(VT) + 2) +
                   (slots(a.g_slice_ptr, k) + slots(a.gt_slice_ptr, k)) * 6;
        };
        const long long room = a.smem_bytes - (20LL * nb + 12LL * wn);
        int lo = 0, hi = ns;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (bytes(mid) <= room) lo = mid;
            else hi = mid - 1;
        }
        const int staged = lo;
        unsigned char* next = reinterpret_cast<unsigned char*>(rsv + nb);
        // every slice is a multiple of 64 slots, so each part is whole 16-byte groups
        auto stage = [&](int m, const long long* sp, auto* val, const short* col) {
            using V = std::remove_const_t<std::remove_pointer_t<decltype(val)>>;
            const long long m0 = ns > 0 ? sp[sb] : 0, ms = slots(sp, staged);
            V* mval = reinterpret_cast<V*>(next);
            short* mcol = reinterpret_cast<short*>(mval + ms);
            next += ms * static_cast<long long>(sizeof(V) + 2);
            const uint4* gv = reinterpret_cast<const uint4*>(val + m0);
            const uint4* gc = reinterpret_cast<const uint4*>(col + m0);
            const long long nv = ms * static_cast<long long>(sizeof(V)) / 16, nc = ms * 2 / 16;
            for (long long i = threadIdx.x; i < nv; i += blockDim.x) reinterpret_cast<uint4*>(mval)[i] = __ldg(gv + i);
            for (long long i = threadIdx.x; i < nc; i += blockDim.x) reinterpret_cast<uint4*>(mcol)[i] = __ldg(gc + i);
            if (threadIdx.x == 0)
                s_stage[m] = make_int4(sb + staged, static_cast<int>(m0), static_cast<int>(ms),
                                       static_cast<int>(reinterpret_cast<unsigned char*>(mval) - smem_raw));
        };
        stage(0, a.slice_ptr, static_cast<const VT*>(a.val), static_cast<const short*>(a.col));
        stage(1, a.g_slice_ptr, static_cast<const float*>(a.g_val), a.g_col16);
        stage(2, a.gt_slice_ptr, static_cast<const float*>(a.gt_val), a.gt_col16);
    }
    // phase clock (per CTA, thread 0): {A work, grid-barrier waits, BC work, D work}
    if (threadIdx.x == 0) {
        for (int k = 0; k < 5; ++k) s_clk[k] = 0;
        s_clk[5] = globaltimer_ns();
        if (lead) a.out->t_start_ns = s_clk[5];
    }
    __syncthreads();
    const int exp_lo = s_exp[0], exp_hi = s_exp[1];
    auto exported = [&](int row) { return row < exp_lo || row >= exp_hi; };
    auto clock = [&](int slot) {
        if (threadIdx.x == 0) {
            const long long t = globaltimer_ns();
            s_clk[slot] += t - s_clk[5];
            s_clk[5] = t;
        }
    };
    int bank = 0;
    auto next_bank = [&]() {
        double* b = a.partial + static_cast<size_t>(bank) * 4 * gridDim.x;
        bank ^= 1;
        return b;
    };
    double* cur_bank = nullptr;

    // The halo of the window [w0, w0 + wn) without the band, in float4 groups: group u < nlo lies
    // below the band, the others above it.
    const int nlo = (r0 - w0) >> 2;
    const int hi0 = (r0 + nb - w0) >> 2;
    const int nh = nlo + (wn >> 2) - hi0;
    const int hbd = static_cast<int>(blockDim.x);
    auto qof = [&](int u) { return u < nlo ? u : hi0 + (u - nlo); };
    float4 hv[kHaloU];
    // the first groups of src's halo into registers, right after the barrier that made it final
    auto issue_halo = [&](const float* src) {
        const float4* s4 = reinterpret_cast<const float4*>(src + w0);
#pragma unroll
        for (int v = 0; v < kHaloU; ++v) {
            const int u = threadIdx.x + v * hbd;
            hv[v] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (u < nh) hv[v] = s4[qof(u)];
        }
    };
    // the halo of the window dst: f(what it holds, src's value)
    auto fill_halo = [&](const float* src, float* dst, auto&& f) {
        const float4* s4 = reinterpret_cast<const float4*>(src + w0);
        float4* d4 = reinterpret_cast<float4*>(dst);
        auto one = [&](int u, const float4& h) {
            float4 d = d4[qof(u)];
            d.x = f(d.x, h.x);
            d.y = f(d.y, h.y);
            d.z = f(d.z, h.z);
            d.w = f(d.w, h.w);
            d4[qof(u)] = d;
        };
#pragma unroll
        for (int v = 0; v < kHaloU; ++v) {
            const int u = threadIdx.x + v * hbd;
            if (u < nh) one(u, hv[v]);
        }
#pragma unroll 2
        for (int u = threadIdx.x + kHaloU * hbd; u < nh; u += hbd) one(u, s4[qof(u)]);
    };
    auto take = [](float, float h) { return h; };

    // breakdown test that opens iteration k (kernels/cuper_pcg_control_kernel.cpp:1069-1235)
    auto open_iteration = [&](int k) {
        if (k >= a.max_iters) {
            st.code = kStop;  // status stays XPLUS_MAX_ITER
        } else if (bad(st.rz) || bad(st.rr) || fabs(st.rz) <= kBreakdownEps) {
            st.status = XPLUS_BREAKDOWN;
            st.code = kStop;
        }
    };
    // ends the last iteration (rep: after a refresh): convergence, beta, the next one's start
    auto finish = [&](bool rep) {
        st.code = kStop;
        const int it = st.iterations - 1;
        if (lead && a.trace && it < a.trace_cap) {
            double* tr = a.trace + 5 * static_cast<size_t>(it);
            tr[0] = st.alpha;
            tr[1] = st.rz / st.rz_old;
            tr[2] = st.rz;
            tr[3] = st.rr;
            tr[4] = sqrt(st.rr > 0.0 ? st.rr : 0.0);
        }
        if (true_mode ? (rep && st.true_rr <= st.tau_true_rr) : (st.rr <= a.tau_rr)) {
            st.status = XPLUS_CONVERGED;
            return;
        }
        if (st.stagnated && st.jac) return;
        if (fabs(st.rz_old) <= kBreakdownEps) {
            st.status = XPLUS_BREAKDOWN;
            return;
        }
        ReplacePolicy pol(a.restart_on_replace, 0.0);
        pol.mode = st.mode;
        const double beta =
            st.restart ? 0.0 : pol.beta(rep, st.drop_replace != 0, st.rz, st.rz_old, st.zap, st.pap);
        if (bad(beta)) {
            st.status = XPLUS_BREAKDOWN;
            return;
        }
        st.be = static_cast<float>(beta);
        st.code = kGo;
        open_iteration(it + 1);
    };
    // after the last reduction of iteration it: r.z and r.r in s_tot
    auto advance = [&](int it) {
        st.code = kStop;
        st.rz_old = st.rz;
        st.rz = s_tot[0];
        st.rr = s_tot[1];
        st.iterations = it + 1;
        if (bad(st.rz) || bad(st.rr)) {
            st.status = XPLUS_BREAKDOWN;
            return;
        }
        bool do_replace = false, drop_replace = false;
        st.restart = 0;
        if (true_mode) {
            if (st.rr <= st.tau_true_rr) do_replace = drop_replace = true;
            if (a.replace_every > 0 && st.iterations % a.replace_every == 0) do_replace = true;
            if (a.replace_drop > 0.0 && st.rr <= a.replace_drop * st.rr_at_replace) do_replace = drop_replace = true;
        }
        // Jacobi fallback: the learned preconditioner stagnated or used up its iterations
        if (!st.jac && (st.stagnated || (a.g_fallback_iters > 0 && st.iterations >= a.g_fallback_iters))) {
            st.jac = 1;
            st.fell_back = st.iterations;
            st.stagnated = 0;
            st.stagnant = 0;
            do_replace = true;
            st.restart = 1;
        }
        st.drop_replace = drop_replace;
        st.zap = 0.0;
        if (do_replace) st.code = kReplace;
        else finish(false);
    };
    // after a refresh (st.rz, rr, true_rr, zap set): the first one starts the solve
    auto refreshed = [&](bool init) {
        if (init) {
            st.rr_at_replace = st.rr;
            const ReplacePolicy pol(a.restart_on_replace, st.true_rr);
            st.mode = pol.mode;
            st.stagnant = pol.stagnant;
            st.best = pol.best;
            st.code = kGo;
            if (true_mode ? (st.true_rr <= st.tau_true_rr) : (st.rr <= a.tau_rr)) {
                st.status = XPLUS_CONVERGED;
                st.code = kStop;
            } else {
                open_iteration(0);
            }
            return;
        }
        ++st.replacements;
        st.rr_at_replace = st.rr;
        ReplacePolicy pol(a.restart_on_replace, st.best);
        pol.mode = st.mode;
        pol.stagnant = st.stagnant;
        if (st.restart) {
            // the switch to Jacobi: the refreshed residual is the new reference
            if (a.restart_on_replace == 3 && pol.mode == 2 && st.true_rr > 4.0 * pol.best) pol.mode = 1;
            pol.best = st.true_rr;
        } else if (pol.after(a.restart_on_replace, st.true_rr, a.stag_factor, a.stag_window)) {
            st.stagnated = 1;
        }
        st.mode = pol.mode;
        st.stagnant = pol.stagnant;
        st.best = pol.best;
        finish(true);
    };

    if (threadIdx.x == 0) {
        st.pap = st.alpha = st.zap = st.rz_old = 0.0;
        st.be = 0.0f;
        st.status = XPLUS_MAX_ITER;
        st.iterations = st.replacements = st.stagnated = st.drop_replace = st.jac = st.restart = 0;
        st.fell_back = -1;
        st.code = kReplace;
    }
    __syncthreads();
    for (int it = 0;; ++it) {
        if (st.code == kReplace) {
            // ---- FP64 residual r = b - A x (stored rounded) and its preconditioning; the first
            //      one (it = 0) also sums ||b||^2 ----
            const bool init = it == 0, jac = st.jac != 0;
            if (!init) {
                for (int t = threadIdx.x; t < nb; t += blockDim.x) a.x64[r0 + t] = xs[t];
                if (!bar.sync(&s_flag)) return;
            }
            {
                double acc[4] = {0.0, 0.0, 0.0, 0.0};
                for (int s = sb + warp; s < se; s += wpb) {
                    const int row = s * 32 + lane;
                    const double y = row_fp64<VT, float, CHUNK, true, short>(a, s, lane, row);
                    const double bv = a.b64[row];
                    const double rt = bv - y;
                    if (init) acc[3] += bv * bv;
                    const float rv = static_cast<float>(rt);
                    rw[row - w0] = rv;
                    r_g[row] = rv;
                    if (jac) {
                        const float z_ = minv[row] * rv;
                        zv[row - r0] = z_;
                        z_g[row] = z_;
                        if (!init) acc[3] += static_cast<double>(z_) * static_cast<double>(apv[row - r0]);
                        acc[0] += static_cast<double>(rv) * static_cast<double>(z_);
                    }
                    acc[1] += static_cast<double>(rv) * static_cast<double>(rv);
                    acc[2] += rt * rt;
                }
                cur_bank = next_bank();
                publish<4>(acc, s_red, cur_bank);
            }
            if (!bar.sync(&s_flag)) return;
            issue_halo(r_g);
            grid_totals(cur_bank, 4, s_tot);
            if (threadIdx.x == 0) {
                st.rz = s_tot[0];
                st.rr = s_tot[1];
                st.true_rr = s_tot[2];
                if (init) {
                    st.tau_true_rr = a.tau2_rel > 0.0 ? a.tau2_rel * s_tot[3] : a.tau_true_rr;
                    if (lead) a.out->bb = s_tot[3];
                } else {
                    st.zap = s_tot[3];
                }
            }
            fill_halo(r_g, rw, take);
            if (!jac) {
                __syncthreads();
                g_rows(g_slots(), rw, w0, [&](int row, float y) {
                    tw[row - w0] = y;
                    if (exported(row)) t_g[row] = y;
                });
                if (!bar.sync(&s_flag)) return;
                issue_halo(t_g);
                fill_halo(t_g, tw, take);
                double acc[2] = {0.0, 0.0};
                __syncthreads();
                g_rows(t_slots(), tw, w0, [&](int row, float y) {
                    zv[row - r0] = y;
                    z_g[row] = y;
                    acc[0] += static_cast<double>(rw[row - w0]) * static_cast<double>(y);
                    if (!init) acc[1] += static_cast<double>(y) * static_cast<double>(apv[row - r0]);
                });
                cur_bank = next_bank();
                publish<2>(acc, s_red, cur_bank);
                if (!bar.sync(&s_flag)) return;
                grid_totals(cur_bank, 2, s_tot);
                if (threadIdx.x == 0) {
                    st.rz = s_tot[0];
                    if (!init) st.zap = s_tot[1];
                }
            }
            issue_halo(z_g);
            if (threadIdx.x == 0) refreshed(init);
            prime_a();
            __syncthreads();
            if (st.code == kStop) break;
        }
        // ---- A: p' over the window, Ap', p'.Ap' ----
        {
            const float be = st.be;
            float4* pw4 = reinterpret_cast<float4*>(pw + (r0 - w0));
            const float4* z4 = reinterpret_cast<const float4*>(zv);
            for (int t4 = threadIdx.x; t4 < (nb >> 2); t4 += blockDim.x) {
                float4 p = pw4[t4];
                const float4 z = z4[t4];
                p.x = node_pnew(z.x, be, p.x);
                p.y = node_pnew(z.y, be, p.y);
                p.z = node_pnew(z.z, be, p.z);
                p.w = node_pnew(z.w, be, p.w);
                pw4[t4] = p;
            }
            fill_halo(z_g, pw, [be](float p, float z) { return node_pnew(z, be, p); });
            __syncthreads();
            double acc[1] = {0.0};
            ring_a.run(bind_a(), pw, w0, [&](int row, float pi, float y) {
                const int t = row - r0;
                const float ap_ = y * a.val_scale + rsv[t] * pi;
                apv[t] = ap_;
                if (exported(row)) ap_g[row] = ap_;
                acc[0] += static_cast<double>(pi) * static_cast<double>(ap_);
            });
            cur_bank = next_bank();
            publish<1>(acc, s_red, cur_bank);
        }
        clock(0);
        if (!bar.sync(&s_flag)) return;
        clock(1);
        issue_halo(ap_g);
        grid_totals(cur_bank, 1, s_tot);
        const double pap = s_tot[0];
        const double alpha = st.rz / pap;
        const bool broken = bad(pap) || fabs(pap) <= kBreakdownEps || bad(alpha);
        if (threadIdx.x == 0) {
            st.pap = pap;
            if (broken) st.status = XPLUS_BREAKDOWN;
            if (!(bad(pap) || fabs(pap) <= kBreakdownEps)) st.alpha = alpha;
        }
        if (broken) break;
        // ---- BC: x, r', r'.r'; t = G r' (or z = M^-1 r' with Jacobi) ----
        const bool jac = st.jac != 0;
        {
            double acc[2] = {0.0, 0.0};
            const float nal = -static_cast<float>(alpha);
#pragma unroll 2
            for (int s = sb + warp; s < se; s += wpb) {
                const int row = s * 32 + lane, t = row - r0;
                const float pv = pw[row - w0];
                xs[t] = xs[t] + alpha * static_cast<double>(pv);
                const float rn = __fmaf_rn(nal, apv[t], rw[row - w0]);
                rw[row - w0] = rn;
                if (jac) {
                    const float z_ = minv[row] * rn;
                    zv[t] = z_;
                    if (exported(row)) z_g[row] = z_;
                    acc[0] += static_cast<double>(rn) * static_cast<double>(z_);
                }
                acc[1] += static_cast<double>(rn) * static_cast<double>(rn);
            }
            if (!jac) {
                fill_halo(ap_g, rw, [nal](float r, float ap_) { return __fmaf_rn(nal, ap_, r); });
                __syncthreads();
                g_rows(g_slots(), rw, w0, [&](int row, float y) {
                    tw[row - w0] = y;
                    if (exported(row)) t_g[row] = y;
                });
                clock(2);
                if (!bar.sync(&s_flag)) return;
                clock(1);
                issue_halo(t_g);
                // ---- D: z = G^T t, r'.z ----
                fill_halo(t_g, tw, take);
                __syncthreads();
                g_rows(t_slots(), tw, w0, [&](int row, float y) {
                    zv[row - r0] = y;
                    if (exported(row)) z_g[row] = y;
                    acc[0] += static_cast<double>(rw[row - w0]) * static_cast<double>(y);
                });
            }
            cur_bank = next_bank();
            publish<2>(acc, s_red, cur_bank);
        }
        clock(jac ? 2 : 3);
        prime_a();
        if (!bar.sync(&s_flag)) return;
        clock(1);
        issue_halo(z_g);
        grid_totals(cur_bank, 2, s_tot);
        if (threadIdx.x == 0) advance(it);
        __syncthreads();
        if (st.code == kStop) break;
    }
    __syncthreads();
    if (threadIdx.x == 0 && st.status == XPLUS_MAX_ITER && !true_mode && st.rr <= a.tau_rr) st.status = XPLUS_CONVERGED;

    // exit: x to global memory, then its FP64 true residual
    for (int t = threadIdx.x; t < nb; t += blockDim.x) a.x64[r0 + t] = xs[t];
    if (!bar.sync(&s_flag)) return;
    {
        double acc[1] = {0.0};
        for (int s = sb + warp; s < se; s += wpb) {
            const int row = s * 32 + lane;
            const double y = row_fp64<VT, float, CHUNK, true, short>(a, s, lane, row);
            const double rt = a.b64[row] - y;
            acc[0] += rt * rt;
        }
        cur_bank = next_bank();
        publish<1>(acc, s_red, cur_bank);
    }
    if (threadIdx.x == 0 && a.block_clk)
        for (int k = 0; k < 4; ++k) a.block_clk[4 * static_cast<size_t>(blockIdx.x) + k] = s_clk[k];
    if (!bar.sync(&s_flag)) return;
    if (blockIdx.x == 0) {
        grid_totals(cur_bank, 1, s_tot);
        if (threadIdx.x == 0) {
            PcgOut* o = a.out;
            o->status = st.status;
            o->iterations = st.iterations;
            o->replacements = st.replacements;
            o->stagnated = st.stagnated;
            o->rz = st.rz;
            o->rr = st.rr;
            o->pap = st.pap;
            o->alpha = st.alpha;
            o->true_rr = s_tot[0];
            o->reserved = static_cast<double>(st.fell_back);
            o->t_end_ns = globaltimer_ns();
            for (int k = 0; k < 4; ++k) o->t_phase[k] = s_clk[k];
        }
    }
}

using GtgKernel = void (*)(PcgArgs);

template <typename VT>
GtgKernel pick_chunk(int chunk) {
    return chunk == 4 ? pcg_gtg_res_kernel<VT, 4> : (chunk == 2 ? pcg_gtg_res_kernel<VT, 2> : nullptr);
}

GtgKernel pick(const KernelKey& k) {
    if (k.xt != XPLUS_F32 || !k.diag || !k.idx16) return nullptr;
    switch (k.vt) {
        case XPLUS_F32: return pick_chunk<float>(k.chunk);
        case XPLUS_F16: return pick_chunk<__half>(k.chunk);
        case XPLUS_BF16: return pick_chunk<__nv_bfloat16>(k.chunk);
    }
    return nullptr;
}

// thread per SELL row of a chunk-2 image whose rows' columns lie within 32767 of them
__global__ void k_gtg_pack16(const long long* __restrict__ slice_ptr, int n_pad, const int* __restrict__ col,
                             short* __restrict__ col16) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n_pad) return;
    const long long b0 = slice_ptr[row >> 5];
    const int w = static_cast<int>((slice_ptr[(row >> 5) + 1] - b0) >> 5);
    for (int j = 0; j < w; j += 2) {
        const long long at = b0 + static_cast<long long>(j) * 32 + (row & 31) * 2;
        const int2 c = *reinterpret_cast<const int2*>(col + at);
        *reinterpret_cast<short2*>(col16 + at) = make_short2(static_cast<short>(c.x - row), static_cast<short>(c.y - row));
    }
}

// The window of band blockIdx.x over the columns of A (offsets from the row), G and G^T.  The three
// patterns differ where A stores one of (i, j) and (j, i) alone: G^T's row j then reaches a column
// that A's row j does not have.  *empty: some slice of G or G^T has no slots.
__global__ void __launch_bounds__(256) k_gtg_windows(GtgPatterns m, int n_slices, int n_pad, int per,
                                                     int2* __restrict__ win, int* __restrict__ empty) {
    __shared__ int s_lo, s_hi;
    const int sb = blockIdx.x * per, se = min(n_slices, sb + per);
    if (threadIdx.x == 0) {
        s_lo = sb * 32;
        s_hi = se * 32;
    }
    __syncthreads();
    int lo = sb * 32, hi = se * 32;
    for (int s = sb + static_cast<int>(threadIdx.x >> 5); s < se; s += 8) {
        const long long b0 = m.slice_ptr[s];
        const int slots = static_cast<int>(m.slice_ptr[s + 1] - b0);
        for (int q = threadIdx.x & 31; q < slots; q += 32) {
            const int c = s * 32 + (q / m.chunk) % 32 + m.col16[b0 + q];
            lo = min(lo, c);
            hi = max(hi, c + 1);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const long long* __restrict__ sp = k == 0 ? m.g_slice_ptr : m.gt_slice_ptr;
            const int* __restrict__ col = k == 0 ? m.g_col : m.gt_col;
            const long long e = sp[s + 1];
            if (sp[s] == e) *empty = 1;
            for (long long q = sp[s] + (threadIdx.x & 31); q < e; q += 32) {
                lo = min(lo, col[q]);
                hi = max(hi, col[q] + 1);
            }
        }
    }
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
    __syncthreads();
    if (threadIdx.x == 0) {
        const int w0 = s_lo & ~3;
        win[blockIdx.x] = se > sb ? make_int2(w0, min(n_pad, (s_hi + 3) & ~3) - w0) : make_int2(0, 0);
    }
}

}  // namespace

bool gtg_res_supported(const KernelKey& k) { return pick(k) != nullptr; }

size_t gtg_res_vector_bytes(int rows, int window) {
    return 20 * static_cast<size_t>(rows) + 12 * static_cast<size_t>(window);
}

cudaError_t gtg_res_prepare(const KernelKey& k, int device, int grid, size_t vector_bytes, size_t matrix_bytes,
                            bool* fits, size_t* smem_bytes) {
    *fits = false;
    GtgKernel f = pick(k);
    if (!f) return cudaSuccess;
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa{};
    e = cudaFuncGetAttributes(&fa, f);
    if (e != cudaSuccess) return e;
    if (vector_bytes + fa.sharedSizeBytes > static_cast<size_t>(optin)) return cudaSuccess;
    // the opt-in is the kernel's, shared by all handles: always the most a launch may ask for
    const size_t limit = static_cast<size_t>(optin) - fa.sharedSizeBytes;
    e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(limit));
    if (e != cudaSuccess) return e;
    const size_t want = std::min(limit, vector_bytes + matrix_bytes);
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, 512, want);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    *smem_bytes = want;
    *fits = grid <= per_sm * sms;  // the grid is the global-memory kernel's, all of it must be resident
    return cudaSuccess;
}

cudaError_t gtg_res_launch(const KernelKey& k, const PcgArgs& a, int grid, size_t smem_bytes, cudaStream_t s) {
    GtgKernel f = pick(k);
    if (!f) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, f, a);
}

cudaError_t gtg_pack16(const long long* slice_ptr, int n_slices, const int* col, short* col16, cudaStream_t s) {
    k_gtg_pack16<<<(n_slices * 32 + 255) / 256, 256, 0, s>>>(slice_ptr, n_slices * 32, col, col16);
    return cudaGetLastError();
}

cudaError_t gtg_windows(const GtgPatterns& m, int n_slices, int n_pad, int grid, int2* win, int* empty, cudaStream_t s) {
    k_gtg_windows<<<grid, 256, 0, s>>>(m, n_slices, n_pad, (n_slices + grid - 1) / grid, win, empty);
    return cudaGetLastError();
}

}  // namespace xplus
