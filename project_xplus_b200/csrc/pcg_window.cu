// pcg_window.cu -- the persistent Jacobi-PCG of pcg_kernels.cu (FP32 vectors, row-sum form, int16
// column offsets) with the search direction's window in shared memory: for systems whose vectors do
// not fit the SM-resident kernel but whose band + halo of one vector does (128^3: 189 KB).
//
// Same arithmetic on every row and the same order of every sum as pcg_persistent_kernel, two grid
// barriers per iteration:
//   phase A  p' = z + beta p over the window [w0, w0 + wn) (a CTA keeps its halo's p itself, so only
//            z is exchanged), Ap' gathered from shared memory while the matrix streams through a
//            register ring, p'.Ap'                                            -> grid barrier
//   phase B  x += alpha p' (FP64), r -= alpha Ap', z = M^-1 r, r.z and r.r     -> grid barrier
// The global-memory form gathers {z, p} records through L1 behind each slot load: two dependent
// round trips for 16 warps, and 8 bytes per row where 4 are enough.
//
// The matrix (200 MB at 128^3) streams past L1 and through L2 at its default priority, beside the
// vectors (67 MB), and no part of L2 is set aside for it: with the persisting set-aside that the
// global-memory form asks for, 128^3 takes 73.5 us per iteration instead of 50.4 (104^3 reads 114 MB
// of DRAM per iteration, its 107 MB of slots and little else).  us per iteration, global-memory form
// -> here: 128^3 FP32 95.7 -> 50.0, BF16 100.6 -> 51.8; 100^3 FP32 46.4 -> 27.8, BF16 40.7 -> 29.0;
// 1400^2 FP32 69.4 -> 32.7.  Of the 50 (median CTA): window and product 36 (DRAM: 200 MB at 6.5 TB/s
// is 31), barriers and totals 6.6, phase B 6.8.
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

constexpr int kWinSlices = 1024;  // slice table capacity per CTA

template <typename VT, int CHUNK>
__global__ void __launch_bounds__(512, 1) pcg_window_kernel(PcgArgs a) {
    extern __shared__ __align__(16) float pw[];  // p' of the window [w0, w0 + wn)
    __shared__ double s_red[32 * 4];
    __shared__ double s_tot[4];
    __shared__ int s_flag;
    __shared__ int2 s_slice[kWinSlices];  // {first slot, width} of the block's slices
    __shared__ long long s_clk[6];
    GridBarrier bar{a.bar, a.err, a.timeout_ns, 0u, a.debug_skip_block};
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    const int per_block = (a.n_slices + gridDim.x - 1) / gridDim.x;
    const int sb = blockIdx.x * per_block;
    const int se = min(a.n_slices, sb + per_block);
    const int2 win = a.win[blockIdx.x];
    const int w0 = win.x, wn = win.y;  // multiples of 4
    const float* __restrict__ minv = static_cast<const float*>(a.minv);
    const float* __restrict__ rowsum = static_cast<const float*>(a.rowsum);
    float* z = static_cast<float*>(a.rec);  // M^-1 r, what the neighbours' windows need of a row
    float* r = static_cast<float*>(a.r);
    float* ap = static_cast<float*>(a.ap);
    for (int t = threadIdx.x; t < wn; t += blockDim.x) pw[t] = 0.0f;
    SlotRing<VT, CHUNK, 2, true> ring;
    ring.val = ring.mval = static_cast<const VT*>(a.val);
    ring.col = ring.mcol = static_cast<const short*>(a.col);
    ring.table = s_slice;
    ring.sb = ring.sm_end = sb;  // no slots in shared memory
    ring.se = se;
    ring.m0 = 0;
    ring.wpb = wpb;
    ring.lane = lane;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    const bool true_mode = a.tau_true_rr >= 0.0;
    for (int k = threadIdx.x; k < se - sb; k += blockDim.x) {
        const long long b0 = a.slice_ptr[sb + k];
        s_slice[k] = make_int2(static_cast<int>(b0), static_cast<int>((a.slice_ptr[sb + k + 1] - b0) >> 5));
    }
    // phase clock of block 0 (globaltimer, in shared memory): work of phase A / B incl. the
    // block reduction, and the grid-barrier waits after each.  Slot 5 is the last mark.
    if (threadIdx.x == 0) {
        for (int k = 0; k < 5; ++k) s_clk[k] = 0;
        s_clk[5] = globaltimer_ns();
        if (lead) a.out->t_start_ns = s_clk[5];
    }
    __syncthreads();
    auto clock = [&](int slot) {
        if (threadIdx.x == 0) {
            const long long t = globaltimer_ns();
            s_clk[slot] += t - s_clk[5];
            s_clk[5] = t;
        }
    };
    // Two banks of 4 partial slots: consecutive publishes alternate banks, so a block that
    // runs ahead can never overwrite partials another block has not read yet (a barrier
    // separates any two publishes, and a bank is reused only two publishes later).
    int bank = 0;
    auto next_bank = [&]() {
        double* b = a.partial + static_cast<size_t>(bank) * 4 * gridDim.x;
        bank ^= 1;
        return b;
    };
    double* cur_bank = nullptr;

    // ---- residual phase: r = b - A x in FP64, stored rounded, z = M^-1 r; partials r.z, r.r, true r.r, and ||b||^2 (init) or z.Ap' ----
    auto residual_phase = [&](bool init) {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int s = sb + warp; s < se; s += wpb) {
            const int row = s * 32 + lane;
            const double y = row_fp64<VT, float, CHUNK, true, short>(a, s, lane, row);
            const double bv = a.b64[row];
            const double rt = bv - y;
            const float rv = static_cast<float>(rt);
            const float zv = minv[row] * rv;
            // slot 3: ||b||^2 in the first pass, z_new . Ap' at a replacement
            acc[3] += init ? bv * bv : static_cast<double>(zv) * static_cast<double>(ap[row]);
            r[row] = rv;
            z[row] = zv;
            acc[0] += static_cast<double>(rv) * static_cast<double>(zv);
            acc[1] += static_cast<double>(rv) * static_cast<double>(rv);
            acc[2] += rt * rt;
        }
        cur_bank = next_bank();
        publish<4>(acc, s_red, cur_bank);
    };

    residual_phase(true);
    if (!bar.sync(&s_flag)) return;
    grid_totals(cur_bank, 4, s_tot);
    double rz = s_tot[0], rr = s_tot[1], true_rr = s_tot[2];
    const double tau_true_rr = a.tau2_rel > 0.0 ? a.tau2_rel * s_tot[3] : a.tau_true_rr;
    if (lead) a.out->bb = s_tot[3];
    double rr_at_replace = rr;
    double pap = 0.0, alpha = 0.0, beta = 0.0;
    int status = XPLUS_MAX_ITER, iterations = 0, replacements = 0, stagnated = 0;
    ReplacePolicy pol(a.restart_on_replace, true_rr);
    const bool converged_now = true_mode ? (true_rr <= tau_true_rr) : (rr <= a.tau_rr);
    clock(4);

    if (converged_now) {
        status = XPLUS_CONVERGED;
    } else {
        for (int it = 0; it < a.max_iters; ++it) {
            if (bad(rz) || bad(rr) || fabs(rz) <= kBreakdownEps) {
                status = XPLUS_BREAKDOWN;
                break;
            }
            // ---- phase A: p' = z + beta p over the window, Ap', p'.Ap' ----
            {
                ring.prime(warp);  // the first slots travel meanwhile
                const float be = static_cast<float>(beta);
                const float4* z4 = reinterpret_cast<const float4*>(z + w0);
                float4* p4 = reinterpret_cast<float4*>(pw);
                constexpr int U = 4;  // loads of one thread in flight
                for (int u0 = threadIdx.x; u0 < (wn >> 2); u0 += U * blockDim.x) {
                    float4 zv[U];
#pragma unroll
                    for (int v = 0; v < U; ++v) {
                        const int u = u0 + v * static_cast<int>(blockDim.x);
                        zv[v] = u < (wn >> 2) ? z4[u] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
#pragma unroll
                    for (int v = 0; v < U; ++v) {
                        const int u = u0 + v * static_cast<int>(blockDim.x);
                        if (u >= (wn >> 2)) break;
                        float4 p = p4[u];
                        p.x = node_pnew(zv[v].x, be, p.x);
                        p.y = node_pnew(zv[v].y, be, p.y);
                        p.z = node_pnew(zv[v].z, be, p.z);
                        p.w = node_pnew(zv[v].w, be, p.w);
                        p4[u] = p;
                    }
                }
                __syncthreads();
                double acc[1] = {0.0};
                ring.run(warp, pw, w0, [&](int row, float pi, float y) {
                    const float yy = y * a.val_scale + rowsum[row] * pi;
                    ap[row] = yy;
                    acc[0] += static_cast<double>(pi) * static_cast<double>(yy);
                });
                cur_bank = next_bank();
                publish<1>(acc, s_red, cur_bank);
            }
            clock(0);
            if (!bar.sync(&s_flag)) return;
            grid_totals(cur_bank, 1, s_tot);
            clock(1);
            pap = s_tot[0];
            if (bad(pap) || fabs(pap) <= kBreakdownEps) {
                status = XPLUS_BREAKDOWN;
                break;
            }
            const double rz_old = rz;
            alpha = rz / pap;
            if (bad(alpha)) {
                status = XPLUS_BREAKDOWN;
                break;
            }
            // ---- phase B: x, r, z and the two dots; four slices per step so the loads of all are
            //      in flight together ----
            {
                double acc[2] = {0.0, 0.0};
                const float al = static_cast<float>(alpha);
                constexpr int NB = 4;  // slices of one warp whose loads are in flight together
                for (int s0 = sb + warp; s0 < se; s0 += NB * wpb) {
                    float apv[NB], rv0[NB], mv[NB];
                    double xv[NB];
#pragma unroll
                    for (int k = 0; k < NB; ++k) {
                        const int s = s0 + k * wpb;
                        const int rr_ = (s < se ? s : s0) * 32 + lane;
                        apv[k] = ap[rr_];
                        rv0[k] = r[rr_];
                        mv[k] = minv[rr_];
                        xv[k] = a.x64[rr_];
                    }
#pragma unroll
                    for (int k = 0; k < NB; ++k) {
                        const int s = s0 + k * wpb;
                        if (s >= se) continue;
                        const int row = s * 32 + lane;
                        const float pv = pw[row - w0];
                        a.x64[row] = xv[k] + alpha * static_cast<double>(pv);
                        const float rv = rv0[k] - al * apv[k];
                        const float zv = mv[k] * rv;
                        r[row] = rv;
                        z[row] = zv;
                        acc[0] += static_cast<double>(rv) * static_cast<double>(zv);
                        acc[1] += static_cast<double>(rv) * static_cast<double>(rv);
                    }
                }
                cur_bank = next_bank();
                publish<2>(acc, s_red, cur_bank);
            }
            clock(2);
            if (!bar.sync(&s_flag)) return;
            grid_totals(cur_bank, 2, s_tot);
            clock(3);
            double rz_new = s_tot[0], rr_new = s_tot[1];
            iterations = it + 1;
            if (bad(rz_new) || bad(rr_new)) {
                rz = rz_new;
                rr = rr_new;
                status = XPLUS_BREAKDOWN;
                break;
            }
            bool do_replace = false, drop_replace = false;
            double zap = 0.0;  // z_new . Ap' of a replacement
            if (true_mode) {
                if (rr_new <= tau_true_rr) do_replace = drop_replace = true;
                if (a.replace_every > 0 && iterations % a.replace_every == 0) do_replace = true;
                if (a.replace_drop > 0.0 && rr_new <= a.replace_drop * rr_at_replace) do_replace = drop_replace = true;
            }
            if (do_replace) {
                residual_phase(false);
                if (!bar.sync(&s_flag)) return;
                grid_totals(cur_bank, 4, s_tot);
                clock(4);
                rz_new = s_tot[0];
                rr_new = s_tot[1];
                true_rr = s_tot[2];
                zap = s_tot[3];
                ++replacements;
                rr_at_replace = rr_new;
                if (pol.after(a.restart_on_replace, true_rr, a.stag_factor, a.stag_window)) stagnated = 1;
            }
            if (lead && a.trace && it < a.trace_cap) {
                double* t = a.trace + 5 * static_cast<size_t>(it);
                t[0] = alpha;
                t[1] = rz_new / rz_old;
                t[2] = rz_new;
                t[3] = rr_new;
                t[4] = sqrt(rr_new > 0.0 ? rr_new : 0.0);
            }
            rz = rz_new;
            rr = rr_new;
            if (true_mode ? (do_replace && true_rr <= tau_true_rr) : (rr <= a.tau_rr)) {
                status = XPLUS_CONVERGED;
                break;
            }
            if (stagnated) break;
            if (fabs(rz_old) <= kBreakdownEps) {
                status = XPLUS_BREAKDOWN;
                break;
            }
            beta = pol.beta(do_replace, drop_replace, rz, rz_old, zap, pap);
            if (bad(beta)) {
                status = XPLUS_BREAKDOWN;
                break;
            }
        }
    }
    if (status == XPLUS_MAX_ITER && !true_mode && rr <= a.tau_rr) status = XPLUS_CONVERGED;

    // ---- exit: FP64 true residual of the final x ----
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
            o->status = status;
            o->iterations = iterations;
            o->replacements = replacements;
            o->stagnated = stagnated;
            o->rz = rz;
            o->rr = rr;
            o->pap = pap;
            o->alpha = alpha;
            o->true_rr = s_tot[0];
            o->t_end_ns = globaltimer_ns();
            for (int k = 0; k < 4; ++k) o->t_phase[k] = s_clk[k];
        }
    }
}


using WindowKernel = void (*)(PcgArgs);

template <typename VT>
WindowKernel pick_chunk(int chunk) {
    return chunk == 4 ? pcg_window_kernel<VT, 4> : (chunk == 2 ? pcg_window_kernel<VT, 2> : nullptr);
}

WindowKernel pick(const KernelKey& k) {
    if (k.xt != XPLUS_F32 || !k.diag || k.gtg || !k.idx16) return nullptr;
    switch (k.vt) {
        case XPLUS_F32: return pick_chunk<float>(k.chunk);
        case XPLUS_BF16: return pick_chunk<__nv_bfloat16>(k.chunk);
        case XPLUS_F16: return pick_chunk<__half>(k.chunk);
    }
    return nullptr;
}

}  // namespace

cudaError_t window_prepare(const KernelKey& k, int device, int n_slices, int grid, int tpb, int window, bool* fits,
                           size_t* smem_bytes) {
    *fits = false;
    WindowKernel f = pick(k);
    if (!f || (n_slices + grid - 1) / grid > kWinSlices) return cudaSuccess;
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa{};
    e = cudaFuncGetAttributes(&fa, f);
    if (e != cudaSuccess) return e;
    const size_t limit = static_cast<size_t>(optin) - fa.sharedSizeBytes, need = sizeof(float) * static_cast<size_t>(window);
    if (tpb > fa.maxThreadsPerBlock || need > limit) return cudaSuccess;
    // the opt-in is the kernel's, shared by all handles: always the most a launch may ask for
    e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(limit));
    if (e != cudaSuccess) return e;
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, tpb, need);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    *smem_bytes = need;
    *fits = grid <= per_sm * sms;
    return cudaSuccess;
}

cudaError_t window_launch(const KernelKey& k, const PcgArgs& a, int grid, int tpb, size_t smem_bytes, cudaStream_t s) {
    WindowKernel f = pick(k);
    if (!f) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(tpb);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, f, a);
}

}  // namespace xplus
