// pcg_small.cu -- the persistent Jacobi-PCG for systems that one CTA solves with FP64 vectors (the
// reference's own problem size, n <= 1024 by include/cg_common.hpp:11): pcg_persistent_kernel's
// iteration, its arithmetic on every row and the order of its sums, without its trips to L2.
//
// Warp w owns slices w, w + W, ... (at most four) and lane l row 32 s + l of each, so a thread's rows'
// x, r, z, p, Ap and M^-1 stay in its registers for the whole solve; the search direction p' is the
// one vector others read and lies in shared memory, with the matrix beside it when it fits (it does at
// n = 1024: 87 KB), else the matrix comes through L1, which no barrier empties here.  A sum over the
// CTA is known to every thread after one CTA barrier (two scratch banks), so an iteration has three:
// p' written, p'.Ap', r.z and r.r.
// What bounds it is the chain of those: two block sums of ten dependent FP64 shuffles and adds, two
// FP64 divisions, one pass over the matrix.  n = 1024, FP64 values: 6.0 us per iteration through the
// global-memory kernel (records, partial sums and Ap through L2), here 2.9 (solve() 0.77 -> 0.42 ms).
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

constexpr int kMaxRows = 4;     // slices (rows per thread) of a warp
constexpr int kMaxSlices = 64;  // 16 warps

// block_sum with the scratch bank given: one CTA barrier, since the bank's last readers have passed
// another one since.
template <int NV>
__device__ __forceinline__ void block_sum_bank(double (&v)[NV], double* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = warp_sum(v[q]);
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) scratch[q * 32 + warp] = v[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = warp_sum(lane < nwarps ? scratch[q * 32 + lane] : 0.0);
}

// kRows: slices of a warp at most, 2 or 4 (straight-line code over a thread's rows)
template <typename VT, int CHUNK, bool DIFF, typename IT, int kRows>
__global__ void __launch_bounds__(512, 1) pcg_small_kernel(PcgArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double s_red[2][32 * 4];
    __shared__ int2 s_slice[kMaxSlices];
    __shared__ long long s_clk[6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const bool lead = threadIdx.x == 0;
    const bool true_mode = a.tau_true_rr >= 0.0;
    double* pw = reinterpret_cast<double*>(smem_raw);
    // every slice is a multiple of 32 slots: 16-byte groups of both arrays
    const long long slots = a.slice_ptr[a.n_slices];
    const VT* val = static_cast<const VT*>(a.val);
    const IT* col = static_cast<const IT*>(a.col);
    if (8LL * a.n_pad + slots * static_cast<long long>(sizeof(VT) + sizeof(IT)) <= a.smem_bytes) {
        VT* mval = reinterpret_cast<VT*>(pw + a.n_pad);
        IT* mcol = reinterpret_cast<IT*>(mval + slots);
        const long long nv = slots * static_cast<long long>(sizeof(VT)) / 16;
        const long long nc = slots * static_cast<long long>(sizeof(IT)) / 16;
        for (long long i = threadIdx.x; i < nv; i += blockDim.x)
            reinterpret_cast<uint4*>(mval)[i] = __ldg(reinterpret_cast<const uint4*>(val) + i);
        for (long long i = threadIdx.x; i < nc; i += blockDim.x)
            reinterpret_cast<uint4*>(mcol)[i] = __ldg(reinterpret_cast<const uint4*>(col) + i);
        val = mval;
        col = mcol;
    }
    // the first slice with slots (n_slices: none): what a slice without any may read
    int with_slots = 0;
    while (with_slots < a.n_slices && a.slice_ptr[with_slots + 1] == a.slice_ptr[with_slots]) ++with_slots;
    const int first_slice = with_slots < a.n_slices ? with_slots : 0;
    for (int k = threadIdx.x; k < a.n_slices; k += blockDim.x) {
        const long long b0 = a.slice_ptr[k];
        s_slice[k] = make_int2(static_cast<int>(b0), static_cast<int>((a.slice_ptr[k + 1] - b0) >> 5));
    }
    double x[kRows], r[kRows], z[kRows], p[kRows], ap[kRows], mi[kRows], rs[kRows];
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
        const int s = warp + k * wpb, row = s * 32 + lane;
        const bool on = s < a.n_slices;
        x[k] = on ? a.x64[row] : 0.0;
        mi[k] = on ? static_cast<const double*>(a.minv)[row] : 0.0;
        rs[k] = DIFF && on ? static_cast<const double*>(a.rowsum)[row] : 0.0;
        r[k] = z[k] = p[k] = ap[k] = 0.0;
    }
    if (lead) {
        for (int k = 0; k < 5; ++k) s_clk[k] = 0;
        s_clk[5] = globaltimer_ns();
        a.out->t_start_ns = s_clk[5];
    }
    __syncthreads();
    auto clock = [&](int slot) {
        if (lead) {
            const long long t = globaltimer_ns();
            s_clk[slot] += t - s_clk[5];
            s_clk[5] = t;
        }
    };
    int bank = 0;
    auto sum = [&](auto& v) {
        block_sum_bank(v, s_red[bank]);
        bank ^= 1;
    };
    // r = b - A x in FP64 of the x in global memory; z = M^-1 r.  Sums r.z, r.r, ||b - A x||^2, and
    // ||b||^2 (init) or z.Ap'
    double res[4];
    auto residual_phase = [&](bool init) {
        res[0] = res[1] = res[2] = res[3] = 0.0;
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const int s = warp + k * wpb;
            if (s >= a.n_slices) continue;
            const int row = s * 32 + lane;
            const double y = row_fp64<VT, double, CHUNK, DIFF, IT>(a, s, lane, row);
            const double bv = a.b64[row];
            const double rt = bv - y;
            const double zv = mi[k] * rt;
            res[3] += init ? bv * bv : zv * ap[k];
            r[k] = rt;
            z[k] = zv;
            res[0] += rt * zv;
            res[1] += rt * rt;
            res[2] += rt * rt;
        }
        sum(res);
    };
    auto store_x = [&]() {
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const int s = warp + k * wpb;
            if (s < a.n_slices) a.x64[s * 32 + lane] = x[k];
        }
        __syncthreads();
    };

    residual_phase(true);
    double rz = res[0], rr = res[1], true_rr = res[2];
    const double tau_true_rr = a.tau2_rel > 0.0 ? a.tau2_rel * res[3] : a.tau_true_rr;
    if (lead) a.out->bb = res[3];
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
            // ---- phase A: p' = z + beta p, Ap', p'.Ap' (the last readers of pw have passed the sum
            // of phase B since) ----
            double acc[1] = {0.0};
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const int s = warp + k * wpb;
                if (s >= a.n_slices) continue;
                p[k] = node_pnew(z[k], beta, p[k]);
                pw[s * 32 + lane] = p[k];
            }
            __syncthreads();
            // all the warp's slices together, chunk by chunk: their chains of dependent FP64 adds
            // overlap.  Beyond its width a slice repeats its last chunk, unused (one without slots:
            // those of the first that has some, which begin the matrix).
            int w[kRows], row[kRows], wmax = 0;
            const VT* vp[kRows];
            const IT* cp[kRows];
            double y[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const int s = warp + k * wpb;
                const int2 sl = s < a.n_slices ? s_slice[s] : make_int2(0, 0);
                w[k] = sl.y;
                wmax = max(wmax, sl.y);
                row[k] = (sl.y > 0 ? s : first_slice) * 32 + lane;
                vp[k] = val + (sl.y > 0 ? sl.x : 0) + lane * CHUNK;
                cp[k] = col + (sl.y > 0 ? sl.x : 0) + lane * CHUNK;
                y[k] = 0.0;
            }
            for (int c = 0; c < wmax; c += CHUNK) {
                typename ValArith<VT>::type v[kRows][CHUNK];
                int cc[kRows][CHUNK];
#pragma unroll
                for (int k = 0; k < kRows; ++k) {
                    const int at = max(0, min(c, w[k] - CHUNK)) * 32;
                    ChunkLoad<VT, CHUNK, kLdPlain>::run(vp[k] + at, v[k]);
                    ColLoad<CHUNK, IT, kLdPlain>::run(cp[k] + at, row[k], cc[k]);
                }
                double pj[kRows][CHUNK];
#pragma unroll
                for (int k = 0; k < kRows; ++k)
#pragma unroll
                    for (int q = 0; q < CHUNK; ++q) pj[k][q] = pw[cc[k][q]];
#pragma unroll
                for (int q = 0; q < CHUNK; ++q)
#pragma unroll
                    for (int k = 0; k < kRows; ++k) {
                        double pd = pj[k][q];
                        if (DIFF) pd -= p[k];
                        double t = y[k];
                        t += static_cast<double>(v[k][q]) * pd;
                        y[k] = c < w[k] ? t : y[k];
                    }
            }
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                if (warp + k * wpb >= a.n_slices) continue;
                if (DIFF) y[k] = y[k] * static_cast<double>(a.val_scale) + rs[k] * p[k];
                ap[k] = y[k];
                acc[0] += p[k] * y[k];
            }
            clock(0);
            sum(acc);
            clock(1);
            pap = acc[0];
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
            // ---- phase B: x, r, z and the two dots ----
            double dots[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                if (warp + k * wpb >= a.n_slices) continue;
                x[k] = x[k] + alpha * p[k];
                const double rv = r[k] - alpha * ap[k];
                const double zv = mi[k] * rv;
                r[k] = rv;
                z[k] = zv;
                dots[0] += rv * zv;
                dots[1] += rv * rv;
            }
            clock(2);
            sum(dots);
            clock(3);
            double rz_new = dots[0], rr_new = dots[1];
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
                store_x();
                residual_phase(false);
                clock(4);
                rz_new = res[0];
                rr_new = res[1];
                true_rr = res[2];
                zap = res[3];
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

    // ---- exit: x to global memory, the FP64 true residual of it ----
    store_x();
    double fin[1] = {0.0};
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
        const int s = warp + k * wpb;
        if (s >= a.n_slices) continue;
        const int row = s * 32 + lane;
        const double rt = a.b64[row] - row_fp64<VT, double, CHUNK, DIFF, IT>(a, s, lane, row);
        fin[0] += rt * rt;
    }
    sum(fin);
    if (lead) {
        if (a.block_clk)
            for (int k = 0; k < 4; ++k) a.block_clk[k] = s_clk[k];
        PcgOut* o = a.out;
        o->status = status;
        o->iterations = iterations;
        o->replacements = replacements;
        o->stagnated = stagnated;
        o->rz = rz;
        o->rr = rr;
        o->pap = pap;
        o->alpha = alpha;
        o->true_rr = fin[0];
        o->t_end_ns = globaltimer_ns();
        for (int k = 0; k < 4; ++k) o->t_phase[k] = s_clk[k];
    }
}

using SmallKernel = void (*)(PcgArgs);

template <typename VT, bool DIFF, typename IT>
SmallKernel pick_rows(int chunk, bool two) {
    switch (chunk) {
        case 1: return two ? pcg_small_kernel<VT, 1, DIFF, IT, 2> : pcg_small_kernel<VT, 1, DIFF, IT, 4>;
        case 2: return two ? pcg_small_kernel<VT, 2, DIFF, IT, 2> : pcg_small_kernel<VT, 2, DIFF, IT, 4>;
        case 4: return two ? pcg_small_kernel<VT, 4, DIFF, IT, 2> : pcg_small_kernel<VT, 4, DIFF, IT, 4>;
    }
    return nullptr;
}
template <typename VT, bool DIFF>
SmallKernel pick_form(const KernelKey& k, bool two) {
    return k.idx16 ? pick_rows<VT, DIFF, short>(k.chunk, two) : pick_rows<VT, DIFF, int>(k.chunk, two);
}

// the value types and forms of pcg_persistent_kernel with FP64 vectors
SmallKernel pick(const KernelKey& k, int n_slices, int tpb) {
    if (k.xt != XPLUS_F64 || k.gtg || n_slices > kMaxRows * (tpb / 32) || n_slices > kMaxSlices) return nullptr;
    const bool two = n_slices <= 2 * (tpb / 32);
    switch (k.vt) {
        case XPLUS_F32: return k.diag ? pick_form<float, true>(k, two) : pick_form<float, false>(k, two);
        case XPLUS_BF16: return k.diag ? pick_form<__nv_bfloat16, true>(k, two) : nullptr;
        case XPLUS_F16: return k.diag ? pick_form<__half, true>(k, two) : nullptr;
        case XPLUS_F64: return k.diag ? nullptr : pick_form<double, false>(k, two);
    }
    return nullptr;
}

}  // namespace

cudaError_t small_prepare(const KernelKey& k, int device, int n_slices, long long matrix_bytes, int tpb, bool* fits,
                          size_t* smem_bytes) {
    *fits = false;
    SmallKernel f = pick(k, n_slices, tpb);
    if (!f) return cudaSuccess;
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa{};
    e = cudaFuncGetAttributes(&fa, f);
    if (e != cudaSuccess) return e;
    const size_t limit = static_cast<size_t>(optin) - fa.sharedSizeBytes;
    const size_t vec = 8 * 32 * static_cast<size_t>(n_slices);
    if (tpb > fa.maxThreadsPerBlock || vec > limit) return cudaSuccess;
    // the opt-in is the kernel's, shared by all handles: always the most a launch may ask for
    e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(limit));
    if (e != cudaSuccess) return e;
    *smem_bytes = vec + static_cast<size_t>(matrix_bytes) <= limit ? vec + static_cast<size_t>(matrix_bytes) : vec;
    *fits = true;
    return cudaSuccess;
}

cudaError_t small_launch(const KernelKey& k, const PcgArgs& a, int tpb, size_t smem_bytes, cudaStream_t s) {
    SmallKernel f = pick(k, a.n_slices, tpb);
    if (!f) return cudaErrorInvalidValue;
    f<<<1, tpb, smem_bytes, s>>>(a);
    return cudaGetLastError();
}

}  // namespace xplus
