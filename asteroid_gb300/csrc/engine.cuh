// engine.cuh -- the context object behind the C ABI and the helpers the kernels share.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <vector>
#include "asteroid_gb300.h"
#include "model.cuh"

extern "C" int ast_set_error(int code, const char* fmt, ...);

#define AST_CUDA(call)                                                                        \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return ast_set_error(AST_E_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call,       \
                                 cudaGetErrorString(e_));                                     \
    } while (0)

namespace ast {

// Device error word: kernels record a wait that ran out of iterations here instead of
// trapping, so the context stays usable and the host returns AST_E_TIMEOUT.
enum : int32_t { kErrNone = 0, kErrStageTimeout = 1 };

struct FitBuffers {
    int64_t slots = 0, slots_pad = 0, chains = 0, groups = 0;
    int32_t n_params = 0, n_filters = 0, cf_bytes = 0;
    void* x = nullptr;        // CF [(N+1)*N][S]
    void* f = nullptr;        // CF [N+1][S]
    uint8_t* ind = nullptr;   // [N+1][S]
    void* x0 = nullptr;       // CF [N][S]
    void* xr = nullptr;       // CF [N][S]
    void* fr = nullptr;       // CF [S]
    int32_t* st = nullptr;    // [S] phase | j << 8 | bad << 16
    int32_t* it = nullptr;    // [S] simplex iterations l
    int32_t* ev = nullptr;    // [S] evaluations of the current chain-stage
    int64_t* chain = nullptr; // [S] chain on the slot, -1 if none
    double* dv = nullptr;     // [NF][S] last delta_V of the slot's chain
    double* chain_f = nullptr;  // [C]
    void* chain_x = nullptr;    // CF [C][N] best vertex
    double* chain_dv = nullptr; // [C][NF]
    void* group_x = nullptr;    // CF [G][N] next stage start
    double* out_f = nullptr;    // [G]
    double* out_p = nullptr;    // [G][N]
    double* out_dv = nullptr;   // [G][NF]
    unsigned long long* ctr = nullptr;  // [0] next chain, [1] finished chains, [2] evals, [3] fits, [4] err
    size_t bytes = 0;
    void* base = nullptr;
};

struct FitRun {
    bool active = false;
    ast_fit_cfg cfg{};
    int32_t stage = 0;
    int32_t reopt = 0;          // reopt of the current stage
    int64_t n_evals = 0, n_fits = 0;
    double kernel_ms = 0;
    int tpb = 256, ctas = 0;
    int lanes = 1;     // threads of a slot (fit_group_kernel)
    int pair = 0;      // integrators of a CTA of fit_pair_kernel, 0: another kernel
    size_t smem = 0;   // dynamic shared memory of the launch (the observation block, or 0)
    int minb = 1;      // register budget variant of fit_kernel
};

}  // namespace ast

struct ast_ctx {
    int device = 0;
    int sm_count = 0;
    size_t smem_optin = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    ast_model model{};
    ast::DevModel dm{};
    int32_t n_data = 0, n_filters = 0;
    double span = 0;  // days from the first observation to the last
    double steps() const { return span / dm.time_step / n_data; }  // the span in RK4 steps an observation
    ast::ObsLayout layout{};
    void* d_obs = nullptr;
    // evaluation scratch
    double* d_params = nullptr;
    double* d_chi2 = nullptr;
    double* d_dv = nullptr;
    int64_t eval_cap = 0;
    // fit
    ast::FitBuffers fb;
    ast::FitRun run;
    int32_t stage_wait = 1 << 22;  // polls of the fit kernel's shared-memory staging wait
};

namespace ast {
// Lets launches of `kern` ask for up to `bytes` of dynamic shared memory (needed above 48 KB; allocates
// nothing).  The limit belongs to the kernel on its device, not to a context or a call: one caller's
// value holds for the launches of every other context and thread.  So `bytes` is the most that any call
// asks of the kernel, the same from every caller, never what this call needs.
template <class K>
inline int allow_smem(K kern, size_t bytes)
{
    AST_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return AST_OK;
}

// Dynamic shared memory for staging an observation block of `bytes` in one CTA of `kern`: the
// block's size when it fits beside the kernel's static shared memory (the double-float trig
// table, the staging barrier) under the per-CTA opt-in limit `optin`, else 0 -- the kernel then
// reads the block from global memory through L1.  When it is staged, the kernel may ask for all
// that the device has beside its static shared memory.
template <class K>
inline int obs_smem_for(K kern, size_t bytes, size_t optin, size_t* smem)
{
    *smem = 0;
    if (!bytes) return AST_OK;
    cudaFuncAttributes a;
    AST_CUDA(cudaFuncGetAttributes(&a, kern));
    if (bytes + a.sharedSizeBytes > optin) return AST_OK;
    if (int rc = allow_smem(kern, optin - a.sharedSizeBytes)) return rc;
    *smem = bytes;
    return AST_OK;
}

// Lanes an FP64 evaluation by the number that run side by side (1: one thread each).  A warp alone on its
// quarter of the SM costs its FP64 instructions times 64 cycles, four on an SM 19 each (group64.cuh):
// eight lanes an evaluation need 2.2 to 3 times fewer, so they win until the SMs hold `most` evaluations, six to
// eight such warps; from there the FP64 unit is full either way and threads do the least.
// Thirty-two lanes share the magnitudes of four times as many observations and win while every
// evaluation still has a quarter of an SM.  Eight lanes against threads, ms, by evaluations an SM (152 SMs, 60
// points, 30 RK4 steps an observation; searches of 13 evaluations a chain, their sines the library's):
//   evaluations, torque     28: 12.9/14.0   32: 14.8/14.0     free 28: 8.7/10.4   32: 9.9/10.4
//   searches, torque        24: 521/571     28: 598/571       free 28: 299/325    32: 342/325
//   the same, 10 steps      28: 199/209     32: 226/209            32: 114/121
//   the same, 3 steps       32: 72/88                              32: 36/51
//   torque, 10 steps: P_PSI 32: 161/173     from a model 24: 155/172  28: 178/172  32: 203/172
//   the ball, whose magnitude is a third: torque, 10 steps 24: 101/109; from a model 3 steps 28: 27/30  32: 31/30
// and 32 lanes against 8, 10 steps an observation: evaluations 4: 3.06/2.97, 6: 3.67/2.97; searches 4: 130/133, 6: 155/134.
// `steps`: the curve's span in RK4 steps an observation.
inline int group_lanes(int64_t n, int sm_count, int most)
{
    return n <= 4 * (int64_t)sm_count ? 32 : n <= (int64_t)most * sm_count ? 8 : 1;
}
inline int group_most_eval(int flags, double steps) { return (flags & AST_TORQUE) && steps >= 15 ? 28 : 32; }
inline int group_most_fit(int flags, bool from_model, double steps)
{
    if (!(flags & AST_TORQUE)) return steps < 15 ? 32 : 28;
    const double w = flags & AST_BW_BALL ? 3 * steps : steps;
    if (from_model) return w < 5 ? 32 : w < 8 ? 28 : 24;
    return w < 5 ? 32 : w < 15 ? (flags & AST_P_PSI ? 32 : 28) : 24;
}

// Integrator warps of a CTA of the paired mixed kernels (mixed.cuh), by the number of evaluations that run
// side by side; 0: one thread an evaluation, both parts.  At most `most` (pair_most_fit).
constexpr int kPairIntegrators = 4;
inline int pair_integrators(int64_t n, int sm_count, int most)
{
    const int64_t k = ((n + 31) / 32 + sm_count - 1) / sm_count;
    return k <= most ? (int)k : 0;
}

// The most integrators a CTA with which pairs are faster than threads.  Beside its step an integrator has
// the general step's code (models that the step declines) and a photometer the NUDGE candidates'; an SM whose
// warps run all of them at once waits for instructions, the more warps the more.  Pairs against threads,
// ms, with 2, 3 and 4 integrators a CTA on 152 SMs; steps: the curve's span in RK4 steps an observation.
//   evaluations, 150 points, steps 2.1: near a model       0.37/0.53    0.39/0.53    0.42/0.53
//                                       from the prior     0.57/0.69    0.77/0.70    0.94/0.71
//                torque, NUDGE: near a model               0.73/0.93    0.86/0.93    0.85/0.94
//                               from the prior             1.18/1.11    1.58/1.14    1.87/1.20
//   fits, 60 points, steps 2.1: free, 16 evaluations a chain  3.4/4.8    4.0/4.9      4.4/4.8
//     100 evaluations:
//                torque, from a model                      21.7/30.0    25.9/30.6    38.6/29.3
//                                        steps 0.1         13.1/19.8    14.1/20.2    16.3/20.0
//                        from the prior                    45.1/46.0    66.7/52.4    88.3/58.6
//                                        steps 9.1         75.3/88.0    84.7/88.4    98.4/89.0
//                                        steps 29          174/190      178/189      182/189
//                        with P_PSI, from the prior        29.9/37.4    36.5/38.6    47.0/38.2
//                torque, NUDGE, from the prior              143/138      206/183      274/205
//                FP32 right-hand side, from a model        21.9/27.2    24.7/29.0    31.7/28.2
//                                        steps 9.1         53.4/61.4    55.5/62.8    57.3/62.0
// Evaluations, which are of models near a solution for the most part, take pairs up to four.  So do batches, whose
// thread kernel keeps three CTAs of 128 an SM (six objects of three variants, 30 evaluations a chain: 26/67,
// 29/68, 36/67).
inline int pair_most_fit(int precision, int flags, bool from_model, double steps)
{
    const bool few = steps >= 1 && steps < 6;  // below, an integrator has little to run
    if (precision == AST_PREC_MIXED_RHS32 && (flags & AST_NUDGE)) return 3;
    if (flags & AST_NUDGE) return steps < 20 ? 2 : 3;
    if (!(flags & AST_TORQUE)) return kPairIntegrators;
    if (precision == AST_PREC_MIXED_RHS32) return few ? 3 : 4;
    // A period's range (P_PSI) keeps most of the prior's models within the compact step, as a model does.
    if (from_model || (flags & AST_P_PSI)) return few ? 3 : 4;
    return steps < 6 ? 2 : steps < 20 ? 3 : 4;
}

int build_dev_model(const ast_model* m, const ast_obs_set* obs, DevModel* dm);
int set_device(int device);
void obs_image(const ast_model* model, const ast_obs_set* obs, const ObsLayout& L, std::vector<unsigned char>& img);
int launch_prep(const DevModel& dm, char* d_block, const ObsLayout& L, int64_t n, cudaStream_t s);
}  // namespace ast
