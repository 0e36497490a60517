// The chunked attention kernels on slices of wider tensors (host-side interface): `ld` is the distance in elements from
// one step of q / k / v to the next (0: dense, H * d); otherwise as the C ABI functions of the same arguments.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mxk.h"

namespace mxk {
namespace linattn {
int forward(const void* q, const void* k, const void* v, long long ld, const float* s0, const float* z0, const uint8_t* done,
            void* o, float* s_last, float* z_last, void* chunk_states, int* status, int B, int T, int H, int d, float eps,
            int feature_map, cudaStream_t stream);
int backward(const void* q, const void* k, const void* v, long long ld, const void* d_o, const void* chunk_states,
             const uint8_t* done, const float* ds_last, const float* dz_last, void* dq, void* dk, void* dv, long long ld_grad,
             float* ds0, float* dz0, int* status, int B, int T, int H, int d, float eps, int feature_map, cudaStream_t stream);
}  // namespace linattn
namespace gdelta {
int forward(const void* q, const void* k, const void* v, long long ld_v, const float* alpha, const float* beta, const float* s0,
            const uint8_t* done, void* o, float* s_last, void* chunk_states, void* workspace, size_t workspace_bytes,
            int* status, int B, int T, int H, int d, cudaStream_t stream);
int backward(const void* q, const void* k, const void* v, const float* alpha, const float* beta, const void* d_o,
             const void* chunk_states, const void* workspace, const uint8_t* done, const float* ds_last, void* dq, void* dk,
             void* dv, long long ld_dv, float* dalpha, float* dbeta, float* ds0, int* status, int B, int T, int H, int d,
             cudaStream_t stream);
}  // namespace gdelta
namespace mlstm_tc {
// ld_qv, hp_qv / ld_grad, hp_grad: pitch of the steps and of the heads of q and v (of dq and dv); k and dk are dense
int forward(const void* q, const void* k, const void* v, long long ld_qv, long long hp_qv, const float* log_i, const float* log_f, const float* c0,
            const float* n0, const float* m0, const float* f0, const uint8_t* done, void* h, float* c_last, float* n_last,
            float* m_last, float* f_last, float* m_steps, void* chunk_states, int* status, int B, int T, int H, int d, float eps,
            cudaStream_t stream);
int backward(const void* q, const void* k, const void* v, long long ld_qv, long long hp_qv, const float* log_i, const float* log_f, const float* c0,
             const float* n0, const float* m0, const uint8_t* done, const void* dh, const float* c_last, const float* n_last,
             const float* m_steps, const void* chunk_states, const float* dc_last, const float* dn_last, const float* dm_last,
             void* dq, void* dk, void* dv, long long ld_grad, long long hp_grad, float* dlog_i, float* dlog_f, float* dc0, float* dn0, float* dm0,
             int* status, int B, int T, int H, int d, float eps, cudaStream_t stream);
}  // namespace mlstm_tc
}  // namespace mxk
