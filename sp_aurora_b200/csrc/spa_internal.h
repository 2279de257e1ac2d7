// Internal declarations shared by the kernels and the C-ABI translation unit.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/spa.h"

namespace spa {

// Error text for spa_last_error(); thread-local.
void set_error(const char* fmt, ...);

// Device-global status word (4 ints) of the current device; allocated lazily,
// zero while no bounded wait has ever given up.
int* device_status_word();

// Encode a 4-D TMA descriptor (dims D, S, H, B; 128-byte swizzle; box of
// `box_rows` sequence rows by 64 two-byte elements). Returns 0 on success.
int encode_rows_map(CUtensorMap* map, const void* ptr, int is_bf16, int D, int64_t S, int H, int B,
                    int64_t stride_s, int64_t stride_h, int64_t stride_b, int box_rows);

// 4-D TMA descriptor over a contiguous fp32 [B,S,H,D] tensor (dims D, S, H, B; no
// swizzle; box of `box_rows` sequence rows by D), used for bulk reduce-add.
int encode_f32_rows_map(CUtensorMap* map, const void* ptr, int D, int64_t S, int H, int B,
                        int box_rows);

// Same tensor, box of `box_rows` sequence rows by 32 floats with the 128-byte swizzle:
// shared-memory slabs of [box_rows][128 B] that a thread per row fills without bank
// conflicts. Used to store or reduce-add dK/dV tiles.
int encode_f32_slab_map(CUtensorMap* map, const void* ptr, int D, int64_t S, int H, int B,
                        int box_rows);

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) applies to the current device only:
// done once per (kernel, device), remembered in a small table. Returns a spa status code.
int ensure_dynamic_smem(const void* kernel, int bytes, const char* what);

// SM count of the current device (cached per device; 148 if the query fails).
int device_sm_count();

// Launchers (return a spa status code). Arguments arrive normalised: zero stride
// triples of spa.h are already replaced by the contiguous strides.
// `workspace` (may be null: then the keys of a block are never split between CTAs) holds
// fwd_sm100_workspace(a) bytes, 16-byte aligned.
int64_t fwd_sm100_workspace(const spa_fwd_args* a);
int launch_fwd_sm100(const spa_fwd_args* a, float* workspace);
int launch_bwd_dq_sm100(const spa_bwd_args* a);       // query-stationary pass: dQ
// K/V-stationary pass: dK, dV. behind_dq: the dQ pass of the same problem is the kernel just
// before it in the stream; the two may then overlap where one drains and the other fills.
int launch_bwd_dkv_sm100(const spa_bwd_args* a, bool behind_dq);
// The same kernels over up to kVarMaxSeqs sequences of a packed batch (B = 1).
int launch_fwd_sm100_var(const spa_fwd_args* a, const spa_seq* seqs, int n_seq);
int launch_bwd_dq_sm100_var(const spa_bwd_args* a, const spa_seq* seqs, int n_seq);
int launch_bwd_dkv_sm100_var(const spa_bwd_args* a, const spa_seq* seqs, int n_seq, bool behind_dq);
// The dQ pass with CTAs that loop over query tiles, and the rule that takes a launch there
// (n_seq = 0: a plain one).
bool dq_loops(const spa_bwd_args* a, const spa_seq* seqs, int n_seq);
int launch_bwd_dq_loop_sm100(const spa_bwd_args* a, const spa_seq* seqs, int n_seq);
int launch_fwd_simt(const spa_fwd_args* a);
int launch_bwd_simt(const spa_bwd_args* a);

// kern<<<grid, threads, smem, stream>>>(args...), with the programmatic attribute: the grid may
// start before the one in front of it has ended (see grid_release / grid_acquire).
template <typename... P, typename... A>
cudaError_t launch_programmatic(void (*kern)(P...), long long grid, int threads, int smem, void* stream,
                                const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

}  // namespace spa
