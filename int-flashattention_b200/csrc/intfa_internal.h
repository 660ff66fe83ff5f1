// Internal declarations shared by the translation units of libintfa.so.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/intfa.h"

namespace intfa {

// Arguments of the attention kernel (plain data, passed by value).
struct KParams {
  const void* qs; const void* ks; const void* vs;   // fp32, or fp16 where scale_f16 says so
  int scale_f16;                 // INTFA_SCALE_F16_* bits
  __half* o;
  long long o_sb, o_sh, o_sn;
  long long qs_sb, qs_sh, ks_sb, ks_sh, vs_sb, vs_sh, vs_sd;
  int B, H, Nq, Nk;
  int dh;                        // head dim of the tensors in memory (16 runs the 32-wide kernel on zero-filled tiles,
                                 // 256 the 128-wide one twice per query tile, once per half of the V channels)
  int hk_ratio;                  // query heads per K/V head (1 unless grouped-query attention)
  int o_bf16;                    // output element type: 0 fp16, 1 bf16
  int causal;
  float c;                       // sm_scale * 1.44269504 (fp32)
  long long q_off, kv_off;
  float* lse; float* st_m; float* st_l; float* st_acc;
  int state_in, state_out, write_o;
  int* dbg_s; void* dbg_p; int dbg_tile, dbg_step;
  int* status;
  int MB, num_tiles;
  int wait_limit_kcycles;        // bounded waits give up after this many thousand SM cycles
  int skip_k_load;               // test hook: 1-based KV step whose K tile the producer leaves out; 0: none
  int kv_desc;                   // 1: KV tiles visited last-to-first
  long long vs_sblk;             // element stride of the KV-tile axis of v_scale; 0: one scale row per (batch, head)
  unsigned int* tile_counter;    // {next work item beyond the first of every CTA, CTAs that are done}, both zero
                                 // between launches; null when every CTA has one work item at most
};

// Records the calling thread's last error (printf-style) and returns `code`.
int set_error(int code, const char* fmt, ...);
// SM count of the current device, cached per device; <=0 on failure.
int sm_count_cached();

// Few query rows against many keys (intfa_decode.cu).  Returns false where the call is not one for that path.
bool decode_dispatch(const IntfaFwdParams* a, cudaStream_t stream, int* rc);
size_t decode_workspace_bytes(const IntfaFwdParams* a);
// Every kernel of this library is launched so that it may begin while the kernel before it on the stream is still running
// (programmatic stream serialisation): its setup and the launch itself overlap the other's tail.  Each begins with
// pdl_wait(), which returns when everything before it on the stream is done and visible, and only then may let the next one
// begin (pdl_launch()): what a kernel reads ahead of its own wait is therefore older than the kernel before it.
// `cluster`: CTAs of a cluster (the x dimension of the grid is a multiple of it).
template <typename K, typename... A>
inline int launch_clusters(const char* what, K kernel, dim3 grid, int cluster, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  return e == cudaSuccess ? INTFA_OK : set_error(INTFA_ERR_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
}
template <typename K, typename... A>
inline int launch_kernel(const char* what, K kernel, dim3 grid, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  return launch_clusters(what, kernel, grid, 1, threads, smem, stream, args...);
}

int fwd_dispatch(const IntfaFwdParams* a, cudaStream_t stream);
int quant_pertoken(const void* x, const int64_t* st, void* x8, float* scale, int B, int H, int N, int D,
                   cudaStream_t stream);
int quant_v(const void* v, const int64_t* st, void* v8, float* scale, int mode, int B, int H, int N, int D,
            void* workspace, cudaStream_t stream);
int v_colmax(const void* v, const int64_t* st, void* colmax, int B, int H, int N, int D, cudaStream_t stream);
int v_quant_from_colmax(const void* v, const int64_t* st, const void* colmax, void* v8, float* scale, int mode, int B,
                        int H, int N, int D, cudaStream_t stream);
constexpr int kStaticColmaxWords = 65536;   // 256 KiB: built-in scratch of intfa_quant_v_static (B*H*D limit)
int quant_v_static(const void* v, const int64_t* st, void* v8, float* scale, int mode, int B, int H, int N, int D,
                   cudaStream_t stream);
int quant_v_partial(const void* v, const int64_t* st, void* v8, float* scale, int mode, int B, int H, int N, int D,
                    void* workspace, cudaStream_t stream);
size_t quant_qkv_workspace_bytes(int B, int Hkv, int Nk, int D);
int quant_qkv(const void* q, const void* k, const void* v, const int64_t* v_st, void* q8, void* k8, void* v8, float* qs,
              float* ks, float* vs, int mode, int B, int H, int Hkv, int Nq, int Nk, int D, void* workspace,
              cudaStream_t stream);
int scales_f16_to_f32(const void* src, float* dst, long long n, cudaStream_t stream);

}  // namespace intfa
