// Host-side helpers shared by the tensor-core kernels (defined in fna_sm100.cu / na_bwd_simt.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200na {

// Tensor map over a heads-last [B, X0, X1, X2, H, D] 16-bit tensor seen as (H*D, X0, X1, X2, B):
// a box of 64 channels x tile[a] * dil[a] positions per axis, traversed with element stride
// dil[a]. B200NA_ERR_UNSUPPORTED when a box exceeds 256 positions or a stride exceeds 8.
// token_stride: elements between tokens (0 = H * D); ndim_sep > 0: the head is an axis of its own,
// (D, H, the ndim_sep layout axes, B), so that channels past a narrow head read as zeros.
struct FoldedAxis {
  int d, g0, groups, len;   // dilation, first group, number of groups, tokens of the layout
};
int fna_make_tensor_map_direct(CUtensorMap* tm, const void* ptr, int dtype, int B, const int* X,
                               int H, int D, const int* tile, const int* dil,
                               long long token_stride = 0, int ndim_sep = 0,
                               const FoldedAxis* fold = nullptr);

// A dilated 1-D layout is (position, group) with both as tensor-map axes: a tile of a group is then
// 128 positions whatever the dilation, where a box of 128 d tokens read with element stride d ends
// at d = 2 (256 positions). Groups g < len % d are one token longer than the others, and a map has
// one extent for all: one launch for each of the two kinds. At d = 2 and an odd length the strided
// box in one launch is kept. Returns the number of launches (0: do not fold).
struct FoldedPart {
  int g0, groups, extent;
};
int fna_fold_parts(int ndim, int len, int d, FoldedPart (&parts)[2]);

// One-time per-device setup of the attention kernels; returns the SM count and the address of the
// device status word that bounded waits report into.
int fna_device_info(int* sms, int** status_ptr);

// A zeroed pair of device counters {next work item, CTAs finished} for one launch on `stream` of a
// persistent kernel that hands out its items dynamically; the kernel's last CTA must zero the
// pair again. Launches on one stream share that stream's pair (they cannot overlap); a launch
// under stream capture gets a pair of its own from a pool of 3072 that is handed out in turn.
int fna_work_counters(unsigned long long** pair, cudaStream_t stream);

// Device memory that a call on `stream` hands from one of its launches to the next, from slots that are
// handed out like the counter pairs; set to 0 on the stream. Another thread's call on the same stream must
// not come between: the caller holds a lock from here to its last launch.
struct CallScratch {
  float norms[2];
  unsigned redo;
  unsigned unused;
};
int fna_call_scratch(CallScratch** scratch, cudaStream_t stream);

// norms[slot] = the largest squared 2-norm of the rows of D fp16 elements (a multiple of 8, at most 128,
// 16-byte aligned) of the inputs with that slot, or what was there. NaN where an input holds one.
struct NormRows {
  const void* rows;
  int64_t tokens;
  int heads;
  int64_t token_stride;   // elements
  int slot;
};
int launch_max_norms(const NormRows* in, int n_inputs, int D, float* norms, cudaStream_t stream);

// delta[row] = sum_d o[row, d] * d_out[row, d] (fp32), rows of D 16-bit elements (a multiple of
// 8, at most 128).
int launch_delta(const void* o, const void* d_out, float* delta, int64_t rows, int D, int dtype,
                 cudaStream_t stream);

// b200na_na_backward_simt; redo not null: dq, dk and dv are there already, and if *redo (device memory) is not
// 0, the 32-row blocks of them that hold a NaN or an infinity are done again (16-bit types, D a multiple of 8).
int simt_backward(
    const void* q, const void* k, const void* v, const void* o, const void* d_out, const float* lse,
    const void* add_k, const void* add_v, int n_extra, void* dq, void* dk, void* dv, void* d_add_k,
    void* d_add_v, float* delta_scratch, int ndim, const int* shape, const int* kernel,
    const int* stride, const int* dilation, const int* causal, int B, int Hq, int Hkv, int D,
    int dtype, float scale, const unsigned* redo, cudaStream_t stream);

}  // namespace b200na
