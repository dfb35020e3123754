// Shared between the chunkwise mLSTM translation units.
#pragma once
#include "common.cuh"

namespace xl {

struct ChunkwiseParams {
    const void *q, *k, *v, *ig, *fg;
    const float *C0, *n0, *m0;
    void *h;
    float *C1, *n1, *m1;
    int B, NH, S, dqk, dv, L;
    float eps, qscale;
    float gate_cap;   // > 0: i and f are soft-capped (cap * tanh(x / cap)) as they are read
    // element strides (batch, head, token); innermost dimension contiguous
    int64_t sq[3], sk[3], sv[3], sh[3], sg[3];
    // optional extra destinations of h (same strides and offsets as `h`): buffers of peer GPUs
    void *h_peer[8];
    int n_peer;
    // > 0: token-sharded destinations instead of replicas - h_peer[r] (r = 0 .. n_peer-1, this rank included, `h` unused)
    // is rank r's [B, tok_per_rank, NH_total, dv] buffer and a tile of tokens goes ONLY to the rank that owns them
    int tok_per_rank;
    int *status;      // status word of the caller's scratch, cleared by the fp32 kernels (no wait of theirs can give up), or NULL
};

// the first bytes of every scratch buffer: the status word that xlstm_mlstm_chunkwise_status() reads
constexpr size_t WS_HEADER = 256;

// fp32 arithmetic, any dqk, dv, S: launches over groups of chunks, chunk states in scratch
size_t mlstm_chunkwise_f32_workspace(int B, int NH, int S, int dqk, int dv);
bool mlstm_chunkwise_f32_supported(const ChunkwiseParams &p, int dtype);
int mlstm_chunkwise_f32(const ChunkwiseParams &p, int dtype, void *workspace, cudaStream_t st);

// the same in one launch without scratch: dqk <= 512, L <= 64
int mlstm_chunkwise_simt(const ChunkwiseParams &p, int dtype, cudaStream_t st);

// up to 128 bf16 tokens to the same accuracy in one launch without scratch: dqk == 256 or 128, dv % 32 == 0, 16-byte aligned
// rows.  inputs_settled: q, k, v and the gates were not written by the launch before (only the state is waited for).  C1 may
// be C0.
bool mlstm_chunkwise_tail_supported(const ChunkwiseParams &p, int dtype);
int mlstm_chunkwise_tail(const ChunkwiseParams &p, bool inputs_settled, cudaStream_t st);

// tcgen05 / TMEM / TMA path: bf16, L == 64, dqk == 256 (or 128/64), dv % 128 == 0, whole chunks
// shape_ok: the shape, strides and alignment fit the tensor-core kernel; driver_ok: the driver entry point
// that encodes TMA descriptors could be resolved; supported = both
bool mlstm_chunkwise_tc_shape_ok(const ChunkwiseParams &p, int dtype);
bool mlstm_chunkwise_tc_driver_ok();
bool mlstm_chunkwise_tc_supported(const ChunkwiseParams &p, int dtype);
size_t mlstm_chunkwise_tc_workspace(int B, int NH, int S, int dqk, int dv, int L);
// scratch of the single-pass mode (no segment states): what the forward needs at least
size_t mlstm_chunkwise_tc_workspace_min(int B, int NH, int S, int dqk, int dv);
int mlstm_chunkwise_tc(const ChunkwiseParams &p, void *workspace, size_t workspace_bytes, cudaStream_t st);
// 1: every head takes the general tensor-core kernel whatever its gates are; 0: per-head choice (default)
void mlstm_chunkwise_tc_set_general_only(int on);
// segments >= 1: cut every sequence into that many segments (segment-parallel two-pass mode); < 1: planned from
// the grid size (default)
void mlstm_chunkwise_tc_set_segments(int segments);

int mlstm_chunkwise_static_scratch(void **out);

}  // namespace xl
