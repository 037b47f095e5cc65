// Attention over host-resident operands: the flat batch * head axis is streamed through two device staging
// buffers in chunks, the host -> device copies of the next chunk and the device -> host copy of the previous one
// overlapping the fused kernel of this one.  Native because a chunk took Python 60 to 80 us to enqueue, which
// set the smallest chunk worth having; what is not overlapped is the first chunk's way in and the last one's
// way out, so chunks want to be small (see host_chunk() in r_attention.py).
#include "common.cuh"

extern "C" int32_t splat_attention_host(const void* q, const void* k, const void* v, void* o, void* const* staging_8,
                                        int64_t chunk, const float* sTod_lin, const float* sTod_tr, const float* nnzs,
                                        int64_t bh, int64_t n_rows, int64_t d, float scale, int32_t dtype, int32_t path,
                                        const int32_t* plan_i32, const int32_t* band_table, int32_t* status_word,
                                        int32_t* path_ran, void* stream_in, void* stream, void* stream_out,
                                        void* const* events_7) {
    if (!q || !k || !v || !o || !staging_8 || !events_7 || chunk < 1 || bh < 0 || n_rows < 0 || d < 1) return SPLAT_ERR_BAD_ARG;
    cudaStream_t s_in = (cudaStream_t)stream_in, s = (cudaStream_t)stream, s_out = (cudaStream_t)stream_out;
    cudaEvent_t ev[7];       // per buffer: inputs ready, kernel done, output gone; the caller's stream
    for (int i = 0; i < 7; ++i) ev[i] = (cudaEvent_t)events_7[i];
    const size_t head = (size_t)n_rows * d * splat::elem_size(dtype);
    bool fine = cudaEventRecord(ev[6], s) == cudaSuccess && cudaStreamWaitEvent(s_in, ev[6], 0) == cudaSuccess;
    int i = 0;
    for (int64_t b = 0; b < bh && fine; b += chunk, ++i) {
        const int64_t n = bh - b < chunk ? bh - b : chunk;
        void* const* buf = staging_8 + (i & 1) * 4;
        cudaEvent_t in_ready = ev[(i & 1) * 3], done = ev[(i & 1) * 3 + 1], gone = ev[(i & 1) * 3 + 2];
        // (the events of a buffer's last use, in this call or an earlier one)
        fine = cudaStreamWaitEvent(s_in, done, 0) == cudaSuccess;
        const void* src[3] = {q, k, v};
        for (int j = 0; j < 3 && fine; ++j)
            fine = cudaMemcpyAsync(buf[j], (const char*)src[j] + b * head, n * head, cudaMemcpyHostToDevice, s_in) == cudaSuccess;
        fine = fine && cudaEventRecord(in_ready, s_in) == cudaSuccess && cudaStreamWaitEvent(s, in_ready, 0) == cudaSuccess &&
               cudaStreamWaitEvent(s, gone, 0) == cudaSuccess;
        if (!fine) break;
        const int32_t rc = splat_attention_fused_table(buf[0], buf[1], n_rows * d, d, 1, buf[2], buf[3], nullptr, sTod_lin,
                                                       sTod_tr, nnzs, n, n_rows, n_rows, d, scale, dtype, path, plan_i32,
                                                       band_table, status_word, path_ran, stream);
        if (rc != SPLAT_OK) return rc;
        fine = cudaEventRecord(done, s) == cudaSuccess && cudaStreamWaitEvent(s_out, done, 0) == cudaSuccess &&
               cudaMemcpyAsync((char*)o + b * head, buf[3], n * head, cudaMemcpyDeviceToHost, s_out) == cudaSuccess &&
               cudaEventRecord(gone, s_out) == cudaSuccess;
    }
    for (int x = 0; x < 2 && fine; ++x) fine = cudaStreamWaitEvent(s, ev[x * 3 + 2], 0) == cudaSuccess;
    if (!fine) (void)cudaGetLastError();
    return fine ? SPLAT_OK : SPLAT_ERR_LAUNCH;
}
