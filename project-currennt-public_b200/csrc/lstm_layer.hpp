// Implementation object behind the opaque b2_lstm handle; also used directly by the layer stack.
#pragma once
#include "common.cuh"

namespace b2 {

struct LstmLayerImpl {
    b2_lstm_desc desc{};
    int D = 1, els = 0;
    int T = 0, Tmin = 0;
    bool forward_done = false;
    int recurrence_mode = 1;   // b2_lstm_set_recurrence_mode
    bool force_ffma = false;
    float x_bound = 0.0f;         // > 0: no |entry| of the layer's input exceeds it (the layer stack knows its layers' ranges)
    bool check_padding = false;   // load_sequences verifies that padding frames trail their sequences
    int *pad_dev = nullptr;       // result word of that check
    LstmBuffers bufs{};
    const int *list = nullptr;    // the frames of the fraction the sweeps run, n_list of them (NULL: the products take all frames)
    int n_list = 0;
    float *ws = nullptr;       // scratch: split-K partials, vector-gradient partials
    size_t ws_floats = 0;
    size_t state_bytes = 0;
    // arena for the tf32 hi/lo operand copies of the tensor-core GEMMs: the layer stack lends its
    // shared one (set before create()); a stand-alone layer makes its own
    TcScratch *scratch = nullptr, *own_scratch = nullptr;
    // persistent kernels: exchange buffers, device status word, running step tag
    unsigned long long *xchg = nullptr;
    int *status_dev = nullptr;
    unsigned tag_next = 1;
    // tensor-core recurrence (large batches): hi/lo buffers, allocated on first use
    TcRecBuffers tcrec{};
    // of lstm_persistent.cu: mode 2 forces clusters, 4 forces L2
    int persistent_transport() const { return recurrence_mode == 2 ? 1 : (recurrence_mode == 4 ? 0 : 2); }
    bool tcrec_used = false;      // this fraction's forward sweep ran on the tensor-core recurrence
    // persistent tensor-core recurrence: weight images, exchange words (allocated on first use)
    PtcBuffers ptc{};
    bool ptc_used = false;        // this fraction's forward sweep ran on the persistent tensor-core kernels
    bool cluster_used = false;    // this fraction's forward sweep ran on the register-resident cluster kernels
    // persistent tensor-core recurrence of wide layers: exchange buffers (allocated on first use)
    WideBuffers wide{};
    bool wide_used = false;       // this fraction's forward sweep ran on them
    bool want_wide() const;
    int ensure_wide();
    bool want_cluster() const;
    bool want_ptc() const;
    int ensure_ptc();
    // which recurrence the last forward / backward sweep actually ran, as a family (b2_lstm_recurrence_path) and by the name of its source file
    // (b2_lstm_recurrence_kernel): families 1 and 5 have two members each
    int fwd_path = -1, bwd_path = -1;
    const char *fwd_kernel = "", *bwd_kernel = "";
    bool want_tc_recurrence() const;
    int ensure_tcrec();
    int check_status(cudaStream_t st);   // synchronises st; returns the kernels' status word
    // optional per-phase timing hooks (set by the layer stack when profiling is on)
    void *prof_ctx = nullptr;
    void (*prof_begin)(void *, const char *) = nullptr;
    void (*prof_end)(void *) = nullptr;

    int create(const b2_lstm_desc &d);
    void destroy();
    LstmShape shape() const;
    int load_sequences(int cur_max, int cur_min, const char *pat_dev);
    // The frames of the loaded fraction that the sweeps run (device list: t below the slot's length or the shortest one), where the products
    // are to leave out the others; NULL: they are not.  A frame that is missing keeps stale pre-activations: the list must hold every such frame.
    void set_frame_list(const int *map, int n);
    int forward(const float *w, const float *x, float *y, cudaStream_t st);
    int backward(const float *w, const float *x, const float *y, const float *dy, float *dx, float *dw,
                 cudaStream_t st);
    int gemm(float *C, long ldc, const float *A, long sam, long sak, const float *B, long sbk, long sbn, int m, int n,
             int k, bool acc, cudaStream_t st);
};

}  // namespace b2
