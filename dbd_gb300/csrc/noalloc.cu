// noalloc.cu -- dbd_spgemm_noalloc: the whole multiply without allocating.
//
// Some callers of this library cannot allocate device memory: code that runs
// while a caching allocator owns the device (an allocator hook, a framework
// that forbids allocation outside its pool), latency-critical loops where
// cudaMalloc/cudaFree's implicit device synchronisation is not acceptable,
// and processes whose device memory is fully reserved up front.  They pass
// device-resident A, B and the output arrays; every temporary array of the
// pipeline (row products, bins, row lists, per-tile offsets, row counts, scan
// partials, dense-window cursors and next columns, the error word) is carved out of the
// file-scope array below instead of cudaMalloc'ed, and the pipeline runs on
// the caller's stream without creating streams or events.  What the host reads
// back (bin sizes, nnz(C), the error word) the kernels leave in pinned words
// allocated by the first call on a device.
//
// The array is kDbdNoallocScratchBytes (32 MiB) per GPU, held by every GPU
// that loads this library until the process exits.
#include <cstdio>
#include <cstring>
#include <mutex>

#include "../../include/dbd.h"
#include "dbd_internal.h"

namespace dbd {

namespace {

constexpr size_t kDbdNoallocScratchBytes = DBD_NOALLOC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kDbdNoallocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
bool g_setup_done[kMaxDevices] = {};
unsigned char *g_scratch_addr[kMaxDevices] = {};
Mailbox *g_mail[kMaxDevices] = {};  // pinned: what a call reads back
thread_local char g_msg[256];

// Failures are reported by the return code and one stderr line.
int report(int code) {
    fprintf(stderr, "dbd_spgemm_noalloc: %s\n", g_msg);
    return code;
}

int fail(int code, const char *msg) {
    snprintf(g_msg, sizeof(g_msg), "%s", msg);
    return report(code);
}

// Device address of the scratch array on the current device and the pinned
// words a call reads back (set-up once per device: kernel attributes and
// loading, cudaGetSymbolAddress, the pinned words).
int device_scratch(int dev, unsigned char **out, Mailbox **mail) {
    if (dev < 0 || dev >= kMaxDevices) return fail(DBD_ERR_INVALID, "device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_setup_mu);
    if (!g_setup_done[dev]) {
        init_kernel_attributes();
        // Every kernel the pipeline launches is loaded here, so that no later
        // call has the CUDA driver load a module (and allocate) on first launch.
        cudaError_t le = preload_analysis_kernels();
        if (le == cudaSuccess) le = preload_spgemm_kernels();
        if (le != cudaSuccess) {
            snprintf(g_msg, sizeof(g_msg), "loading the kernels: %s", cudaGetErrorString(le));
            return report(DBD_ERR_CUDA);
        }
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) {
            snprintf(g_msg, sizeof(g_msg), "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
            return report(DBD_ERR_CUDA);
        }
        // Allowed beside another thread's capture, which it has no part in.
        void *h = nullptr;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        e = cudaMallocHost(&h, sizeof(Mailbox));
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) {
            snprintf(g_msg, sizeof(g_msg), "cudaMallocHost: %s", cudaGetErrorString(e));
            return report(DBD_ERR_OOM_HOST);
        }
        g_mail[dev] = static_cast<Mailbox *>(h);
        g_scratch_addr[dev] = static_cast<unsigned char *>(p);
        g_setup_done[dev] = true;
    }
    *out = g_scratch_addr[dev];
    *mail = g_mail[dev];
    return DBD_OK;
}

struct Carver {
    unsigned char *base;
    size_t off = 0;
    template <class T> T *take(size_t count) {
        off = (off + 255) & ~size_t(255);
        T *p = reinterpret_cast<T *>(base + off);
        off += sizeof(T) * (count > 0 ? count : 1);
        return p;
    }
};

// Bytes of scratch that m rows and nnzA entries of A and mB rows of B count
// for: what callers size their inputs by.  The carving below in
// dbd_spgemm_noalloc takes the same regions in this order, some of them
// joined (the two columns of B's rows) or shared (the scan partials).
size_t scratch_bytes(int64_t m, int64_t nnzA, int64_t mB) {
    Carver c{nullptr};
    const size_t nt = (size_t)ceil_div(m, kTileRows) + 1;
    c.take<int32_t>((size_t)mB);                   // first columns of B's rows
    c.take<int32_t>((size_t)mB);                   // last columns
    c.take<int32_t>((size_t)m);                    // rowLo
    c.take<int32_t>((size_t)m);                    // rowHi
    c.take<int64_t>((size_t)m);                    // rowP
    c.take<uint8_t>((size_t)m);                    // symBin
    c.take<uint8_t>((size_t)m);                    // numBin
    c.take<int32_t>((size_t)m);                    // rowNnz
    c.take<int32_t>((size_t)m);                    // symList
    c.take<int32_t>((size_t)m);                    // numList
    c.take<int32_t>(kMaxBins * nt);                // hist
    c.take<int32_t>(kMaxBins * nt);                // symTileOff
    c.take<int32_t>(kMaxBins * nt);                // numTileOff
    c.take<int32_t>(kMaxBins + 1);                 // symStart
    c.take<int32_t>(kMaxBins + 1);                 // numStart
    c.take<int64_t>((size_t)ceil_div(m, kScanTile) + 1);  // scan partials
    c.take<int32_t>(2 * (size_t)nnzA);             // dense-window state
    c.take<int>(4);                                // err + flags
    c.take<uint32_t>(CTR_COUNT);                   // persistent kernels' row counters
    return c.off;
}

#define NA_CK(call)                                                                  \
    do {                                                                             \
        cudaError_t _e = (call);                                                     \
        if (_e != cudaSuccess) {                                                     \
            snprintf(g_msg, sizeof(g_msg), "%s: %s", #call, cudaGetErrorString(_e)); \
            return report(_e == cudaErrorMemoryAllocation ? DBD_ERR_OOM_DEVICE : DBD_ERR_CUDA); \
        }                                                                            \
    } while (0)

}  // namespace

}  // namespace dbd

using namespace dbd;

extern "C" int dbd_spgemm_noalloc(const dbd_csr_view *a, const dbd_csr_view *b, int64_t *c_row_ptr,
                                  int32_t *c_col_idx, double *c_val, int64_t c_capacity, int64_t *c_nnz,
                                  void *stream_handle) {
    g_msg[0] = '\0';
    if (!a || !c_row_ptr || !c_nnz) return fail(DBD_ERR_INVALID, "null argument");
    if (!b) b = a;
    *c_nnz = -1;
    if (!a->on_device || !b->on_device) return fail(DBD_ERR_INVALID, "operands must be device-resident");
    if (a->val_fp32 || b->val_fp32) return fail(DBD_ERR_INVALID, "operands must hold FP64 values");
    if (a->n_cols != b->n_rows) return fail(DBD_ERR_INVALID, "inner dimensions differ");
    if (a->n_rows < 0 || a->n_rows >= INT32_MAX || b->n_cols > INT32_MAX || a->nnz < 0 || b->nnz < 0 ||
        a->nnz > INT32_MAX || b->nnz > INT32_MAX)
        return fail(DBD_ERR_INVALID, "size out of range");
    if ((a->nnz > 0 && (!a->col_idx || !a->val)) || (b->nnz > 0 && (!b->col_idx || !b->val)) || !a->row_ptr ||
        !b->row_ptr)
        return fail(DBD_ERR_INVALID, "null operand array");
    const int64_t m = a->n_rows;
    const size_t need = scratch_bytes(m, a->nnz, b->n_rows);
    if (need > kDbdNoallocScratchBytes) {
        snprintf(g_msg, sizeof(g_msg),
                 "needs %zu bytes of scratch for %lld rows and %lld entries of A; the limit is %zu bytes",
                 need, (long long)m, (long long)a->nnz, kDbdNoallocScratchBytes);
        return report(DBD_ERR_BUDGET);
    }
    cudaStream_t s = (cudaStream_t)stream_handle;
    // The call synchronises with the host (bin sizes, nnz(C), the error word),
    // which a stream capture cannot hold: refuse it before anything is enqueued,
    // and before the set-up, whose pinned allocation would break the capture.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
        cudaGetLastError();
        cap = cudaStreamCaptureStatusNone;
    }
    if (cap != cudaStreamCaptureStatusNone)
        return fail(DBD_ERR_INVALID, "the stream is capturing: this call synchronises and cannot be captured");
    int dev = 0;
    NA_CK(cudaGetDevice(&dev));
    unsigned char *base = nullptr;
    Mailbox *box = nullptr;
    int rc = device_scratch(dev, &base, &box);
    if (rc) return rc;
    Carver c{base};  // the layout of scratch_bytes()
    const size_t nt = (size_t)ceil_div(m, kTileRows) + 1;
    int2 *range = c.take<int2>((size_t)b->n_rows);
    RowInfo ri;
    ri.lo = c.take<int32_t>((size_t)m);
    ri.hi = c.take<int32_t>((size_t)m);
    int64_t *rowP = c.take<int64_t>((size_t)m);
    ri.rowP = rowP;
    uint8_t *symBin = c.take<uint8_t>((size_t)m);
    uint8_t *numBin = c.take<uint8_t>((size_t)m);
    int32_t *rowNnz = c.take<int32_t>((size_t)m);
    int32_t *symList = c.take<int32_t>((size_t)m);
    int32_t *numList = c.take<int32_t>((size_t)m);
    int32_t *hist = c.take<int32_t>(kMaxBins * nt);
    int32_t *symTileOff = c.take<int32_t>(kMaxBins * nt);
    int32_t *numTileOff = c.take<int32_t>(kMaxBins * nt);
    int32_t *symStart = c.take<int32_t>(kMaxBins + 1);
    int32_t *numStart = c.take<int32_t>(kMaxBins + 1);
    // The tiles' entry sums take the symbolic tile offsets' place, which are
    // read last when the symbolic lists are written.
    static_assert(sizeof(int32_t) * kMaxBins >= sizeof(int64_t), "a tile's sum fits in its offsets");
    int64_t *tileSum = reinterpret_cast<int64_t *>(symTileOff);
    int32_t *state = c.take<int32_t>(2 * (size_t)a->nnz);
    int32_t *ctl = c.take<int32_t>(CTL_COUNT);
    int *err = ctl + CTL_ERR;
    uint32_t *ctrs = reinterpret_cast<uint32_t *>(ctl + CTL_CTR);

    // The array keeps the previous call's contents: clear what starts at zero.
    NA_CK(cudaMemsetAsync(ctl, 0, sizeof(int32_t) * CTL_COUNT, s));
    CsrDev A, B;
    A.m = a->n_rows; A.n = a->n_cols; A.nnz = a->nnz;
    A.ptr = a->row_ptr; A.idx = a->col_idx; A.val = (const double *)a->val;
    B.m = b->n_rows; B.n = b->n_cols; B.nnz = b->nnz;
    B.ptr = b->row_ptr; B.idx = b->col_idx; B.val = (const double *)b->val;
    int sms = 0;
    NA_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // Both operands are checked before any kernel gathers through them (the
    // work estimate looks at the flags; the host reads them with its results).
    // A's row ranges (into rowP, which the analysis fills later) are not used.
    if (b != a)
        launch_check_operand(A, reinterpret_cast<int2 *>(rowP), ctl + CTL_A, ctl + CTL_A + 1, ctl + CTL_A + 2, s, sms);
    launch_check_operand(B, range, ctl + CTL_B, ctl + CTL_B + 1, ctl + CTL_B + 2, s, sms);
    launch_row_minmax(B, range, ctl + CTL_B, ctl + CTL_B + 2, s, sms);
    // Analysis: products per row, symbolic bins, row lists.
    launch_row_products(A, B.ptr, range, ri, symBin, err, ctl, Tuning{}, s, sms);
    Binning sb{symBin, symList, hist, symTileOff, symStart};
    Mail mail;
    mail.to = box;
    mail.ctl = ctl;
    mail.binStart = symStart;
    launch_sym_lists(m, sb, ri, rowNnz, nullptr, 0, nullptr, nullptr, mail, s);
    NA_CK(cudaStreamSynchronize(s));
    NA_CK(cudaGetLastError());
    for (const int32_t *f : {box->flags + CTL_A, box->flags + CTL_B}) {
        if (f[0]) return fail(DBD_ERR_INVALID, "malformed row_ptr");
        if (f[1]) return fail(DBD_ERR_INVALID, "column index out of range");
    }
    if (box->err) return fail(DBD_ERR_DEVICE_CHECK, "a row has more than 2^31 products");
    int32_t symStart_h[kMaxBins + 1];
    memcpy(symStart_h, box->binStart, sizeof(symStart_h));
    const int sorted = box->flags[CTL_B + 2] ? 0 : 1;
    // Symbolic, row pointer, numeric bins.
    SymArgs sa;
    sa.A = A;
    sa.B = B;
    sa.list = symList;
    sa.binStart = symStart;
    sa.rowNnz = rowNnz;
    sa.ctr = ctrs;
    sa.numSms = sms;
    sa.bSorted = sorted;
    sa.err = err;
    sa.rowLo = ri.lo;
    sa.rowP = ri.rowP;
    sa.bRange = range;
    sa.rowHi = ri.hi;
    int launches = 0;
    for (int bin = SB_TINY; bin < SB_COUNT; ++bin)
        launch_symbolic_bin(sa, bin, symStart_h[bin], symStart_h[bin + 1] - symStart_h[bin], s, &launches);
    Binning nb{numBin, numList, hist, numTileOff, numStart};
    mail.binStart = numStart;
    mail.nnz = c_row_ptr + m;
    launch_num_lists(m, nb, ri, A.ptr, rowNnz, Tuning{}, tileSum, c_row_ptr, mail, s);
    NA_CK(cudaStreamSynchronize(s));
    NA_CK(cudaGetLastError());
    if (box->err) return fail(DBD_ERR_DEVICE_CHECK, "symbolic phase: device check failed");
    const int64_t nnz = box->nnz;
    int32_t numStart_h[kMaxBins + 1];
    memcpy(numStart_h, box->binStart, sizeof(numStart_h));
    *c_nnz = nnz;
    if (nnz > c_capacity) {
        snprintf(g_msg, sizeof(g_msg), "output needs %lld entries, capacity is %lld", (long long)nnz,
                 (long long)c_capacity);
        return report(DBD_ERR_BUDGET);
    }
    if (nnz > 0 && (!c_col_idx || !c_val)) return fail(DBD_ERR_INVALID, "null output array");
    NumArgs na;
    na.A = A;
    na.B = B;
    na.list = numList;
    na.Cp = c_row_ptr;
    na.outBase = 0;
    na.Ci = c_col_idx;
    na.Cv = c_val;
    na.state = state;
    na.bSorted = sorted;
    na.err = err;
    na.rowP = rowP;
    na.rowLo = ri.lo;
    na.numSms = sms;
    na.rowHi = ri.hi;
    na.ctr = ctrs;
    for (int bin = NB_TINY; bin < NB_COUNT; ++bin)
        launch_numeric_bin(na, bin, numStart_h[bin], numStart_h[bin + 1], s, &launches);
    NA_CK(cudaMemcpyAsync(&box->err, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    NA_CK(cudaStreamSynchronize(s));
    NA_CK(cudaGetLastError());
    if (box->err) return fail(DBD_ERR_DEVICE_CHECK, "numeric phase: device check failed");
    return DBD_OK;
}
