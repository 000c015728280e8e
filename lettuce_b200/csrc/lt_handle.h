// The lattice handle behind the C ABI's opaque lt_lattice, shared by the translation units
// that implement the ABI (lt_capi.cu, lt_ensemble.cu).
#pragma once
#include <vector>

#include "lettuce_b200.h"
#include "lt_backend.h"
#include "lt_host.h"

namespace lt {
// Records a CUDA error as this thread's last error; returns LT_ERR_NOMEM or LT_ERR_CUDA.
int cuda_error(cudaError_t e, const char* what);

// Makes a handle's device current for one C-ABI call and restores the caller's device after
struct DeviceScope
{
    int prev = -1;
    explicit DeviceScope(int dev)
    {
        int cur;
        if (cudaGetDevice(&cur) == cudaSuccess && cur != dev && cudaSetDevice(dev) == cudaSuccess) prev = cur;
    }
    ~DeviceScope()
    {
        if (prev >= 0) cudaSetDevice(prev);
    }
    DeviceScope(const DeviceScope&) = delete;
    DeviceScope& operator=(const DeviceScope&) = delete;
};

// Device memory of the lattice handles and ensembles.  A handle's buffers go back to a per-device store when
// it is destroyed and serve the next handle that asks for the same size (a flowed copy made for each
// measurement, one field after another): a cudaMalloc or cudaFree of a field takes from one to tens of
// milliseconds, more than most calls that need it (the measurement bundle on one flow level at 32 x 24^3
// in FP64: 10.3 ms a call with them, 5.1 without).  The store keeps at most an eighth of the device's memory,
// oldest given up first, and gives everything back when the last handle or ensemble goes.  Scratch that a call
// can do without is borrowed for the call: after it the buffer stays with its handle, and the pointer that
// holds it is set to null when the memory is taken.  An allocation that fails empties the store, takes the
// idle scratch of all handles and waits for the scratch of other threads' calls; borrowing only empties the
// store, and what was refused is not asked for again until another buffer has been returned.  Safe
// from any thread.
cudaError_t dev_alloc(int device, void** p, size_t bytes);
void dev_free(int device, void** p);    // expects no work in flight on the buffer
bool dev_borrow(int device, void** p, size_t bytes, uint64_t* refused);
void dev_lend(int device, void** p, cudaStream_t stream, bool keep);   // ends it; idle once the stream is, or kept
bool dev_claim(int device, void** p);   // makes an idle buffer the handle's own; false if there is none (any more)
void dev_release(int device);           // gives back all that no call needs: the store and the lent scratch
size_t dev_test(int device, size_t limit, bool deny);   // lt_memory_test; returns the bytes held
void dev_handle_created(int device);    // lattices and ensembles
void dev_handle_gone(int device);
} // namespace lt

#define LT_CK(call)                                                  \
    do {                                                             \
        cudaError_t e_ = (call);                                     \
        if (e_ != cudaSuccess) return lt::cuda_error(e_, #call);     \
    } while (0)

#define LT_TRY(call)                                                 \
    do {                                                             \
        int r_ = (call);                                             \
        if (r_ != LT_OK) return r_;                                  \
    } while (0)

struct lt_lattice
{
    int ext[4];
    int prec;
    int device = 0;
    lt::Geom g;
    const lt::Backend* be;
    cudaStream_t stream = nullptr;
    void* U = nullptr;       // links
    void* U2 = nullptr;      // ping-pong partner for flow / stout
    void* Z = nullptr;       // flow Z (algebra)
    void* P = nullptr;       // HMC momenta (algebra)
    void* F = nullptr;       // metadynamics force / Sigma (algebra)
    void* Ubak = nullptr;    // HMC backup of the links
    void* R = nullptr;       // clover planes
    void* Lam = nullptr;     // Lambda (algebra)
    void* Lt = nullptr;      // U^dag Lambda U (algebra)
    void* corners = nullptr; // corner sums of the clover planes (the clover derivative)
    void* Tloc = nullptr;    // link-local recursion term (full matrix)
    std::vector<void*> levels;   // smeared levels 1..n of the MetaD chain
    std::vector<void*> staples;  // the staples of levels 0..n-1 (full 3x3 per link), for the adjoint
    double* partials = nullptr;
    double* results = nullptr;
    double* h_results = nullptr; // pinned
    void* h_stage = nullptr;     // pinned: FP32 links packed in the device layout on the host (upload)
    int uploads = 0;             // lt_upload_links calls so far (the staging is set up from the second)
    double* d_aos = nullptr;     // staging buffer for host transfers (reference layout)
    unsigned* status = nullptr;  // device status word (lt_status_word) and scratch words
    void* chainA = nullptr;      // straight-line link products of lt_wilson_loop (FP64 full matrices)
    void* chainB = nullptr;
    // the chain kept between lt_wilson_loop_chain calls (the reference's U_chain): the buffer
    // holding it and the product U(x + o mu) ... U(x + (o + n - 1) mu) it holds (n = -1: none)
    void* chain_cur = nullptr;
    int chain_origin = 0, chain_len = -1;
    bool chain_contig = true;
    // gauge action of staples, sweeps, HMC forces / Hamiltonian and flow (lt_set_gauge_action):
    // stencil radius 1 (Wilson, the default) or 2 (plaquettes and 1x2 rectangles)
    int act_radius = 1;
    double act_cp = 1.0, act_cr = 0.0;
    // force of the gradient flow run into this handle (lt_set_flow_action): the gauge action's
    // (LT_FLOW_ACTION_GAUGE, the reference's GradientFlowKernel) or the Zeuthen flow's
    int flow_action = LT_FLOW_ACTION_GAUGE;
    void* planes = nullptr;      // plaquette planes of the Wilson force
    void* rectD = nullptr;       // two-link products of the rectangle forces (link field)
    void* rectE = nullptr;       // and their outer staples (full matrices)
    void* Xz = nullptr;          // Luescher-Weisz force of a Zeuthen flow stage (algebra)
    double* tensor = nullptr;    // FullTensor4D of lt_clover_tensor (FP64, reference layout)
    uint64_t refused = ~0ull;    // state of the store when it had no memory for scratch
    bool captured = false;       // a call has been captured into a graph: scratch stays
    mutable unsigned order = 0;  // launches of the order-alternating sweep and flow kernels

    lt::Ctx ctx() const
    {
        lt::Ctx c;
        c.g = g;
        c.stream = stream;
        c.partials = partials;
        c.results = results;
        c.status = status;
        c.rect = act_radius == 2;
        c.cp = act_cp;
        c.cr = act_cr;
        c.order = &order;
        return c;
    }
};
