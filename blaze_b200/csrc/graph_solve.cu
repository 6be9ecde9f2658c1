// graph_solve.cu — the residual-controlled pressure solve as one CUDA graph.
//
// The host loop of blz_solve synchronises after every residual check to
// decide whether to continue (one device->host round trip per check_every
// sweeps).  Here the decision stays on the device: a conditional WHILE node
// runs {check_every sweeps, FP64 residual} until the residual's last kernel
// clears the condition (converged, or max_iter sweeps done); that kernel and
// the residual's first one also keep the loop's counters and times, so a check
// is two launches, not five.  The
// schedule is the host loop's exactly: one check before any sweep, then one
// after every check_every sweeps, capped at max_iter (a multiple of
// check_every on this path).
#include <cmath>

#include "kernels.cuh"

namespace blz {

#define CKG(x)                                      \
    do {                                            \
        cudaError_t e_ = (x);                       \
        if (e_ != cudaSuccess) { err = e_; goto done; } \
    } while (0)

cudaError_t build_solve_graph(const Geom &g, const SolveParams &sp, const float *rhs_r, const float *rhs_b,
                              float *p_r, float *p_b, double *partials, int n_partials, double *norm2,
                              SolveCtl *ctl, int chunk, int max_iter, double tol, int variant, cudaStream_t st,
                              cudaGraphExec_t *exec_out, int *body_kernels, int *prologue_kernels, float *q_r,
                              float *q_b, const DefectArrays *dfa, const ResidentWork &res) {
    cudaError_t err = cudaSuccess, swept = cudaSuccess;
    cudaGraph_t graph = nullptr, body = nullptr;
    cudaGraphConditionalHandle handle;
    cudaGraphNode_t cond_node;
    long long dummy = 0;
    bool broken = false;                                 // the body's capture has not ended well
    *exec_out = nullptr;
    // The stopping test: the FP64 residual of (rhs, p); for a defect-
    // correction solve (after sweeps) d folded into p and a fresh defect,
    // whose norms are those of the pressure p + d.  Returns its launches.
    auto check = [&](bool after) -> int {
        const LoopCheck loop{ctl, handle, after, chunk, max_iter, tol};
        if (!dfa) return launch_residual(g, sp, rhs_r, rhs_b, p_r, p_b, partials, n_partials, norm2, st, &loop);
        int n = 0;
        if (after) { launch_fold(g, dfa->p_r, dfa->p_b, dfa->d_r, dfa->d_b, st, &loop); ++n; }
        return n + launch_defect(g, sp, dfa->rhs_r, dfa->rhs_b, dfa->p_r, dfa->p_b, dfa->d_r, dfa->d_b, dfa->df_r,
                                 dfa->df_b, partials, n_partials, norm2, st, &loop);
    };
    CKG(cudaGraphCreate(&graph, 0));
    CKG(cudaGraphConditionalHandleCreate(&handle, graph, 0, 0));
    // Prologue: one check before any sweep, which resets the control block.
    CKG(cudaStreamBeginCaptureToGraph(st, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    *prologue_kernels = check(false);
    {
        cudaStreamCaptureStatus status;
        const cudaGraphNode_t *deps = nullptr;
        size_t ndeps = 0;
        CKG(cudaStreamGetCaptureInfo(st, &status, nullptr, nullptr, &deps, &ndeps));
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = handle;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        CKG(cudaGraphAddNode(&cond_node, graph, deps, ndeps, &cp));
        body = cp.conditional.phGraph_out[0];
        CKG(cudaStreamUpdateCaptureDependencies(st, &cond_node, 1, cudaStreamSetCaptureDependencies));
    }
    CKG(cudaStreamEndCapture(st, &graph));
    // Body: chunk sweeps (timed with the global timer), residual, decision.
    CKG(cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    broken = true;
    swept = launch_rbgs_sweeps(g, sp, rhs_r, rhs_b, p_r, p_b, chunk, st, &dummy, variant, q_r, q_b, res);
    *body_kernels = (int)dummy + check(true);
    CKG(cudaStreamEndCapture(st, &body));
    broken = false;
    CKG(swept);                                          // without its sweeps the loop would only check
    CKG(cudaGraphInstantiate(exec_out, graph, 0));
done:
    if (err != cudaSuccess) {
        cudaStreamCaptureStatus status;
        if (cudaStreamIsCapturing(st, &status) == cudaSuccess && status != cudaStreamCaptureStatusNone) {
            cudaGraph_t junk = nullptr;
            cudaStreamEndCapture(st, &junk);
            if (junk) cudaGraphDestroy(junk);
        }
        cudaGetLastError();
    }
    // A graph whose body's capture failed is left: destroying it crashes the driver
    // (580.159).
    if (graph && !broken) cudaGraphDestroy(graph);
    return err;
}

} // namespace blz
