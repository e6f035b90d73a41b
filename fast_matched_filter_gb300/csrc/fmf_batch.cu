// fmf_batch.cu -- many independent searches of uneven sizes in one graph.
//
// The reference runs one search per call (matched_filter.cu:171-399).  A
// batch records any number of searches (device pointers, each with its own
// T, S, C, L, N, step, normalisation and output layout) and runs them as one
// CUDA graph: every search's preprocessing kernels, then, for the tensor-core
// form, one persistent launch per mode and up to 64 searches that fit together over
// a shared tile queue (fmf_tc.cu); small FP32 searches run on the CUDA cores.  The graph is
// captured on the first run (on a stream the batch owns, joined to the
// caller's stream with events) and replayed afterwards; its scratch lives in
// graph memory nodes.  The searches' preprocessing (and the FP32 searches)
// are captured on kBatchBranches forked streams, so they become concurrent
// branches of the graph: each is small and would leave most of the GPU idle
// if they ran one after another.  Inputs are read when the graph runs, so a
// batch can be re-run after its input buffers were refilled.
#include <algorithm>
#include <cstring>
#include <memory>
#include <vector>

#include "fmf_common.cuh"

namespace fmf {
constexpr int kBatchBranches = 8;  // concurrent graph branches for the per-search work
// A graph holds the operand blocks of all its searches at once: FP32 searches with
// more than this stay on the CUDA cores, and so do all of a batch whose operands the
// device has no memory for (batch_fits).
constexpr size_t kBatchTemplateBytes = (size_t)1 << 30;
}

struct fmf_batch {
    int precision = FMF_PREC_SPLIT_BF16;
    int tile = 0;      // forced lag blocks per tensor-core tile (0 = largest that fits)
    int group = 0;     // templates interleaved per group of tile-queue items (0 = default)
    int device = -1;
    std::vector<fmf::Args> searches;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev_in = nullptr, ev_out = nullptr;
    // fork/join of the capture: branch streams and their events
    cudaStream_t branch[fmf::kBatchBranches] = {};
    cudaEvent_t ev_fork = nullptr, ev_main = nullptr;
    cudaEvent_t ev_join[fmf::kBatchBranches] = {}, ev_rejoin[fmf::kBatchBranches] = {};
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int launches = 0;  // kernel launches in one replay
    bool operands = false;  // it holds operands of FP32 searches on the tensor cores
};

namespace fmf {

// cuda_cores: FP32 searches run there without the tensor cores' operands.
static int batch_record(fmf_batch *b, cudaStream_t s, bool cuda_cores)
{
    int rc;
    cudaError_t e;
    // fork: the branch streams join the capture
    if ((e = cudaEventRecord(b->ev_fork, s)) != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "forking the batch capture: %s", cudaGetErrorString(e));
    for (int k = 0; k < kBatchBranches; k++)
        if ((e = cudaStreamWaitEvent(b->branch[k], b->ev_fork, 0)) != cudaSuccess)
            return set_error(FMF_ERR_CUDA, "forking the batch capture: %s", cudaGetErrorString(e));
    int status = FMF_OK;
    {
        std::vector<std::unique_ptr<Scratch>> bws;  // per-branch scratch, freed on its branch
        for (int k = 0; k < kBatchBranches; k++)
            bws.emplace_back(new Scratch(b->branch[k]));
        const size_t n = b->searches.size();
        std::vector<Problem> P(n);
        const int form = tc_form(b->precision);
        const bool fp32 = form == TC_FORM_FP32;
        std::vector<int> nb(n, 0);  // lag blocks per tile; 0: the CUDA cores
        const size_t psz = tc_prob_size();
        std::vector<unsigned char> probs(psz * n);
        for (size_t i = 0; i < n && status == FMF_OK; i++) {
            const int k = (int)(i % kBatchBranches);
            cudaStream_t si = b->branch[k];
            const Args &a = b->searches[i];
            nb[i] = fp32 ? (cuda_cores ? 0 : tc_fp32_nb(a.T, a.S * a.C, a.L, a.step, a.n_corr))
                         : tc_choose_nb((int)a.L, (int)a.step, form != TC_FORM_BF16, b->tile);
            if (!fp32 && nb[i] == 0) {
                status = set_error(FMF_ERR_SMEM, "search %zu: template length %zu with step %zu does not "
                                                 "fit a tensor-core tile", i, a.L, a.step);
                break;
            }
            if ((status = prepare_problem(a, *bws[k], si, &P[i], tc_pad(nb[i]), fp32 && nb[i])))
                break;
            if (fp32 && nb[i] && tc_template_bytes(P[i], nb[i]) > kBatchTemplateBytes)
                nb[i] = 0;
            if ((status = clear_outputs(P[i], si)))
                break;
            b->operands = b->operands || (fp32 && nb[i]);
            if (nb[i] == 0)
                status = launch_plain_all(P[i], si);
            else
                status = tc_prepare(P[i], form, nb[i], b->group, *bws[k], si,
                                    reinterpret_cast<TcProb *>(probs.data() + psz * i));
        }
        // join the branches, then the persistent launches on s
        for (int k = 0; k < kBatchBranches; k++)
            if ((e = cudaEventRecord(b->ev_join[k], b->branch[k])) != cudaSuccess ||
                (e = cudaStreamWaitEvent(s, b->ev_join[k], 0)) != cudaSuccess)
                status = status ? status : set_error(FMF_ERR_CUDA, "joining the batch capture: %s",
                                                     cudaGetErrorString(e));
        if (status == FMF_OK) {
            unsigned *err = nullptr;
            if ((status = device_error_word(&err)) == FMF_OK) {
                // One persistent launch per normalisation and output layout (each runs the
                // instantiation of its own mode) for the searches whose buffers fit together
                // (tc_group), each mode on a branch of its own: a mode's blocks start as the SMs
                // finish the one before.  The items of a launch are taken up in order of their
                // work, the long ones (1.3 ms of 7.4 in the uneven batch of 24) first.
                std::vector<size_t> order;
                for (size_t i = 0; i < n; i++)
                    if (nb[i])
                        order.push_back(i);
                const auto work = [&](size_t i) { return (size_t)P[i].SC * (P[i].L + 128 * P[i].step) * nb[i]; };
                std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) { return work(x) > work(y); });
                if ((e = cudaEventRecord(b->ev_main, s)) != cudaSuccess)
                    status = set_error(FMF_ERR_CUDA, "ordering the batch launches: %s", cudaGetErrorString(e));
                for (int mode = 0; mode < 4 && status == FMF_OK; mode++) {
                    cudaStream_t sm = b->branch[mode];
                    std::vector<unsigned char> grp;
                    for (size_t i : order)
                        if (P[i].normalize == (mode & 1) && (P[i].network_sum == 0) == (mode >> 1))
                            grp.insert(grp.end(), probs.begin() + psz * i, probs.begin() + psz * (i + 1));
                    const size_t ng = grp.size() / psz;
                    if (ng && (e = cudaStreamWaitEvent(sm, b->ev_main, 0)) != cudaSuccess)
                        status = set_error(FMF_ERR_CUDA, "ordering the batch launches: %s", cudaGetErrorString(e));
                    std::vector<unsigned char> taken(ng), shared;
                    int members[TC_MAX_PROBS];
                    for (int m; status == FMF_OK && (m = tc_group(reinterpret_cast<const TcProb *>(grp.data()), (int)ng,
                                                                  form, taken.data(), members)) > 0;) {
                        shared.clear();
                        for (int j = 0; j < m; j++)
                            shared.insert(shared.end(), grp.begin() + psz * members[j],
                                          grp.begin() + psz * (members[j] + 1));
                        unsigned long long *queue = nullptr;
                        if ((status = bws[mode]->get(&queue, 1, "tile queue")))
                            break;
                        if ((e = cudaMemsetAsync(queue, 0, sizeof(*queue), sm)) != cudaSuccess) {
                            status = set_error(FMF_ERR_CUDA, "clearing the tile queue: %s", cudaGetErrorString(e));
                            break;
                        }
                        status = tc_run(reinterpret_cast<const TcProb *>(shared.data()), m, form, 1, queue, err, sm);
                    }
                    if (ng && ((e = cudaEventRecord(b->ev_join[mode], sm)) != cudaSuccess ||
                               (e = cudaStreamWaitEvent(s, b->ev_join[mode], 0)) != cudaSuccess))
                        status = status ? status : set_error(FMF_ERR_CUDA, "joining the batch capture: %s",
                                                             cudaGetErrorString(e));
                }
                // FP32: the searches whose operands' flags leave them to the CUDA cores
                for (size_t i = 0; i < n && fp32 && status == FMF_OK; i++)
                    if (nb[i]) {
                        P[i].only_if = P[i].scan + 3 * P[i].SC;
                        P[i].left = err + kLeftWord;
                        status = launch_plain_all(P[i], s);
                    }
            }
        }
        // the branch scratch is freed after the work on s that reads it
        if ((e = cudaEventRecord(b->ev_main, s)) == cudaSuccess)
            for (int k = 0; k < kBatchBranches && e == cudaSuccess; k++)
                e = cudaStreamWaitEvent(b->branch[k], b->ev_main, 0);
        if (e != cudaSuccess && status == FMF_OK)
            status = set_error(FMF_ERR_CUDA, "ordering the batch scratch: %s", cudaGetErrorString(e));
    }  // branch scratch freed here, on the branch streams
    // rejoin the branches before the capture ends
    for (int k = 0; k < kBatchBranches; k++)
        if ((e = cudaEventRecord(b->ev_rejoin[k], b->branch[k])) != cudaSuccess ||
            (e = cudaStreamWaitEvent(s, b->ev_rejoin[k], 0)) != cudaSuccess)
            status = status ? status : set_error(FMF_ERR_CUDA, "joining the batch capture: %s",
                                                 cudaGetErrorString(e));
    rc = status;
    return rc;
}

static void batch_reset_graph(fmf_batch *b)
{
    if (b->exec)
        cudaGraphExecDestroy(b->exec);
    if (b->graph)
        cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}

// Records the searches into b->graph; *bytes: the scratch it asks for.
static int batch_capture(fmf_batch *b, bool cuda_cores, size_t *bytes)
{
    unsigned *err = nullptr;  // allocated outside the capture
    int rc = device_error_word(&err);
    if (rc)
        return rc;
    cudaError_t e = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "beginning graph capture: %s", cudaGetErrorString(e));
    const int before = fmf_last_launch_count();
    const size_t asked = scratch_asked();
    b->operands = false;
    rc = batch_record(b, b->stream, cuda_cores);
    *bytes = scratch_asked() - asked;
    b->launches = fmf_last_launch_count() - before;
    cudaGraph_t g = nullptr;
    e = cudaStreamEndCapture(b->stream, &g);
    if (rc) {
        if (g)
            cudaGraphDestroy(g);
        return rc;
    }
    if (e != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "ending graph capture: %s", cudaGetErrorString(e));
    b->graph = g;
    return FMF_OK;
}

// Whether the device has `bytes` for a graph's scratch, given back by the default pool if
// need be.  A graph takes its memory when it is launched, and what a launch that failed
// for want of it had taken stays lost to the process, so the batch asks first.  (A
// sixteenth and 128 MB more: the driver takes memory in large pieces.)
static bool batch_fits(int device, size_t bytes)
{
    const size_t need = bytes + bytes / 16 + ((size_t)128 << 20);
    unsigned long long used = 0, reserved = 0;
    size_t free = 0, total = 0;
    cudaMemPool_t pool;
    for (int attempt = 0; attempt < 2; attempt++) {
        if (cudaDeviceGetGraphMemAttribute(device, cudaGraphMemAttrUsedMemCurrent, &used) != cudaSuccess ||
            cudaDeviceGetGraphMemAttribute(device, cudaGraphMemAttrReservedMemCurrent, &reserved) != cudaSuccess ||
            cudaMemGetInfo(&free, &total) != cudaSuccess)
            break;
        if (need <= free + (reserved - used))
            return true;
        if (attempt == 0 && (cudaDeviceGetDefaultMemPool(&pool, device) != cudaSuccess ||
                             cudaMemPoolTrimTo(pool, 0) != cudaSuccess))
            break;
    }
    cudaGetLastError();
    return false;
}

}  // namespace fmf

extern "C" {

int fmf_batch_create(fmf_batch **out, int precision)
{
    fmf::set_error(FMF_OK, "");
    if (!out)
        return fmf::set_error(FMF_ERR_ARG, "null batch pointer");
    *out = nullptr;
    if (precision < FMF_PREC_FP32 || precision > FMF_PREC_BF16)
        return fmf::set_error(FMF_ERR_ARG, "unknown precision %d", precision);
    fmf_batch *b = new fmf_batch();
    b->precision = precision;
    cudaError_t e = cudaGetDevice(&b->device);
    if (e == cudaSuccess)
        e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess)
        e = cudaEventCreateWithFlags(&b->ev_in, cudaEventDisableTiming);
    if (e == cudaSuccess)
        e = cudaEventCreateWithFlags(&b->ev_out, cudaEventDisableTiming);
    if (e == cudaSuccess)
        e = cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming);
    if (e == cudaSuccess)
        e = cudaEventCreateWithFlags(&b->ev_main, cudaEventDisableTiming);
    for (int k = 0; k < fmf::kBatchBranches && e == cudaSuccess; k++) {
        e = cudaStreamCreateWithFlags(&b->branch[k], cudaStreamNonBlocking);
        if (e == cudaSuccess)
            e = cudaEventCreateWithFlags(&b->ev_join[k], cudaEventDisableTiming);
        if (e == cudaSuccess)
            e = cudaEventCreateWithFlags(&b->ev_rejoin[k], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) {
        fmf_batch_destroy(b);
        return fmf::set_error(FMF_ERR_CUDA, "creating a batch: %s", cudaGetErrorString(e));
    }
    *out = b;
    return FMF_OK;
}

int fmf_batch_set_tiles(fmf_batch *b, int lag_blocks, int template_group)
{
    fmf::set_error(FMF_OK, "");
    if (!b)
        return fmf::set_error(FMF_ERR_ARG, "null batch");
    if (lag_blocks != 0 && lag_blocks != 32 && lag_blocks != 64 && lag_blocks != 128)
        return fmf::set_error(FMF_ERR_ARG, "lag_blocks must be 0, 32, 64 or 128");
    if (template_group < 0 || template_group > 1024)
        return fmf::set_error(FMF_ERR_ARG, "template_group must be in [0, 1024]");
    b->tile = lag_blocks;
    b->group = template_group;
    fmf::batch_reset_graph(b);
    return FMF_OK;
}

int fmf_batch_add(fmf_batch *b, const float *templates, const float *sum_square_templates,
                  const int *moveouts, const float *data, const float *weights, size_t step,
                  size_t n_samples_template, size_t n_samples_data, size_t n_templates,
                  size_t n_stations, size_t n_components, size_t n_corr, float *cc_out,
                  int normalize, int sum_cc_mode)
{
    fmf::set_error(FMF_OK, "");
    if (!b)
        return fmf::set_error(FMF_ERR_ARG, "null batch");
    fmf::Args a;
    a.tpl = templates;
    a.sst = sum_square_templates;
    a.mo = moveouts;
    a.data = data;
    a.w = weights;
    a.out = cc_out;
    a.step = step;
    a.L = n_samples_template;
    a.N = n_samples_data;
    a.T = n_templates;
    a.S = n_stations;
    a.C = n_components;
    a.n_corr = n_corr;
    a.normalize = normalize;
    a.sum_mode = sum_cc_mode;
    a.precision = b->precision;
    a.flags = FMF_FLAG_DEVICE_POINTERS;
    int rc = fmf::validate_args(a);
    if (rc)
        return rc;
    b->searches.push_back(a);
    fmf::batch_reset_graph(b);
    return FMF_OK;
}

int fmf_batch_run(fmf_batch *b, void *stream)
{
    fmf::set_error(FMF_OK, "");
    if (!b)
        return fmf::set_error(FMF_ERR_ARG, "null batch");
    if (b->searches.empty())
        return fmf::set_error(FMF_ERR_ARG, "empty batch");
    int dev = -1;
    cudaGetDevice(&dev);
    if (dev != b->device)
        return fmf::set_error(FMF_ERR_ARG, "batch created on device %d, current device is %d", b->device,
                              dev);
    cudaGetLastError();
    cudaStream_t user = (cudaStream_t)stream;
    cudaError_t e;
    if (!b->exec) {
        size_t bytes = 0;
        int rc = fmf::batch_capture(b, false, &bytes);
        if (rc == FMF_OK && b->operands && !fmf::batch_fits(dev, bytes)) {
            fmf::batch_reset_graph(b);
            rc = fmf::batch_capture(b, true, &bytes);
        }
        if (rc)
            return rc;
        e = cudaGraphInstantiate(&b->exec, b->graph, 0);
        if (e != cudaSuccess) {
            fmf::batch_reset_graph(b);
            return fmf::set_error(FMF_ERR_CUDA, "instantiating the batch graph: %s", cudaGetErrorString(e));
        }
    }
    if ((e = cudaEventRecord(b->ev_in, user)) != cudaSuccess ||
        (e = cudaStreamWaitEvent(b->stream, b->ev_in, 0)) != cudaSuccess ||
        (e = cudaGraphLaunch(b->exec, b->stream)) != cudaSuccess ||
        (e = cudaEventRecord(b->ev_out, b->stream)) != cudaSuccess ||
        (e = cudaStreamWaitEvent(user, b->ev_out, 0)) != cudaSuccess)
        return fmf::set_error(FMF_ERR_CUDA, "launching the batch graph: %s", cudaGetErrorString(e));
    return FMF_OK;
}

int fmf_batch_launch_count(const fmf_batch *b) { return b ? b->launches : 0; }

int fmf_batch_destroy(fmf_batch *b)
{
    if (!b)
        return FMF_OK;
    if (b->stream)
        cudaStreamSynchronize(b->stream);
    fmf::batch_reset_graph(b);
    if (b->ev_in)
        cudaEventDestroy(b->ev_in);
    if (b->ev_out)
        cudaEventDestroy(b->ev_out);
    if (b->ev_fork)
        cudaEventDestroy(b->ev_fork);
    if (b->ev_main)
        cudaEventDestroy(b->ev_main);
    for (int k = 0; k < fmf::kBatchBranches; k++) {
        if (b->ev_join[k])
            cudaEventDestroy(b->ev_join[k]);
        if (b->ev_rejoin[k])
            cudaEventDestroy(b->ev_rejoin[k]);
        if (b->branch[k])
            cudaStreamDestroy(b->branch[k]);
    }
    if (b->stream)
        cudaStreamDestroy(b->stream);
    delete b;
    return FMF_OK;
}

}  // extern "C"
