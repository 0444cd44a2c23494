// batch.cuh -- batched rendering of many scenes of uneven size and sample
// budget in ONE persistent kernel launch, captured in a CUDA graph (included
// by integrator.cu: it reuses shade_path, the traversal and the camera).
//
// Work is a flat list of units (item, pixel, chunk of `chunk_spp` samples),
// chunk-major within an item so that a warp's 32 consecutive units are 32
// neighbouring pixels of one chunk.  Warps fetch 32 units at a time from a
// global counter (dynamic load balance across scenes of 1k..2M triangles and
// 16..512 spp).  Each thread traces its unit's samples end to end (camera ray,
// bounces, shadow rays traced inline), sums the clamped sample radiance with
// Neumaier compensation and stores the chunk partial; a resolve kernel sums
// the chunks of every pixel in chunk order.  The result is deterministic and
// independent of the launch shape.  Launch shape (block size, blocks per SM)
// and chunk size come from the autotuner below.

namespace ptb {

struct BatchItemDev {
    DeviceScene scene;
    pt_camera_frame cam;
    int32_t  width, height, spp, spf, max_depth, sampler, arg_rtl, watertight;
    uint32_t pcg_seed, first_frame, chunk_spp, chunks;
    unsigned long long unit_begin;   // first global unit of this item
    unsigned long long pixel_begin;  // first global pixel of this item
    float4*  partial;                // chunks x pixels: rgb sum, w = samples
    float4*  out;                    // pixels: mean, w = 1
};

__device__ __forceinline__ int find_item(const BatchItemDev* items, int n, unsigned long long u, bool by_pixel) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const unsigned long long b = by_pixel ? __ldg(&items[mid].pixel_begin) : __ldg(&items[mid].unit_begin);
        if (b <= u) lo = mid; else hi = mid - 1;
    }
    return lo;
}

struct BatchCounters { uint32_t camera, ext, shadow; };

// One sample of pathTrace (path.cu:62-206) traced end to end.
__device__ f3 trace_path_inline(const BatchItemDev& it, int x, int y, PathRng& rng, BatchCounters& bc,
                                uint32_t& err) {
    f3 o, d;
    camera_ray(it.cam, it.width, it.height, x, y, rng, o, d);
    f3 T = mk(1.0f), L = mk(0.0f);
    float last_pdf = 0.0f;
    bool last_delta = true;
    InlineSink sink{it.scene, it.watertight != 0, mk(0.0f), 0u, 0u, TraceCounters{0, 0}};
    TraceCounters tc{0, 0};
    for (int depth = 0; depth < it.max_depth; ++depth) {
        const RayInv r = make_ray_inv(o.x, o.y, o.z, d.x, d.y, d.z);
        float t, u, v;
        const int prim = trace_closest(it.scene, r, it.watertight != 0, t, u, v, err, tc);
        if (depth == 0) ++bc.camera; else ++bc.ext;
        const bool last = depth == it.max_depth - 1;
        f3 no, nd;
        const bool cont = shade_path<false>(it.scene, it.arg_rtl, depth, last, o, d, make_float4(t, __int_as_float(prim), u, v),
                                     T, last_pdf, last_delta, L, rng, no, nd, sink);
        if (!cont || last) break;
        o = no;
        d = nd;
    }
    err |= sink.err;
    bc.shadow += sink.rays;
    L += sink.acc;
    return mk(fminf(L.x, 100.0f), fminf(L.y, 100.0f), fminf(L.z, 100.0f));
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_batch_persistent(const BatchItemDev* __restrict__ items, int n_items,
                                                             unsigned long long total_units,
                                                             unsigned long long* next_unit,
                                                             unsigned long long* stats, uint32_t* err_out) {
    const int lane = threadIdx.x & 31;
    BatchCounters bc{0, 0, 0};
    uint32_t err = 0;
    uint32_t paths = 0;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(next_unit, 32ull);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= total_units) break;
        const unsigned long long u = base + static_cast<unsigned long long>(lane);
        if (u < total_units) {
            const int k = find_item(items, n_items, u, false);
            const BatchItemDev& it = items[k];
            const unsigned long long local = u - it.unit_begin;
            const uint32_t npix = static_cast<uint32_t>(it.width) * static_cast<uint32_t>(it.height);
            const uint32_t chunk = static_cast<uint32_t>(local / npix);
            const uint32_t pix = static_cast<uint32_t>(local % npix);
            const int x = static_cast<int>(pix % static_cast<uint32_t>(it.width));
            const int y = static_cast<int>(pix / static_cast<uint32_t>(it.width));
            const uint32_t s0 = chunk * it.chunk_spp;
            const uint32_t s1 = min(s0 + it.chunk_spp, static_cast<uint32_t>(it.spp));
            float sx = 0.0f, sy = 0.0f, sz = 0.0f, cx = 0.0f, cy = 0.0f, cz = 0.0f;
            for (uint32_t s = s0; s < s1; ++s) {
                const uint32_t frame = it.first_frame + s / static_cast<uint32_t>(it.spf);
                const uint32_t i = s % static_cast<uint32_t>(it.spf);
                PathRng rng = make_rng(it.sampler, x, y, frame, static_cast<uint32_t>(it.spf), i, it.pcg_seed);
                const f3 L = trace_path_inline(it, x, y, rng, bc, err);
                neumaier(sx, cx, L.x);
                neumaier(sy, cy, L.y);
                neumaier(sz, cz, L.z);
                ++paths;
            }
            it.partial[static_cast<size_t>(chunk) * npix + pix] =
                make_float4(sx + cx, sy + cy, sz + cz, static_cast<float>(s1 - s0));
        }
    }
    warp_count(stats + kStatCameraRays, bc.camera);
    warp_count(stats + kStatExtRays, bc.ext);
    warp_count(stats + kStatShadowRays, bc.shadow);
    warp_count(stats + kStatPaths, paths);
    if (err) atomicOr(err_out, err);
}

__global__ void k_batch_resolve(const BatchItemDev* __restrict__ items, int n_items, unsigned long long total_pixels) {
    for (unsigned long long g = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; g < total_pixels;
         g += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        const int k = find_item(items, n_items, g, true);
        const BatchItemDev& it = items[k];
        const uint32_t npix = static_cast<uint32_t>(it.width) * static_cast<uint32_t>(it.height);
        const uint32_t pix = static_cast<uint32_t>(g - it.pixel_begin);
        float sx = 0.0f, sy = 0.0f, sz = 0.0f, cx = 0.0f, cy = 0.0f, cz = 0.0f, n = 0.0f;
        for (uint32_t c = 0; c < it.chunks; ++c) {
            const float4 p = it.partial[static_cast<size_t>(c) * npix + pix];
            neumaier(sx, cx, p.x);
            neumaier(sy, cy, p.y);
            neumaier(sz, cz, p.z);
            n += p.w;
        }
        it.out[pix] = n > 0.0f ? make_float4((sx + cx) / n, (sy + cy) / n, (sz + cz) / n, 1.0f)
                               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

struct BatchPlan {
    std::vector<BatchItemDev> items;
    unsigned long long total_units = 0, total_pixels = 0;
    size_t partial_floats4 = 0, out_floats4 = 0;
};

int launch_persistent(int block, int grid, const BatchItemDev* d_items, int n, unsigned long long total,
                      unsigned long long* next, unsigned long long* stats, uint32_t* err, cudaStream_t st) {
    switch (block) {
        case 64: k_batch_persistent<64><<<grid, 64, 0, st>>>(d_items, n, total, next, stats, err); break;
        case 128: k_batch_persistent<128><<<grid, 128, 0, st>>>(d_items, n, total, next, stats, err); break;
        case 256: k_batch_persistent<256><<<grid, 256, 0, st>>>(d_items, n, total, next, stats, err); break;
        default: set_error("block size must be 64, 128 or 256"); return PT_ERR_INVALID;
    }
    PT_CU(cudaGetLastError());
    return PT_OK;
}

int max_blocks_per_sm(int block) {
    int v = 1;
    const void* k = block == 64 ? reinterpret_cast<const void*>(k_batch_persistent<64>)
                  : block == 128 ? reinterpret_cast<const void*>(k_batch_persistent<128>)
                                 : reinterpret_cast<const void*>(k_batch_persistent<256>);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k, block, 0) != cudaSuccess || v < 1) { cudaGetLastError(); v = 1; }
    return v;
}

// The camera an item renders: its own, else its scene's.
const pt_camera& item_camera(const pt_batch_item& it) { return it.camera ? *it.camera : it.scene->host.camera; }

BatchPlan make_plan(const pt_batch_item* in, uint32_t n, uint32_t chunk_spp, int cap_spp) {
    BatchPlan plan;
    plan.items.resize(n);
    for (uint32_t k = 0; k < n; ++k) {
        const pt_scene* s = in[k].scene;
        const pt_camera& cam = item_camera(in[k]);
        BatchItemDev& it = plan.items[k];
        std::memset(&it, 0, sizeof(it));
        it.scene = device_view(s);
        it.cam = camera_frame(cam);
        it.width = cam.width;
        it.height = cam.height;
        it.spp = cap_spp > 0 ? std::min(cap_spp, in[k].spp) : in[k].spp;
        it.spf = s->host.settings.sample_per_frame;
        it.max_depth = in[k].max_depth >= 0 ? in[k].max_depth : s->host.settings.max_depth;
        it.sampler = s->host.settings.sampler_type;
        it.arg_rtl = s->host.settings.arg_order == PT_ARGS_RTL ? 1 : 0;
        it.watertight = (s->host.settings.flags & PT_FLAG_WATERTIGHT) ? 1 : 0;
        it.pcg_seed = s->host.settings.pcg_seed;
        it.first_frame = in[k].first_frame;
        it.chunk_spp = chunk_spp;
        it.chunks = (static_cast<uint32_t>(it.spp) + chunk_spp - 1) / chunk_spp;
        const unsigned long long npix = static_cast<unsigned long long>(it.width) * it.height;
        it.unit_begin = plan.total_units;
        it.pixel_begin = plan.total_pixels;
        plan.total_units += npix * it.chunks;
        plan.total_pixels += npix;
        plan.partial_floats4 += npix * it.chunks;
        plan.out_floats4 += npix;
    }
    return plan;
}

// ---- wavefront mode: every item runs the wavefront integrator as one branch
//      of a single CUDA graph (branches run concurrently) ----
struct BatchSlot {
    const pt_scene* scene = nullptr;
    int             dup = 0;          // k-th item of the batch with this scene
    pt_integrator*  integ = nullptr;
    pt_film*        film = nullptr;
    // a guided item samples through a view of its guide: the guide's network
    // (read only), this slot's own mixture buffer -- items that share one
    // guide run concurrently in the batch graph
    GuideState      gview{};
};
std::mutex g_slot_mu;
// one integrator + film per scene, reused across batches (heap cells: the
// addresses handed out stay valid while the list grows)
std::vector<std::unique_ptr<BatchSlot>> g_slots;
std::vector<std::pair<int, std::vector<cudaStream_t>>> g_side_streams;   // per device
constexpr int kBatchBranches = 16;

void slot_release(BatchSlot& sl) {
    if (sl.integ) { integrator_free(sl.integ); delete sl.integ; }
    if (sl.film) { film_free(sl.film); delete sl.film; }
    sl.gview.params = nullptr;   // owned by the guide
    guide_free(sl.gview);
    sl = BatchSlot{};
}

// Integrator and film for the dup-th batch item rendering scene s at w x h
// on its device; caller holds g_slot_mu.
int batch_slot(const pt_scene* s, int dup, int w, int h, BatchSlot*& out) {
    const int dev = s->dev.device;
    out = nullptr;
    for (auto& cell : g_slots) {
        BatchSlot& sl = *cell;
        if (sl.scene != s || sl.dup != dup) continue;
        if (sl.film->width == w && sl.film->height == h && sl.film->device == dev) { out = &sl; return PT_OK; }
        slot_release(sl);
        sl.scene = s;
        out = &sl;
        break;
    }
    if (!out) {
        g_slots.push_back(std::make_unique<BatchSlot>());
        out = g_slots.back().get();
        out->scene = s;
        out->dup = dup;
    }
    out->integ = new pt_integrator();
    out->film = new pt_film();
    out->film->width = w; out->film->height = h; out->film->device = dev;
    return film_alloc(out->film);
}

int side_streams(int device, std::vector<cudaStream_t>*& out) {
    for (auto& kv : g_side_streams) if (kv.first == device) { out = &kv.second; return PT_OK; }
    g_side_streams.emplace_back(device, std::vector<cudaStream_t>(kBatchBranches, nullptr));
    out = &g_side_streams.back().second;
    for (cudaStream_t& x : *out) PT_CU(cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking));
    return PT_OK;
}

__global__ void k_batch_film_mean(const float4* sum, const float4* comp, float4* out, int n) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float4 s = sum[p], c = comp[p];
        out[p] = s.w > 0.0f ? make_float4((s.x + c.x) / s.w, (s.y + c.y) / s.w, (s.z + c.z) / s.w, 1.0f)
                            : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// Renders the batch in wavefront mode: the path slots (budget) are shared
// among the items in proportion to their work (pixels x spp), every item gets
// at least one sample per pixel in flight.  Returns the graph's device time.
// write_out = false (calibration) skips the output.
int batch_wavefront(const pt_batch_item* in, uint32_t n, int out_is_device, int64_t budget, bool write_out,
                    cudaStream_t st, float* ms_out, pt_render_stats* stats) {
    std::lock_guard<std::mutex> lk(g_slot_mu);
    const int device = in[0].scene->dev.device;
    std::vector<cudaStream_t>* side = nullptr;
    if (int rc = side_streams(device, side)) return rc;
    double work_total = 0.0;
    for (uint32_t k = 0; k < n; ++k)
        work_total += static_cast<double>(item_camera(in[k]).width) * item_camera(in[k]).height * in[k].spp;
    std::vector<BatchSlot*> slots(n, nullptr);
    std::vector<WaveParams> P(n);
    std::vector<int64_t> total(n);
    for (uint32_t k = 0; k < n; ++k) {
        pt_scene* s = in[k].scene;
        int dup = 0;   // items sharing a scene need their own wavefront and film
        for (uint32_t j = 0; j < k; ++j) dup += in[j].scene == s ? 1 : 0;
        const pt_camera& cam = item_camera(in[k]);
        if (int rc = batch_slot(s, dup, cam.width, cam.height, slots[k])) return rc;
        pt_scene_params prm;
        if (int rc = pt_scene_build_params(s, &prm)) return rc;
        if (in[k].camera) {
            prm.camera = camera_frame(cam);
            prm.width = cam.width;
            prm.height = cam.height;
        }
        // guide view (or none) for this item's wavefront
        if (!slots[k]->integ->wf) slots[k]->integ->wf = new Wavefront();
        GuideState* gs_k = nullptr;
        if (in[k].guide) {
            const GuideState& g = guide_state(in[k].guide);
            GuideState& v = slots[k]->gview;
            if (v.device != g.device || v.net.w != g.net.w) {
                v.params = nullptr;
                guide_free(v);
                v = GuideState{};
                v.device = g.device;
            }
            v.net = g.net;
            v.step = g.step;
            v.alpha = g.alpha;
            v.lr = g.lr;
            v.infer = g.infer;
            v.mode = PT_GUIDE_USE;
            gs_k = &v;
        }
        if (slots[k]->integ->wf->guide != gs_k) {
            slots[k]->integ->wf->guide = gs_k;
            Wavefront& wfk = *slots[k]->integ->wf;
            if (wfk.graph) { cudaGraphExecDestroy(wfk.graph); wfk.graph = nullptr; wfk.graph_key.clear(); }
        }
        if (in[k].max_depth >= 0) prm.max_depth = in[k].max_depth;
        const int64_t npix = static_cast<int64_t>(prm.width) * prm.height;
        total[k] = in[k].spp;
        const double share = static_cast<double>(budget) * (static_cast<double>(npix) * in[k].spp / work_total);
        const int64_t item_budget = std::max<int64_t>(npix, static_cast<int64_t>(share));
        int lanes = 1;
        if (int rc = prepare_wave(slots[k]->integ, slots[k]->film, s, &prm, total[k], item_budget, P[k], lanes)) return rc;
        if (int rc = film_clear(slots[k]->film)) return rc;
        if (int rc = integrator_reset_stats(slots[k]->integ)) return rc;
    }
    PT_CU(cudaDeviceSynchronize());
    cudaEvent_t fork = nullptr, e0 = nullptr, e1 = nullptr;
    std::vector<cudaEvent_t> join(kBatchBranches, nullptr);
    struct EvGuard { std::vector<cudaEvent_t*> ev; ~EvGuard() { for (auto* e : ev) if (*e) cudaEventDestroy(*e); } } eg;
    eg.ev = {&fork, &e0, &e1};
    PT_CU(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    PT_CU(cudaEventCreate(&e0));
    PT_CU(cudaEventCreate(&e1));
    for (cudaEvent_t& e : join) { PT_CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)); eg.ev.push_back(&e); }
    const int branches = static_cast<int>(std::min<uint32_t>(n, kBatchBranches));
    cudaGraph_t graph = nullptr;
    PT_CU(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    int rc = PT_OK;
    cudaError_t ce = cudaEventRecord(fork, st);
    for (int j = 0; j < branches && ce == cudaSuccess; ++j) ce = cudaStreamWaitEvent((*side)[j], fork, 0);
    for (uint32_t k = 0; k < n && ce == cudaSuccess && rc == PT_OK; ++k) {
        cudaStream_t bs = (*side)[k % branches];
        Wavefront& wf = *slots[k]->integ->wf;
        k_begin<<<1, 1, 0, bs>>>(P[k].pass, in[k].first_frame);
        rc = enqueue_batch(wf, P[k], total[k], bs, nullptr, wf.guide, false);
        if (rc == PT_OK && write_out) {
            const int np = P[k].npix;
            float4* out = out_is_device ? reinterpret_cast<float4*>(in[k].out_rgba)
                                        : static_cast<float4*>(slots[k]->film->resolve);
            k_batch_film_mean<<<std::min((np + 255) / 256, wf.sms * 8), 256, 0, bs>>>(
                P[k].f_sum, P[k].f_comp, out, np);
        }
    }
    for (int j = 0; j < branches && ce == cudaSuccess; ++j) {
        ce = cudaEventRecord(join[j], (*side)[j]);
        if (ce == cudaSuccess) ce = cudaStreamWaitEvent(st, join[j], 0);
    }
    const cudaError_t ec = cudaStreamEndCapture(st, &graph);
    if (rc != PT_OK || ce != cudaSuccess || ec != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        if (rc == PT_OK) {
            set_error(std::string("batch graph capture: ") + cudaGetErrorString(ce != cudaSuccess ? ce : ec));
            rc = PT_ERR_CUDA;
        }
        return rc;
    }
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) { set_error(std::string("batch graph instantiate: ") + cudaGetErrorString(ei)); return PT_ERR_CUDA; }
    PT_CU(cudaEventRecord(e0, st));
    const cudaError_t el = cudaGraphLaunch(exec, st);
    PT_CU(cudaEventRecord(e1, st));
    const cudaError_t es = cudaStreamSynchronize(st);
    cudaGraphExecDestroy(exec);
    if (el != cudaSuccess || es != cudaSuccess) {
        set_error(std::string("batch launch: ") + cudaGetErrorString(el != cudaSuccess ? el : es));
        return PT_ERR_CUDA;
    }
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms_out) *ms_out = ms;
    pt_render_stats sum;
    std::memset(&sum, 0, sizeof(sum));
    for (uint32_t k = 0; k < n; ++k) {
        if (int rc2 = integrator_check(slots[k]->integ, false)) return rc2;
        pt_render_stats s1;
        if (int rc2 = integrator_stats(slots[k]->integ, &s1)) return rc2;
        sum.camera_rays += s1.camera_rays; sum.extension_rays += s1.extension_rays;
        sum.shadow_rays += s1.shadow_rays; sum.paths += s1.paths;
        if (write_out && !out_is_device)
            PT_CU(cudaMemcpy(in[k].out_rgba, slots[k]->film->resolve,
                             static_cast<size_t>(P[k].npix) * sizeof(float4), cudaMemcpyDeviceToHost));
    }
    if (stats) {
        *stats = sum;
        stats->total_ms = ms;
        uint64_t launches = 0;
        for (uint32_t k = 0; k < n; ++k) {
            const int lanes = std::max(1, P[k].npath / std::max(P[k].npix, 1));
            const uint64_t passes = static_cast<uint64_t>((total[k] + lanes - 1) / lanes);
            launches += 1 + passes * (1 + 4 * static_cast<uint64_t>(P[k].max_depth)) + (write_out ? 1 : 0);
        }
        stats->kernel_launches = launches;
    }
    return PT_OK;
}

// The autotuner's choice for a batch class: the persistent kernel's block size
// and blocks per SM, or wavefront mode with its queue capacity (paths).
struct BatchTune { int block, blocks_per_sm, chunk_spp; double ms; int mode; int64_t paths; };
std::mutex g_tune_mu;
std::vector<std::pair<std::string, BatchTune>> g_tune_cache;

std::string tune_key(int device, const pt_batch_item* items, uint32_t n) {
    uint64_t tris = 0, pix = 0, spp = 0;
    for (uint32_t k = 0; k < n; ++k) {
        tris += items[k].scene->host.faces.size();
        pix += static_cast<uint64_t>(item_camera(items[k]).width) * item_camera(items[k]).height;
        spp += static_cast<uint64_t>(items[k].spp);
    }
    auto lg = [](uint64_t v) { int b = 0; while (v > 1) { v >>= 1; ++b; } return b; };
    return std::to_string(device) + ":" + std::to_string(n) + ":" + std::to_string(lg(tris)) + ":" +
           std::to_string(lg(pix)) + ":" + std::to_string(lg(spp / std::max<uint32_t>(n, 1)));
}

}  // namespace

// Renders every item; stats accumulate over the batch.
int render_batch(const pt_batch_item* in, uint32_t n, int out_is_device, pt_batch_config* cfg, pt_render_stats* stats) {
    if (n == 0) return PT_OK;
    const int device = in[0].scene->dev.device;
    for (uint32_t k = 0; k < n; ++k) {
        if (!in[k].scene || !in[k].scene->dev.uploaded) { set_error("batch item " + std::to_string(k) + ": scene not uploaded"); return PT_ERR_STATE; }
        if (in[k].scene->dev.device != device) { set_error("batch items must live on one device"); return PT_ERR_INVALID; }
        if (in[k].spp <= 0 || !in[k].out_rgba) { set_error("batch item " + std::to_string(k) + ": invalid spp or output"); return PT_ERR_INVALID; }
        if (in[k].camera && (in[k].camera->width <= 0 || in[k].camera->height <= 0)) {
            set_error("batch item " + std::to_string(k) + ": camera resolution must be positive");
            return PT_ERR_INVALID;
        }
        if (in[k].guide && guide_state(in[k].guide).device != device) {
            set_error("batch item " + std::to_string(k) + ": guide lives on another device");
            return PT_ERR_INVALID;
        }
    }
    if (int rc = ensure_device(device)) return rc;
    int sms = 0;
    PT_CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    cudaStream_t st;
    PT_CU(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    struct Guard { std::vector<void*> bufs; cudaStream_t st; ~Guard() { for (void* b : bufs) cudaFree(b); cudaStreamDestroy(st); } } g{{}, st};
    auto alloc = [&](size_t bytes) -> void* {
        void* p = nullptr;
        if (cudaMalloc(&p, std::max<size_t>(bytes, 16)) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        g.bufs.push_back(p);
        return p;
    };
    unsigned long long* d_misc = static_cast<unsigned long long*>(alloc(64 * 8));
    if (!d_misc) { set_error("batch: allocation failed"); return PT_ERR_NOMEM; }
    unsigned long long* d_next = d_misc;
    unsigned long long* d_stats = d_misc + 8;
    uint32_t* d_err = reinterpret_cast<uint32_t*>(d_misc + 32);

    int req_mode = cfg ? cfg->mode : PT_BATCH_AUTO;
    if (req_mode != PT_BATCH_AUTO && req_mode != PT_BATCH_PERSISTENT && req_mode != PT_BATCH_WAVEFRONT) {
        set_error("unknown batch mode");
        return PT_ERR_INVALID;
    }
    bool guided = false, textured = false;
    for (uint32_t k = 0; k < n; ++k) {
        guided = guided || in[k].guide != nullptr;
        textured = textured || !in[k].scene->host.textures.empty();
    }
    if (guided || textured) {
        // the persistent kernel traces whole paths per thread with the
        // untextured shading and has no warp-wide network evaluation: guided
        // items and scenes with material textures run in wavefront mode
        if (req_mode == PT_BATCH_PERSISTENT) {
            set_error(guided ? "guided batch items need wavefront mode" : "textured scenes need wavefront mode");
            return PT_ERR_INVALID;
        }
        req_mode = PT_BATCH_WAVEFRONT;
    }
    const int64_t budget = cfg && cfg->paths_in_flight > 0 ? cfg->paths_in_flight : kDefaultPathsInFlight;
    auto run_wavefront = [&](float tuned_ms, int64_t paths) -> int {
        float ms = 0.0f;
        if (int rc = batch_wavefront(in, n, out_is_device, paths, true, st, &ms, stats)) return rc;
        if (cfg) {
            cfg->mode = PT_BATCH_WAVEFRONT;
            cfg->paths_in_flight = static_cast<int32_t>(paths);
            cfg->tuned_ms = tuned_ms;
        }
        return PT_OK;
    };
    if (req_mode == PT_BATCH_WAVEFRONT) return run_wavefront(0.0f, budget);

    // ---- pick the mode and launch shape (autotuner) ----
    // work units of the persistent kernel: chunk_spp samples of an item's
    // pixels (16 unless fixed in cfg; the calibration batch caps every item at
    // 8 spp, so the unit size is not among the timed candidates)
    BatchTune tune{cfg && cfg->block_size ? cfg->block_size : 128,
                   cfg && cfg->blocks_per_sm ? cfg->blocks_per_sm : 0,
                   cfg && cfg->chunk_spp ? cfg->chunk_spp : 16, 0.0, PT_BATCH_PERSISTENT, budget};
    const bool autotune = !cfg || cfg->autotune;
    const std::string key = tune_key(device, in, n) + ":" + std::to_string(req_mode);
    bool cached = false;
    if (autotune) {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        for (auto& kv : g_tune_cache) if (kv.first == key) { tune = kv.second; cached = true; }
    }
    if (autotune && !cached) {
        // time candidate shapes on a calibration batch: every item capped at 8 spp
        std::vector<BatchTune> cands;
        for (int block : {64, 128, 256}) {
            const int mx = max_blocks_per_sm(block);
            for (int bps : {mx, std::max(1, mx / 2)}) cands.push_back({block, bps, 8, 0.0, PT_BATCH_PERSISTENT, budget});
        }
        BatchPlan cal = make_plan(in, n, 8, 8);
        BatchItemDev* d_items = static_cast<BatchItemDev*>(alloc(cal.items.size() * sizeof(BatchItemDev)));
        float4* part = static_cast<float4*>(alloc(cal.partial_floats4 * sizeof(float4)));
        if (!d_items || !part) { set_error("batch: calibration allocation failed"); return PT_ERR_NOMEM; }
        size_t off = 0;
        for (auto& it : cal.items) {
            it.partial = part + off;
            it.out = nullptr;
            off += static_cast<size_t>(it.width) * it.height * it.chunks;
        }
        PT_CU(cudaMemcpyAsync(d_items, cal.items.data(), cal.items.size() * sizeof(BatchItemDev), cudaMemcpyHostToDevice, st));
        cudaEvent_t e0, e1;
        PT_CU(cudaEventCreate(&e0));
        PT_CU(cudaEventCreate(&e1));
        double best = 1e30;
        for (BatchTune& c : cands) {
            for (int rep = 0; rep < 2; ++rep) {
                PT_CU(cudaMemsetAsync(d_next, 0, 8, st));
                PT_CU(cudaEventRecord(e0, st));
                if (int rc = launch_persistent(c.block, c.blocks_per_sm * sms, d_items, static_cast<int>(n),
                                               cal.total_units, d_next, d_stats, d_err, st)) return rc;
                PT_CU(cudaEventRecord(e1, st));
                PT_CU(cudaEventSynchronize(e1));
                float ms = 0.0f;
                PT_CU(cudaEventElapsedTime(&ms, e0, e1));
                c.ms = ms;   // second repetition counts (first is warm-up)
            }
            if (c.ms < best) { best = c.ms; tune = c; tune.chunk_spp = cfg && cfg->chunk_spp ? cfg->chunk_spp : 16; }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        // the wavefront mode on the same calibration batch, at three queue
        // capacities (paths in flight shared by the items) unless fixed in cfg
        if (req_mode == PT_BATCH_AUTO) {
            std::vector<pt_batch_item> capped(in, in + n);
            for (pt_batch_item& it : capped) it.spp = std::min(it.spp, 8);
            std::vector<int64_t> caps;
            if (cfg && cfg->paths_in_flight > 0) caps.push_back(cfg->paths_in_flight);
            else caps = {int64_t(1) << 25, int64_t(1) << 26, int64_t(1) << 27};
            for (int64_t paths : caps) {
                float wms = 0.0f;
                for (int rep = 0; rep < 2; ++rep)
                    if (int rc = batch_wavefront(capped.data(), n, 0, paths, false, st, &wms, nullptr)) return rc;
                if (wms < best) { best = wms; tune.mode = PT_BATCH_WAVEFRONT; tune.ms = wms; tune.paths = paths; }
            }
        }
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune_cache.emplace_back(key, tune);
    }
    if (tune.mode == PT_BATCH_WAVEFRONT && req_mode == PT_BATCH_AUTO)
        return run_wavefront(static_cast<float>(tune.ms), tune.paths);
    if (tune.blocks_per_sm <= 0) tune.blocks_per_sm = max_blocks_per_sm(tune.block);

    // ---- the batch itself: one persistent launch + resolve, captured in a graph ----
    BatchPlan plan = make_plan(in, n, static_cast<uint32_t>(tune.chunk_spp), 0);
    BatchItemDev* d_items = static_cast<BatchItemDev*>(alloc(plan.items.size() * sizeof(BatchItemDev)));
    float4* part = static_cast<float4*>(alloc(plan.partial_floats4 * sizeof(float4)));
    float4* outs = out_is_device ? nullptr : static_cast<float4*>(alloc(plan.out_floats4 * sizeof(float4)));
    if (!d_items || !part || (!out_is_device && !outs)) { set_error("batch: allocation failed (partials)"); return PT_ERR_NOMEM; }
    size_t off = 0, ooff = 0;
    for (uint32_t k = 0; k < n; ++k) {
        BatchItemDev& it = plan.items[k];
        it.partial = part + off;
        off += static_cast<size_t>(it.width) * it.height * it.chunks;
        it.out = out_is_device ? reinterpret_cast<float4*>(in[k].out_rgba) : outs + ooff;
        ooff += static_cast<size_t>(it.width) * it.height;
    }
    PT_CU(cudaMemcpyAsync(d_items, plan.items.data(), plan.items.size() * sizeof(BatchItemDev), cudaMemcpyHostToDevice, st));
    PT_CU(cudaMemsetAsync(d_stats, 0, 24 * 8, st));
    PT_CU(cudaMemsetAsync(d_err, 0, 4, st));
    PT_CU(cudaStreamSynchronize(st));
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    PT_CU(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(d_next, 0, 8, st);
    int rc = launch_persistent(tune.block, tune.blocks_per_sm * sms, d_items, static_cast<int>(n), plan.total_units,
                               d_next, d_stats, d_err, st);
    k_batch_resolve<<<sms * 8, 256, 0, st>>>(d_items, static_cast<int>(n), plan.total_pixels);
    const cudaError_t ec = cudaStreamEndCapture(st, &graph);
    if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
    if (ec != cudaSuccess) { set_error(std::string("batch graph capture: ") + cudaGetErrorString(ec)); return PT_ERR_CUDA; }
    const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) { set_error(std::string("batch graph instantiate: ") + cudaGetErrorString(ei)); return PT_ERR_CUDA; }
    cudaEvent_t e0, e1;
    PT_CU(cudaEventCreate(&e0));
    PT_CU(cudaEventCreate(&e1));
    PT_CU(cudaEventRecord(e0, st));
    const cudaError_t el = cudaGraphLaunch(exec, st);
    PT_CU(cudaEventRecord(e1, st));
    const cudaError_t es = cudaStreamSynchronize(st);
    cudaGraphExecDestroy(exec);
    if (el != cudaSuccess || es != cudaSuccess) {
        set_error(std::string("batch launch: ") + cudaGetErrorString(el != cudaSuccess ? el : es));
        cudaEventDestroy(e0); cudaEventDestroy(e1);
        return PT_ERR_CUDA;
    }
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    uint32_t err = 0;
    PT_CU(cudaMemcpy(&err, d_err, 4, cudaMemcpyDeviceToHost));
    if (err) { set_error("batch: device error word " + std::to_string(err)); return PT_ERR_DEVICE; }
    if (!out_is_device) {
        for (uint32_t k = 0; k < n; ++k) {
            const BatchItemDev& it = plan.items[k];
            PT_CU(cudaMemcpy(in[k].out_rgba, it.out, static_cast<size_t>(it.width) * it.height * sizeof(float4),
                             cudaMemcpyDeviceToHost));
        }
    }
    if (stats) {
        unsigned long long s[kStatCount];
        PT_CU(cudaMemcpy(s, d_stats, sizeof(s), cudaMemcpyDeviceToHost));
        std::memset(stats, 0, sizeof(*stats));
        stats->camera_rays = s[kStatCameraRays];
        stats->extension_rays = s[kStatExtRays];
        stats->shadow_rays = s[kStatShadowRays];
        stats->paths = s[kStatPaths];
        stats->total_ms = ms;
        stats->kernel_launches = 2;
    }
    if (cfg) {
        cfg->block_size = tune.block;
        cfg->blocks_per_sm = tune.blocks_per_sm;
        cfg->chunk_spp = tune.chunk_spp;
        cfg->tuned_ms = static_cast<float>(tune.ms);
        cfg->mode = PT_BATCH_PERSISTENT;
    }
    return PT_OK;
}

// Drops the cached wavefront slot of a scene that is being destroyed.
void batch_forget_scene(const pt_scene* s) {
    std::lock_guard<std::mutex> lk(g_slot_mu);
    for (size_t i = 0; i < g_slots.size();) {
        if (g_slots[i]->scene != s) { ++i; continue; }
        slot_release(*g_slots[i]);
        g_slots.erase(g_slots.begin() + static_cast<long>(i));
    }
}

}  // namespace ptb
