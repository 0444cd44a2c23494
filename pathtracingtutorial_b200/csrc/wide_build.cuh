// wide_build.cuh -- collapses the binary tree into the four-wide one on the
// device (included by integrator.cu; layout and argument in wide.h).
//
// A wide node starts as one binary inner node's two children; while it has
// fewer than four, its inner child of the largest surface area is replaced by
// that child's own two.  The wide nodes keep the depth-first order of their
// binary nodes.  One cooperative launch walks the levels from the root, a scan
// numbers the nodes, one launch writes them and one the triangle records:
// bound by launches and, on large scenes, HBM (64 B read per binary node, 64 B
// written per wide node and triangle).

#include <cooperative_groups.h>

namespace ptb {

// Slot of a binary node: node << 1 | side; kWideRoot: the root itself.
constexpr uint32_t kWideRoot = 0xffffffffu;

struct WideStatus { uint32_t tail, bad, need, pad; };

// Scratch of one collapse, per binary inner node.
struct WideScratch {
    uint4*    slots;    // children of the wide node that starts here (slots of binary nodes)
    uint2*    order;
    uint32_t* queue;    // slots whose subtree starts a wide node, in level order
    uint32_t* mark;     // 0, or the number of children
    uint32_t* before;   // deferred entries a walk can hold when it arrives here
    uint32_t* index;    // exclusive sums of (mark != 0)
    WideStatus* status;
};
constexpr size_t kWideScratchPerNode = 16 + 8 + 4 * 4;

struct Box6 { float lo[3], hi[3]; };

__device__ __forceinline__ uint32_t slot_ref(const InnerNode& n, uint32_t side) { return side ? n.ref1 : n.ref0; }
__device__ __forceinline__ Box6 slot_box(const InnerNode& n, uint32_t side) {
    Box6 b;
    if (side == 0) {
        b.lo[0] = n.c0lo[0]; b.lo[1] = n.c0lo[1]; b.lo[2] = n.c0lo[2];
        b.hi[0] = n.c0hi_x; b.hi[1] = n.c0hi_yz[0]; b.hi[2] = n.c0hi_yz[1];
    } else {
        b.lo[0] = n.c1lo_xy[0]; b.lo[1] = n.c1lo_xy[1]; b.lo[2] = n.c1lo_z;
        b.hi[0] = n.c1hi[0]; b.hi[1] = n.c1hi[1]; b.hi[2] = n.c1hi[2];
    }
    return b;
}
__device__ __forceinline__ float box_area(const Box6& b) {
    const float x = b.hi[0] - b.lo[0], y = b.hi[1] - b.lo[1], z = b.hi[2] - b.lo[2];
    return x * y + y * z + z * x;
}
// Usable as a child of `own`: finite, ordered and inside it.
__device__ __forceinline__ bool box_sound(const Box6& b, const Box6& own) {
    bool ok = true;
    for (int a = 0; a < 3; ++a)
        ok = ok && fabsf(b.lo[a]) <= 1e30f && fabsf(b.hi[a]) <= 1e30f && b.lo[a] <= b.hi[a] && b.lo[a] >= own.lo[a] &&
             b.hi[a] <= own.hi[a];
    return ok;
}

// The collapse.  Cooperative: the grid meets between levels.
__global__ void __launch_bounds__(128, 4) k_wide_collapse(const InnerNode* __restrict__ inner, uint32_t ni, Box6 root,
                                                       WideScratch sc) {
    const cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t i = tid; i < ni; i += stride) sc.mark[i] = 0u;
    if (tid == 0) {
        sc.queue[0] = kWideRoot;
        sc.before[0] = 0u;
        *sc.status = WideStatus{1u, 0u, 0u, 0u};
    }
    grid.sync();
    uint32_t begin = 0, end = 1;
    for (int level = 0; begin < end && level < 128; ++level) {
        for (uint32_t q = begin + tid; q < end; q += stride) {
            const uint32_t code = sc.queue[q];
            const uint32_t node = code == kWideRoot ? 0u : slot_ref(inner[code >> 1], code & 1u);
            const Box6 own = code == kWideRoot ? root : slot_box(inner[code >> 1], code & 1u);
            uint32_t slot[4] = {node << 1, (node << 1) | 1u, 0u, 0u};
            float area[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // of inner children; 0 for leaves
            uint32_t list[4];                           // per octant: the slots in visiting order, nibbles
            bool ok = true;
            auto look = [&](int k) {
                const InnerNode& n = inner[slot[k] >> 1];
                area[k] = (slot_ref(n, slot[k] & 1u) & kLeafBit) ? 0.0f
                                                                 : fmaxf(box_area(slot_box(n, slot[k] & 1u)), FLT_MIN);
            };
            auto right_first = [&](const InnerNode& n, uint32_t octant) {
                return ((octant >> (n.meta & 3u)) & 1u) == ((n.meta >> 2) & 1u);
            };
            {
                const InnerNode& n = inner[node];
                ok = box_sound(slot_box(n, 0), own) && box_sound(slot_box(n, 1), own);
                for (uint32_t o = 0; o < 4; ++o) list[o] = right_first(n, o) ? 0x01u : 0x10u;
                look(0);
                look(1);
            }
            int cnt = 2;
            while (cnt < 4) {
                int k = 0;
                for (int c = 1; c < cnt; ++c) if (area[c] > area[k]) k = c;
                if (area[k] <= 0.0f) break;
                const InnerNode& up = inner[slot[k] >> 1];
                const Box6 ub = slot_box(up, slot[k] & 1u);
                const uint32_t child = slot_ref(up, slot[k] & 1u);
                const InnerNode& n = inner[child];
                ok = ok && box_sound(slot_box(n, 0), ub) && box_sound(slot_box(n, 1), ub);
                for (uint32_t o = 0; o < 4; ++o) {
                    // entry k becomes the pair (k, cnt) in the order of its node
                    uint32_t out = 0;
                    int w = 0;
                    for (int p = 0; p < cnt; ++p) {
                        const uint32_t e = (list[o] >> (4 * p)) & 15u;
                        if (static_cast<int>(e) == k) {
                            const bool rf = right_first(n, o);
                            out |= (rf ? static_cast<uint32_t>(cnt) : e) << (4 * w++);
                            out |= (rf ? e : static_cast<uint32_t>(cnt)) << (4 * w++);
                        } else {
                            out |= e << (4 * w++);
                        }
                    }
                    list[o] = out;
                }
                slot[k] = child << 1;
                slot[cnt] = (child << 1) | 1u;
                look(k);
                look(cnt);
                ++cnt;
            }
            uint32_t after[4];
            for (uint32_t o = 0; o < 4; ++o) {
                uint32_t a = 0, later = 0;
                for (int p = cnt - 1; p >= 0; --p) {
                    const uint32_t e = (list[o] >> (4 * p)) & 15u;
                    a |= later << (4 * e);
                    later |= 1u << e;
                }
                after[o] = a;
            }
            sc.slots[node] = make_uint4(slot[0], slot[1], slot[2], slot[3]);
            sc.order[node] = make_uint2(after[0] | (after[1] << 16), after[2] | (after[3] << 16));
            sc.mark[node] = static_cast<uint32_t>(cnt);
            const uint32_t before = sc.before[node];
            atomicMax(&sc.status->need, before + 3u);
            if (!ok) sc.status->bad = 1u;
            for (int c = 0; c < cnt; ++c) {
                const uint32_t r = slot_ref(inner[slot[c] >> 1], slot[c] & 1u);
                if (r & kLeafBit) continue;
                sc.before[r] = before + static_cast<uint32_t>(cnt) - 1u;
                const uint32_t at = atomicAdd(&sc.status->tail, 1u);
                if (at < ni) sc.queue[at] = slot[c];
            }
        }
        grid.sync();
        begin = end;
        end = min(*reinterpret_cast<volatile uint32_t*>(&sc.status->tail), ni);
        grid.sync();
    }
    for (uint32_t i = tid; i < ni; i += stride) sc.index[i] = sc.mark[i] ? 1u : 0u;
}

__global__ void __launch_bounds__(128) k_wide_emit(const InnerNode* __restrict__ inner, uint32_t ni, WideScratch sc,
                                                   WideNode* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ni; i += gridDim.x * blockDim.x) {
        const uint32_t cnt = sc.mark[i];
        if (cnt == 0u) continue;
        const uint4 s4 = sc.slots[i];
        const uint32_t slot[4] = {s4.x, s4.y, s4.z, s4.w};
        Box6 b[4];
        WideNode w;
        for (uint32_t c = 0; c < 4; ++c) {
            w.ref[c] = kNoRef;
            if (c >= cnt) continue;
            const InnerNode& n = inner[slot[c] >> 1];
            b[c] = slot_box(n, slot[c] & 1u);
            const uint32_t r = slot_ref(n, slot[c] & 1u);
            w.ref[c] = (r & kLeafBit) ? r : sc.index[r];
        }
        w.exps = ((1u << cnt) - 1u) << 24;
        for (int a = 0; a < 3; ++a) {
            float mn = b[0].lo[a], mx = b[0].hi[a];
            for (uint32_t c = 1; c < cnt; ++c) { mn = fminf(mn, b[c].lo[a]); mx = fmaxf(mx, b[c].hi[a]); }
            uint32_t e = 0;
            if (!wide_frame(mn, mx, w.base[a], e)) sc.status->bad = 1u;
            const float s = wide_scale(e);
            w.exps |= e << (8 * a);
            w.qlo[a] = w.qhi[a] = 0u;
            for (uint32_t c = 0; c < cnt; ++c) {
                w.qlo[a] |= wide_code_lo(b[c].lo[a], w.base[a], s) << (8 * c);
                w.qhi[a] |= wide_code_hi(b[c].hi[a], w.base[a], s) << (8 * c);
            }
        }
        const uint2 o = sc.order[i];
        w.order[0] = o.x;
        w.order[1] = o.y;
        out[sc.index[i]] = w;
    }
}

// Triangle records with their leaf's box, leaf by leaf (ni = 0: one leaf, the
// root box).
__global__ void __launch_bounds__(128) k_wide_tris(const InnerNode* __restrict__ inner, uint32_t ni, Box6 root,
                                                   const TriRecord* __restrict__ tris, uint32_t n,
                                                   WideTri* __restrict__ out) {
    auto leaf = [&](uint32_t first, const Box6& b) {
        for (uint32_t t = first; t < n; ++t) {
            const TriRecord r = tris[t];
            WideTri w;
            w.v0[0] = r.v0[0]; w.v0[1] = r.v0[1]; w.v0[2] = r.v0[2];
            w.e1[0] = r.e1x; w.e1[1] = r.e1yz[0]; w.e1[2] = r.e1yz[1];
            w.e2xy[0] = r.e2xy[0]; w.e2xy[1] = r.e2xy[1];
            w.e2z = r.e2z;
            w.flags = r.flags;
            for (int a = 0; a < 3; ++a) { w.lo[a] = b.lo[a]; w.hi[a] = b.hi[a]; }
            out[t] = w;
            if (r.flags & 1u) break;
        }
    };
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (ni == 0u && tid == 0u) leaf(0u, root);
    for (uint32_t i = tid; i < 2u * ni; i += gridDim.x * blockDim.x) {
        const InnerNode& nd = inner[i >> 1];
        const uint32_t r = slot_ref(nd, i & 1u);
        if (r & kLeafBit) leaf(r & ~kLeafBit, slot_box(nd, i & 1u));
    }
}

// Builds the wide tree of a scene from its binary tree on the device, once per
// upload of new arrays: nothing reads d.wide and d.wtris yet.  Scratch lives
// where the triangle records go afterwards.
static int build_wide(const SceneTables& t, uint32_t n_faces, DeviceSceneBuffers& d) {
    d.wide_on = false;
    d.wide_need = 0;
    const uint32_t ni = static_cast<uint32_t>(t.inner.size());
    if (n_faces == 0) return PT_OK;
    Box6 root;
    bool finite = true;
    for (int a = 0; a < 3; ++a) {
        root.lo[a] = t.root_lo[a];
        root.hi[a] = t.root_hi[a];
        finite = finite && std::fabs(root.lo[a]) <= 1e30f && std::fabs(root.hi[a]) <= 1e30f && root.lo[a] <= root.hi[a];
        // (at least 2^-80: see the pads in wide.h)
        d.coord_max[a] = std::max(std::max(std::fabs(root.lo[a]), std::fabs(root.hi[a])), 8.2718061e-25f);
    }
    if (!finite) return PT_OK;
    size_t scan_tmp = 0;
    PT_CU(cub::DeviceScan::ExclusiveSum(nullptr, scan_tmp, static_cast<uint32_t*>(nullptr),
                                        static_cast<uint32_t*>(nullptr), static_cast<int>(std::max(ni, 1u))));
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t scratch = up(ni * size_t(16)) + up(ni * size_t(8)) + 4 * up(ni * size_t(4)) + 256 + up(scan_tmp);
    const size_t want_tris = std::max(size_t(n_faces) * sizeof(WideTri), scratch);
    // a node with fewer than four children has only leaves below it, so there
    // are at most 2/3 as many wide nodes as binary ones (and one)
    const size_t want_nodes = (size_t(ni) * 2 / 3 + 2) * sizeof(WideNode);
    // without room for both the scene keeps the binary walk
    if (cudaMalloc(&d.wide, want_nodes) != cudaSuccess || cudaMalloc(&d.wtris, want_tris) != cudaSuccess) {
        cudaGetLastError();
        if (d.wide) cudaFree(d.wide);
        d.wide = d.wtris = nullptr;
        return PT_OK;
    }
    d.wide_bytes = want_nodes;
    d.wtris_bytes = want_tris;
    const InnerNode* inner = static_cast<const InnerNode*>(d.inner);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d.device);
    WideStatus st{0, 0, 0, 0};
    if (ni > 0) {
        char* cur = static_cast<char*>(d.wtris);
        auto take = [&](size_t bytes) { char* p = cur; cur += up(bytes); return p; };
        WideScratch sc;
        sc.slots = reinterpret_cast<uint4*>(take(ni * size_t(16)));
        sc.order = reinterpret_cast<uint2*>(take(ni * size_t(8)));
        sc.queue = reinterpret_cast<uint32_t*>(take(ni * size_t(4)));
        sc.mark = reinterpret_cast<uint32_t*>(take(ni * size_t(4)));
        sc.before = reinterpret_cast<uint32_t*>(take(ni * size_t(4)));
        sc.index = reinterpret_cast<uint32_t*>(take(ni * size_t(4)));
        sc.status = reinterpret_cast<WideStatus*>(take(sizeof(WideStatus)));
        void* tmp = take(scan_tmp);
        uint32_t nn = ni;
        const int grid = static_cast<int>(std::min<uint32_t>((ni + 127) / 128, static_cast<uint32_t>(sms) * 4u));
        void* args[] = {&inner, &nn, &root, &sc};
        PT_CU(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_wide_collapse), dim3(grid), dim3(128), args, 0,
                                          nullptr));
        PT_CU(cub::DeviceScan::ExclusiveSum(tmp, scan_tmp, sc.index, sc.index, static_cast<int>(ni)));
        const int wide_grid = static_cast<int>(std::min<uint32_t>((ni + 127) / 128, static_cast<uint32_t>(sms) * 16u));
        k_wide_emit<<<wide_grid, 128>>>(inner, ni, sc, static_cast<WideNode*>(d.wide));
        PT_CU(cudaMemcpyAsync(&st, sc.status, sizeof(st), cudaMemcpyDeviceToHost));   // (the records go over it)
    }
    k_wide_tris<<<static_cast<int>(std::min<uint32_t>((2 * ni + 128) / 128, static_cast<uint32_t>(sms) * 16u)), 128>>>(
        inner, ni, root, static_cast<const TriRecord*>(d.tris), n_faces, static_cast<WideTri*>(d.wtris));
    PT_CU(cudaGetLastError());
    PT_CU(cudaStreamSynchronize(nullptr));
    d.wide_on = st.bad == 0;
    d.wide_need = st.need;
    d.wide_root = ni > 0 ? 0u : (kLeafBit | 0u);
    return PT_OK;
}

}  // namespace ptb
