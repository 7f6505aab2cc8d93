// lbmx_pair_kernels.cuh -- two steps of the fused D2Q9 step in one pass over
// memory, instantiated once per storage type by lbmx_pair_{f32,f16,bf16}.cu.
//
// A neighbour-access step (parity 1) followed by an own-node step (parity 0)
// maps the populations of one own-node layout to the next: every node's nine
// slots after the pair depend on the slots within two nodes of it before.
// Each work item is a tile of W x H nodes (pair_w, pair_h): the producer warp brings
// the tile's slots and two nodes around it into shared memory by TMA, the
// consumers run the first step there on the tile and one node around it --
// in place, since a node reads and writes the same slots (the AA pattern) --
// and the second step on the tile, whose results go to the lattice's second
// population buffer.  Nothing a tile reads is written in the same launch, so
// tiles need no order.
//
// The arithmetic of a node is the single-step kernel's (unit_collide,
// node_collide), and so are the random bits of 16-bit stores, so a pair gives
// what two single steps give.  Nodes computed by two tiles (the ring around
// each) come out alike in both.
//
// Single steps of a large FP32 lattice are bound by HBM (72 bytes a node and
// step, issue slots a third busy); a pair moves the same bytes for two steps
// and is bound by issue and latency instead: MRT cavity 8192^2 740 -> 397 us
// a step (90.7 -> 169 GLUPS), 1024^2, in L2, 12.1 -> 8.4 us, 256^2 vortex 4.3
// -> 2.6 us (half the launches), FP16 8192^2 414 -> 391 us (issue-bound both
// ways).  Tile shapes and their choice: pair_shape in lbmx_internal.h.
#pragma once
#include <algorithm>

#include "lbmx_kernels.cuh"

namespace lbmx {

template <typename T, int SHAPE>
struct PairStaging {
    using Elem = T;
    static constexpr int W = pair_w(SHAPE), H = pair_h(SHAPE, (int)sizeof(T));
    static constexpr int A = 16 / (int)sizeof(T);  // elements per 16-byte chunk
    static constexpr int BW = W + 2 * A;           // box: the tile, two nodes (one chunk) each side
    static constexpr int BH = H + 2;               //   and the row above and below, shifted by the plane's c_y
    static constexpr int NST = kPairStages;
    static constexpr int BOX_ELEMS = BW * BH;
    static constexpr int SLAB = (int)(((BOX_ELEMS * sizeof(T) + 127) / 128) * 128 / sizeof(T));
    static constexpr int STAGE_ELEMS = 9 * SLAB;
    static constexpr unsigned STAGE_BYTES = (unsigned)(9 * BOX_ELEMS * sizeof(T));
    static constexpr size_t BUF_BYTES = (size_t)NST * STAGE_ELEMS * sizeof(T);
    // after the buffers: ready, full, mid, empty [NST] mbarriers, one work slot per stage
    static constexpr size_t SMEM = BUF_BYTES + 4 * NST * sizeof(uint64_t) + NST * 2 * sizeof(int4);
};

// Slot of plane p at node (x0 + dx + c_x, y0 + dy + c_y), c the plane's
// velocity, is element pair_at(p, dx, dy): the nine slots that node (dx, dy)
// of the tile reads and writes in the first step sit at one place of the nine
// slabs, but for the x shift.
template <typename St>
__device__ __forceinline__ constexpr int pair_at(int p, int dx, int dy) {
    return p * St::SLAB + (dy + 1) * St::BW + dx + St::A + CX(p);
}
// slot of plane p at the node (dx, dy) itself
template <typename St>
__device__ __forceinline__ constexpr int pair_own(int p, int dx, int dy) {
    return pair_at<St>(p, dx - CX(p), dy - CY(p));
}

// The sums of a kModeSums pair, exact in the same fixed point as everywhere
// (fix): a thread's terms of each step stay in 32 bits -- each below one half
// of 2^30, a unit's mass less the 2 it has at rest -- and a warp adds its
// total to its own 64-bit accumulators in shared memory when one of its
// threads' sums passes kUnitSumLimit at the end of a tile (at most three
// units more fit then), and at the end, the rest mass by the count of units.  Terms out of that range go to the
// warp's accumulators by themselves.  (64-bit accumulators of both steps in
// every thread cost 12 registers and twice the instructions; a warp's total
// after every tile and step: 1024^2 FP32 with sums 10.2 us a step, 9.9 now,
// lean 8.4.)
constexpr int kUnitSumLimit = 1 << 29;
struct UnitSums {
    int m = 0, x = 0, y = 0, units = 0;
};
// 64-bit terms of a whole warp (general-path nodes; any: the tile has some)
__device__ __forceinline__ void node_sums_add(const Acc t[3], bool any, unsigned long long* acc) {
    if (!any) return;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        Acc v = t[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) acc[k] += (unsigned long long)v;
    }
    __syncwarp();
}
__device__ __forceinline__ void unit_sums_count(UnitSums& u, unsigned long long* acc, float m, float jx, float jy) {
    const float dm = m - 2.0f;  // exact for m in [1, 4]
    if (fabsf(dm) < 0.5f && fabsf(jx) < 0.5f && fabsf(jy) < 0.5f) {
        u.m += __float2int_rn(__fmul_rn(dm, kFixScale));
        u.x += __float2int_rn(__fmul_rn(jx, kFixScale));
        u.y += __float2int_rn(__fmul_rn(jy, kFixScale));
        u.units++;
    } else {
        atomicAdd(acc, (unsigned long long)fix(m));
        atomicAdd(acc + 1, (unsigned long long)fix(jx));
        atomicAdd(acc + 2, (unsigned long long)fix(jy));
    }
}
__device__ __forceinline__ bool unit_sums_large(const UnitSums& u) {
    return abs(u.m) > kUnitSumLimit || abs(u.x) > kUnitSumLimit || abs(u.y) > kUnitSumLimit;
}
// every lane of a consumer warp; lane k adds the warp's total of sum k
__device__ __forceinline__ void unit_sums_add(UnitSums& u, unsigned long long* acc) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    // in halves: a warp's sum of 32-bit terms may need more than 32
    const int mh = __reduce_add_sync(0xffffffffu, u.m >> 16), ml = __reduce_add_sync(0xffffffffu, u.m & 0xFFFF);
    const int xh = __reduce_add_sync(0xffffffffu, u.x >> 16), xl = __reduce_add_sync(0xffffffffu, u.x & 0xFFFF);
    const int yh = __reduce_add_sync(0xffffffffu, u.y >> 16), yl = __reduce_add_sync(0xffffffffu, u.y & 0xFFFF);
    // the units' rest mass, 2 * 2^30 each, in 64 bits: near rest nothing calls
    // for a warp's total before the end of the launch, and a warp of a large
    // lattice has more than 2^16 units by then
    const int units = __reduce_add_sync(0xffffffffu, u.units);
    const int hi = lane == 0 ? mh : lane == 1 ? xh : yh, lo = lane == 0 ? ml : lane == 1 ? xl : yl;
    if (lane < 3)
        acc[lane] += (unsigned long long)(((Acc)hi << 16) + (Acc)lo + (lane == 0 ? (Acc)units << 31 : 0));
    __syncwarp();
    u = UnitSums();
}

// First step of two x-neighbouring interior nodes, in shared memory.
template <typename St, int OP, int MODE>
__device__ __forceinline__ void pair_unit_first(const StepArgs& a, typename St::Elem* sb, int dx, int dy, int x, int y,
                                                Acc v[kNumSums], bool own, UnitSums& us, unsigned long long* tsums) {
    using T = typename St::Elem;
    V2 f[9];
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const T* s = sb + pair_at<St>(OPP(q), dx, dy);
        f[q].v = CX(q) != 0 ? Store<T>::ld2r_u(s) : Store<T>::ld2r(s);
    }
    const long long off = (long long)y * a.g.pitch + x;
    V2 mom[5];
    unit_collide<T, OP, MODE, true>(a, off, f, v, own, nullptr, mom);
    if (MODE == kModeSums && own && a.partials)
        unit_sums_count(us, tsums, mom[0].v.x + mom[0].v.y, mom[1].v.x + mom[1].v.y, mom[2].v.x + mom[2].v.y);
    if (kOffset<T> && a.sr) {
        const uint32_t h = sr_hash(((uint32_t)off >> 1) + a.sr_unit_origin, a.sr_seed);
#pragma unroll
        for (int q = 0; q < 9; q++) {
            T* p = sb + pair_at<St>(q, dx, dy);
            const uint32_t r = sr_bits(h, q);
            if (CX(q) == 0) Store<T>::st2r_sr(p, f[q].v, r);
            else Store<T>::st2r_sr_u(p, f[q].v, r);
        }
    } else {
#pragma unroll
        for (int q = 0; q < 9; q++) {
            T* p = sb + pair_at<St>(q, dx, dy);
            if (CX(q) == 0) Store<T>::st2r(p, f[q].v);
            else Store<T>::st2r_u(p, f[q].v);
        }
    }
}

// Second step of two x-neighbouring nodes, from shared memory to b.f.
template <typename St, int OP, int MODE>
__device__ __forceinline__ void pair_unit_second(const StepArgs& b, const typename St::Elem* sb, int dx, int dy, int x, int y,
                                                 Acc v[kNumSums], UnitSums& us, unsigned long long* tsums) {
    using T = typename St::Elem;
    V2 f[9];
#pragma unroll
    for (int q = 0; q < 9; q++) f[q].v = Store<T>::ld2r(sb + pair_own<St>(q, dx, dy));
    const long long off = (long long)y * b.g.pitch + x;
    V2 mom[5];
    unit_collide<T, OP, MODE, true>(b, off, f, v, true, nullptr, mom);
    if (MODE == kModeSums) {
        unit_sums_count(us, tsums, mom[0].v.x + mom[0].v.y, mom[1].v.x + mom[1].v.y, mom[2].v.x + mom[2].v.y);
        if (b.rho_out) {
            *reinterpret_cast<float2*>(b.rho_out + off) = mom[0].v;
            *reinterpret_cast<float2*>(b.u_out + off) = mom[3].v;
            *reinterpret_cast<float2*>(b.u_out + b.g.plane + off) = mom[4].v;
        }
    }
    // plane bases are the same for every thread; a plane's bytes fit 32 bits
    // (checked where pairs are enabled), so an address is one register
    const uint32_t o = (uint32_t)(y * b.g.pitch + x) * (uint32_t)sizeof(T);
    char* base = static_cast<char*>(b.f);
    if (kOffset<T> && b.sr) {
        const uint32_t h = sr_hash(((uint32_t)off >> 1) + b.sr_unit_origin, b.sr_seed);
#pragma unroll
        for (int q = 0; q < 9; q++)
            Store<T>::st2r_sr(reinterpret_cast<T*>(base + b.st_off[q] + o), f[q].v, sr_bits(h, q));
    } else {
#pragma unroll
        for (int q = 0; q < 9; q++) Store<T>::st2r(reinterpret_cast<T*>(base + b.st_off[q] + o), f[q].v);
    }
}

// The results of one node of the first step's general path into the tile's
// slots; `own`: the tile's own node, which also updates the edge store.
template <typename St>
__device__ __forceinline__ void pair_put_first(const StepArgs& a, float* edge_out, typename St::Elem* sb, int dx, int dy,
                                               int x, int y, const float f[9], unsigned outmask, uint8_t fl, bool own) {
    using T = typename St::Elem;
    const Geometry& g = a.g;
    const uint32_t off = (uint32_t)(y * g.pitch + x);
    const bool hw = is_halfway(fl);
    const bool sr = kOffset<T> && a.sr;
    const uint32_t h = sr ? sr_hash((off >> 1) + a.sr_unit_origin, a.sr_seed) : 0u;
    const int lane = (int)(off & 1);
    auto put = [&](T* p, float val, int q) {
        if (sr) Store<T>::st_sr(p, val, WQ(q), sr_lane16(sr_bits(h, q), lane));
        else Store<T>::st(p, val, WQ(q));
    };
    put(sb + pair_at<St>(0, dx, dy), f[0], 0);
#pragma unroll
    for (int q = 1; q < 9; q++) {
        const int tx = x + CX(q), ty = y + CY(q);
        const bool out = (CX(q) != 0 && !g.periodic_x && (tx < 0 || tx >= g.nx)) ||
                         (CY(q) != 0 && !g.periodic_y && (ty < 0 || ty >= g.ny));
        if (!out) put(sb + pair_at<St>(q, dx, dy), f[q], q);
        else if (hw && own) put(sb + pair_own<St>(OPP(q), dx, dy), f[q] - wall_term(a, q, fl), q);
    }
    if (outmask && !hw && own) {
        float* E = edge_out + ((long long)g.perimeter + edge_index(x, y, g.nx, g.ny)) * 9;
#pragma unroll
        for (int q = 1; q < 9; q++)
            if (outmask & (1u << q)) E[q] = f[q];
    }
}

// Second step of one of the tile's nodes through the general path: its own
// slots from shared memory, the edge store's old values from edge_in; b.edge
// is the new edge store.
template <typename St, int OP>
__device__ __forceinline__ void pair_node_second(const StepArgs& b, const float* edge_in, const typename St::Elem* sb, int dx,
                                                 int dy, int x, int y, uint8_t fl, Acc v[kNumSums]) {
    using T = typename St::Elem;
    const Geometry& g = b.g;
    const long long off = (long long)y * g.pitch + x;
    const bool hw = is_halfway(fl);
    const float* E = edge_in + (long long)(on_edge(g, x, y) ? edge_index(x, y, g.nx, g.ny) : 0) * 9;
    unsigned m = 0;
    float f[9];
    f[0] = Store<T>::ld(sb + pair_own<St>(0, dx, dy), WQ(0));
#pragma unroll
    for (int q = 1; q < 9; q++) {
        const int sx = x - CX(q), sy = y - CY(q);
        const bool out = (CX(q) != 0 && !g.periodic_x && (sx < 0 || sx >= g.nx)) ||
                         (CY(q) != 0 && !g.periodic_y && (sy < 0 || sy >= g.ny));
        if (out) m |= 1u << q;
        f[q] = out && !hw ? E[q] : Store<T>::ld(sb + pair_own<St>(q, dx, dy), WQ(q));
    }
    if (fl) apply_bc(b, f, x, y, fl);
    node_collide<OP>(b, off, f, v, true);
    store_post_collision<T>(b, x, y, f, m, fl, b.sr_seed);
}

// The grid sums of both steps of a kModeFull pair; the last CTA publishes.
__device__ __forceinline__ void pair_block_sums(const PairArgs& p, const Acc v1[kNumSums], const Acc v2[kNumSums]) {
    __shared__ bool is_last;
    const int tid = threadIdx.x;
    const unsigned mask1 = sums_mask(p.a.ke != 0, false), mask2 = sums_mask(p.b.ke != 0, false);
    if (p.a.partials) warp_sums(p.a.partials, v1, mask1);
    if (p.b.partials) warp_sums(p.b.partials, v2, mask2);
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        is_last = atomicAdd(p.b.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last || tid >= 32) return;
    __threadfence();
    double s[kNumSums];
    if (p.a.partials) {
        collect_sums(p.a.partials, mask1, s, nullptr, tid);
        if (tid == 0) write_sums(s, p.a.sums, p.a.series, p.a.ke != 0);
    }
    if (p.b.partials) {
        collect_sums(p.b.partials, mask2, s, nullptr, tid);
        if (tid == 0) write_sums(s, p.b.sums, p.b.series, p.b.ke != 0);
    }
    if (tid == 0) {
        *p.b.counter = 0u;
        __threadfence();
    }
}

// Persistent CTAs, warp-specialised as the single-step kernel's: one producer
// warp claims tiles (those with general-path nodes first) and fills the ring,
// eight consumer warps run the two steps.  ready[s]: the stage's slot is
// written; full[s]: its bytes have landed; mid[s]: all consumer warps are done
// with the first step; empty[s]: with the second.  Every wait is bounded, and
// a warp gives up as a whole.
template <typename T, int OP, int MODE, int SHAPE>
__global__ void __launch_bounds__(kStepThreads, pair_ctas(SHAPE, (int)sizeof(T), MODE))
    pair_kernel(const __grid_constant__ PairArgs p, const __grid_constant__ CUtensorMap tmap) {
    using St = PairStaging<T, SHAPE>;
    constexpr int W = St::W, H = St::H;
    Acc v1[kNumSums] = {0, 0, 0, 0, 0, 0}, v2[kNumSums] = {0, 0, 0, 0, 0, 0};
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* bufs = reinterpret_cast<T*>(smem_raw);
    uint64_t* ready = reinterpret_cast<uint64_t*>(smem_raw + St::BUF_BYTES);
    uint64_t* full = ready + St::NST;
    uint64_t* mid = full + St::NST;
    uint64_t* empty = mid + St::NST;
    int4* slot = reinterpret_cast<int4*>(empty + St::NST);
    // kModeSums: each consumer warp's totals of mass and momentum, first and
    // second step
    __shared__ unsigned long long tsums_buf[kConsumerWarps * 6];
    unsigned long long* tsums = MODE == kModeSums ? tsums_buf + 6 * (warp % kConsumerWarps) : nullptr;
    if (MODE == kModeSums && tid < 6 * kConsumerWarps) tsums_buf[tid] = 0ull;
    if (tid == 0) {
        for (int s = 0; s < St::NST; s++) {
            mbar_init(&ready[s], 1);
            mbar_init(&full[s], 1);
            mbar_init(&mid[s], kConsumerWarps);
            mbar_init(&empty[s], kConsumerWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // The previous step's grid may still be draining (programmatic dependent
    // launch): the first tile's place in the lists, which no step writes, is
    // looked up before the wait, everything else after it.
    const StepArgs& a = p.a;
    const StepArgs& b = p.b;
    const Geometry& g = a.g;
    if (warp == kConsumerWarps) {
        if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
        int k = 0;
        bool failed = false;
        for (;; k++) {
            const int s = k % St::NST;
            if (k >= St::NST && !mbar_wait(&empty[s], (unsigned)(((k / St::NST) - 1) & 1), kWaitLimit)) {
                if (lane == 0) atomicOr(a.error_word, 2u);
                failed = true;
                break;
            }
            // a CTA's first tile is its own (there are no more CTAs than
            // tiles), the counter hands out the rest
            int item = (int)blockIdx.x;
            if (k > 0) {
                if (lane == 0) item = (int)gridDim.x + (int)atomicAdd(p.counter, 1ull);
                item = __shfl_sync(0xffffffffu, item, 0);
            }
            int4* sl = slot + 2 * s;
            if (item >= p.ntiles) {
                if (lane == 0) {
                    put_slot(sl, -1, 0, 0, 0);
                    mbar_arrive(&ready[s]);
                }
                break;
            }
            const int tile =
                __ldg(p.order + (p.reverse && item >= p.nfirst ? p.nfirst + p.ntiles - 1 - item : item));
            const int ty = tile / p.tiles_x, tx = tile - ty * p.tiles_x;
            const int x0 = tx * W, y0 = ty * H;
            const auto publish_slot = [&]() {
                if (lane != 0) return;
                const int b1 = __ldg(p.sp1_at + tile), e1 = __ldg(p.sp1_at + tile + 1);
                const int b0 = __ldg(p.sp0_at + tile), e0 = __ldg(p.sp0_at + tile + 1);
                // a tile with no general-path node whose ring lies off the
                // domain's edge needs no test per unit
                const bool clean = b1 == e1 && x0 > 0 && y0 > 1 && x0 + W + 2 < g.nx && y0 + H < g.ny - 1;
                put_slot(sl, clean ? 1 : 0, x0, y0, 0);
                put_slot(sl + 1, b1, e1, b0, e0);
                mbar_arrive(&ready[s]);
            };
            // before the wait for the first tile, behind the fill for the others
            if (k == 0) {
                publish_slot();
                asm volatile("griddepcontrol.wait;" ::: "memory");
                asm volatile("griddepcontrol.launch_dependents;" :::);
                // the work counters of the launches that may come next
                if (lane == 0 && blockIdx.x == 0) {
                    *p.counter_next = 0ull;
                    p.step_counters[0] = 0ull;
                    p.step_counters[1] = 0ull;
                }
            }
            if (lane == 0) {
                fence_proxy_async_smem();
                mbar_expect_tx(&full[s], St::STAGE_BYTES);
            }
            __syncwarp();
            if (lane < 9) {
                int cy;
                switch (lane) {
                case 2: case 5: case 6: cy = 1; break;
                case 4: case 7: case 8: cy = -1; break;
                default: cy = 0;
                }
                tma_load_3d(bufs + (size_t)s * St::STAGE_ELEMS + (size_t)lane * St::SLAB, &tmap, x0 - St::A,
                            y0 - 1 + cy, lane, &full[s]);
            }
            if (k > 0) publish_slot();
            // the last launch's sums, if it left them (after the first fill
            // is under way)
            if (k == 0 && blockIdx.x == 0) {
                if (a.pub_acc) publish_sums(a.pub_acc, a.pub_sums, a.pub_series, lane);
                if (p.pub_acc2) publish_sums(p.pub_acc2, a.pub_sums, p.pub_series2, lane);
            }
        }
        // as in the single-step kernel: fills nobody waited for land first
        if (failed && lane == 0)
            for (int j = max(0, k - St::NST); j < k; j++)
                mbar_wait(&full[j % St::NST], (unsigned)((j / St::NST) & 1), kWaitLimit);
    } else {
        constexpr int UW = W / 2 + 2;  // units of a ring row
        constexpr int NT = kConsumerWarps * 32;
        static_assert(UW * (H + 2) <= 3 * NT, "UnitSums: at most three units a thread");
        bool waited = false;  // for the previous grid
        UnitSums us1, us2;    // kModeSums: terms of the first and the second step
        for (int i = 0;; i++) {
            const int s = i % St::NST;
            const unsigned phase = (unsigned)((i / St::NST) & 1);
            bool ok = mbar_wait(&ready[s], phase, kWaitLimit);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) atomicOr(a.error_word, 2u);
                break;
            }
            const int4 sl = get_slot(slot + 2 * s), sp = get_slot(slot + 2 * s + 1);
            if (sl.x == -1) break;
            const bool clean = sl.x != 0;
            const int x0 = sl.y, y0 = sl.z;
            T* sb = bufs + (size_t)s * St::STAGE_ELEMS;
            // first step, general-path nodes: their populations come from the
            // source buffer, so their loads and arithmetic run while the
            // tile's bytes are on their way
            bool landed = false;
            Acc ns[3] = {0, 0, 0};
            for (int e = sp.x + (NT - 1 - tid); e < sp.y; e += NT) {
                const int w = p.sp1[e];
                const int dx = (w & 255) - 1, dy = (w >> 8 & 255) - 1;
                const uint8_t fl = (uint8_t)(w >> 16);
                int x = x0 + dx, y = y0 + dy;
                const bool own = dx >= 0 && dx < W && dy >= 0 && dy < H && x < g.nx && y < g.ny;
                // a ring node beyond a periodic edge is the one across it
                x = x < 0 ? x + g.nx : (x >= g.nx ? x - g.nx : x);
                y = y < 0 ? y + g.ny : (y >= g.ny ? y - g.ny : y);
                float f[9];
                unsigned outmask;
                Acc t[kNumSums] = {0, 0, 0, 0, 0, 0};
                if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
                waited = true;
                load_post_stream<T>(a, x, y, fl, f, &outmask);
                if (fl) apply_bc(a, f, x, y, fl);
                node_collide<OP>(a, (long long)y * g.pitch + x, f, t, own);
                if (!landed) ok = mbar_wait(&full[s], phase, kWaitLimit);
                landed = true;
                if (ok) pair_put_first<St>(a, b.edge, sb, dx, dy, x, y, f, outmask, fl, own);
                if (MODE == kModeSums)
#pragma unroll
                    for (int k = 0; k < 3; k++) ns[k] += t[k];
                if (MODE == kModeFull && a.partials)
#pragma unroll
                    for (int k = 0; k < kNumSums; k++) v1[k] += t[k];
            }
            if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
            waited = true;
            if (!landed) ok = mbar_wait(&full[s], phase, kWaitLimit);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) atomicOr(a.error_word, 2u);
                break;
            }
            if (MODE == kModeSums) node_sums_add(ns, a.partials && sp.x < sp.y, tsums);
            // first step: the tile and the ring around it
#pragma unroll 1
            for (int u = tid; u < UW * (H + 2); u += NT) {
                const int r = u / UW, c = u - r * UW;
                const int dx = 2 * c - 2, dy = r - 1;
                const int x = x0 + dx, y = y0 + dy;
                bool live = clean;
                if (!clean) {
                    live = y > 0 && y < g.ny - 1 && x > 0 && x + 1 < g.nx - 1;
                    if (live && a.special_bits) {
                        const long long unit = ((long long)y * g.pitch + x) >> 1;
                        live = ((a.special_bits[unit >> 5] >> (unit & 31)) & 1u) == 0;
                    }
                }
                if (live)
                    pair_unit_first<St, OP, MODE>(a, sb, dx, dy, x, y, v1, dx >= 0 && dx < W && dy >= 0 && dy < H, us1,
                                                  tsums);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&mid[s]);
            ok = mbar_wait(&mid[s], phase, kWaitLimit);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) atomicOr(a.error_word, 2u);
                break;
            }
            // second step: general-path nodes on the last warps, which have
            // fewer units to do
            ns[0] = ns[1] = ns[2] = 0;
            for (int e = sp.z + (NT - 1 - tid); e < sp.w; e += NT) {
                const int w = p.sp0[e];
                const int dx = (w & 255) - 1, dy = (w >> 8 & 255) - 1;
                Acc t[kNumSums] = {0, 0, 0, 0, 0, 0};
                pair_node_second<St, OP>(b, p.edge_in, sb, dx, dy, x0 + dx, y0 + dy, (uint8_t)(w >> 16), t);
                if (MODE == kModeSums)
#pragma unroll
                    for (int k = 0; k < 3; k++) ns[k] += t[k];
                if (MODE == kModeFull && b.partials)
#pragma unroll
                    for (int k = 0; k < kNumSums; k++) v2[k] += t[k];
            }
            if (MODE == kModeSums) node_sums_add(ns, sp.z < sp.w, tsums + 3);
            // second step: the tile
#pragma unroll 1
            for (int u = tid; u < W / 2 * H; u += NT) {
                const int dy = u / (W / 2), dx = 2 * (u - dy * (W / 2));
                const int x = x0 + dx, y = y0 + dy;
                bool live = clean;
                if (!clean) {
                    live = y < g.ny && x + 1 < g.nx;
                    if (live && b.special_bits) {
                        const long long unit = ((long long)y * g.pitch + x) >> 1;
                        live = ((b.special_bits[unit >> 5] >> (unit & 31)) & 1u) == 0;
                    }
                }
                if (live) pair_unit_second<St, OP, MODE>(b, sb, dx, dy, x, y, v2, us2, tsums + 3);
            }
            // the next fill of this stage (async proxy) follows these accesses
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (MODE == kModeSums && __any_sync(0xffffffffu, unit_sums_large(us1) || unit_sums_large(us2))) {
                unit_sums_add(us1, tsums);
                unit_sums_add(us2, tsums + 3);
            }
        }
        if (MODE == kModeSums) {
            unit_sums_add(us1, tsums);
            unit_sums_add(us2, tsums + 3);
        }
    }
    if (MODE == kModeSums) {
        __syncthreads();
        if (tid < 6) {
            double* part = tid < 3 ? a.partials : b.partials;
            unsigned long long* acc =
                reinterpret_cast<unsigned long long*>(part) + (blockIdx.x % kSumSlots) * kNumSums + tid % 3;
            unsigned long long t = 0;
            for (int w = 0; w < kConsumerWarps; w++) t += tsums_buf[6 * w + tid];
            if (part && t != 0) atomicAdd(acc, t);
        }
    } else if (MODE == kModeFull && (a.partials || b.partials)) {
        pair_block_sums(p, v1, v2);
    }
}

template <typename T, int OP, int MODE, int SHAPE>
static cudaError_t launch_pair_variant(const PairArgs& p, const CUtensorMap& tmap, cudaStream_t s) {
    using St = PairStaging<T, SHAPE>;
    static unsigned long long configured = 0;  // the attribute, set once per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (!(configured >> (dev & 63) & 1ull)) {
        cudaError_t e = cudaFuncSetAttribute(pair_kernel<T, OP, MODE, SHAPE>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)St::SMEM);
        if (e != cudaSuccess) return e;
        configured |= 1ull << (dev & 63);
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)std::min(p.ntiles, pair_ctas(SHAPE, (int)sizeof(T), MODE) * p.num_sms));
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = St::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, pair_kernel<T, OP, MODE, SHAPE>, p, tmap);
}

template <typename T, int OP, int SHAPE>
static cudaError_t launch_pair_shape(const PairArgs& p, const CUtensorMap& tmap, cudaStream_t s) {
    switch (pair_mode(p)) {
    case kModeLean: return launch_pair_variant<T, OP, kModeLean, SHAPE>(p, tmap, s);
    case kModeSums: return launch_pair_variant<T, OP, kModeSums, SHAPE>(p, tmap, s);
    case kModeField: return launch_pair_variant<T, OP, kModeField, SHAPE>(p, tmap, s);
    default: return launch_pair_variant<T, OP, kModeFull, SHAPE>(p, tmap, s);
    }
}

// the shapes pair_shape chooses for the type and operator
template <typename T, int OP>
static cudaError_t launch_pair_op(const PairArgs& p, const CUtensorMap& tmap, cudaStream_t s) {
    constexpr bool half = sizeof(T) == 2;
    if (p.shape == 0)
        if constexpr (half || OP != LBMX_CM) return launch_pair_shape<T, OP, 0>(p, tmap, s);
    if (p.shape == 1)
        if constexpr (half || OP == LBMX_CM) return launch_pair_shape<T, OP, 1>(p, tmap, s);
    if (p.shape == 2) return launch_pair_shape<T, OP, 2>(p, tmap, s);
    if (p.shape == 3) return launch_pair_shape<T, OP, 3>(p, tmap, s);
    return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_pair(const PairArgs& p, const CUtensorMap& tmap, int op, cudaStream_t s) {
    switch (op) {
    case LBMX_BGK: return launch_pair_op<T, LBMX_BGK>(p, tmap, s);
    case LBMX_MRT: return launch_pair_op<T, LBMX_MRT>(p, tmap, s);
    case LBMX_CM: return launch_pair_op<T, LBMX_CM>(p, tmap, s);
    default: return cudaErrorInvalidValue;
    }
}

#define LBMX_INSTANTIATE_PAIR(T) \
    template cudaError_t launch_pair<T>(const PairArgs&, const CUtensorMap&, int, cudaStream_t);

}  // namespace lbmx
