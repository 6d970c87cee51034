// FP32 pair passes over neighbour lists and staged windows, one thread per
// particle.
//
// A tile is 128 consecutive slots (a thread block). Particles are stored in cell
// order, so the neighbours of a tile's particles lie in a few contiguous slot
// ranges: for every run of the tile's particles that share a cell row (and
// instance), the three neighbouring rows' cells from one before the run's
// first to one after its last. These ranges, each widened to multiples of four
// slots, are the tile's window (TileWin, written at a neighbour rebuild): about
// 470 slots on a lattice at rest. A pass copies the arrays it reads of
// neighbours into shared memory once per tile (16-byte asynchronous copies,
// 3.7 slots a particle instead of 21 gathers from L1), and a particle's
// neighbours are 16-bit byte offsets into that window.
//
//   candidates  per particle, the rebuild-time neighbours (the set bits of its
//               row masks, in slot order), written after a rebuild or when a
//               restored state has masks but no list
//   in support  per particle, this step's neighbours with r^2 < 4h^2, written
//               by the density pass and read by the later passes of the step
//
// Lists are stored as quads of four offsets, [tile][quad][thread], so a warp reads
// four neighbours of all its particles in one coalesced 8-byte load; the last
// quad is padded with the particle's last entry. Visiting order, pair terms and
// sums are those of the mask walks (for_each_neighbor), operation by operation,
// so results are the same bits; what goes away is the walk itself: finding set
// bits, moving from word to word (some lane of a warp does that in nearly every
// iteration), and 64-bit addresses for every array. A tile whose window exceeds
// its capacity keeps lists of slots, and its passes read memory (TileKind). Particles
// that have no list (more than 48 candidates, or in a tile of more than 8 runs or with
// a window wider than 16 bits) are marked and take the mask walk.
//
// Bound: shared-memory wavefronts and issue slots together (accel at 1M: 71% of
// the wavefront rate, 57% of the issue slots, 913 warp instructions a warp where
// the mask walk ran 1449). Measured per launch at 1,048,576 particles, mask walk
// -> lists: density 58.1 -> 45.5 us, accel 59.2 -> 47.8, accel + drag 70.8 -> 49.8,
// pass 1 82.7 -> 61.5, pass 2 64.1 -> 48.3; a rebuild's masks and lists 52 -> 72 us
// (k_nl_window), 111 with the step's density (k_nl_density_win).
// Reading the lists two quads ahead (accel 46 -> 49 us), copying a tile's lists
// to shared memory first (density 45 -> 51) and 16-byte interleaved windows
// (below) were slower.
#pragma once

#include "sph_kernels.cuh"

namespace sphgb {

constexpr int kTile = 128;     // slots of a tile = threads of its block
constexpr int kWinMax = 640;   // window capacity in slots (rest: ~470)
constexpr int kRunMax = 8;     // cell-row runs of a tile
constexpr int kRangeMax = 3 * kRunMax;
constexpr int kQuads = 12;     // list capacity: 48 entries
constexpr int kNoList = 255;   // count of a particle without a list
constexpr int kSpilled = 64;   // flag beside the candidate count of a particle whose rows
                               // exceed the 64-slot masks
// While lists are collected, entry k of thread t lies at row k, column t: a store
// has a two-way bank conflict at most, wherever each lane's list ends (a run of
// entries per thread, its stride an odd number of words: 3.4 wavefronts on
// average, mask and list build of 1M particles 69.1 us against 66.5)
constexpr int kRow = 2 * kTile;            // bytes of a row
constexpr int kListStride = 8 * kQuads + 4; // bytes per thread: the list and two rows more
constexpr int kNlStride = 8 * kQuads + 20;  // the same with room for eight entries past
                                            // the capacity (nl_window)

struct TileWin {
    int32_t nr;               // ranges (0: no window)
    int32_t pad[3];
    int32_t start[kRangeMax]; // first slot, a multiple of 4 (no window: of all ranges)
    int32_t base[kRangeMax + 1]; // first window slot; base[nr] = window slots
    int32_t pad2[3];
};

// The lists of one state (device pointers; win NULL: it has none and every
// particle takes the mask walk).
struct WinLists {
    TileWin *win;
    uint2 *cand, *supp;        // [tile][kQuads][kTile]
    uint8_t *candCnt, *suppCnt; // per slot; kNoList: mask walk
};

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}
// Element at byte offset o of a staged array (s_win is in shared memory).
__device__ __forceinline__ float2 lds2(const unsigned char *sw, uint32_t o)
{
    return *reinterpret_cast<const float2 *>(sw + o);
}
__device__ __forceinline__ float lds1(const unsigned char *sw, uint32_t o)
{
    return *reinterpret_cast<const float *>(sw + o);
}
__device__ __forceinline__ void copy16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Bytes of a staged array.
constexpr int kWin8 = 8 * kWinMax;
constexpr int kWin4 = 4 * kWinMax;

// Where a pass reads its neighbours: float2 array k and, behind N8 of those, a float
// array, at a list's entry e.
struct InWindow { // staged, e a byte offset
    const unsigned char *sw;
    __device__ __forceinline__ float2 a(int k, uint32_t e) const { return lds2(sw + k * kWin8, e); }
    template <int N8> __device__ __forceinline__ float f(uint32_t e) const
    {
        return lds1(sw + N8 * kWin8, e >> 1);
    }
};
struct InMemory { // of a tile without a window, e a slot from its first one on
    const float2 *p0, *p1, *p2, *p3;
    const float *pf;
    __device__ __forceinline__ float2 a(int k, uint32_t e) const
    {
        return (k == 0 ? p0 : k == 1 ? p1 : k == 2 ? p2 : p3)[e];
    }
    template <int N8> __device__ __forceinline__ float f(uint32_t e) const { return pf[e]; }
};

// Copy the tile's window of the given arrays into shared memory at sw, sw +
// kWin8, ... (N8 float2 arrays), then a float array. Range ends are multiples of
// four slots, so a copy may read up to three elements past the last particle:
// every staged array has room for them. All threads of the block call it. Returns the
// ranges: 0 is a tile without a window, whose lists hold slots from w->start[0] on.
//
// Neighbours are then read eight bytes at a time: 4.2 wavefronts a warp read
// (2.1 per 16 lanes; bank padding, swizzles, 4-byte arrays were no better), and
// 16-byte reads of interleaved arrays measured slower (8.8 wavefronts where two
// 8-byte reads take 8.4: accel 46 -> 55 us, pass 1 60 -> 74 us at 1M).
template <int N8, bool F4>
__device__ __forceinline__ int stage_window(const TileWin *__restrict__ w,
                                             const unsigned char *sw, const float2 *a0,
                                             const float2 *a1, const float2 *a2, const float2 *a3,
                                             const float *f)
{
    const uint32_t sm = smem_addr(sw);
    const int lane = (int)(threadIdx.x & 31u);
    const int nr = w->nr;
    const int st = lane < nr ? w->start[lane] : 0;
    const int bs = lane <= nr ? w->base[lane] : 0;
    const int total = __shfl_sync(0xffffffffu, bs, nr);
    const int rounds = (total / 2 + kTile - 1) / kTile;
    for (int q = 0; q < rounds; ++q) {
        const int k = 2 * (q * kTile + (int)threadIdx.x);
        int r = 0;
        for (int t = 1; t < nr; ++t) r += k >= __shfl_sync(0xffffffffu, bs, t) ? 1 : 0;
        const int src = __shfl_sync(0xffffffffu, st, r) + k - __shfl_sync(0xffffffffu, bs, r);
        if (k < total) {
            const uint32_t d = sm + 8 * k;
            copy16(d, a0 + src);
            if (N8 > 1) copy16(d + kWin8, a1 + src);
            if (N8 > 2) copy16(d + 2 * kWin8, a2 + src);
            if (N8 > 3) copy16(d + 3 * kWin8, a3 + src);
            if (F4 && !(k & 2)) copy16(sm + N8 * kWin8 + 4 * k, f + src);
        }
    }
    copy_wait();
    __syncthreads();
    return nr;
}

__device__ __forceinline__ uint32_t entry_of(const uint2 &e, int k)
{
    const uint32_t w = k < 2 ? e.x : e.y;
    return (k & 1) ? w >> 16 : w & 0xffffu;
}

// The collected list of a thread (n entries at its place in shared memory) to
// its quads, the last one padded with the last entry.
__device__ __forceinline__ void write_list(unsigned char *place, int n, uint2 *__restrict__ out)
{
    const uint16_t *p = reinterpret_cast<const uint16_t *>(place);
    int q = 0;
    for (; 4 * q + 4 <= n; ++q, p += 4 * kTile)
        out[q * kTile] = make_uint2(p[0] | (uint32_t)p[kTile] << 16,
                                    p[2 * kTile] | (uint32_t)p[3 * kTile] << 16);
    if (const int left = n & 3) { // padded with the last entry
        const uint32_t a = p[0], b = p[left > 1 ? kTile : 0];
        const uint32_t c = left > 2 ? p[2 * kTile] : b;
        out[q * kTile] = make_uint2(a | b << 16, c | c << 16);
    }
}

// The window of a tile whose particles lie in cells (cx, cy) of instance b:
// TileWin, and for this thread's run the window slot of a slot j of row r as
// T.base[3 run + r] + j - T.start[3 run + r]. Returns kWindow if the window fits. If it
// does not, but its slots span 16 bits, kFar: the lists hold slots from T.first on and the
// passes read memory. (Where a column has pressed through a wall, a border cell holds
// what would be many cells, and such a tile's walk over rows of some hundred slots was
// the end of every pass: a batch of eight, 51,500 particles, 1000 steps on, 32 steps with
// gradient 8.8 ms, so 2.7; 90,000 particles 6.4 ms, so 2.5.) Otherwise kNone: the mask walk. All threads call it; it ends with a
// barrier.
enum TileKind : int { kNone = 0, kFar, kWindow };
struct TileShared {
    int key[kTile], cnt[kTile / 32];
    int lo[kRunMax], hi[kRunMax], inst[kRunMax], cy[kRunMax];
    int start[32], len[32], base[33];
    int first, span;
};
template <bool MULTI>
__device__ __forceinline__ int tile_window(TileShared &T, const Inst<float> &one,
                                            const Inst<float> *inst,
                                            const int32_t *__restrict__ cellStart, bool live, int b,
                                            int cx, int cy, TileWin *W, int &run, int &nrun)
{
    const int t = (int)threadIdx.x, lane = t & 31, warp = t >> 5;
    const int key = live ? (b << 15) | cy : -1;
    T.key[t] = key;
    if (t < kRunMax) {
        T.lo[t] = INT_MAX;
        T.hi[t] = 0;
    }
    if (t < 32) T.len[t] = 0;
    __syncthreads();
    const bool first = live && (t == 0 || T.key[t - 1] != key);
    const unsigned fm = __ballot_sync(0xffffffffu, first);
    if (lane == 0) T.cnt[warp] = __popc(fm);
    __syncthreads();
    run = __popc(fm & (0xffffffffu >> (31 - lane))) - 1;
    nrun = 0;
#pragma unroll
    for (int w = 0; w < kTile / 32; ++w) {
        if (w < warp) run += T.cnt[w];
        nrun += T.cnt[w];
    }
    // each run's first and last cell: one atomic pair per run and warp
    if (live && run < kRunMax) {
        const unsigned peers = __match_any_sync(__activemask(), run);
        const int lo = __reduce_min_sync(peers, cx), hi = __reduce_max_sync(peers, cx);
        if (lane == __ffs((int)peers) - 1) {
            atomicMin(&T.lo[run], lo);
            atomicMax(&T.hi[run], hi);
        }
        if (first) {
            T.inst[run] = b;
            T.cy[run] = cy;
        }
    }
    __syncthreads();
    bool ok = nrun <= kRunMax;
    if (ok && t < 3 * nrun) {
        const int q = t / 3;
        decltype(auto) I = pick_inst<MULTI>(one, inst, T.inst[q]);
        const int jy = T.cy[q] + t % 3 - 1;
        int a = 0, e = 0;
        if (jy >= 1 && jy <= I.ny) {
            const int xa = T.lo[q] - 1 > 1 ? T.lo[q] - 1 : 1;
            const int xb = T.hi[q] + 1 < I.nx ? T.hi[q] + 1 : I.nx;
            const int row = I.coff + (jy - 1) * I.nx;
            a = cellStart[row + xa - 1];
            e = cellStart[row + xb];
        }
        T.start[t] = a & ~3;
        T.len[t] = e > a ? ((e - (a & ~3) + 3) & ~3) : 0;
    }
    __syncthreads();
    if (t < 32) {
        const int n = T.len[t];
        int x = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        T.base[t] = x - n;
        const int lo = __reduce_min_sync(0xffffffffu, n ? T.start[t] : INT_MAX);
        const int hi = __reduce_max_sync(0xffffffffu, n ? T.start[t] + n : 0);
        if (t == 31) {
            T.base[32] = x;
            T.first = x ? lo : 0;
            T.span = x ? hi - lo : 0;
        }
    }
    __syncthreads();
    const bool far = ok && T.base[32] > kWinMax && T.span <= 65536;
    ok = ok && T.base[32] <= kWinMax;
    if (t == 0) W->nr = ok ? 3 * nrun : 0;
    if (t < kRangeMax) W->start[t] = ok && t < 3 * nrun ? T.start[t] : t == 0 ? T.first : 0;
    if (t <= kRangeMax) W->base[t] = ok ? T.base[t] : 0;
    return ok ? kWindow : far ? kFar : kNone;
}

// Which of the kAhead slots from j on (below e) are neighbours of a particle at xr, by the
// positions x of the rebuild. Their loads overlap: such a row has hundreds of slots.
constexpr int kAhead = 8;
__device__ __forceinline__ uint32_t test_slots(const Inst<float> &I, const float2 &xr,
                                               const float2 *x, int j, int e)
{
    float2 xj[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) xj[k] = x[j + k < e ? j + k : j];
    uint32_t in = 0;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
        const float r2 = r2_exact<float>(sub_rn(xr.x, xj[k].x), sub_rn(xr.y, xj[k].y));
        in |= (uint32_t)(j + k < e && lt_nonneg(I.r2min, r2) && lt_nonneg(r2, I.rc2)) << k;
    }
    return in;
}

// The candidate list of a particle in cell (cx, cy) by the test of its rows' rebuild
// positions x (its own is xr), as for_each_neighbor takes it: entries off(slot), at most
// maxnb of them; its length, or kNoList if it does not fit.
template <typename Off>
__device__ __forceinline__ int scan_list(const Inst<float> &I, int cx, int cy, const float2 &xr,
                                         const float2 *x, const int32_t *cellStart, uint16_t *to,
                                         Off &&off)
{
    const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
    const int jx1 = cx + 1 < I.nx ? cx + 1 : I.nx;
    int n = 0;
#pragma unroll 1
    for (int r = 0; r < 3; ++r) {
        const int jy = cy + r - 1;
        if (jy < 1 || jy > I.ny) continue;
        const int row = I.coff + (jy - 1) * I.nx;
        const int e = cellStart[row + jx1];
        for (int j = cellStart[row + jx0 - 1]; j < e; j += kAhead) {
            uint32_t in = test_slots(I, xr, x, j, e);
            for (; in; in &= in - 1u) {
                if (n >= I.maxnb) return n;
                if (n == 4 * kQuads) return kNoList;
                to[kTile * n++] = (uint16_t)off(r, j + __ffs((int)in) - 1);
            }
        }
    }
    return n;
}

// density_kernel! + eos_kernel! of one particle and its in-support list, from its n
// candidates: cand(q) gives the q-th four entries (past the last one, any of them). The list is collected at `place`, which may hold the
// candidates: an entry is written behind those already read. The arithmetic of
// density_pairs_f32, two candidates at a time, or for a particle with spilled rows that
// of density_spill_sum, which scales each pair's term.
template <bool MULTI, typename Read, typename Cand>
__device__ __forceinline__ void density_list(const NLView<float> &v, const WinLists &L, int tile,
                                             int64_t i, const Read &rd, unsigned char *place, int n, bool spilled,
                                             Cand &&cand, float *__restrict__ rho,
                                             float2 *__restrict__ prho)
{
    decltype(auto) I = load_inst<MULTI>(v, i);
    const float r2max = I.p.r2max, invh = I.p.invh, m = I.p.m, A = I.p.A;
    const float2 xi = v.pos[i];
    const float2 ih2 = make_float2(invh, invh), mh = make_float2(-0.5f, -0.5f);
    const float2 one2 = make_float2(1.0f, 1.0f), two2 = make_float2(2.0f, 2.0f);
    const int64_t lbase = (int64_t)tile * (kQuads * kTile) + (int)threadIdx.x;
    int ns = 0;
    float acc = 0.0f;
    // one quad of candidates, `left` of them in the list
    auto quad = [&](const uint2 &cur, int left) {
        float2 xj[4];
        bool in[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) xj[k] = rd.a(0, entry_of(cur, k));
#pragma unroll
        for (int h = 0; h < 4; h += 2) {
            const float2 da = fsub2(xi, xj[h]);
            const float2 db = fsub2(xi, xj[h + 1]);
            const float r2a = da.x * da.x + da.y * da.y;
            const float r2b = db.x * db.x + db.y * db.y;
            in[h] = h < left && r2a < r2max;
            in[h + 1] = h + 1 < left && r2b < r2max;
            const float2 qq = fmul2(make_float2(pair_sqrt(r2a), pair_sqrt(r2b)), ih2);
            float2 u = ffma2(qq, mh, one2); // 1 - q/2
            u.x = in[h] ? u.x : 0.0f;
            u.y = in[h + 1] ? u.y : 0.0f;
            const float2 u2 = fmul2(u, u);
            const float2 u4 = fmul2(u2, u2);
            const float2 w = ffma2(qq, two2, one2); // 2q + 1
            acc = fmaf(u4.x, w.x, acc);
            acc = fmaf(u4.y, w.y, acc);
        }
        // every entry is written, and kept by moving on (ns <= 48: the write
        // after the last kept entry stays inside this thread's place)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            *reinterpret_cast<uint16_t *>(place + ns) = (uint16_t)entry_of(cur, k);
            if (in[k]) ns += kRow;
        }
    };
    if (!spilled) {
        uint2 e = n ? cand(0) : make_uint2(0u, 0u);
        int q = 0;
        for (; q < (n >> 2); ++q) {
            const uint2 cur = e;
            if (4 * q + 4 < n) e = cand(q + 1);
            quad(cur, 4);
        }
        if (n & 3) quad(e, n & 3);
        acc = mul_rn(mul_rn(m, A), acc);
    } else {
#pragma unroll 1
        for (int q = 0; 4 * q < n; ++q) {
            const uint2 cur = cand(q);
#pragma unroll 1
            for (int k = 0; k < 4 && 4 * q + k < n; ++k) {
                const uint32_t o = entry_of(cur, k);
                const float2 xj = rd.a(0, o);
                const float dx = xi.x - xj.x;
                const float dy = xi.y - xj.y;
                const float r2 = dx * dx + dy * dy;
                if (r2 < r2max) {
                    acc += density_pair<float>(r2, invh, m, A);
                    *reinterpret_cast<uint16_t *>(place + ns) = (uint16_t)o;
                    ns += kRow;
                }
            }
        }
    }
    ns /= kRow;
    write_list(place, ns, L.supp + lbase);
    L.suppCnt[i] = (uint8_t)ns;
    density_finish<float>(I, i, acc, rho, prho);
}

// _nl_build! (nl_build_one), the tile's window and the candidate lists of a fresh
// cell list: the rows are scanned in the staged window, and every passing slot
// goes both to its row mask and to the list. One pass instead of a mask build
// (52 us at 1M particles) and a walk of the masks (43 us): 72 us, bound by issue
// slots and shared-memory wavefronts (some 80% of either's rate); 8.4M dense
// particles 775 -> 647 us.
// DENS: the density pass of the same particles follows in the staged window, from
// the lists in shared memory (k_nl_density_win).
template <bool MULTI, bool DENS = false>
__device__ __forceinline__ void nl_window(int64_t N, const Inst<float> &one,
                                          const Inst<float> *inst,
                                          const uint16_t *__restrict__ pinst,
                                          const float2 *__restrict__ pos,
                                          const int32_t *__restrict__ cellStart,
                                          const NlOut<float> &out, const WinLists &L, int tile,
                                          const NLView<float> *v = nullptr, float *rho = nullptr,
                                          float2 *prho = nullptr)
{
    __shared__ TileShared T;
    __shared__ __align__(16) unsigned char s_win[kWin8];
    __shared__ __align__(8) unsigned char s_list[kTile * kNlStride];
    auto walk = [&](int64_t i) { // the density of a particle without a list
        if constexpr (DENS) {
            L.suppCnt[i] = kNoList;
            density_walk<float, MULTI, true>(*v, i, rho, prho, nullptr);
        }
    };
    const int t = (int)threadIdx.x;
    const int64_t i = (int64_t)tile * kTile + t;
    const bool live = i < N;
    const int b = MULTI && live ? (int)pinst[i] : 0;
    decltype(auto) I = pick_inst<MULTI>(one, inst, b);
    const int nx = I.nx, ny = I.ny;
    const float2 xi = live ? pos[i] : make_float2(0.0f, 0.0f);
    const int cx = cell_coord<float>(xi.x * I.invcs, nx);
    const int cy = cell_coord<float>(xi.y * I.invcs, ny);
    int run, nrun;
    const int kind = tile_window<MULTI>(T, one, inst, cellStart, live, b, cx, cy, L.win + tile,
                                        run, nrun);
    unsigned char *const place = s_list + 2 * t;
    uint2 *const list = L.cand + (int64_t)tile * (kQuads * kTile) + t;
    // the density from the list just collected
    auto density = [&](const auto &rd, int n, bool spilled) {
        if constexpr (DENS) {
            const uint16_t *p = reinterpret_cast<const uint16_t *>(place);
            auto four = [&](int q) {
                auto at = [&](int k) {
                    return (uint32_t)p[(4 * q + k < n ? 4 * q + k : n - 1) * kTile];
                };
                return make_uint2(at(0) | at(1) << 16, at(2) | at(3) << 16);
            };
            density_list<MULTI>(*v, L, tile, i, rd, place, n, spilled, four, rho, prho);
        }
    };
    if (kind != kWindow) {
        if (!live) return;
        nl_build_one<float>(N, I, b, i, pos, cellStart, out.center, out.masks, out.nbcount,
                            out.flags);
        int n = kNoList;
        if (kind == kFar)
            n = scan_list(I, cx, cy, xi, pos, cellStart, reinterpret_cast<uint16_t *>(place),
                          [&](int, int j) { return j - T.first; });
        if (n == kNoList) {
            L.candCnt[i] = kNoList;
            walk(i);
            return;
        }
        const bool spilled = out.center[i] >> 31;
        write_list(place, n, list);
        L.candCnt[i] = (uint8_t)(spilled ? n | kSpilled : n);
        density(InMemory{pos + T.first, nullptr, nullptr, nullptr, nullptr}, n, spilled);
        return;
    }
    const int total = T.base[32];
    for (int k = 2 * t; k < total; k += 2 * kTile) {
        int r = 0;
        for (int q = 1; q < 3 * nrun; ++q) r += k >= T.base[q] ? 1 : 0;
        copy16(smem_addr(s_win) + 8 * k, pos + T.start[r] + k - T.base[r]);
    }
    copy_wait();
    __syncthreads();
    if (!live) return;
    const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
    const int jx1 = cx + 1 < nx ? cx + 1 : nx;
    const float rc2 = I.rc2, r2min = I.r2min;
    unsigned char *const full = place + 4 * kQuads * kRow;
    unsigned char *to = place; // the list's end; held at `full` once it is reached
    uint32_t spill = 0;
    uint32_t word[6];
    int cnt[3];
    // every slot's offset is written at the list's end and kept by moving on
    // (writing the passing ones alone, branched or predicated: 74 us instead of 69)
    auto pass = [&](uint32_t o) {
        const float2 d = fsub2(xi, lds2(s_win, o));
        const float2 q = fmul2(d, d);
        const float r2 = add_rn(q.x, q.y);
        const bool in = lt_nonneg(r2min, r2) && lt_nonneg(r2, rc2);
        *reinterpret_cast<uint16_t *>(to) = (uint16_t)o;
        if (in) to += kRow;
        return in;
    };
    // passing slots among the len (at most 32) from offset o, eight at a time
    auto scan32 = [&](uint32_t o, int len) {
        uint32_t w = 0u;
        int k = 0;
        for (; k + 8 <= len; k += 8) {
            uint32_t w8 = 0u;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (pass(o + 8u * (uint32_t)(k + u))) w8 |= 1u << u;
            w |= w8 << k;
            to = to < full ? to : full;
        }
        for (; k < len; ++k)
            if (pass(o + 8u * (uint32_t)k)) w |= 1u << k;
        to = to < full ? to : full;
        return w;
    };
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        word[2 * r] = word[2 * r + 1] = 0u;
        cnt[r] = 0;
        const int jy = cy + r - 1;
        if (jy < 1 || jy > ny) continue;
        const int row = I.coff + (jy - 1) * nx;
        const int a = cellStart[row + jx0 - 1];
        const int len = cellStart[row + jx1] - a;
        if (len > 64) spill = 1;
        const uint32_t o = 8u * (uint32_t)(T.base[3 * run + r] + a - T.start[3 * run + r]);
        word[2 * r] = scan32(o, len < 32 ? len : 32);
        if (len > 32) word[2 * r + 1] = scan32(o + 256u, len < 64 ? len - 32 : 32);
        cnt[r] = __popc(word[2 * r]) + __popc(word[2 * r + 1]);
        for (int k = 64; k < len; k += 32) // only counted
            cnt[r] += __popc(scan32(o + 8u * (uint32_t)k, len - k < 32 ? len - k : 32));
    }
    const int all = cnt[0] + cnt[1] + cnt[2], maxnb = I.maxnb;
    if (all > maxnb) { // keep the first maxnb, as nl_build_one
        int room = maxnb;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int nlo = __popc(word[2 * r]), nhi = __popc(word[2 * r + 1]);
            if (room <= 0) {
                word[2 * r] = word[2 * r + 1] = 0u;
            } else if (room < nlo) {
                word[2 * r] &= (1u << select_bit(word[2 * r], room)) - 1u;
                word[2 * r + 1] = 0u;
            } else if (room < nlo + nhi) {
                word[2 * r + 1] &= (1u << select_bit(word[2 * r + 1], room - nlo)) - 1u;
            }
            room -= cnt[r];
        }
        atomicOr(out.flags + b, FLAG_NL_OVERFLOW);
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) out.masks[(int64_t)q * N + i] = word[q];
    const int n = all < maxnb ? all : maxnb;
    out.center[i] = (uint32_t)cx | ((uint32_t)cy << 16) | (spill << 31);
    out.nbcount[i] = n;
    if (n > 4 * kQuads) {
        L.candCnt[i] = kNoList;
        walk(i);
        return;
    }
    write_list(place, n, list);
    L.candCnt[i] = (uint8_t)(spill ? n | kSpilled : n);
    density(InWindow{s_win}, n, spill != 0);
}

template <bool MULTI>
__global__ void __launch_bounds__(kTile)
    k_nl_window(int64_t N, const Inst<float> one, const Inst<float> *__restrict__ inst,
                const uint16_t *__restrict__ pinst, const float2 *__restrict__ pos,
                const int32_t *__restrict__ cellStart, const NlOut<float> out, const WinLists L)
{
    pdl_enter();
    nl_window<MULTI>(N, one, inst, pinst, pos, cellStart, out, L, (int)blockIdx.x);
}

// The same and the density pass of the step in one launch, which saves the launch, the
// second staging of the window and the read of the lists: 20,000 particles' 16 steps
// 271 -> 267 us, 249,001 particles 41.3 -> 35.9 us a rebuild, 1M 116 -> 111, 8.4M 1030
// -> 1014.
template <bool MULTI>
__global__ void __launch_bounds__(kTile)
    k_nl_density_win(const __grid_constant__ NLView<float> v, const NlOut<float> out,
                     const WinLists L, float *__restrict__ rho, float2 *__restrict__ prho)
{
    pdl_enter();
    nl_window<MULTI, true>(v.N, v.one, v.inst, v.pinst, v.pos, v.cellStart, out, L,
                           (int)blockIdx.x, &v, rho, prho);
}

// Windows and candidate lists from the row masks, after a snapshot was restored (a
// snapshot holds the masks, not the lists).
template <bool MULTI>
__device__ __forceinline__ void window_lists(const NLView<float> &v, const WinLists &L, int tile)
{
    __shared__ TileShared T;
    __shared__ __align__(8) unsigned char s_list[kTile * kListStride];
    const int t = (int)threadIdx.x;
    const int64_t i = (int64_t)tile * kTile + t;
    const bool live = i < v.N;
    const uint32_t cc = live ? v.center[i] : 0u;
    const int cx = (int)(cc & 0xffffu);
    const int cy = (int)((cc >> 16) & 0x7fffu);
    const int b = MULTI && live ? (int)v.pinst[i] : 0;
    int run, nrun;
    const int kind = tile_window<MULTI>(T, v.one, v.inst, v.cellStart, live, b, cx, cy,
                                        L.win + tile, run, nrun);
    if (!live) return;
    if (kind == kNone) {
        L.candCnt[i] = kNoList;
        return;
    }
    // the walk of for_each_neighbor over the masks, as offsets into the window
    decltype(auto) I = pick_inst<MULTI>(v.one, v.inst, b);
    const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
    const int row0 = I.coff + (jx0 - 1) + (cy - 2) * I.nx;
    unsigned char *const place = s_list + 2 * t;
    uint2 *const list = L.cand + (int64_t)tile * (kQuads * kTile) + t;
    if (kind == kFar || (cc >> 31)) { // no window, or rows beyond the masks
        const int n = scan_list(I, cx, cy, v.xref[i], v.xref, v.cellStart,
                                reinterpret_cast<uint16_t *>(place), [&](int r, int j) {
                                    return kind == kFar ? j - T.first
                                                        : 8 * (T.base[3 * run + r] + j -
                                                               T.start[3 * run + r]);
                                });
        if (n != kNoList) write_list(place, n, list);
        L.candCnt[i] = (uint8_t)(n != kNoList && (cc >> 31) ? n | kSpilled : n);
        return;
    }
    uint64_t m[3];
    int off[3];
    int n = 0;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        m[r] = ((uint64_t)v.masks[(2 * r + 1) * v.N + i] << 32) | v.masks[2 * r * v.N + i];
        n += __popcll(m[r]);
        off[r] = m[r] ? 8 * (T.base[3 * run + r] + v.cellStart[row0 + r * I.nx] -
                             T.start[3 * run + r])
                      : 0;
    }
    if (n > 4 * kQuads) {
        L.candCnt[i] = kNoList;
        return;
    }
    uint16_t *to = reinterpret_cast<uint16_t *>(place);
    uint32_t w = (uint32_t)m[0];
    int base = off[0], word = 0;
    for (;;) {
        if (w == 0u) {
            if (++word == 6) break;
            const uint64_t mr = word < 2 ? m[0] : (word < 4 ? m[1] : m[2]);
            base = (word < 2 ? off[0] : (word < 4 ? off[1] : off[2])) + ((word & 1) << 8);
            w = (word & 1) ? (uint32_t)(mr >> 32) : (uint32_t)mr;
            continue;
        }
        const int k = __ffs((int)w) - 1;
        w &= w - 1u;
        *to = (uint16_t)(base + 8 * k);
        to += kTile;
    }
    write_list(place, n, list);
    L.candCnt[i] = (uint8_t)n;
}

template <bool MULTI>
__global__ void __launch_bounds__(kTile)
    k_window_lists(const __grid_constant__ NLView<float> v, const WinLists L)
{
    pdl_enter();
    window_lists<MULTI>(v, L, (int)blockIdx.x);
}

// density_kernel! + eos_kernel! and this step's in-support lists.
template <bool MULTI>
__device__ __forceinline__ void density_window(const NLView<float> &v, const WinLists &L, int tile,
                                               float *__restrict__ rho,
                                               float2 *__restrict__ prho)
{
    __shared__ __align__(16) unsigned char s_win[kWin8];
    __shared__ __align__(8) unsigned char s_list[kTile * kListStride];
    const int t = (int)threadIdx.x;
    const int64_t i = (int64_t)tile * kTile + t;
    const bool live = i < v.N;
    const unsigned char *sw = s_win;
    const int c = live ? (int)L.candCnt[i] : 0;
    const int nr =
        stage_window<1, false>(L.win + tile, sw, v.pos, nullptr, nullptr, nullptr, nullptr);
    if (!live) return;
    if (c == kNoList) {
        L.suppCnt[i] = kNoList;
        density_walk<float, MULTI, true>(v, i, rho, prho, nullptr);
        return;
    }
    const uint2 *list = L.cand + (int64_t)tile * (kQuads * kTile) + t;
    const auto cand = [&](int q) { return list[q * kTile]; };
    const int n = c & (kSpilled - 1);
    const bool spilled = (c & kSpilled) != 0;
    unsigned char *const place = s_list + 2 * t;
    if (nr)
        density_list<MULTI>(v, L, tile, i, InWindow{sw}, place, n, spilled, cand, rho, prho);
    else
        density_list<MULTI>(v, L, tile, i,
                            InMemory{v.pos + L.win[tile].start[0], nullptr, nullptr, nullptr,
                                     nullptr},
                            place, n, spilled, cand, rho, prho);
}

template <bool MULTI>
__global__ void __launch_bounds__(kTile, 11)
    k_density_win(const __grid_constant__ NLView<float> v, const WinLists L,
                  float *__restrict__ rho, float2 *__restrict__ prho)
{
    pdl_enter();
    density_window<MULTI>(v, L, (int)blockIdx.x, rho, prho);
}

// Visit a particle's in-support list: f(offset) for each of its n entries, in
// slot order. Whole quads run four pairs at once, so their loads overlap.
template <typename F>
__device__ __forceinline__ void for_each_entry(const uint2 *__restrict__ list, int n, F &&f)
{
    const int nq = n >> 2;
    uint2 e = n ? list[0] : make_uint2(0u, 0u);
    for (int q = 0; q < nq; ++q) {
        const uint2 cur = e;
        if (4 * q + 4 < n) e = list[(q + 1) * kTile];
#pragma unroll
        for (int k = 0; k < 4; ++k) f(entry_of(cur, k));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (k < (n & 3)) f(entry_of(e, k));
}

// Pressure + viscosity sum of accel_sum over a list: positions, velocities,
// {p/rho^2, 1/rho} (and densities for the artificial viscosity).
template <bool AV, typename Read>
__device__ __forceinline__ void accel_sum_win(const Inst<float> &I, const Read &rd,
                                              const uint2 *__restrict__ list, int n,
                                              const float2 &xi, const float2 &vi,
                                              const float2 &pi, float rhoi, float &ax, float &ay)
{
    const float invh = I.p.invh, m = I.p.m, Fc = I.p.Fc;
    // the model is chosen outside the pair loop, so each loop is one straight
    // body whose multiply-adds contract as in the mask walks' loops
    Visc<float> vc = visc_of<float>(I);
    const float pti = pi.x, iri = pi.y;
    if (!AV || vc.kind != 1) {
        const float tmm = vc.twomumass;
        float2 acc = make_float2(0.0f, 0.0f);
        for_each_entry(list, n, [&](uint32_t o) {
            const float2 xj = rd.a(0, o);
            const float2 vj = rd.a(1, o);
            const float2 pj = rd.a(2, o);
            const float2 d = fsub2(xi, xj);
            const float r2 = d.x * d.x + d.y * d.y;
            const float q = pair_sqrt(r2) * invh;
            const float u = 1.0f - 0.5f * q;
            const float F = Fc * u * u * u;
            const float PF = m * (pti + pj.x) * F;
            const float C = tmm * iri * pj.y * F;
            acc = ffma2(make_float2(-PF, -PF), d, acc);
            acc = ffma2(make_float2(C, C), fsub2(vi, vj), acc);
        });
        ax = acc.x;
        ay = acc.y;
    } else {
        ax = 0.0f;
        ay = 0.0f;
        for_each_entry(list, n, [&](uint32_t o) {
            const float2 xj = rd.a(0, o);
            const float2 vj = rd.a(1, o);
            const float2 pj = rd.a(2, o);
            const float rhoj = rd.template f<3>(o);
            const float dx = xi.x - xj.x;
            const float dy = xi.y - xj.y;
            const float r2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
            accel_add_av(dx, dy, r2, invh, m, Fc, vc, pti, rhoi, rhoj, vi, pj.x, vj, ax, ay);
        });
    }
}

// The sum of particle i of a tile: its list (nr: ranges of the tile's window), or the mask
// walk of a marked one.
template <bool MULTI, bool AV>
__device__ __forceinline__ void accel_any(const NLView<float> &v, const WinLists &L, int tile,
                                          const unsigned char *sw, int nr, int64_t i, const Inst<float> &I,
                                          const float2 *__restrict__ vel,
                                          const float2 *__restrict__ prho,
                                          const float *__restrict__ rho, const float2 &xi,
                                          const float2 &vi, float &ax, float &ay)
{
    const int n = L.win ? (int)L.suppCnt[i] : kNoList;
    if (n == kNoList) {
        accel_sum<float, AV>(v, I, vel, prho, rho, i, xi, vi, ax, ay);
        return;
    }
    const float rhoi = AV && I.p.visc == 1 ? rho[i] : 0.0f;
    const uint2 *list = L.supp + (int64_t)tile * (kQuads * kTile) + threadIdx.x;
    if (nr) {
        accel_sum_win<AV>(I, InWindow{sw}, list, n, xi, vi, prho[i], rhoi, ax, ay);
    } else {
        const int f = L.win[tile].start[0];
        accel_sum_win<AV>(I, InMemory{v.pos + f, vel + f, prho + f, nullptr, AV ? rho + f : nullptr},
                          list, n, xi, vi, prho[i], rhoi, ax, ay);
    }
}

template <bool AV> constexpr int kAccelSmem = 3 * kWin8 + (AV ? kWin4 : 0);

// accel_kernel! + integrate_kernel!
template <bool MULTI, bool AV>
__global__ void __launch_bounds__(kTile, AV ? 1 : 12)
    k_accel_win(const __grid_constant__ NLView<float> v, const WinLists L,
                const float2 *__restrict__ vel, const float2 *__restrict__ prho,
                const float *__restrict__ rho, const float *__restrict__ theta,
                float2 *__restrict__ posOut, float2 *__restrict__ velOut,
                float2 *__restrict__ aOut, float *__restrict__ alphaOut,
                uint32_t *__restrict__ flags, const int32_t *__restrict__ perm,
                float2 *__restrict__ tx, float2 *__restrict__ tv)
{
    pdl_enter();
    __shared__ __align__(16) unsigned char s_win[kAccelSmem<AV>];
    const unsigned char *sw = s_win;
    const int nr = stage_window<3, AV>(L.win + blockIdx.x, sw, v.pos, vel, prho, nullptr, rho);
    const int64_t i = (int64_t)blockIdx.x * kTile + threadIdx.x;
    if (i >= v.N) return;
    const int b = MULTI ? inst_of(v, i) : 0;
    decltype(auto) I = load_inst<MULTI>(v, i);
    const float2 xi = v.pos[i];
    const float2 vi = vel[i];
    float ax, ay;
    accel_any<MULTI, AV>(v, L, (int)blockIdx.x, sw, nr, i, I, vel, prho, rho, xi, vi, ax, ay);
    accel_integrate_finish<float>(I, b, i, xi, vi, ax, ay, theta, posOut, velOut, aOut, alphaOut,
                                  flags, perm, tx, tv);
}

// Largest exponent of the lanes of each instance in the warp, one atomic each.
__device__ __forceinline__ void warp_emax(bool live, int b, int e, int *__restrict__ emax,
                                          int parity, bool multi)
{
    const unsigned act = __ballot_sync(0xffffffffu, live);
    if (!live) return;
    const unsigned peers = multi ? __match_any_sync(act, b) : act;
    const int mx = __reduce_max_sync(peers, e);
    if ((int)lane_id() == __ffs((int)peers) - 1 && mx != INT_MIN)
        atomicMax(emax + 2 * b + parity, mx);
}

// Accel recompute + _adj_integrate! + _adj_drag!
template <bool MULTI, bool AV>
__global__ void __launch_bounds__(kTile, AV ? 1 : 12)
    k_drag_win(const __grid_constant__ NLView<float> v, const WinLists L,
               const float2 *__restrict__ vel, const float2 *__restrict__ prho,
               const float *__restrict__ rho, const float *__restrict__ theta,
               const float2 *__restrict__ gX, float2 *__restrict__ gV, float2 *__restrict__ abar,
               float *__restrict__ galpha, int *__restrict__ emax, int parity)
{
    pdl_enter();
    __shared__ __align__(16) unsigned char s_win[kAccelSmem<AV>];
    const unsigned char *sw = s_win;
    const int nr = stage_window<3, AV>(L.win + blockIdx.x, sw, v.pos, vel, prho, nullptr, rho);
    const int64_t i = (int64_t)blockIdx.x * kTile + threadIdx.x;
    const bool live = i < v.N;
    int e = INT_MIN, b = 0;
    if (live) {
        b = MULTI ? inst_of(v, i) : 0;
        decltype(auto) I = load_inst<MULTI>(v, i);
        const float2 xi = v.pos[i];
        const float2 vi = vel[i];
        float ax, ay;
        accel_any<MULTI, AV>(v, L, (int)blockIdx.x, sw, nr, i, I, vel, prho, rho, xi, vi, ax, ay);
        e = drag_adj_finish<float>(I, i, xi, vi, ax, ay, theta, gX, gV, abar, galpha);
    }
    warp_emax(live, b, e, emax, parity, MULTI);
}

// The pair sums of pass1_sum over a list: positions, velocities, {p/rho^2, 1/rho}, abar
// (and densities).
template <bool AV, typename Read>
__device__ __forceinline__ void pass1_sum_win(const Inst<float> &I, const Read &rd,
                                              const uint2 *__restrict__ list, int n,
                                              const float2 &xi, const float2 &vi,
                                              const float2 &ab, const float2 &pi, float rhoi,
                                              float &gx, float &gy, float &gvx, float &gvy,
                                              float &grh, float &sumS)
{
    const float invh = I.p.invh, m = I.p.m, Fc = I.p.Fc, Gc = I.p.Gc;
    Visc<float> vc = visc_of<float>(I);
    const float pti = pi.x, iri = pi.y;
    if (!AV || vc.kind != 1) {
        const float tmm = vc.twomumass;
        float2 g = make_float2(0.0f, 0.0f), gv = make_float2(0.0f, 0.0f);
        float gr = 0.0f, sS = 0.0f;
        for_each_entry(list, n, [&](uint32_t o) {
            const float2 xj = rd.a(0, o);
            const float2 vj = rd.a(1, o);
            const float2 pj = rd.a(2, o);
            const float2 abj = rd.a(3, o);
            const float2 d = fsub2(xi, xj);
            const float r2 = d.x * d.x + d.y * d.y;
            const float rinv = r2 > 0.0f ? rsqrtf(r2) : 0.0f;
            const float r = r2 * rinv;
            const float q = r * invh;
            const float u = 1.0f - 0.5f * q;
            const float F = Fc * u * u * u;
            const float G = Gc * u * u;
            const float PF = m * (pti + pj.x) * F;
            const float Cbase = tmm * iri * pj.y;
            const float C = Cbase * F;
            const float2 da = fsub2(ab, abj);
            const float2 dv = fsub2(vi, vj);
            const float ad_d = -(da.x * d.x + da.y * d.y);
            const float ad_v = da.x * dv.x + da.y * dv.y;
            const float Fbar = m * (pti + pj.x) * ad_d + Cbase * ad_v;
            const float w = Fbar * G * invh * rinv;
            g = ffma2(make_float2(-PF, -PF), da, g);
            g = ffma2(make_float2(w, w), d, g);
            gv = ffma2(make_float2(C, C), da, gv);
            gr -= C * ad_v * iri;
            sS += F * ad_d;
        });
        gx = g.x;
        gy = g.y;
        gvx = gv.x;
        gvy = gv.y;
        grh = gr;
        sumS = sS;
    } else {
        vc.kind = 1;
        gx = 0, gy = 0, gvx = 0, gvy = 0, grh = 0, sumS = 0;
        for_each_entry(list, n, [&](uint32_t o) {
            const float2 xj = rd.a(0, o);
            const float2 vj = rd.a(1, o);
            const float2 pj = rd.a(2, o);
            const float2 abj = rd.a(3, o);
            const float rhoj = rd.template f<4>(o);
            const float dx = xi.x - xj.x;
            const float dy = xi.y - xj.y;
            const float r2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
            const Pass1Pair<float> t = pass1_pair<float, AV>(r2, dx, dy, invh, m, Fc, Gc, vc, pti,
                                                             iri, rhoi, rhoj, vi, ab, pj, abj, vj);
            gx -= t.gxs;
            gy -= t.gys;
            gx += t.gxa;
            gy += t.gya;
            gvx += t.gvx;
            gvy += t.gvy;
            grh -= t.grs;
            sumS += t.sS;
        });
    }
}

template <bool AV> constexpr int kPass1Smem = 4 * kWin8 + (AV ? kWin4 : 0);

template <bool MULTI, bool AV>
__device__ __forceinline__ void pass1_window(const NLView<float> &v, const WinLists &L, int tile,
                                             const unsigned char *sw, const float2 *__restrict__ vel,
                                             const float2 *__restrict__ prho,
                                             const float *__restrict__ rho,
                                             const float *__restrict__ theta,
                                             const float2 *__restrict__ abar,
                                             const float *__restrict__ galpha,
                                             float2 *__restrict__ gXs, float *__restrict__ grho,
                                             float2 *__restrict__ gV)
{
    int nr = 0;
    if (L.win) nr = stage_window<4, AV>(L.win + tile, sw, v.pos, vel, prho, abar, rho);
    const int64_t i = (int64_t)tile * kTile + threadIdx.x;
    if (i >= v.N) return;
    decltype(auto) I = load_inst<MULTI>(v, i);
    const float2 xi = v.pos[i];
    const float2 vi = vel[i];
    const float2 ab = abar[i];
    const float2 pi = prho[i];
    float gx, gy, gvx, gvy, grh, sumS;
    const int n = L.win ? (int)L.suppCnt[i] : kNoList;
    if (n == kNoList)
        pass1_sum<float, AV>(v, I, i, vel, prho, rho, abar, xi, vi, ab, pi, gx, gy, gvx, gvy, grh,
                             sumS);
    else {
        const uint2 *list = L.supp + (int64_t)tile * (kQuads * kTile) + threadIdx.x;
        const float r = AV && I.p.visc == 1 ? rho[i] : 0.0f;
        if (nr) {
            pass1_sum_win<AV>(I, InWindow{sw}, list, n, xi, vi, ab, pi, r, gx, gy, gvx, gvy, grh,
                              sumS);
        } else {
            const int f = L.win[tile].start[0];
            pass1_sum_win<AV>(I, InMemory{v.pos + f, vel + f, prho + f, abar + f,
                                          AV ? rho + f : nullptr},
                              list, n, xi, vi, ab, pi, r, gx, gy, gvx, gvy, grh, sumS);
        }
    }
    const float rhoi = I.p.eos == 1 || (AV && I.p.visc == 1) ? rho[i] : 0.0f;
    pass1_finish<float>(I, i, xi, ab, pi, rhoi, gx, gy, gvx, gvy, grh, sumS, theta, galpha, gXs,
                        grho, gV);
}

// adj_pass1_kernel! + the gXs half of adj_design_kernel! + _axpy2!(gV, gVs)
template <bool MULTI, bool AV>
__global__ void __launch_bounds__(kTile)
    k_pass1_win(const __grid_constant__ NLView<float> v, const WinLists L,
                const float2 *__restrict__ vel, const float2 *__restrict__ prho,
                const float *__restrict__ rho, const float *__restrict__ theta,
                const float2 *__restrict__ abar, const float *__restrict__ galpha,
                float2 *__restrict__ gXs, float *__restrict__ grho, float2 *__restrict__ gV)
{
    pdl_enter();
    __shared__ __align__(16) unsigned char s_win[kPass1Smem<AV>];
    pass1_window<MULTI, AV>(v, L, (int)blockIdx.x, s_win, vel, prho, rho, theta, abar,
                            galpha, gXs, grho, gV);
}

// The pair sum of pass2_sum over the staged window: positions and grho.
template <bool MULTI>
__device__ __forceinline__ void pass2_window(const NLView<float> &v, const WinLists &L, int tile,
                                             const unsigned char *sw, const float *__restrict__ grho,
                                             const float2 *__restrict__ gXs,
                                             float2 *__restrict__ gX,
                                             const float *__restrict__ galpha,
                                             const int *__restrict__ emax, int parity,
                                             unsigned long long *__restrict__ thetaAcc)
{
    int nr = 0;
    if (L.win) nr = stage_window<1, true>(L.win + tile, sw, v.pos, nullptr, nullptr, nullptr, grho);
    const int64_t i = (int64_t)tile * kTile + threadIdx.x;
    const bool live = i < v.N;
    const int64_t s = live ? i : v.N - 1;
    const int b = MULTI ? inst_of(v, s) : 0;
    decltype(auto) I = load_inst<MULTI>(v, s);
    const float2 xi = v.pos[s];
    float gx = 0.0f, gy = 0.0f;
    if (live) {
        const int n = L.win ? (int)L.suppCnt[i] : kNoList;
        if (n == kNoList) {
            pass2_sum<float>(v, I, i, xi, grho, gx, gy);
        } else {
            const float invh = I.p.invh, m = I.p.m, Fc = I.p.Fc;
            const float gri = grho[i];
            float2 acc = make_float2(0.0f, 0.0f);
            const auto sum = [&](const auto &rd) {
                for_each_entry(L.supp + (int64_t)tile * (kQuads * kTile) + threadIdx.x, n,
                               [&](uint32_t o) {
                                   const float2 xj = rd.a(0, o);
                                   const float grj = rd.template f<1>(o);
                                   const float2 d = fsub2(xi, xj);
                                   const float r2 = d.x * d.x + d.y * d.y;
                                   const float w = pass2_weight<float>(r2, invh, m, Fc, gri, grj);
                                   acc = ffma2(make_float2(w, w), d, acc);
                               });
            };
            if (nr) {
                sum(InWindow{sw});
            } else {
                const int f = L.win[tile].start[0];
                sum(InMemory{v.pos + f, nullptr, nullptr, nullptr, grho + f});
            }
            gx = acc.x;
            gy = acc.y;
        }
    }
    pass2_finish_warp<float>(live, I, b, i, xi, gx, gy, gXs, gX, galpha, emax, parity, thetaAcc);
}

// adj_pass2_kernel! + _axpy2!(gX, gXs) + the exact theta write-back
template <bool MULTI>
__global__ void __launch_bounds__(kTile, 14)
    k_pass2_win(const __grid_constant__ NLView<float> v, const WinLists L,
                const float *__restrict__ grho, const float2 *__restrict__ gXs,
                float2 *__restrict__ gX, const float *__restrict__ galpha,
                const int *__restrict__ emax, int parity,
                unsigned long long *__restrict__ thetaAcc)
{
    pdl_enter();
    __shared__ __align__(16) unsigned char s_win[kWin8 + kWin4];
    pass2_window<MULTI>(v, L, (int)blockIdx.x, s_win, grho, gXs, gX, galpha, emax,
                        parity, thetaAcc);
}

} // namespace sphgb
