// Group-per-particle variants of the neighbour-list and pair-sum kernels, for
// single states too small to fill the GPU one thread per particle (a 2072-
// particle dam break runs 17 blocks; in FP64 those 17 SMs are bound by the
// double-precision pipe while 135 SMs idle). With 16-lane groups the same
// state runs 259 blocks of 128 threads on every SM and its pass-1 kernel
// keeps the FP64 pipe ~70% busy.
//
// A group of G lanes (16 or 32) owns one particle. The particle's candidate
// neighbours (the set bits of its six mask words, in slot order = the
// reference's scan order) are dealt out G at a time: lane g of round r takes
// candidate r*G + g and computes that pair's terms with the same per-pair
// functions as the thread-per-particle kernels. The terms go to shared
// memory, and one lane per running sum adds them in candidate order, so
// every sum sees exactly the operations and the order of the serial loop:
// results are bit-identical to the thread-per-particle kernels (and, in the
// FP64 build, to the reference's). A particle whose rows spill past 64 slots
// (a compressed region: the small dam break has up to ~130 of them while its
// front runs along the floor) has masks for the first 64 slots only; its group scans the rows, keeps
// the reference's row in slot order in shared memory and deals that list out
// the same way (the serial path on one lane, used before, made those steps
// 6-10x slower). Only a row limit maxnb above kSpillList falls back to the
// serial walk on the group's first lane.
#pragma once

#include "sph_kernels.cuh"

namespace sphgb {

constexpr int kCoopBlock = 128;
constexpr int kSpillList = 64; // neighbour list of a spilled particle, in shared memory

// Lanes of one group inside its warp.
template <int G> struct Group {
    int gl;         // lane within the group
    int gi;         // group within the block
    int shift;      // first warp lane of the group
    unsigned mask;  // warp lanes of the group
    __device__ __forceinline__ Group()
    {
        const int lane = (int)(threadIdx.x & 31u);
        gl = lane & (G - 1);
        gi = (int)threadIdx.x / G;
        shift = lane & ~(G - 1);
        mask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << shift);
    }
    __device__ __forceinline__ unsigned ballot(bool p) const
    {
        return __ballot_sync(mask, p) >> shift;
    }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
    template <typename V> __device__ __forceinline__ V from(V x, int src) const
    {
        return __shfl_sync(mask, x, src, G);
    }
};

// One running sum over a round's G term slots, n of them dealt out, those with
// their bit in `inm` in the support: "minus one slot, plus one slot" per pair (sub
// may be NULL). FP32 adds all of them eight at a time: a slot without a pair is a
// zero, and a sum that starts at +0 never becomes -0, so x - 0 and x + 0 leave it as
// it is (pass 1 of 1500 particles, skipping them by their bits: 6.1 us, so 5.5). In
// FP64 an addition takes 64 cycles, and skipping is the shorter way.
template <typename T, int G>
__device__ __forceinline__ T coop_fold(T acc, const T *sub, const T *add, int n, unsigned inm)
{
    if constexpr (sizeof(T) == 4) {
        auto read8 = [](const T *p, float (&x)[8]) {
            const float4 a = *reinterpret_cast<const float4 *>(p);
            const float4 c = *reinterpret_cast<const float4 *>(p + 4);
            x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
            x[4] = c.x, x[5] = c.y, x[6] = c.z, x[7] = c.w;
        };
#pragma unroll
        for (int t = 0; t < G; t += 8) {
            if (t >= n) break;
            float a[8], s[8];
            read8(add + t, a);
            if (sub) read8(sub + t, s);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (sub) acc -= s[u];
                acc += a[u];
            }
        }
    } else {
        for (int t = 0; t < n; ++t)
            if ((inm >> t) & 1u) {
                if (sub) acc -= sub[t];
                acc += add[t];
            }
    }
    return acc;
}

// The candidates of a particle, numbered 0..total-1 in slot order: the set
// bits of its six words (row r = words 2r, 2r+1), or for a spilled particle
// the list spill_list built.
template <typename T> struct Cands {
    uint32_t wd[6];
    int bs[6];  // slot of bit 0 of each word
    int pre[7]; // candidates before each word
    const int32_t *lst; // spilled particle: its neighbour slots (shared memory)
    int nl;
    __device__ __forceinline__ void init_list(const int32_t *l, int n)
    {
        lst = l;
        nl = n;
    }
    __device__ __forceinline__ void init(const NLView<T> &v, const Inst<T> &I, int64_t i,
                                         uint32_t cc, const uint32_t *__restrict__ mk)
    {
        lst = nullptr;
        const int cx = (int)(cc & 0xffffu);
        const int cy = (int)((cc >> 16) & 0x7fffu);
        const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
        const int row0 = I.coff + (jx0 - 1) + (cy - 2) * I.nx; // cell (jx0, cy - 1)
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            wd[2 * r] = mk[(int64_t)(2 * r) * v.N + i];
            wd[2 * r + 1] = mk[(int64_t)(2 * r + 1) * v.N + i];
            const int b = (wd[2 * r] | wd[2 * r + 1]) ? v.cellStart[row0 + r * I.nx] : 0;
            bs[2 * r] = b;
            bs[2 * r + 1] = b + 32;
        }
        pre[0] = 0;
#pragma unroll
        for (int w = 0; w < 6; ++w) pre[w + 1] = pre[w] + __popc(wd[w]);
    }
    // from the words in registers, rows starting at slots b
    __device__ __forceinline__ void init_words(const uint32_t (&words)[6], const int (&b)[3])
    {
        lst = nullptr;
        pre[0] = 0;
#pragma unroll
        for (int w = 0; w < 6; ++w) {
            wd[w] = words[w];
            bs[w] = b[w >> 1] + 32 * (w & 1);
            pre[w + 1] = pre[w] + __popc(wd[w]);
        }
    }
    __device__ __forceinline__ int total() const { return lst ? nl : pre[6]; }
    // slot of candidate k < total(); w, bit: its word and bit (w = -1 for a
    // listed candidate: a spilled particle has no in-support words)
    __device__ __forceinline__ int slot(int k, int &w, int &bit) const
    {
        if (lst) {
            w = -1;
            bit = 0;
            return lst[k];
        }
        uint32_t word = wd[0];
        int base = bs[0], rem = k;
        w = 0;
#pragma unroll
        for (int q = 1; q < 6; ++q)
            if (k >= pre[q]) {
                word = wd[q];
                base = bs[q];
                rem = k - pre[q];
                w = q;
            }
        bit = select_bit(word, rem);
        return base + bit;
    }
};

// The neighbour row of a spilled particle as the generic walk of
// for_each_neighbor visits it: r2min < r^2 < rc^2 on the rebuild positions,
// rows ddy = -1..1, slot order, at most maxnb (<= kSpillList) entries. Each
// round tests G consecutive slots; a ballot gives the kept ones, which are
// written to lst at their rank. Returns the count (the same on every lane).
template <typename T, int G>
__device__ __forceinline__ int spill_list(const Group<G> &g, const NLView<T> &v,
                                          const Inst<T> &I, int64_t i, uint32_t cc,
                                          int32_t *__restrict__ lst)
{
    const int cx = (int)(cc & 0xffffu);
    const int cy = (int)((cc >> 16) & 0x7fffu);
    const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
    const int jx1 = cx + 1 < I.nx ? cx + 1 : I.nx;
    const T2<T> xr = v.xref[i];
    const int maxnb = I.maxnb;
    int cnt = 0;
#pragma unroll 1
    for (int r = 0; r < 3; ++r) {
        const int jy = cy + r - 1;
        if (jy < 1 || jy > I.ny) continue;
        const int row = I.coff + (jy - 1) * I.nx;
        const int b = v.cellStart[row + jx0 - 1];
        const int e = v.cellStart[row + jx1];
        for (int base = b; base < e && cnt < maxnb; base += G) {
            const int j = base + g.gl;
            bool pass = false;
            if (j < e) {
                const T2<T> xj = v.xref[j];
                const T r2 = r2_exact<T>(sub_rn(xr.x, xj.x), sub_rn(xr.y, xj.y));
                pass = lt_nonneg(I.r2min, r2) && lt_nonneg(r2, I.rc2);
            }
            uint32_t kept = g.ballot(pass);
            const int room = maxnb - cnt;
            if (__popc(kept) > room) kept &= (1u << select_bit(kept, room)) - 1u;
            if ((kept >> g.gl) & 1u) lst[cnt + __popc(kept & ((1u << g.gl) - 1u))] = j;
            cnt += __popc(kept);
        }
    }
    g.sync();
    return cnt;
}

// _nl_build! (src/neighbors.jl:192-245) with the row scan spread over the
// group: each round tests G consecutive slots, a ballot gives the passing
// ones, and the first (maxnb - kept) of them are kept, in slot order. The three
// rows' bounds, then their first rounds' positions, are loaded together. Writes
// the particle's masks, count and cell and leaves them in wd, n and the return
// value, with the rows' first slots in bs.
template <typename T, int G>
__device__ __forceinline__ uint32_t nl_group(const Group<G> &g, int64_t N, const Inst<T> &I,
                                             int64_t i, const T2<T> *__restrict__ pos,
                                             const int32_t *__restrict__ cellStart,
                                             const NlOut<T> &out, uint32_t (&wd)[6], int (&bs)[3],
                                             int &n)
{
    const int nx = I.nx, ny = I.ny, maxnb = I.maxnb;
    const T2<T> xi = pos[i];
    const NlTest<T> test(I, xi);
    const int cx = cell_coord<T>(xi.x * I.invcs, nx);
    const int cy = cell_coord<T>(xi.y * I.invcs, ny);
    const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
    const int jx1 = cx + 1 < nx ? cx + 1 : nx;
    int e[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int jy = cy + r - 1;
        const int row = I.coff + (jy - 1) * nx;
        const bool is = jy >= 1 && jy <= ny;
        bs[r] = is ? cellStart[row + jx0 - 1] : 0;
        e[r] = is ? cellStart[row + jx1] : 0;
    }
    T2<T> x0[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) x0[r] = pos[bs[r] + g.gl < e[r] ? bs[r] + g.gl : i];
    uint32_t spill = 0;
    int m = 0;
    bool over = false;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        uint32_t lo = 0, hi = 0;
        const int b = bs[r], len = e[r] - b;
        if (len > 64) spill = 1;
        for (int off = 0; off < len; off += G) {
            const int j = b + off + g.gl;
            bool pass = false;
            if (off + g.gl < len && j != (int)i) pass = test(off == 0 ? x0[r] : pos[j]);
            uint32_t kept = g.ballot(pass);
            const int np = __popc(kept), room = maxnb - m;
            if (np > room) {
                over = true;
                kept = room > 0 ? kept & ((1u << select_bit(kept, room)) - 1u) : 0u;
            }
            m += __popc(kept);
            if (off < 64) {
                const uint64_t w64 = (uint64_t)kept << off;
                lo |= (uint32_t)w64;
                hi |= (uint32_t)(w64 >> 32);
            }
        }
        wd[2 * r] = lo;
        wd[2 * r + 1] = hi;
    }
    const uint32_t cc = (uint32_t)cx | ((uint32_t)cy << 16) | (spill << 31);
    n = m;
    if (g.gl == 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) out.masks[(int64_t)q * N + i] = wd[q];
        out.center[i] = cc;
        out.nbcount[i] = m;
        if (over) atomicOr(out.flags, FLAG_NL_OVERFLOW);
    }
    return cc;
}

template <typename T, int G>
__global__ void __launch_bounds__(kCoopBlock)
    k_nl_build_coop(int64_t N, const Inst<T> I, const T2<T> *__restrict__ pos,
                    const int32_t *__restrict__ cellStart, const NlOut<T> out)
{
    pdl_enter();
    const Group<G> g;
    const int64_t i = (int64_t)blockIdx.x * (kCoopBlock / G) + g.gi;
    if (i >= N) return; // the whole group
    uint32_t wd[6];
    int bs[3], n;
    nl_group<T, G>(g, N, I, i, pos, cellStart, out, wd, bs, n);
}

// density_kernel! + eos_kernel!, and this step's in-support words. BUILD: of a fresh
// cell list; the group builds its particle's masks first and takes them from its
// registers. One launch and one read of the masks less per rebuild: 48 steps of 1500
// FP32 particles with gradient 1.45 -> 1.38 ms.
template <typename T, int G, bool BUILD>
__global__ void __launch_bounds__(kCoopBlock)
    k_density_eos_coop(const __grid_constant__ NLView<T> v, T *__restrict__ rho,
                       T2<T> *__restrict__ prho, uint32_t *__restrict__ tmaskOut,
                       const ThetaFlush<T> flush, const NlOut<T> out)
{
    pdl_enter();
    if (theta_flush<T>(flush)) return;
    constexpr int NG = kCoopBlock / G;
    __shared__ __align__(16) T buf[NG][G];
    __shared__ uint32_t tws[NG][6];
    __shared__ int32_t lst[NG][kSpillList];
    const Group<G> g;
    const int64_t i = (int64_t)blockIdx.x * NG + g.gi;
    if (i >= v.N) return;
    const Inst<T> &I = v.one;
    const T r2max = I.p.r2max, invh = I.p.invh, m = I.p.m, A = I.p.A;
    const T2<T> xi = v.pos[i];
    uint32_t wd[6], cc;
    int bs[3], nb;
    if (BUILD) cc = nl_group<T, G>(g, v.N, I, i, v.pos, v.cellStart, out, wd, bs, nb);
    else cc = v.center[i];
    if ((cc >> 31) && I.maxnb > kSpillList) {
        g.sync(); // the masks just written are read here
        if (g.gl == 0) density_finish<T>(I, i, density_spill_sum<T>(v, I, i, xi, tmaskOut), rho, prho);
        return;
    }
    Cands<T> cd;
    if (cc >> 31) cd.init_list(lst[g.gi], spill_list<T, G>(g, v, I, i, cc, lst[g.gi]));
    else if (BUILD) cd.init_words(wd, bs);
    else cd.init(v, I, i, cc, v.masks);
    const int K = cd.total();
    if (g.gl < 6) tws[g.gi][g.gl] = 0u;
    g.sync();
    T acc = (T)0;
    for (int base = 0; base < K; base += G) {
        const int k = base + g.gl;
        T c = (T)0;
        bool in = false;
        if (k < K) {
            int w, bit;
            const T2<T> xj = v.pos[cd.slot(k, w, bit)];
            const T dx = xi.x - xj.x;
            const T dy = xi.y - xj.y;
            const T r2 = dx * dx + dy * dy;
            if (lt_nonneg(r2, r2max)) {
                in = true;
                c = density_pair<T>(r2, invh, m, A);
                if (w >= 0) atomicOr(&tws[g.gi][w], 1u << bit);
            }
        }
        buf[g.gi][g.gl] = c;
        const unsigned inm = g.ballot(in);
        g.sync();
        if (g.gl == 0)
            acc = coop_fold<T, G>(acc, nullptr, buf[g.gi], K - base < G ? K - base : G, inm);
        g.sync();
    }
    if (tmaskOut && g.gl < 6) tmaskOut[(int64_t)g.gl * v.N + i] = tws[g.gi][g.gl];
    if (g.gl == 0) density_finish<T>(I, i, acc, rho, prho);
}

// Pressure + viscosity pair sum of one particle by its group; lane 0 returns
// (ax, ay).
// The candidates of particle i for a pass after the density pass: this step's
// in-support words, or for a spilled particle its listed row.
template <typename T, int G>
__device__ __forceinline__ Cands<T> pass_cands(const Group<G> &g, const NLView<T> &v,
                                               const Inst<T> &I, int64_t i, uint32_t cc,
                                               int32_t *__restrict__ lst)
{
    Cands<T> cd;
    if (cc >> 31) cd.init_list(lst, spill_list<T, G>(g, v, I, i, cc, lst));
    else cd.init(v, I, i, cc, v.tmask ? v.tmask : v.masks);
    return cd;
}

template <typename T, int G, int NG>
__device__ __forceinline__ void accel_sum_coop(const Group<G> &g, T (*buf)[4][G],
                                               const NLView<T> &v, const Inst<T> &I, int64_t i,
                                               const Cands<T> &cd, const T2<T> *__restrict__ vel,
                                               const T2<T> *__restrict__ prho,
                                               const T *__restrict__ rho, const T2<T> &xi,
                                               const T2<T> &vi, T &ax, T &ay)
{
    const T r2max = I.p.r2max, invh = I.p.invh, m = I.p.m, Fc = I.p.Fc;
    const Visc<T> vc = visc_of<T>(I);
    const T2<T> pi = prho[i];
    const T pti = pi.x, iri = pi.y;
    const T rhoi = vc.kind == 1 ? rho[i] : (T)0;
    const int K = cd.total();
    T acc = (T)0; // lane 0: ax, lane 1: ay
    for (int base = 0; base < K; base += G) {
        const int k = base + g.gl;
        AccelPair<T> t = {(T)0, (T)0, (T)0, (T)0};
        bool in = false;
        if (k < K) {
            int w, bit;
            const int j = cd.slot(k, w, bit);
            const T2<T> xj = v.pos[j];
            const T dx = xi.x - xj.x;
            const T dy = xi.y - xj.y;
            const T r2 = dx * dx + dy * dy;
            if (lt_nonneg(r2, r2max)) {
                in = true;
                const T rhoj = vc.kind == 1 ? rho[j] : (T)0;
                t = accel_pair<T>(r2, dx, dy, invh, m, Fc, vc, pti, iri, rhoi, rhoj, vi, prho[j],
                                  vel[j]);
            }
        }
        buf[g.gi][0][g.gl] = t.px;
        buf[g.gi][1][g.gl] = t.py;
        buf[g.gi][2][g.gl] = t.cx;
        buf[g.gi][3][g.gl] = t.cy;
        const unsigned inm = g.ballot(in);
        g.sync();
        if (g.gl < 2)
            acc = coop_fold<T, G>(acc, buf[g.gi][g.gl], buf[g.gi][2 + g.gl],
                                  K - base < G ? K - base : G, inm);
        g.sync();
    }
    ax = acc;
    ay = g.from(acc, 1);
}

// The passes below have a fifth warp. While the four with the groups go through
// their pairs, its lane t does what the block's t-th particle needs besides the pair
// sums: the design field and the walls (two dependent loads and a division), the
// tape. One lane per group did that behind the sums: 48 steps of 1500 FP32 particles
// with gradient 1.52 -> 1.45 ms.
constexpr int kCoopThreads = kCoopBlock + 32;

// accel_kernel! + integrate_kernel!
template <typename T, int G>
__global__ void __launch_bounds__(kCoopThreads)
    k_accel_integrate_coop(const __grid_constant__ NLView<T> v, const T2<T> *__restrict__ vel,
                           const T2<T> *__restrict__ prho, const T *__restrict__ rho,
                           const T *__restrict__ theta,
                           T2<T> *__restrict__ posOut, T2<T> *__restrict__ velOut,
                           T2<T> *__restrict__ aOut, T *__restrict__ alphaOut,
                           uint32_t *__restrict__ flags, const int32_t *__restrict__ perm,
                           T2<T> *__restrict__ tx, T2<T> *__restrict__ tv)
{
    pdl_enter();
    constexpr int NG = kCoopBlock / G;
    __shared__ __align__(16) T buf[NG][4][G];
    __shared__ int32_t lst[NG][kSpillList];
    __shared__ SideForce<T> side[NG];
    const Group<G> g;
    const bool fifth = threadIdx.x >= kCoopBlock;
    const int q = fifth ? (int)threadIdx.x - kCoopBlock : g.gi;
    const int64_t i = (int64_t)blockIdx.x * NG + q;
    const bool live = q < NG && i < v.N; // of a group: all its lanes or none
    const Inst<T> &I = v.one;
    T2<T> xi = mk2<T>((T)0, (T)0), vi = xi;
    T ax = (T)0, ay = (T)0;
    if (live) {
        xi = v.pos[i];
        vi = vel[i];
        if (fifth) {
            if (tx) {
                // _tape_store! (src/driver.jl:73-77) of the pre-step state, in
                // particle-id order
                const int32_t id = perm[i];
                tx[id] = xi;
                tv[id] = vi;
            }
            side[q] = side_force<T>(I, xi, theta);
        } else {
            const uint32_t cc = v.center[i];
            if ((cc >> 31) && I.maxnb > kSpillList) {
                if (g.gl == 0) accel_sum<T, true>(v, I, vel, prho, rho, i, xi, vi, ax, ay);
            } else {
                const Cands<T> cd = pass_cands<T, G>(g, v, I, i, cc, lst[g.gi]);
                accel_sum_coop<T, G, NG>(g, buf, v, I, i, cd, vel, prho, rho, xi, vi, ax, ay);
            }
        }
    }
    __syncthreads();
    if (!live || fifth || g.gl != 0) return;
    const SideForce<T> f = side[q];
    ax += f.gx;
    ay += f.gy;
    if (aOut) aOut[i] = mk2<T>(ax, ay);
    if (alphaOut) alphaOut[i] = f.al;
    const T dt = I.p.dt;
    const T v1 = (vi.x + dt * ax) * f.D;
    const T v2 = (vi.y + dt * ay) * f.D;
    const T x1 = xi.x + dt * v1;
    const T x2 = xi.y + dt * v2;
    velOut[i] = mk2<T>(v1, v2);
    posOut[i] = mk2<T>(x1, x2);
    if (!(isfinite(x1) && isfinite(x2) && isfinite(v1) && isfinite(v2)))
        atomicOr(flags, FLAG_NONFINITE);
}

// Accel recompute + _adj_integrate! + _adj_drag!; one exponent update per
// particle (these launches cover few particles).
template <typename T, int G>
__global__ void __launch_bounds__(kCoopThreads)
    k_accel_drag_adj_coop(const __grid_constant__ NLView<T> v, const T2<T> *__restrict__ vel,
                          const T2<T> *__restrict__ prho, const T *__restrict__ rho,
                          const T *__restrict__ theta,
                          const T2<T> *__restrict__ gX, T2<T> *__restrict__ gV,
                          T2<T> *__restrict__ abar, T *__restrict__ galpha,
                          int *__restrict__ emax, int parity)
{
    pdl_enter();
    constexpr int NG = kCoopBlock / G;
    __shared__ __align__(16) T buf[NG][4][G];
    __shared__ int32_t lst[NG][kSpillList];
    __shared__ SideForce<T> side[NG];
    __shared__ T2<T> s_gv[NG];
    const Group<G> g;
    const bool fifth = threadIdx.x >= kCoopBlock;
    const int q = fifth ? (int)threadIdx.x - kCoopBlock : g.gi;
    const int64_t i = (int64_t)blockIdx.x * NG + q;
    const bool live = q < NG && i < v.N;
    const Inst<T> &I = v.one;
    const T dt = I.p.dt;
    T2<T> vi = mk2<T>((T)0, (T)0);
    T ax = (T)0, ay = (T)0;
    if (live) {
        const T2<T> xi = v.pos[i];
        vi = vel[i];
        if (fifth) {
            const T2<T> gx = gX[i];
            T2<T> gv = gV[i];
            const SideForce<T> f = side_force<T>(I, xi, theta);
            gv.x += dt * gx.x;
            gv.y += dt * gx.y;
            abar[i] = mk2<T>(dt * f.D * gv.x, dt * f.D * gv.y);
            gV[i] = mk2<T>(f.D * gv.x, f.D * gv.y);
            side[q] = f;
            s_gv[q] = gv;
        } else {
            const uint32_t cc = v.center[i];
            if ((cc >> 31) && I.maxnb > kSpillList) {
                if (g.gl == 0) accel_sum<T, true>(v, I, vel, prho, rho, i, xi, vi, ax, ay);
            } else {
                const Cands<T> cd = pass_cands<T, G>(g, v, I, i, cc, lst[g.gi]);
                accel_sum_coop<T, G, NG>(g, buf, v, I, i, cd, vel, prho, rho, xi, vi, ax, ay);
            }
        }
    }
    __syncthreads();
    if (!live || fifth || g.gl != 0) return;
    const SideForce<T> f = side[q];
    const T2<T> gv = s_gv[q];
    ax += f.gx;
    ay += f.gy;
    const T vx = (vi.x + dt * ax) * f.D;
    const T vy = (vi.y + dt * ay) * f.D;
    const T ga = -dt * f.D * (vx * gv.x + vy * gv.y);
    galpha[i] = ga;
    if (ga != (T)0 && isfinite(ga)) atomicMax(emax + parity, ilogb((double)ga) + 1); // |ga| < 2^e
}

// adj_pass1_kernel! + the gXs half of adj_design_kernel! + _axpy2!(gV, gVs).
// Lanes 0..5 keep gx, gy, gvx, gvy, grho, S.
template <typename T, int G>
__global__ void __launch_bounds__(kCoopThreads)
    k_pass1_design_coop(const __grid_constant__ NLView<T> v, const T2<T> *__restrict__ vel,
                        const T2<T> *__restrict__ prho, const T *__restrict__ rho,
                        const T *__restrict__ theta,
                        const T2<T> *__restrict__ abar, const T *__restrict__ galpha,
                        T2<T> *__restrict__ gXs, T *__restrict__ grho, T2<T> *__restrict__ gV)
{
    pdl_enter();
    constexpr int NG = kCoopBlock / G;
    __shared__ __align__(16) T buf[NG][9][G]; // eight term slots and a row of zeros
    __shared__ int32_t lst[NG][kSpillList];
    __shared__ Pass1Side<T> side[NG];
    const Group<G> g;
    const bool fifth = threadIdx.x >= kCoopBlock;
    const int q = fifth ? (int)threadIdx.x - kCoopBlock : g.gi;
    const int64_t i = (int64_t)blockIdx.x * NG + q;
    const bool live = q < NG && i < v.N;
    const Inst<T> &I = v.one;
    const T2<T> zero = mk2<T>((T)0, (T)0);
    const T2<T> xi = live ? v.pos[i] : zero;
    const T2<T> vi = live ? vel[i] : zero;
    const T2<T> ab = live ? abar[i] : zero;
    const T2<T> pi = live ? prho[i] : zero;
    const uint32_t cc = live ? v.center[i] : 0u;
    T gx = (T)0, gy = (T)0, gvx = (T)0, gvy = (T)0, grh = (T)0, sumS = (T)0;
    if (fifth) {
        if (live) side[q] = pass1_side<T>(I, i, xi, theta, galpha, gV);
    } else if (!live) {
    } else if ((cc >> 31) && I.maxnb > kSpillList) {
        if (g.gl == 0)
            pass1_sum<T, true>(v, I, i, vel, prho, rho, abar, xi, vi, ab, pi, gx, gy, gvx, gvy,
                               grh, sumS);
    } else {
        const T r2max = I.p.r2max, invh = I.p.invh, m = I.p.m, Fc = I.p.Fc, Gc = I.p.Gc;
        const Visc<T> vc = visc_of<T>(I);
        const T pti = pi.x, iri = pi.y;
        const T rhoi = vc.kind == 1 ? rho[i] : (T)0;
        const Cands<T> cd = pass_cands<T, G>(g, v, I, i, cc, lst[g.gi]);
        const int K = cd.total();
        // term slots: 0 gx-, 1 gx+, 2 gy-, 3 gy+, 4 gvx+, 5 gvy+, 6 grho-, 7 S+,
        // 8 zeros. Every running sum takes "minus one slot, plus one slot" per
        // pair, a zero where it has no such term: a sum that starts at +0 never
        // becomes -0, so x - 0 and x + 0 leave it unchanged and each sum sees
        // exactly the serial loop's operations, while all six fold lanes run
        // the same instructions.
        T(*b)[G] = buf[g.gi];
        b[8][g.gl] = (T)0;
        const int fold = g.gl < 6 ? g.gl : 0;
        const T *fsub = b[fold == 0 ? 0 : fold == 1 ? 2 : fold == 4 ? 6 : 8];
        const T *fadd = b[fold == 0 ? 1 : fold == 1 ? 3 : fold == 2 ? 4 : fold == 3 ? 5 : fold == 5 ? 7 : 8];
        T acc = (T)0;
        for (int base = 0; base < K; base += G) {
            const int k = base + g.gl;
            Pass1Pair<T> t = {(T)0, (T)0, (T)0, (T)0, (T)0, (T)0, (T)0, (T)0};
            bool in = false;
            if (k < K) {
                int w, bit;
                const int j = cd.slot(k, w, bit);
                const T2<T> xj = v.pos[j];
                const T dx = xi.x - xj.x;
                const T dy = xi.y - xj.y;
                const T r2 = dx * dx + dy * dy;
                if (lt_nonneg(r2, r2max)) {
                    in = true;
                    const T rhoj = vc.kind == 1 ? rho[j] : (T)0;
                    t = pass1_pair<T>(r2, dx, dy, invh, m, Fc, Gc, vc, pti, iri, rhoi, rhoj, vi,
                                      ab, prho[j], abar[j], vel[j]);
                }
            }
            b[0][g.gl] = t.gxs;
            b[1][g.gl] = t.gxa;
            b[2][g.gl] = t.gys;
            b[3][g.gl] = t.gya;
            b[4][g.gl] = t.gvx;
            b[5][g.gl] = t.gvy;
            b[6][g.gl] = t.grs;
            b[7][g.gl] = t.sS;
            const unsigned inm = g.ballot(in);
            g.sync();
            if (g.gl < 6)
                acc = coop_fold<T, G>(acc, fsub, fadd, K - base < G ? K - base : G, inm);
            g.sync();
        }
        gx = acc;
        gy = g.from(acc, 1);
        gvx = g.from(acc, 2);
        gvy = g.from(acc, 3);
        grh = g.from(acc, 4);
        sumS = g.from(acc, 5);
    }
    __syncthreads();
    if (!live || fifth || g.gl != 0) return;
    const T rhoi = needs_rho_dev(I) ? rho[i] : (T)0;
    pass1_put<T>(I, i, side[q], ab, pi, rhoi, gx, gy, gvx, gvy, grh, sumS, gXs, grho, gV);
}

// adj_pass2_kernel! + _axpy2!(gX, gXs) + the exact theta write-back. A fifth warp
// writes theta back, a lane per particle and corner (a corner waits for the old
// value of its accumulator, so one lane took four waits after the pair sums), and
// loads the next tape state: 1500 FP32 particles 6.4 -> 4.3 us, its floor of a
// launch being 2.
template <typename T, int G>
__global__ void __launch_bounds__(kCoopThreads)
    k_pass2_axpy_coop(const __grid_constant__ NLView<T> v, const T *__restrict__ grho,
                      const T2<T> *__restrict__ gXs, T2<T> *__restrict__ gX,
                      const T *__restrict__ galpha, const int *__restrict__ emax, int parity,
                      unsigned long long *__restrict__ thetaAcc, NextState<T> next)
{
    pdl_enter();
    constexpr int NG = kCoopBlock / G;
    __shared__ __align__(16) T buf[NG][2][G];
    __shared__ int32_t lst[NG][kSpillList];
    const Group<G> g;
    const Inst<T> &I = v.one;
    if (threadIdx.x >= kCoopBlock) {
        const int t = (int)threadIdx.x - kCoopBlock;
        const int64_t i0 = (int64_t)blockIdx.x * NG, it = i0 + (t >> 2);
        const bool load = t < NG && i0 + t < v.N;
        if (load) next.read(i0 + t);
        if (t < 4 * NG && it < v.N)
            theta_add_corner<T>(I, 0, it, v.pos[it], t & 3, galpha, emax, parity, thetaAcc);
        if (load) next.write(i0 + t);
        return;
    }
    const int64_t i = (int64_t)blockIdx.x * NG + g.gi;
    if (i >= v.N) return;
    const T r2max = I.p.r2max, invh = I.p.invh, m = I.p.m, Fc = I.p.Fc;
    const T2<T> xi = v.pos[i];
    const T gri = grho[i];
    const uint32_t cc = v.center[i];
    T gx = (T)0, gy = (T)0;
    if ((cc >> 31) && I.maxnb > kSpillList) {
        if (g.gl != 0) return;
        for_each_neighbor<T>(v, I, i, [&](int j) {
            const T2<T> xj = v.pos[j];
            const T dx = xi.x - xj.x;
            const T dy = xi.y - xj.y;
            const T r2 = dx * dx + dy * dy;
            if (lt_nonneg(r2, r2max)) {
                const T w = pass2_weight<T>(r2, invh, m, Fc, gri, grho[j]);
                gx += w * dx;
                gy += w * dy;
            }
        });
    } else {
        const Cands<T> cd = pass_cands<T, G>(g, v, I, i, cc, lst[g.gi]);
        const int K = cd.total();
        T acc = (T)0;
        for (int base = 0; base < K; base += G) {
            const int k = base + g.gl;
            T tx = (T)0, ty = (T)0;
            bool in = false;
            if (k < K) {
                int w, bit;
                const int j = cd.slot(k, w, bit);
                const T2<T> xj = v.pos[j];
                const T dx = xi.x - xj.x;
                const T dy = xi.y - xj.y;
                const T r2 = dx * dx + dy * dy;
                if (lt_nonneg(r2, r2max)) {
                    in = true;
                    const T wt = pass2_weight<T>(r2, invh, m, Fc, gri, grho[j]);
                    tx = wt * dx;
                    ty = wt * dy;
                }
            }
            buf[g.gi][0][g.gl] = tx;
            buf[g.gi][1][g.gl] = ty;
            const unsigned inm = g.ballot(in);
            g.sync();
            if (g.gl < 2)
                acc = coop_fold<T, G>(acc, nullptr, buf[g.gi][g.gl], K - base < G ? K - base : G,
                                      inm);
            g.sync();
        }
        gx = acc;
        gy = g.from(acc, 1);
        if (g.gl != 0) return;
    }
    pass2_axpy<T>(i, gx, gy, gXs, gX);
}

} // namespace sphgb
