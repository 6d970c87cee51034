// FP64 pair passes with one lane per pair (Morris viscosity).
//
// These passes are bound by GB300's FP64 pipe (1.8 results per clock and SM), in
// which a warp instruction costs the same whatever number of lanes take part.
// With one thread per particle a third of the lanes idle (neighbour counts
// differ, candidates outside the support diverge); with a lane group per
// particle the last round of a group is part empty and each group's first
// lanes fold its sums alone. Here a block takes P consecutive particles and
// deals their pairs out as one flat sequence (particle by particle, in slot
// order), so every lane has a pair:
//
//   density   every candidate's r^2; the in-support pairs are compacted in order
//             into a dense sequence, and only those run the kernel function.
//             The pass leaves, per block, the dense pairs (particle, slot), each
//             pair's F = Fc u^3, and the particles' offsets.
//   force and adjoint passes read that sequence: no masks, no support test, and
//             8 to 10 FP64 operations a pair fewer (r, F and each particle's 2 m mu /
//             rho come with it).
//
// Each pair's terms go to shared memory, and one lane per running sum adds them
// in sequence order, so every sum sees the operations of the serial walk in its
// order: results are the same bits as the other forms'. 32 particles a block
// fill the folding warps; states below 152 x 2 x 32 particles take fewer, so
// that every SM has two blocks. A particle the sequence does not hold (a spilled
// row with maxnb > 64, or more than 64 candidates) is walked by one thread.
//
// FP64 operations a pair, before -> now: density 14 + 5 per candidate outside ->
// 17 + 5, accel 25 -> 18, pass 1 49 -> 46, pass 2 17 -> 9 (square roots and
// divisions not counted, sph_exact64.cuh). Measured per launch, 66,013 particles,
// one thread per particle -> one lane per pair: density 78.2 -> 61.6 us, accel
// 100.6 -> 71.7, accel + drag 104.3 -> 70.7, pass 1 184.7 -> 151.2 (FP64 pipe 79%
// busy), pass 2 69.9 -> 41.2; the solve 5.51 -> 4.22 ms, and with the r, 2 m mu /
// rho and fifth warp of the later passes 3.70 ms. Small states are chains of
// latencies (pass 2 at 240 particles: 4 us), so the density's first warp prepares the
// block alone, a part's loads are issued together, and the folds run ahead of
// their chain: 240 particles 200 steps 9.86 -> 8.22 ms, 925 particles 50 steps 0.92
// -> 0.80, 2072 particles 128 steps 7.09 -> 6.58 (lane groups: 12.0), 66,013 the
// same within 0.3%.
#pragma once

#include "sph_coop.cuh"
#include "sph_window.cuh"

namespace sphgb {

constexpr int kFlatBlock = 128;
constexpr int kFlatMax = 32;    // particles of a block, at most
constexpr int kFlatRow = 64;    // pairs of a particle, at most
constexpr int kFlatChunk = 384; // pairs folded at a time
constexpr int kFlatTest = 256;  // candidates tested at a time (384: density 64.3 us, 62.9 at 256)
constexpr int kFlatOff = kFlatMax + 2; // offsets of a block, then its serial mask
constexpr int kFlatSlotBits = 27;

struct FlatLists {
    double *F, *r;  // [block][P * kFlatRow]
    double *tm;     // per slot: 2 m mu / rho
    uint32_t *pair; // local particle << kFlatSlotBits | neighbour slot
    int32_t *off;   // [block][kFlatOff]
    int P;          // particles of a block
};

// Particles per block: two blocks on each of 152 SMs for small states.
__host__ __device__ __forceinline__ int flat_particles(int64_t N)
{
    const int64_t p = (N + 303) / 304;
    return p < 4 ? 4 : (p > kFlatMax ? kFlatMax : (int)p);
}

// Exclusive scan of one int per lane of a warp.
__device__ __forceinline__ int warp_scan(int x)
{
    const int lane = (int)(threadIdx.x & 31u);
    int s = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    return s - x;
}

// One running sum per lane: the terms k0 .. k1 - 1 in order, sub (may be NULL)
// subtracted before each added one. All lanes of the warp call it (k0 == k1: no
// sum). A dependent FP64 addition takes 64 cycles, so nothing else may stand in
// the chain: the lanes run the same number of steps, a missing term is a zero
// (a sum that starts at +0 never becomes -0, so x + 0 and x - 0 leave it as it
// is), and four terms are read ahead of the four being added. 141 cycles an
// addition with a loop per lane, about 90 this way.
__device__ __forceinline__ double flat_fold(double acc, const double *sub, const double *add,
                                            int k0, int k1)
{
    const int n = k1 > k0 ? k1 - k0 : 0;
    const int most = __reduce_max_sync(0xffffffffu, n);
    double a[4], s[4];
    auto term = [&](const double *p, int k) {
        const double x = p[k < n ? k0 + k : 0];
        return k < n ? x : 0.0;
    };
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        a[u] = term(add, u);
        s[u] = sub ? term(sub, u) : 0.0;
    }
    for (int k = 0; k < most; k += 4) {
        double a2[4], s2[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            a2[u] = term(add, k + 4 + u);
            s2[u] = sub ? term(sub, k + 4 + u) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (sub) acc -= s[u];
            acc += a[u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            a[u] = a2[u];
            s[u] = s2[u];
        }
    }
    return acc;
}

// density_kernel! + eos_kernel!, and the block's dense pairs.
// BUILD: of a fresh cell list of a small single state; the block builds its
// particles' masks first, a warp per particle. 200 steps of 240 particles with
// gradient 8.26 -> 7.90 ms, 50 steps of 925 0.80 -> 0.76, 128 of 2072 6.57 -> 6.46. With
// more particles a block, the warps go through too many in turn: 32 steps at 10 a
// block 2.00 ms either way, at 16 2.35 (a launch of its own) against 2.37, at 32
// 3.55 against 3.64.
constexpr int kFlatBuild = 8; // particles of a block up to which it builds them
template <bool MULTI, bool BUILD>
__global__ void __launch_bounds__(kFlatBlock)
    k_density_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                   double *__restrict__ rho, double2 *__restrict__ prho,
                   const ThetaFlush<double> flush, const NlOut<double> out)
{
    pdl_enter();
    if (theta_flush<double>(flush)) return;
    __shared__ double s_r2[kFlatMax * kFlatRow];
    __shared__ int32_t s_lst[kFlatMax][kFlatRow]; // rows of spilled particles
    __shared__ uint32_t s_wd[kFlatMax][6];
    __shared__ int s_bs[kFlatMax][3], s_pre[kFlatMax][6];
    __shared__ int s_off[kFlatMax + 1], s_cnt[kFlatMax], s_in[kFlatMax];
    __shared__ uint8_t s_own[kFlatMax * kFlatRow];
    __shared__ int s_warp[2][kFlatTest / 32]; // kept per warp and part, by round parity
    __shared__ uint32_t s_spill, s_serial;
    const int t = (int)threadIdx.x, P = B.P;
    const int64_t i0 = (int64_t)blockIdx.x * P;
    const int np = v.N - i0 < P ? (int)(v.N - i0) : P;
    if constexpr (BUILD) {
        const Group<32> g;
        for (int a = t >> 5; a < np; a += kFlatBlock / 32) {
            uint32_t wd[6];
            int bs[3], n;
            const uint32_t cc = nl_group<double, 32>(g, v.N, v.one, i0 + a, v.pos, v.cellStart,
                                                     out, wd, bs, n);
            if (g.gl < 3) s_bs[a][g.gl] = g.gl == 0 ? bs[0] : g.gl == 1 ? bs[1] : bs[2];
            if (g.gl == 0) {
                int k = 0;
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    s_wd[a][q] = wd[q];
                    s_pre[a][q] = k;
                    k += __popc(wd[q]);
                }
                s_cnt[a] = cc >> 31 ? -1 : k;
            }
        }
        __syncthreads();
    }
    if (t < 32) { // the first warp: each particle's candidates and their offsets
        int n = 0;
        bool isSpill = false, isSerial = false;
        if (BUILD) {
            n = t < np ? s_cnt[t] : 0;
            isSerial = n > kFlatRow || (n < 0 && v.one.maxnb > kFlatRow);
            isSpill = n < 0 && !isSerial;
            if (isSerial || isSpill) n = 0;
        } else if (t < np) {
            const int64_t i = i0 + t;
            decltype(auto) I = load_inst<MULTI>(v, i);
            const uint32_t cc = v.center[i];
            uint32_t w[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) w[q] = v.masks[(int64_t)q * v.N + i];
            if (cc >> 31) {
                isSerial = I.maxnb > kFlatRow;
                isSpill = !isSerial;
            } else {
                const int cx = (int)(cc & 0xffffu), cy = (int)((cc >> 16) & 0x7fffu);
                const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
                const int row0 = I.coff + (jx0 - 1) + (cy - 2) * I.nx; // cell (jx0, cy - 1)
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    s_bs[t][r] = (w[2 * r] | w[2 * r + 1]) ? v.cellStart[row0 + r * I.nx] : 0;
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    s_wd[t][q] = w[q];
                    s_pre[t][q] = n;
                    n += __popc(w[q]);
                }
                if (n > kFlatRow) {
                    isSerial = true;
                    n = 0;
                }
            }
        }
        const unsigned sp = __ballot_sync(0xffffffffu, isSpill);
        const unsigned se = __ballot_sync(0xffffffffu, isSerial);
        const int o = warp_scan(n);
        s_cnt[t] = n;
        s_in[t] = 0;
        s_off[t] = o;
        if (t == 31) s_off[32] = o + n;
        if (t == 0) {
            s_spill = sp;
            s_serial = se;
        }
    }
    __syncthreads();
    const uint32_t spill = s_spill, serial = s_serial;
    if (spill) { // list their rows, a warp per particle, and number the candidates again
        const Group<32> g;
        for (int a = t >> 5; a < np; a += kFlatBlock / 32)
            if ((spill >> a) & 1u) {
                const int64_t i = i0 + a;
                decltype(auto) I = load_inst<MULTI>(v, i);
                const int n = spill_list<double, 32>(g, v, I, i, v.center[i], s_lst[a]);
                if ((t & 31) == 0) s_cnt[a] = n;
            }
        __syncthreads();
        if (t < 32) {
            const int n = s_cnt[t], o = warp_scan(n);
            s_off[t] = o;
            if (t == 31) s_off[32] = o + n;
        }
        __syncthreads();
    }
    const int tot = s_off[np];

    const int64_t bb = (int64_t)blockIdx.x * P * kFlatRow;
    const unsigned below = (1u << (t & 31)) - 1u;
    int D = 0; // dense pairs so far
    for (int base = 0, par = 0; base < tot; base += kFlatTest, par ^= 1) {
        constexpr int U = kFlatTest / kFlatBlock;
        // candidate base + 128 u + t: its particle and slot, then all positions,
        // then the test, so that the parts' loads overlap
        int own[U], slot[U];
        double2 xi[U], xj[U];
        double r2[U];
        unsigned in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int p = base + u * kFlatBlock + t;
            own[u] = 0;
            slot[u] = (int)i0;
            if (p < tot) {
                int a = 0;
#pragma unroll
                for (int h = kFlatMax / 2; h > 0; h >>= 1)
                    if (a + h < np && s_off[a + h] <= p) a += h;
                const int k = p - s_off[a];
                own[u] = a;
                if ((spill >> a) & 1u) {
                    slot[u] = s_lst[a][k];
                } else {
                    int w = 0;
#pragma unroll
                    for (int q = 1; q < 6; ++q) w = k >= s_pre[a][q] ? q : w;
                    slot[u] = s_bs[a][w >> 1] + 32 * (w & 1) +
                              select_bit(s_wd[a][w], k - s_pre[a][w]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            xi[u] = v.pos[i0 + own[u]];
            xj[u] = v.pos[slot[u]];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (base + u * kFlatBlock >= tot) { // nothing in this part
                in[u] = 0u;
                continue;
            }
            decltype(auto) I = load_inst<MULTI>(v, i0 + own[u]);
            const double dx = xi[u].x - xj[u].x;
            const double dy = xi[u].y - xj[u].y;
            r2[u] = dx * dx + dy * dy;
            in[u] = __ballot_sync(0xffffffffu, base + u * kFlatBlock + t < tot &&
                                                   lt_nonneg(r2[u], I.p.r2max));
        }
        if ((t & 31) == 0)
#pragma unroll
            for (int u = 0; u < U; ++u) s_warp[par][u * (kFlatBlock / 32) + (t >> 5)] = __popc(in[u]);
        __syncthreads();
        int kept = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int pos = D + kept;
#pragma unroll
            for (int w = 0; w < kFlatBlock / 32; ++w) {
                const int n = s_warp[par][u * (kFlatBlock / 32) + w];
                pos += w < (t >> 5) ? n : 0;
                kept += n;
            }
            if ((in[u] >> (t & 31)) & 1u) {
                pos += __popc(in[u] & below);
                s_r2[pos] = r2[u];
                s_own[pos] = (uint8_t)own[u];
                B.pair[bb + pos] = (uint32_t)own[u] << kFlatSlotBits | (uint32_t)slot[u];
                atomicAdd(&s_in[own[u]], 1);
            }
        }
        D += kept;
    }
    __syncthreads();
    for (int d = t; d < D; d += kFlatBlock) {
        decltype(auto) I = load_inst<MULTI>(v, i0 + s_own[d]);
        const double r = pair_sqrt(s_r2[d]);
        const double q = r * I.p.invh;
        const double u = 1.0 - half_of(q);
        const double u2 = u * u;
        B.F[bb + d] = I.p.Fc * u * u * u;
        B.r[bb + d] = r;
        s_r2[d] = I.p.m * (I.p.A * u2 * u2 * (twice_of(q) + 1.0));
    }
    __syncthreads();
    if (t >= 32) return;
    const int nin = s_in[t], o = warp_scan(nin);
    int32_t *off = B.off + (int64_t)blockIdx.x * kFlatOff;
    if (t <= np) off[t] = o;
    if (t == 31 && np == 32) off[32] = o + nin;
    if (t == 0) off[kFlatOff - 1] = (int)serial;
    if (t >= np) return;
    const int64_t i = i0 + t;
    if ((serial >> t) & 1u) {
        density_walk<double, MULTI, false>(v, i, rho, prho, nullptr);
        decltype(auto) I = load_inst<MULTI>(v, i);
        B.tm[i] = I.p.twomumass * prho[i].y;
        return;
    }
    double acc = 0.0;
#pragma unroll 4
    for (int k = o; k < o + nin; ++k) acc += s_r2[k];
    decltype(auto) I = load_inst<MULTI>(v, i);
    B.tm[i] = I.p.twomumass * density_finish<double>(I, i, acc, rho, prho).y;
}

// ---- the passes that read the dense pairs --------------------------------------
// Five warps: four take the pairs, the fifth meanwhile does what its particles'
// results need besides the pair sums (design field, walls, the theta write-back,
// the next tape state), so that a short pass is one chain of loads, pair terms,
// fold and a few last operations.
constexpr int kFlatThreads = kFlatBlock + 32;
constexpr int kFlatAhead = kFlatChunk / kFlatBlock;

struct FlatShared {
    int off[kFlatMax + 1];
    uint32_t serial;
};

// Where a pass stands: its particles [i0, i0 + np), the thread's role, and the
// first chunk's pairs, read before the offsets that tell how many there are.
template <bool MULTI> struct FlatPass {
    const NLView<double> &v;
    const FlatLists &B;
    int64_t i0, bb;
    int np, t;
    uint32_t e[kFlatAhead];
    double F[kFlatAhead];
    __device__ __forceinline__ FlatPass(const NLView<double> &view, const FlatLists &L,
                                        FlatShared &S)
        : v(view), B(L), i0((int64_t)blockIdx.x * L.P), bb(i0 * kFlatRow), t((int)threadIdx.x)
    {
        np = v.N - i0 < B.P ? (int)(v.N - i0) : B.P;
        const int32_t *o = B.off + (int64_t)blockIdx.x * kFlatOff;
#pragma unroll
        for (int u = 0; u < kFlatAhead; ++u) {
            const int p = t + u * kFlatBlock;
            e[u] = 0u;
            F[u] = 0.0;
            if (t < kFlatBlock && p < B.P * kFlatRow) {
                e[u] = B.pair[bb + p];
                F[u] = B.F[bb + p];
            }
        }
        if (t <= np) S.off[t] = o[t];
        if (t == kFlatBlock) S.serial = (uint32_t)o[kFlatOff - 1];
        __syncthreads();
    }
    // f(place in the chunk, particle, neighbour, F) of the chunk's m pairs, done by
    // the first four warps
    template <typename Fn> __device__ __forceinline__ void pairs(int base, int m, Fn &&f) const
    {
        if (t >= kFlatBlock) return;
#pragma unroll
        for (int u = 0; u < kFlatAhead; ++u) {
            const int p = t + u * kFlatBlock;
            if (p < m) {
                const uint32_t q = base ? B.pair[bb + base + p] : e[u];
                f(p, i0 + (q >> kFlatSlotBits), (int)(q & ((1u << kFlatSlotBits) - 1u)),
                  base ? B.F[bb + base + p] : F[u]);
            }
        }
    }
    // The pairs of the chunk from pair `base` of particle a on: those of the next 16
    // particles where they fit, so that the warp whose lanes fold 16 particles runs
    // once; a moves to the particle after them.
    __device__ __forceinline__ int chunk(const FlatShared &S, int base, int &a) const
    {
        const int n = S.off[np], a1 = (a & ~15) + 16 < np ? (a & ~15) + 16 : np;
        if (S.off[a1] - base <= kFlatChunk) {
            a = a1;
            return S.off[a1] - base;
        }
        return n - base < kFlatChunk ? n - base : kFlatChunk;
    }
    // the particle of the fifth warp's lane (-1: none)
    __device__ __forceinline__ int64_t aside() const
    {
        return t >= kFlatBlock && t - kFlatBlock < np ? i0 + t - kFlatBlock : -1;
    }
};

// A barrier of the four pair warps alone: the fifth is not waited for until the
// results are put together. Not the aligned form (bar.sync): the lanes of a warp come
// from pair terms that only some of them had.
__device__ __forceinline__ void pair_sync()
{
    asm volatile("barrier.sync 1, 128;" ::: "memory");
}

// Pressure + Morris viscosity of the block's particles (accel_pair): s_acc[2 a],
// s_acc[2 a + 1]. side() is what the fifth warp does during the first chunk. All
// threads call it; ends with a barrier.
template <bool MULTI, typename Side>
__device__ __forceinline__ void flat_accel(const FlatPass<MULTI> &Q, const FlatShared &S,
                                           double (*s_t)[kFlatChunk], double *s_acc,
                                           const double2 *__restrict__ vel,
                                           const double2 *__restrict__ prho, Side &&side)
{
    const NLView<double> &v = Q.v;
    const FlatLists &B = Q.B;
    const int n = S.off[Q.np], a2 = Q.t >> 1, c2 = Q.t & 1;
    const int b0 = a2 < Q.np ? S.off[a2] : 0, b1 = a2 < Q.np ? S.off[a2 + 1] : 0;
    double acc = 0.0;
    side();
    for (int base = 0, at = 0, m; Q.t < kFlatBlock && base < n; base += m) {
        m = Q.chunk(S, base, at);
        Q.pairs(base, m, [&](int p, int64_t i, int j, double F) {
            decltype(auto) I = load_inst<MULTI>(v, i);
            const double2 xi = v.pos[i], vi = vel[i], pi = prho[i];
            const double2 xj = v.pos[j], vj = vel[j], pj = prho[j];
            const double Pij = I.p.m * (pi.x + pj.x);
            s_t[0][p] = Pij * F * (xi.x - xj.x);
            s_t[1][p] = Pij * F * (xi.y - xj.y);
            const double C = B.tm[i] * pj.y * F;
            s_t[2][p] = C * (vi.x - vj.x);
            s_t[3][p] = C * (vi.y - vj.y);
        });
        pair_sync();
        if (Q.t < 2 * kFlatMax) {
            const int k0 = (b0 > base ? b0 : base) - base;
            const int k1 = (b1 < base + m ? b1 : base + m) - base;
            acc = flat_fold(acc, s_t[c2], s_t[2 + c2], k0, k1);
        }
        if (base + m < n) pair_sync();
    }
    if (a2 < Q.np) s_acc[Q.t] = acc;
    __syncthreads();
}

// The force sum of the particle this thread finishes (t < np).
template <bool MULTI>
__device__ __forceinline__ void flat_force(const NLView<double> &v, uint32_t serial, int64_t i,
                                           const double *s_acc, const double2 *__restrict__ vel,
                                           const double2 *__restrict__ prho, const double2 &xi,
                                           const double2 &vi, double &ax, double &ay)
{
    const int t = (int)threadIdx.x;
    if ((serial >> t) & 1u) {
        decltype(auto) I = load_inst<MULTI>(v, i);
        accel_sum<double, false>(v, I, vel, prho, nullptr, i, xi, vi, ax, ay);
    } else {
        ax = s_acc[2 * t];
        ay = s_acc[2 * t + 1];
    }
}

// accel_kernel! + integrate_kernel! (accel_integrate_finish)
template <bool MULTI>
__global__ void __launch_bounds__(kFlatThreads)
    k_accel_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                 const double2 *__restrict__ vel, const double2 *__restrict__ prho,
                 const double *__restrict__ theta, double2 *__restrict__ posOut,
                 double2 *__restrict__ velOut, double2 *__restrict__ aOut,
                 double *__restrict__ alphaOut, uint32_t *__restrict__ flags,
                 const int32_t *__restrict__ perm, double2 *__restrict__ tx,
                 double2 *__restrict__ tv)
{
    pdl_enter();
    __shared__ double s_t[4][kFlatChunk], s_acc[2 * kFlatMax];
    __shared__ SideForce<double> s_f[kFlatMax];
    __shared__ FlatShared S;
    const FlatPass<MULTI> Q(v, B, S);
    flat_accel<MULTI>(Q, S, s_t, s_acc, vel, prho, [&] {
        const int64_t i = Q.aside();
        if (i < 0) return;
        decltype(auto) I = load_inst<MULTI>(v, i);
        const double2 xi = v.pos[i];
        if (tx) {
            const int32_t id = perm[i];
            tx[id] = xi;
            tv[id] = vel[i];
        }
        const SideForce<double> f = side_force<double>(I, xi, theta);
        if (alphaOut) alphaOut[i] = f.al;
        s_f[Q.t - kFlatBlock] = f;
    });
    if (Q.t >= Q.np) return;
    const int64_t i = Q.i0 + Q.t;
    const int b = MULTI ? inst_of(v, i) : 0;
    decltype(auto) I = load_inst<MULTI>(v, i);
    const double2 xi = v.pos[i], vi = vel[i];
    const SideForce<double> f = s_f[Q.t];
    double ax, ay;
    flat_force<MULTI>(v, S.serial, i, s_acc, vel, prho, xi, vi, ax, ay);
    ax += f.gx;
    ay += f.gy;
    if (aOut) aOut[i] = make_double2(ax, ay);
    const double dt = I.p.dt;
    const double v1 = (vi.x + dt * ax) * f.D;
    const double v2 = (vi.y + dt * ay) * f.D;
    const double x1 = xi.x + dt * v1;
    const double x2 = xi.y + dt * v2;
    velOut[i] = make_double2(v1, v2);
    posOut[i] = make_double2(x1, x2);
    if (!(isfinite(x1) && isfinite(x2) && isfinite(v1) && isfinite(v2)))
        atomicOr(flags + b, FLAG_NONFINITE);
}

// Accel recompute + _adj_integrate! + _adj_drag! (drag_adj_finish)
template <bool MULTI>
__global__ void __launch_bounds__(kFlatThreads)
    k_drag_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                const double2 *__restrict__ vel, const double2 *__restrict__ prho,
                const double *__restrict__ theta, const double2 *__restrict__ gX,
                double2 *__restrict__ gV, double2 *__restrict__ abar,
                double *__restrict__ galpha, int *__restrict__ emax, int parity)
{
    pdl_enter();
    __shared__ double s_t[4][kFlatChunk], s_acc[2 * kFlatMax];
    __shared__ SideForce<double> s_f[kFlatMax];
    __shared__ double2 s_gv[kFlatMax];
    __shared__ FlatShared S;
    const FlatPass<MULTI> Q(v, B, S);
    flat_accel<MULTI>(Q, S, s_t, s_acc, vel, prho, [&] {
        const int64_t i = Q.aside();
        if (i < 0) return;
        decltype(auto) I = load_inst<MULTI>(v, i);
        const SideForce<double> f = side_force<double>(I, v.pos[i], theta);
        const double dt = I.p.dt;
        const double2 gx = gX[i];
        double2 gv = gV[i];
        gv.x += dt * gx.x;
        gv.y += dt * gx.y;
        abar[i] = make_double2(dt * f.D * gv.x, dt * f.D * gv.y);
        gV[i] = make_double2(f.D * gv.x, f.D * gv.y);
        s_f[Q.t - kFlatBlock] = f;
        s_gv[Q.t - kFlatBlock] = gv;
    });
    if (Q.t >= 32) return;
    const int64_t i = Q.i0 + Q.t;
    int e = INT_MIN, b = 0;
    if (Q.t < Q.np) {
        b = MULTI ? inst_of(v, i) : 0;
        decltype(auto) I = load_inst<MULTI>(v, i);
        const double2 xi = v.pos[i], vi = vel[i];
        const SideForce<double> f = s_f[Q.t];
        const double2 gv = s_gv[Q.t];
        double ax, ay;
        flat_force<MULTI>(v, S.serial, i, s_acc, vel, prho, xi, vi, ax, ay);
        ax += f.gx;
        ay += f.gy;
        const double dt = I.p.dt;
        const double vx = (vi.x + dt * ax) * f.D;
        const double vy = (vi.y + dt * ay) * f.D;
        const double ga = -dt * f.D * (vx * gv.x + vy * gv.y);
        galpha[i] = ga;
        e = (ga != 0.0 && isfinite(ga)) ? ilogb(ga) + 1 : INT_MIN;
    }
    warp_emax(Q.t < Q.np, b, e, emax, parity, MULTI);
}

// adj_pass1_kernel! + the gXs half of adj_design_kernel! + _axpy2!(gV, gVs)
template <bool MULTI>
__global__ void __launch_bounds__(kFlatThreads)
    k_pass1_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                 const double2 *__restrict__ vel, const double2 *__restrict__ prho,
                 const double *__restrict__ rho, const double *__restrict__ theta,
                 const double2 *__restrict__ abar, const double *__restrict__ galpha,
                 double2 *__restrict__ gXs, double *__restrict__ grho, double2 *__restrict__ gV)
{
    pdl_enter();
    __shared__ double s_t[8][kFlatChunk];
    __shared__ double s_acc[6 * kFlatMax]; // gx gy per particle, then gvx gvy grho S
    __shared__ double s_side[4][kFlatMax]; // wall and design-field terms of gXs
    __shared__ FlatShared S;
    const FlatPass<MULTI> Q(v, B, S);
    const int t = Q.t, np = Q.np;
    if (t < kFlatBlock)
        for (int k = t; k < 6 * kFlatMax; k += kFlatBlock) s_acc[k] = 0.0;
    if (const int64_t i = Q.aside(); i >= 0) {
        decltype(auto) I = load_inst<MULTI>(v, i);
        const double2 x = v.pos[i], ab = abar[i];
        double al, dadx, dady;
        interp_alpha<double>(theta + I.toff, x.x, x.y, I.p, al, dadx, dady);
        const double ga = galpha[i];
        s_side[0][t - kFlatBlock] = ab.x * wall_daccel<double>(x.x, I.p.Lx, I.p.kw);
        s_side[1][t - kFlatBlock] = ab.y * wall_daccel<double>(x.y, I.p.Ly, I.p.kw);
        s_side[2][t - kFlatBlock] = ga * dadx;
        s_side[3][t - kFlatBlock] = ga * dady;
    }
    const int n = S.off[np];
    for (int base = 0, at = 0, m; t < kFlatBlock && base < n; base += m) {
        m = Q.chunk(S, base, at);
        Q.pairs(base, m, [&](int p, int64_t i, int j, double F) {
            decltype(auto) I = load_inst<MULTI>(v, i);
            const double2 xi = v.pos[i], vi = vel[i], pi = prho[i], ab = abar[i];
            const double2 xj = v.pos[j], vj = vel[j], pj = prho[j], abj = abar[j];
            // pass1_pair, with F from the density pass
            const double dx = xi.x - xj.x;
            const double dy = xi.y - xj.y;
            const double r = B.r[Q.bb + base + p];
            const double q = r * I.p.invh;
            const double u = 1.0 - half_of(q);
            const double G = I.p.Gc * u * u;
            const double Pij = I.p.m * (pi.x + pj.x);
            const double Cbase = B.tm[i] * pj.y;
            const double C = Cbase * F;
            const double dax = ab.x - abj.x;
            const double day = ab.y - abj.y;
            const double ad_d = -(dax * dx + day * dy);
            const double ad_v = dax * (vi.x - vj.x) + day * (vi.y - vj.y);
            const double Fbar = Pij * ad_d + Cbase * ad_v;
            const double w = div_rn(Fbar * G * I.p.invh, r);
            s_t[0][p] = Pij * F * dax;
            s_t[1][p] = Pij * F * day;
            s_t[2][p] = w * dx;
            s_t[3][p] = w * dy;
            s_t[4][p] = C * dax;
            s_t[5][p] = C * day;
            s_t[6][p] = -(C * ad_v * pi.y); // subtracted
            s_t[7][p] = F * ad_d;
        });
        pair_sync();
        // gx and gy (two terms a pair) on the first warps, the four sums with one
        // term from the last warp down
        auto range = [&](int a, int &k0, int &k1) {
            k0 = a < np && S.off[a] > base ? S.off[a] - base : 0;
            k1 = a >= np ? 0 : S.off[a + 1] < base + m ? S.off[a + 1] - base : m;
        };
        int k0, k1;
        if (t < 2 * kFlatMax) {
            range(t >> 1, k0, k1);
            s_acc[t] = flat_fold(s_acc[t], s_t[t & 1], s_t[2 + (t & 1)], k0, k1);
        }
        const int c = kFlatBlock - 1 - t;
        range(c >> 2, k0, k1);
        double &x = s_acc[2 * kFlatMax + c];
        x = flat_fold(x, nullptr, s_t[4 + (c & 3)], k0, k1);
        pair_sync();
    }
    __syncthreads();
    if (t >= np) return;
    const int64_t i = Q.i0 + t;
    decltype(auto) I = load_inst<MULTI>(v, i);
    const double2 pi = prho[i];
    double gx = s_acc[2 * t], gy = s_acc[2 * t + 1];
    const double *o = s_acc + 2 * kFlatMax + 4 * t;
    double gvx = o[0], gvy = o[1], grh = o[2], sumS = o[3];
    if ((S.serial >> t) & 1u)
        pass1_sum<double, false>(v, I, i, vel, prho, rho, abar, v.pos[i], vel[i], abar[i], pi, gx,
                                 gy, gvx, gvy, grh, sumS);
    // pass1_finish
    grh += (-2.0 * I.p.m * pi.x * pi.y) * sumS;
    if (I.p.eos == 1)
        grh += I.p.dB * pow_fold<double>(div_rn(rho[i], I.p.rho0), I.p.gam - 1) * I.p.m * pi.y *
               pi.y * sumS;
    else
        grh += I.p.c2 * I.p.m * pi.y * pi.y * sumS;
    gx += s_side[0][t];
    gy += s_side[1][t];
    gXs[i] = make_double2(gx + s_side[2][t], gy + s_side[3][t]);
    grho[i] = grh;
    double2 g = gV[i];
    g.x += gvx;
    g.y += gvy;
    gV[i] = g;
}

// adj_pass2_kernel! + _axpy2!(gX, gXs) + the exact theta write-back
template <bool MULTI>
__global__ void __launch_bounds__(kFlatThreads)
    k_pass2_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                 const double *__restrict__ grho, const double2 *__restrict__ gXs,
                 double2 *__restrict__ gX, const double *__restrict__ galpha,
                 const int *__restrict__ emax, int parity,
                 unsigned long long *__restrict__ thetaAcc, NextState<double> next)
{
    pdl_enter();
    __shared__ double s_t[2][kFlatChunk], s_acc[2 * kFlatMax];
    __shared__ FlatShared S;
    const FlatPass<MULTI> Q(v, B, S);
    const int t = Q.t, np = Q.np;
    if (t >= kFlatBlock) { // the theta write-back and the next tape state
        const int64_t own = Q.aside(), i = own >= 0 ? own : Q.i0;
        if (own >= 0) next.read(i);
        const int b = MULTI ? inst_of(v, i) : 0;
        decltype(auto) I = load_inst<MULTI>(v, i);
        const double2 x = v.pos[i];
        const double ga = galpha[i];
        const int em = emax[2 * b + parity];
        int ci, cj;
        double fx, fy, ax, ay;
        interp_cell<double>(x.x, x.y, I.p, ci, cj, fx, fy, ax, ay);
        theta_add_warp<double>(own >= 0 && ga != 0.0 && em != INT_MIN,
                               I.toff + cj + ci * I.p.ngy, I.p.ngy, theta_scale(em, I.lgN), ga, fx,
                               fy, thetaAcc);
        if (own >= 0) next.write(i);
    }
    const int n = S.off[np], a2 = t >> 1, c2 = t & 1;
    const int b0 = a2 < np ? S.off[a2] : 0, b1 = a2 < np ? S.off[a2 + 1] : 0;
    double acc = 0.0;
    for (int base = 0, at = 0, m; t < kFlatBlock && base < n; base += m) {
        m = Q.chunk(S, base, at);
        Q.pairs(base, m, [&](int p, int64_t i, int j, double F) {
            decltype(auto) I = load_inst<MULTI>(v, i);
            const double2 xi = v.pos[i], xj = v.pos[j];
            const double w = I.p.m * F * (grho[i] + grho[j]);
            s_t[0][p] = w * (xi.x - xj.x);
            s_t[1][p] = w * (xi.y - xj.y);
        });
        pair_sync();
        if (t < 2 * kFlatMax) {
            const int k0 = (b0 > base ? b0 : base) - base;
            const int k1 = (b1 < base + m ? b1 : base + m) - base;
            acc = flat_fold(acc, nullptr, s_t[c2], k0, k1);
        }
        if (base + m < n) pair_sync();
    }
    if (a2 < np) s_acc[t] = acc;
    __syncthreads();
    if (t >= np) return;
    const int64_t i = Q.i0 + t;
    double gx = s_acc[2 * t], gy = s_acc[2 * t + 1];
    if ((S.serial >> t) & 1u) {
        decltype(auto) I = load_inst<MULTI>(v, i);
        pass2_sum<double>(v, I, i, v.pos[i], grho, gx, gy);
    }
    pass2_axpy<double>(i, gx, gy, gXs, gX);
}

} // namespace sphgb
