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
//             8 to 10 FP64 operations a pair fewer (r^2, q, u and F are not formed
//             again; pass 1 needs r itself).
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
// busy), pass 2 69.9 -> 41.2; the solve 5.51 -> 4.22 ms. 2072 particles, lane
// groups -> this: 128 steps 12.0 -> 9.1 ms.
#pragma once

#include "sph_coop.cuh"
#include "sph_window.cuh"

namespace sphgb {

constexpr int kFlatBlock = 128;
constexpr int kFlatMax = 32;    // particles of a block, at most
constexpr int kFlatRow = 64;    // pairs of a particle, at most
constexpr int kFlatChunk = 384; // pairs folded at a time
constexpr int kFlatOff = kFlatMax + 2; // offsets of a block, then its serial mask
constexpr int kFlatSlotBits = 27;

struct FlatLists {
    double *F;      // [block][P * kFlatRow]
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

// Exclusive scan of one int per thread over the block; tot: the sum.
__device__ __forceinline__ int flat_scan(int x, int *s_warp, int &tot)
{
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    int s = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    if (lane == 31) s_warp[warp] = s;
    __syncthreads();
    int before = 0;
    tot = 0;
#pragma unroll
    for (int w = 0; w < kFlatBlock / 32; ++w) {
        before += w < warp ? s_warp[w] : 0;
        tot += s_warp[w];
    }
    __syncthreads();
    return before + s - x;
}

// density_kernel! + eos_kernel!, and the block's dense pairs.
template <bool MULTI>
__global__ void __launch_bounds__(kFlatBlock)
    k_density_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                   double *__restrict__ rho, double2 *__restrict__ prho,
                   const ThetaFlush<double> flush)
{
    pdl_enter();
    if (theta_flush<double>(flush)) return;
    __shared__ double s_r2[kFlatMax * kFlatRow];
    __shared__ int32_t s_lst[kFlatMax][kFlatRow]; // rows of spilled particles
    __shared__ uint32_t s_wd[kFlatMax][6];
    __shared__ int s_bs[kFlatMax][3], s_pre[kFlatMax][6];
    __shared__ int s_off[kFlatMax + 1], s_cnt[kFlatMax], s_in[kFlatMax];
    __shared__ uint8_t s_own[kFlatMax * kFlatRow];
    __shared__ int s_warp[kFlatBlock / 32];
    __shared__ uint32_t s_spill, s_serial;
    const int t = (int)threadIdx.x, P = B.P;
    const int64_t i0 = (int64_t)blockIdx.x * P;
    const int np = v.N - i0 < P ? (int)(v.N - i0) : P;
    if (t == 0) s_spill = s_serial = 0u;
    __syncthreads();
    if (t < np) {
        const int64_t i = i0 + t;
        decltype(auto) I = load_inst<MULTI>(v, i);
        const uint32_t cc = v.center[i];
        int n = 0;
        if (cc >> 31) {
            atomicOr(I.maxnb > kFlatRow ? &s_serial : &s_spill, 1u << t);
        } else {
            const int cx = (int)(cc & 0xffffu), cy = (int)((cc >> 16) & 0x7fffu);
            const int jx0 = cx - 1 > 1 ? cx - 1 : 1;
            const int row0 = I.coff + (jx0 - 1) + (cy - 2) * I.nx; // cell (jx0, cy - 1)
            uint32_t w[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) w[q] = v.masks[(int64_t)q * v.N + i];
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
                atomicOr(&s_serial, 1u << t);
                n = 0;
            }
        }
        s_cnt[t] = n;
    }
    if (t < kFlatMax) s_in[t] = 0;
    __syncthreads();
    const uint32_t spill = s_spill, serial = s_serial;
    if (spill) { // list their rows, a warp per particle
        const Group<32> g;
        for (int a = t >> 5; a < np; a += kFlatBlock / 32)
            if ((spill >> a) & 1u) {
                const int64_t i = i0 + a;
                decltype(auto) I = load_inst<MULTI>(v, i);
                const int n = spill_list<double, 32>(g, v, I, i, v.center[i], s_lst[a]);
                if ((t & 31) == 0) s_cnt[a] = n;
            }
        __syncthreads();
    }
    int tot;
    const int pre = flat_scan(t < np ? s_cnt[t] : 0, s_warp, tot);
    if (t <= np) s_off[t] = pre;
    __syncthreads();

    const int64_t bb = (int64_t)blockIdx.x * P * kFlatRow;
    int D = 0; // dense pairs so far
    for (int base = 0; base < tot; base += kFlatChunk) {
        constexpr int U = kFlatChunk / kFlatBlock;
        double r2v[U];
        uint32_t pj[U];
        int cnt = 0, a = 0;
        const int p0 = base + U * t;
        if (p0 < tot) { // the particle that owns pair p0
            int hi = np - 1;
            while (a < hi) {
                const int mid = (a + hi + 1) >> 1;
                if (s_off[mid] <= p0) a = mid;
                else hi = mid - 1;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int p = p0 + u;
            pj[u] = 0xffffffffu;
            if (p < tot) {
                while (p >= s_off[a + 1]) ++a;
                const int k = p - s_off[a];
                int j;
                if ((spill >> a) & 1u) {
                    j = s_lst[a][k];
                } else {
                    int w = 0;
#pragma unroll
                    for (int q = 1; q < 6; ++q) w = k >= s_pre[a][q] ? q : w;
                    j = s_bs[a][w >> 1] + 32 * (w & 1) + select_bit(s_wd[a][w], k - s_pre[a][w]);
                }
                decltype(auto) I = load_inst<MULTI>(v, i0 + a);
                const double2 xi = v.pos[i0 + a], xj = v.pos[j];
                const double dx = xi.x - xj.x;
                const double dy = xi.y - xj.y;
                r2v[u] = dx * dx + dy * dy;
                if (lt_nonneg(r2v[u], I.p.r2max)) {
                    pj[u] = (uint32_t)a << kFlatSlotBits | (uint32_t)j;
                    ++cnt;
                }
            }
        }
        int n;
        int pos = D + flat_scan(cnt, s_warp, n);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (pj[u] != 0xffffffffu) {
                const int own = (int)(pj[u] >> kFlatSlotBits);
                s_r2[pos] = r2v[u];
                s_own[pos] = (uint8_t)own;
                B.pair[bb + pos] = pj[u];
                atomicAdd(&s_in[own], 1);
                ++pos;
            }
        D += n;
    }
    __syncthreads();
    for (int d = t; d < D; d += kFlatBlock) {
        decltype(auto) I = load_inst<MULTI>(v, i0 + s_own[d]);
        const double q = pair_sqrt(s_r2[d]) * I.p.invh;
        const double u = 1.0 - half_of(q);
        const double u2 = u * u;
        B.F[bb + d] = I.p.Fc * u * u * u;
        s_r2[d] = I.p.m * (I.p.A * u2 * u2 * (twice_of(q) + 1.0));
    }
    int all;
    const int o = flat_scan(t < np ? s_in[t] : 0, s_warp, all); // ends with a barrier
    if (t <= np) B.off[(int64_t)blockIdx.x * kFlatOff + t] = o;
    if (t == 0) B.off[(int64_t)blockIdx.x * kFlatOff + kFlatOff - 1] = (int)serial;
    if (t >= np) return;
    const int64_t i = i0 + t;
    if ((serial >> t) & 1u) {
        density_walk<double, MULTI, false>(v, i, rho, prho, nullptr);
        return;
    }
    double acc = 0.0;
    const int e = o + s_in[t];
#pragma unroll 4
    for (int k = o; k < e; ++k) acc += s_r2[k];
    decltype(auto) I = load_inst<MULTI>(v, i);
    density_finish<double>(I, i, acc, rho, prho);
}

// The offsets of a block's particles in its dense pairs; s_off[np] pairs.
__device__ __forceinline__ void flat_offsets(const FlatLists &B, int np, int *s_off,
                                             uint32_t *s_serial)
{
    const int t = (int)threadIdx.x;
    const int32_t *o = B.off + (int64_t)blockIdx.x * kFlatOff;
    if (t <= np) s_off[t] = o[t];
    if (t == 0) *s_serial = (uint32_t)o[kFlatOff - 1];
}

// One lane per running sum: chain c adds the terms of its particle's pairs that
// this chunk holds. sub (may be NULL): a term subtracted before each added one.
__device__ __forceinline__ double flat_fold(double acc, const double *sub, const double *add,
                                            int k0, int k1)
{
    if (sub) {
#pragma unroll 4
        for (int k = k0; k < k1; ++k) {
            acc -= sub[k];
            acc += add[k];
        }
    } else {
#pragma unroll 4
        for (int k = k0; k < k1; ++k) acc += add[k];
    }
    return acc;
}

// Pressure + Morris viscosity of the block's particles (accel_pair): s_acc[2 a],
// s_acc[2 a + 1]. All threads call it; ends with a barrier.
template <bool MULTI>
__device__ __forceinline__ void flat_accel(const NLView<double> &v, const FlatLists &B, int np,
                                           const int *s_off, double (*s_t)[kFlatChunk],
                                           double *s_acc, const double2 *__restrict__ vel,
                                           const double2 *__restrict__ prho)
{
    const int t = (int)threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * B.P, bb = i0 * kFlatRow;
    const int n = s_off[np], a2 = t >> 1, c2 = t & 1;
    const int b0 = a2 < np ? s_off[a2] : 0, b1 = a2 < np ? s_off[a2 + 1] : 0;
    double acc = 0.0;
    for (int base = 0; base < n; base += kFlatChunk) {
        const int m = n - base < kFlatChunk ? n - base : kFlatChunk;
        for (int p = t; p < m; p += kFlatBlock) {
            const uint32_t e = B.pair[bb + base + p];
            const double F = B.F[bb + base + p];
            const int64_t i = i0 + (e >> kFlatSlotBits);
            const int j = (int)(e & ((1u << kFlatSlotBits) - 1u));
            decltype(auto) I = load_inst<MULTI>(v, i);
            const double2 xi = v.pos[i], vi = vel[i], pi = prho[i];
            const double2 xj = v.pos[j], vj = vel[j], pj = prho[j];
            const double Pij = I.p.m * (pi.x + pj.x);
            s_t[0][p] = Pij * F * (xi.x - xj.x);
            s_t[1][p] = Pij * F * (xi.y - xj.y);
            const double C = I.p.twomumass * pi.y * pj.y * F;
            s_t[2][p] = C * (vi.x - vj.x);
            s_t[3][p] = C * (vi.y - vj.y);
        }
        __syncthreads();
        if (a2 < np) {
            const int k0 = (b0 > base ? b0 : base) - base;
            const int k1 = (b1 < base + m ? b1 : base + m) - base;
            acc = flat_fold(acc, s_t[c2], s_t[2 + c2], k0, k1);
        }
        __syncthreads();
    }
    if (a2 < np) s_acc[t] = acc;
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

// accel_kernel! + integrate_kernel!
template <bool MULTI>
__global__ void __launch_bounds__(kFlatBlock)
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
    __shared__ int s_off[kFlatMax + 1];
    __shared__ uint32_t s_serial;
    const int64_t i0 = (int64_t)blockIdx.x * B.P;
    const int np = v.N - i0 < B.P ? (int)(v.N - i0) : B.P;
    flat_offsets(B, np, s_off, &s_serial);
    __syncthreads();
    flat_accel<MULTI>(v, B, np, s_off, s_t, s_acc, vel, prho);
    const int t = (int)threadIdx.x;
    if (t >= np) return;
    const int64_t i = i0 + t;
    const int b = MULTI ? inst_of(v, i) : 0;
    decltype(auto) I = load_inst<MULTI>(v, i);
    const double2 xi = v.pos[i], vi = vel[i];
    double ax, ay;
    flat_force<MULTI>(v, s_serial, i, s_acc, vel, prho, xi, vi, ax, ay);
    accel_integrate_finish<double>(I, b, i, xi, vi, ax, ay, theta, posOut, velOut, aOut, alphaOut,
                                   flags, perm, tx, tv);
}

// Accel recompute + _adj_integrate! + _adj_drag!
template <bool MULTI>
__global__ void __launch_bounds__(kFlatBlock)
    k_drag_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                const double2 *__restrict__ vel, const double2 *__restrict__ prho,
                const double *__restrict__ theta, const double2 *__restrict__ gX,
                double2 *__restrict__ gV, double2 *__restrict__ abar,
                double *__restrict__ galpha, int *__restrict__ emax, int parity)
{
    pdl_enter();
    __shared__ double s_t[4][kFlatChunk], s_acc[2 * kFlatMax];
    __shared__ int s_off[kFlatMax + 1];
    __shared__ uint32_t s_serial;
    const int64_t i0 = (int64_t)blockIdx.x * B.P;
    const int np = v.N - i0 < B.P ? (int)(v.N - i0) : B.P;
    flat_offsets(B, np, s_off, &s_serial);
    __syncthreads();
    flat_accel<MULTI>(v, B, np, s_off, s_t, s_acc, vel, prho);
    const int t = (int)threadIdx.x;
    if (t >= 32) return;
    const int64_t i = i0 + t;
    int e = INT_MIN, b = 0;
    if (t < np) {
        b = MULTI ? inst_of(v, i) : 0;
        decltype(auto) I = load_inst<MULTI>(v, i);
        const double2 xi = v.pos[i], vi = vel[i];
        double ax, ay;
        flat_force<MULTI>(v, s_serial, i, s_acc, vel, prho, xi, vi, ax, ay);
        e = drag_adj_finish<double>(I, i, xi, vi, ax, ay, theta, gX, gV, abar, galpha);
    }
    warp_emax(t < np, b, e, emax, parity, MULTI);
}

// adj_pass1_kernel! + the gXs half of adj_design_kernel! + _axpy2!(gV, gVs)
template <bool MULTI>
__global__ void __launch_bounds__(kFlatBlock)
    k_pass1_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                 const double2 *__restrict__ vel, const double2 *__restrict__ prho,
                 const double *__restrict__ rho, const double *__restrict__ theta,
                 const double2 *__restrict__ abar, const double *__restrict__ galpha,
                 double2 *__restrict__ gXs, double *__restrict__ grho, double2 *__restrict__ gV)
{
    pdl_enter();
    __shared__ double s_t[8][kFlatChunk];
    __shared__ double s_acc[6 * kFlatMax]; // gx gy per particle, then gvx gvy grho S
    __shared__ int s_off[kFlatMax + 1];
    __shared__ uint32_t s_serial;
    const int t = (int)threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * B.P, bb = i0 * kFlatRow;
    const int np = v.N - i0 < B.P ? (int)(v.N - i0) : B.P;
    flat_offsets(B, np, s_off, &s_serial);
    for (int k = t; k < 6 * kFlatMax; k += kFlatBlock) s_acc[k] = 0.0;
    __syncthreads();
    const int n = s_off[np];
    for (int base = 0; base < n; base += kFlatChunk) {
        const int m = n - base < kFlatChunk ? n - base : kFlatChunk;
        for (int p = t; p < m; p += kFlatBlock) {
            const uint32_t e = B.pair[bb + base + p];
            const double F = B.F[bb + base + p];
            const int64_t i = i0 + (e >> kFlatSlotBits);
            const int j = (int)(e & ((1u << kFlatSlotBits) - 1u));
            decltype(auto) I = load_inst<MULTI>(v, i);
            const double2 xi = v.pos[i], vi = vel[i], pi = prho[i], ab = abar[i];
            const double2 xj = v.pos[j], vj = vel[j], pj = prho[j], abj = abar[j];
            // pass1_pair, with F from the density pass
            const double dx = xi.x - xj.x;
            const double dy = xi.y - xj.y;
            const double r = pair_sqrt(dx * dx + dy * dy);
            const double q = r * I.p.invh;
            const double u = 1.0 - half_of(q);
            const double G = I.p.Gc * u * u;
            const double Pij = I.p.m * (pi.x + pj.x);
            const double Cbase = I.p.twomumass * pi.y * pj.y;
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
        }
        __syncthreads();
        // gx and gy (two terms a pair) on the first warps, then the four sums
        // with one
        for (int c = t; c < 2 * np; c += kFlatBlock) {
            const int a = c >> 1, k0 = s_off[a] > base ? s_off[a] - base : 0;
            const int k1 = s_off[a + 1] < base + m ? s_off[a + 1] - base : m;
            s_acc[c] = flat_fold(s_acc[c], s_t[c & 1], s_t[2 + (c & 1)], k0, k1);
        }
        for (int c = kFlatBlock - 1 - t; c < 4 * np; c += kFlatBlock) {
            const int a = c >> 2, k0 = s_off[a] > base ? s_off[a] - base : 0;
            const int k1 = s_off[a + 1] < base + m ? s_off[a + 1] - base : m;
            double &x = s_acc[2 * kFlatMax + c];
            x = flat_fold(x, nullptr, s_t[4 + (c & 3)], k0, k1);
        }
        __syncthreads();
    }
    if (t >= np) return;
    const int64_t i = i0 + t;
    decltype(auto) I = load_inst<MULTI>(v, i);
    const double2 xi = v.pos[i], ab = abar[i], pi = prho[i];
    double gx = s_acc[2 * t], gy = s_acc[2 * t + 1];
    const double *o = s_acc + 2 * kFlatMax + 4 * t;
    double gvx = o[0], gvy = o[1], grh = o[2], sumS = o[3];
    if ((s_serial >> t) & 1u)
        pass1_sum<double, false>(v, I, i, vel, prho, rho, abar, xi, vel[i], ab, pi, gx, gy, gvx,
                                 gvy, grh, sumS);
    const double rhoi = I.p.eos == 1 ? rho[i] : 0.0;
    pass1_finish<double>(I, i, xi, ab, pi, rhoi, gx, gy, gvx, gvy, grh, sumS, theta, galpha, gXs,
                         grho, gV);
}

// adj_pass2_kernel! + _axpy2!(gX, gXs) + the exact theta write-back
template <bool MULTI>
__global__ void __launch_bounds__(kFlatBlock)
    k_pass2_flat(const __grid_constant__ NLView<double> v, const FlatLists B,
                 const double *__restrict__ grho, const double2 *__restrict__ gXs,
                 double2 *__restrict__ gX, const double *__restrict__ galpha,
                 const int *__restrict__ emax, int parity,
                 unsigned long long *__restrict__ thetaAcc, NextState<double> next)
{
    pdl_enter();
    __shared__ double s_t[2][kFlatChunk], s_acc[2 * kFlatMax];
    __shared__ int s_off[kFlatMax + 1];
    __shared__ uint32_t s_serial;
    const int t = (int)threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * B.P, bb = i0 * kFlatRow;
    const int np = v.N - i0 < B.P ? (int)(v.N - i0) : B.P;
    flat_offsets(B, np, s_off, &s_serial);
    const int nt = kFlatBlock - 1 - t; // the last threads load the next state
    if (nt < np) next.read(i0 + nt);
    __syncthreads();
    const int n = s_off[np], a2 = t >> 1, c2 = t & 1;
    const int b0 = a2 < np ? s_off[a2] : 0, b1 = a2 < np ? s_off[a2 + 1] : 0;
    double acc = 0.0;
    for (int base = 0; base < n; base += kFlatChunk) {
        const int m = n - base < kFlatChunk ? n - base : kFlatChunk;
        for (int p = t; p < m; p += kFlatBlock) {
            const uint32_t e = B.pair[bb + base + p];
            const double F = B.F[bb + base + p];
            const int64_t i = i0 + (e >> kFlatSlotBits);
            const int j = (int)(e & ((1u << kFlatSlotBits) - 1u));
            decltype(auto) I = load_inst<MULTI>(v, i);
            const double2 xi = v.pos[i], xj = v.pos[j];
            const double w = I.p.m * F * (grho[i] + grho[j]);
            s_t[0][p] = w * (xi.x - xj.x);
            s_t[1][p] = w * (xi.y - xj.y);
        }
        __syncthreads();
        if (a2 < np) {
            const int k0 = (b0 > base ? b0 : base) - base;
            const int k1 = (b1 < base + m ? b1 : base + m) - base;
            acc = flat_fold(acc, nullptr, s_t[c2], k0, k1);
        }
        __syncthreads();
    }
    if (a2 < np) s_acc[t] = acc;
    if (nt < np) next.write(i0 + nt);
    __syncthreads();
    if (t >= 32) return;
    const bool live = t < np;
    const int64_t i = i0 + (live ? t : np - 1);
    const int b = MULTI ? inst_of(v, i) : 0;
    decltype(auto) I = load_inst<MULTI>(v, i);
    const double2 xi = v.pos[i];
    double gx = live ? s_acc[2 * t] : 0.0, gy = live ? s_acc[2 * t + 1] : 0.0;
    if (live && ((s_serial >> t) & 1u)) pass2_sum<double>(v, I, i, xi, grho, gx, gy);
    pass2_finish_warp<double>(live, I, b, i, xi, gx, gy, gXs, gX, galpha, emax, parity, thetaAcc);
}

} // namespace sphgb
