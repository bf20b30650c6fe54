// Row-marching forward step for displacement-free SH and P-SV batches.
//
// Same arithmetic per cell as the tiled step kernels of step.cu (and so as
// the reference's div_sy / div_sxz, stf_dsy / stf_dsxz, add_vy / add_vxz,
// div_vy / div_vxz, add_sy / add_sxz and save_obs, solver.py:54-156), with a
// layout that keeps the instruction count per cell low enough for the step to
// be bound by HBM rather than by issue:
//
//   * A CTA spans the whole z extent of the grid -- thread t owns the four
//     columns 4t .. 4t+3 (up to 1024 columns) -- and marches down a
//     contiguous range of x rows of one shot.  Every shared-memory access
//     and every store is a 16-byte vector for four cells; the z neighbours
//     come from one 8- and one 4-byte load beside it.  The 4th-order x
//     derivatives of the stress come from register windows of five rows, and
//     the arithmetic is packed two cells to an instruction (fma.f32x2 and the
//     like; each cell's operations and roundings are the scalar kernels').
//   * Two rows per block barrier: the new velocity of rows r, r+1 goes to a
//     ring of six rows in shared memory (only rows r-2, r-1 are read across
//     threads, for D+z, so a row may be overwritten one iteration after its
//     own column's last use); after the barrier the stress of rows r-2, r-1
//     follows.  Rows away from a range's ends, the grid's first and last rows
//     and any source or receiver run a version without a branch, which gives
//     the compiler one long block to schedule.
//   * Rows of the state (stress, velocity) stream into a ring of N row slots
//     in shared memory with untiled bulk copies (cp.async.bulk, one per field
//     and row, each issued by its own lane of the last warp, completion on an
//     mbarrier per slot, bounded waits by every warp for itself).  The model,
//     shared by the shots and resident in L2, is read with 16-byte loads one
//     iteration ahead, outside the branches: a load inside one is waited for
//     where the branches join.
//   * What bounds it (P-SV 512 x 512, 32 shots): latency with 12 warps per SM
//     (issue 45 %, 326 MB of DRAM traffic at 53 % of the device's nominal
//     throughput), not the 336 MB that a step has to move, the state's 40 B
//     per cell (51 us at the measured copy rate; the shots share the model,
//     which L2 holds).  One row per barrier, scalar arithmetic and one thread
//     issuing all copies: 88.7 us and 52.1 M warp instructions per step; this:
//     69.7 us, 34 M.  1021 x 511, 64 shots: 284 -> 245 us (1.34 GB: 204 us at
//     the copy rate).  SH 512 x 512, 32 shots: 56 -> 41 us.  256 x 256, one SH
//     shot: 11.2 -> 5.6 us, where the serial searches of the receiver list
//     by one thread were most of the step (now a warp tests 32 places at once,
//     and before the previous step is waited for).
//   * The rows of all shots form one sequence, split evenly over a grid of
//     resident CTAs (one pass, no tail wave); a CTA whose range starts in
//     the middle of a shot recomputes the velocity of the row above its range
//     and of the two below it (the D+x stencil needs them).
//   * No displacement field: the displacement only feeds the receivers, so
//     the kernel records the new velocity at the receivers and
//     displacement_traces_kernel turns each trace into the running sum
//     u(it) = u(it-1) + v(it) dt afterwards -- the same float operations in
//     the same order as the displacement update of add_vy / add_vxz
//     (solver.py:95-109), so the traces are bit-identical.
//   * Sources and receivers are visited in cell order: the injection entries
//     of a shot must be sorted by cell (entries at one cell keep their order,
//     so the per-cell sums are unchanged) and rec_order lists the receivers
//     by cell.  Each CTA stages the points of its rows in shared-memory
//     windows and walks them with the march.
#include <cooperative_groups.h>

#include <atomic>
#include <cstdio>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "stencil.cuh"

namespace cg = cooperative_groups;

namespace fwi {

// Status word of the row-marching kernels (a bounded wait gave up).
__device__ int g_march_status = 0;

int march_device_status(int clear, int *status) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_march_status, sizeof(int)) != cudaSuccess)
        return set_error(FWI_ECUDA, "fwi_device_status: reading the row-marching kernels' status failed");
    if (clear && v) {
        const int z = 0;
        if (cudaMemcpyToSymbol(g_march_status, &z, sizeof(int)) != cudaSuccess)
            return set_error(FWI_ECUDA, "fwi_device_status: clearing the row-marching kernels' status failed");
    }
    *status = v;
    return 0;
}

constexpr int kPts = 128;        // points (injection entries, receivers) staged per window
constexpr int kMaxPitch = 1024;  // row length (floats) a CTA can span: 256 threads of 4 columns
constexpr int kVRing = 6;        // rows of the new-velocity ring (r-4 .. r+1)

struct MarchArgs {
    int nx, nz, pitch, nt, it, nrec;
    int rl;                 // shared-memory row length (floats)
    int nslots;             // row slots of the staging ring
    long long rows_total;   // nshots * nx
    float cx1, cx2, cz1, cz2, dt;
    const float *sig_in[3];
    float *sig_out[3];
    const float *vel_in[2];
    float *vel_out[2];
    const float *buo, *bound;
    const float *ip[2];     // SH: mu | P-SV: lam, mu
    const int *inj_ptr, *inj_cell, *inj_row;
    const float *stf[2];    // injected components in slot order
    const int *rec_cell, *rec_order;
    float *obs[2];          // per velocity component, NULL skips
    float *seg_e[3];        // per-step strain store of this step (slot-offset), or NULL
    float *seg_ds[2];       // per-step divergence store, or NULL
};

// Shared-memory layout, in floats: ring [nslots][NF][rl], velocity ring
// [kVRing][NV][rl], injection window (cells, NINJ value rows), receiver
// window (cells, ids), two double-buffered cursors, then the mbarriers
// (8-byte aligned).
struct MarchLayout {
    int vring, icell, ival, rcell, rid, cur, bar;
    size_t bytes;
};

__host__ __device__ inline MarchLayout march_layout(int nf, int nv, int ninj, int rl, int nslots) {
    MarchLayout L;
    L.vring = nslots * nf * rl;
    L.icell = L.vring + kVRing * nv * rl;
    L.ival = L.icell + kPts;
    L.rcell = L.ival + ninj * kPts;
    L.rid = L.rcell + kPts;
    L.cur = L.rid + kPts;  // two double-buffered cursors (16 ints)
    L.bar = (L.cur + 16 + 1) / 2 * 2;
    L.bytes = sizeof(float) * (size_t)L.bar + 8 * (size_t)nslots;
    return L;
}

// First index in [lo, hi) whose key is >= v (keys non-decreasing); key(i) =
// cell[perm ? perm[i] : i].  Warp-wide: every round tests 32 positions at
// once, so a list of n points takes log33(n) rounds of dependent loads.
__device__ __forceinline__ int warp_lower_bound(const int *cell, const int *perm, int lo, int hi, int v) {
    const int lane = threadIdx.x & 31;
    while (hi - lo > 0) {
        const long long n = hi - lo;
        const int q = lo + (int)(n * (lane + 1) / 33);  // non-decreasing in lane, in [lo, hi)
        const bool below = cell[perm ? perm[q] : q] < v;
        const int k = __popc(__ballot_sync(0xffffffffu, below));  // lanes 0 .. k-1 are below
        const int nlo = k > 0 ? lo + (int)(n * k / 33) + 1 : lo;  // past the last position below
        hi = k < 32 ? lo + (int)(n * (k + 1) / 33) : hi;          // at the first position not below
        lo = nlo;
    }
    return lo;
}

// The same by one thread.
__device__ __forceinline__ int thread_lower_bound(const int *cell, const int *perm, int lo, int hi, int v) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cell[perm ? perm[mid] : mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// A window of consecutive points [w0, w0+wn) of the range [p, end) staged in
// shared memory; p is the next point to visit.  Kept in shared memory; the
// march holds only the cell of the next point in a register and reads the
// cursor on the rows that have points.  Every thread sees the same values,
// so branches on them are block-uniform.
struct Cursor {
    int p, end, w0, wn;
};
constexpr int kNone = 0x7fffffff;  // "no further point"

// Four adjacent columns as two register pairs: the packed FP32 instructions
// (one issue slot for two cells) take them as they are loaded.
struct Q4 {
    float2 a, b;
};
__device__ __forceinline__ Q4 ld4(const float *p) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    return Q4{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ Q4 ldg4(const float *p) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
    return Q4{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ void st4(float *p, const Q4 &q) {
    *reinterpret_cast<float4 *>(p) = make_float4(q.a.x, q.a.y, q.b.x, q.b.y);
}
__device__ __forceinline__ Q4 zero4() { return Q4{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
// the four values with those whose mask is off set to zero
__device__ __forceinline__ Q4 keep4(const Q4 &q, const bool (&m)[4]) {
    return Q4{make_float2(m[0] ? q.a.x : 0.f, m[1] ? q.a.y : 0.f), make_float2(m[2] ? q.b.x : 0.f, m[3] ? q.b.y : 0.f)};
}
__device__ __forceinline__ float2 bc2(float x) { return make_float2(x, x); }

// Finite difference c1 (a - b) - c2 (c - d) of two cells: two differences, the
// second product, one fused multiply-add -- the operations (and roundings)
// the scalar kernels' expressions compile to.
struct Coef {
    float2 c1, n2;  // c1, -c2
};
__device__ __forceinline__ float2 fd2(const Coef &k, float2 a, float2 b, float2 c, float2 d) {
    const float2 m1 = make_float2(-1.f, -1.f);
    return __ffma2_rn(k.c1, __ffma2_rn(b, m1, a), __fmul2_rn(k.n2, __ffma2_rn(d, m1, c)));
}
__device__ __forceinline__ Q4 fdx(const Coef &k, const Q4 &a, const Q4 &b, const Q4 &c, const Q4 &d) {
    return Q4{fd2(k, a.a, b.a, c.a, d.a), fd2(k, a.b, b.b, c.b, d.b)};
}
// D-z of a row at this thread's columns: taps j, j-1, j+1, j-2 around the
// centre values c; s points at the row in shared memory
__device__ __forceinline__ Q4 dzm4(const Coef &k, const float *s, const Q4 &c) {
    const float2 l = *reinterpret_cast<const float2 *>(s - 2);
    const float r = s[4];
    const float2 m0 = make_float2(l.y, c.a.x), m1 = make_float2(c.a.y, c.b.x), m2 = make_float2(c.b.y, r);
    return Q4{fd2(k, c.a, m0, m1, l), fd2(k, c.b, m1, m2, c.a)};
}
// D+z: taps j+1, j, j+2, j-1
__device__ __forceinline__ Q4 dzp4(const Coef &k, const float *s, const Q4 &c) {
    const float l = s[-1];
    const float2 r = *reinterpret_cast<const float2 *>(s + 4);
    const float2 m0 = make_float2(l, c.a.x), m1 = make_float2(c.a.y, c.b.x), m2 = make_float2(c.b.y, r.x);
    return Q4{fd2(k, m1, c.a, c.b, m0), fd2(k, m2, c.b, r, m1)};
}
__device__ __forceinline__ Q4 add4(const Q4 &x, const Q4 &y) { return Q4{__fadd2_rn(x.a, y.a), __fadd2_rn(x.b, y.b)}; }
__device__ __forceinline__ Q4 mul4(const Q4 &x, const Q4 &y) { return Q4{__fmul2_rn(x.a, y.a), __fmul2_rn(x.b, y.b)}; }
__device__ __forceinline__ Q4 fma4(const Q4 &x, const Q4 &y, const Q4 &z) {
    return Q4{__ffma2_rn(x.a, y.a, z.a), __ffma2_rn(x.b, y.b, z.b)};
}
__device__ __forceinline__ float &elem(Q4 &q, int e) { return e == 0 ? q.a.x : e == 1 ? q.a.y : e == 2 ? q.b.x : q.b.y; }

template <int MODE, int WIDE, bool SEG>
__global__ void __launch_bounds__(WIDE ? 256 : 128, MODE == FWI_SH ? (WIDE ? 2 : 4) : (WIDE ? 1 : 3)) march_kernel(const __grid_constant__ MarchArgs a) {
    using F = Fields<MODE>;
    constexpr int NS = F::NS, NV = F::NV, NF = NS + NV, NINJ = F::NINJ;
    // stress fields with an x register window (D-x) and the one without
    constexpr int FX0 = 0, FX1 = MODE == FWI_SH ? 0 : 2, FZ = 1;
    constexpr int NW = MODE == FWI_SH ? 1 : 2;
    extern __shared__ __align__(128) float smem[];
    const int RL = a.rl, N = a.nslots;
    const MarchLayout L = march_layout(NF, NV, NINJ, RL, N);
    int *const i_cell = reinterpret_cast<int *>(smem + L.icell);
    float *const i_val = smem + L.ival;
    int *const r_cell = reinterpret_cast<int *>(smem + L.rcell);
    int *const r_id = reinterpret_cast<int *>(smem + L.rid);
    // cursors [list][buffer]: list 0 injection, 1 receivers; the buffer in use flips at every store
    Cursor *const cur_s = reinterpret_cast<Cursor *>(smem + L.cur);
    uint64_t *const full = reinterpret_cast<uint64_t *>(smem + L.bar);

    const int tid = threadIdx.x, j0 = 4 * tid, lane = tid & 31, nwarps = blockDim.x >> 5, warp = tid >> 5;
    const int nx = a.nx, nz = a.nz, pitch = a.pitch, nt = a.nt, it = a.it;
    const bool tin = j0 < pitch;  // this thread's four columns lie in the rows
    const Coef kx{bc2(a.cx1), bc2(-a.cx2)}, kz{bc2(a.cz1), bc2(-a.cz2)};
    const Q4 dt4{bc2(a.dt), bc2(a.dt)};
    const uint32_t row_bytes = 4u * (uint32_t)pitch;
    // row buffers start 4 floats into their slot so that columns -4 .. rl-5 are addressable
    float *const ring0 = smem + 4 + j0;
    const int slot_len = NF * RL;

    grid_dep_trigger();
    if (tid == 0) {
        for (int i = 0; i < N; i++) mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // the field whose rows this lane of the issuing warp streams in, one bulk copy per field and row
    const bool issuer = warp == nwarps - 1 && lane < NF;
    const float *my_field = nullptr;
#pragma unroll
    for (int f = 0; f < NF; f++)
        if (lane == f) my_field = f < NS ? a.sig_in[f] : a.vel_in[f < NS ? 0 : f - NS];

    // issuing warp, lanes 0 .. NF-1: row q of the shot at soff into ring slot `slot`
    auto issue = [&](long long soff, int q, int slot) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        if (lane == 0) mbar_expect_tx(&full[slot], NF * row_bytes);
        bulk_load(smem + slot * slot_len + lane * RL + 4, my_field + soff + (long long)q * pitch, row_bytes, &full[slot]);
    };
    // per-column masks, fixed for the whole march: D-z (2 <= j < nz-2),
    // D+z (1 <= j < nz-2) and "inside the grid" (j < nz)
    bool zm[4], zp[4], zin[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int c = j0 + e;
        zm[e] = c >= 2 && c < nz - 2;
        zp[e] = c >= 1 && c < nz - 2;
        zin[e] = c < nz;
    }
    // warps without a masked column (all but those at the z edges) skip the masks
    const bool zedge = __any_sync(0xffffffffu, !(j0 >= 2 && j0 + 3 < nz - 2));

    const bool rec_on = a.rec_order && a.nrec > 0 && (a.obs[0] || (NV > 1 && a.obs[1]));
    const bool inj_on = a.inj_ptr != nullptr;
    const int R = (int)a.rows_total, G = gridDim.x;
    int Lrow = (int)((long long)R * blockIdx.x / G);
    const int Lend = (int)((long long)R * (blockIdx.x + 1) / G);
    int islot = 0;          // ring slot of the next row to issue
    int wslot = 0;          // ring slot of the next row to wait for
    uint32_t wphase = 0;    // and the parity of its barrier

    // wait for the next row of the ring (every warp for itself: a row that has
    // landed costs one test, and no block barrier has to follow)
    auto wait_next = [&]() -> bool {
        const bool ok = mbar_try_wait(&full[wslot], wphase) || mbar_wait(&full[wslot], wphase);
        if (++wslot == N) {
            wslot = 0;
            wphase ^= 1;
        }
        return ok;
    };
    // a wait gave up: record it and let the copies still in flight land
    auto give_up = [&] {
        if (tid == 0) atomicExch(&g_march_status, 1);
        for (int k = 0; k < N; k++) wait_next();
    };

    // stage the window of points starting at c.p (block-wide: every thread
    // calls it with the same cursor, which it updates in place)
    auto load_inj = [&](Cursor &c) {
        __syncthreads();
        const int n = min(kPts, c.end - c.p);
        for (int k = tid; k < n; k += blockDim.x) {
            const int e = c.p + k;
            i_cell[k] = a.inj_cell[e];
            const long long src = (long long)a.inj_row[e] * nt + it;
#pragma unroll
            for (int q = 0; q < NINJ; q++) i_val[q * kPts + k] = a.stf[q][src];
        }
        c.w0 = c.p;
        c.wn = n;
        __syncthreads();
    };
    auto load_rec = [&](Cursor &c) {
        __syncthreads();
        const int n = min(kPts, c.end - c.p);
        for (int k = tid; k < n; k += blockDim.x) {
            const int r = a.rec_order[c.p + k];
            r_id[k] = r;
            r_cell[k] = a.rec_cell[r];
        }
        c.w0 = c.p;
        c.wn = n;
        __syncthreads();
    };
    // after the points of a row: store the cursor into the other buffer of
    // its list (slow threads may still read the one in use) and return the
    // cell of the next point, or kNone.  Every thread holds the same cursor;
    // the barrier orders the store before the next use.
    auto park = [&](Cursor &c, int which, int &buf, bool inj) -> int {
        if (c.p < c.end && c.p - c.w0 >= c.wn) {
            if (inj) load_inj(c);
            else load_rec(c);
        }
        const int nxt = c.p < c.end ? (inj ? i_cell : r_cell)[c.p - c.w0] : kNone;
        buf ^= 1;
        if (tid == 0) cur_s[2 * which + buf] = c;
        __syncthreads();
        return nxt;
    };
    // this thread's columns of the model (the first four columns for threads past the row: unused)
    const long long mcol = tin ? j0 : 0;
    // model row `row`, or the nearest row of the grid (values outside the grid are not used)
    auto ld_model = [&](const float *p, int row) -> Q4 {
        return ldg4(p + (long long)min(max(row, 0), nx - 1) * pitch + mcol);
    };
    auto wrap = [&](int slot) -> int { return slot >= N ? slot - N : slot; };

    bool first = true;
    while (Lrow < Lend) {
        const int shot = Lrow / nx, a0 = Lrow - shot * nx;
        const int b0 = min(nx, a0 + (Lend - Lrow));
        Lrow += b0 - a0;
        const long long soff = (long long)shot * nx * pitch;
        const int va = max(a0 - 1, 0), vb = min(b0 + 2, nx);  // velocity rows computed
        const int qa = max(va - 2, 0), qb = min(vb + 1, nx);  // rows streamed through the ring
        int nexti = min(qa + N, qb);                           // next row to issue
        const int slot_a = islot;                              // ring slot of row qa
        __syncthreads();  // the previous range's cursors and ring rows are done with
        if (!first && issuer)
            for (int q = qa, sl = slot_a; q < nexti; q++, sl = wrap(sl + 1)) issue(soff, q, sl);
        islot = (slot_a + (nexti - qa)) % N;
        // the points of this range, found by one warp per list; nothing here depends on the previous
        // step, so the first range's search runs while that step may still be finishing
        if (warp == 0) {
            int p0 = 0, p1 = 0;
            if (inj_on) {
                p0 = a.inj_ptr[shot];
                p1 = a.inj_ptr[shot + 1];
            }
            const int i0 = inj_on ? warp_lower_bound(a.inj_cell, nullptr, p0, p1, va * nz) : 0;
            const int i1 = inj_on ? warp_lower_bound(a.inj_cell, nullptr, i0, p1, vb * nz) : 0;
            if (lane == 0) cur_s[0] = Cursor{i0, i1, i0, 0};
        }
        if (warp == (nwarps > 1 ? 1 : 0)) {
            const int r0 = rec_on ? warp_lower_bound(a.rec_cell, a.rec_order, 0, a.nrec, a0 * nz) : 0;
            const int r1 = rec_on ? warp_lower_bound(a.rec_cell, a.rec_order, r0, a.nrec, b0 * nz) : 0;
            if (lane == 0) cur_s[2] = Cursor{r0, r1, r0, 0};
        }
        // model of the rows of the coming iteration: dt/rho and sponge of rows r, r+1, stiffness of rows
        // r-2, r-1; each is reloaded for the next iteration right after its use
        Q4 buo[2], bnd[2], ip0[2], ip1[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            buo[k] = ld_model(a.buo, va + k);
            bnd[k] = ld_model(a.bound, va + k);
            ip0[k] = ld_model(a.ip[0], va - 2 + k);
            if (MODE == FWI_PSV) ip1[k] = ld_model(a.ip[1], va - 2 + k);
        }
        __syncthreads();
        int inj_next, rec_next;  // row of the next injection entry / receiver, or kNone
        int ib = 0, rb = 0;      // cursor buffers in use
        {
            Cursor c = cur_s[0];
            inj_next = c.p < c.end ? park(c, 0, ib, true) / nz : kNone;
            c = cur_s[2];
            rec_next = c.p < c.end ? park(c, 1, rb, false) / nz : kNone;
        }
        if (first) {
            // the previous step (state rows, and the stress / velocity buffers this step overwrites) is
            // complete from here on
            grid_dep_wait();
            if (issuer)
                for (int q = qa, sl = slot_a; q < nexti; q++, sl = wrap(sl + 1)) issue(soff, q, sl);
            first = false;
        }

        bool ok = true;
        // Register windows: the D-x stress fields at rows r-2 .. r+2 (SH:
        // sxy; P-SV: sxx, sxz), the other stress field at rows r-2 .. r+1
        // (SH: szy; P-SV: szz).
        Q4 wx[NW][5], wz[4];
        // rows va-2 .. va must have landed before the first iteration
        for (int q = qa; q <= va; q++) ok = wait_next() && ok;
        if (__syncthreads_or(!ok)) return give_up();
        int scur = slot_a;  // ring slot of row r
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (va - 2 + k >= qa) {
                const float *s = ring0 + scur * slot_len;
                wx[0][k] = ld4(s + FX0 * RL);
                if (NW > 1) wx[NW - 1][k] = ld4(s + FX1 * RL);
                scur = wrap(scur + 1);
            } else {
                wx[0][k] = wx[NW - 1][k] = zero4();
            }
            wz[k] = zero4();
        }
        {
            const float *s = ring0 + scur * slot_len;
            wx[0][2] = ld4(s + FX0 * RL);
            if (NW > 1) wx[NW - 1][2] = ld4(s + FX1 * RL);
        }
        // rows above va are consumed once every thread has its window: their
        // slots take the next rows
        __syncthreads();
        for (int q = qa; q < va; q++)
            if (nexti < qb) {
                if (issuer) issue(soff, nexti, islot);
                islot = wrap(islot + 1);
                nexti++;
            }

        // this thread's place in row r of the shot (velocity stores; the stress rows lie 2 rows above)
        long long grow = soff + (long long)va * pitch + j0;
        // new-velocity ring, three pairs of rows: (r, r+1), (r-2, r-1), (r-4, r-3)
        float *pa = smem + L.vring + 4 + j0, *pb = pa + 2 * NV * RL, *pc = pb + 2 * NV * RL;

        for (int r = va; r < b0 + 2; r += 2) {
            const int s1 = wrap(scur + 1), s2 = wrap(scur + 2);
            if (r + 1 < qb) ok = wait_next() && ok;
            if (r + 2 < qb) ok = wait_next() && ok;
            Q4 vn[2][NV];
            // ---- velocity of rows r, r+1; K: which of the two.  FAST: both rows are this CTA's own, away
            // from the first and last rows of the grid and without points, so that the row is one stretch
            // of code without a branch; ZE: this warp holds columns near a z edge (per-column masks).
            auto velocity = [&](auto k_t, auto fast_t, auto ze_t, const float *scr, const float *snx) {
                constexpr int K = decltype(k_t)::value;
                constexpr bool FAST = decltype(fast_t)::value, ZE = decltype(ze_t)::value;
                const int row = r + K;
                if (!FAST && row >= vb) {
#pragma unroll
                    for (int c = 0; c < NV; c++) {
                        vn[K][c] = zero4();
                        st4(pa + (K * NV + c) * RL, vn[K][c]);
                    }
                    return;
                }
                if (FAST || row + 1 < qb) {
                    wx[0][3 + K] = ld4(snx + FX0 * RL);
                    if (NW > 1) wx[NW - 1][3 + K] = ld4(snx + FX1 * RL);
                } else {
                    wx[0][3 + K] = wx[NW - 1][3 + K] = zero4();
                }
                wz[2 + K] = ld4(scr + FZ * RL);
                Q4 ds[NV];
                Q4 zz[NV];  // the z derivative of each component (SH: szy; P-SV: sxz, szz)
                if constexpr (MODE == FWI_SH) {
                    zz[0] = dzm4(kz, scr + FZ * RL, wz[2 + K]);
                } else {
                    zz[0] = dzm4(kz, scr + FX1 * RL, wx[1][2 + K]);
                    zz[NV - 1] = dzm4(kz, scr + FZ * RL, wz[2 + K]);
                }
                if (ZE) {
#pragma unroll
                    for (int c = 0; c < NV; c++) zz[c] = keep4(zz[c], zm);
                }
                if (FAST || (row >= 2 && row < nx - 2)) {
#pragma unroll
                    for (int c = 0; c < NV; c++)
                        ds[c] = add4(fdx(kx, wx[c][2 + K], wx[c][1 + K], wx[c][3 + K], wx[c][K]), zz[c]);
                } else {
#pragma unroll
                    for (int c = 0; c < NV; c++) ds[c] = zz[c];
                }
                // sources of the row, summed per cell in entry order (stf_dsy / stf_dsxz, solver.py:78-93)
                if (!FAST && inj_next <= row) {
                    const int lo = row * nz, hi = lo + nz;
                    Q4 acc[NINJ];
#pragma unroll
                    for (int q = 0; q < NINJ; q++) acc[q] = zero4();
                    Cursor c = cur_s[ib];
                    while (c.p < c.end) {
                        if (c.p - c.w0 >= c.wn) load_inj(c);
                        const int k = c.p - c.w0, cell = i_cell[k];
                        if (cell >= hi) break;
                        const int off = cell - lo - j0;
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (off == e) {
#pragma unroll
                                for (int q = 0; q < NINJ; q++) elem(acc[q], e) += i_val[q * kPts + k];
                            }
                        c.p++;
                    }
                    const int nxt = park(c, 0, ib, true);
                    inj_next = nxt == kNone ? kNone : nxt / nz;
#pragma unroll
                    for (int q = 0; q < NV; q++) ds[q] = add4(ds[q], acc[q]);
                }
                const bool own = (FAST || (row >= a0 && row < b0)) && (!ZE || tin);
#pragma unroll
                for (int c = 0; c < NV; c++) {
                    const Q4 vold = ld4(scr + (NS + c) * RL);
                    vn[K][c] = mul4(bnd[K], fma4(ds[c], buo[K], vold));
                    if (ZE) {  // padding columns stay zero
                        vn[K][c] = keep4(vn[K][c], zin);
                        ds[c] = keep4(ds[c], zin);
                    }
                    st4(pa + (K * NV + c) * RL, vn[K][c]);
                    if (own) {
                        st4(a.vel_out[c] + grow + K * pitch, vn[K][c]);
                        if (SEG && a.seg_ds[c]) st4(a.seg_ds[c] + grow + K * pitch, ds[c]);
                    }
                }
                // receivers of the row record the new velocity (save_obs, solver.py:151-156)
                if (!FAST && rec_next <= row) {
                    const int lo = row * nz, hi = lo + nz;
                    Cursor c = cur_s[2 + rb];
                    while (c.p < c.end) {
                        if (c.p - c.w0 >= c.wn) load_rec(c);
                        const int k = c.p - c.w0, cell = r_cell[k];
                        if (cell >= hi) break;
                        const int off = cell - lo - j0;
                        if (off >= 0 && off < 4) {
                            const long long o = ((long long)shot * a.nrec + r_id[k]) * nt + it;
#pragma unroll
                            for (int e = 0; e < 4; e++)
                                if (off == e) {
#pragma unroll
                                    for (int q = 0; q < NV; q++)
                                        if (a.obs[q]) a.obs[q][o] = elem(vn[K][q], e);
                                }
                        }
                        c.p++;
                    }
                    const int nxt = park(c, 1, rb, false);
                    rec_next = nxt == kNone ? kNone : nxt / nz;
                }
            };
            {
                const float *c0 = ring0 + scur * slot_len, *c1 = ring0 + s1 * slot_len, *c2 = ring0 + s2 * slot_len;
                const std::integral_constant<int, 0> k0{};
                const std::integral_constant<int, 1> k1{};
                const std::true_type yes{};
                const std::false_type no{};
                if (r >= max(a0, 2) && r + 1 < min(b0, nx - 2) && min(inj_next, rec_next) > r + 1) {
                    if (zedge) {
                        velocity(k0, yes, yes, c0, c1);
                        velocity(k1, yes, yes, c1, c2);
                    } else {
                        velocity(k0, yes, no, c0, c1);
                        velocity(k1, yes, no, c1, c2);
                    }
                } else {
                    velocity(k0, no, yes, c0, c1);
                    velocity(k1, no, yes, c1, c2);
                }
            }
            // the next iteration's dt/rho and sponge, in flight during the barrier and the stress half (loaded
            // here and not in the branches above, whose join would wait for them)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                buo[k] = ld_model(a.buo, r + 2 + k);
                bnd[k] = ld_model(a.bound, r + 2 + k);
            }
            if (__syncthreads_or(!ok)) return give_up();
            // rows r and r+1 are consumed: their slots take rows r + N, r + N + 1
            scur = s2;
#pragma unroll
            for (int k = 0; k < 2; k++)
                if (nexti < qb) {
                    if (issuer) issue(soff, nexti, islot);
                    islot = wrap(islot + 1);
                    nexti++;
                }

            // ---- stress of rows r-2, r-1 (add_sy / add_sxz, solver.py:128-149)
            Q4 vw[NV][3];  // new velocity of rows r-3, r-2, r-1
#pragma unroll
            for (int c = 0; c < NV; c++) {
                vw[c][0] = ld4(pc + (NV + c) * RL);
                vw[c][1] = ld4(pb + c * RL);
                vw[c][2] = ld4(pb + (NV + c) * RL);
            }
            auto stress = [&](auto k_t, auto fast_t, auto ze_t) {
                constexpr int K = decltype(k_t)::value;
                constexpr bool FAST = decltype(fast_t)::value, ZE = decltype(ze_t)::value;
                const int s = r - 2 + K;
                if ((FAST || (s >= a0 && s < b0)) && (!ZE || tin)) {
                    Q4 ex[NV], ez[NV];
#pragma unroll
                    for (int c = 0; c < NV; c++) {
                        const Q4 &v0 = vw[c][K], &v1 = vw[c][1 + K];
                        const Q4 &v2 = K == 0 ? vw[c][2] : vn[0][c], &v3 = vn[K][c];
                        ez[c] = dzp4(kz, pb + (K * NV + c) * RL, v1);
                        if (ZE) ez[c] = keep4(ez[c], zp);
                        if (FAST || (s >= 1 && s < nx - 2)) ex[c] = fdx(kx, v2, v1, v3, v0);
                        else ex[c] = zero4();
                    }
                    Q4 o[NS], shear = zero4();
                    if constexpr (MODE == FWI_SH) {
                        const Q4 dm = mul4(dt4, ip0[K]);
                        o[0] = fma4(dm, ex[0], wx[0][K]);
                        o[1] = fma4(dm, ez[0], wz[K]);
                    } else {
                        shear = add4(ez[0], ex[NV - 1]);
                        const Q4 two{bc2(2.f), bc2(2.f)};
                        const Q4 l2m = fma4(two, ip1[K], ip0[K]);
                        o[0] = fma4(dt4, fma4(l2m, ex[0], mul4(ip0[K], ez[NV - 1])), wx[0][K]);
                        o[1] = fma4(dt4, fma4(ip0[K], ex[0], mul4(l2m, ez[NV - 1])), wz[K]);
                        o[NS - 1] = fma4(dt4, mul4(ip1[K], shear), wx[NW - 1][K]);
                    }
                    if (ZE) {  // padding columns stay zero
#pragma unroll
                        for (int f = 0; f < NS; f++) o[f] = keep4(o[f], zin);
                        if (SEG && MODE == FWI_PSV) shear = keep4(shear, zin);
                    }
                    const long long gs = grow + (K - 2) * pitch;
#pragma unroll
                    for (int f = 0; f < NS; f++) st4(a.sig_out[f] + gs, o[f]);
                    if (SEG && a.seg_e[0]) {
                        st4(a.seg_e[0] + gs, ex[0]);
                        st4(a.seg_e[1] + gs, ez[NV - 1]);
                        if (MODE == FWI_PSV) st4(a.seg_e[NS - 1] + gs, shear);
                    }
                }
            };
            {
                const std::integral_constant<int, 0> k0{};
                const std::integral_constant<int, 1> k1{};
                const std::true_type yes{};
                const std::false_type no{};
                if (r - 2 >= max(a0, 1) && r - 1 < min(b0, nx - 2)) {
                    if (zedge) {
                        stress(k0, yes, yes);
                        stress(k1, yes, yes);
                    } else {
                        stress(k0, yes, no);
                        stress(k1, yes, no);
                    }
                } else {
                    stress(k0, no, yes);
                    stress(k1, no, yes);
                }
            }
            // and its stiffness, in flight during the next velocity half
#pragma unroll
            for (int k = 0; k < 2; k++) {
                ip0[k] = ld_model(a.ip[0], r + k);
                if (MODE == FWI_PSV) ip1[k] = ld_model(a.ip[1], r + k);
            }
            // the windows move down two rows
#pragma unroll
            for (int w = 0; w < NW; w++) {
                wx[w][0] = wx[w][2];
                wx[w][1] = wx[w][3];
                wx[w][2] = wx[w][4];
            }
            wz[0] = wz[2];
            wz[1] = wz[3];
            float *const t = pc;
            pc = pb;
            pb = pa;
            pa = t;
            grow += 2 * pitch;
        }
    }
}

// ------------------------------------------------- small grids: resident steps
//
// All steps of one fwi_run call on a grid whose shots fit the shared memory of
// a cluster: a cluster of C CTAs holds one shot for the whole call, CTA k the
// rows [nx k/C, nx (k+1)/C), stress and velocity in shared memory, the model of
// a thread's cells in its registers.  A thread owns four adjacent columns of up
// to kResRows consecutive rows, so the x taps of the stencils are read once per
// row.  Per step: velocity of the own rows and of the three halo rows the D+x
// taps reach (computed twice, so that only stress is exchanged), a block
// barrier, stress of the own rows, whose first and last three the owner also
// writes into the neighbours' halo rows (distributed shared memory, two copies
// by the parity of the step), a cluster barrier.  Sources and receivers as in
// march_kernel: the points of a thread's cells are ranges of the cell-sorted
// lists, found once per call.  The arithmetic per cell is march_kernel's.
//
// A launched step cannot be shorter than a launch and a pass through L2, 5.6 us
// (SH) to 8 us (P-SV) here; a resident one costs its arithmetic, bound by the
// latency of 16 warps' shared-memory loads and packed operations, and two
// barriers: one SH shot on 256 x 256 5.9 -> 2.8 us, P-SV 183 x 270, 3 shots
// 8.5 -> 4.8 us, 256 x 128, 16 shots 12.4 -> 5.8 us, 64 x 64, 64 shots 13.4 ->
// 3.4 us a step.

constexpr int kResThreads = 512;
constexpr int kResPts = 64;  // source values and receiver numbers staged in shared memory

struct ResidentArgs {
    int nx, nz, pitch, nt, it0, nsteps, nrec;
    int rows_max;           // rows of a CTA, at most
    int groups, segs;       // column groups of four per row; row segments (threads = groups x segs)
    float cx1, cx2, cz1, cz2, dt;
    const float *sig_in[3];
    float *sig_out[3];
    const float *vel_in[2];
    float *vel_out[2];
    float *sig_prev[3], *vel_prev[2];  // the other half: the state before the last step
    const float *buo, *bound;
    const float *ip[2];
    const int *inj_ptr, *inj_cell, *inj_row;
    const float *stf[2];
    const int *rec_cell, *rec_order;
    float *obs[2];
};

// Floats of shared memory: stress rows (own, and two copies of the three halo
// rows on either side) and velocity rows of RL floats, then the staged points.
template <int MODE>
static size_t resident_bytes(int rows, int pitch) {
    using F = Fields<MODE>;
    return sizeof(float) * ((size_t)(F::NS * (rows + 12) + F::NV * (rows + 3)) * (pitch + 8) +
                            (size_t)kResPts * (2 * F::NINJ + 3));
}

template <int MODE, int I>
__global__ void __launch_bounds__(kResThreads, 1) resident_kernel(const __grid_constant__ ResidentArgs a) {
    using F = Fields<MODE>;
    constexpr int NS = F::NS, NV = F::NV, NINJ = F::NINJ;
    constexpr int FX0 = 0, FX1 = MODE == FWI_SH ? 0 : 2, FZ = 1;
    extern __shared__ __align__(128) float smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int nx = a.nx, nz = a.nz, pitch = a.pitch, nt = a.nt, RL = pitch + 8, RM = a.rows_max;
    const int shot = blockIdx.y, tid = threadIdx.x;
    const int row0 = (int)((long long)nx * rank / C), n = (int)((long long)nx * (rank + 1) / C) - row0;
    const int FS = (RM + 12) * RL, FV = (RM + 3) * RL;  // field strides
    // stress row q = 0 .. n+5 is grid row row0-3+q; the halo rows q < 3 and q >= n+3 of an odd step sit in the
    // last six rows of the field.  Velocity row q = 0 .. n+2 is grid row row0-1+q.
    float *const S = smem, *const V = smem + NS * FS;
    float *const pts = V + NV * FV;  // source values [2][NINJ][kResPts]; source cells, receiver numbers and cells
    int *const i_cell = reinterpret_cast<int *>(pts + 2 * NINJ * kResPts), *const r_id = i_cell + kResPts,
              *const r_cell = r_id + kResPts;
    const int cg4 = tid % a.groups, seg = tid / a.groups, j0 = 4 * cg4;
    const bool work = seg < a.segs;
    const Coef kx{bc2(a.cx1), bc2(-a.cx2)}, kz{bc2(a.cz1), bc2(-a.cz2)};
    const Q4 dt4{bc2(a.dt), bc2(a.dt)};
    const long long soff = (long long)shot * nx * pitch;
    bool zm[4], zp[4], zin[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int c = j0 + e;
        zm[e] = c >= 2 && c < nz - 2;
        zp[e] = c >= 1 && c < nz - 2;
        zin[e] = c < nz;
    }
    // this thread's velocity rows [v0, v0+nv) of n+3 and stress rows [s0, s0+ns) of n, as local rows
    const int iv = (n + 3 + a.segs - 1) / a.segs, is = (n + a.segs - 1) / a.segs;
    const int v0 = seg * iv, nv = work ? min(iv, n + 3 - v0) : 0;
    const int s0 = seg * is, ns = work ? min(is, n - s0) : 0;

    // ---- state into shared memory (zero outside the grid and in the padding columns, where it stays zero)
    for (int q = tid; q < (n + 6) * a.groups; q += kResThreads) {
        const int r = q / a.groups, c = 4 * (q - r * a.groups), gr = row0 - 3 + r;
        const bool in = gr >= 0 && gr < nx;
        const bool cin[4] = {c < nz, c + 1 < nz, c + 2 < nz, c + 3 < nz};
#pragma unroll
        for (int f = 0; f < NS; f++) {
            const Q4 v = in ? keep4(ld4(a.sig_in[f] + soff + (long long)gr * pitch + c), cin) : zero4();
            st4(S + f * FS + r * RL + 4 + c, v);
            // the odd copies of halo rows outside the grid stay zero; the others are written by the first step
            if (r < 3) st4(S + f * FS + (RM + 6 + r) * RL + 4 + c, zero4());
            if (r >= n + 3) st4(S + f * FS + (RM + 9 + r - n - 3) * RL + 4 + c, zero4());
        }
        if (r >= 2 && r < n + 5) {
#pragma unroll
            for (int c2 = 0; c2 < NV; c2++)
                st4(V + c2 * FV + (r - 2) * RL + 4 + c,
                    in ? keep4(ld4(a.vel_in[c2] + soff + (long long)gr * pitch + c), cin) : zero4());
        }
    }
    // ---- model of this thread's cells (zero in the padding columns, which keeps them zero)
    Q4 buo[I], bnd[I], ip0[I], ip1[I];
    // points of its velocity cells: first entry and count of the two lists
    int inj_lo[I], rec_lo[I];
    unsigned cnt[I];  // injection count | receiver count << 16
    const bool rec_on = a.rec_order && a.nrec > 0 && (a.obs[0] || (NV > 1 && a.obs[1]));
    int p0 = 0, p1 = 0;
    if (a.inj_ptr) {
        p0 = a.inj_ptr[shot];
        p1 = a.inj_ptr[shot + 1];
    }
    // the entries of the CTA's rows, of which the first kResPts are staged
    const int clo = max(row0 - 1, 0) * nz, chi = min(row0 + n + 2, nx) * nz;
    const int il = thread_lower_bound(a.inj_cell, nullptr, p0, p1, clo), ih = thread_lower_bound(a.inj_cell, nullptr, il, p1, chi);
    const int rl = rec_on ? thread_lower_bound(a.rec_cell, a.rec_order, 0, a.nrec, row0 * nz) : 0;
    const int rh = rec_on ? thread_lower_bound(a.rec_cell, a.rec_order, rl, a.nrec, (row0 + n) * nz) : 0;
    const int ni = min(ih - il, kResPts), nr = min(rh - rl, kResPts);
#pragma unroll
    for (int k = 0; k < I; k++) {
        const int gr = row0 - 1 + v0 + k;
        const bool in = k < nv && gr >= 0 && gr < nx;
        buo[k] = in ? keep4(ldg4(a.buo + (long long)gr * pitch + j0), zin) : zero4();
        bnd[k] = in ? keep4(ldg4(a.bound + (long long)gr * pitch + j0), zin) : zero4();
        const int gs = row0 + s0 + k;
        ip0[k] = k < ns ? keep4(ldg4(a.ip[0] + (long long)gs * pitch + j0), zin) : zero4();
        if (MODE == FWI_PSV) ip1[k] = k < ns ? keep4(ldg4(a.ip[1] + (long long)gs * pitch + j0), zin) : zero4();
        inj_lo[k] = rec_lo[k] = 0;
        cnt[k] = 0;
        if (in && j0 < nz) {
            const int c0 = gr * nz + j0, c1 = gr * nz + min(j0 + 4, nz);
            inj_lo[k] = thread_lower_bound(a.inj_cell, nullptr, il, ih, c0);
            cnt[k] = thread_lower_bound(a.inj_cell, nullptr, inj_lo[k], ih, c1) > inj_lo[k] ? 1u : 0u;
            if (gr >= row0 && gr < row0 + n && rh > rl) {
                rec_lo[k] = thread_lower_bound(a.rec_cell, a.rec_order, rl, rh, c0);
                cnt[k] |= thread_lower_bound(a.rec_cell, a.rec_order, rec_lo[k], rh, c1) > rec_lo[k] ? 2u : 0u;
            }
        }
    }
    // source values of a step, staged one step ahead
    auto stage = [&](int it) {
        if (tid < ni) {
            const long long src = (long long)a.inj_row[il + tid] * nt + it;
#pragma unroll
            for (int q = 0; q < NINJ; q++) pts[((it & 1) * NINJ + q) * kResPts + tid] = a.stf[q][src];
        }
    };
    stage(a.it0);
    if (tid < ni) i_cell[tid] = a.inj_cell[il + tid];
    if (tid < nr) {
        r_id[tid] = a.rec_order[rl + tid];
        r_cell[tid] = a.rec_cell[r_id[tid]];
    }
    cluster.sync();

    // the state of the own rows to global memory
    auto store_state = [&](float *const(&sig)[3], float *const(&vel)[2]) {
        for (int q = tid; q < n * a.groups; q += kResThreads) {
            const int r = q / a.groups, c = 4 * (q - r * a.groups);
            const long long g = soff + (long long)(row0 + r) * pitch + c;
#pragma unroll
            for (int f = 0; f < NS; f++) st4(sig[f] + g, ld4(S + f * FS + (r + 3) * RL + 4 + c));
#pragma unroll
            for (int c2 = 0; c2 < NV; c2++) st4(vel[c2] + g, ld4(V + c2 * FV + (r + 1) * RL + 4 + c));
        }
    };
    float *const up = rank > 0 ? cluster.map_shared_rank(S, rank - 1) : nullptr;
    float *const down = rank + 1 < C ? cluster.map_shared_rank(S, rank + 1) : nullptr;
    const int n_up = row0 - (rank > 0 ? (int)((long long)nx * (rank - 1) / C) : 0);  // rows of the CTA above
    // all steps but the last; then, once the state before it is in the other half (as launched steps leave it), the
    // last.  Two loops, since a branch in the time loop costs every step 2-3 %.
    for (int step = 0, end = a.nsteps - 1;; end++) {
        for (; step < end; step++) {
            const int it = a.it0 + step, par = step & 1;
            // stress row q of this step at this thread's columns
            auto srow = [&](int q) -> float * {
                int r = q;
                if (par && q < 3) r = RM + 6 + q;
                if (par && q >= n + 3) r = RM + 9 + q - n - 3;
                return S + r * RL + 4 + j0;
            };
            // ---- velocity
            if (nv > 0) {
                Q4 w0[4], w1[4];  // D-x windows
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const float *s = srow(v0 + k);
                    w0[k] = ld4(s + FX0 * FS);
                    if (NV > 1) w1[k] = ld4(s + FX1 * FS);
                }
#pragma unroll
                for (int k = 0; k < I; k++) {
                    if (k < nv) {
                        const int gr = row0 - 1 + v0 + k;
                        const float *s = srow(v0 + k + 3), *sc = srow(v0 + k + 2);
                        w0[(k + 3) & 3] = ld4(s + FX0 * FS);
                        if (NV > 1) w1[(k + 3) & 3] = ld4(s + FX1 * FS);
                        if (gr >= 0 && gr < nx) {
                            const Q4 cz = ld4(sc + FZ * FS);
                            Q4 ds[NV], vn[NV];
                            if constexpr (MODE == FWI_SH) {
                                ds[0] = keep4(dzm4(kz, sc + FZ * FS, cz), zm);
                            } else {
                                ds[0] = keep4(dzm4(kz, sc + FX1 * FS, w1[(k + 2) & 3]), zm);
                                ds[NV - 1] = keep4(dzm4(kz, sc + FZ * FS, cz), zm);
                            }
                            if (gr >= 2 && gr < nx - 2) {
                                ds[0] = add4(fdx(kx, w0[(k + 2) & 3], w0[(k + 1) & 3], w0[(k + 3) & 3], w0[k & 3]), ds[0]);
                                if (NV > 1)
                                    ds[NV - 1] = add4(fdx(kx, w1[(k + 2) & 3], w1[(k + 1) & 3], w1[(k + 3) & 3], w1[k & 3]),
                                                      ds[NV - 1]);
                            }
                            if (cnt[k] & 1) {  // sources, summed per cell in entry order (stf_dsy / stf_dsxz, solver.py:78-93)
                                Q4 acc[NINJ];
#pragma unroll
                                for (int q = 0; q < NINJ; q++) acc[q] = zero4();
                                const int base = gr * nz + j0, end = gr * nz + min(j0 + 4, nz);
                                for (int e = inj_lo[k]; e < ih; e++) {
                                    const int at = e - il, cell = at < kResPts ? i_cell[at] : a.inj_cell[e];
                                    if (cell >= end) break;
#pragma unroll
                                    for (int q = 0; q < NINJ; q++) {
                                        const float val = at < kResPts ? pts[((it & 1) * NINJ + q) * kResPts + at]
                                                                       : a.stf[q][(long long)a.inj_row[e] * nt + it];
#pragma unroll
                                        for (int x = 0; x < 4; x++)
                                            if (cell - base == x) elem(acc[q], x) += val;
                                    }
                                }
#pragma unroll
                                for (int q = 0; q < NV; q++) ds[q] = add4(ds[q], acc[q]);
                            }
#pragma unroll
                            for (int c = 0; c < NV; c++) {
                                float *v = V + c * FV + (v0 + k) * RL + 4 + j0;
                                vn[c] = mul4(bnd[k], fma4(ds[c], buo[k], ld4(v)));
                                st4(v, vn[c]);
                            }
                            if (cnt[k] & 2) {  // receivers record the new velocity (save_obs, solver.py:151-156)
                                const int base = gr * nz + j0, end = gr * nz + min(j0 + 4, nz);
                                for (int e = rec_lo[k]; e < rh; e++) {
                                    const int at = e - rl, id = at < kResPts ? r_id[at] : a.rec_order[e];
                                    const int cell = at < kResPts ? r_cell[at] : a.rec_cell[id];
                                    if (cell >= end) break;
                                    const long long o = ((long long)shot * a.nrec + id) * nt + it;
#pragma unroll
                                    for (int x = 0; x < 4; x++)
                                        if (cell - base == x) {
#pragma unroll
                                            for (int q = 0; q < NV; q++)
                                                if (a.obs[q]) a.obs[q][o] = elem(vn[q], x);
                                        }
                                }
                            }
                        }
                    }
                }
            }
            __syncthreads();
            if (step + 1 < a.nsteps) stage(it + 1);
            // ---- stress
            if (ns > 0) {
                Q4 w[NV][4];  // velocity rows s-1 .. s+2
#pragma unroll
                for (int k = 0; k < 3; k++)
#pragma unroll
                    for (int c = 0; c < NV; c++) w[c][k] = ld4(V + c * FV + (s0 + k) * RL + 4 + j0);
#pragma unroll
                for (int k = 0; k < I; k++) {
                    if (k < ns) {
                        const int gs = row0 + s0 + k;
                        Q4 ex[NV], ez[NV];
#pragma unroll
                        for (int c = 0; c < NV; c++) {
                            const float *v = V + c * FV + (s0 + k) * RL + 4 + j0;
                            w[c][(k + 3) & 3] = ld4(v + 3 * RL);
                            ez[c] = keep4(dzp4(kz, v + RL, w[c][(k + 1) & 3]), zp);
                            if (gs >= 1 && gs < nx - 2) ex[c] = fdx(kx, w[c][(k + 2) & 3], w[c][(k + 1) & 3], w[c][(k + 3) & 3], w[c][k & 3]);
                            else ex[c] = zero4();
                        }
                        float *s = S + (s0 + k + 3) * RL + 4 + j0;
                        Q4 o[NS];
                        if constexpr (MODE == FWI_SH) {
                            const Q4 dm = mul4(dt4, ip0[k]);
                            o[0] = fma4(dm, ex[0], ld4(s));
                            o[1] = fma4(dm, ez[0], ld4(s + FS));
                        } else {
                            const Q4 two{bc2(2.f), bc2(2.f)};
                            const Q4 l2m = fma4(two, ip1[k], ip0[k]);
                            o[0] = fma4(dt4, fma4(l2m, ex[0], mul4(ip0[k], ez[NV - 1])), ld4(s));
                            o[1] = fma4(dt4, fma4(ip0[k], ex[0], mul4(l2m, ez[NV - 1])), ld4(s + FS));
                            o[NS - 1] = fma4(dt4, mul4(ip1[k], add4(ez[0], ex[NV - 1])), ld4(s + (NS - 1) * FS));
                        }
                        const int q = s0 + k;
#pragma unroll
                        for (int f = 0; f < NS; f++) {
                            st4(s + f * FS, o[f]);
                            // the neighbours' halo rows of the next step (even steps read the rows in place)
                            if (up && q < 3) st4(up + f * FS + ((par ? n_up + 3 : RM + 9) + q) * RL + 4 + j0, o[f]);
                            if (down && q >= n - 3) st4(down + f * FS + ((par ? 0 : RM + 6) + q - n + 3) * RL + 4 + j0, o[f]);
                        }
                    }
                }
            }
            cluster.sync();
        }
        if (end == a.nsteps) break;
        store_state(a.sig_prev, a.vel_prev);
        __syncthreads();
    }
    store_state(a.sig_out, a.vel_out);
}

// Displacement traces from velocity traces: u(it) = u(it-1) + v(it) dt over
// steps [it0, it0+n) of every trace ([trace][nt]), u(it0-1) being the
// trace's value before it0 (0 at it0 = 0) -- the displacement update of
// add_vy / add_vxz (solver.py:95-109) in the same float operations.
__global__ void displacement_traces_kernel(float *obs, long long ntr, int nt, int it0, int n, float dt) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntr) return;
    float *p = obs + t * nt;
    float u = it0 > 0 ? p[it0 - 1] : 0.f;
    for (int i = it0; i < it0 + n; i++) {
        u = u + p[i] * dt;
        p[i] = u;
    }
}

// ------------------------------------------------------------- host side

static int comp_slot_of(int mode, int q) { return mode == FWI_SH ? 1 : (q == 0 ? 0 : 2); }

// Shared-memory bytes of a ring depth for a row length.
static size_t march_bytes(int mode, int rl, int n) {
    const int nf = mode == FWI_SH ? 3 : 5, nv = mode == FWI_SH ? 1 : 2, ninj = mode == FWI_SH ? 1 : 2;
    return march_layout(nf, nv, ninj, rl, n).bytes;
}

bool march_supported(const fwi_batch *b) {
    return (b->mode == FWI_SH || b->mode == FWI_PSV) && b->pitch <= kMaxPitch;
}

constexpr size_t kMaxSmem = 227 * 1024;

// The calling thread's device: a kernel's attributes and what fits at once are
// kept per device.
static int current_device() {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess ? dev : 0;
}

// Ring depth and resident CTAs per SM for a launch shape: the requested
// depth, or the one with the most resident CTAs (shared memory and
// registers both counted), the deepest among those.  Made once per device and
// shape; the kernel's dynamic shared memory limit is the SM's throughout, so
// that a shape's plan does not depend on which other shapes have run.
struct MarchPlan {
    int dev, nthr, rl, want, n, occ;
    size_t bytes;
};

template <int MODE, int WIDE, bool SEG>
static int march_choose(int nthr, int rl, int want, MarchPlan *out) {
    static std::mutex lock;
    static std::vector<MarchPlan> plans;
    const auto kernel = march_kernel<MODE, WIDE, SEG>;
    const int dev = current_device();
    std::lock_guard<std::mutex> hold(lock);
    bool first = true;  // on this device
    for (const MarchPlan &p : plans)
        if (p.dev == dev) {
            first = false;
            if (p.nthr == nthr && p.rl == rl && p.want == want) {
                *out = p;
                return 0;
            }
        }
    if (first) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
        if (e != cudaSuccess) return set_error(FWI_ECUDA, "march_kernel shared memory: %s", cudaGetErrorString(e));
    }
    MarchPlan best{dev, nthr, rl, want, 0, 0, 0};
    for (int n : {3, 4, 6, 8}) {
        if (want && n != want) continue;
        const size_t b = march_bytes(MODE, rl, n);
        if (b > kMaxSmem) continue;
        int occ = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, nthr, b);
        if (e != cudaSuccess) return set_error(FWI_ECUDA, "march_kernel occupancy: %s", cudaGetErrorString(e));
        if (occ >= 1 && occ >= best.occ) {
            best.n = n;
            best.occ = occ;
            best.bytes = b;
        }
    }
    if (!best.n) return set_error(FWI_ERANGE, "row-marching step: rows of %d floats do not fit an SM", rl - 8);
    plans.push_back(best);
    *out = best;
    return 0;
}

static int sm_count() {
    static std::atomic<int> sms[16];  // of the first devices, 0 until asked for
    const int dev = current_device();
    int n = dev < 16 ? sms[dev].load(std::memory_order_relaxed) : 0;
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
        if (dev < 16) sms[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

template <int MODE, int WIDE, bool SEG>
static int launch_march_mode(MarchArgs &a, int nthr, int want, int cap, bool pdl, cudaStream_t st) {
    MarchPlan p;
    const int rc = march_choose<MODE, WIDE, SEG>(nthr, a.rl, want, &p);
    if (rc) return rc;
    a.nslots = p.n;
    const int occ = cap > 0 && cap < p.occ ? cap : p.occ;
    const long long slots = (long long)sm_count() * occ;
    const long long grid = a.rows_total < slots ? a.rows_total : slots;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(nthr, 1, 1);
    cfg.dynamicSmemBytes = p.bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    set_pdl_attr(attr[0], true);
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, march_kernel<MODE, WIDE, SEG>, a);
    if (e != cudaSuccess) return launch_failed("march_kernel", e);
    return check_launch("march_kernel");
}

template <int MODE>
static int launch_march_any(MarchArgs &a, int nthr, int want, int cap, bool pdl, cudaStream_t st) {
    const bool seg = a.seg_e[0] || a.seg_ds[0] || a.seg_ds[1];
    if (nthr > 128)
        return seg ? launch_march_mode<MODE, 1, true>(a, nthr, want, cap, pdl, st)
                   : launch_march_mode<MODE, 1, false>(a, nthr, want, cap, pdl, st);
    return seg ? launch_march_mode<MODE, 0, true>(a, nthr, want, cap, pdl, st)
               : launch_march_mode<MODE, 0, false>(a, nthr, want, cap, pdl, st);
}

// ------------------------------------------------------------ resident steps

// Fewer steps in one call are launched one by one: a resident call takes 9 to
// 14 us more besides its steps than a launched one, and from 8 steps on is still
// the faster (8 steps, launched -> resident: SH 256 x 256, 1 shot 48 -> 37 us;
// P-SV 128 x 96, 4 shots 67 -> 39 us; 183 x 270, 3 shots 75 -> 58 us).
constexpr int kResMinSteps = 8;

// Clusters of csize CTAs of the resident kernel the GPU holds at once (0: none).
template <int MODE, int I>
static int resident_clusters(int csize, size_t bytes) {
    static std::mutex lock;
    struct Known {
        int dev, csize, clusters;
        size_t bytes;
    };
    static std::vector<Known> known;
    const int dev = current_device();
    std::lock_guard<std::mutex> hold(lock);
    const auto kernel = resident_kernel<MODE, I>;
    bool first = true;  // on this device
    for (const Known &k : known)
        if (k.dev == dev) {
            first = false;
            if (k.csize == csize && k.bytes == bytes) return k.clusters;
        }
    if (first &&
        (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) != cudaSuccess ||
         cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(csize, 1, 1);
    cfg.blockDim = dim3(kResThreads, 1, 1);
    cfg.dynamicSmemBytes = bytes;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();  // a cluster this large or this much shared memory: not available
        n = 0;
    }
    if (known.size() >= 1024) known.clear();
    known.push_back(Known{dev, csize, n, bytes});
    return n;
}

template <int MODE, int I>
static int launch_resident_kernel(const ResidentArgs &a, int csize, int nshots, size_t bytes, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(csize, nshots, 1);
    cfg.blockDim = dim3(kResThreads, 1, 1);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, resident_kernel<MODE, I>, a);
    if (e != cudaSuccess) return launch_failed("resident_kernel", e);
    return check_launch("resident_kernel");
}

template <int MODE>
static int resident_clusters_i(int i, int csize, size_t bytes) {
    switch (i) {
        case 1: return resident_clusters<MODE, 1>(csize, bytes);
        case 2: return resident_clusters<MODE, 2>(csize, bytes);
        case 3: return resident_clusters<MODE, 3>(csize, bytes);
        default: return resident_clusters<MODE, 4>(csize, bytes);
    }
}

// Microseconds of a step, fitted to measurements and indexed by wave type (SH,
// P-SV).  Launched: a + b per cell of the batch (one SH shot on 256 x 256 5.9,
// 16 shots 10.6; P-SV 183 x 270, 3 shots 8.5, 256 x 128, 16 shots 12.4).
// Resident: a + b per velocity and per stress row of a thread (SH 256 x 256 on
// 16 CTAs, 3 + 2 rows, 2.8; on 9 CTAs, 4 + 4 rows, 4.0; P-SV 128 x 96 on 16
// CTAs, 1 + 1 rows, 2.4; 64 x 64 on 2 CTAs, 2 + 2 rows, 3.4; 183 x 270 on 16
// CTAs, 3 + 2 rows, 4.8), more where the model of 3 or 4 rows of P-SV cells
// spills registers (256 x 128 on 6 CTAs, 3 + 3 rows, 5.8; 183 x 270 on 8 CTAs,
// 4 + 4 rows, 8.2), times the waves of clusters that the GPU does not hold at
// once.  Resident wins for every batch that one wave holds and loses to
// launched steps from three or four waves on.
static double launched_us(int mode, double cells) {
    return mode == FWI_SH ? 5.5 + 4.9e-6 * cells : 7.5 + 8.3e-6 * cells;
}
static double resident_us(int mode, int vel_rows, int stress_rows) {
    if (mode == FWI_SH) return 0.75 + 0.4 * (vel_rows + stress_rows);
    const double spill = vel_rows == 4 ? 2.0 : vel_rows == 3 && stress_rows == 3 ? 0.9 : 0.0;
    return 1.0 + 0.65 * (vel_rows + stress_rows) + spill;
}

constexpr double kResCallUs = 10.0;  // of a call besides its steps, more than a launched call's (9 to 14 us)

// The cluster size and rows per thread that finish a call first, or false
// where launched steps do or a shot does not fit.
struct ResidentPlan {
    int csize, rows, groups, segs, i;
    size_t bytes;
};
template <int MODE>
static bool resident_plan(const fwi_batch *b, int nsteps, ResidentPlan *out) {
    const int groups = b->pitch / 4;
    if (groups > kResThreads) return false;
    // a call also loads and stores the state and finds the points
    double best = 0.9 * launched_us(MODE, (double)b->nx * b->pitch * b->nshots) - kResCallUs / nsteps;
    bool found = false;
    for (int c = 1; c <= 16; c++) {
        const int rows = (b->nx + c - 1) / c;
        if (b->nx / c < 3) break;  // the three rows a neighbour needs come from one CTA
        const int segs = kResThreads / groups, i = (rows + 3 + segs - 1) / segs, is = (rows + segs - 1) / segs;
        const size_t bytes = resident_bytes<MODE>(rows, b->pitch);
        if (i > 4 || bytes > kMaxSmem) continue;
        const int n = resident_clusters_i<MODE>(i, c, bytes);
        if (n < 1) continue;
        const double t = (b->nshots + n - 1) / n * resident_us(MODE, i, is);
        if (t < best) {
            best = t;
            found = true;
            *out = ResidentPlan{c, rows, groups, segs, i, bytes};
        }
    }
    return found;
}

// All steps [it0, it0 + nsteps) of a displacement-free forward batch on the
// resident kernel, the state going from half cur to the half that many
// single steps would end in, the state one step earlier to the other; 1 if the batch is left to launched steps.
int launch_resident(const fwi_batch *b, int it0, int nsteps, cudaStream_t st) {
    const int mode = b->mode;
    // segment stores come from launched steps
    const bool seg = it0 + nsteps > b->seg0 && it0 < b->seg0 + b->nseg;
    if (nsteps < kResMinSteps || seg || b->ring || b->ctas_per_sm) return 1;
    ResidentPlan p;
    if (!(mode == FWI_SH ? resident_plan<FWI_SH>(b, nsteps, &p) : resident_plan<FWI_PSV>(b, nsteps, &p))) return 1;
    ResidentArgs a;
    a.nx = b->nx;
    a.nz = b->nz;
    a.pitch = b->pitch;
    a.nt = b->nt;
    a.it0 = it0;
    a.nsteps = nsteps;
    a.nrec = b->nrec;
    a.rows_max = p.rows;
    a.groups = p.groups;
    a.segs = p.segs;
    a.cx1 = (float)(9.0 / (8.0 * (double)b->dx));
    a.cx2 = (float)(1.0 / (24.0 * (double)b->dx));
    a.cz1 = (float)(9.0 / (8.0 * (double)b->dz));
    a.cz2 = (float)(1.0 / (24.0 * (double)b->dz));
    a.dt = (float)b->dt;
    const int cur = b->cur, end = cur ^ (nsteps & 1), ns = mode == FWI_SH ? 2 : 3, nv = mode == FWI_SH ? 1 : 2;
    for (int f = 0; f < 3; f++) {
        a.sig_in[f] = f < ns ? b->sig[cur][f] : nullptr;
        a.sig_out[f] = f < ns ? b->sig[end][f] : nullptr;
        a.sig_prev[f] = f < ns ? b->sig[1 - end][f] : nullptr;
    }
    for (int q = 0; q < 2; q++) {
        const bool on = q < nv;
        a.vel_in[q] = on ? b->vel[cur][q] : nullptr;
        a.vel_out[q] = on ? b->vel[end][q] : nullptr;
        a.vel_prev[q] = on ? b->vel[1 - end][q] : nullptr;
        a.obs[q] = on ? b->obs[comp_slot_of(mode, q)] : nullptr;
    }
    a.buo = b->buo;
    a.bound = b->bound;
    a.ip[0] = mode == FWI_SH ? b->mu : b->lam;
    a.ip[1] = mode == FWI_SH ? nullptr : b->mu;
    a.inj_ptr = b->inj_ptr;
    a.inj_cell = b->inj_cell;
    a.inj_row = b->inj_row;
    a.stf[0] = mode == FWI_SH ? b->stf[1] : b->stf[0];
    a.stf[1] = mode == FWI_SH ? nullptr : b->stf[2];
    a.rec_cell = b->rec_cell;
    a.rec_order = b->rec_order;
    const int n = b->nshots;
    if (mode == FWI_SH) {
        switch (p.i) {
            case 1: return launch_resident_kernel<FWI_SH, 1>(a, p.csize, n, p.bytes, st);
            case 2: return launch_resident_kernel<FWI_SH, 2>(a, p.csize, n, p.bytes, st);
            case 3: return launch_resident_kernel<FWI_SH, 3>(a, p.csize, n, p.bytes, st);
            default: return launch_resident_kernel<FWI_SH, 4>(a, p.csize, n, p.bytes, st);
        }
    }
    switch (p.i) {
        case 1: return launch_resident_kernel<FWI_PSV, 1>(a, p.csize, n, p.bytes, st);
        case 2: return launch_resident_kernel<FWI_PSV, 2>(a, p.csize, n, p.bytes, st);
        case 3: return launch_resident_kernel<FWI_PSV, 3>(a, p.csize, n, p.bytes, st);
        default: return launch_resident_kernel<FWI_PSV, 4>(a, p.csize, n, p.bytes, st);
    }
}

int launch_march(const fwi_batch *b, int it, bool pdl, cudaStream_t st) {
    MarchArgs a;
    const int mode = b->mode;
    a.nx = b->nx;
    a.nz = b->nz;
    a.pitch = b->pitch;
    a.nt = b->nt;
    a.it = it;
    a.nrec = b->nrec;
    a.rows_total = (long long)b->nshots * b->nx;
    if (a.rows_total >= (1ll << 31))
        return set_error(FWI_ERANGE, "row-marching step: nshots * nx = %lld rows exceed 2^31", a.rows_total);
    a.cx1 = (float)(9.0 / (8.0 * (double)b->dx));
    a.cx2 = (float)(1.0 / (24.0 * (double)b->dx));
    a.cz1 = (float)(9.0 / (8.0 * (double)b->dz));
    a.cz2 = (float)(1.0 / (24.0 * (double)b->dz));
    a.dt = (float)b->dt;
    const int cur = b->cur, nxt = 1 - cur;
    const int ns = mode == FWI_SH ? 2 : 3, nv = mode == FWI_SH ? 1 : 2, ne = ns == 2 ? 2 : 3;
    for (int f = 0; f < 3; f++) {
        a.sig_in[f] = f < ns ? b->sig[cur][f] : nullptr;
        a.sig_out[f] = f < ns ? b->sig[nxt][f] : nullptr;
    }
    const long long field = (long long)b->nshots * b->nx * b->pitch;
    const bool seg = it - b->seg0 >= 0 && it - b->seg0 < b->nseg;
    for (int q = 0; q < 2; q++) {
        const bool on = q < nv;
        const int slot = on ? comp_slot_of(mode, q) : 0;
        a.vel_in[q] = on ? b->vel[cur][q] : nullptr;
        a.vel_out[q] = on ? b->vel[nxt][q] : nullptr;
        a.obs[q] = on ? b->obs[slot] : nullptr;
        a.seg_ds[q] = (on && seg && b->seg_ds[slot]) ? b->seg_ds[slot] + (long long)(it - b->seg0) * field : nullptr;
    }
    for (int k = 0; k < 3; k++)
        a.seg_e[k] = (seg && k < ne && b->seg_e[k]) ? b->seg_e[k] + (long long)(it - b->seg0) * field : nullptr;
    a.buo = b->buo;
    a.bound = b->bound;
    a.ip[0] = mode == FWI_SH ? b->mu : b->lam;
    a.ip[1] = mode == FWI_SH ? nullptr : b->mu;
    a.inj_ptr = b->inj_ptr;
    a.inj_cell = b->inj_cell;
    a.inj_row = b->inj_row;
    a.stf[0] = mode == FWI_SH ? b->stf[1] : b->stf[0];
    a.stf[1] = mode == FWI_SH ? nullptr : b->stf[2];
    a.rec_cell = b->rec_cell;
    a.rec_order = b->rec_order;
    // four columns per thread, whole warps
    const int nthr = ((b->pitch / 4 + 31) / 32) * 32;
    a.rl = 4 * nthr + 8;
    return mode == FWI_SH ? launch_march_any<FWI_SH>(a, nthr, b->ring, b->ctas_per_sm, pdl, st)
                          : launch_march_any<FWI_PSV>(a, nthr, b->ring, b->ctas_per_sm, pdl, st);
}

// A bounded wait on an mbarrier that nothing ever completes: the wait runs
// out after the current poll limit, the kernel records it in the status word
// like a step kernel whose copies were lost, and returns.  No copy is in
// flight, so giving up is harmless; used to test the failure path.
__global__ void wait_selftest_kernel() {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if (!mbar_wait(&bar, 0)) atomicExch(&g_march_status, 1);
    }
}

int launch_wait_selftest(cudaStream_t st) {
    wait_selftest_kernel<<<1, 32, 0, st>>>();
    return check_launch("wait_selftest_kernel");
}

// Binary version (major*10 + minor) of the device code the library loaded.
int kernel_binary_version(int *v) {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, displacement_traces_kernel);
    if (e != cudaSuccess) return set_error(FWI_ECUDA, "cudaFuncGetAttributes: %s", cudaGetErrorString(e));
    *v = fa.binaryVersion;
    return 0;
}

int launch_displacement_traces(float *obs, long long ntr, int nt, int it0, int n, double dt, cudaStream_t st) {
    if (ntr <= 0 || n <= 0) return 0;
    const int th = 128;
    displacement_traces_kernel<<<(unsigned)((ntr + th - 1) / th), th, 0, st>>>(obs, ntr, nt, it0, n, (float)dt);
    return check_launch("displacement_traces_kernel");
}

}  // namespace fwi

cudaError_t fwi::march_set_wait_limit(int polls) { return fwi::set_wait_limit_here(polls); }
