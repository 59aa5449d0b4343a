// k_pair32.cuh -- the particle loop of the FP32 form's full substep, two
// particles of a cell per lane and iteration (included by k_tiles.cuh).
//
// One lane owns one grid cell and walks its particles two at a time. Nearly
// all FP32 arithmetic -- B-spline weights, G2P, the strain update, the
// invariants and the stress, P2G -- is done for both particles at once in
// the two halves of sm_100's packed f32x2 instructions, and the bookkeeping,
// the loads of the cell's 9 node velocities and the branches are paid once
// for two particles.
#pragma once

namespace icm {

__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }

// The 27 P2G sums of one cell: momentum, and the sums of the weights (the
// mass is a common factor). One partial sum per half would save 18
// multiply-adds a pair but holds 18 more registers, which the third warp
// per scheduler and then some would pay for.
struct PairSums {
    float x[9], y[9], m[9];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int q = 0; q < 9; q++) x[q] = y[q] = m[q] = 0.f;
    }
    __device__ __forceinline__ void add(int q, const float2 W, const float2 a0, const float2 a1)
    {
        m[q] += W.x + W.y;
        x[q] = fmaf(W.x, a0.x, fmaf(W.y, a0.y, x[q]));
        y[q] = fmaf(W.x, a1.x, fmaf(W.y, a1.y, y[q]));
    }
    __device__ __forceinline__ void flush(float4 &ac, int q, float mass) const
    {
        const float4 v = ac;
        ac = make_float4(v.x + x[q], v.y + y[q], fmaf(mass, m[q], v.z), v.w);
    }
};

// B-spline weight of node c (0, 1, 2) for two particles, from
// g = X - 1/2 - base in [0, 1]
__device__ __forceinline__ float2 pair_weight(const float2 g, int c)
{
    if (c == 1) {
        const float2 d = __fadd2_rn(g, bcast2(-0.5f));
        return __ffma2_rn(make_float2(-d.x, -d.y), d, bcast2(0.75f));
    }
    const float2 a = c == 0 ? __fadd2_rn(bcast2(1.0f), make_float2(-g.x, -g.y)) : g;
    return __fmul2_rn(__fmul2_rn(bcast2(0.5f), a), a);
}

__device__ __forceinline__ float pair_weight_at(const float g, int c)
{
    if (c == 1) return 0.75f - (g - 0.5f) * (g - 0.5f);
    const float a = c == 0 ? 1.0f - g : g;
    return 0.5f * a * a;
}

// The packed base node of a position (cell word and fixed-point fractions):
// base = floor(X - 1/2). Below the grid (X < 1/2, where the reference
// truncates towards zero) and for cells outside [0, 32767] it equals no
// cell of the grid, and the particle takes the general path.
__device__ __forceinline__ uint32_t pair_base(uint32_t cell, uint32_t ux, uint32_t uy)
{
    return cell + (ux >> 31) + ((uy >> 31) << 16) - 0x00010001u;
}

// g of a fixed-point fraction: the fraction of X - 1/2, rounded for use only
__device__ __forceinline__ float2 pair_g(uint32_t ua, uint32_t ub)
{
    return __fmul2_rn(make_float2(__uint2float_rn(ua ^ 0x80000000u), __uint2float_rn(ub ^ 0x80000000u)),
                      bcast2(2.3283064365386963e-10f));
}

// G2P of one particle from the region's velocities; n points at its base
// node, g as in pair_g. Bp lacks the factor 4/h.
__device__ __forceinline__ G2POut<float> pair_gather(const float4 *n, const int RX, const float gx, const float gy)
{
    const float vc0 = n[RX + 1].x, vc1 = n[RX + 1].z;
    float wy[3], wyd[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        wy[j] = pair_weight(bcast2(gy), j).x;
        wyd[j] = wy[j] * ((float)j - 0.5f - gy);
    }
    G2POut<float> o{0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 3; i++) {
        float a0 = 0, a1 = 0, b0 = 0, b1 = 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const float4 v = n[j * RX + i];
            const float n0 = v.x - vc0, n1 = v.z - vc1;
            a0 += wy[j] * n0;
            a1 += wy[j] * n1;
            b0 += wyd[j] * n0;
            b1 += wyd[j] * n1;
        }
        const float wx = pair_weight(bcast2(gx), i).x, wxd = wx * ((float)i - 0.5f - gx);
        o.v0 += wx * a0;
        o.v1 += wx * a1;
        o.B0 += wxd * a0;
        o.B2 += wxd * a1;
        o.B1 += wx * b0;
        o.B3 += wx * b1;
    }
    o.v0 += vc0;  // sum W = 1
    o.v1 += vc1;
    return o;
}

__device__ __forceinline__ bool pair_in_grid(uint32_t base, int GX, int GY)
{
    return cell_x(base) >= 0 && cell_y(base) >= 0 && cell_x(base) + 2 < GX && cell_y(base) + 2 < GY;
}

// P2G of one particle by the whole warp: lane q < 9 adds the particle's
// contribution to node (q / 3, q % 3) of its stencil -- plain additions to
// the warp's region where the stencil lies inside it (float additions to
// shared memory compile to compare-and-swap loops, 27 of them a particle:
// 11,000 cycles for the first stray of an iteration, now about 150), vector
// reductions into the scatter buffer beyond it. c = (u0, u1, S00, S01),
// d = (S10, S11, gx, gy) as in the pair loop; the base is inside the grid.
template <int TX, int TY>
__device__ __forceinline__ void pair_scatter(const TileRun &R, const int GX, const int rx0, const int ry0, float4 *wacc,
                                             const uint32_t base, const float4 c, const float4 d, const float mass)
{
    constexpr int RX = TX + 4, RY = TY + 4;
    const int lane = threadIdx.x & 31, i = lane / 3, j = lane % 3;
    if (lane < 9) {
        const float W = pair_weight_at(d.z, i) * pair_weight_at(d.w, j);
        const float m = W * mass, x = W * (c.x + (float)i * c.z + (float)j * c.w),
                    y = W * (c.y + (float)i * d.x + (float)j * d.y);
        const int gx = cell_x(base) + i, gy = cell_y(base) + j, lx = cell_x(base) - rx0, ly = cell_y(base) - ry0;
        if (lx >= 0 && ly >= 0 && lx + 2 < RX && ly + 2 < RY) {
            acc_add(wacc[(ly + j) * RX + lx + i], m, x, y);
        } else {
            node_add_global((float4 *)R.gB, (size_t)gy * GX + gx, m, x, y);
            R.dB[(gy / TY) * R.ntx + gx / TX] = 1;
        }
    }
    __syncwarp();
}

// The whole substep of one particle that the pair loop leaves aside (out of
// line): one whose constitutive step needs FP64, and one whose stencil leaves
// the CTA's node region before the substep or the grid after it. G2P from the CTA's node region or node by
// node beyond it, advection, Pol32's constitutive step, store, and P2G with
// shared or global atomics. (cbx, cby) is the cell it was binned to.
struct Deferred { int bad, redo, stray; };

template <int TX, int TY>
static __device__ __noinline__ Deferred pair_deferred(const icy_SimParams &P, const Consts32 &K, const Parts32 &A,
                                                      const TileRun &R, const int p, const float4 *s_v, float4 *wacc,
                                                      const int rx0, const int ry0, const int cbx, const int cby)
{
    constexpr int RX = TX + 4, RY = TY + 4;
    Pol32::St s = Pol32::load(A, p);
    const float jp_old = s.Jp;
    G2POut<float> o{0, 0, 0, 0, 0, 0};
    {
        const Pol32::Sten st = Pol32::stencil(P, K, s);
        const int lx = st.bx - rx0, ly = st.by - ry0;
        if (lx >= 0 && ly >= 0 && lx + 2 < RX && ly + 2 < RY && st.bx >= 0 && st.by >= 0 && st.bx + 2 < P.GridX &&
            st.by + 2 < P.GridY) {
            const int q0 = ly * RX + lx;
            const float vc0 = s_v[q0 + RX + 1].x, vc1 = s_v[q0 + RX + 1].z;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                float a0 = 0, a1 = 0, b0 = 0, b1 = 0;
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const float4 n = s_v[q0 + j * RX + i];
                    const float n0 = n.x - vc0, n1 = n.z - vc1, wyd = st.wy[j] * ((float)j - st.fy);
                    a0 += st.wy[j] * n0;
                    a1 += st.wy[j] * n1;
                    b0 += wyd * n0;
                    b1 += wyd * n1;
                }
                const float wxd = st.wx[i] * ((float)i - st.fx);
                o.v0 += st.wx[i] * a0;
                o.v1 += st.wx[i] * a1;
                o.B0 += wxd * a0;
                o.B2 += wxd * a1;
                o.B1 += st.wx[i] * b0;
                o.B3 += st.wx[i] * b1;
            }
            o.B0 *= K.four_h_inv; o.B1 *= K.four_h_inv; o.B2 *= K.four_h_inv; o.B3 *= K.four_h_inv;
            o.v0 += vc0;  // sum W = 1
            o.v1 += vc1;
        } else {
            o = far_gather<Pol32>(P, K, (const float4 *)R.gA, st.bx, st.by, st.fx, st.fy, st.wx[0], st.wx[1],
                                  st.wx[2], st.wy[0], st.wy[1], st.wy[2], R.ind_x, R.ind_y);
        }
    }
    Deferred d{0, 0, 0};
    const float B[4] = {o.B0, o.B1, o.B2, o.B3};
    float p_tr, q_tr;
    const Tau<float> tau = Pol32::advance(P, K, GrainStrengths32{K}, s, o.v0, o.v1, B, p_tr, q_tr, d.redo);
    Pol32::store(A, p, s, jp_old, 0u);
    if (R.record_pq) A.pq[p] = make_float2(p_tr, q_tr);
    const Pol32::Sten st = Pol32::stencil(P, K, s);
    d.stray = !(st.bx == cbx && st.by == cby && cbx + 2 < P.GridX && cby + 2 < P.GridY);
    const float m = K.mass, h = K.h, sc = K.stress_c;
    const float S00 = h * (m * B[0] - sc * tau.t00), S01 = h * (m * B[1] - sc * tau.t01);
    const float S10 = h * (m * B[2] - sc * tau.t10), S11 = h * (m * B[3] - sc * tau.t11);
    d.bad = stray_p2g<Pol32, TX, TY>(wacc, rx0, ry0, P.GridX, P.GridY, (float4 *)R.gB, R.dB, R.ntx,
                                     st.bx, st.by, st.wx[0], st.wx[1], st.wx[2], st.wy[0], st.wy[1], st.wy[2], m,
                                     o.v0 * m - (S00 * st.fx + S01 * st.fy), o.v1 * m - (S10 * st.fx + S11 * st.fy), S00,
                                     S01, S10, S11);
    return d;
}

// The listed nodes' velocities, in place, and the reaction of those that the
// tile owns (count) to the force bins: as Pol32::node_velocity. The last
// threads take them, which have the fewest of the region's other nodes.
template <int TX, int TY>
static __device__ __noinline__ void pair_contact_nodes(const icy_SimParams &P, const Consts32 &K, const TileRun &R,
                                                       const int x0, const int y0, const bool count, const bool staged,
                                                       float4 *s_v, const ContactList C)
{
    constexpr int RX = TX + 4;
    const int nthr = blockDim.x, n = *C.n;
    const float4 *gA = (const float4 *)R.gA;
    NodeForce force;
    for (int e = nthr - 1 - (int)threadIdx.x; e < n; e += nthr) {
        const int k = C.code[e] & 0xffff, bin = C.code[e] >> 16, x = x0 - 1 + k % RX, y = y0 - 1 + k / RX;
        const double2 nrm = C.normal[e];
        float4 nd = make_float4(0.f, 0.f, 0.f, 0.f);
        if (staged) nd = s_v[k];
        else if (x >= 0 && y >= 0 && x < P.GridX && y < P.GridY) nd = gA[(size_t)y * P.GridX + x];
        float a, b;
        double f0, f1;
        if (Pol32::contact_velocity(P, K, nd, x, y, nrm.x, nrm.y, a, b, f0, f1) && count && x >= x0 && x < x0 + TX &&
            y >= y0 && y < y0 + TY)
            force.add(R, bin, f0, f1);
        s_v[k] = make_float4(a, a, b, b);
    }
    force.total(R);
}

// The node region's copy did not complete within the poll limit: the thread
// raises the error word, gives the copy a second chance to land before its
// space is written, and reads its nodes with plain loads instead.
static __device__ __noinline__ void pair_copy_late(uint64_t *bar, int *err)
{
    atomicOr(err, kErrTmaTimeout);
    tc05::mbar_wait(bar, 0, kTmaPolls);
}

// iterations of a group that the pair loop walks (a bit per particle says
// which it leaves aside); the particles of a cell beyond them take
// pair_deferred
constexpr int kPairIters = 32;
// warps per CTA at most (512 threads of 128 registers fill an SM)
constexpr int kPairMaxWarps = 16;
// threads per cell of a tile at most: with one warp per 16 cells two warps
// share a group, each taking every second pair of its rounds
constexpr int kPairWidest = 2;

// Dynamic shared memory of a CTA: the node region (as the tensor copy
// delivers it, then in place the velocities as {vx, vx, vy, vy}, so that one
// load gives both halves), the warps' P2G regions, and two staging buffers
// per warp. The second staging buffers hold the list of contact nodes until
// the particle loop starts.
__host__ __device__ constexpr size_t pair_dyn_bytes(int RN, int nwarps)
{
    const size_t stage = (size_t)nwarps * sizeof(Pol32::PairStage), bins = contact_bytes(RN);
    return (size_t)RN * 16 * (1 + nwarps) + stage + (stage > bins ? stage : bins);
}

// The place q of a warp's j-th group in the CTA's lists: the groups' order
// (group_of), or with more warps than groups the warp itself.
template <bool WIDE> __device__ __forceinline__ int pair_place(int j, int warp, int nwarps)
{
    if (WIDE) return j == 0 ? warp : kPairMaxWarps;
    return group_of(j, warp, nwarps, 0);
}

// The particles that a warp left aside, and those of a cell beyond its
// kPairIters iterations (out of line: the common path keeps no registers for it).
// They are dealt out to the lanes, 32 particles of a cell at a time, through a
// list of slots in the warp's staging space.
template <int TX, int TY, bool WIDE>
static __device__ __noinline__ void pair_aside(const icy_SimParams &P, const Consts32 &K, const Parts32 &A,
                                               const TileRun &R, const int x0, const int y0, const int step,
                                               const float4 *s_v, float4 *wacc, Pol32::PairStage *stage,
                                               const int2 *s_group, const uint32_t (*s_wc)[32],
                                               const unsigned long long (*s_aside)[32])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // 1,024 slots at most, 512 in each of the two staging buffers
    int *list = reinterpret_cast<int *>(stage);
    const int list_stride = nwarps * (int)(sizeof(Pol32::PairStage) / sizeof(int));
    int bad = 0;
    unsigned redo_count = 0, stray_count = 0;
    constexpr int kPlaces = WIDE ? kPairMaxWarps : TX * TY / 32;
    for (int j = 0, q; (q = pair_place<WIDE>(j, warp, nwarps)) < kPlaces; j++) {
        const int2 g = s_group[q];
        if (g.y <= 0) break;
        const unsigned long long aside = s_aside[q][lane];
        const int cl = (int)(s_wc[q][lane] >> kLaneCountBits);
        // 32 particles of each cell at a time: particle r of the part's is
        // in round (r / 2) step + r % 2
        for (int r0 = 0; (r0 >> 1) * step < g.y; r0 += 32) {
            unsigned bits = r0 == 0 ? (unsigned)aside : (unsigned)(aside >> 32);
            if (r0 >= 2 * kPairIters) {
                const int cnt = (int)(s_wc[q][lane] & kLaneCountMask);
                bits = 0;
                for (int r = 0; r < 32; r++)
                    if (((r0 + r) >> 1) * step + (r & 1) < cnt) bits |= 1u << r;
            }
            if (!__any_sync(0xffffffffu, bits != 0u)) continue;
            int at = __popc(bits);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, at, o);
                if (lane >= o) at += y;
            }
            const int total = __shfl_sync(0xffffffffu, at, 31);
            at -= __popc(bits);
            __syncwarp();
            for (; bits; bits &= bits - 1, at++)
            {
                const int r = r0 + __ffs(bits) - 1;
                list[(at >> 9) * list_stride + (at & 511)] = g.x + 32 * ((r >> 1) * step + (r & 1)) + lane;
            }
            __syncwarp();
            for (int b = lane; b - lane < total; b += 32) {
                const int slot = b < total ? list[(b >> 9) * list_stride + (b & 511)] : 0;
                // the cell it was binned to: that of the slot's lane
                const int c = __shfl_sync(0xffffffffu, cl, slot & 31);
                if (b >= total) continue;
                const Deferred d =
                    pair_deferred<TX, TY>(P, K, A, R, slot, s_v, wacc, x0 - 1, y0 - 1, x0 + c % TX, y0 + c / TX);
                bad |= d.bad;
                redo_count += d.redo;
                stray_count += d.stray;
            }
        }
    }
    if (stray_count && R.strays) atomicAdd(R.strays, (unsigned long long)stray_count);
    if (bad) *R.err = 1;
    if (redo_count && R.fp64_redo) atomicAdd(R.fp64_redo, (unsigned long long)redo_count);
}

// One substep of one tile with particles, as tile_body (k_tiles.cuh) but for
// the pair loop. Every return is uniform over the CTA.
template <int TX, int TY, bool WIDE>
__device__ __forceinline__ void pair_tile_body(const icy_SimParams &P, const Consts32 &K, const Parts32 &A,
                                               const TileRun &R, const int t, const CUtensorMap *tmaps,
                                               const bool tmaps_in_global, const int part)
{
    constexpr int RX = TX + 4, RY = TY + 4, RN = RX * RY, CELLS = TX * TY, NGT = CELLS / 32;
    extern __shared__ __align__(128) unsigned char s_dyn[];
    __shared__ uint64_t s_tma_bar;
    __shared__ int s_any;  // a warp left a particle aside
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    float4 *s_v = reinterpret_cast<float4 *>(s_dyn);
    float4 *s_acc = s_v + RN, *wacc = s_acc + warp * RN;
    Pol32::PairStage *s_stage = reinterpret_cast<Pol32::PairStage *>(s_acc + nwarps * RN);
    const ContactList s_con(s_stage + nwarps, RN);
    const int tx = t % R.ntx, ty = t / R.ntx;
    const int x0 = tx * TX, y0 = ty * TY, rx0 = x0 - 1, ry0 = y0 - 1;
    const int GX = P.GridX, GY = P.GridY;

    // What depends only on the binning is read before the wait for the
    // previous substep: of each of the warp's groups the lane words and the
    // first slot and rounds (the fullest groups come first, so a group
    // without rounds ends the list). With more warps than groups (WIDE) nip
    // warps share each group and take every nip-th pair of its rounds; the
    // words and rounds then count from the warp's first pair on.
    constexpr int kPlaces = WIDE ? kPairMaxWarps : NGT;
    const int nip = WIDE ? nwarps / NGT : 1, ip = WIDE ? warp / NGT : 0;
    __shared__ uint32_t s_wc[kPlaces][32];
    __shared__ unsigned long long s_aside[kPlaces][32];  // bit r: the lane's particle r is left aside
    __shared__ int2 s_group[kPlaces];
    {
        constexpr int NJ = 2;  // loads in flight together
        for (int j0 = 0; pair_place<WIDE>(j0, warp, nwarps) < kPlaces; j0 += NJ) {
            uint32_t w[NJ];
            int b0[NJ], b1[NJ];
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int q = pair_place<WIDE>(j0 + j, warp, nwarps);
                const int g = q - (WIDE ? ip * NGT : 0), m = part == 0 ? g : 2 * g + (part - 1);
                w[j] = 0u;
                b0[j] = b1[j] = 0;
                if (q < kPlaces && m < NGT) {
                    w[j] = R.lane_cell[t * CELLS + m * 32 + lane];
                    b0[j] = R.group_base[t * NGT + m];
                    b1[j] = R.group_base[t * NGT + m + 1];
                }
            }
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int q = pair_place<WIDE>(j0 + j, warp, nwarps);
                if (q >= kPlaces) continue;
                const int cnt = (int)(w[j] & kLaneCountMask);
                if (cnt > 0xffff) atomicOr(R.err, kErrCellOverflow);  // the cell's later particles are not advanced
                s_wc[q][lane] = (w[j] & ~kLaneCountMask) | (uint32_t)max(min(cnt, 0xffff) - 2 * ip, 0);
                if (lane == 0) s_group[q] = make_int2(b0[j] + 64 * ip, ((b1[j] - b0[j]) >> 5) - 2 * ip);
            }
        }
    }
    __syncwarp();
    // the warp's j-th group and its place (no rounds: no more groups)
    auto group = [&](int j, int &q) {
        q = pair_place<WIDE>(j, warp, nwarps);
        return q < kPlaces ? s_group[q] : make_int2(0, 0);
    };
    // rounds of an iteration: the group's other warps take those in between
    const int step = WIDE ? 2 * nip : 2;
    const bool busy = R.group_base[t * NGT + 1] > R.group_base[t * NGT];
    const bool contact = region_touches_indenter<TX, TY>(P, R, t);
    const bool staging = tmaps && (tc05::smem_u32(s_dyn) & 127u) == 0;
    if (staging && tid == 0) {
        if (tmaps_in_global)
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(tmaps + R.bufA) : "memory");
        tc05::mbar_init(&s_tma_bar, 1);
    }
    if (tid == 0) s_any = 0;
    if (contact && busy) {
        for (int k = tid; k < 1 + contact_mask_words(RN); k += nthr) s_con.n[k] = 0;  // the mask behind it
        __syncthreads();
        contact_list<TX, TY>(P, R, x0, y0, s_con);
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!busy) {
        const bool z = part != 2 && R.dC[t], c = part != 2 && contact && R.dA[t];
        empty_tile<Pol32, TX, TY>(P, K, R, t, z, c);
        __syncthreads();  // every thread has read the flag
        if (z && tid == 0) R.dC[t] = 0;
        return;
    }
    // the node region and the first particles come in while the CTA zeroes
    // its accumulators and its nodes in the next-but-one buffer
    if (staging && tid == 0) tma_region_load(tmaps + R.bufA, s_v, rx0, ry0, (uint32_t)(RN * 16), &s_tma_bar);
    auto issue = [&](int left, int p, Pol32::PairStage &S) {
        if (left > 0) {
            __pipeline_memcpy_async(&S.X[0][lane], &A.X[p], 16);
            __pipeline_memcpy_async(&S.H[0][lane], &A.H[p], 16);
            __pipeline_memcpy_async(&S.Jp[0][lane], &A.Jp[p], 4);
        }
        if (left > 1) {
            __pipeline_memcpy_async(&S.X[1][lane], &A.X[p + 32], 16);
            __pipeline_memcpy_async(&S.H[1][lane], &A.H[p + 32], 16);
            __pipeline_memcpy_async(&S.Jp[1][lane], &A.Jp[p + 32], 4);
        }
    };
    int q;
    int2 g = group(0, q);
    if (g.y > 0) issue((int)(s_wc[q][lane] & kLaneCountMask), g.x + lane, s_stage[warp]);
    __pipeline_commit();
    for (int k = lane; k < RN; k += 32) acc_zero(wacc[k]);
    // grid update of the region, in place (node k and its velocity share
    // their 16 bytes; nodes beyond the grid read as zero). Four nodes per
    // thread and pass, so that their loads and divisions overlap.
    bool staged = staging && tc05::mbar_wait(&s_tma_bar, 0, kTmaPolls);
    if (staging && !staged) pair_copy_late(&s_tma_bar, R.err);
    if (contact) pair_contact_nodes<TX, TY>(P, K, R, x0, y0, part != 2, staged, s_v, s_con);
    {
        const float4 *gA = (const float4 *)R.gA;
        const bool edge = rx0 <= 2 || ry0 <= 2 || rx0 + RX > GX - 3 || ry0 + RY > GY - 3;
        const int dkx = nthr % RX, dky = nthr / RX;
        int kx = tid % RX, ky = tid / RX;
        constexpr int NB = 4;
        for (int k0 = tid; k0 < RN; k0 += NB * nthr) {
            float4 nd[NB];
            int gx[NB], gy[NB];
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const int k = k0 + b * nthr;
                gx[b] = rx0 + kx;
                gy[b] = ry0 + ky;
                kx += dkx;
                ky += dky;
                if (kx >= RX) { kx -= RX; ky++; }
                nd[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k < RN) {
                    if (staged) nd[b] = s_v[k];
                    else if (gx[b] >= 0 && gy[b] >= 0 && gx[b] < GX && gy[b] < GY) nd[b] = gA[(size_t)gy[b] * GX + gx[b]];
                }
            }
            float va[NB], vb[NB];
#pragma unroll
            for (int b = 0; b < NB; b++) {  // Pol32::node_velocity beyond the indenter's reach
                const float m = nd[b].x;
                const float inv_m = 1.0f / (m != 0.0f ? m : 1.0f);
                float a = nd[b].y * inv_m, c = nd[b].z * inv_m;
                c -= K.dt_g;
                const float n2 = a * a + c * c;
                if (n2 > K.vmax * K.vmax) {
                    const float sc = K.vmax * rsqrtf(n2);
                    a *= sc;
                    c *= sc;
                }
                va[b] = m != 0.0f ? a : 0.0f;
                vb[b] = m != 0.0f ? c : 0.0f;
            }
            if (edge) {
#pragma unroll
                for (int b = 0; b < NB; b++) {
                    if (gy[b] <= 2) { va[b] = 0.0f; vb[b] = 0.0f; }
                    else if (gy[b] >= GY - 3 && vb[b] > 0.0f) vb[b] = 0.0f;
                    if (gx[b] <= 2 && va[b] < 0.0f) va[b] = 0.0f;
                    else if (gx[b] >= GX - 3 && va[b] > 0.0f) va[b] = 0.0f;
                }
            }
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const int k = k0 + b * nthr;
                if (k >= RN || (contact && (s_con.mask[k >> 5] >> (k & 31) & 1))) continue;
                s_v[k] = make_float4(va[b], va[b], vb[b], vb[b]);
            }
        }
    }
    __syncthreads();

    // the particles of the warp's groups
    int stage = 0;
    for (int gj = 0; g.y > 0; gj++) {
        const uint32_t wc = s_wc[q][lane];
        const int cnt = (int)(wc & kLaneCountMask), cl = (int)(wc >> kLaneCountBits);
        const int iters = min((g.y + step - 1) / step, kPairIters);
        const int clx = cl % TX, cly = cl / TX, cbx = x0 + clx, cby = y0 + cly;
        // a cell whose stencil leaves the grid sends every particle down the
        // general path, which raises the error word as v2_kernel_p2g does
        const bool cell_ok = cbx + 2 < GX && cby + 2 < GY;
        const uint32_t cell_base = (uint32_t)cbx | ((uint32_t)cby << 16);
        const int q0 = (cly + 1) * RX + (clx + 1);  // the cell's base node in the region
        PairSums sums;
        sums.zero();
        s_aside[q][lane] = 0;
        for (int i = 0; i < iters; i++) {
            {
                Pol32::PairStage &N = s_stage[(stage ^ 1) * nwarps + warp];
                if (i + 1 < iters) {
                    issue(cnt - step * (i + 1), g.x + 32 * step * (i + 1) + lane, N);
                } else {
                    int qn;
                    const int2 gn = group(gj + 1, qn);
                    if (gn.y > 0) issue((int)(s_wc[qn][lane] & kLaneCountMask), gn.x + lane, N);
                }
            }
            __pipeline_commit();
            __pipeline_wait_prior(1);
            const Pol32::PairStage &S = s_stage[stage * nwarps + warp];
            stage ^= 1;
            bool out_a = false, out_b = false;  // out of the cell: scattered below
            if (step * i < cnt) {
                // a missing second particle is computed as a copy of the first
                // and takes no part in stores and sums
                const bool has1 = step * i + 1 < cnt;
                const int p = g.x + 32 * step * i + lane;
                const int h1 = has1 ? 1 : 0;
                float4 Xa = S.X[0][lane], Xb = S.X[h1][lane];
                uint32_t uxa = __float_as_uint(Xa.x), uya = __float_as_uint(Xa.y), ca = __float_as_uint(Xa.z),
                         ma = __float_as_uint(Xa.w);
                uint32_t uxb = __float_as_uint(Xb.x), uyb = __float_as_uint(Xb.y), cb = __float_as_uint(Xb.z),
                         mb = __float_as_uint(Xb.w);
                // on: the pair loop settles the particle (it is not left aside)
                bool on_a = true, on_b = has1;

                // G2P (Bp from velocities relative to the centre node, as Pol32)
                float2 v0, v1, B0, B1, B2, B3;
                {
                    const float2 gx = pair_g(uxa, uxb), gy = pair_g(uya, uyb);
                    float2 wy[3], wyd[3];
#pragma unroll
                    for (int j = 0; j < 3; j++) wy[j] = pair_weight(gy, j);
                    const float2 ngy = make_float2(-gy.x, -gy.y), ngx = make_float2(-gx.x, -gx.y);
                    wyd[0] = __fmul2_rn(wy[0], __fadd2_rn(ngy, bcast2(-0.5f)));
                    wyd[1] = __fmul2_rn(wy[1], __fadd2_rn(ngy, bcast2(0.5f)));
                    wyd[2] = __fmul2_rn(wy[2], __fadd2_rn(ngy, bcast2(1.5f)));
                    const float4 vc = s_v[q0 + RX + 1];
                    const float2 nc0 = make_float2(-vc.x, -vc.y), nc1 = make_float2(-vc.z, -vc.w);
                    v0 = v1 = B0 = B1 = B2 = B3 = make_float2(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        float2 a0, a1, b0, b1;
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            if (c == 1 && j == 1) continue;  // the centre node itself: zero
                            const float4 n = s_v[q0 + j * RX + c];
                            const float2 n0 = __fadd2_rn(make_float2(n.x, n.y), nc0);
                            const float2 n1 = __fadd2_rn(make_float2(n.z, n.w), nc1);
                            if (j == 0) {
                                a0 = __fmul2_rn(wy[0], n0);
                                a1 = __fmul2_rn(wy[0], n1);
                                b0 = __fmul2_rn(wyd[0], n0);
                                b1 = __fmul2_rn(wyd[0], n1);
                            } else {
                                a0 = __ffma2_rn(wy[j], n0, a0);
                                a1 = __ffma2_rn(wy[j], n1, a1);
                                b0 = __ffma2_rn(wyd[j], n0, b0);
                                b1 = __ffma2_rn(wyd[j], n1, b1);
                            }
                        }
                        const float2 wx = pair_weight(gx, c);
                        const float2 wxd = __fmul2_rn(wx, __fadd2_rn(ngx, bcast2((float)c - 0.5f)));
                        v0 = __ffma2_rn(wx, a0, v0);
                        v1 = __ffma2_rn(wx, a1, v1);
                        B0 = __ffma2_rn(wxd, a0, B0);
                        B2 = __ffma2_rn(wxd, a1, B2);
                        B1 = __ffma2_rn(wx, b0, B1);
                        B3 = __ffma2_rn(wx, b1, B3);
                    }
                    const float2 f = bcast2(K.four_h_inv);
                    v0 = __fadd2_rn(v0, make_float2(vc.x, vc.y));  // sum W = 1
                    v1 = __fadd2_rn(v1, make_float2(vc.z, vc.w));
                    // a particle that left its cell gathers on its own from
                    // the region (beyond the region it is left aside)
                    const bool out_a = !(cell_ok && pair_base(ca, uxa, uya) == cell_base);
                    const bool out_b = has1 && !(cell_ok && pair_base(cb, uxb, uyb) == cell_base);
                    if (out_a || out_b) {
#pragma unroll 1
                        for (int h = out_a ? 0 : 1; h < (out_b ? 2 : 1); h++) {
                            const uint32_t wb = h ? pair_base(cb, uxb, uyb) : pair_base(ca, uxa, uya);
                            const int bx = cell_x(wb), by = cell_y(wb), lx = bx - rx0, ly = by - ry0;
                            if (!(bx >= 0 && by >= 0 && lx >= 0 && ly >= 0 && lx + 2 < RX && ly + 2 < RY && bx + 2 < GX &&
                                  by + 2 < GY)) {
                                if (h) on_b = false;
                                else on_a = false;
                                continue;
                            }
                            const G2POut<float> o = pair_gather(s_v + ly * RX + lx, RX, h ? gx.y : gx.x, h ? gy.y : gy.x);
                            if (h) { v0.y = o.v0; v1.y = o.v1; B0.y = o.B0; B1.y = o.B1; B2.y = o.B2; B3.y = o.B3; }
                            else { v0.x = o.v0; v1.x = o.v1; B0.x = o.B0; B1.x = o.B1; B2.x = o.B2; B3.x = o.B3; }
                        }
                    }
                    B0 = __fmul2_rn(B0, f);
                    B1 = __fmul2_rn(B1, f);
                    B2 = __fmul2_rn(B2, f);
                    B3 = __fmul2_rn(B3, f);
                }
                // advection (Pol32::advect): displacement in units of 2^-32
                // cells added to the fixed-point fraction, carries to the cell
                {
                    const float2 d0 = __fmul2_rn(__fmul2_rn(v0, bcast2(K.dt_h_inv)), bcast2(4294967296.0f));
                    const float2 d1 = __fmul2_rn(__fmul2_rn(v1, bcast2(K.dt_h_inv)), bcast2(4294967296.0f));
                    const long long xa = (long long)uxa + __float2ll_rn(d0.x), ya = (long long)uya + __float2ll_rn(d1.x);
                    const long long xb = (long long)uxb + __float2ll_rn(d0.y), yb = (long long)uyb + __float2ll_rn(d1.y);
                    ca = __byte_perm(ca + (uint32_t)(xa >> 32), (ca >> 16) + (uint32_t)(ya >> 32), 0x5410);
                    cb = __byte_perm(cb + (uint32_t)(xb >> 32), (cb >> 16) + (uint32_t)(yb >> 32), 0x5410);
                    uxa = (uint32_t)xa; uya = (uint32_t)ya;
                    uxb = (uint32_t)xb; uyb = (uint32_t)yb;
                }
                // in: the particle adds to its cell's sums; out of its cell
                // it scatters on its own, or is left aside where a node of
                // its stencil lies beyond the grid
                const bool in_a = cell_ok && pair_base(ca, uxa, uya) == cell_base;
                const bool in_b = cell_ok && pair_base(cb, uxb, uyb) == cell_base;
                if (!in_a) on_a = on_a && pair_in_grid(pair_base(ca, uxa, uya), GX, GY);
                if (!in_b) on_b = on_b && pair_in_grid(pair_base(cb, uxb, uyb), GX, GY);
                // H_new = H + dt (C + C H)
                float2 H0, H1, H2, H3;
                {
                    const float4 Ha = S.H[0][lane], Hb = S.H[h1][lane];
                    const float2 h0 = make_float2(Ha.x, Hb.x), h1_ = make_float2(Ha.y, Hb.y), h2 = make_float2(Ha.z, Hb.z),
                                 h3 = make_float2(Ha.w, Hb.w), dt = bcast2(K.dt);
                    const float2 c0 = __fmul2_rn(dt, B0), c1 = __fmul2_rn(dt, B1), c2 = __fmul2_rn(dt, B2),
                                 c3 = __fmul2_rn(dt, B3);
                    H0 = __fadd2_rn(h0, __ffma2_rn(c0, h0, __ffma2_rn(c1, h2, c0)));
                    H1 = __fadd2_rn(h1_, __ffma2_rn(c0, h1_, __ffma2_rn(c1, h3, c1)));
                    H2 = __fadd2_rn(h2, __ffma2_rn(c2, h0, __ffma2_rn(c3, h2, c2)));
                    H3 = __fadd2_rn(h3, __ffma2_rn(c2, h1_, __ffma2_rn(c3, h3, c3)));
                }
                // invariants and stress (invariants32, tau32)
                float2 t00, t01, t11;
                {
                    const float2 nH1 = make_float2(-H1.x, -H1.y), nH2 = make_float2(-H2.x, -H2.y),
                                 nH3 = make_float2(-H3.x, -H3.y);
                    const float2 tr = __fadd2_rn(H0, H3);
                    const float2 Jm1 = __fadd2_rn(tr, __ffma2_rn(H0, H3, __fmul2_rn(nH1, H2)));
                    const float2 J = __fadd2_rn(Jm1, bcast2(1.0f));
                    const float2 b01 = __fadd2_rn(__fadd2_rn(H1, H2), __ffma2_rn(H0, H2, __fmul2_rn(H1, H3)));
                    const float2 hd =
                        __ffma2_rn(__fadd2_rn(H0, nH3), __ffma2_rn(bcast2(0.5f), tr, bcast2(1.0f)),
                                   __fmul2_rn(__fmul2_rn(bcast2(0.5f), __fadd2_rn(H1, nH2)), __fadd2_rn(H1, H2)));
                    const float2 s1 = make_float2(__fdividef(K.mu, J.x), __fdividef(K.mu, J.y));
                    const float2 s2 = __fmul2_rn(__fmul2_rn(bcast2(K.kappa), Jm1), __fadd2_rn(J, bcast2(1.0f)));
                    t00 = __ffma2_rn(s1, hd, s2);
                    t01 = __fmul2_rn(s1, b01);
                    t11 = __ffma2_rn(make_float2(-s1.x, -s1.y), hd, s2);
                    // settled here: an intact particle of a grain with a
                    // non-negative id whose (p, q) lies in the box inside every
                    // failure surface (p = -s2/2, q = 2 s1 |(hd, b01)|; MPa)
                    const float2 pm = __fmul2_rn(s2, bcast2(-0.5e-6f));
                    const float2 qs = __fmul2_rn(s1, bcast2(2e-6f));
                    const float2 r2 = __ffma2_rn(hd, hd, __fmul2_rn(b01, b01));
                    const float2 q2 = __fmul2_rn(__fmul2_rn(qs, qs), r2);
                    const uint32_t kind = kMetaNonNeg | kMetaCrushed;
                    const bool box_a = (ma & kind) == kMetaNonNeg && J.x > 0.25f && pm.x > K.inside_plo &&
                                       pm.x < K.inside_phi && q2.x < K.inside_q2;
                    const bool box_b = (mb & kind) == kMetaNonNeg && J.y > 0.25f && pm.y > K.inside_plo &&
                                       pm.y < K.inside_phi && q2.y < K.inside_q2;
                    if (R.record_pq) {
                        if (on_a) A.pq[p] = make_float2(-0.5f * s2.x, 2.0f * s1.x * approx_sqrt(r2.x));
                        if (on_b) A.pq[p + 32] = make_float2(-0.5f * s2.y, 2.0f * s1.y * approx_sqrt(r2.y));
                    }
                    // the others, one at a time: an intact particle is checked
                    // against its own failure surface, a crushed one projected
                    // (Drucker-Prager map), in FP32; what FP32 does not settle
                    // is left aside
                    if ((on_a && !box_a) || (on_b && !box_b)) {
                        // (v and Bp wait in the staging space, already read,
                        // so that the branch costs the common path no registers)
                        float4 *keep = &s_stage[(stage ^ 1) * nwarps + warp].X[0][lane];
                        keep[0] = make_float4(v0.x, v0.y, v1.x, v1.y);
                        keep[32] = make_float4(B0.x, B0.y, B1.x, B1.y);
                        s_stage[(stage ^ 1) * nwarps + warp].H[0][lane] = make_float4(B2.x, B2.y, B3.x, B3.y);
#pragma unroll 1
                        for (int h = (on_a && !box_a) ? 0 : 1; h < ((on_b && !box_b) ? 2 : 1); h++) {
                            M2f F{h ? H0.y : H0.x, h ? H1.y : H1.x, h ? H2.y : H2.x, h ? H3.y : H3.x};
                            const uint32_t meta = h ? mb : ma;
                            bool ok = (h ? J.y : J.x) > 0.25f;
                            if (!(meta & kMetaCrushed)) {
                                const float pp = -0.5f * (h ? s2.y : s2.x);
                                const float qq = 2.0f * (h ? s1.y : s1.x) * approx_sqrt(h ? r2.y : r2.x);
                                ok = ok && failure_side32(GrainStrengths32{K}, meta, pp, qq) == 0;
                            } else if (ok) {
                                const float jp_old = S.Jp[h][lane];
                                float jp = jp_old;
                                const Inv32 v = invariants32(F, K.mu, K.kappa);
                                const float rho = sqrtf(v.hd * v.hd + v.b01 * v.b01);
                                const float pp = -0.5f * v.s2, qq = 2.0f * v.s1 * rho;
                                ok = !K.harvest && dp_map32(K, F, jp, v, pp, qq, rho) == kC32_OK;
                                if (ok) {
                                    const Tau32 tau = tau32(invariants32(F, K.mu, K.kappa));
                                    if (h) {
                                        H0.y = F.a00; H1.y = F.a01; H2.y = F.a10; H3.y = F.a11;
                                        t00.y = tau.t00; t01.y = tau.t01; t11.y = tau.t11;
                                    } else {
                                        H0.x = F.a00; H1.x = F.a01; H2.x = F.a10; H3.x = F.a11;
                                        t00.x = tau.t00; t01.x = tau.t01; t11.x = tau.t11;
                                    }
                                    if (jp != jp_old) A.Jp[p + 32 * h] = jp;
                                    if (R.record_pq) A.pq[p + 32 * h] = make_float2(pp, qq);
                                }
                            }
                            if (h) on_b = on_b && ok;
                            else on_a = on_a && ok;
                        }
                        float4 k4 = keep[0];
                        v0 = make_float2(k4.x, k4.y);
                        v1 = make_float2(k4.z, k4.w);
                        k4 = keep[32];
                        B0 = make_float2(k4.x, k4.y);
                        B1 = make_float2(k4.z, k4.w);
                        k4 = s_stage[(stage ^ 1) * nwarps + warp].H[0][lane];
                        B2 = make_float2(k4.x, k4.y);
                        B3 = make_float2(k4.z, k4.w);
                    }
                }
                if (on_a) {
                    A.X[p] = make_float4(__uint_as_float(uxa), __uint_as_float(uya), __uint_as_float(ca), __uint_as_float(ma));
                    A.H[p] = make_float4(H0.x, H1.x, H2.x, H3.x);
                }
                if (on_b) {
                    A.X[p + 32] =
                        make_float4(__uint_as_float(uxb), __uint_as_float(uyb), __uint_as_float(cb), __uint_as_float(mb));
                    A.H[p + 32] = make_float4(H0.y, H1.y, H2.y, H3.y);
                }

                // P2G: node (i, j) gets W_ij (m, c + S_h (i, j)^T) with
                // S_h = h (m Bp - dt Vp Dinv tau), c = m v - S_h (fx, fy)^T
                {
                    const float2 pm = bcast2(K.mass), nsc = bcast2(-K.stress_c), h = bcast2(K.h);
                    float2 S00 = __fmul2_rn(h, __ffma2_rn(pm, B0, __fmul2_rn(nsc, t00)));
                    float2 S01 = __fmul2_rn(h, __ffma2_rn(pm, B1, __fmul2_rn(nsc, t01)));
                    float2 S10 = __fmul2_rn(h, __ffma2_rn(pm, B2, __fmul2_rn(nsc, t01)));
                    float2 S11 = __fmul2_rn(h, __ffma2_rn(pm, B3, __fmul2_rn(nsc, t11)));
                    const float2 gx = pair_g(uxa, uxb), gy = pair_g(uya, uyb);
                    // f = g + 1/2
                    const float2 nfx = __fadd2_rn(make_float2(-gx.x, -gx.y), bcast2(-0.5f));
                    const float2 nfy = __fadd2_rn(make_float2(-gy.x, -gy.y), bcast2(-0.5f));
                    float2 u0 = __ffma2_rn(v0, pm, __ffma2_rn(S00, nfx, __fmul2_rn(S01, nfy)));
                    float2 u1 = __ffma2_rn(v1, pm, __ffma2_rn(S10, nfx, __fmul2_rn(S11, nfy)));
                    float2 on = make_float2(1.f, 1.f);
                    if (!(on_a && in_a && on_b && in_b)) {
                        // what a particle out of its cell scatters waits in
                        // the staging space, already read
                        Pol32::PairStage &W = s_stage[(stage ^ 1) * nwarps + warp];
                        out_a = on_a && !in_a;
                        out_b = on_b && !in_b;
                        if (out_a) {
                            W.X[0][lane] = make_float4(u0.x, u1.x, S00.x, S01.x);
                            W.H[0][lane] = make_float4(S10.x, S11.x, gx.x, gy.x);
                            W.Jp[0][lane] = __uint_as_float(pair_base(ca, uxa, uya));
                        }
                        if (out_b) {
                            W.X[1][lane] = make_float4(u0.y, u1.y, S00.y, S01.y);
                            W.H[1][lane] = make_float4(S10.y, S11.y, gx.y, gy.y);
                            W.Jp[1][lane] = __uint_as_float(pair_base(cb, uxb, uyb));
                        }
                        const unsigned long long bits = (on_a ? 0ull : 1ull) | (on_b || !has1 ? 0ull : 2ull);
                        if (bits) {
                            s_aside[q][lane] |= bits << (2 * i);
                            s_any = 1;
                        }
                        // a half that is out or left aside adds zeros to the sums
                        if (!(on_a && in_a)) on.x = u0.x = u1.x = S00.x = S01.x = S10.x = S11.x = 0.f;
                        if (!(on_b && in_b)) on.y = u0.y = u1.y = S00.y = S01.y = S10.y = S11.y = 0.f;
                    }
                    float2 wy[3];
#pragma unroll
                    for (int j = 0; j < 3; j++) wy[j] = __fmul2_rn(on, pair_weight(gy, j));
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        if (c) {
                            u0 = __fadd2_rn(u0, S00);
                            u1 = __fadd2_rn(u1, S10);
                        }
                        const float2 wx = pair_weight(gx, c);
                        float2 a0 = u0, a1 = u1;
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            if (j) {
                                a0 = __fadd2_rn(a0, S01);
                                a1 = __fadd2_rn(a1, S11);
                            }
                            const float2 W = __fmul2_rn(wx, wy[j]);
                            sums.add(c * 3 + j, W, a0, a1);
                        }
                    }
                }
            }
            const unsigned oa = __ballot_sync(0xffffffffu, out_a), ob = __ballot_sync(0xffffffffu, out_b);
            if (oa | ob) {
                __syncwarp();
                const Pol32::PairStage &W = s_stage[(stage ^ 1) * nwarps + warp];
                if (lane == 0 && R.strays) atomicAdd(R.strays, (unsigned long long)(__popc(oa) + __popc(ob)));
#pragma unroll 1
                for (int h = 0; h < 2; h++)
                    for (unsigned b = h ? ob : oa; b; b &= b - 1) {
                        const int l = __ffs(b) - 1;
                        pair_scatter<TX, TY>(R, GX, rx0, ry0, wacc, __float_as_uint(W.Jp[h][l]), W.X[h][l], W.H[h][l],
                                             K.mass);
                    }
            }
        }
        if (g.y > step * kPairIters && lane == 0) s_any = 1;
        // the cell's sums into the warp's region: 9 read-modify-write steps,
        // one warp barrier after each (two cells a row apart reach the same
        // node in different steps; lanes hold distinct cells, and a lane
        // without particles adds zeros)
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                sums.flush(wacc[q0 + j * RX + c], c * 3 + j, K.mass);
                __syncwarp();
            }
        g = group(gj + 1, q);
    }
    __pipeline_wait_prior(0);
    __syncwarp();
    if (*(volatile int *)&s_any) pair_aside<TX, TY, WIDE>(P, K, A, R, x0, y0, step, s_v, wacc, &s_stage[warp], s_group, s_wc, s_aside);
    __syncthreads();

    // the tile's nodes in the next-but-one buffer (a tile with particles had
    // mass there two substeps ago)
    if (part != 2) {
        float4 *gC = (float4 *)R.gC;
        for (int k = tid; k < CELLS; k += nthr) {
            const int gx = x0 + k % TX, gy = y0 + k / TX;
            if (gx < GX && gy < GY) node_zero(gC, (size_t)gy * GX + gx);
        }
        if (tid == 0) R.dC[t] = 0;
    }
    // the warps' regions to the scatter buffer
    {
        float4 *gB = (float4 *)R.gB;
        const int dkx = nthr % RX, dky = nthr / RX;
        int kx = tid % RX, ky = tid / RX;
        unsigned marks = 0;  // the tiles of the 3 x 3 neighbourhood that got mass
        constexpr int NB = 4;
        for (int k0 = tid; k0 < RN; k0 += NB * nthr) {
            float4 sum[NB];
#pragma unroll
            for (int b = 0; b < NB; b++) sum[b] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int w = 0; w < nwarps; w++) {
#pragma unroll
                for (int b = 0; b < NB; b++) {
                    if (k0 + b * nthr >= RN) break;
                    const float4 o = s_acc[w * RN + k0 + b * nthr];
                    acc_add(sum[b], acc_m(o), acc_x(o), acc_y(o));
                }
            }
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const int gx = rx0 + kx, gy = ry0 + ky;
                // (a node beyond the grid has no mass: such stencils take the general path)
                if (acc_m(sum[b]) != 0.f && gx >= 0 && gy >= 0 && gx < GX && gy < GY) {
                    node_add_global(gB, (size_t)gy * GX + gx, acc_m(sum[b]), acc_x(sum[b]), acc_y(sum[b]));
                    marks |= 1u << (((ky + TY - 1) / TY) * 3 + (kx + TX - 1) / TX);
                }
                kx += dkx;
                ky += dky;
                if (kx >= RX) { kx -= RX; ky++; }
            }
        }
        marks = __reduce_or_sync(0xffffffffu, marks);
        if (lane < 9 && (marks >> lane & 1u)) {
            const int nx = tx + lane % 3 - 1, ny = ty + lane / 3 - 1;
            if (nx >= 0 && ny >= 0 && nx < R.ntx && ny < R.nty) R.dB[ny * R.ntx + nx] = 1;
        }
    }
}

}  // namespace icm
