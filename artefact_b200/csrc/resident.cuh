// On-chip solver: the whole fixed-count iteration loop of an image as one
// launch, its state held in shared memory.
//
// The image is cut into tiles of RES_TW columns x res_rows rows, one block
// each, all resident at once. A block keeps the FISTA point y (with a two-pixel
// halo), the gradient g, the iterate x, the DCT-distance plane P and the
// coefficients of its tile on chip; per iteration only the norm partials and
// the tile borders of y cross blocks: through distributed shared memory where
// the image's blocks form one cluster, else through L2. Per iteration:
//   1. gradient sweep of the tile, one warp per 28-column strip and a quarter
//      of the tile's rows, from y in shared memory;
//   2. sums of g^2 per strip, sent to the block or blocks that add them;
//   3. sigma from all strips' sums;
//   4. step and projection of the tile's blocks, border pixels of y sent to
//      the neighbouring tiles; image-wide barrier.
// Every per-pixel expression is k_grad_sweep_n's and k_project's, and the sums
// of g^2 are formed in the order of k_grad_sweep_n with strips of 28 columns x
// strip_rows rows in groups of eight, so the result equals theirs bit for bit.
//
// What bounds it: the chain of barriers and short phases, not bandwidth. With
// one launch pair per iteration a small image spent 17-18 us per iteration in
// the latency of global loads (16 rows one after the other, block start-up,
// last-block reduction, projection round trips) whatever its size; here it
// spends 8-10 us (96x64 4:2:0: sweep 3.3, projection 2.7, the sums and the two
// exchanges 3). plan_resident has the measured solves.
#pragma once

#include "solver_kernels.cuh"

namespace art {

constexpr int RES_TW = 112;            // tile columns: four 28-column strips, a multiple of the 16-pixel cells
constexpr int RES_YP = RES_TW + 8;     // row pitch of y in shared memory (column 0 is image column x0 - 4)
constexpr int RES_GP = RES_TW + 1;     // row pitch of g: 8x8 blocks of it serve as transpose scratch, and with an
                                       // odd pitch of 17 mod 32 rows and columns of four adjacent blocks are
                                       // conflict-free
constexpr int RES_WARPS = 16;
constexpr int RES_THREADS = RES_WARPS * 32;
constexpr int RES_STRIP = 28;          // columns of a norm strip (SWEEP_OUT_N)
constexpr int RES_CLUSTER = 16;        // blocks of a cluster, at most (a lane each to send a strip's sums to)
constexpr int RES_CLUSTER_STRIPS = 256;                 // norm strips of an image solved by one cluster, at most
constexpr int RES_GROUPS = 512;                         // groups of eight norm strips of an image, at most
constexpr unsigned RES_ERR_TIMEOUT = 2u;                // bit of the solve's error flag
constexpr long long RES_WAIT_LIMIT = 4000000000LL;      // clock cycles a wait of a solve may take (about 2 s)

// Shared-memory layout of one tile (offsets in floats; coef in int16 from its
// own float offset).
struct ResLayout {
    int y, g, x, p[3], coef[3], total;
};

__host__ __device__ inline ResLayout res_layout(const ImgDev &im)
{
    ResLayout L;
    const int th = im.res_rows;
    int at = 0;
    L.y = at;
    at += im.nch * (th + 4) * RES_YP;
    L.g = at;
    at += (im.nch * th * RES_GP + 3) / 4 * 4;
    for (int c = 0; c < 3; c++) {
        L.p[c] = at;
        if (c < im.nch) at += (th / im.ch[c].sv) * (RES_TW / im.ch[c].sh);
    }
    L.x = at;
    at += im.nch * th * RES_TW;
    for (int c = 0; c < 3; c++) {
        L.coef[c] = at;
        if (c < im.nch) at += (th / im.ch[c].sv) * (RES_TW / im.ch[c].sh) / 2;
    }
    L.total = at;
    return L;
}

// How blocks of one image talk. In a cluster: stores into each other's shared
// memory, ordered by the hardware barrier (res_cluster_sync). In a cooperative
// launch (all blocks are resident): every word that crosses blocks carries a
// tag, the iteration's number in the life of the context, in the same atomic
// access as its data, and the reader polls until the tag is the one it waits
// for. A tagged word needs no fence, no counter and no second read: with a
// counter barrier an exchange cost fence, arrival, poll and load, about 2.3 us
// each twice an iteration. The norm partials are double-buffered (a block may
// post the next iteration's before another has read this one's; it cannot get
// two ahead, since it needs everybody's partials in between); border pixels
// are not: the next ones are sent only after everybody's next partials, which
// follow their reading. Polls are bounded: a block that gives up raises the
// error flag and leaves without posting what it could not form, and so do those
// that wait for it.
__device__ __forceinline__ void res_cluster_sync()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// {value, tag} as one 64-bit access at L2.
__device__ __forceinline__ void res_post(unsigned long long *p, float v, unsigned tag)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p),
                 "l"(__float_as_uint(v) | (unsigned long long)tag << 32)
                 : "memory");
}
__device__ __forceinline__ unsigned long long res_peek(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Gives up a wait that has lasted longer than `limit` clock cycles.
__device__ __forceinline__ bool res_gave_up(long long t0, long long limit, int *s_abort, unsigned *err)
{
    if (clock64() - t0 <= limit) return false;
    *s_abort = 1;
    atomicOr(err, RES_ERR_TIMEOUT);
    return true;
}

// Stores to the same place of the shared memory of block `rank` of the cluster.
__device__ __forceinline__ unsigned res_peer(const void *smem, int rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(smem)), "r"(rank));
    return a;
}
__device__ __forceinline__ void res_store_peer(unsigned addr, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// 8x8 transpose among the 8 lanes of a group through its own block of the
// consumed g tile (T: row pitch RES_GP). Inactive groups only take part in the
// warp barriers.
__device__ __forceinline__ void res_transpose8(float *T, int r, float *v, bool act)
{
    __syncwarp();
    if (act) {
#pragma unroll
        for (int u = 0; u < 8; u++) T[r * RES_GP + u] = v[u];
    }
    __syncwarp();
    if (act) {
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = T[k * RES_GP + r];
    }
}

// Sends the tile's two-pixel border of y to its neighbours' halos: in a cluster
// straight into the neighbouring blocks' shared memory, otherwise as tagged
// words to the image's exchange plane. Warp w takes
// row and column w % 4 of the border of channel w / 4. (Sent by the projecting
// lanes themselves, a border column was one lane's serial loop over its rows
// and doubled the projection's time on a one-tile-high image.)
template <int NCH, bool CLUSTER>
__device__ __forceinline__ void res_send_border(const float *ys, int ych, int warp, int lane, int th, int rows, int cols,
                                                int tile, int tiles_x, bool left, bool right, bool up, bool down,
                                                unsigned long long *yx, long long cs, int pitch, unsigned tag)
{
    if (warp >= 4 * NCH) return;
    const int c = warp >> 2, q = warp & 3;
    const float *t0 = ys + c * ych + 2 * RES_YP + 4;  // the tile's pixel (0, 0)
    const int r = q < 2 ? q : th + q - 4, x = q < 2 ? q : RES_TW + q - 4;
    const int dr = q < 2 ? -1 : 1, dc = dr;
    const bool vert = q < 2 ? up : down, hor = q < 2 ? left : right;
    if constexpr (CLUSTER) {
        // Pixel (r, x) here is pixel (r - dr th, x - dc RES_TW) of the tile (dr, dc) away.
        if (vert) {
            const float *dst = t0 + (r - dr * th) * RES_YP;
            const unsigned a = res_peer(dst, tile + dr * tiles_x);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int xx = lane + 32 * i;
                if (xx < cols) res_store_peer(a + 4 * xx, t0[r * RES_YP + xx]);
            }
            if (lane < 2 && left)
                res_store_peer(res_peer(dst + RES_TW + lane, tile + dr * tiles_x - 1), t0[r * RES_YP + lane]);
            if (lane < 2 && right)
                res_store_peer(res_peer(dst - 2 + lane, tile + dr * tiles_x + 1), t0[r * RES_YP + RES_TW - 2 + lane]);
        }
        if (hor) {
            const unsigned a = res_peer(t0 + x - dc * RES_TW, tile + dc);
            for (int rr = lane; rr < rows; rr += 32) res_store_peer(a + 4 * rr * RES_YP, t0[rr * RES_YP + x]);
        }
    } else {
        unsigned long long *dst = yx + c * cs;
        if (vert) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int xx = lane + 32 * i;
                if (xx < cols) res_post(dst + (long long)r * pitch + xx, t0[r * RES_YP + xx], tag);
            }
        }
        if (hor)
            for (int rr = lane; rr < rows; rr += 32) res_post(dst + (long long)rr * pitch + x, t0[rr * RES_YP + x], tag);
    }
}

// The parts of the projection that depend on the sampling. res_step: x' = y -
// sigma g into v, and the cell means (compute_projection.rs:18-32); res_write:
// x_{k+1} and the next y from v, the means and the projected means. Pointers
// are to the lane's first sample; v holds its 8 SV x SH samples.
template <int SH, int SV>
__device__ __forceinline__ void res_step(const float *y, const float *g, float sg, float (&v)[32], float (&mean)[8])
{
    const bool stepped = sg != 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        float acc = 0.f;
#pragma unroll
        for (int sy = 0; sy < SV; sy++) {
            const int r = k * SV + sy;
            float yv[2];
            if constexpr (SH == 2) {
                const float2 t = *reinterpret_cast<const float2 *>(y + r * RES_YP);
                yv[0] = t.x;
                yv[1] = t.y;
            } else {
                yv[0] = y[r * RES_YP];
            }
#pragma unroll
            for (int sx = 0; sx < SH; sx++) {
                v[r * SH + sx] = stepped ? fmaf(-sg, g[r * RES_GP + sx], yv[sx]) : yv[sx];
                acc += v[r * SH + sx];
            }
        }
        mean[k] = SH * SV > 1 ? acc / (float)(SH * SV) : acc;
    }
}

template <int SH, int SV>
__device__ __forceinline__ void res_write(float *y, float *x, const float (&v)[32], const float (&mean)[8],
                                          const float (&m)[8], float fnext)
{
#pragma unroll
    for (int k = 0; k < 8 * SV; k++) {
        const int kc = k / SV;
        float xo[2], xn[2], yn[2];
        if constexpr (SH == 2) {
            const float2 t = *reinterpret_cast<const float2 *>(x + k * RES_TW);
            xo[0] = t.x;
            xo[1] = t.y;
        } else {
            xo[0] = x[k * RES_TW];
        }
#pragma unroll
        for (int sx = 0; sx < SH; sx++) {
            xn[sx] = SH * SV > 1 ? (v[k * SH + sx] - mean[kc]) + m[kc] : m[kc];
            yn[sx] = fmaf(fnext, xn[sx] - xo[sx], xn[sx]);
        }
        if constexpr (SH == 2) {
            *reinterpret_cast<float2 *>(x + k * RES_TW) = make_float2(xn[0], xn[1]);
            *reinterpret_cast<float2 *>(y + k * RES_YP) = make_float2(yn[0], yn[1]);
        } else {
            x[k * RES_TW] = xn[0];
            y[k * RES_YP] = yn[0];
        }
    }
}

// Step, projection and next FISTA point of four blocks (one per lane group) of
// channel c of a tile: k_project's arithmetic on the tile in shared memory.
// y, g, x point at the lane's first sample, T at the group's block
// of g. One copy of the transforms serves every sampling mode (the code of an
// iteration, run once a phase, has to stay in the instruction cache), and the
// two IDCTs run side by side so that their chains overlap.
__device__ __forceinline__ void res_project(const ImgDev &im, int c, int j, bool act, float *y, const float *g, float *T,
                                            float *x, float *P, const int16_t *coef_row, float sg, float fnext)
{
    const ChanDev &cd = im.ch[c];
    const int sh = cd.sh, sv = cd.sv, mode = (sh - 1) * 2 + sv - 1;
    float co[8], v[32], m[8], mean[8];
    load_coef_row(coef_row, co);
    if (mode == 0)
        res_step<1, 1>(y, g, sg, v, mean);
    else if (mode == 3)
        res_step<2, 2>(y, g, sg, v, mean);
    else if (mode == 2)
        res_step<2, 1>(y, g, sg, v, mean);
    else
        res_step<1, 2>(y, g, sg, v, mean);
#pragma unroll
    for (int u = 0; u < 8; u++) m[u] = mean[u];
    dct8(m);
    res_transpose8(T, j, m, act);
    dct8(m);
    const float ap = cd.alpha_p;  // warp-uniform
    const float *qt = &im.q[c][j * 8], *it = &im.invq2[c][j * 8];
    float d[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const float qv = qt[u], iq = it[u];
        const float cl = fminf(fmaxf(m[u], (co[u] - 0.5f) * qv), (co[u] + 0.5f) * qv);
        m[u] = cl;
        d[u] = __fmul_rn(cl - co[u] * qv, iq);  // rounded on its own, not into the IDCT's first sums
    }
    idct8(m);
    idct8(d);
    res_transpose8(T, j, m, act);
    res_transpose8(T, j, d, act);
    idct8(m);
    idct8(d);
    if (!act) return;
    if (ap != 0.f) {
        const int pp = RES_TW / sh;
#pragma unroll
        for (int k = 0; k < 8; k++) P[k * pp] = ap * d[k];
    }
    if (mode == 0)
        res_write<1, 1>(y, x, v, mean, m, fnext);
    else if (mode == 3)
        res_write<2, 2>(y, x, v, mean, m, fnext);
    else if (mode == 2)
        res_write<2, 1>(y, x, v, mean, m, fnext);
    else
        res_write<1, 2>(y, x, v, mean, m, fnext);
}

// Gradient of rows [r0, r0 + nr) of one 28-column strip of the tile into g
// (k_grad_sweep_n's rows on y and P in shared memory; nr a multiple of 4). Cells
// of y outside the image are zero. pa / pb: this lane's column of P in an even
// row's and an odd row's component row, pstep: to the next pair of rows.
template <int NCH, bool EDGE>
__device__ __forceinline__ void res_sweep_rows(const float *y, int ych, float *g, int gch, const float *const (&pa)[NCH],
                                               const int (&podd)[NCH], const int (&pstep)[NCH], int lane, int strip,
                                               int r0, int nr, int x0, int y0, int W, int H, float at, float ag, float2 nz)
{
    constexpr bool SOLO = NCH & 1, PAIR = NCH >= 2;
    constexpr int P0 = SOLO ? 1 : 0;
    const int gx = x0 + strip * RES_STRIP - 2 + lane;
    const bool colin = gx >= 0 && gx < W, tx0 = gx > 0, xin = gx < W - 1;
    const bool outlane = lane >= 2 && lane < 30 && gx < W;
    const float *yc[NCH], *pc[NCH];
    float *gc[NCH];
#pragma unroll
    for (int c = 0; c < NCH; c++) {
        yc[c] = y + c * ych + r0 * RES_YP + strip * RES_STRIP + 2 + lane;  // column gx of row r0 - 2
        gc[c] = g + c * gch + r0 * RES_GP + strip * RES_STRIP - 2 + lane;
        pc[c] = pa[c] + (r0 / 2) * pstep[c];
    }
    NarrowGroup<float> A;
    NarrowGroup<float2> B;
    if constexpr (SOLO) {
        const float *q = yc[0];
        const float v0[3] = {q[-1], q[0], q[1]}, v1[3] = {q[RES_YP - 1], q[RES_YP], q[RES_YP + 1]};
        narrow_begin(A, v0, v1, xin);
    }
    if constexpr (PAIR) {
        auto l2 = [&](int o) { return make_float2(yc[P0][o], yc[P0 + 1][o]); };
        const float2 v0[3] = {l2(-1), l2(0), l2(1)}, v1[3] = {l2(RES_YP - 1), l2(RES_YP), l2(RES_YP + 1)};
        narrow_begin(B, v0, v1, xin);
    }
    // Two rows a turn: terms of rows t and t + 1, gradient rows t - 1 and t.
#pragma unroll 1
    for (int t = r0 - 1; t <= r0 + nr; t += 2) {
        const bool out = t > r0;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int ta = y0 + t + k;  // image row of the terms
            narrow_row<NCH, EDGE>(
                A, B, [&](int c, int d) { return yc[c][(2 + k) * RES_YP + d]; }, [&](int c) { return pc[c][k * podd[c]]; },
                colin && ta >= 0 && ta < H, tx0, ta > 0, xin, ta < H - 1, at, ag, nz, [&]() {
                    if (!out || !outlane || (EDGE && ta - 1 >= H)) return;
                    if constexpr (SOLO) gc[0][k * RES_GP] = vadd(A.Gm, A.pr);
                    if constexpr (PAIR) {
                        const float2 gv = vadd(B.Gm, B.pr);
                        gc[P0][k * RES_GP] = gv.x;
                        gc[P0 + 1][k * RES_GP] = gv.y;
                    }
                });
        }
#pragma unroll
        for (int c = 0; c < NCH; c++) {
            yc[c] += 2 * RES_YP;
            if (out) {
                gc[c] += 2 * RES_GP;
                pc[c] += pstep[c];
            }
        }
    }
}

// One block a tile of the image; sched[k] = {fnext, stepmul} of iteration k, whose
// tag is epoch + 1 + k. In CLUSTER launches the tiles are one cluster (blocks
// whose index lies past the last tile only keep the barriers complete).
template <int NCH, bool CLUSTER>
__global__ void __launch_bounds__(RES_THREADS, 1) k_resident(const ImgDev *__restrict__ img,
                                                             const float2 *__restrict__ sched, int iterations,
                                                             unsigned epoch, long long wait_limit, unsigned *err)
{
    extern __shared__ float4 s_dyn[];
    __shared__ double s_dred[8][NCH];
    __shared__ float s_sigma[NCH];
    __shared__ int s_abort;
    __shared__ float s_part[NCH][CLUSTER ? RES_CLUSTER_STRIPS : 1];  // every strip's sums of g^2, from all blocks
    __shared__ float s_grp[CLUSTER ? 1 : RES_GROUPS][NCH];       // sums of groups of eight strips
    float *sm = reinterpret_cast<float *>(s_dyn);
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    __shared__ ImgDev s_im;  // the descriptor, read in every phase
    const int tile = blockIdx.x;
    for (int i = tid; i < (int)(sizeof(ImgDev) / 4); i += RES_THREADS)
        reinterpret_cast<unsigned *>(&s_im)[i] = __ldg(reinterpret_cast<const unsigned *>(img) + i);
    if (tid == 0) s_abort = 0;
    __syncthreads();
    const ImgDev &im = s_im;
    const int ntiles = im.res_tiles;
    if (CLUSTER && tile >= ntiles) {
        for (int it = 0; it < 2 * iterations; it++) res_cluster_sync();
        return;
    }
    const int W = im.W, H = im.H, pitch = im.pitch, th = im.res_rows, R = im.strip_rows;
    const int x0 = (tile % im.res_tiles_x) * RES_TW, y0 = (tile / im.res_tiles_x) * th;
    const ResLayout L = res_layout(im);
    const int ych = (th + 4) * RES_YP, gch = th * RES_GP;
    float *ys = sm + L.y, *gs = sm + L.g;
    const int cols = min(RES_TW, W - x0), rows = min(th, H - y0);  // tile inside the image
    const long long cs = im.cstride, o0 = (long long)y0 * pitch + x0;

    // Load the tile: y with its halo (zero outside the image), x, P, coefficients.
    for (int i = tid; i < NCH * ych; i += RES_THREADS) {
        const int c = i / ych, k = i - c * ych, r = k / RES_YP - 2, x = k % RES_YP - 4;
        const bool in = y0 + r >= 0 && y0 + r < H && x0 + x >= 0 && x0 + x < W;
        ys[i] = in ? __ldcg(im.y + c * cs + o0 + (long long)r * pitch + x) : 0.f;
    }
    for (int i = tid; i < NCH * th * RES_TW; i += RES_THREADS) {
        const int c = i / (th * RES_TW), k = i - c * th * RES_TW, r = k / RES_TW, x = k % RES_TW;
        sm[L.x + i] = r < rows && x < cols ? __ldcg(im.x + c * cs + o0 + (long long)r * pitch + x) : 0.f;
    }
#pragma unroll
    for (int c = 0; c < NCH; c++) {
        const ChanDev &cd = im.ch[c];
        const int pw = RES_TW / cd.sh, ph = th / cd.sv, cx0 = x0 / cd.sh, cy0 = y0 / cd.sv;
        int16_t *sc = reinterpret_cast<int16_t *>(sm + L.coef[c]);
        for (int i = tid; i < pw * ph; i += RES_THREADS) {
            const int r = cy0 + i / pw, x = cx0 + i % pw;
            const bool in = r < cd.chh && x < cd.cw;
            sm[L.p[c] + i] = in ? __ldcg(cd.P + (long long)r * cd.ppitch + x) : 0.f;
            sc[i] = in ? __ldg(cd.coef + (long long)r * cd.cpitch + x) : (int16_t)0;
        }
    }
    // Gradient-sweep task of this warp: strip warp % 4, quarter warp / 4 of the rows.
    const int strip = warp & 3, nr = th / 4, r0 = (warp >> 2) * nr;
    const bool sweeps = x0 + strip * RES_STRIP < W && y0 + r0 < H;
    const int xs = x0 + strip * RES_STRIP;
    const bool interior = xs - 2 >= 1 && xs + 29 <= W - 1 && y0 + r0 - 1 >= 1 && y0 + r0 + nr + 1 <= H - 1;
    const float *pa[NCH];
    int pstep[NCH], podd[NCH];
#pragma unroll
    for (int c = 0; c < NCH; c++) {
        const ChanDev &cd = im.ch[c];
        const int lx = max(strip * RES_STRIP - 2 + lane, 0);
        pa[c] = sm + L.p[c] + (lx >> (cd.sh - 1));
        podd[c] = cd.sv == 1 ? RES_TW / cd.sh : 0;
        pstep[c] = (RES_TW / cd.sh) * (cd.sv == 1 ? 2 : 1);
    }
    const float at = im.alpha_tv, ag = im.alpha_tgv;
    const float2 nz = make_float2(im.neg_zero, im.neg_zero);
    const int tcol = tile % im.res_tiles_x, trow = tile / im.res_tiles_x;
    const bool left = tcol > 0, right = tcol + 1 < im.res_tiles_x, up = trow > 0, down = y0 + th < H;
    const int strip0 = (y0 / R) * im.strips_x + x0 / RES_STRIP;  // the tile's first norm strip
    unsigned long long *yx = im.res_y + o0;
    if constexpr (CLUSTER) res_cluster_sync();
    else __syncthreads();

    for (int it = 0; it < iterations; it++) {
        const float2 sc = __ldg(sched + it);  // fnext, stepmul
        if (sweeps) {
            if (interior)
                res_sweep_rows<NCH, false>(ys, ych, gs, gch, pa, podd, pstep, lane, strip, r0, nr, x0, y0, W, H, at, ag, nz);
            else
                res_sweep_rows<NCH, true>(ys, ych, gs, gch, pa, podd, pstep, lane, strip, r0, nr, x0, y0, W, H, at, ag, nz);
        }
        __syncthreads();
        // Sums of g^2 of the tile's norm strips: each column down its rows,
        // then the warp tree of k_grad_sweep_n.
        const unsigned tag = epoch + 1 + it;
        unsigned long long *part = im.res_part + (it & 1) * NCH * im.nstrips;  // [channel][strip]
        for (int i = warp; i < 4 * (th / R); i += RES_WARPS) {
            const int s = i & 3, sr = i >> 2, sy = y0 + sr * R;
            if (x0 + s * RES_STRIP >= W || sy >= H) continue;  // warp-uniform
            const int col = s * RES_STRIP - 2 + lane;
            float v[3] = {0.f, 0.f, 0.f};
            if (lane >= 2 && lane < 30 && x0 + col < W) {
                const float *gp = gs + sr * R * RES_GP + col;
                const int n = min(R, H - sy);  // a multiple of 8
#pragma unroll 8
                for (int r = 0; r < n; r++) {
#pragma unroll
                    for (int c = 0; c < NCH; c++) {
                        const float gv = gp[c * gch + r * RES_GP];
                        v[c] = __fmaf_rn(gv, gv, v[c]);
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int c = 0; c < NCH; c++) v[c] += __shfl_xor_sync(FULL, v[c], o);
            }
            const int to = strip0 + sr * im.strips_x + s;
            if constexpr (CLUSTER) {
                if (lane < ntiles) {
#pragma unroll
                    for (int c = 0; c < NCH; c++) res_store_peer(res_peer(&s_part[c][to], lane), v[c]);
                }
            } else {
                if (lane < NCH) res_post(part + lane * im.nstrips + to, lane == 0 ? v[0] : lane == 1 ? v[1] : v[2], tag);
            }
        }
        // sigma_c = step / ||g_c||: in a cluster every block adds all strips, in
        // a grid the first tile's block does and posts the result. (Every block
        // polling every strip's words queued their writes behind the polls: with
        // 130 blocks a wait of 5300 to 10000 clocks.)
        if constexpr (CLUSTER) res_cluster_sync();
        if (CLUSTER || tile == 0) {
            const int n = im.nstrips;
            if constexpr (!CLUSTER) {
                // 32 neighbouring strips a load; groups of eight added in order.
                for (int i0 = warp * 32; i0 < n; i0 += RES_THREADS) {
                    const int i = i0 + lane;
                    float e[NCH];
#pragma unroll
                    for (int c = 0; c < NCH; c++) e[c] = 0.f;
                    if (i < n) {
                        unsigned long long v[NCH];
                        const long long t0 = clock64();
                        for (;;) {
                            bool all = true;
#pragma unroll
                            for (int c = 0; c < NCH; c++) v[c] = res_peek(part + c * n + i);
#pragma unroll
                            for (int c = 0; c < NCH; c++) all &= (unsigned)(v[c] >> 32) == tag;
                            if (all || res_gave_up(t0, wait_limit, &s_abort, err)) break;
                        }
#pragma unroll
                        for (int c = 0; c < NCH; c++) e[c] = __uint_as_float((unsigned)v[c]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < NCH; c++) {
                        float t = e[c];
#pragma unroll
                        for (int w = 1; w < 8; w++) t += __shfl_down_sync(FULL, e[c], w);
                        if ((lane & 7) == 0 && i < n) s_grp[i >> 3][c] = t;
                    }
                }
                __syncthreads();
            }
            if (tid < 256)
                sigma_trees_of<NCH>((n + 7) / 8, s_dred, [&](int b, float(&t)[NCH]) {
#pragma unroll
                    for (int c = 0; c < NCH; c++) {
                        if constexpr (CLUSTER) {
                            t[c] = 0.f;
#pragma unroll
                            for (int w = 0; w < 8; w++) t[c] += b * 8 + w < n ? s_part[c][b * 8 + w] : 0.f;
                        } else {
                            t[c] = s_grp[b][c];
                        }
                    }
                });
            __syncthreads();
            if (tid < NCH) {
                const float sg = sigma_final<NCH>(s_dred, tid, im.step * sc.y);
                s_sigma[tid] = sg;
                // Sums of which some never came are nobody's step.
                if (!CLUSTER && !s_abort) res_post(im.res_sigma + tid, sg, tag);
            }
        } else if (tid < NCH) {
            const long long t0 = clock64();
            unsigned long long v;
            do v = res_peek(im.res_sigma + tid);
            while ((unsigned)(v >> 32) != tag && !res_gave_up(t0, wait_limit, &s_abort, err));
            s_sigma[tid] = __uint_as_float((unsigned)v);
        }
        __syncthreads();
        if (!CLUSTER && s_abort) return;
        // Step and projection, four blocks per warp.
        int c = 0, first = warp;  // this warp's next task, counted from channel c's first
#pragma unroll 1
        for (;;) {
            int nbx = 0, nblk = 0;
            for (; c < NCH; c++) {
                nbx = cols / (8 * im.ch[c].sh);
                nblk = nbx * (rows / (8 * im.ch[c].sv));
                const int ntask = (nblk + 3) / 4;
                if (first < ntask) break;
                first -= ntask;
            }
            if (c == NCH) break;
            const ChanDev &cd = im.ch[c];
            const int sh = cd.sh, sv = cd.sv, grp = lane >> 3, j = lane & 7;
            const bool act = first * 4 + grp < nblk;
            const int blk = act ? first * 4 + grp : 0, by = blk / nbx, bx = blk - by * nbx;
            const int col = (bx * 8 + j) * sh, row0 = by * 8 * sv, pw = RES_TW / sh;
            res_project(im, c, j, act, ys + c * ych + (2 + row0) * RES_YP + 4 + col, gs + c * gch + row0 * RES_GP + col,
                        gs + c * gch + row0 * RES_GP + bx * 8 * sh, sm + L.x + (c * th + row0) * RES_TW + col,
                        sm + L.p[c] + by * 8 * pw + bx * 8 + j,
                        reinterpret_cast<const int16_t *>(sm + L.coef[c]) + (by * 8 + j) * pw + bx * 8, s_sigma[c], sc.x);
            first += RES_WARPS;
        }
        if (it + 1 == iterations) break;
        __syncthreads();
        if (ntiles > 1)
            res_send_border<NCH, CLUSTER>(ys, ych, warp, lane, th, rows, cols, tile, im.res_tiles_x, left, right, up, down,
                                          yx, cs, pitch, tag);
        if constexpr (CLUSTER) {
            res_cluster_sync();
        } else if (ntiles > 1) {
            // Halo of y: warp w takes row and column w % 4 of the halo of channel w / 4.
            if (warp < 4 * NCH) {
                const int c = warp >> 2, q = warp & 3;
                const unsigned long long *src = yx + c * cs;
                float *dst = ys + c * ych + 2 * RES_YP + 4;
                const int r = q < 2 ? q - 2 : th + q - 2, x = q < 2 ? q - 2 : RES_TW + q - 2;
                const bool rin = y0 + r >= 0 && y0 + r < H, xin = x0 + x >= 0 && x0 + x < W;
                const unsigned long long none = (unsigned long long)tag << 32;
                unsigned long long v[4], w[4];
                const long long t0 = clock64();
                for (;;) {
                    bool all = true;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int xx = lane + 32 * i - 2, rr = lane + 32 * i;
                        const bool vin = rin && xx < RES_TW + 2 && x0 + xx >= 0 && x0 + xx < W;
                        v[i] = vin ? res_peek(src + (long long)r * pitch + xx) : none;
                        w[i] = xin && rr < rows ? res_peek(src + (long long)rr * pitch + x) : none;
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) all &= (unsigned)(v[i] >> 32) == tag && (unsigned)(w[i] >> 32) == tag;
                    if (all || res_gave_up(t0, wait_limit, &s_abort, err)) break;
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int xx = lane + 32 * i - 2, rr = lane + 32 * i;
                    if (rin && xx < RES_TW + 2) dst[r * RES_YP + xx] = __uint_as_float((unsigned)v[i]);
                    if (xin && rr < rows) dst[rr * RES_YP + x] = __uint_as_float((unsigned)w[i]);
                }
            }
            __syncthreads();
            if (s_abort) return;
        }
    }
    __syncthreads();
    for (int i = tid; i < NCH * th * RES_TW; i += RES_THREADS) {
        const int c = i / (th * RES_TW), k = i - c * th * RES_TW, r = k / RES_TW, x = k % RES_TW;
        if (r < rows && x < cols) im.x[c * cs + o0 + (long long)r * pitch + x] = sm[L.x + i];
    }
}

}  // namespace art
