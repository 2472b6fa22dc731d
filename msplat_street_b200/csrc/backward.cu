// Fused per-Gaussian backward + Adam + densification statistics.
//
// A block of Gaussians replaces four reference passes:
//  1. reduce_isect_grads (core/cpu/msplat_cpu.cpp:1034-1064): each visible Gaussian's
//     intersection slots, found through the inverse sort permutation, are summed;
//  2. project_and_sh_backward_adam (:1068-1139): projection, EWA and covariance VJPs
//     (:197-291) for visible Gaussians, SH gradients fused into Adam for DC and rest;
//  3. adam_dense (:1142-1147) over ALL N for means, scales, quats and opacity
//     (invisible Gaussians see a zero gradient, their moments decay);
//  4. the densification statistics (:1312-1324).
// The block first lists its visible Gaussians (a street view sees a tenth to a third of
// them, scattered over the indices), so that the slot sums and the VJPs run on full
// warps; the gradients pass through shared memory to the Adam steps, which walk each
// parameter array as one flat range, coalesced, a thread's loads issued together.
// Compiled with -fmad=false; expressions keep the reference's operation order.
#include "common.cuh"
#include "kernels.h"

namespace msplat {

namespace {

// pixel-centre VJP through the perspective divide (:197-205)
__device__ __forceinline__ V3 center_vjp(const float *P, V3 p, uint32_t w, uint32_t h, float gx, float gy) {
    float hx = P[0] * p.x + P[1] * p.y + P[2] * p.z + P[3];
    float hy = P[4] * p.x + P[5] * p.y + P[6] * p.z + P[7];
    float hw = P[12] * p.x + P[13] * p.y + P[14] * p.z + P[15];
    float rw = 1.f / (hw + 1e-6f);
    float nx = 0.5f * (float)w * gx, ny = 0.5f * (float)h * gy;
    float px = nx * rw, py = ny * rw, pz = 0.f, pw = -(nx * hx + ny * hy) * rw * rw;
    return V3{P[0] * px + P[4] * py + P[8] * pz + P[12] * pw, P[1] * px + P[5] * py + P[9] * pz + P[13] * pw,
              P[2] * px + P[6] * py + P[10] * pz + P[14] * pw};
}

// conic VJP, -X G X with 2x2 column-major products (:207-214)
__device__ __forceinline__ void conic_vjp(V3 cn, V3 g, float *out) {
    const float X00 = cn.x, X01 = cn.y, X10 = cn.y, X11 = cn.z;  // X[col][row]
    const float G00 = g.x, G01 = g.y, G10 = g.y, G11 = g.z;
    // P = X * G
    const float P00 = X00 * G00 + X10 * G01, P01 = X01 * G00 + X11 * G01;
    const float P10 = X00 * G10 + X10 * G11, P11 = X01 * G10 + X11 * G11;
    // Q = P * X
    const float Q00 = P00 * X00 + P10 * X01, Q01 = P01 * X00 + P11 * X01;
    const float Q10 = P00 * X10 + P10 * X11, Q11 = P01 * X10 + P11 * X11;
    const float S00 = Q00 * -1.f, S01 = Q01 * -1.f, S10 = Q10 * -1.f, S11 = Q11 * -1.f;
    out[0] = S00;
    out[1] = S10 + S01;
    out[2] = S11;
}

// EWA VJP (:216-255); adds the mean gradient into gm
__device__ __forceinline__ void ewa_vjp(const float *cov, const float *vm, float fx, float fy, float tfx, float tfy,
                                        V3 gc2, float *gm, float *gc3, V3 pv) {
    float lx = 1.3f * tfx, ly = 1.3f * tfy;
    pv.x = pv.z * fminf(lx, fmaxf(-lx, pv.x / pv.z));
    pv.y = pv.z * fminf(ly, fmaxf(-ly, pv.y / pv.z));
    float rz = 1.f / pv.z, rz2 = rz * rz;
    M3 W = m3(vm[0], vm[4], vm[8], vm[1], vm[5], vm[9], vm[2], vm[6], vm[10]);
    M3 J = m3(fx * rz, 0.f, 0.f, 0.f, fy * rz, 0.f, -fx * pv.x * rz2, -fy * pv.y * rz2, 0.f);
    M3 V = m3(cov[0], cov[1], cov[2], cov[1], cov[3], cov[4], cov[2], cov[4], cov[5]);
    M3 G = m3(gc2.x, 0.5f * gc2.y, 0.f, 0.5f * gc2.y, gc2.z, 0.f, 0.f, 0.f, 0.f);
    M3 T = mul(J, W);
    M3 gV = mul(mul(tr(T), G), T);
    M3 gT = plus(mul(mul(G, T), tr(V)), mul(mul(tr(G), T), V));
    gc3[0] = gV.c[0].x;
    gc3[1] = gV.c[0].y + gV.c[1].x;
    gc3[2] = gV.c[0].z + gV.c[2].x;
    gc3[3] = gV.c[1].y;
    gc3[4] = gV.c[1].z + gV.c[2].y;
    gc3[5] = gV.c[2].z;
    M3 gJ = mul(gT, tr(W));
    float fxr2 = fx * rz2, fyr2 = fy * rz2, rz3 = rz2 * rz;
    V3 gt{-fxr2 * gJ.c[2].x, -fyr2 * gJ.c[2].y,
          -fxr2 * gJ.c[0].x + 2.f * fx * pv.x * rz3 * gJ.c[2].x - fyr2 * gJ.c[1].y + 2.f * fy * pv.y * rz3 * gJ.c[2].y};
    gm[0] += dot3(gt, W.c[0]);
    gm[1] += dot3(gt, W.c[1]);
    gm[2] += dot3(gt, W.c[2]);
}

// rotation VJP, tangent to the unit sphere (:259-274). G(col, row) of the column-major v_R.
__device__ __forceinline__ Q4 rotmat_vjp(Q4 q, const M3 &g) {
    float s = 1.f / sqrtf(q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z);
    float w = q.x * s, x = q.y * s, y = q.z * s, z = q.w * s;
#define G(col, row) el(g.c[col], row)
    Q4 r;
    r.x = 2.f * (x * (G(1, 2) - G(2, 1)) + y * (G(2, 0) - G(0, 2)) + z * (G(0, 1) - G(1, 0)));
    r.y = 2.f * (-2.f * x * (G(1, 1) + G(2, 2)) + y * (G(0, 1) + G(1, 0)) + z * (G(0, 2) + G(2, 0)) +
                 w * (G(1, 2) - G(2, 1)));
    r.z = 2.f * (x * (G(0, 1) + G(1, 0)) - 2.f * y * (G(0, 0) + G(2, 2)) + z * (G(1, 2) + G(2, 1)) +
                 w * (G(2, 0) - G(0, 2)));
    r.w = 2.f * (x * (G(0, 2) + G(2, 0)) + y * (G(1, 2) + G(2, 1)) - 2.f * z * (G(0, 0) + G(1, 1)) +
                 w * (G(0, 1) - G(1, 0)));
#undef G
    float radial = r.x * w + r.y * x + r.z * y + r.w * z;
    return Q4{(r.x - radial * w) * s, (r.y - radial * x) * s, (r.z - radial * y) * s, (r.w - radial * z) * s};
}

// covariance VJP to scale and quaternion (:276-291)
__device__ __forceinline__ void cov3d_vjp(V3 sc, float gs, Q4 q, const float *gc, float *gsv, float *gq) {
    M3 gV = m3(gc[0], 0.5f * gc[1], 0.5f * gc[2], 0.5f * gc[1], gc[3], 0.5f * gc[4], 0.5f * gc[2], 0.5f * gc[4], gc[5]);
    M3 R = rotmat(q);
    M3 S = diag_scale(sc, gs);
    M3 M = mul(R, S);
    M3 gM = smul(2.f, mul(gV, M));
    gsv[0] = dot3(R.c[0], gM.c[0]);
    gsv[1] = dot3(R.c[1], gM.c[1]);
    gsv[2] = dot3(R.c[2], gM.c[2]);
    Q4 r = rotmat_vjp(q, mul(gM, S));
    gq[0] = r.x;
    gq[1] = r.y;
    gq[2] = r.z;
    gq[3] = r.w;
}


constexpr int MAX_REST = 15;  // SH bases beyond DC that the backward updates (degree <= 3)

// A block's visible Gaussians, and the sums of their intersection slots.
template <int NB>
struct VisibleList {
    int count;
    int warp_count[NB / 32];
    uint16_t idx[NB];   // local indices, ascending
    float s9[NB * 9];   // by local index: xy(2) conic(3) rgb(3) opacity
    float depth[NB];    // aux mode: dL/d(view depth)
    int64_t first[NB];  // by local index: first emission index and tiles
    int tiles[NB];
    // listed ones whose slots four lanes, a warp, or the whole block add
    int n_mid, n_wide, n_large;
    uint16_t mid[NB], wide[NB], large[NB];
    __device__ __forceinline__ void store(int i, const float p[9], float pd) {
#pragma unroll
        for (int c = 0; c < 9; c++) s9[i * 9 + c] = p[c];
        depth[i] = pd;
    }
    __device__ __forceinline__ void store_share(int i, int part, const float p[3]) {  // add_share's
        s9[i * 9 + part] = p[0];
        s9[i * 9 + part + 4] = p[1];
        if (part == 0) s9[i * 9 + 8] = p[2];
        if (part == 1) depth[i] = p[2];
    }
};

// Lists the threads with vis set. Every thread of the block must call it; on return the
// list is complete (block-wide).
template <int NB>
__device__ __forceinline__ void list_visible(bool vis, VisibleList<NB> &L) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(0xffffffffu, vis);
    if (lane == 0) L.warp_count[warp] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < NB / 32; w++) {
        const int c = L.warp_count[w];
        if (w < warp) before += c;
        all += c;
    }
    if (vis) L.idx[before + __popc(m & ((1u << lane) - 1u))] = (uint16_t)threadIdx.x;
    if (threadIdx.x == 0) {
        L.count = all;
        L.n_mid = L.n_wide = L.n_large = 0;
    }
    __syncthreads();
}

// Lists the visible ones of a block's instances g0 .. g0 + rows - 1 with their slots'
// emission indices.
template <int NB>
__device__ __forceinline__ bool list_instances(VisibleList<NB> &L, int64_t g0, int rows, const int32_t *radii,
                                               const int64_t *offsets, const int32_t *n_tiles) {
    const int t = threadIdx.x;
    const bool in = t < rows, vis = in && radii[g0 + t] > 0;
    const int64_t first = in ? offsets[g0 + t] : 0;  // not behind the radius: one latency for all three
    const int tiles = in ? n_tiles[g0 + t] : 0;
    L.first[t] = first;
    L.tiles[t] = tiles;
    list_visible<NB>(vis, L);
    return vis;
}

// Sums of the 9 (with slots_depth: 10) raster-backward values over each listed
// Gaussian's intersection slots. Of up to SLOT_SERIAL tiles, every value is added slot
// after slot; of more (near the camera: hundreds), lane l of a warp adds slots l,
// l + 32, ... and a fixed butterfly the lanes. The orders are fixed, so the sums do not
// depend on scheduling. Every thread of the block must call it; the sums are complete
// after the next block barrier.
//
// Bound by the latency of two dependent loads a slot (its sorted position, then the slot
// in L2), about a microsecond. A Gaussian of up to SLOT_LANE_MAX tiles is one lane's; of
// up to SLOT_SERIAL, four neighbouring lanes', which share out its values (two or three
// each) and fetch SLOT_AHEAD slots before they add any; of up to SLOT_WARP_MAX, a warp's,
// and of more a warp's too where there is one for every warp, the rest the block's, whose
// warps share out the values. One lane walking its Gaussian's slots alone (34 on average
// in an early street view) and one warp walking the 2000 of a single Gaussian in front of
// the camera were most of the kernel's time; but blocks full of large Gaussians are bound
// by the slots' sectors, which warps that share out the values read four times: 4000
// Gaussians of 2700 tiles each 2.80 -> 1.64 ms (2.22 with one thread a Gaussian), 300 of
// 5300 3.63 -> 2.04 (3.02), an early street view 66 -> 60 us.
constexpr int SLOT_LANE_MAX = 8, SLOT_SERIAL = 64, SLOT_WARP_MAX = 256, SLOT_AHEAD = 8;

// All values of the slots first, first + step, ... of cnt, two slots fetched at a time.
__device__ __forceinline__ void add_slots(int first, int step, const int32_t *pos, int cnt, const float *slots,
                                          const float *slots_depth, float p[9], float &pd) {
#pragma unroll
    for (int c = 0; c < 9; c++) p[c] = 0.f;
    pd = 0.f;
    int32_t k0 = first < cnt ? pos[first] : 0, k1 = first + step < cnt ? pos[first + step] : 0;
    int j = first;
    for (; j + step < cnt; j += 2 * step) {
        const int32_t n0 = j + 2 * step < cnt ? pos[j + 2 * step] : 0;  // the next two's places, with these two
        const int32_t n1 = j + 3 * step < cnt ? pos[j + 3 * step] : 0;
        const float *s0 = slots + (size_t)k0 * 9, *s1 = slots + (size_t)k1 * 9;
        float a[9], b[9];
#pragma unroll
        for (int c = 0; c < 9; c++) {
            a[c] = s0[c];
            b[c] = s1[c];
        }
#pragma unroll
        for (int c = 0; c < 9; c++) p[c] = (p[c] + a[c]) + b[c];
        if (slots_depth) pd = (pd + slots_depth[k0]) + slots_depth[k1];
        k0 = n0;
        k1 = n1;
    }
    if (j < cnt) {
        const float *s = slots + (size_t)k0 * 9;
#pragma unroll
        for (int c = 0; c < 9; c++) p[c] += s[c];
        if (slots_depth) pd += slots_depth[k0];
    }
}

// One share of a Gaussian's sums over its slots first, first + step, ... of cnt: values
// part and part + 4, and for part 0 value 8, for part 1 the depth.
__device__ __forceinline__ void add_share(int part, int first, int step, const int32_t *pos, int cnt,
                                          const float *slots, const float *slots_depth, float p[3]) {
    p[0] = p[1] = p[2] = 0.f;
    int32_t k[SLOT_AHEAD];
#pragma unroll
    for (int u = 0; u < SLOT_AHEAD; u++) k[u] = first + u * step < cnt ? pos[first + u * step] : 0;
    for (int j = first; j < cnt; j += step * SLOT_AHEAD) {
        int32_t next[SLOT_AHEAD];  // the places of the slots after these, with these
        float v[3][SLOT_AHEAD];
        const int jn = j + step * SLOT_AHEAD;
#pragma unroll
        for (int u = 0; u < SLOT_AHEAD; u++) next[u] = jn + u * step < cnt ? pos[jn + u * step] : 0;
#pragma unroll
        for (int u = 0; u < SLOT_AHEAD; u++) {
            const float *s = slots + (size_t)k[u] * 9 + part;
            const bool in = j + u * step < cnt;
            v[0][u] = in ? s[0] : 0.f;
            v[1][u] = in ? s[4] : 0.f;
            v[2][u] = 0.f;
            if (in && part == 0) v[2][u] = s[8];
            if (in && part == 1 && slots_depth) v[2][u] = slots_depth[k[u]];
        }
#pragma unroll
        for (int u = 0; u < SLOT_AHEAD; u++)
            if (j + u * step < cnt) {
                p[0] += v[0][u];
                p[1] += v[1][u];
                p[2] += v[2][u];
            }
#pragma unroll
        for (int u = 0; u < SLOT_AHEAD; u++) k[u] = next[u];
    }
}

template <int NB>
__device__ __forceinline__ void sum_slots(VisibleList<NB> &L, const int32_t *inv, const float *slots,
                                          const float *slots_depth) {
    static_assert(NB == 128, "four warps share the values of a large Gaussian");
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    float p[9], pd;
    if (t < L.count) {
        const int i = L.idx[t], cnt = L.tiles[i];
        if (cnt <= SLOT_LANE_MAX) {
            add_slots(0, 1, inv + L.first[i], cnt, slots, slots_depth, p, pd);
            L.store(i, p, pd);
        } else {  // the order of a list changes no sum
            int *n = cnt <= SLOT_SERIAL ? &L.n_mid : cnt <= SLOT_WARP_MAX ? &L.n_wide : &L.n_large;
            uint16_t *list = cnt <= SLOT_SERIAL ? L.mid : cnt <= SLOT_WARP_MAX ? L.wide : L.large;
            list[atomicAdd(n, 1)] = (uint16_t)i;
        }
    }
    __syncthreads();
    for (int li = t / 4; li < L.n_mid; li += NB / 4) {
        const int i = L.mid[li], part = t & 3;
        add_share(part, 0, 1, inv + L.first[i], L.tiles[i], slots, slots_depth, p);
        L.store_share(i, part, p);
    }
    __syncwarp();
    const int whole = L.n_large / (NB / 32) * (NB / 32);  // large ones that keep every warp busy alone
    for (int li = warp; li < L.n_wide + whole; li += NB / 32) {  // warp-uniform
        const int i = li < whole ? L.large[li] : L.wide[li - whole];
        add_slots(lane, 32, inv + L.first[i], L.tiles[i], slots, slots_depth, p, pd);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int c = 0; c < 9; c++) p[c] += __shfl_xor_sync(0xffffffffu, p[c], o);
            if (slots_depth) pd += __shfl_xor_sync(0xffffffffu, pd, o);
        }
        if (lane == 0) L.store(i, p, pd);
    }
    for (int q = whole; q < L.n_large; q++) {  // block-uniform
        const int i = L.large[q];
        add_share(warp, lane, 32, inv + L.first[i], L.tiles[i], slots, slots_depth, p);
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) p[c] += __shfl_xor_sync(0xffffffffu, p[c], o);
        if (lane == 0) L.store_share(i, warp, p);
    }
}

// Projection, EWA and covariance VJPs of one visible Gaussian i seen by camera cam
// (core/cpu/msplat_cpu.cpp:1068-1110): mean, scale and quaternion gradients from its
// summed xy / conic gradients, and its unit view direction for the SH gradients.
// v_depth: dL/d(view-space depth), from the aux mode's expected-depth loss (else 0).
__device__ __forceinline__ void projection_vjp(const CamParams &cam, const float *means, const float *scales,
                                               const float *quats, float glob_scale, const Splat *sp, int i,
                                               const float s9[9], float gm[3], float gsv[3], float gq[4], V3 &dir,
                                               float v_depth = 0.f) {
    const float *vm = cam.viewmat;
    V3 pw = ld3(means, i);
    V3 vmn = center_vjp(cam.projmat, pw, cam.width, cam.height, s9[0], s9[1]);
    vmn = add(vmn, scl(V3{vm[8], vm[9], vm[10]}, v_depth));
    gm[0] = vmn.x;
    gm[1] = vmn.y;
    gm[2] = vmn.z;
    const float4 sp0 = reinterpret_cast<const float4 *>(sp)[0];
    const float4 sp1 = reinterpret_cast<const float4 *>(sp)[1];
    float gc2[3];
    conic_vjp(V3{sp0.z, sp0.w, sp1.x}, V3{s9[2], s9[3], s9[4]}, gc2);
    V3 ls = ld3(scales, i);
    // gradient arithmetic: single-precision exp (within 2 ulps) is enough here
    V3 es{expf(ls.x), expf(ls.y), expf(ls.z)};
    const float4 qq = reinterpret_cast<const float4 *>(quats)[i];
    Q4 q{qq.x, qq.y, qq.z, qq.w};
    float cov[6];
    cov3d_of(es, glob_scale, q, cov);
    const float tfx = 0.5f * (float)cam.width / cam.fx, tfy = 0.5f * (float)cam.height / cam.fy;
    V3 pv{vm[0] * pw.x + vm[1] * pw.y + vm[2] * pw.z + vm[3], vm[4] * pw.x + vm[5] * pw.y + vm[6] * pw.z + vm[7],
          vm[8] * pw.x + vm[9] * pw.y + vm[10] * pw.z + vm[11]};
    float gc3[6];
    ewa_vjp(cov, vm, cam.fx, cam.fy, tfx, tfy, V3{gc2[0], gc2[1], gc2[2]}, gm, gc3, pv);
    cov3d_vjp(es, glob_scale, q, gc3, gsv, gq);
    gsv[0] *= es.x;
    gsv[1] *= es.y;
    gsv[2] *= es.z;
    dir = unit(sub(pw, V3{cam.cam_pos[0], cam.cam_pos[1], cam.cam_pos[2]}));
}

// The 15 SH basis values beyond DC for unit direction (x, y, z)
// (core/cpu/msplat_cpu.cpp:101-130).
__device__ __forceinline__ void sh_rest_basis(V3 d, float *bs) {
    float x = d.x, y = d.y, z = d.z;
    float xx = x * x, xy = x * y, xz = x * z, yy = y * y, yz = y * z, zz = z * z;
    bs[0] = -SH_C1 * y;
    bs[1] = SH_C1 * z;
    bs[2] = -SH_C1 * x;
    bs[3] = SH_C2_0 * xy;
    bs[4] = SH_C2_1 * yz;
    bs[5] = SH_C2_2 * (2.f * zz - xx - yy);
    bs[6] = SH_C2_3 * xz;
    bs[7] = SH_C2_4 * (xx - yy);
    bs[8] = SH_C3_0 * y * (3.f * xx - yy);
    bs[9] = SH_C3_1 * xy * z;
    bs[10] = SH_C3_2 * y * (4.f * zz - xx - yy);
    bs[11] = SH_C3_3 * z * (2.f * zz - 3.f * xx - 3.f * yy);
    bs[12] = SH_C3_4 * x * (4.f * zz - xx - yy);
    bs[13] = SH_C3_5 * z * (xx - yy);
    bs[14] = SH_C3_6 * x * (xx - 3.f * yy);
}

// Adam over one array of a block's Gaussians, `count` consecutive floats of it with
// their gradients in shared memory: every access of a warp covers 32 consecutive floats.
// load() only reads, so that a thread can have two arrays' loads on their way at once.
// use(j): whether element j is updated.
template <int NB, int U>
struct AdamFlat {
    float pv[U], v1[U], v2[U];
    template <typename Use>
    __device__ __forceinline__ void load(const float *p, const float *m1, const float *m2, int count, Use use) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = u * NB + (int)threadIdx.x;
            if (j < count && use(j)) {
                pv[u] = p[j];
                v1[u] = m1[j];
                v2[u] = m2[j];
            }
        }
    }
    template <typename Use>
    __device__ __forceinline__ void update(float *p, float *m1, float *m2, const float *g, int count, float ss,
                                           float b1, float b2, float bc2, float eps, Use use) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = u * NB + (int)threadIdx.x;
            if (!(j < count && use(j))) continue;
            adam_step(pv[u], v1[u], v2[u], g[j], ss, b1, b2, bc2, eps);
            p[j] = pv[u];
            m1[j] = v1[u];
            m2[j] = v2[u];
        }
    }
};

// The dense groups and DC of a block's Gaussians (all but the SH rest).
template <int NB>
__device__ __forceinline__ void adam_groups(float *const p[6], float *const m1[6], float *const m2[6], int64_t g0,
                                            int rows, const float *s_mean, const float *s_scale, const float *s_quat,
                                            const float *s_op, const float *s_dc, const uint8_t *s_vis,
                                            const float *ss, const float *bc2, float b1, float b2, float eps) {
    auto all = [](int) { return true; };
    auto seen = [&](int j) { return s_vis[j / 3] != 0; };
    const size_t o3 = 3 * (size_t)g0, o4 = 4 * (size_t)g0;
    const bool op = m1[5] != nullptr;
    AdamFlat<NB, 3> mean, scale, dc;
    AdamFlat<NB, 4> quat;
    AdamFlat<NB, 1> opac;
    mean.load(p[0] + o3, m1[0] + o3, m2[0] + o3, 3 * rows, all);
    scale.load(p[1] + o3, m1[1] + o3, m2[1] + o3, 3 * rows, all);
    mean.update(p[0] + o3, m1[0] + o3, m2[0] + o3, s_mean, 3 * rows, ss[0], b1, b2, bc2[0], eps, all);
    quat.load(p[2] + o4, m1[2] + o4, m2[2] + o4, 4 * rows, all);
    scale.update(p[1] + o3, m1[1] + o3, m2[1] + o3, s_scale, 3 * rows, ss[1], b1, b2, bc2[1], eps, all);
    dc.load(p[3] + o3, m1[3] + o3, m2[3] + o3, 3 * rows, seen);
    quat.update(p[2] + o4, m1[2] + o4, m2[2] + o4, s_quat, 4 * rows, ss[2], b1, b2, bc2[2], eps, all);
    if (op) opac.load(p[5] + g0, m1[5] + g0, m2[5] + g0, rows, all);
    dc.update(p[3] + o3, m1[3] + o3, m2[3] + o3, s_dc, 3 * rows, ss[3], b1, b2, bc2[3], eps, seen);
    if (op) opac.update(p[5] + g0, m1[5] + g0, m2[5] + g0, s_op, rows, ss[5], b1, b2, bc2[5], eps, all);
}

// Adam over the SH-rest rows (`stride` floats, of which the first `used` have gradients)
// of `rows` Gaussians: row(r) is the r-th one's local index, grad(i, base, c, e) the
// gradient of local Gaussian i's float e = 3 base + c. A warp takes as many whole rows at
// a time as fit six floats a lane (four of 45 floats, eight of 24, 21 of 9), as one flat
// range, all loads issued before any update.
template <int NB, typename Row, typename Grad>
__device__ __forceinline__ void adam_rest(float *__restrict__ p, float *__restrict__ m1, float *__restrict__ m2,
                                          int rows, int stride, int used, Row row, Grad grad, float ss, float b1,
                                          float b2, float bc2, float eps) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int E = 6;
    const int per = 32 * E / used;
    int r[E], e[E];  // the lane's floats: row within the step, float within the row
#pragma unroll
    for (int q = 0; q < E; q++) {
        const int k = q * 32 + lane;
        r[q] = k / used;
        e[q] = k - r[q] * used;
    }
    for (int r0 = warp * per; r0 < rows; r0 += NB / 32 * per) {
        float pv[E], v1[E], v2[E];
        int at[E];
#pragma unroll
        for (int q = 0; q < E; q++) {
            at[q] = r[q] < per && r0 + r[q] < rows ? row(r0 + r[q]) : -1;
            if (at[q] < 0) continue;
            const size_t j = (size_t)at[q] * stride + e[q];
            pv[q] = p[j];
            v1[q] = m1[j];
            v2[q] = m2[j];
        }
#pragma unroll
        for (int q = 0; q < E; q++) {
            if (at[q] < 0) continue;
            const size_t j = (size_t)at[q] * stride + e[q];
            const int base = e[q] / 3;
            adam_step(pv[q], v1[q], v2[q], grad(at[q], base, e[q] - 3 * base, e[q]), ss, b1, b2, bc2, eps);
            p[j] = pv[q];
            m1[j] = v1[q];
            m2[j] = v2[q];
        }
    }
}

// Writes every SH-rest gradient row of a block (gradient-only mode): grad(i, base, c, e)
// where e < used, else 0.
template <int NB, typename Grad>
__device__ __forceinline__ void write_rest(float *__restrict__ out, int rows, int stride, int used, Grad grad) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = warp; i < rows; i += NB / 32)
        for (int e = lane; e < stride; e += 32) {
            const int base = e / 3;
            out[(size_t)i * stride + e] = e < used ? grad(i, base, e - 3 * base, e) : 0.f;
        }
}

// The bases beyond DC that get gradients at an SH degree in use.
__device__ __forceinline__ int active_bases(uint32_t dtu) { return dtu < 1 ? 0 : dtu < 2 ? 3 : dtu < 3 ? 8 : 15; }

}  // namespace

// Gaussians (and threads) a block. 64 was no faster for a 10 k scene (29.7 against 29.2
// us).
constexpr int NB = 128;

// The gradient arrays of one Gaussian (those that are asked for).
__device__ __forceinline__ void write_grads(const BackwardArgs &a, size_t i, const float s9[9], float depth,
                                            const float gm[3], const float gsv[3], const float gq[4]) {
    if (a.v_xy) {
        a.v_xy[2 * i] = s9[0];
        a.v_xy[2 * i + 1] = s9[1];
    }
    if (a.v_conic)
        for (int c = 0; c < 3; c++) a.v_conic[3 * i + c] = s9[2 + c];
    if (a.v_rgb)
        for (int c = 0; c < 3; c++) a.v_rgb[3 * i + c] = s9[5 + c];
    if (a.v_opacity) a.v_opacity[i] = s9[8];
    if (a.v_depth) a.v_depth[i] = depth;
    if (a.v_mean3d) {
        for (int c = 0; c < 3; c++) {
            a.v_mean3d[3 * i + c] = gm[c];
            a.v_scale[3 * i + c] = gsv[c];
        }
        for (int c = 0; c < 4; c++) a.v_quat[4 * i + c] = gq[c];
    }
    if (a.g_dc)
        for (int c = 0; c < 3; c++) a.g_dc[3 * i + c] = SH_C0 * s9[5 + c];
}

// The gradients on their way to the Adam steps.
template <int NB>
struct AdamGrads {
    float mean[NB * 3], scale[NB * 3], quat[NB * 4], op[NB], dc[NB * 3];
};

// Bound by the latency of its chain of phases (radii; slot positions; slots; parameters;
// three rounds of Adam loads) and, where most Gaussians are visible and SH degree 3 is in
// use, by issue (Adam's exact square root and divisions). Against one thread a Gaussian
// with its slots, VJPs and Adam in one lane (whose order of additions the slot sums
// keep): a 1 M-Gaussian street step at 1600 x 1060 545 -> 345 us, an early 100 k street
// view 100 -> 76 us.
//
// ADAM: the update step; else gradients (and statistics) only, which go to their arrays
// from the thread that computed them: 63 us for 200 k Gaussians, all visible, and 176 for
// 600 k, where passing them through shared memory as the update does took 70 and 201 and
// one thread a Gaussian 66 and 185.
template <bool ADAM>
__global__ void __launch_bounds__(NB, 1024 / NB) backward_adam_kernel(BackwardArgs a) {
    __shared__ VisibleList<NB> L;
    __shared__ AdamGrads<ADAM ? NB : 1> s;
    __shared__ float s_basis[NB][MAX_REST + 2];
    __shared__ uint8_t s_vis[NB];
    const int t = threadIdx.x;
    const int64_t g0 = (int64_t)blockIdx.x * NB;
    const int rows = (int)min((int64_t)NB, (int64_t)a.n - g0);
    const int active = active_bases(a.cam.degrees_to_use);

    // 1. the visible Gaussians and their slot sums; the others' gradients are zero
    const bool vis = list_instances<NB>(L, g0, rows, a.radii, a.offsets, a.n_tiles);
    if (!vis) {
        if constexpr (ADAM) {
#pragma unroll
            for (int c = 0; c < 9; c++) L.s9[t * 9 + c] = 0.f;
            L.depth[t] = 0.f;
#pragma unroll
            for (int c = 0; c < 3; c++) s.mean[t * 3 + c] = s.scale[t * 3 + c] = s.dc[t * 3 + c] = 0.f;
#pragma unroll
            for (int c = 0; c < 4; c++) s.quat[t * 4 + c] = 0.f;
            s.op[t] = 0.f;
        } else if (t < rows) {
            const float zero[9] = {};
            write_grads(a, (size_t)g0 + t, zero, 0.f, zero, zero, zero);
        }
    }
    s_vis[t] = vis;
    sum_slots<NB>(L, a.inv, a.slots, a.slots_depth);
    __syncthreads();

    // 2. projection VJPs and densification statistics, a listed Gaussian per thread
    if (t < L.count) {
        const int li = L.idx[t], i = (int)g0 + li;
        float s9[9], gm[3], gsv[3], gq[4];
#pragma unroll
        for (int c = 0; c < 9; c++) s9[c] = L.s9[li * 9 + c];
        const float depth = a.slots_depth ? L.depth[li] : 0.f;
        V3 dir;
        projection_vjp(a.cam, a.means, a.scales, a.quats, a.glob_scale, a.splats + i, i, s9, gm, gsv, gq, dir, depth);
        if constexpr (!ADAM) {
            write_grads(a, (size_t)i, s9, depth, gm, gsv, gq);
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++) {
                s.mean[li * 3 + c] = gm[c];
                s.scale[li * 3 + c] = gsv[c];
                s.dc[li * 3 + c] = SH_C0 * s9[5 + c];
            }
#pragma unroll
            for (int c = 0; c < 4; c++) s.quat[li * 4 + c] = gq[c];
            s.op[li] = s9[8];
        }
        if (active > 0) sh_rest_basis(dir, s_basis[li]);
        if (a.vis_counts) {
            a.vis_counts[i] += 1.0f;
            a.xys_grad_norm[i] += sqrtf(s9[0] * s9[0] + s9[1] * s9[1]);
            a.max_2d_size[i] = fmaxf(a.max_2d_size[i], (float)a.radii[i] * a.inv_max_dim);
        }
    }
    __syncthreads();

    const float b1 = a.beta1, b2 = a.beta2, eps = a.eps;
    const int stride = a.rest_stride, used = 3 * active;
    auto grad = [&](int i, int base, int c, int) { return s_basis[i][base] * L.s9[i * 9 + 5 + c]; };
    const size_t off = (size_t)g0 * (size_t)max(stride, 0);
    if constexpr (!ADAM) {  // 3. the SH rest's gradient rows
        if (stride > 0 && a.g_rest)
            write_rest<NB>(a.g_rest + off, rows, stride, used,
                           [&](int i, int base, int c, int e) { return s_vis[i] ? grad(i, base, c, e) : 0.f; });
        return;
    } else {
        if (t < rows)
            write_grads(a, (size_t)g0 + t, L.s9 + t * 9, L.depth[t], s.mean + t * 3, s.scale + t * 3, s.quat + t * 4);
        // 3. Adam: means, scales, quats, opacity of all N; DC and the SH rest of the visible
        adam_groups<NB>(a.p, a.m1, a.m2, g0, rows, s.mean, s.scale, s.quat, s.op, s.dc, s_vis, a.ss, a.bc2, b1, b2,
                        eps);
        // needle cap after the scale update (scale_ratio_cap, core/cpu/msplat_cpu.cpp:1295-1309)
        if (a.log_max_scale_ratio > 0.f) {  // grid-uniform
            __syncthreads();  // a Gaussian's three scales were updated by three threads
            if (t < rows) {
                float *sc = a.p[1] + 3 * ((size_t)g0 + t);
                const float x = sc[0], y = sc[1], z = sc[2];
                const float mx = fmaxf(x, fmaxf(y, z)), mn = fminf(x, fminf(y, z));
                const float cap = (x + y + z - mx - mn) + a.log_max_scale_ratio;
                if (mx > cap) {
                    if (x == mx) sc[0] = cap;
                    else if (y == mx) sc[1] = cap;
                    else sc[2] = cap;
                }
            }
        }
        if (stride <= 0 || active == 0) return;
        adam_rest<NB>(a.p[4] + off, a.m1[4] + off, a.m2[4] + off, L.count, stride, used,
                      [&](int r) { return (int)L.idx[r]; }, grad, a.ss[4], b1, b2, a.bc2[4], eps);
    }
}

void launch_backward_adam(const BackwardArgs &a, cudaStream_t st) {
    if (a.n <= 0) return;
    const int blocks = (a.n + NB - 1) / NB;
    if (a.do_adam) backward_adam_kernel<true><<<blocks, NB, 0, st>>>(a);
    else backward_adam_kernel<false><<<blocks, NB, 0, st>>>(a);
}

// The multi-view form: a block walks the batch's views in order, lists the Gaussians each
// view sees, sums their slots (instance v * n + i), runs that view's projection VJPs and
// accumulates the gradients in shared memory, then applies one Adam step. The
// densification statistics advance once per view that sees the Gaussian, as consecutive
// single-view steps would advance them. A one-view batch reproduces
// backward_adam_kernel's update. Eight street views of 100 k Gaussians: 916 -> 654 us
// against one thread a Gaussian.
__global__ void __launch_bounds__(NB, 768 / NB) backward_adam_batch_kernel(BackwardBatchArgs a) {
    __shared__ VisibleList<NB> L;
    __shared__ float s_mean[NB * 3], s_scale[NB * 3], s_quat[NB * 4], s_op[NB], s_dc[NB * 3];
    __shared__ uint8_t s_vis[NB];
    extern __shared__ float s_rest[];  // [NB][3 * MAX_REST], when an SH degree above 0 is in use
    if (a.skip && *a.skip) return;  // block-uniform: the step overflowed its capacity
    const int t = threadIdx.x;
    const int64_t g0 = (int64_t)blockIdx.x * NB;
    const int rows = (int)min((int64_t)NB, (int64_t)a.n - g0);
    const int active = active_bases(a.degrees_to_use), used = 3 * active;
#pragma unroll
    for (int c = 0; c < 3; c++) s_mean[t * 3 + c] = s_scale[t * 3 + c] = s_dc[t * 3 + c] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; c++) s_quat[t * 4 + c] = 0.f;
    s_op[t] = 0.f;
    s_vis[t] = 0;
    if (active > 0)
        for (int j = 0; j < 3 * MAX_REST; j++) s_rest[t * 3 * MAX_REST + j] = 0.f;
    for (int v = 0; v < a.n_views; v++) {  // block-uniform
        const int64_t gv = (int64_t)v * a.n + g0;
        list_instances<NB>(L, gv, rows, a.radii, a.offsets, a.n_tiles);
        sum_slots<NB>(L, a.inv, a.slots, nullptr);
        __syncthreads();
        if (t < L.count) {
            const int li = L.idx[t], i = (int)g0 + li;
            const int64_t g = gv + li;
            float s9[9], vm[3], vs[3], vq[4];
#pragma unroll
            for (int c = 0; c < 9; c++) s9[c] = L.s9[li * 9 + c];
            V3 dir;
            projection_vjp(a.proj[v].cam, a.means, a.scales, a.quats, a.glob_scale, a.splats + g, i, s9, vm, vs, vq,
                           dir);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                s_mean[li * 3 + c] += vm[c];
                s_scale[li * 3 + c] += vs[c];
                s_dc[li * 3 + c] += SH_C0 * s9[5 + c];
            }
#pragma unroll
            for (int c = 0; c < 4; c++) s_quat[li * 4 + c] += vq[c];
            s_op[li] += s9[8];
            s_vis[li] = 1;
            if (active > 0) {
                float bs[MAX_REST];
                sh_rest_basis(dir, bs);
                float *r = s_rest + li * 3 * MAX_REST;
#pragma unroll
                for (int k = 0; k < MAX_REST; k++) {
                    if (k >= active) break;
#pragma unroll
                    for (int c = 0; c < 3; c++) r[3 * k + c] += bs[k] * s9[5 + c];
                }
            }
            if (a.vis_counts) {
                a.vis_counts[i] += 1.0f;
                a.xys_grad_norm[i] += sqrtf(s9[0] * s9[0] + s9[1] * s9[1]);
                a.max_2d_size[i] = fmaxf(a.max_2d_size[i], (float)a.radii[g] * a.inv_max_dim[v]);
            }
        }
        __syncthreads();  // the list and the statistics are another thread's in the next view
    }
    if (t < rows && a.g[0]) {  // summed gradients (zero for Gaussians no view sees)
        const size_t i = (size_t)g0 + t;
        for (int c = 0; c < 3; c++) {
            a.g[0][3 * i + c] = s_mean[t * 3 + c];
            a.g[1][3 * i + c] = s_scale[t * 3 + c];
            a.g[3][3 * i + c] = s_dc[t * 3 + c];
        }
        for (int c = 0; c < 4; c++) a.g[2][4 * i + c] = s_quat[t * 4 + c];
        a.g[5][i] = s_op[t];
    }
    const float *ss = a.adam_scalars, *bc2 = a.adam_scalars + 6;
    const float b1 = a.beta1, b2 = a.beta2, eps = a.eps;
    if (a.do_adam) {
        adam_groups<NB>(a.p, a.m1, a.m2, g0, rows, s_mean, s_scale, s_quat, s_op, s_dc, s_vis, ss, bc2, b1, b2, eps);
    }
    // SH rest: the summed gradient rows (zero where no view saw the Gaussian), and Adam
    const int stride = a.rest_stride;
    if (stride <= 0) return;
    auto grad = [&](int i, int, int, int e) { return s_rest[i * 3 * MAX_REST + e]; };
    const size_t off = (size_t)g0 * stride;
    if (a.g[4]) write_rest<NB>(a.g[4] + off, rows, stride, used, grad);
    if (!a.do_adam || active == 0) return;
    list_visible<NB>(s_vis[t] != 0, L);
    adam_rest<NB>(a.p[4] + off, a.m1[4] + off, a.m2[4] + off, L.count, stride, used,
                  [&](int r) { return (int)L.idx[r]; }, grad, ss[4], b1, b2, bc2[4], eps);
}

void launch_backward_adam_batch(const BackwardBatchArgs &a, cudaStream_t st) {
    if (a.n <= 0) return;
    const size_t smem = a.degrees_to_use > 0 ? NB * 3 * MAX_REST * sizeof(float) : 0;
    backward_adam_batch_kernel<<<(a.n + NB - 1) / NB, NB, smem, st>>>(a);
}

}  // namespace msplat
