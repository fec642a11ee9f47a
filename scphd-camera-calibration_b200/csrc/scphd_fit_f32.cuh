// scphd_fit_f32.cuh — the single-precision cloud fit: cloud_fit_body's work (what it covers
// and the reference's lines are listed there) with four samples per lane.
//
// Why.  The one-sample-per-lane form is bound by instruction issue: 1669 warp instructions
// per fitted Gaussian at 100 samples, 0.76 per scheduler and cycle, no pipe above 40 %.
// sm_100's packed operations (fma, mul, add.rn.f32x2) work on two FP32 values per
// instruction, each rounded like its scalar form.  Two neighbouring samples of a Gaussian
// make a pair and a lane holds two pairs, so the algebra of a sample (factor times normals,
// both camera transforms, the motion, the moment rows) takes half the instructions, one
// 16-byte access moves four samples of a cloud or a staged row, and the factor row and the
// poses are read once for four samples.  Philox, the logarithm, root, sine and cosine stay
// one per sample.  1024 instructions per fitted Gaussian at 0.56 per scheduler and cycle; one
// launch over 4096 parents x 256 Gaussians x 100 samples takes 1.59 ms instead of 1.98 ms.
//
// What bounds it now: the multiply-add pipe that runs packed operations and Philox's 64-bit
// products (54 % busy), shared-memory and L1 data (53 %) and issue (56 %), with four warps per
// scheduler (128 registers).  Measured and not better: two samples per lane at 28 warps per
// SM (1.90 ms: the constants are read for half as many samples, 64 % of the shared-memory
// data path), 20 or 18 warps of 96 registers (2.05, 1.81 ms: spills that the small L1 beside
// 220 KB of shared memory does not hold), 12 of 160 (1.71 ms), prefetching the next round's
// clouds into L2 (1.63 ms), the normals in scalar operations (1.59 ms).
//
// Constants that a packed operation needs twice (factor rows, poses, model) are doubled in
// shared memory: building a pair from one value costs the move that packing saves.
//
// Sample layout.  A Gaussian's samples are units of four (P = 100: 25).  A warp sorts its
// Gaussians, up to 32 at a time, the drawn (merged) ones before the carried clouds, so that
// lanes of a pass take different paths in one pass at most, and deals their units out to its
// lanes in order, without regard to where a Gaussian ends: five Gaussians fill four passes
// (125 of 128 lanes).  Moment rows are staged per Gaussian in a ring; two complete Gaussians
// are summed at a time.
//
// The sums.  The 29 moments are products of two of eight rows (r d[6], r, w').  A lane that
// sums one product reads two rows; here it reads three, x, y, z, and sums xx, xy, xz and yz
// over every second pair of samples: the seven lines of the Fano plane hold each of the 21
// pairs of r d[6], r once, an eighth lane takes w'w', so 16 lanes sum a Gaussian and the
// shared-memory data read falls from 200 to 75 cycles per Gaussian.
//
// Every operation is the one-sample form's, in its order and with its contractions (fused
// multiply-adds are written out), and each moment runs over the same partial sums in the same
// order: fitted rows and clouds are the one-sample form's bit for bit.  (rcp, rsqrt and lg2
// flush subnormal inputs here, which only a subnormal depth or disparity could be.)
#pragma once

namespace scphd {

typedef unsigned long long F2;   // two FP32 values, the lower sample in the low half

__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ F2 f2_dup(float a) { return pack_f32x2(a, a); }
__device__ __forceinline__ float f2_lo(F2 v) {
    return __uint_as_float((uint32_t)v);
}
__device__ __forceinline__ float f2_hi(F2 v) {
    return __uint_as_float((uint32_t)(v >> 32));
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_ftz(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Box-Muller for two samples: the pair of normals Pair<float>::two gives for (wa0, wb0) in
// the low halves and for (wa1, wb1) in the high ones.  n = -r; unlike there, nothing guards the
// root: its argument -2 ln u is positive for every u the clamp lets through (the smallest is
// 1.6e-8, for the largest u, 0.99999994, whose approximate logarithm is -1.2e-8 where -8.6e-8
// is exact).  tests/cpp/normals_check.cu runs all values of [0.5, 1].
__device__ __forceinline__ void normals_pair(uint32_t wa0, uint32_t wb0, uint32_t wa1, uint32_t wb1, F2& z0, F2& z1) {
    const F2 ua = f2_fma(pack_f32x2((float)wa0, (float)wa1), f2_dup(0x1p-32f), f2_dup(0x1p-33f));
    const F2 lg = pack_f32x2(lg2_ftz(fminf(f2_lo(ua), 0.99999994f)), lg2_ftz(fminf(f2_hi(ua), 0.99999994f)));
    const F2 q = f2_mul(lg, f2_dup(1.3862943611198906f));   // -(r r)
    const F2 n = f2_mul(q, pack_f32x2(rsqrt_ftz(-f2_lo(q)), rsqrt_ftz(-f2_hi(q))));
    const F2 th = f2_fma(pack_f32x2((float)wb0, (float)wb1), f2_dup(6.283185307179586f * 0x1p-32f),
                         f2_dup(6.283185307179586f * (0x1p-33f - 0.5f)));
    float s0, c0, s1, c1;
    __sincosf(f2_lo(th), &s0, &c0);
    __sincosf(f2_hi(th), &s1, &c1);
    z0 = f2_mul(n, pack_f32x2(c0, c1));
    z1 = f2_mul(n, pack_f32x2(s0, s1));
}

// Doubled constants of one block, in the order the passes read them.
struct alignas(16) QuadTable {
    F2 inv[6];       // -u0, -v0, B, fx / fy, -(fx B), -1
    F2 src_r[9], src_t[3];   // pose the merged components are drawn with (world = R' c + t)
    F2 pred[6];      // feature noise (3), dt, dt^2 / 2, (unused)
    F2 upd_t[4];     // -t of this frame's pose, (unused)
    F2 upd_r[9];     // R of this frame's pose
    F2 meas[5];      // -fx, -fy, u0, v0, -(fx B)
};

constexpr int kQuadWarps = 4;
// units (four samples) per Gaussian
__host__ __device__ constexpr int quad_units(int P) { return (P + 3) / 4; }
// Gaussians per round: as many as fill whole passes of 32 units best (P = 100: 5, 125 of 128)
__host__ __device__ constexpr int quad_round(int P) {
    const int nu = quad_units(P), t = nu <= 32 ? 128 / nu : 256 / nu;
    const int cap = nu <= 32 ? 16 : 5;
    return t < cap ? t : cap;
}
// Gaussians whose rows are held at once: those a pass touches, and one that waits for its
// partner (two are fitted at a time)
__host__ __device__ constexpr int quad_ring(int P) {
    const int nu = quad_units(P), n = quad_round(P) * nu;
    int span = 1;
    for (int u = 0; u < n; u += 32) {
        const int last = u + 31 < n ? u + 31 : n - 1;
        const int k = last / nu - u / nu + 1;
        span = k > span ? k : span;
    }
    return 1 + span;
}
// floats of one Gaussian's staged rows (r d[6], r, w')
__host__ __device__ constexpr int quad_rows(int P) { return kStageRows * stage_stride<float>((P + 3) & ~3); }
// bytes of one Gaussian's marks: per unit, samples in view (bits 0-3), of non-zero weight (4-7)
__host__ __device__ constexpr int quad_marks(int P) { return (quad_units(P) + 15) & ~15; }
// per warp: the ring's rows and negated shifts (6, doubled), the round's doubled factor rows
// (28), the slots of up to kQuadSlots Gaussians
constexpr int kQuadSlots = 32;
__host__ __device__ constexpr size_t quad_warp_bytes(int P) {
    return (size_t)quad_ring(P) * (quad_rows(P) * 4 + 48 + quad_marks(P)) + (size_t)quad_round(P) * 28 * 8 + kQuadSlots * 16;
}
// the mean pD of a Gaussian with n of its samples in view, n = 0..P (cloud_fit_body)
__host__ __device__ constexpr size_t quad_pbar_bytes(int P) { return (size_t)((P + 4) & ~3) * 4; }
__host__ __device__ constexpr size_t quad_fit_smem_bytes(int P) {
    return sizeof(QuadTable) + quad_pbar_bytes(P) + (size_t)kQuadWarps * quad_warp_bytes(P);
}

// predict_features with feature noise on two samples: w0, w1 their Philox words
__device__ __forceinline__ void quad_predict(const QuadTable& tab, const uint32_t w0[4], const uint32_t w1[4], F2 (&X)[6]) {
    F2 z[4];
    normals_pair(w0[0], w0[1], w1[0], w1[1], z[0], z[1]);
    normals_pair(w0[2], w0[3], w1[2], w1[3], z[2], z[3]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const F2 a2 = f2_mul(tab.pred[i], z[i]);
        X[i] = f2_fma(a2, tab.pred[4], f2_fma(X[i + 3], tab.pred[3], X[i]));
        X[i + 3] = f2_fma(a2, tab.pred[3], X[i + 3]);
    }
}

// measure() on two samples
__device__ __forceinline__ void quad_measure(const QuadTable& tab, const F2 (&X)[6], F2 (&y)[6]) {
    const F2 d0 = f2_add(X[0], tab.upd_t[0]), d1 = f2_add(X[1], tab.upd_t[1]), d2 = f2_add(X[2], tab.upd_t[2]);
    F2 xc[3], vc[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const F2 r0 = tab.upd_r[3 * i], r1 = tab.upd_r[3 * i + 1], r2 = tab.upd_r[3 * i + 2];
        xc[i] = f2_fma(r2, d2, f2_fma(r0, d0, f2_mul(r1, d1)));
        vc[i] = f2_fma(r2, X[5], f2_fma(r0, X[3], f2_mul(r1, X[4])));
    }
    const F2 iz = pack_f32x2(rcp_ftz(f2_lo(xc[2])), rcp_ftz(f2_hi(xc[2]))), iz2 = f2_mul(iz, iz);
    const F2 nvz = f2_mul(vc[2], tab.inv[5]), nfx = tab.meas[0], nfy = tab.meas[1], nfxB = tab.meas[4];
    y[0] = f2_fma(f2_mul(nfx, iz), xc[0], tab.meas[2]);
    y[1] = f2_fma(f2_mul(nfy, iz), xc[1], tab.meas[3]);
    y[2] = f2_mul(nfxB, iz);
    y[3] = f2_mul(f2_mul(nfx, f2_fma(vc[0], xc[2], f2_mul(nvz, xc[0]))), iz2);
    y[4] = f2_mul(f2_mul(nfy, f2_fma(vc[1], xc[2], f2_mul(nvz, xc[1]))), iz2);
    y[5] = f2_mul(f2_mul(nfxB, nvz), iz2);
}

// invert() on two samples
__device__ __forceinline__ void quad_invert(const QuadTable& tab, const F2 (&y)[6], F2 (&X)[6]) {
    const F2 id = pack_f32x2(rcp_ftz(f2_lo(y[2])), rcp_ftz(f2_hi(y[2]))), id2 = f2_mul(id, id);
    const F2 du = f2_add(y[0], tab.inv[0]), dv = f2_add(y[1], tab.inv[1]);
    const F2 B = tab.inv[2], fr = tab.inv[3], nvd = f2_mul(y[5], tab.inv[5]);
    F2 c[6];
    c[0] = f2_mul(f2_mul(du, B), id);
    c[1] = f2_mul(f2_mul(f2_mul(fr, dv), B), id);
    c[2] = f2_mul(tab.inv[4], id);
    c[3] = f2_mul(f2_mul(B, f2_fma(y[3], y[2], f2_mul(nvd, du))), id2);
    c[4] = f2_mul(f2_mul(f2_mul(fr, f2_fma(y[4], y[2], f2_mul(nvd, dv))), B), id2);
    c[5] = f2_mul(f2_mul(tab.inv[4], nvd), id2);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const F2 r0 = tab.src_r[i], r3 = tab.src_r[3 + i], r6 = tab.src_r[6 + i];
        X[i] = f2_add(f2_fma(r6, c[2], f2_fma(r0, c[0], f2_mul(r3, c[1]))), tab.src_t[i]);
        X[3 + i] = f2_fma(r6, c[5], f2_fma(r0, c[3], f2_mul(r3, c[4])));
    }
}

// y = L z + mean on two samples: el holds the factor (packed lower, 21) and the mean (6)
__device__ __forceinline__ void quad_ltz(const F2 (&el)[28], const F2 (&z)[6], F2 (&y)[6]) {
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        F2 t = 0ull;
#pragma unroll
        for (int k = 0; k <= a; ++k) t = f2_fma(el[tri(a, k)], z[k], t);
        y[a] = f2_add(t, el[21 + a]);
    }
}

// The six normals of two drawn samples s, s + 1 (component key key_i of map row `row`)
__device__ __forceinline__ void quad_draw(const uint32_t* rk, uint32_t s, uint32_t key_i, uint32_t row, uint32_t frame, F2 (&z)[6]) {
    uint32_t a0[4], a1[4], b0[4], b1[4];
    const uint32_t c0 = ctr_word3(frame, ST_SAMPLE, 0), c1 = ctr_word3(frame, ST_SAMPLE, 1);
    philox_rk(s, key_i, row, c0, rk, a0);
    philox_rk(s + 1u, key_i, row, c0, rk, a1);
    philox_rk(s, key_i, row, c1, rk, b0);
    philox_rk(s + 1u, key_i, row, c1, rk, b1);
    normals_pair(a0[0], a0[1], a1[0], a1[1], z[0], z[1]);
    normals_pair(a0[2], a0[3], a1[2], a1[3], z[2], z[3]);
    normals_pair(b0[0], b0[1], b1[0], b1[1], z[4], z[5]);
}

// The unweighted fit of a Gaussian in view whose in-view samples all have zero weight
// (pD = 1 and sample weights of 0, which set_state can bring in): every sample weighted 1
// (exp(LOG0 - LOG0)), the unnormalised mean (sum of the samples) and covariance x (P + P)/P.
// One warp, its samples made once more; ent: the map row, rows: 6 rows of stride sY.
// Returns element `lane` of the fitted row (lanes 2..28).
static __device__ __noinline__ float quad_unweighted(const Params& prm, const QuadTable& tab, const float* ent,
                                                     const float* cloud, int Ps, int ref, int j, int p, int row, int has_pred,
                                                     uint32_t pred_frame, uint32_t sample_frame, float* rows, int sY, int ra,
                                                     int rb) {
    const int lane = threadIdx.x & 31, P = prm.P;
    for (int s = lane; s < P; s += 32) {
        F2 X[6], y[6];
        if (ref < 0) {
            F2 z[6], el[28];
            quad_draw(prm.rk, (uint32_t)s, (uint32_t)(-1 - ref), (uint32_t)row, sample_frame, z);
#pragma unroll
            for (int i = 0; i < 21; ++i) el[i] = f2_dup(ent[7 + i]);
#pragma unroll
            for (int i = 0; i < 6; ++i) el[21 + i] = f2_dup(ent[1 + i]);
            quad_ltz(el, z, y);
            quad_invert(tab, y, X);
        } else {
#pragma unroll
            for (int a = 0; a < 6; ++a) X[a] = f2_dup(cloud[((size_t)ref * 7 + a) * Ps + s]);
        }
        if (has_pred) {
            uint32_t w[4];
            philox_rk((uint32_t)s, (uint32_t)j, (uint32_t)p, ctr_word3(pred_frame, ST_FEAT, 0), prm.rk, w);
            quad_predict(tab, w, w, X);
        }
        quad_measure(tab, X, y);
#pragma unroll
        for (int a = 0; a < 6; ++a) rows[a * sY + s] = f2_lo(y[a]);
    }
    __syncwarp();
    float mu = 0;
    if (lane < 6)
        for (int i = 0; i < P; ++i) mu += rows[lane * sY + i];
    const float ma = __shfl_sync(0xffffffffu, mu, ra < 6 ? ra : 0), mb = __shfl_sync(0xffffffffu, mu, rb < 6 ? rb : 0);
    float cva = 0;
    if (lane >= 8 && lane < 29)
        for (int i = 0; i < P; ++i) cva += (rows[ra * sY + i] - ma) * (rows[rb * sY + i] - mb);
    const float scale = ((float)P * (float)P + (float)P) / (float)P;
    const float mu_e = __shfl_sync(0xffffffffu, mu, (lane - 2) & 31);   // mean element lane - 2
    return lane < 8 ? mu_e : cva * scale;
}

template <int K, int PC = 0>
__device__ __forceinline__ void cloud_fit_f32_body(const Params& prm, const Bufs<float>& b, int cur, int M, int fixed,
                                                   int has_pred, double dt, uint32_t pred_frame, uint32_t sample_frame,
                                                   const double* zu, const double* zv, const double* zd, int p, int c,
                                                   int split, unsigned char* smem) {
    if (p == 0 && c == 0 && zu != nullptr) {   // this frame's measurements into the FP32 layout (u, v, d)
        for (int mm = threadIdx.x; mm < M; mm += blockDim.x) {
            b.z[mm * 3 + 0] = (float)zu[mm];
            b.z[mm * 3 + 1] = (float)zv[mm];
            b.z[mm * 3 + 2] = (K == 3 && zd) ? (float)zd[mm] : 0.0f;
        }
    }
    const int warp = threadIdx.x >> 5;
    int lane;   // (volatile: read once and kept, not read again from the special register)
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    const int gw = c * kQuadWarps + warp, nwp = split * kQuadWarps;
    const int row = b.src[p];
    const int G = min(b.map_n[cur][row], prm.Gcap);
    const int P = PC > 0 ? PC : prm.P, Ps = PC > 0 ? cloud_stride<float>(PC) : prm.Ps;
    const int nu = quad_units(P), TG = quad_round(P), NR = quad_ring(P);
    const int sY = stage_stride<float>((P + 3) & ~3), rowsz = quad_rows(P);

    QuadTable& tab = *reinterpret_cast<QuadTable*>(smem);
    float* s_pbar = reinterpret_cast<float*>(smem + sizeof(QuadTable));
    unsigned char* wsm = smem + sizeof(QuadTable) + quad_pbar_bytes(P) + warp * quad_warp_bytes(P);
    float* rows = reinterpret_cast<float*>(wsm);                   // ring slot r: 8 rows
    F2* nsh = reinterpret_cast<F2*>(rows + NR * rowsz);            // ring slot r: -shift, doubled
    unsigned char* marks = reinterpret_cast<unsigned char*>(nsh + NR * 6);   // ring slot r: the units' marks
    F2* Lw = reinterpret_cast<F2*>(marks + NR * quad_marks(P));    // round's Gaussian q: factor and mean, doubled
    int4* slots = reinterpret_cast<int4*>(Lw + TG * 28);           // ref, W, j, ring slot
    __shared__ int s_rd, s_wr;

    for (int i = threadIdx.x; i <= P; i += blockDim.x) s_pbar[i] = (float)((double)i * prm.model.pd / (double)P);
    const ModelF& mf = prm.model_f;
    if (threadIdx.x == 32) {
        const Pose<float> ps = make_pose<float>(b.map_ext[cur] + 12 * row);
#pragma unroll
        for (int i = 0; i < 9; ++i) tab.src_r[i] = f2_dup(ps.R[i]);
#pragma unroll
        for (int i = 0; i < 3; ++i) tab.src_t[i] = f2_dup(ps.t[i]);
    }
    if (threadIdx.x == 64) {
        const float nfxB = -mf.fx * mf.B;
        tab.inv[0] = f2_dup(-mf.u0);
        tab.inv[1] = f2_dup(-mf.v0);
        tab.inv[2] = f2_dup(mf.B);
        tab.inv[3] = f2_dup(mf.fx / mf.fy);
        tab.inv[4] = f2_dup(nfxB);
        tab.inv[5] = f2_dup(-1.0f);
#pragma unroll
        for (int q = 0; q < 3; ++q) tab.pred[q] = f2_dup(mf.feat_std[q]);
        tab.pred[3] = f2_dup((float)dt);
        tab.pred[4] = f2_dup(0.5f * (float)dt * (float)dt);
        tab.meas[0] = f2_dup(-mf.fx);
        tab.meas[1] = f2_dup(-mf.fy);
        tab.meas[2] = f2_dup(mf.u0);
        tab.meas[3] = f2_dup(mf.v0);
        tab.meas[4] = f2_dup(nfxB);
    }
    if (threadIdx.x == 0) {
        if (p == 0 && c == 0) b.flags[3] = b.flags[1] = 0;   // no parent listed for a second merge launch yet
        double zero[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        const Pose<float> pu = make_pose<float>(fixed ? zero : b.ext + 12 * p);
#pragma unroll
        for (int i = 0; i < 9; ++i) tab.upd_r[i] = f2_dup(pu.R[i]);
#pragma unroll
        for (int i = 0; i < 3; ++i) tab.upd_t[i] = f2_dup(-pu.t[i]);
        if (c == 0) {
            b.surv_n[p] = 0;
            atomicAdd(&b.counters[6], (unsigned long long)G * (unsigned long long)M);
            atomicAdd(&b.counters[10], (unsigned long long)G);
        }
        s_rd = 0;
        s_wr = 0;
    }
    __syncthreads();

    const float invP = 1.0f / (float)P;
    const float min_w = (float)prm.min_weight;
    const float two_u0 = 2 * mf.u0, two_v0 = 2 * mf.v0;
    // fitted row element of this lane: W, pD, mean (lanes 2-7), covariance entry (ra, rb) (8-28)
    int ra = 6, rb = 6;
    if (lane >= 8 && lane < 29) {
        int e = lane - 8, aa = 0;
        while ((aa + 1) * (aa + 2) / 2 <= e) ++aa;
        ra = aa;
        rb = e - aa * (aa + 1) / 2;
    }
    // moments this lane sums (see the sweep below): rows x, y, z; places of xx, xy, xz, yz among the moments
    const int task = lane & 7, cls = (lane >> 3) & 1, hf = lane >> 4;
    const int tx = moment_row_x(task), ty = moment_row_y(task), tz = moment_row_z(task);
    const int pl_xx = moment_place(tx, tx), pl_xy = moment_place(tx, ty), pl_xz = moment_place(tx, tz), pl_yz = moment_place(ty, tz);

    const int nW = G > gw ? (G - gw + nwp - 1) / nwp : 0;   // this warp's Gaussians
    for (int k0 = 0; k0 < nW; k0 += kQuadSlots) {
        const int nS = min(kQuadSlots, nW - k0);
        int n_merged;
        {   // lane k < nS: entry of Gaussian k, then sorted into slots (drawn ones first)
            int my_ref = 0;
            float my_W = 0.0f;
            if (lane < nS) {
                const size_t erow = (size_t)row * prm.Gcap + gw + nwp * (k0 + lane);
                my_ref = b.map_ref[cur][erow];
                my_W = has_pred ? b.map[cur][erow * kRow] * (float)prm.ps : b.map[cur][erow * kRow];
            }
            const unsigned merged = __ballot_sync(0xffffffffu, lane < nS && my_ref < 0);
            const unsigned writes = __ballot_sync(0xffffffffu, lane < nS && my_W >= min_w);
            n_merged = __popc(merged);
            if (lane == 0) {
                atomicAdd(&s_rd, nS - n_merged);
                atomicAdd(&s_wr, __popc(writes));
            }
            if (lane < nS) {
                const int below = __popc(merged & ((1u << lane) - 1u));
                const int at = (merged >> lane) & 1u ? below : n_merged + lane - below;
                slots[at] = make_int4(my_ref, __float_as_int(my_W), gw + nwp * (k0 + lane), at % NR);
            }
            __syncwarp();
        }
        int swept = 0;
        for (int g0 = 0; g0 < nS; g0 += TG) {
            const int nR = min(TG, nS - g0);
            // factor (21) and mean (6) of the round's drawn ones: every load before the first store
            // (at PC, where the round's size is known)
            constexpr int kAhead = PC > 0 ? quad_round(PC) : 1;
            for (int q0 = 0; q0 < nR; q0 += kAhead) {
                float lv[kAhead];
#pragma unroll
                for (int q = 0; q < kAhead; ++q)
                    if (q0 + q < nR && g0 + q0 + q < n_merged && lane < 27)
                        lv[q] = __ldg(b.map[cur] + ((size_t)row * prm.Gcap + slots[g0 + q0 + q].z) * kRow + (lane < 21 ? 7 + lane : lane - 20));
#pragma unroll
                for (int q = 0; q < kAhead; ++q)
                    if (q0 + q < nR && g0 + q0 + q < n_merged && lane < 27) Lw[(q0 + q) * 28 + lane] = f2_dup(lv[q]);
            }
            __syncwarp();
            const int nunits = nR * nu;
            int q = lane / nu, i4 = lane - q * nu;   // this lane's unit: Gaussian q of the round, its samples 4 i4 ..
            for (int u0 = 0; u0 < nunits; u0 += 32) {
                // lanes past the last unit repeat it: they store the same values to the same places
                int uq = q, ui = i4;
                if (u0 + lane >= nunits) {
                    uq = nR - 1;
                    ui = nu - 1;
                }
                const int s = 4 * ui, og = g0 + uq;
                const int4 sl = slots[og];
                const int ref = sl.x, j = sl.z, ring = sl.w;
                F2 X[2][6];
                float om[4] = {invP, invP, invP, invP};
                if (ref < 0) {   // merged component: draw (.cu:640-690) and map to world (.cu:1222-1286)
                    const uint32_t key_i = (uint32_t)(-1 - ref);
                    F2 z[2][6];
                    quad_draw(prm.rk, (uint32_t)s, key_i, (uint32_t)row, sample_frame, z[0]);
                    quad_draw(prm.rk, (uint32_t)s + 2u, key_i, (uint32_t)row, sample_frame, z[1]);
                    // y = L z + mean
                    const ulonglong2* line = reinterpret_cast<const ulonglong2*>(Lw + uq * 28);
                    F2 el[28], y[2][6];
#pragma unroll
                    for (int i = 0; i < 14; ++i) {
                        const ulonglong2 v = line[i];
                        el[2 * i] = v.x;
                        el[2 * i + 1] = v.y;
                    }
                    quad_ltz(el, z[0], y[0]);
                    quad_ltz(el, z[1], y[1]);
                    quad_invert(tab, y[0], X[0]);
                    quad_invert(tab, y[1], X[1]);
                } else {         // non-detection cloud carried from the previous frame
                    // (only read in this kernel; 16-byte aligned: rows of Ps values, a multiple of 8)
                    const float* cl = b.cloud[cur] + (size_t)ref * 7 * Ps + s;
#pragma unroll
                    for (int a = 0; a < 6; ++a) {
                        const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(cl + a * Ps));
                        X[0][a] = v.x;
                        X[1][a] = v.y;
                    }
                    const float4 v = __ldg(reinterpret_cast<const float4*>(cl + 6 * Ps));
                    om[0] = v.x;
                    om[1] = v.y;
                    om[2] = v.z;
                    om[3] = v.w;
                }
                if (has_pred) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t w0[4], w1[4];
                        const uint32_t c0 = ctr_word3(pred_frame, ST_FEAT, 0), s0 = (uint32_t)(s + 2 * h);
                        philox_rk(s0, (uint32_t)j, (uint32_t)p, c0, prm.rk, w0);
                        philox_rk(s0 + 1u, (uint32_t)j, (uint32_t)p, c0, prm.rk, w1);
                        quad_predict(tab, w0, w1, X[h]);
                    }
                }
                F2 y[2][6];
                quad_measure(tab, X[0], y[0]);
                quad_measure(tab, X[1], y[1]);
                // in view (kernels.cu:37-41), pD, the sample's weight
                bool in[4], nz[4];
                float pd[4], wp[4];
                const bool whole = P % 4 == 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    auto at = [&](int a) { return i & 1 ? f2_hi(y[i >> 1][a]) : f2_lo(y[i >> 1][a]); };
                    in[i] = (whole || s + i < P) && at(0) >= 0.0f && at(0) <= two_u0 && at(1) >= 0.0f && at(1) <= two_v0 &&
                            at(2) >= 0.0f;
                    pd[i] = in[i] ? mf.pd : 0.0f;
                    wp[i] = om[i] * pd[i];
                    nz[i] = wp[i] != 0.0f;
                }
                // the candidate non-detection cloud (evict-first: read again only next frame)
                if (__int_as_float(sl.y) >= min_w) {
                    float* co = b.cloud[cur ^ 1] + ((size_t)p * prm.Gcap + j) * 7 * Ps + s;
#pragma unroll
                    for (int a = 0; a < 6; ++a)
                    {
                        __stcs(reinterpret_cast<F2*>(co + a * Ps), X[0][a]);
                        __stcs(reinterpret_cast<F2*>(co + a * Ps + 2), X[1][a]);
                    }
                    __stcs(reinterpret_cast<float4*>(co + 6 * Ps), make_float4(1.0f - pd[0], 1.0f - pd[1], 1.0f - pd[2], 1.0f - pd[3]));
                }
                // the shift: the Gaussian's first sample, if finite, else 0
                if (s == 0) {
#pragma unroll
                    for (int a = 0; a < 6; ++a) {
                        const float v = f2_lo(y[0][a]);
                        nsh[ring * 6 + a] = f2_dup(isfinite(v) ? -v : -0.0f);
                    }
                }
                marks[ring * quad_marks(P) + ui] =
                    (unsigned char)((in[0] ? 1 : 0) | (in[1] ? 2 : 0) | (in[2] ? 4 : 0) | (in[3] ? 8 : 0) | (nz[0] ? 16 : 0) |
                                    (nz[1] ? 32 : 0) | (nz[2] ? 64 : 0) | (nz[3] ? 128 : 0));
                __syncwarp();
                // moment rows r d, r, w' (zeros for a sample of zero weight); r = sqrt(w')
                {
                    float* Ys = rows + ring * rowsz + s;
                    float r[4];
                    bool tiny = false;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool norm = wp[i] >= 1.17549435e-38f;
                        r[i] = norm ? wp[i] * rsqrt_ftz(wp[i]) : 0.0f;
                        tiny |= nz[i] && !norm;
                    }
                    if (tiny) {   // subnormal weights (or a negative or NaN one, set by the caller)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (nz[i] && !(wp[i] >= 1.17549435e-38f)) r[i] = sqrtf(wp[i]);
                    }
                    const F2 ra2 = pack_f32x2(r[0], r[1]), rb2 = pack_f32x2(r[2], r[3]);
                    const ulonglong2* sh = reinterpret_cast<const ulonglong2*>(nsh + ring * 6);
                    F2 t0[6], t1[6];
#pragma unroll
                    for (int a = 0; a < 6; ++a) {
                        const F2 v = a & 1 ? sh[a >> 1].y : sh[a >> 1].x;
                        t0[a] = f2_mul(ra2, f2_add(y[0][a], v));
                        t1[a] = f2_mul(rb2, f2_add(y[1][a], v));
                    }
                    if (!__all_sync(0xffffffffu, nz[0] && nz[1] && nz[2] && nz[3])) {   // (0 times inf or NaN is NaN)
#pragma unroll
                        for (int a = 0; a < 6; ++a) {
                            t0[a] = pack_f32x2(nz[0] ? f2_lo(t0[a]) : 0.0f, nz[1] ? f2_hi(t0[a]) : 0.0f);
                            t1[a] = pack_f32x2(nz[2] ? f2_lo(t1[a]) : 0.0f, nz[3] ? f2_hi(t1[a]) : 0.0f);
                        }
                    }
#pragma unroll
                    for (int a = 0; a < 6; ++a) *reinterpret_cast<ulonglong2*>(Ys + a * sY) = make_ulonglong2(t0[a], t1[a]);
                    *reinterpret_cast<float4*>(Ys + 6 * sY) = make_float4(r[0], r[1], r[2], r[3]);
                    *reinterpret_cast<float4*>(Ys + 7 * sY) = make_float4(wp[0], wp[1], wp[2], wp[3]);
                }
                q += 32 / nu;
                i4 += 32 % nu;
                if (i4 >= nu) {
                    i4 -= nu;
                    ++q;
                }
                __syncwarp();
                // ---- fit the Gaussians whose samples are all staged, two at a time
                const int done = g0 + min(nR, (u0 + 32) / nu);
                while (done - swept >= 2 || (done == nS && swept < nS)) {
                    const int n = min(2, done - swept);
                    {   // the sweep: lanes 16 g + 8 k + t sum the products of rows x, y, z of
                        // Gaussian g over the samples 4 i + 2 k, 4 i + 2 k + 1
                        const float* base = rows + ((swept + (hf < n ? hf : 0)) % NR) * rowsz + 2 * cls;
                        const float *px = base + tx * sY, *py = base + ty * sY, *pz = base + tz * sY;
                        F2 xx = 0ull, xy = 0ull, xz = 0ull, yz = 0ull;
#pragma unroll 5
                        for (int i = 0; i < nu; ++i) {
                            const F2 vx = *reinterpret_cast<const F2*>(px + 4 * i), vy = *reinterpret_cast<const F2*>(py + 4 * i),
                                     vz = *reinterpret_cast<const F2*>(pz + 4 * i);
                            xx = f2_fma(vx, vx, xx);
                            xy = f2_fma(vx, vy, xy);
                            xz = f2_fma(vx, vz, xz);
                            yz = f2_fma(vy, vz, yz);
                        }
                        float m0 = f2_lo(xx) + f2_hi(xx), m1 = f2_lo(xy) + f2_hi(xy), m2 = f2_lo(xz) + f2_hi(xz),
                              m3 = f2_lo(yz) + f2_hi(yz);
                        m0 += __shfl_xor_sync(0xffffffffu, m0, 8);
                        m1 += __shfl_xor_sync(0xffffffffu, m1, 8);
                        m2 += __shfl_xor_sync(0xffffffffu, m2, 8);
                        m3 += __shfl_xor_sync(0xffffffffu, m3, 8);
                        __syncwarp();   // every row is read: the moments go where Gaussian g's first row was
                        if (cls == 0 && hf < n) {
                            float* d = rows + ((swept + hf) % NR) * rowsz;
                            d[pl_xx] = m0;
                            if (task != 7) {
                                d[pl_xy] = m1;
                                d[pl_xz] = m2;
                                d[pl_yz] = m3;
                            }
                        }
                        __syncwarp();
                    }
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        if (g >= n) break;
                        const int4 sg = slots[swept + g];
                        const int rg = sg.w;
                        unsigned mk = 0;   // samples in view + 512 x units with a weight
                        for (int i = lane; i < nu; i += 32) {
                            const unsigned m = marks[rg * quad_marks(P) + i];
                            mk += __popc(m & 15u) + (m > 15u ? 512u : 0u);
                        }
                        mk = __reduce_add_sync(0xffffffffu, mk);
                        const float pbar = s_pbar[mk & 511u], W = __int_as_float(sg.y);
                        const float* mg = rows + rg * rowsz;
                        float fv = lane == 0 ? W : pbar;
                        if (mk > 511u) {
                            const float S0 = mg[0], S2 = mg[1];
                            const float inv = __frcp_rn(S0), scale = 1.0f + S2 * inv * inv;
                            if (lane >= 8)
                                fv = __fmaf_rn(-__fmul_rn(mg[2 + ra], inv), __fmul_rn(mg[2 + rb], inv), __fmul_rn(mg[lane], inv)) * scale;
                            else if (lane >= 2) fv = __fadd_rn(__fmul_rn(mg[lane], inv), -f2_lo(nsh[rg * 6 + lane - 2]));
                        } else if (pbar > 0.0f) {
                            const float v = quad_unweighted(prm, tab, b.map[cur] + ((size_t)row * prm.Gcap + sg.z) * kRow,
                                                            b.cloud[cur], Ps, sg.x, sg.z, p, row, has_pred, pred_frame,
                                                            sample_frame, rows + rg * rowsz, sY, ra, rb);
                            if (lane >= 2) fv = v;
                            if (lane == 0) atomicAdd(&b.counters[14], 1ull);
                        } else {   // entirely out of view: never used downstream (its log-constant is -inf)
                            if (lane >= 8) fv = 0.0f;
                            else if (lane >= 2) fv = -f2_lo(nsh[rg * 6 + lane - 2]);
                        }
                        float* fr = b.fit + ((size_t)p * prm.Gcap + sg.z) * kRow;
                        if (lane < 29) fr[lane] = fv;
                    }
                    __syncwarp();   // the rows' reads end before their next staging
                    swept += n;
                }
            }
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&b.counters[8], (unsigned long long)s_rd);
        atomicAdd(&b.counters[9], (unsigned long long)s_wr);
    }
}

}  // namespace scphd
