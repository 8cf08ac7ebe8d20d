// stage_quad.cuh -- one RK stage with four real strips per transform unit.
//
// A quad is four adjacent strips of one job: two complex strips A = s0 + i s1
// and B = s2 + i s3 (neighbours share a transform, and with it its rounding:
// their amplitudes are closest), stored position by position as one 16-byte
// element (s0, s2, s1, s3) = (re A, re B, im A, im B).  What this buys over the
// complex-strip form of stage_kernel.cuh, which computes the same transform
// with the same constants:
//   * a column job's element is four adjacent columns of one row, i.e. one
//     16-byte global access and one 16-byte shared access, no shuffling; a row
//     job turns four 16-byte row loads into four elements by renaming registers;
//   * sums and rotations act on both complex strips at once (add / sub / fma
//     .f32x2; on sm_103a such an instruction occupies the issue port for two
//     cycles -- 2.0-2.2 measured -- so it does not raise the FP32 rate, but it
//     halves the code: the plain form stalls 1.7 cycles per issue on
//     instruction fetch);
//   * twiddles, filter values and addresses are formed once for four strips,
//     and shared memory is accessed with half as many instructions.
//
// A job is described by one self-contained 208-byte record (QJob): sources,
// neighbours, coefficients and output, so a CTA reads its record and then its
// data -- two dependent round trips where the plain form chains five (job,
// domain, first-step flag, neighbour domain, data).  That chain, not the
// arithmetic, is what a stage of a small scene spends its time on.
//
// Measured (GB300, one RK stage of a 96-scene batch, fastest complex-strip
// variant -> fastest of these, us): length 128 240 -> 172, 256 107 -> 73, 512
// 160 -> 118, 1024 177 -> 139, 2048 53 -> 49; length 8192 of the 8192^2 scene
// 2833 -> 2380.  (Length 128 took 163 as first built, with strips 0 and 2, 1 and
// 3 sharing a transform; neighbours share one for their rounding.)  What bounds
// lengths up to 1024 there: the L1 data path (69-76 % of its wavefronts; DRAM
// 26-37 %, issue 44-49 %), i.e. the passes' trips through shared memory; about
// 30 % of the shared load wavefronts are bank conflicts.  Counters:
// profiles/stage_quad_batch.md.
//
// The kernels may be launched with programmatic stream serialisation: a CTA
// reads its record and copies its tables before it waits for the previous
// launch (griddepcontrol.wait), and lets the next launch start only after
// that wait, so a launch that has started knows that everything before its
// predecessor has completed.
#pragma once
#include "stage_kernel.cuh"

namespace pstd {

// ---------------------------------------------------------------- packed pairs
using u64 = unsigned long long;
__device__ __forceinline__ u64 pk(float2 a) { return (u64)__float_as_uint(a.x) | ((u64)__float_as_uint(a.y) << 32); }
__device__ __forceinline__ float2 upk(u64 a) {
    return make_float2(__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)));
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}

// the same position of both complex strips
struct Q2 {
    float2 re, im;
};
__device__ __forceinline__ Q2 qadd(Q2 a, Q2 b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ Q2 qsub(Q2 a, Q2 b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a + rot(b), a - rot(b) with rot = * -i (forward) or * +i (inverse)
template <bool INV>
__device__ __forceinline__ Q2 qaddrot(Q2 a, Q2 b) {
    return INV ? Q2{sub2(a.re, b.im), add2(a.im, b.re)} : Q2{add2(a.re, b.im), sub2(a.im, b.re)};
}
template <bool INV>
__device__ __forceinline__ Q2 qsubrot(Q2 a, Q2 b) {
    return INV ? Q2{add2(a.re, b.im), sub2(a.im, b.re)} : Q2{sub2(a.re, b.im), add2(a.im, b.re)};
}
// both strips times the same complex number (scalar products: a broadcast pair
// would cost two moves per component and issue no faster)
__device__ __forceinline__ Q2 qmul(Q2 a, float2 w) {
    const float2 u = cmul(make_float2(a.re.x, a.im.x), w), v = cmul(make_float2(a.re.y, a.im.y), w);
    return {make_float2(u.x, v.x), make_float2(u.y, v.y)};
}
__device__ __forceinline__ Q2 qmulc(Q2 a, float2 w) {
    const float2 u = cmulc(make_float2(a.re.x, a.im.x), w), v = cmulc(make_float2(a.re.y, a.im.y), w);
    return {make_float2(u.x, v.x), make_float2(u.y, v.y)};
}
__device__ __forceinline__ Q2 q_of(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
__device__ __forceinline__ float4 f4_of(Q2 v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }

template <int K, bool INV>
__device__ __forceinline__ Q2 qtw16(Q2 a) {   // a * exp(-/+ 2 pi i K / 16), K not a multiple of 4
    constexpr float sg = INV ? 1.f : -1.f;
    constexpr float c = K == 2 ? PSTD_R2 : K == 6 ? -PSTD_R2 : K == 1 ? PSTD_C8 : K == 3 ? PSTD_S8
                      : K == 5 ? -PSTD_S8 : -PSTD_C8;
    constexpr float s = (K == 2 || K == 6) ? PSTD_R2 : (K == 1 || K == 7) ? PSTD_S8 : PSTD_C8;
    return qmul(a, make_float2(c, sg * s));
}

// the butterflies of stage_kernel.cuh (same order of operations) on a quad
template <int R, bool INV>
struct QDFT;
template <bool INV>
struct QDFT<2, INV> {
    static __device__ __forceinline__ void run(Q2* x) {
        const Q2 a = x[0], b = x[1];
        x[0] = qadd(a, b);
        x[1] = qsub(a, b);
    }
};
template <bool INV>
struct QDFT<4, INV> {
    static __device__ __forceinline__ void run(Q2* x) {
        const Q2 a = qadd(x[0], x[2]), b = qsub(x[0], x[2]);
        const Q2 c = qadd(x[1], x[3]), d = qsub(x[1], x[3]);
        x[0] = qadd(a, c);
        x[2] = qsub(a, c);
        x[1] = qaddrot<INV>(b, d);
        x[3] = qsubrot<INV>(b, d);
    }
};
template <bool INV>
struct QDFT<8, INV> {
    static __device__ __forceinline__ void run(Q2* x) {
        Q2 e[4] = {x[0], x[2], x[4], x[6]};
        Q2 o[4] = {x[1], x[3], x[5], x[7]};
        QDFT<4, INV>::run(e);
        QDFT<4, INV>::run(o);
        o[1] = qtw16<2, INV>(o[1]);
        o[3] = qtw16<6, INV>(o[3]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (k == 2) {
                x[k] = qaddrot<INV>(e[k], o[k]);
                x[k + 4] = qsubrot<INV>(e[k], o[k]);
            } else {
                x[k] = qadd(e[k], o[k]);
                x[k + 4] = qsub(e[k], o[k]);
            }
        }
    }
};
template <bool INV>
struct QDFT<16, INV> {
    static __device__ __forceinline__ void run(Q2* x) {
        Q2 e[8], o[8];
#pragma unroll
        for (int k = 0; k < 8; k++) { e[k] = x[2 * k]; o[k] = x[2 * k + 1]; }
        QDFT<8, INV>::run(e);
        QDFT<8, INV>::run(o);
        o[1] = qtw16<1, INV>(o[1]);
        o[2] = qtw16<2, INV>(o[2]);
        o[3] = qtw16<3, INV>(o[3]);
        o[5] = qtw16<5, INV>(o[5]);
        o[6] = qtw16<6, INV>(o[6]);
        o[7] = qtw16<7, INV>(o[7]);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (k == 4) {
                x[k] = qaddrot<INV>(e[k], o[k]);
                x[k + 8] = qsubrot<INV>(e[k], o[k]);
            } else {
                x[k] = qadd(e[k], o[k]);
                x[k + 8] = qsub(e[k], o[k]);
            }
        }
    }
};

// ---------------------------------------------------------------- variants
// L, quads per CTA, threads, min CTAs per SM, radices; TSM = 1: twiddles and
// the job's filter are copied to shared memory while the strips are on their
// way (a CTA that runs alone on its SM finds them in no cache)
// FUSE = 1: the last pass updates the fields itself
template <int L_, int CS_, int NT_, int MINB_, int R0_, int R1_, int R2_ = 0, int R3_ = 0, int TSM_ = 0, int FUSE_ = 0>
struct QCfg {
    static constexpr int L = L_, CS = CS_, NT = NT_, MINB = MINB_, TSM = TSM_, CTW = 1, FUSE = FUSE_;
    static constexpr int R0 = R0_, R1 = R1_, R2 = R2_, R3 = R3_;
    static constexpr int NP = R3_ ? 4 : (R2_ ? 3 : 2);
    static_assert(R0 * R1 * (R2 ? R2 : 1) * (R3 ? R3 : 1) == L, "radix plan must multiply to L");
    static_assert(NT % CS == 0 && CS <= NT, "threads are split evenly over the quads");
    static constexpr int RL = R3 ? R3 : (R2 ? R2 : R1);   // last radix
    // one padding element per 2^SH positions: the last pass's threads read
    // blocks RL apart, eight of them must meet distinct 16-byte bank groups
    static constexpr int SH = RL >= 16 ? 4 : 3;
    static constexpr int RAW = (L + (L >> SH) + 7) / 8 * 8;
    // pitch of a quad: CS quads at one position (a column job's accesses) in distinct bank groups
    static constexpr int SP = RAW + (CS == 1 ? 0 : CS >= 8 ? 1 : 8 / CS);
    static constexpr int M1 = L / R0, M2 = R1 ? M1 / R1 : 1;
    static constexpr int T1 = (L / R0) * tw_entry(R0);
    static constexpr int T2 = T1 + (NP > 2 ? (M1 / R1) * tw_entry(R1) : 0);
    static constexpr int TWN = T2 + (NP > 3 ? (M2 / R2) * tw_entry(R2) : 0);
    static constexpr int DATA = CS * SP * 16;
    static constexpr int JOB = DATA + (TSM ? (TWN + L) * 8 : 0);   // byte offset of the job record's copy
    static constexpr int SMEM = JOB + (int)sizeof(QJob);
    static_assert(sizeof(QJob) % 16 == 0 && JOB % 16 == 0, "the record is copied in 16-byte pieces");
    static constexpr int TPQ = NT / CS;   // threads per quad in gather and epilogue
    // 16-byte loads of a column job's thread in flight (two fields each), and
    // row-job chunks: twice as many where a thread has that many elements and
    // the register budget is 100 and more (shorter strips: the loads past the
    // end cost a small scene's chained step 10 us of 55)
    static constexpr int UC = 65536 / (NT * MINB) >= 100 && L / TPQ >= 16 ? 8 : 4;
    static constexpr int PRE = UC == 8;   // stage-start values loaded ahead of the last inverse pass
};

template <class C>
__device__ __forceinline__ constexpr int qoff(int p) { return p + (p >> C::SH); }

template <class C, int R, int M, int TOFF, bool PRUNE>
__device__ __forceinline__ void qfwd_pass(float4* sm, const float2* tw, int tid, int lim) {
    constexpr int Q = M / R, PER = C::L / R, ITEMS = C::CS * PER;
#pragma unroll 1
    for (int it = tid; it < ITEMS; it += C::NT) {
        const int g = it / PER, b = it % PER, blk = b / Q, n1 = b % Q;
        float4* base = sm + g * C::SP + blk * (M + (M >> C::SH)) + n1 + (n1 >> C::SH);
        float2 w[R];
        pass_twiddles<C, R, C::TSM != 0>(tw + TOFF, n1, w);
        Q2 x[R];
#pragma unroll
        for (int q = 0; q < R; q++)
            x[q] = (!PRUNE || n1 + q * Q < lim) ? q_of(base[qoff<C>(q * Q)]) : Q2{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        QDFT<R, false>::run(x);
        base[0] = f4_of(x[0]);
#pragma unroll
        for (int k = 1; k < R; k++) base[qoff<C>(k * Q)] = f4_of(qmul(x[k], w[k]));
    }
}

template <class C, int R, int M, int TOFF, bool PRUNE>
__device__ __forceinline__ void qinv_pass(float4* sm, const float2* tw, int tid, int lo, int hi) {
    constexpr int Q = M / R, PER = C::L / R, ITEMS = C::CS * PER;
#pragma unroll 1
    for (int it = tid; it < ITEMS; it += C::NT) {
        const int g = it / PER, b = it % PER, blk = b / Q, n1 = b % Q;
        float4* base = sm + g * C::SP + blk * (M + (M >> C::SH)) + n1 + (n1 >> C::SH);
        float2 w[R];
        pass_twiddles<C, R, C::TSM != 0>(tw + TOFF, n1, w);
        Q2 x[R];
        x[0] = q_of(base[0]);
#pragma unroll
        for (int k = 1; k < R; k++) x[k] = qmulc(q_of(base[qoff<C>(k * Q)]), w[k]);
        QDFT<R, true>::run(x);
#pragma unroll
        for (int q = 0; q < R; q++)
            if (!PRUNE || (n1 + q * Q >= lo && n1 + q * Q < hi)) base[qoff<C>(q * Q)] = f4_of(x[q]);
    }
}

// last forward pass, filter ([h][block] pairs of values), first inverse pass
template <class C, int R>
__device__ __forceinline__ void qmid_pass(float4* sm, const float4* filt, int tid) {
    constexpr int PER = C::L / R, ITEMS = C::CS * PER;
#pragma unroll 1
    for (int it = tid; it < ITEMS; it += C::NT) {
        const int g = it / PER, blk = it % PER;
        float4* base = sm + g * C::SP + qoff<C>(blk * R);
        Q2 x[R];
#pragma unroll
        for (int q = 0; q < R; q++) x[q] = q_of(base[q]);
        QDFT<R, false>::run(x);
#pragma unroll
        for (int h = 0; h < R / 2; h++) {
            const float4 v = tload<C::TSM != 0>(filt + h * PER + blk);
            x[2 * h] = qmul(x[2 * h], make_float2(v.x, v.y));
            x[2 * h + 1] = qmul(x[2 * h + 1], make_float2(v.z, v.w));
        }
        QDFT<R, true>::run(x);
#pragma unroll
        for (int q = 0; q < R; q++) base[q] = f4_of(x[q]);
    }
}

// all passes but the last inverse one
template <class C>
__device__ __forceinline__ void qconvolve(float4* sm, const float2* tw, const float4* filt, int tid, int z0) {
    qfwd_pass<C, C::R0, C::L, 0, true>(sm, tw, tid, z0);
    __syncthreads();
    if constexpr (C::NP > 2) {
        qfwd_pass<C, C::R1, C::M1, C::T1, false>(sm, tw, tid, 0);
        __syncthreads();
    }
    if constexpr (C::NP > 3) {
        qfwd_pass<C, C::R2, C::M2, C::T2, false>(sm, tw, tid, 0);
        __syncthreads();
    }
    qmid_pass<C, C::RL>(sm, filt, tid);
    __syncthreads();
    if constexpr (C::NP > 3) {
        qinv_pass<C, C::R2, C::M2, C::T2, false>(sm, tw, tid, 0, 0);
        __syncthreads();
    }
    if constexpr (C::NP > 2) {
        qinv_pass<C, C::R1, C::M1, C::T1, false>(sm, tw, tid, 0, 0);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- loads
// Field loads stay out of L1 (streamed once per job; and a launch that starts
// early must not see lines an earlier launch left there).
__device__ __forceinline__ float qld(const float* p) { return __ldcg(p); }
__device__ __forceinline__ float4 qld4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }

struct QPtr {
    const float *a, *b;   // b: py where p0 = px + py is formed on the way, else nullptr
    int pitch, flags;
};

__device__ __forceinline__ QPtr qsource(const StageArgs& A, const QSrc& s, bool vel, bool first) {
    const float* base = (s.flags & QS_FIXED) ? A.fixed : A.in;
    QPtr r;
    r.pitch = s.pitch;
    r.flags = s.flags;
    r.a = base + s.oa;
    r.b = nullptr;
    if (!vel) {
        if (A.stage == 0 && ((s.flags & QS_PML) || first)) r.a = A.p0 + s.op0;   // stale / initial p0
        else r.b = base + s.ob;
    }
    return r;
}

// element (strips 4g .. 4g+3) of position `pos` of a source; absent strips are zero
__device__ __forceinline__ float4 qelem(const QPtr& s, bool ydir, int g, long long pos, int count) {
    float4 v;
    if (ydir && (s.flags & QS_ALIGNED)) {
        const long long e = pos * s.pitch + 4 * g;
        v = qld4(s.a + e);
        if (s.b) v = add4(v, qld4(s.b + e));
        if (4 * g + 4 > count) {
            if (4 * g + 1 > count) v.x = 0.f;
            if (4 * g + 2 > count) v.y = 0.f;
            if (4 * g + 3 > count) v.z = 0.f;
            v.w = 0.f;
        }
    } else {
        float t[4];
        const long long e0 = ydir ? pos * s.pitch + 4 * g : (long long)(4 * g) * s.pitch + pos;
        const long long st = ydir ? 1 : s.pitch;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            t[q] = 0.f;
            if (4 * g + q < count) {
                t[q] = qld(s.a + e0 + q * st);
                if (s.b) t[q] = __fadd_rn(t[q], qld(s.b + e0 + q * st));
            }
        }
        v = make_float4(t[0], t[1], t[2], t[3]);
    }
    return v;
}

__device__ __forceinline__ float4 qband(float4 raw, float4 mir, float T, float R, float w) {
    const float2 t2 = make_float2(T, T), r2 = make_float2(R, R), w2 = make_float2(w, w);
    const float2 a = mul2(add2(mul2(make_float2(raw.x, raw.y), t2), mul2(make_float2(mir.x, mir.y), r2)), w2);
    const float2 b = mul2(add2(mul2(make_float2(raw.z, raw.w), t2), mul2(make_float2(mir.z, mir.w), r2)), w2);
    return make_float4(a.x, a.y, b.x, b.y);
}

// ---------------------------------------------------------------- gather
// Strips to positions W .. W+n of each quad, the two interface bands around
// them.  The neighbours' values are loaded before the strips, the mirrored own
// values are read back from shared memory (the strip's ends), so every field
// value is loaded once.  All loads of a thread are issued before the first one
// is used (sums px + py come after them): with a sum behind every load a job
// paid one memory round trip per load.
__device__ __forceinline__ float4 qperm(float4 v) { return make_float4(v.x, v.z, v.y, v.w); }   // strips <-> element

enum QKind { QK_ROWS, QK_COLS, QK_ANY };   // x strips; y strips on 16-byte boundaries; y strips elsewhere

__device__ __forceinline__ float4 qmask(float4 v, int m) {   // keep the first m strips
    if (m < 1) v.x = 0.f;
    if (m < 2) v.y = 0.f;
    if (m < 3) v.z = 0.f;
    if (m < 4) v.w = 0.f;
    return v;
}

template <class C, int KIND, bool TWO>
__device__ __forceinline__ void qgather_k(float4* smq, const StageArgs& A, const QJob& J, const QPtr& own, const QPtr& lo,
                                          const QPtr& hi, int g, int l) {
    constexpr int TPQ = C::TPQ, NB = (64 + TPQ - 1) / TPQ < 4 ? (64 + TPQ - 1) / TPQ : 4;
    const bool vel = J.kind & JK_VEL, h1 = !(lo.flags & QS_NONE), h2 = !(hi.flags & QS_NONE);
    const int W = J.W, n = J.n, s0 = 4 * g, m = J.count - s0;   // m: live strips of the quad
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* wl = A.win + J.wtab;   // window.head(W) at 0, its tail at W + 1
    float4 ra[NB], rb[NB];
    float wv[NB];
#pragma unroll
    for (int q = 0; q < NB; q++) {
        const int j = l + q * TPQ;
        const bool low = j < W, need = j < 2 * W && m > 0 && (low ? h1 : h2);
        const float *sa = low ? lo.a : hi.a, *sb = low ? lo.b : hi.b;
        const long long pitch = low ? lo.pitch : hi.pitch;
        const int pos = low ? j : j - W;
        ra[q] = rb[q] = zero;
        wv[q] = 0.f;
        if (j < 2 * W) wv[q] = __ldg(wl + j + (low ? 0 : 1));
        if constexpr (KIND == QK_ROWS) {
            const float *pa = sa + s0 * pitch + pos, *pb = sb + s0 * pitch + pos;
            if (need) ra[q].x = qld(pa);
            if (need && m > 1) ra[q].y = qld(pa + pitch);
            if (need && m > 2) ra[q].z = qld(pa + 2 * pitch);
            if (need && m > 3) ra[q].w = qld(pa + 3 * pitch);
            if constexpr (TWO) {
                const bool nb = need && sb;
                if (nb) rb[q].x = qld(pb);
                if (nb && m > 1) rb[q].y = qld(pb + pitch);
                if (nb && m > 2) rb[q].z = qld(pb + 2 * pitch);
                if (nb && m > 3) rb[q].w = qld(pb + 3 * pitch);
            }
        } else if constexpr (KIND == QK_COLS) {
            const long long e = pos * pitch + s0;
            if (need) ra[q] = qld4(sa + e);
            if (TWO && need && sb) rb[q] = qld4(sb + e);
        } else {
            if (need) ra[q] = qelem(low ? lo : hi, true, g, pos, J.count);
        }
    }
    if constexpr (KIND == QK_COLS) {
        const float *a = own.a + s0, *b = own.b + s0;
        const long long pitch = own.pitch;
#pragma unroll 1
        for (int i0 = l; i0 < n; i0 += C::UC * TPQ) {
            float4 ua[C::UC], ub[C::UC];
#pragma unroll
            for (int q = 0; q < C::UC; q++) {
                const int i = i0 + q * TPQ;
                ua[q] = ub[q] = zero;
                if (i < n && m > 0) ua[q] = qld4(a + i * pitch);
                if (TWO && i < n && m > 0 && own.b) ub[q] = qld4(b + i * pitch);
            }
#pragma unroll
            for (int q = 0; q < C::UC; q++) {
                const int i = i0 + q * TPQ;
                if constexpr (TWO) ua[q] = add4(ua[q], ub[q]);
                if (m < 4) ua[q] = qmask(ua[q], m);
                if (i < n) smq[qoff<C>(W + i)] = qperm(ua[q]);
            }
        }
    } else if constexpr (KIND == QK_ROWS) {
        // four rows, four positions each: rows start on 128-byte boundaries and
        // are padded past their last quad
        const int chunks = (n + 3) >> 2;
        const long long pitch = own.pitch;
        const float *a = own.a + s0 * pitch, *b = own.b + s0 * pitch;
        constexpr int UR = C::UC / 4;
#pragma unroll 1
        for (int c0 = l; c0 < chunks; c0 += UR * TPQ) {
            float4 u[UR][4], v[UR][4];
#pragma unroll
            for (int h = 0; h < UR; h++) {
                const int i = (c0 + h * TPQ) << 2;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    u[h][r] = v[h][r] = zero;
                    if (r < m && i < n) u[h][r] = qld4(a + r * pitch + i);
                    if (TWO && r < m && i < n && own.b) v[h][r] = qld4(b + r * pitch + i);
                }
            }
#pragma unroll
            for (int h = 0; h < UR; h++) {
                const int i = (c0 + h * TPQ) << 2, p = W + i;
                if constexpr (TWO) {
#pragma unroll
                    for (int r = 0; r < 4; r++) u[h][r] = add4(u[h][r], v[h][r]);
                }
                if (i < n) smq[qoff<C>(p)] = make_float4(u[h][0].x, u[h][2].x, u[h][1].x, u[h][3].x);
                if (i + 1 < n) smq[qoff<C>(p + 1)] = make_float4(u[h][0].y, u[h][2].y, u[h][1].y, u[h][3].y);
                if (i + 2 < n) smq[qoff<C>(p + 2)] = make_float4(u[h][0].z, u[h][2].z, u[h][1].z, u[h][3].z);
                if (i + 3 < n) smq[qoff<C>(p + 3)] = make_float4(u[h][0].w, u[h][2].w, u[h][1].w, u[h][3].w);
            }
        }
    } else {
#pragma unroll 1
        for (int i = l; i < n; i += TPQ) smq[qoff<C>(W + i)] = m > 0 ? qperm(qelem(own, true, g, i, J.count)) : zero;
    }
    __syncthreads();
    auto store = [&](int j, float4 r, float w) {
        const bool low = j < W;
        const int mp = low ? (vel ? W - j : W - 1 - j) : (vel ? n - 2 - (j - W) : n - 1 - (j - W));   // mirrored own position
        const float4 v = qband(qperm(r), smq[qoff<C>(W + mp)], low ? J.T1 : J.T2, low ? J.R1 : J.R2, w);
        smq[qoff<C>(low ? j : n + j)] = (low ? h1 : h2) ? v : zero;
    };
#pragma unroll
    for (int q = 0; q < NB; q++) {
        const int j = l + q * TPQ;
        if constexpr (TWO && KIND != QK_ANY) ra[q] = add4(ra[q], rb[q]);
        if (KIND == QK_COLS && m < 4) ra[q] = qmask(ra[q], m);
        if (j < 2 * W) store(j, ra[q], wv[q]);
    }
#pragma unroll 1
    for (int j = l + NB * TPQ; j < 2 * W; j += TPQ) {   // windows wider than 32
        const bool low = j < W;
        const float4 r = m > 0 && (low ? h1 : h2) ? qelem(low ? lo : hi, KIND != QK_ROWS, g, low ? j : j - W, J.count) : zero;
        store(j, r, __ldg(wl + j + (low ? 0 : 1)));
    }
    __syncthreads();
}

template <class C>
__device__ __forceinline__ void qgather(float4* sm, const StageArgs& A, const QJob& J, int tid) {
    const bool vel = J.kind & JK_VEL, ydir = J.kind & JK_Y;
    const bool first = A.stage == 0 && __ldcg(A.first_step + J.scene) != 0;
    // column jobs: neighbouring threads on neighbouring quads of one row; row
    // jobs: on neighbouring positions of one quad
    const int g = ydir ? tid % C::CS : tid / C::TPQ, l = ydir ? tid / C::CS : tid % C::TPQ;
    float4* smq = sm + g * C::SP;
    const QPtr own = qsource(A, J.own, vel, first), lo = qsource(A, J.lo, vel, first), hi = qsource(A, J.hi, vel, first);
    if (!ydir) {
        if (vel) qgather_k<C, QK_ROWS, false>(smq, A, J, own, lo, hi, g, l);
        else qgather_k<C, QK_ROWS, true>(smq, A, J, own, lo, hi, g, l);
    } else if ((own.flags & QS_ALIGNED) && (lo.flags & (QS_ALIGNED | QS_NONE)) && (hi.flags & (QS_ALIGNED | QS_NONE))) {
        if (vel) qgather_k<C, QK_COLS, false>(smq, A, J, own, lo, hi, g, l);
        else qgather_k<C, QK_COLS, true>(smq, A, J, own, lo, hi, g, l);
    } else {
        qgather_k<C, QK_ANY, true>(smq, A, J, own, lo, hi, g, l);
    }
}

// ---------------------------------------------------------------- epilogue
template <bool VEL>
__device__ __forceinline__ float2 qrk(float2 p, float2 d, float cdt, float rho, float c2, float rinv) {
    const float2 k = make_float2(cdt, cdt);
    if constexpr (VEL) {
        return sub2(p, mul2(k, mul2(mul2(d, make_float2(rho, rho)), make_float2(c2, c2))));
    } else {
        return make_float2(__fsub_rn(p.x, __fmul_rn(cdt, div_rho(d.x, rho, rinv))),
                           __fsub_rn(p.y, __fmul_rn(cdt, div_rho(d.y, rho, rinv))));
    }
}

// Stage-start values of a thread's first outputs, loaded before the last
// inverse pass (where the register budget allows): that pass hides their latency.
template <class C>
struct QPrev {
    float4 v[C::UC];
};
template <class C>
__device__ __forceinline__ void qprefetch(QPrev<C>& P, const StageArgs& A, const QJob& J, int tid) {
    const bool ydir = J.kind & JK_Y;
    const int g = ydir ? tid % C::CS : tid / C::TPQ, l = ydir ? tid / C::CS : tid % C::TPQ;
    const int count = J.count, nout = (J.kind & JK_VEL) ? J.n - 1 : J.n + 1, s0 = 4 * g;
    const long long pitch = J.pitch_out;
    const float* prev = A.prev + J.o_out;
    if (ydir) {
        if (!(J.own.flags & QS_ALIGNED) || s0 + 4 > count) return;
#pragma unroll
        for (int q = 0; q < C::UC; q++) {
            const int i = l + q * C::TPQ;
            if (i < nout) P.v[q] = qld4(prev + i * pitch + s0);
        }
    } else {
#pragma unroll
        for (int q = 0; q < C::UC; q++) {
            const int i = (l + (q >> 2) * C::TPQ) << 2, r = q & 3;
            if (i < nout && s0 + r < count) P.v[q] = qld4(prev + (s0 + r) * pitch + i);
        }
    }
}

template <class C, bool VEL, bool ATT, bool YDIR>
__device__ __forceinline__ void qepilogue_k(const float4* sm, const StageArgs& A, const QJob& J, int tid, const QPrev<C>& P) {
    const int g = YDIR ? tid % C::CS : tid / C::TPQ, l = YDIR ? tid / C::CS : tid % C::TPQ;
    const float4* smq = sm + g * C::SP;
    const int W = J.W, count = J.count, nout = VEL ? J.n - 1 : J.n + 1, s0 = 4 * g;
    const float cdt = J.cdt[A.stage], rho = J.rho, c2 = J.c2, rinv = J.rinv;
    const long long pitch = J.pitch_out;
    const float* prev = A.prev + J.o_out;
    float* out = A.out + J.o_out;
    const float* att = A.att + J.att;
    if (s0 >= count) return;
    if constexpr (YDIR) {
        if ((J.own.flags & QS_ALIGNED) && s0 + 4 <= count) {
#pragma unroll 1
            for (int i0 = l; i0 < nout; i0 += C::UC * C::TPQ) {
                float4 pv[C::UC];
#pragma unroll
                for (int q = 0; q < C::UC; q++) {
                    const int i = i0 + q * C::TPQ;
                    if (C::PRE && i0 == l) pv[q] = P.v[q];
                    else if (i < nout) pv[q] = qld4(prev + i * pitch + s0);
                }
#pragma unroll
                for (int q = 0; q < C::UC; q++) {
                    const int i = i0 + q * C::TPQ;
                    if (i >= nout) break;
                    const float4 d = qperm(smq[qoff<C>(W + i)]);
                    float2 u = qrk<VEL>(make_float2(pv[q].x, pv[q].y), make_float2(d.x, d.y), cdt, rho, c2, rinv);
                    float2 v = qrk<VEL>(make_float2(pv[q].z, pv[q].w), make_float2(d.z, d.w), cdt, rho, c2, rinv);
                    if constexpr (ATT) {
                        const float a = __ldg(att + i);
                        u = mul2(u, make_float2(a, a));
                        v = mul2(v, make_float2(a, a));
                    }
                    *reinterpret_cast<float4*>(out + i * pitch + s0) = make_float4(u.x, u.y, v.x, v.y);
                }
            }
        } else {
#pragma unroll 1
            for (int i = l; i < nout; i += C::TPQ) {
                const float4 d4 = qperm(smq[qoff<C>(W + i)]);
                const float d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (s0 + q >= count) break;
                    float v = rk_update(qld(prev + i * pitch + s0 + q), d[q], VEL, cdt, rho, c2, rinv);
                    if constexpr (ATT) v = __fmul_rn(v, __ldg(att + i));
                    out[i * pitch + s0 + q] = v;
                }
            }
        }
    } else {
        const int chunks = (nout + 3) >> 2;
#pragma unroll 1
        for (int c = l; c < chunks; c += C::TPQ) {
            const int i = c << 2;
            float4 pv[4];
#pragma unroll
            for (int r = 0; r < 4; r++)
                if (C::PRE && c == l) pv[r] = P.v[r];
                else if (C::PRE && C::UC == 8 && c == l + C::TPQ) pv[r] = P.v[r + C::UC - 4];
                else if (s0 + r < count) pv[r] = qld4(prev + (s0 + r) * pitch + i);   // rows are padded past their last quad
                else pv[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 d[4];
#pragma unroll
            for (int e = 0; e < 4; e++) d[e] = i + e < nout ? smq[qoff<C>(W + i + e)] : make_float4(0.f, 0.f, 0.f, 0.f);
            float a[4];
            if constexpr (ATT) {
#pragma unroll
                for (int e = 0; e < 4; e++) a[e] = i + e < nout ? __ldg(att + i + e) : 1.f;
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                if (s0 + r >= count) break;
                float v[4] = {pv[r].x, pv[r].y, pv[r].z, pv[r].w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float dv = r == 0 ? d[e].x : r == 1 ? d[e].z : r == 2 ? d[e].y : d[e].w;
                    v[e] = rk_update(v[e], dv, VEL, cdt, rho, c2, rinv);
                    if constexpr (ATT) v[e] = __fmul_rn(v[e], a[e]);
                }
                float* o = out + (s0 + r) * pitch + i;
                if (i + 4 <= nout) {
                    *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (i + e < nout) o[e] = v[e];
                }
            }
        }
    }
}

template <class C>
__device__ __forceinline__ void qepilogue(const float4* sm, const StageArgs& A, const QJob& J, int tid, const QPrev<C>& P) {
    const bool ydir = J.kind & JK_Y;
    if (J.kind & JK_VEL) {
        if (ydir) qepilogue_k<C, true, false, true>(sm, A, J, tid, P);
        else qepilogue_k<C, true, false, false>(sm, A, J, tid, P);
    } else if (A.last && J.att >= 0) {   // PML multiply of vx / vy at the sixth stage
        if (ydir) qepilogue_k<C, false, true, true>(sm, A, J, tid, P);
        else qepilogue_k<C, false, true, false>(sm, A, J, tid, P);
    } else {
        if (ydir) qepilogue_k<C, false, false, true>(sm, A, J, tid, P);
        else qepilogue_k<C, false, false, false>(sm, A, J, tid, P);
    }
}

// ---------------------------------------------------------------- fused last pass
// A thread of the last inverse pass updates the elements it ends up with: saves
// the trip of the results through shared memory and a barrier, but reaches row
// jobs' fields with 4-byte accesses.  The same for the first pass (each thread
// loading its own elements, mirrored values read twice) was 1.1-1.9 times
// slower at every length and is not here.

// m: live strips of the quad (1..4)
template <bool VEC>
__device__ __forceinline__ float4 qfetch(const float* p, long long ss, int m) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!p) return v;
    if constexpr (VEC) {
        v = qld4(p);
    } else {
        v.x = qld(p);
        if (m > 1) v.y = qld(p + ss);
        if (m > 2) v.z = qld(p + 2 * ss);
        if (m > 3) v.w = qld(p + 3 * ss);
    }
    return v;
}

template <class C, bool VEL, bool ATT, bool VEC>
__device__ __forceinline__ void qlast_pass(float4* sm, const StageArgs& A, const QJob& J, const float2* tw, int tid) {
    constexpr int R = C::R0, Q = C::L / R, ITEMS = C::CS * Q;
    const bool ydir = J.kind & JK_Y;
    const int W = J.W, count = J.count, nout = VEL ? J.n - 1 : J.n + 1;
    const float cdt = J.cdt[A.stage], rho = J.rho, c2 = J.c2, rinv = J.rinv;
    const long long sp = ydir ? J.pitch_out : 1, ss = ydir ? 1 : J.pitch_out;
#pragma unroll 1
    for (int it = tid; it < ITEMS; it += C::NT) {
        const int g = ydir ? it % C::CS : it / Q, n1 = ydir ? it / C::CS : it % Q;
        const int m = count - 4 * g;
        if (m <= 0) continue;
        const float4* base = sm + g * C::SP + n1 + (n1 >> C::SH);
        float2 w[R];
        pass_twiddles<C, R, C::TSM != 0>(tw, n1, w);
        Q2 x[R];
        x[0] = q_of(base[0]);
#pragma unroll
        for (int k = 1; k < R; k++) x[k] = qmulc(q_of(base[qoff<C>(k * Q)]), w[k]);
        QDFT<R, true>::run(x);
        const long long o = J.o_out + (long long)(4 * g) * ss + (n1 - W) * sp;   // output of q: + q * Q * sp
        const float* prev = A.prev + o;
        float* out = A.out + o;
        const float* att = A.att + J.att + n1 - W;
        constexpr int G = R < 4 ? R : 4;
#pragma unroll
        for (int q0 = 0; q0 < R; q0 += G) {
            float4 pv[G];
#pragma unroll
            for (int u = 0; u < G; u++) {
                const int i = n1 + (q0 + u) * Q - W;
                pv[u] = qfetch<VEC>(i >= 0 && i < nout ? prev + (q0 + u) * Q * sp : nullptr, ss, m);
            }
#pragma unroll
            for (int u = 0; u < G; u++) {
                const int q = q0 + u, i = n1 + q * Q - W;
                if (i < 0 || i >= nout) continue;
                float2 a = qrk<VEL>(make_float2(pv[u].x, pv[u].z), x[q].re, cdt, rho, c2, rinv);
                float2 b = qrk<VEL>(make_float2(pv[u].y, pv[u].w), x[q].im, cdt, rho, c2, rinv);
                if constexpr (ATT) {
                    const float t = __ldg(att + q * Q);
                    a = mul2(a, make_float2(t, t));
                    b = mul2(b, make_float2(t, t));
                }
                float* d = out + q * Q * sp;
                if (VEC && m >= 4) {
                    *reinterpret_cast<float4*>(d) = make_float4(a.x, b.x, a.y, b.y);
                } else {
                    d[0] = a.x;
                    if (m > 1) d[ss] = b.x;
                    if (m > 2) d[2 * ss] = a.y;
                    if (m > 3) d[3 * ss] = b.y;
                }
            }
        }
    }
}

template <class C, bool VEC>
__device__ __forceinline__ void qlast(float4* sm, const StageArgs& A, const QJob& J, const float2* tw, int tid) {
    if (J.kind & JK_VEL) qlast_pass<C, true, false, VEC>(sm, A, J, tw, tid);
    else if (A.last && J.att >= 0) qlast_pass<C, false, true, VEC>(sm, A, J, tw, tid);
    else qlast_pass<C, false, false, VEC>(sm, A, J, tw, tid);
}

// ---------------------------------------------------------------- kernels
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// strips, transform, update of one job
template <class C>
__device__ __forceinline__ void quad_body(float4* sm, const StageArgs& A, const QJob& J, const float2* tw, const float4* filt,
                                          int tid) {
    qgather<C>(sm, A, J, tid);
    const int lo = J.W, hi = J.W + ((J.kind & JK_VEL) ? J.n - 1 : J.n + 1);
    qconvolve<C>(sm, tw, filt, tid, 2 * J.W + J.n);
    QPrev<C> P;
    if constexpr (!C::FUSE) {
        if constexpr (C::PRE) qprefetch<C>(P, A, J, tid);
        qinv_pass<C, C::R0, C::L, 0, true>(sm, tw, tid, lo, hi);
        __syncthreads();
    }
    if constexpr (C::FUSE) {
        if ((J.kind & JK_Y) && (J.own.flags & QS_ALIGNED)) qlast<C, true>(sm, A, J, tw, tid);
        else qlast<C, false>(sm, A, J, tw, tid);
    } else {
        qepilogue<C>(sm, A, J, tid, P);
    }
}

// one job: its record (and, TSM, tables) into shared memory before the
// previous launch is waited for -- read where it is used, its second line cost
// a job of a small scene another memory round trip
template <class C>
__device__ __forceinline__ void quad_job(float4* sm, const StageArgs& A, const QJob& job, const float2* tw_global, int tid) {
    const float2* tw = tw_global;
    const float4* filt = reinterpret_cast<const float4*>(A.filt + job.dtab);
    auto copy = [&](float4* d, const float4* s) {
        const unsigned a = (unsigned)__cvta_generic_to_shared(d);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(a), "l"(s) : "memory");
    };
    float4* js = sm + C::JOB / 16;
    if (tid < (int)sizeof(QJob) / 16) copy(js + tid, reinterpret_cast<const float4*>(&job) + tid);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if constexpr (C::TSM) {
        float4* tws = sm + C::DATA / 16;
        float4* fls = tws + C::TWN / 2;
        const float4* t4 = reinterpret_cast<const float4*>(tw_global);
        for (int i = tid; i < C::TWN / 2; i += C::NT) copy(tws + i, t4 + i);
        for (int i = tid; i < C::L / 2; i += C::NT) copy(fls + i, filt + i);
        tw = reinterpret_cast<const float2*>(tws);
        filt = fls;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");   // the record
    __syncthreads();
    const QJob& J = *reinterpret_cast<const QJob*>(js);
    grid_wait();
    grid_release();
    asm volatile("cp.async.wait_group 0;" ::: "memory");   // the tables: visible after the gather's barriers
    quad_body<C>(sm, A, J, tw, filt, tid);
}

template <class C>
__global__ void __launch_bounds__(C::NT, C::MINB) stage_quad(const __grid_constant__ StageArgs A) {
    extern __shared__ __align__(16) float4 smq[];
    const QJob& J = A.qjobs[blockIdx.x];
    if (J.kind & JK_COPY) {
        grid_wait();
        grid_release();
        copy_axis<C::NT>(A, A.doms[J.dom], J.kind & JK_Y, threadIdx.x);
        return;
    }
    quad_job<C>(smq, A, J, A.tw, threadIdx.x);
}

// Serving loop: a record table whose length is read from device memory, one
// CTA per entry of a grid that covers it; CTAs past the length, free entries
// (all zero) and jobs of scenes that have taken all their steps leave at once.
// As a loop over the table with resident CTAs the body spilled 0.2-1.3 KB a
// thread (72-128 registers; called from the loop as a function, as much): 1500
// resident scenes ran at 3.57 Gcell-steps/s, where the complex-strip loop before
// it had made 3.94.  One job per CTA spills at most 144 bytes: 6.76.
template <class C>
__global__ void __launch_bounds__(C::NT, C::MINB) stage_quad_dev(const __grid_constant__ StageArgs A, const int* count) {
    extern __shared__ __align__(16) float4 smq[];
    if ((int)blockIdx.x >= *count) return;
    const QJob& J = A.qjobs[blockIdx.x];
    const bool copy = J.kind & JK_COPY;
    if ((J.L == 0 && !copy) || (A.scene_limit && A.scene_step[J.scene] >= A.scene_limit[J.scene])) return;
    if (copy) {
        copy_axis<C::NT>(A, A.doms[J.dom], J.kind & JK_Y, threadIdx.x);
        return;
    }
    quad_job<C>(smq, A, J, A.tw, threadIdx.x);
}

template <class C>
cudaError_t launch_quad_dev_t(const int* count, int grid, const StageArgs& a, cudaStream_t st) {
    if (grid <= 0) return cudaSuccess;
    stage_quad_dev<C><<<grid, C::NT, C::SMEM, st>>>(a, count);
    return cudaGetLastError();
}

template <class C>
cudaError_t prepare_quad_dev_t() {
    return cudaFuncSetAttribute(stage_quad_dev<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
}

template <class C>
cudaError_t launch_quad_t(int n_jobs, const StageArgs& a, cudaStream_t st) {
    stage_quad<C><<<n_jobs, C::NT, C::SMEM, st>>>(a);
    return cudaGetLastError();
}

template <class C>
cudaError_t prepare_quad_t() {
    return cudaFuncSetAttribute(stage_quad<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
}

template <class C>
size_t quad_smem(int) {
    return (size_t)C::SMEM;
}

template <class C>
StageVariant make_quad_variant(const char* name) {
    StageVariant v;
    v.L = C::L; v.CS = 2 * C::CS; v.NT = C::NT; v.smem = C::SMEM; v.np = C::NP;
    v.r[0] = C::R0; v.r[1] = C::R1; v.r[2] = C::R2; v.r[3] = C::R3;
    v.persistent = false;
    v.pipe = false;
    v.bf16 = false;
    v.ctw = 1;
    v.quad = 1;
    v.launch = &launch_quad_t<C>;
    v.prepare = &prepare_quad_t<C>;
    v.smem_for = &quad_smem<C>;
    v.name = name;
    return v;
}

// with the serving loop's form
template <class C>
StageVariant make_quad_dev_variant(const char* name) {
    StageVariant v = make_quad_variant<C>(name);
    v.launch_dev = &launch_quad_dev_t<C>;
    v.prepare_dev = &prepare_quad_dev_t<C>;
    return v;
}

}  // namespace pstd
