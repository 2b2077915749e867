// fft_regs.cuh -- complex 32-bit Fourier transforms of 8, 16 and 32 points held in a
// thread's registers (Cooley-Tukey, J. W. Cooley and J. W. Tukey, Math. Comp. 19, 1965).
// Every index is known at compile time, so outputs that are not used cost nothing.
#pragma once
#include <cuda_runtime.h>

namespace ion {

struct C2 { float x, y; };

// cos(2 pi j / 32), j = 0..8 (rounded from the exact values)
__host__ __device__ constexpr double cos32(int j) {
    constexpr double t[9] = {1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
                             0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173,
                             0.19509032201612826785, 0.0};
    const int k = j & 31;
    return k <= 8 ? t[k] : k <= 16 ? -t[16 - k] : k <= 24 ? -t[k - 16] : t[32 - k];
}
__host__ __device__ constexpr double sin32(int j) { return cos32(j + 24); }  // cos(a - pi/2)

// v * exp(SIGN 2 pi i j / 32)
template <int SIGN>
__device__ __forceinline__ C2 twist(const C2 v, const int j) {
    const int k = j & 31;
    if (k == 0) return v;
    if (k == 8) return SIGN > 0 ? C2{-v.y, v.x} : C2{v.y, -v.x};
    if (k == 16) return {-v.x, -v.y};
    if (k == 24) return SIGN > 0 ? C2{v.y, -v.x} : C2{-v.y, v.x};
    const float c = (float)cos32(k), s = (float)(SIGN * sin32(k));
    return {fmaf(v.x, c, -(v.y * s)), fmaf(v.x, s, v.y * c)};
}
// a + v exp(SIGN 2 pi i j / 32)
template <int SIGN>
__device__ __forceinline__ C2 add_twist(const C2 a, const C2 v, const int j) {
    const int k = j & 31;
    if (k % 8 == 0) {
        const C2 w = twist<SIGN>(v, j);
        return {a.x + w.x, a.y + w.y};
    }
    const float c = (float)cos32(k), s = (float)(SIGN * sin32(k));
    return {fmaf(v.x, c, fmaf(-v.y, s, a.x)), fmaf(v.x, s, fmaf(v.y, c, a.y))};
}

template <int SIGN>
__device__ __forceinline__ void dft4(C2& a, C2& b, C2& c, C2& d) {
    const C2 s0 = {a.x + c.x, a.y + c.y}, d0 = {a.x - c.x, a.y - c.y};
    const C2 s1 = {b.x + d.x, b.y + d.y}, d1 = {b.x - d.x, b.y - d.y};
    const C2 r = SIGN > 0 ? C2{-d1.y, d1.x} : C2{d1.y, -d1.x};  // +-i d1
    a = {s0.x + s1.x, s0.y + s1.y};
    b = {d0.x + r.x, d0.y + r.y};
    c = {s0.x - s1.x, s0.y - s1.y};
    d = {d0.x - r.x, d0.y - r.y};
}

// dft4 with b and d times sg = +-1 (exact; a fused step costs what the addition does):
// with -1 the outputs come half a turn on, c d a b
template <int SIGN>
__device__ __forceinline__ void dft4_turn(C2& a, C2& b, C2& c, C2& d, const float sg) {
    const C2 s0 = {a.x + c.x, a.y + c.y}, d0 = {a.x - c.x, a.y - c.y};
    const C2 s1 = {b.x + d.x, b.y + d.y}, d1 = {b.x - d.x, b.y - d.y};
    const C2 r = SIGN > 0 ? C2{-d1.y, d1.x} : C2{d1.y, -d1.x};  // +-i d1
    a = {fmaf(s1.x, sg, s0.x), fmaf(s1.y, sg, s0.y)};
    b = {fmaf(r.x, sg, d0.x), fmaf(r.y, sg, d0.y)};
    c = {fmaf(-s1.x, sg, s0.x), fmaf(-s1.y, sg, s0.y)};
    d = {fmaf(-r.x, sg, d0.x), fmaf(-r.y, sg, d0.y)};
}

// v[n] <- sum_k v[k] exp(SIGN 2 pi i n k / N).  TURN (N = 8, 16): with sg = -1 the outputs are
// stored N/2 on, v[n] = output (n + N/2) mod N
template <int N, int SIGN, bool TURN = false>
__device__ __forceinline__ void fft_regs(C2 (&v)[N], const float sg = 1.0f) {
    static_assert(N == 8 || N == 16 || (N == 32 && !TURN), "transform sizes in use");
    if constexpr (N == 8) {  // k = 2a + b, n = c + 4d
        C2 t[2][4];
#pragma unroll
        for (int b = 0; b < 2; b++) {
#pragma unroll
            for (int a = 0; a < 4; a++) t[b][a] = v[2 * a + b];
            dft4<SIGN>(t[b][0], t[b][1], t[b][2], t[b][3]);
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const C2 w = twist<SIGN>(t[1][c], 4 * c);
            if constexpr (TURN) {
                v[c] = {fmaf(w.x, sg, t[0][c].x), fmaf(w.y, sg, t[0][c].y)};
                v[c + 4] = {fmaf(-w.x, sg, t[0][c].x), fmaf(-w.y, sg, t[0][c].y)};
            } else {
                v[c] = {t[0][c].x + w.x, t[0][c].y + w.y};
                v[c + 4] = {t[0][c].x - w.x, t[0][c].y - w.y};
            }
        }
    } else if constexpr (N == 16) {  // k = 4a + b, n = c + 4d
        C2 t[4][4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
#pragma unroll
            for (int a = 0; a < 4; a++) t[b][a] = v[4 * a + b];
            dft4<SIGN>(t[b][0], t[b][1], t[b][2], t[b][3]);
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            C2 q[4];
#pragma unroll
            for (int b = 0; b < 4; b++) q[b] = twist<SIGN>(t[b][c], 2 * b * c);
            if constexpr (TURN) dft4_turn<SIGN>(q[0], q[1], q[2], q[3], sg);
            else dft4<SIGN>(q[0], q[1], q[2], q[3]);
#pragma unroll
            for (int d = 0; d < 4; d++) v[c + 4 * d] = q[d];
        }
    } else {  // even and odd k
        C2 e[16], o[16];
#pragma unroll
        for (int k = 0; k < 16; k++) { e[k] = v[2 * k]; o[k] = v[2 * k + 1]; }
        fft_regs<16, SIGN>(e);
        fft_regs<16, SIGN>(o);
#pragma unroll
        for (int n = 0; n < 16; n++) {
            v[n] = add_twist<SIGN>(e[n], o[n], n);
            v[n + 16] = add_twist<SIGN>(e[n], o[n], n + 16);
        }
    }
}

}  // namespace ion
