// Device kernels that evaluate the branch-free FP64 routines (csrc/fast64.cuh,
// csrc/solve64.cuh, csrc/update64.cuh) beside the plain ones on given operands
// and states, for tests/test_gpu_fast64.py: out[0 .. n) fast, out[n .. 2n) plain.
#include "../../dragon_b200/csrc/step_mhd.cuh"
#include "../../dragon_b200/csrc/update64.cuh"

using namespace dgpu;

namespace {

__global__ void k_arith(int op, long long n, const double* a, const double* b, double* out, int* flag) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    f64::Chk ck;
    double x = 0, y = 0;
    if (op == 0) { f64::quots(f64::rec(b[i], ck), ck, x = a[i]); y = a[i] / b[i]; }
    if (op == 1) { x = f64::div(a[i], b[i], ck); y = a[i] / b[i]; }
    if (op == 2) { x = f64::root(a[i], ck); y = sqrt(a[i]); }
    if (op == 3) { x = f64::root0(a[i], ck); y = sqrt(a[i]); }
    if (op == 4) { x = f64::by_gm1(a[i]); y = a[i] / kGm1; }
    if (op == 5) { x = f64::by_gamma(a[i]); y = a[i] / kGamma; }
    if (op == 6) { x = f64::by_sq4pi(a[i]); y = a[i] / sq4pi(); }
    out[i] = x;
    out[n + i] = y;
    flag[i] = ck.bad;
}

template <bool MHD>
__device__ Prim<double> get(const double* s, long long i) {
    constexpr int NF = MHD ? 8 : 5;
    const double* q = s + i * NF;
    Prim<double> w{q[0], q[1], q[2], q[3], q[4], 0, 0, 0};
    if (MHD) { w.Bx = q[5]; w.By = q[6]; w.Bz = q[7]; }
    return w;
}
__device__ void put(double* o, const Prim<double>& w) {
    const double v[8] = {w.rho, w.p, w.vx, w.vy, w.vz, w.Bx, w.By, w.Bz};
    for (int f = 0; f < 8; f++) o[f] = v[f];
}
__device__ void put(double* o, const Cons<double>& u) {
    const double v[8] = {u.rho, u.E, u.mx, u.my, u.mz, u.Bx, u.By, u.Bz};
    for (int f = 0; f < 8; f++) o[f] = v[f];
}

// 10 values per face: the flux, whether it is physical, the fallbacks taken
template <bool MHD, int SOLVER>
__global__ void k_face(long long n, const double* L, const double* R, double dt_dx, double* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ExactOpts eo{6, 1e-12, 0, NewtonLog{nullptr, nullptr, 0, 1}, 0.0};
    for (int k = 0; k < 2; k++) {
        FaceStats st{};
        Cons<double> F{};
        const bool ok = k == 0 ? f64::face_flux_x<MHD, SOLVER>(get<MHD>(L, i), get<MHD>(R, i), dt_dx, eo, F, &st)
                               : face_flux_x<MHD, SOLVER>(get<MHD>(L, i), get<MHD>(R, i), dt_dx, eo, F, &st);
        double* o = out + (k * n + i) * 10;
        put(o, F);
        o[8] = ok;
        o[9] = st.pivot_exact + 16 * st.hlld_to_hlle;
    }
}

// 17 values per cell: both half states, whether they are second order
template <bool MHD>
__global__ void k_muscl(long long n, int lim, const double* L, const double* C, const double* R, double dt_dx, double* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double dB = MHD ? 0.01 * (double)(i % 5 - 2) : 0.0;
    for (int k = 0; k < 2; k++) {
        Prim<double> a{}, b{};
        const bool ok = k == 0 ? f64::muscl<MHD>(lim, get<MHD>(L, i), a, get<MHD>(C, i), b, get<MHD>(R, i), dt_dx, dB, -dB, 0.5 * dB)
                               : muscl<MHD>(lim, get<MHD>(L, i), a, get<MHD>(C, i), b, get<MHD>(R, i), dt_dx, dB, -dB, 0.5 * dB);
        double* o = out + (k * n + i) * 17;
        put(o, a);
        put(o + 8, b);
        o[16] = ok;
    }
}

// 18 values per cell: a corrected state, an updated cell with stage (or finite
// and physical) and speed
template <bool MHD>
__global__ void k_cell(long long n, const double* W, const double* D, StepArgs sa, double* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Prim<double> w = get<MHD>(W, i), d = get<MHD>(D, i);
    const Cons<double> u{d.rho, d.p, d.vx, d.vy, d.vz, d.Bx, d.By, d.Bz};
    const Cons<double> v = c_mul<MHD>(u, -0.4);
    const f64::MhdField b{w.Bx + u.Bx, w.By - u.By, w.Bz};
    for (int k = 0; k < 2; k++) {
        double* o = out + (k * n + i) * 18;
        Prim<double> c = w;
        if constexpr (MHD) {
            if (k == 0) c = f64::corrected_mhd<1>(w, u, b.by);
            else f64::corrected_mhd_plain(&c, &u, 1, b.by);
            f64::MhdCell r;
            r.w = w;
            const Cons<double> all[2] = {u, v};
            if (k == 0) r = f64::mhd_cell<true>(w, sa, b, u, v);
            else f64::mhd_cell_plain<true>(&r, all, 2, &b, &sa);
            put(o + 8, r.w);
            o[16] = r.finite + 2 * r.physical;
            o[17] = r.speed;
        } else {
            if (k == 0) c = f64::corrected<false>(w, u);
            else f64::corrected_plain<false>(&c, &u);
            f64::Updated r;
            r.w = w;
            const Cons<double> all[2] = {u, v};
            if (k == 0) r = f64::updated<false>(w, sa, f64::widths(2, sa.dx, sa.dy, 0.0), u, v);
            else f64::updated_plain<false>(&r, all, 2, &sa);
            put(o + 8, r.w);
            o[16] = r.stage;
            o[17] = r.speed;
        }
        put(o, c);
    }
}

struct Buf {
    double* p = nullptr;
    Buf(const double* h, size_t n) {
        if (cudaMalloc(&p, n * 8) == cudaSuccess && h) cudaMemcpy(p, h, n * 8, cudaMemcpyHostToDevice);
    }
    ~Buf() { cudaFree(p); }
};
int done(const Buf& o, double* out, size_t n) {
    if (cudaGetLastError() != cudaSuccess) return 1;
    return cudaMemcpy(out, o.p, n * 8, cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : 1;
}

}  // namespace

extern "C" {

int f64_arith(int op, long long n, const double* a, const double* b, double* out, int* flag) {
    Buf A(a, n), B(b, n), O(nullptr, 2 * n);
    int* F = nullptr;
    cudaMalloc(&F, n * sizeof(int));
    k_arith<<<(int)((n + 127) / 128), 128>>>(op, n, A.p, B.p, O.p, F);
    const int rc = done(O, out, 2 * n);
    cudaMemcpy(flag, F, n * sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(F);
    return rc;
}

int f64_face(int mhd, int solver, long long n, const double* L, const double* R, double dt_dx, double* out) {
    const int nf = mhd ? 8 : 5, g = (int)((n + 127) / 128);
    Buf A(L, n * nf), B(R, n * nf), O(nullptr, 20 * n);
    if (mhd) {
        if (solver == RS_HLLE) k_face<true, RS_HLLE><<<g, 128>>>(n, A.p, B.p, dt_dx, O.p);
        else k_face<true, RS_HLLD><<<g, 128>>>(n, A.p, B.p, dt_dx, O.p);
    } else if (solver == RS_HLL) k_face<false, RS_HLL><<<g, 128>>>(n, A.p, B.p, dt_dx, O.p);
    else if (solver == RS_HLLE) k_face<false, RS_HLLE><<<g, 128>>>(n, A.p, B.p, dt_dx, O.p);
    else if (solver == RS_ROE) k_face<false, RS_ROE><<<g, 128>>>(n, A.p, B.p, dt_dx, O.p);
    else if (solver == RS_EXACT) k_face<false, RS_EXACT><<<g, 128>>>(n, A.p, B.p, dt_dx, O.p);
    else k_face<false, RS_HLLC><<<g, 128>>>(n, A.p, B.p, dt_dx, O.p);
    return done(O, out, 20 * n);
}

int f64_muscl(int mhd, int lim, long long n, const double* L, const double* C, const double* R, double dt_dx, double* out) {
    const int nf = mhd ? 8 : 5, g = (int)((n + 127) / 128);
    Buf A(L, n * nf), B(C, n * nf), D(R, n * nf), O(nullptr, 34 * n);
    if (mhd) k_muscl<true><<<g, 128>>>(n, lim, A.p, B.p, D.p, dt_dx, O.p);
    else k_muscl<false><<<g, 128>>>(n, lim, A.p, B.p, D.p, dt_dx, O.p);
    return done(O, out, 34 * n);
}

int f64_cell(int mhd, int cfl, long long n, const double* W, const double* dU, double* out) {
    const int nf = mhd ? 8 : 5, g = (int)((n + 127) / 128);
    Buf A(W, n * nf), B(dU, n * nf), O(nullptr, 36 * n);
    StepArgs sa{};
    sa.dx = 1.0 / 96;
    sa.dy = 1.0 / 77;
    sa.cfl = cfl;
    sa.ct_energy = 2;
    if (mhd) k_cell<true><<<g, 128>>>(n, A.p, B.p, sa, O.p);
    else k_cell<false><<<g, 128>>>(n, A.p, B.p, sa, O.p);
    return done(O, out, 36 * n);
}

}  // extern "C"
