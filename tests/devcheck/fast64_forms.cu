// Device kernels for tests/test_gpu_fast64_forms.py: the forms of the branch-free
// routines that the 1D, 3D and 3D MHD steps use (small numerators divided on the
// spot, one and three axes) beside the plain ones, out[0 .. n) fast and
// out[n .. 2n) plain, and the flags the routines raise.
#include "../../dragon_b200/csrc/step_mhd.cuh"
#include "../../dragon_b200/csrc/update64.cuh"

using namespace dgpu;

namespace {

template <bool MHD>
__device__ Prim<double> get(const double* s, long long i) {
    const double* q = s + i * (MHD ? 8 : 5);
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
__device__ Cons<double> cons_of(const Prim<double>& d) { return Cons<double>{d.rho, d.p, d.vx, d.vy, d.vz, d.Bx, d.By, d.Bz}; }
__device__ ExactOpts opts() { return ExactOpts{6, 1e-12, 0, NewtonLog{nullptr, nullptr, 0, 1}, 0.0}; }

// 14 values: the flux, whether it is physical, the counters
template <bool MHD, int SOLVER, bool LOCAL>
__global__ void k_face(long long n, const double* L, const double* R, double dt_dx, double* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < 2; k++) {
        FaceStats st{};
        Cons<double> F{};
        const Prim<double> l = get<MHD>(L, i), r = get<MHD>(R, i);
        const bool ok = k == 0 ? f64::face_flux_x<MHD, SOLVER, LOCAL>(l, r, dt_dx, opts(), F, &st)
                               : face_flux_x<MHD, SOLVER>(l, r, dt_dx, opts(), F, &st);
        double* o = out + (k * n + i) * 14;
        put(o, F);
        o[8] = ok;
        o[9] = st.pivot_exact + 16 * st.hlld_to_hlle;
        o[10] = st.newton_iters;
        o[11] = st.exact_calls;
        o[12] = st.trrs;
        o[13] = st.cap_hits;
    }
}

// 17 values: both half states, whether they are second order
template <bool LOCAL>
__global__ void k_muscl(long long n, int lim, const double* L, const double* C, const double* R, double dt_dx, double* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < 2; k++) {
        Prim<double> a{}, b{};
        const Prim<double> l = get<false>(L, i), c = get<false>(C, i), r = get<false>(R, i);
        const bool ok = k == 0 ? f64::muscl<false, LOCAL>(lim, l, a, c, b, r, dt_dx, 0.0, 0.0, 0.0)
                               : muscl<false>(lim, l, a, c, b, r, dt_dx, 0.0, 0.0, 0.0);
        double* o = out + (k * n + i) * 17;
        put(o, a);
        put(o + 8, b);
        o[16] = ok;
    }
}

// 18 values: a corrected state (hydro, small numerators on the spot), an updated
// cell of nd axes with its stage (or finite and physical) and speed
template <bool MHD, int ND>
__global__ void k_cell(long long n, const double* W, const double* D, StepArgs sa, double* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Prim<double> w = get<MHD>(W, i);
    const Cons<double> u = cons_of(get<MHD>(D, i)), v = c_mul<MHD>(u, -0.4), x = c_mul<MHD>(u, 0.15);
    const Cons<double> all[3] = {u, v, x};
    const f64::MhdField b{w.Bx + u.Bx, w.By - u.By, w.Bz};
    for (int k = 0; k < 2; k++) {
        double* o = out + (k * n + i) * 18;
        Prim<double> c = w;
        if constexpr (!MHD) {
            if (k == 0) c = f64::corrected<false, true>(w, u);
            else f64::corrected_plain<false>(&c, &u);
        }
        put(o, c);
        if constexpr (MHD && ND == 3) {
            f64::MhdCell r;
            r.w = w;
            if (k == 0) r = f64::mhd_cell<true>(w, sa, b, u, v, x);
            else f64::mhd_cell_plain<true>(&r, all, 3, &b, &sa);
            put(o + 8, r.w);
            o[16] = r.finite + 2 * r.physical;
            o[17] = r.speed;
        } else {
            f64::Updated r;
            r.w = w;
            if (k == 0) {
                if constexpr (ND == 1) r = f64::updated<MHD>(w, sa, f64::Widths{}, u);
                else r = f64::updated<MHD>(w, sa, f64::widths(3, sa.dx, sa.dy, sa.dz), u, v, x);
            } else {
                f64::updated_plain<MHD>(&r, all, ND, &sa);
            }
            put(o + 8, r.w);
            o[16] = r.stage;
            o[17] = r.speed;
        }
    }
}

// flags of a face's solve, a cell's reconstruction and the cell widths
template <bool MHD, int SOLVER>
__global__ void k_flags(long long n, int lim, const double* L, const double* C, const double* R, double dt_dx, double dx,
                        int* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    FaceStats st{};
    Cons<double> F;
    double ps;
    f64::Chk face, cell;
    f64::face_body<MHD, SOLVER>(get<MHD>(C, i), get<MHD>(R, i), dt_dx, opts(), F, &st, ps, face);
    Prim<double> a, b;
    f64::muscl_body<MHD>(lim, get<MHD>(L, i), a, get<MHD>(C, i), b, get<MHD>(R, i), dt_dx, 0.0, 0.0, 0.0, cell);
    out[i] = face.bad + 2 * cell.bad + 4 * f64::widths(3, dx, dx, dx).bad;
}

// quotients of large divisors: a WideRec's (0), a division of its own (1), a
// slope's (2: the constant floor, 3: a sum of squares)
__global__ void k_arith(int op, long long n, const double* a, const double* b, double* out, int* flag) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    f64::Chk ck;
    double x = a[i];
    if (op == 0) f64::quots(f64::widerec(b[i], ck), ck, x);
    if (op == 1) x = f64::div(a[i], b[i], ck);
    if (op == 2) x = f64::slope_quot<false>(a[i], b[i], true, ck);
    if (op == 3) x = f64::slope_quot<true>(a[i], b[i], true, ck);
    out[i] = x;
    out[n + i] = a[i] / b[i];
    flag[i] = ck.bad;
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
int grid_of(long long n) { return (int)((n + 127) / 128); }

template <bool MHD, int S>
int flags(long long n, int lim, const double* L, const double* C, const double* R, double dt_dx, double dx, int* out) {
    const int nf = MHD ? 8 : 5;
    Buf A(L, n * nf), B(C, n * nf), D(R, n * nf);
    int* F = nullptr;
    cudaMalloc(&F, n * sizeof(int));
    k_flags<MHD, S><<<grid_of(n), 128>>>(n, lim, A.p, B.p, D.p, dt_dx, dx, F);
    const int rc = cudaGetLastError() != cudaSuccess || cudaMemcpy(out, F, n * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(F);
    return rc;
}

}  // namespace

extern "C" {

int forms_arith(int op, long long n, const double* a, const double* b, double* out, int* flag) {
    Buf A(a, n), B(b, n), O(nullptr, 2 * n);
    int* F = nullptr;
    cudaMalloc(&F, n * sizeof(int));
    k_arith<<<grid_of(n), 128>>>(op, n, A.p, B.p, O.p, F);
    const int rc = done(O, out, 2 * n) || cudaMemcpy(flag, F, n * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(F);
    return rc;
}

int forms_face(int solver, int local, long long n, const double* L, const double* R, double dt_dx, double* out) {
    Buf A(L, n * 5), B(R, n * 5), O(nullptr, 28 * n);
#define FACE(S)                                                                                  \
    if (solver == S && local) k_face<false, S, true><<<grid_of(n), 128>>>(n, A.p, B.p, dt_dx, O.p); \
    if (solver == S && !local) k_face<false, S, false><<<grid_of(n), 128>>>(n, A.p, B.p, dt_dx, O.p);
    FACE(RS_HLLC) FACE(RS_HLL) FACE(RS_HLLE) FACE(RS_ROE) FACE(RS_EXACT)
#undef FACE
    return done(O, out, 28 * n);
}

int forms_mhd_face(int solver, long long n, const double* L, const double* R, double dt_dx, double* out) {
    Buf A(L, n * 8), B(R, n * 8), O(nullptr, 28 * n);
    if (solver == RS_HLLE) k_face<true, RS_HLLE, false><<<grid_of(n), 128>>>(n, A.p, B.p, dt_dx, O.p);
    else k_face<true, RS_HLLD, false><<<grid_of(n), 128>>>(n, A.p, B.p, dt_dx, O.p);
    return done(O, out, 28 * n);
}

int forms_muscl(int local, int lim, long long n, const double* L, const double* C, const double* R, double dt_dx, double* out) {
    Buf A(L, n * 5), B(C, n * 5), D(R, n * 5), O(nullptr, 34 * n);
    if (local) k_muscl<true><<<grid_of(n), 128>>>(n, lim, A.p, B.p, D.p, dt_dx, O.p);
    else k_muscl<false><<<grid_of(n), 128>>>(n, lim, A.p, B.p, D.p, dt_dx, O.p);
    return done(O, out, 34 * n);
}

int forms_cell(int mhd, int nd, int cfl, long long n, const double* W, const double* dU, double* out) {
    Buf A(W, n * (mhd ? 8 : 5)), B(dU, n * (mhd ? 8 : 5)), O(nullptr, 36 * n);
    StepArgs sa{};
    sa.dx = 1.0 / 96;
    sa.dy = 1.0 / 77;
    sa.dz = 1.0 / 50;
    sa.cfl = cfl;
    sa.ct_energy = 2;
    if (mhd && nd == 1) k_cell<true, 1><<<grid_of(n), 128>>>(n, A.p, B.p, sa, O.p);
    else if (mhd) k_cell<true, 3><<<grid_of(n), 128>>>(n, A.p, B.p, sa, O.p);
    else if (nd == 1) k_cell<false, 1><<<grid_of(n), 128>>>(n, A.p, B.p, sa, O.p);
    else k_cell<false, 3><<<grid_of(n), 128>>>(n, A.p, B.p, sa, O.p);
    return done(O, out, 36 * n);
}

int forms_flags(int mhd, int solver, int lim, long long n, const double* L, const double* C, const double* R, double dt_dx,
                double dx, int* out) {
    if (mhd && solver == RS_HLLE) return flags<true, RS_HLLE>(n, lim, L, C, R, dt_dx, dx, out);
    if (mhd) return flags<true, RS_HLLD>(n, lim, L, C, R, dt_dx, dx, out);
    if (solver == RS_HLL) return flags<false, RS_HLL>(n, lim, L, C, R, dt_dx, dx, out);
    if (solver == RS_HLLE) return flags<false, RS_HLLE>(n, lim, L, C, R, dt_dx, dx, out);
    if (solver == RS_ROE) return flags<false, RS_ROE>(n, lim, L, C, R, dt_dx, dx, out);
    if (solver == RS_EXACT) return flags<false, RS_EXACT>(n, lim, L, C, R, dt_dx, dx, out);
    return flags<false, RS_HLLC>(n, lim, L, C, R, dt_dx, dx, out);
}

}  // extern "C"
