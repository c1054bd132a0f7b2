// beam.cuh — the beam of neighbouring rays around a pixel ray (geodesic
// deviation), and the magnification it gives.
//
// The reference's BeamIntegratorD (INBI001A.h:178-363) carries a Jacobian J of
// Boyer-Lindquist coordinates along a leapfrog ray with a Jacobi equation in
// the Riemann tensor, and reports 1 / |det| of J's (theta, phi) block. Here the
// same idea is restated on the engine's Hamiltonian form: the ray y = (x^mu,
// p_mu) carries two tangent vectors V_u = dy/du, V_v = dy/dv (u, v: the pixel
// coordinates of its start), which obey the linearised equation
//   dV/dlambda = (df/dy) V,   f = (dx/dlambda, dp/dlambda)
// (the geodesic deviation equation in first-order form). df/dy V is the
// Jacobian-vector product of the closed-form right-hand side (dual numbers with one
// tangent); the ray and its tangents advance together by Dormand-Prince 5(4) steps
// controlled on the ray. When the ray
// escapes, its unit direction n and the tangents' dn/du, dn/dv give the solid
// angle the pixel maps to on the sky, |dn/du x dn/dv| du dv; the pixel's own
// solid angle is |dd/du x dd/dv| du dv with d the start direction in the
// camera frame; the magnification is their ratio (1 in flat space) and the
// parity is the sign of the map (negative for a mirror-reversed image).
//
// This file is a fragment of engine.cu's kernel section (it uses the engine's
// find_frame and globaltimer) and is included there.
#pragma once

// start direction of pixel position (u, v) (pixel units, the centre of pixel
// (px, py) is (px + 0.5, py + 0.5)) in FP64 without the camera's FP32
// roundings, so that its derivatives are smooth
__device__ __forceinline__ void camera_dir_exact(const FrameDev& F, double u, double v, double dir[4]) {
    dir[0] = 0.0;
    if (F.projection == SIRIUS_CAMERA_EQUIRECTANGULAR) {
        const double psi = (2.0 * u / F.width - 1.0) * kPi;
        const double chi = (1.0 - 2.0 * v / F.height) * (0.5 * kPi);
        double sc, cc, sps, cps;
        sincos(chi, &sc, &cc);
        sincos(psi, &sps, &cps);
        dir[1] = -cc * cps;
        dir[2] = -sc;
        dir[3] = cc * sps;
        return;
    }
    const double pxn = (2.0 * u / F.width - 1.0) * double(F.aspect), pyn = 1.0 - 2.0 * v / F.height;
    const double T = F.tan_half_fov;
    const double dx = pxn * T, dy = pyn * T, dz = -1.0;
    const double cR = F.cR, sR = F.sR, cP = F.cP, sP = F.sP, cY = F.cY, sY = F.sY;
    const double rx = dx * cR - dy * sR, ry = dx * sR + dy * cR;
    const double ry2 = ry * cP - dz * sP, rz = ry * sP + dz * cP;
    const double rx2 = rx * cY + rz * sY, rz2 = -rx * sY + rz * cY;
    const double len = sqrt(rx2 * rx2 + ry2 * ry2 + rz2 * rz2);
    dir[1] = rz2 / len;
    dir[2] = -ry2 / len;
    dir[3] = rx2 / len;
}

__device__ __forceinline__ void beam_start(const FrameDev& F, double u, double v, double y[8]) {
    double dir[4];
    camera_dir_exact(F, u, v, dir);
    init_state(F, dir, y, y + 4);
}

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double c[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

struct BeamParams {
    const FrameDev* frames;
    int n_frames;
    long long total;
    CfgDev c;
    sirius_beam_result* out;
    unsigned long long watchdog_ns;
    int* status;
};

// f of a state and of its tangent: y = (x, p) and V in, k and dk out (8 components)
template <bool RING>
__device__ __forceinline__ void beam_rhs(const MetricDev& m, const double y[8], const double V[8], double f[8],
                                         double fV[8]) {
    D1<double> x[4], p[4], k[4], g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] = D1<double>(y[i], V[i]);
        p[i] = D1<double>(y[4 + i], V[4 + i]);
    }
    ks_rhs_closed<RING>(m, x, p, k, g);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[i] = k[i].v; fV[i] = k[i].d;
        f[4 + i] = g[i].v; fV[4 + i] = g[i].d;
    }
}

// Two neighbouring lanes trace a beam: both carry the ray (the same operations on
// the same values, so the same bits and the same steps), the even lane the tangent
// along u and the odd lane the one along v; they meet at the end, for the solid
// angles. A small map is bound by one beam's dependent chain and a large one by
// FP64 issue: a lane's stage is one right-hand side with one tangent (about 250
// operations, three of them roots or reciprocals), where one thread with both
// tangents as central differences took five right-hand sides a stage and kept its
// seven stage derivatives of 24 components in local memory (120 x 68 beams to
// R = 1000 M: 22.3 -> 3.1 ms; magnifications against the same steps with exact
// tangents in 64 bits: both within the rounding of a float). The sums of the stages
// are those of dp45_attempt_f64. RING: the beams of the frames of class kClassRing, without it the others'.
template <bool RING>
__global__ void __launch_bounds__(64) beam_kernel(const __grid_constant__ BeamParams B) {
    const long long thread = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long idx = thread >> 1;
    const int dir = int(thread & 1);  // 0: the tangent along u, 1: along v
    if (idx >= B.total) return;
    const unsigned pair = 3u << (threadIdx.x & 30);
    const int fi = B.n_frames > 1 ? find_frame(B.frames, B.n_frames, idx) : 0;
    const FrameDev& F = B.frames[fi];
    if ((F.cls == kClassRing) != RING) return;
    const CfgDev& c = B.c;
    const MetricDev m = F.m;
    const long long pix = idx - F.ray_offset;
    const double u0 = double(pix % F.width) + 0.5, v0 = double(F.row0 + pix / F.width) + 0.5;
    // start: the ray, its tangent along this lane's direction, and the derivative of
    // the pixel direction
    double y[8], V[8], dd[3];
    beam_start(F, u0, v0, y);
    {
        const double hpx = 1e-3;
        double yp[8], ym[8], dp[4], dm[4];
        const double du = dir == 0 ? hpx : 0.0, dv = dir == 0 ? 0.0 : hpx;
        beam_start(F, u0 + du, v0 + dv, yp);
        beam_start(F, u0 - du, v0 - dv, ym);
        for (int i = 0; i < 8; ++i) V[i] = (yp[i] - ym[i]) / (2.0 * hpx);
        camera_dir_exact(F, u0 + du, v0 + dv, dp);
        camera_dir_exact(F, u0 - du, v0 - dv, dm);
        for (int i = 0; i < 3; ++i) dd[i] = (dp[1 + i] - dm[1 + i]) / (2.0 * hpx);
    }

    const DPTable& D = kDPd;
    double h = c.h0;
    double k1[8], j1[8];  // f of the ray and of its tangent at the current state
    beam_rhs<RING>(m, y, V, k1, j1);
    int outcome = SIRIUS_MAX_STEPS, steps = 0;
    const unsigned long long t0 = globaltimer();
    double r_prev = ks_radius(m, y);
    for (int it = 0; it < 4 * c.max_steps && steps < c.max_steps; ++it) {
        if ((it & 63) == 0) {
            // one answer for the pair: lanes that left the loop apart could not meet again
            const bool late = globaltimer() - t0 > B.watchdog_ns;
            if (__any_sync(pair, late)) {
                atomicOr(B.status, 1);
                break;
            }
        }
        constexpr int C[7] = {0, 1, 2, 3, 5, 6, 7};  // p_0 and its tangent are constant
        double k2[8], k3[8], k4[8], j2[8], j3[8], j4[8], yn[8], Vn[8], sy[7], sV[7];
        double a6[7], b[7], A6[7], Bv[7], e[4];
        yn[4] = y[4];
        Vn[4] = V[4];
        auto stage = [&](double kk[8], double jj[8]) {
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                yn[C[q]] = y[C[q]] + h * sy[q];
                Vn[C[q]] = V[C[q]] + h * sV[q];
            }
            beam_rhs<RING>(m, yn, Vn, kk, jj);
        };
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            sy[q] = D.A[0][0] * k1[C[q]];
            sV[q] = D.A[0][0] * j1[C[q]];
        }
        stage(k2, j2);
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            sy[q] = D.A[0][1] * k1[C[q]] + D.A[1][0] * k2[C[q]];
            sV[q] = D.A[0][1] * j1[C[q]] + D.A[1][0] * j2[C[q]];
        }
        stage(k3, j3);
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            sy[q] = D.A[0][2] * k1[C[q]] + D.A[1][1] * k2[C[q]] + D.A[2][0] * k3[C[q]];
            sV[q] = D.A[0][2] * j1[C[q]] + D.A[1][1] * j2[C[q]] + D.A[2][0] * j3[C[q]];
        }
        stage(k4, j4);
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const int i = C[q];
            sy[q] = D.A[0][3] * k1[i] + D.A[1][2] * k2[i] + D.A[2][1] * k3[i] + D.A[3][0] * k4[i];
            a6[q] = D.A[0][4] * k1[i] + D.A[1][3] * k2[i] + D.A[2][2] * k3[i] + D.A[3][1] * k4[i];
            b[q] = D.A[0][5] * k1[i] + D.A[2][3] * k3[i] + D.A[3][2] * k4[i];
            if (i < 4) e[i] = D.E[0] * k1[i] + D.E[2] * k3[i] + D.E[3] * k4[i];
            sV[q] = D.A[0][3] * j1[i] + D.A[1][2] * j2[i] + D.A[2][1] * j3[i] + D.A[3][0] * j4[i];
            A6[q] = D.A[0][4] * j1[i] + D.A[1][3] * j2[i] + D.A[2][2] * j3[i] + D.A[3][1] * j4[i];
            Bv[q] = D.A[0][5] * j1[i] + D.A[2][3] * j3[i] + D.A[3][2] * j4[i];
        }
        stage(k2, j2);  // k_5
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const int i = C[q];
            sy[q] = a6[q] + D.A[4][0] * k2[i];
            b[q] += D.A[4][1] * k2[i];
            if (i < 4) e[i] += D.E[4] * k2[i];
            sV[q] = A6[q] + D.A[4][0] * j2[i];
            Bv[q] += D.A[4][1] * j2[i];
        }
        stage(k3, j3);  // k_6
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const int i = C[q];
            sy[q] = b[q] + D.A[5][0] * k3[i];
            if (i < 4) e[i] += D.E[5] * k3[i];
            sV[q] = Bv[q] + D.A[5][0] * j3[i];
        }
        stage(k2, j2);  // k_7 at the fifth-order solution (yn, Vn)
        // error on the position components
        double err2 = 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double sc = c.atol + c.rtol * fmax(fabs(y[i]), fabs(yn[i]));
            const double q = h * (e[i] + D.E[6] * k2[i]) * rcp_(sc);
            err2 += q * q;
        }
        const double err = sqrt(err2 / 4.0);
        if (!(err == err)) {
            outcome = SIRIUS_NUMERICAL_FAILURE;
            break;
        }
        if (err > 1.0 && h > c.hmin) {
            h = fmax(c.hmin, optimal_step(h, err, c));
            continue;
        }
        const double z0 = y[3];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            y[i] = yn[i]; V[i] = Vn[i];
            k1[i] = k2[i]; j1[i] = j2[i];
        }
        ++steps;
        h = optimal_step(h, err, c);
        const double r = ks_radius(m, y);
        if (F.has_horizon && r < F.r_hor) {
            outcome = SIRIUS_HORIZON;
            break;
        }
        if (c.enable_disk && z0 * y[3] < 0.0) {
            const double rc = 0.5 * (r + r_prev);
            if (rc >= F.disk_in && rc <= F.disk_out) {
                outcome = SIRIUS_DISK_HIT;
                break;
            }
        }
        r_prev = r;
        const double R2 = y[1] * y[1] + y[2] * y[2] + y[3] * y[3];
        const double out = y[1] * k1[1] + y[2] * k1[2] + y[3] * k1[3];
        if (R2 > c.escape_r * c.escape_r && out > 0.0) {
            outcome = SIRIUS_ESCAPED;
            break;
        }
    }
    __syncwarp(pair);
    // n = k / |k| (spatial, contravariant), dn = (dk - n (n . dk)) / |k| along this lane's tangent
    const double kn = sqrt(k1[1] * k1[1] + k1[2] * k1[2] + k1[3] * k1[3]);
    const double n[3] = {k1[1] / kn, k1[2] / kn, k1[3] / kn};
    const double nd = n[0] * j1[1] + n[1] * j1[2] + n[2] * j1[3];
    double dn[3], ddo[3], dno[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        dn[i] = (j1[1 + i] - n[i] * nd) / kn;
        ddo[i] = __shfl_xor_sync(pair, dd[i], 1);
        dno[i] = __shfl_xor_sync(pair, dn[i], 1);
    }
    if (dir != 0) return;
    sirius_beam_result res{};
    res.outcome = outcome;
    res.steps = steps;
    if (outcome == SIRIUS_ESCAPED) {
        double d0[4], cimg[3], cs[3];
        camera_dir_exact(F, u0, v0, d0);
        cross3(dd, ddo, cimg);
        const double omega_img = sqrt(cimg[0] * cimg[0] + cimg[1] * cimg[1] + cimg[2] * cimg[2]);
        const double sgn_img = cimg[0] * d0[1] + cimg[1] * d0[2] + cimg[2] * d0[3] >= 0.0 ? 1.0 : -1.0;
        cross3(dn, dno, cs);
        const double omega_src = sqrt(cs[0] * cs[0] + cs[1] * cs[1] + cs[2] * cs[2]);
        const double sgn_src = cs[0] * n[0] + cs[1] * n[1] + cs[2] * n[2] >= 0.0 ? 1.0 : -1.0;
        res.magnification = omega_src > 0.0 ? float(omega_img / omega_src) : 1e30f;
        res.parity = float(sgn_img * sgn_src);
        for (int i = 0; i < 3; ++i) res.final_dir[i] = float(n[i]);
    }
    B.out[idx] = res;
}
