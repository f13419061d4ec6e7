// adjoint.cuh — reverse-mode derivative (vector-Jacobian product) of one
// force evaluation of the particle system: density with the three unrolled
// smoothing-length passes and the gradient pass, EOS and Balsara switch, tree
// gravity (particles and monopole nodes), hydro, and the alpha source.
//
// Given the adjoints (dL/d output) of the evaluation's outputs — total
// acceleration, du/dt, d(alpha)/dt, the final smoothing length h (the next
// evaluation's first guess), and optionally the potential and the density —
// it accumulates the adjoints of its inputs: predicted position and velocity,
// internal energy, alpha, and the first guess of h.  Every formula is the
// derivative of the forward code path (pair_kernels.cuh, system.cu glue):
//
//   density   rho_k = c0 h_k^-3 sum_j m_j W0(r/h_k), h_{k+1} = eta ksrh (m/rho_k)^(1/3),
//             k = 0,1,2; rho = rho_2, h = h_3 (hdr_density.hpp:264-302)
//   gradient  Sg = sum_j m_j (3 c0 W0 + c1 q W1), grdh = -h^-4 Sg,
//             Omega = 1/(1 + h grdh/(3 rho)), D = sum_{j!=i} (u.d) m_j W1/r,
//             R = sum_{j!=i} (u x d) m_j W1/r, divv = -c1 h^-4 D Omega/rho,
//             rotv = c1 h^-4 |R| Omega/rho (hdr_density.hpp:304-349)
//   EOS       P = rho u/1.5, c = sqrt(10 u/9), bswt = |divv|/(|divv|+|rotv|+1e-4 c ksrh/h)
//   gravity   acc = -1/2 sum m (Ri^3+Rj^3) d, pot = -1/2 sum m (Ri+Rj), etas = sum m Ri^3,
//             R = (r^2 + eps^2)^-1/2; nodes carry (centre of mass, mass-weighted eps^2)
//             (hdr_gravity.hpp:286-342); a_g2 = G acc, eta = eps^2 Omega/(3 rho) etas
//   hydro     hdr_hydro.hpp:349-398 with alpha_u = 0 (its channel is then inert)
//   alpha     adot = -(alpha - amin) tau^-1 + max(-divv (amax - alpha), 0),
//             tau^-1 = ksrh c/(4 h) (hdr_hgas.hpp:750-762)
//
// Non-smooth points: away from the kink min(w, 0) and max(., 0) take their
// active branch and |x| its sign; exactly at it (which uniform velocities
// reach: w = 0, div v = 0) the mean of both one-sided derivatives, 1/2 and 0,
// the value central differences converge to.  The lists, tree and time step are those of the
// forward evaluation and are held fixed (the density and hydro kernels are
// C2 at their support, so list membership does not change their values).
// Arithmetic is FP64 throughout.
//
// The hydro and density-gradient pairs are gathered: a pair inside either
// support is in the rows of both particles (the forward evaluation's hydro
// rows, ~60 entries), and each particle adds what both ends' equations pass to
// it, without atomics; eight lanes per particle.  The three h passes have
// supports of their own, one-sided: their j-side goes out by atomics from rows
// marked for them.  The gravity lists are one-sided too: a warp holds 32
// i-particles against tiles of 32 list entries, lane l starting at entry l, so
// that each entry's adjoints are added up in shared memory and sent out once
// per tile.
#pragma once

#include "rows.cuh"
#include "sph_device.cuh"

namespace sphadj {

using sphk::CEFF0;
using sphk::CEFF1;
using sphk::KSRH;
using sphk::FULL;

struct AdjState {
    int n;
    const dbl4 *pos;        // predicted position, mass
    const dbl4 *vel;        // predicted velocity
    const double *uene, *alph, *h0, *h, *dens, *grdh, *divv, *rotv, *pres, *vsnd, *bswt, *eps2, *eta, *etas;
    const dbl4 *mom;        // tree nodes: centre of mass, mass
    const double *neps2;    // tree nodes: mass-weighted eps^2
    const int *parent;      // tree nodes: parent (root: -1); leaf of particle p: n - 1 + p
    const int *d_off, *d_idx, *h_off, *h_idx, *g_off, *g_idx;   // density, hydro, gravity lists per walk
    const int *h_rows, *d_rows;       // rows of the hydro pairs and of the h passes
    const int2 *h_info, *d_info;      // their entries (> ROW_CAP: the walk's list instead) and walks
    const long long *id;
    double slack;                     // radius of the rows of the h passes over the first guess
    double G, amax, amin, eta_ksrh;
};

// Seeds (adjoints of the outputs), in sorted particle order.
struct AdjSeed {
    const double *acc;      // 3 per particle
    const double *udot, *adot, *h, *pot, *dens;   // pot / dens may be null
};

// Accumulators, in sorted particle order (zeroed before the first stage).
struct AdjAcc {
    double *x, *v;          // 3 per particle
    double *u, *alph, *h0;  // outputs: internal energy, alpha, first guess of h
    double *h, *rho, *omega, *divv, *rotv, *c, *b, *pc, *eta, *e2, *hinv, *etas, *bswt;
    double *node;           // 4 per tree node: centre of mass (3), eps^2
    double *coef;           // 5 per particle: adjoints of its gradient-pass sums (D, R, Sg)
};

// Wendland C2: W0 = u^4 (1+4q), W1 = -5 q u^3 (the reference's u^4 - u^3 (1+4q)),
// and their q-derivatives, zero for q >= 1.
__device__ __forceinline__ void wendland(double q, double &w0, double &w0p, double &w1, double &w1p) {
    if (q < 1.0) {
        const double u = 1.0 - q, u2 = u * u, u3 = u2 * u;
        w0 = u2 * u2 * (1.0 + 4.0 * q);
        w0p = -20.0 * q * u3;
        w1 = -5.0 * q * u3;
        w1p = -5.0 * u2 * (1.0 - 4.0 * q);
    } else {
        w0 = w0p = w1 = w1p = 0.0;
    }
}

// Eight lanes per particle: its candidate pairs are its row, or its walk's
// whole list where it has none.
constexpr int LANES = 8;
__device__ __forceinline__ double lsum(double v) { return sphk::seg_sum(v, LANES); }
struct Candidates {
    const int *p;
    int n;
    __device__ __forceinline__ Candidates(const int *rows, const int2 *info, const int *off, const int *idx, int i) {
        const int2 f = info[i];
        if (f.x <= sphk::ROW_CAP) {
            p = rows + (size_t)i * sphk::ROW_CAP;
            n = f.x;
        } else {
            p = idx + off[f.y];
            n = off[f.y + 1] - off[f.y];
        }
    }
};
// particle of this lane's segment (-1 beyond n), grid-stride over particles
#define ADJ_PARTICLES(i, n)                                                                                      \
    for (int k0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (32 / LANES), i = k0 + (threadIdx.x & 31) / LANES; \
         k0 < (n); k0 += ((gridDim.x * blockDim.x) >> 5) * (32 / LANES), i = k0 + (threadIdx.x & 31) / LANES)

// -------------------------------------------------------------- stage A
// alpha source and the seeds that need no pair loop
__global__ void adj_alpha(AdjState s, AdjSeed sd, AdjAcc a) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        a.h[i] += sd.h ? sd.h[i] : 0.0;
        if (sd.dens) a.rho[i] += sd.dens[i];
        const double ad = sd.adot[i];
        const double h = s.h[i], c = s.vsnd[i], al = s.alph[i], dv = s.divv[i];
        const double tauinv = 0.25 * KSRH * c / h;
        const double src = -dv * (s.amax - al);
        const double on = src > 0.0 ? 1.0 : (src == 0.0 ? 0.5 : 0.0);
        a.alph[i] += ad * (-tauinv + on * dv);
        a.divv[i] += ad * on * (-(s.amax - al));
        a.c[i] += ad * (-(al - s.amin)) * 0.25 * KSRH / h;
        a.h[i] += ad * (al - s.amin) * tauinv / h;
    }
}

// -------------------------------------------------------------- stage B
// hydro pairs: seeds acch (= acc / 2 per pair sum), accg (= G acc / 2), udot / 2
// of both ends of each pair, gathered over the forward's hydro rows (a pair is
// in the rows of both ends), eight lanes per particle: no atomics, and 1/15 of
// the listed entries (100k, this stage and the density's: 145 -> 44 ms).  FP64
// pipe bound.
__global__ void __launch_bounds__(128) adj_hydro(AdjState s, AdjSeed sd, AdjAcc a) {
    const int sub = threadIdx.x & (LANES - 1);
    ADJ_PARTICLES(ip, s.n) {
        const bool act = ip < s.n;
        const int i = act ? ip : s.n - 1;
        const dbl4 xi = s.pos[i], vi = s.vel[i];
        const double hi_len = s.h[i], hi = 1.0 / hi_len, hi3 = hi * hi * hi, hi4 = hi3 * hi;
        const double rho_i = s.dens[i], c_i = s.vsnd[i], b_i = 0.5 * s.bswt[i], al_i = s.alph[i];
        const double pc_i = s.pres[i] * s.grdh[i] / (rho_i * rho_i), et_i = s.eta[i];
        const double Ahx = 0.5 * sd.acc[3 * i], Ahy = 0.5 * sd.acc[3 * i + 1], Ahz = 0.5 * sd.acc[3 * i + 2];
        const double Us_i = 0.5 * sd.udot[i];
        const long long idi = s.id[i];
        double xb0 = 0, xb1 = 0, xb2 = 0, vb0 = 0, vb1 = 0, vb2 = 0;
        double hinvb = 0, cb = 0, rb = 0, bb = 0, ab = 0, pcb = 0, etb = 0;
        const Candidates cand(s.h_rows, s.h_info, s.h_off, s.h_idx, i);
        for (int e = sub; e < (act ? cand.n : 0); e += LANES) {
            const int j = cand.p[e];
            const dbl4 xj = s.pos[j];
            const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double hj_len = s.h[j];
            const double hm = fmax(hi_len, hj_len);
            if (!(r2 < hm * hm) || s.id[j] == idi) continue;
            const dbl4 vj = s.vel[j];
            const double mi = xi.w, mj = xj.w;
            const double hj = 1.0 / hj_len, hj4 = hj * hj * hj * hj;
            const double rho_j = s.dens[j], b_j = 0.5 * s.bswt[j], al_j = s.alph[j];
            const double pc_j = s.pres[j] * s.grdh[j] / (rho_j * rho_j), et_j = s.eta[j];
            const double Bhx = 0.5 * sd.acc[3 * j], Bhy = 0.5 * sd.acc[3 * j + 1], Bhz = 0.5 * sd.acc[3 * j + 2];
            const double Us_j = 0.5 * sd.udot[j];
            const double ux = vi.x - vj.x, uy = vi.y - vj.y, uz = vi.z - vj.z;
            const double ri = sphk::rsqrt_r(r2), r = r2 * ri;
            double w0, w0p, w1i, w1pi, w1j, w1pj;
            wendland(r * hi, w0, w0p, w1i, w1pi);
            wendland(r * hj, w0, w0p, w1j, w1pj);
            const double dWi = CEFF1 * hi4 * w1i, dWj = CEFF1 * hj4 * w1j;
            // the equations of i and of j: separation d and -d, velocity u and
            // -u, the same w, viscosity and pressure factor
            const double kaI = (dWi + dWj) * mj, kaJ = (dWi + dWj) * mi;
            const double du = dx * ux + dy * uy + dz * uz;
            const double w = du * ri;
            const double wn = w < 0.0 ? w : 0.0;
            const double vs = c_i + s.vsnd[j] - 3.0 * wn;
            const double rh = 1.0 / (rho_i + rho_j);
            const double B = b_i + b_j, A = al_i + al_j;
            const double av = B * A * vs * wn;
            const double T = pc_i + pc_j - 0.5 * av * rh;
            const double taI = T * kaI * ri, taJ = T * kaJ * ri;
            const double Eg = et_i * dWi + et_j * dWj;
            const double dgI = s.G * mj * ri * Eg, dgJ = s.G * mi * ri * Eg;
            // reverse
            const double ad = Ahx * dx + Ahy * dy + Ahz * dz, bd = Bhx * dx + Bhy * dy + Bhz * dz;
            const double ci = dgI - taI, cj = taJ - dgJ;
            double ddx = ci * Ahx + cj * Bhx, ddy = ci * Ahy + cj * Bhy, ddz = ci * Ahz + cj * Bhz;
            const double TbI = -ad * kaI * ri, TbJ = bd * kaJ * ri, Tb = TbI + TbJ;
            const double DG = s.G * (ad * mj - bd * mi);
            const double visc = 0.25 * rh * av * wn;
            const double KB = (Us_i * (pc_i * w - visc) - ad * T * ri) * mj + (Us_j * (pc_j * w - visc) + bd * T * ri) * mi;
            const double UI = Us_i * kaI, UJ = Us_j * kaJ, UK = UI + UJ;
            pcb += UI * w + Tb;
            double wb = UI * pc_i + UJ * pc_j;
            const double rhb = -av * (0.25 * wn * UK + 0.5 * Tb);
            const double avb = -rh * (0.25 * wn * UK + 0.5 * Tb);
            double rib = T * (bd * kaJ - ad * kaI) + DG * Eg;
            etb += DG * ri * dWi;
            const double dWib = DG * ri * et_i + KB, dWjb = DG * ri * et_j + KB;
            const double avw = avb * wn;
            bb += avw * A * vs;
            ab += avw * B * vs;
            const double vsb = avw * B * A;
            cb += vsb;
            const double wnb = -0.25 * rh * av * UK + avb * B * A * vs - 3.0 * vsb;
            if (w < 0.0) wb += wnb;
            else if (w == 0.0) wb += 0.5 * wnb;
            const double wr = wb * ri;
            ddx += wr * ux; ddy += wr * uy; ddz += wr * uz;
            vb0 += wr * dx; vb1 += wr * dy; vb2 += wr * dz;
            rib += wb * du;
            rb -= rhb * rh * rh;
            // dW = c1 hinv^4 W1(r hinv)
            hinvb += dWib * CEFF1 * (4.0 * hi3 * w1i + hi4 * w1pi * r);
            const double rb_ = CEFF1 * (dWib * hi4 * w1pi * hi + dWjb * hj4 * w1pj * hj);
            const double r2b2 = (rb_ - rib * ri * ri) * ri;   // twice the adjoint of r^2
            xb0 += ddx + r2b2 * dx;
            xb1 += ddy + r2b2 * dy;
            xb2 += ddz + r2b2 * dz;
        }
        xb0 = lsum(xb0); xb1 = lsum(xb1); xb2 = lsum(xb2);
        vb0 = lsum(vb0); vb1 = lsum(vb1); vb2 = lsum(vb2);
        hinvb = lsum(hinvb); cb = lsum(cb); rb = lsum(rb); bb = lsum(bb);
        ab = lsum(ab); pcb = lsum(pcb); etb = lsum(etb);
        if (act && sub == 0) {
            a.x[3 * i] += xb0; a.x[3 * i + 1] += xb1; a.x[3 * i + 2] += xb2;
            a.v[3 * i] += vb0; a.v[3 * i + 1] += vb1; a.v[3 * i + 2] += vb2;
            a.hinv[i] += hinvb;
            a.c[i] += cb;
            a.rho[i] += rb;
            a.b[i] += bb;
            a.alph[i] += ab;
            a.pc[i] += pcb;
            a.eta[i] += etb;
        }
    }
}

// -------------------------------------------------------------- stage C
// hydro inputs: hinv = 1/h, presc = P Omega/rho^2, b = bswt/2,
// eta = eps^2 Omega etas/(3 rho), P = rho u/1.5
__global__ void adj_hydro_prep(AdjState s, AdjAcc a) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        const double h = s.h[i], rho = s.dens[i], P = s.pres[i], om = s.grdh[i], e2 = s.eps2[i];
        const double et = s.etas[i], u = s.uene[i];
        a.h[i] += -a.hinv[i] / (h * h);
        const double pcb = a.pc[i];
        double Pb = pcb * om / (rho * rho);
        a.omega[i] += pcb * P / (rho * rho);
        a.rho[i] += -2.0 * pcb * P * om / (rho * rho * rho);
        a.bswt[i] += 0.5 * a.b[i];
        const double etb = a.eta[i];
        a.e2[i] += etb * om * et / (3.0 * rho);
        a.omega[i] += etb * e2 * et / (3.0 * rho);
        a.rho[i] += -etb * e2 * om * et / (3.0 * rho * rho);
        a.etas[i] = etb * e2 * om / (3.0 * rho);
        a.rho[i] += Pb * u / 1.5;
        a.u[i] += Pb * rho / 1.5;
    }
}

// -------------------------------------------------------------- stage D
// gravity pairs: seeds acc_sum (G acc), pot_sum (G pot), etas
// Bound by the FP64 pipe (two operations per clock and SM; 86% busy): 46
// operations per pair, of 54 with the adjoints formed one by one (100k: the
// whole derivative 39.3 -> 34.8 ms).
constexpr int AG_WARPS = 4, AG_PARTS = 4;
__global__ void __launch_bounds__(AG_WARPS * 32) adj_gravity(AdjState s, AdjSeed sd, AdjAcc a,
                                                             const sphk::WorkItem *items, int n_items, int *queue) {
    __shared__ dbl4 s_x[AG_WARPS][32];
    __shared__ double s_e[AG_WARPS][32], s_b[AG_WARPS][4][32];
    __shared__ int s_j[AG_WARPS][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n = s.n;
    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(queue, 1);
        it = __shfl_sync(FULL, it, 0);
        if (it >= n_items * AG_PARTS) return;
        // a quarter of an item's list per turn
        const sphk::WorkItem t = items[it / AG_PARTS];
        const int part = it % AG_PARTS;
        const int tpi = sphk::lanes_per_i(t.z);
        const int li = lane / tpi;
        const bool act = li < t.z;
        const int i = t.y + (act ? li : 0);
        const dbl4 xi = s.pos[i];
        const double e2i = s.eps2[i];
        const double sc = act ? 1.0 : 0.0;
        // half the seed of the acceleration, and -3 of those halves
        const double Cx = 0.5 * s.G * sd.acc[3 * i] * sc, Cy = 0.5 * s.G * sd.acc[3 * i + 1] * sc,
                     Cz = 0.5 * s.G * sd.acc[3 * i + 2] * sc;
        const double Dx = -3.0 * Cx, Dy = -3.0 * Cy, Dz = -3.0 * Cz;
        const double Ph = sd.pot ? 0.5 * s.G * sd.pot[i] * sc : 0.0;
        const double Eb3 = 3.0 * a.etas[i] * sc;
        double xs0 = 0, xs1 = 0, xs2 = 0, gs = 0, e2b = 0;
        const int kb = s.g_off[t.x], tiles = (s.g_off[t.x + 1] - kb + 31) / 32;
        const int ke = min(s.g_off[t.x + 1], kb + 32 * (tiles * (part + 1) / AG_PARTS));
        for (int k0 = kb + 32 * (tiles * part / AG_PARTS); k0 < ke; k0 += 32) {
            const int m = min(32, ke - k0);
            __syncwarp();
            int j = -1;
            dbl4 xj = make_dbl4(0.0, 0.0, 0.0, 0.0);   // no entry: mass 0, beside the particle
            double e2 = 1.0;
            if (lane < m) {
                j = s.g_idx[k0 + lane];
                xj = j >= n ? s.mom[j - n] : s.pos[j];
                e2 = j >= n ? s.neps2[j - n] : s.eps2[j];
            } else {
                xj.x = xi.x + 1.0; xj.y = xi.y; xj.z = xi.z;
            }
            xj.w *= 0.5;
            s_x[wid][lane] = xj;
            s_e[wid][lane] = e2;
            s_j[wid][lane] = j;
#pragma unroll
            for (int c = 0; c < 4; ++c) s_b[wid][c][lane] = 0.0;
            __syncwarp();
            // lane l takes entry l + u: the lanes' entries differ, so each
            // entry's sums have one writer per round (and the tpi lanes of a
            // particle take the entries of their own residue)
            for (int u = 0; u < 32; u += tpi) {
                const int k = (lane + u) & 31;
                const dbl4 q = s_x[wid][k];
                const double dx = xi.x - q.x, dy = xi.y - q.y, dz = xi.z - q.z;
                const double r2 = dx * dx + dy * dy + dz * dz;
                const double Ri = sphk::rsqrt_r(r2 + e2i), Rj = sphk::rsqrt_r(r2 + s_e[wid][k]);
                const double Ri2 = Ri * Ri, Rj2 = Rj * Rj;
                const double Ai = q.w * (Ri2 * Ri), Aj = q.w * (Rj2 * Rj);
                const double w = Dx * dx + Dy * dy + Dz * dz;   // 3/2 x the adjoint of g
                // adjoints of a = r^2 + eps^2 (negated), R = a^(-1/2): R^3/2 times that of R
                const double aib = Ai * (Ri2 * (w + Eb3) - Ph);
                const double ajb = Aj * (Rj2 * w - Ph);
                const bool self = s_j[wid][k] == i;   // d = 0, and its eps_j is eps_i
                const double g = self ? 0.0 : Ai + Aj, sum = aib + ajb;
                // -1/2 of the pair's position adjoint: sum d + g C; the
                // particle's C is multiplied in at the end
                xs0 += sum * dx; xs1 += sum * dy; xs2 += sum * dz;
                gs += g;
                e2b += self ? sum : aib;
                s_b[wid][0][k] += sum * dx + g * Cx;
                s_b[wid][1][k] += sum * dy + g * Cy;
                s_b[wid][2][k] += sum * dz + g * Cz;
                s_b[wid][3][k] += self ? 0.0 : ajb;
                __syncwarp();
            }
            if (lane < m) {
                double *x = j >= n ? a.node + 4 * (size_t)(j - n) : a.x + 3 * (size_t)j;
                double *e = j >= n ? x + 3 : a.e2 + j;
#pragma unroll
                for (int c = 0; c < 3; ++c) atomicAdd(x + c, 2.0 * s_b[wid][c][lane]);
                atomicAdd(e, -s_b[wid][3][lane]);
            }
        }
        if (act) {
            atomicAdd(&a.x[3 * i + 0], -2.0 * (xs0 + gs * Cx));
            atomicAdd(&a.x[3 * i + 1], -2.0 * (xs1 + gs * Cy));
            atomicAdd(&a.x[3 * i + 2], -2.0 * (xs2 + gs * Cz));
            atomicAdd(&a.e2[i], -e2b);
        }
    }
}

// -------------------------------------------------------------- stage E
// node moments to particles: centre = sum m x / M, eps^2 = sum m eps^2 / M,
// so particle p receives m_p sum over the nodes containing it of node_adj / M
__global__ void adj_nodes(AdjState s, AdjAcc a) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < s.n; p += gridDim.x * blockDim.x) {
        double sx = 0, sy = 0, sz = 0, se = 0;
        for (int v = s.n - 1 + p; v >= 0; v = s.parent[v]) {
            const double *nb = a.node + 4 * (size_t)v;
            const double inv = 1.0 / s.mom[v].w;
            sx += nb[0] * inv; sy += nb[1] * inv; sz += nb[2] * inv; se += nb[3] * inv;
        }
        const double m = s.pos[p].w;
        a.x[3 * p] += m * sx;
        a.x[3 * p + 1] += m * sy;
        a.x[3 * p + 2] += m * sz;
        a.e2[p] += m * se;
    }
}

// -------------------------------------------------------------- stage F
// eps^2 = (h/ksrh)^2, Balsara switch, sound speed c = sqrt(10 u/9)
__global__ void adj_switch(AdjState s, AdjAcc a) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
        const double h = s.h[i], c = s.vsnd[i];
        a.h[i] += a.e2[i] * 2.0 * h / (KSRH * KSRH);
        const double dv = s.divv[i], rv = s.rotv[i];
        const double ad = fabs(dv), ar = fabs(rv);
        const double k = 1e-4 * KSRH;
        const double S = ad + ar + k * c / h;
        const double bb = a.bswt[i];
        if (S > 0.0 && bb != 0.0) {
            const double iS2 = 1.0 / (S * S);
            a.divv[i] += bb * (S - ad) * iS2 * (dv < 0.0 ? -1.0 : (dv > 0.0 ? 1.0 : 0.0));
            a.rotv[i] += bb * (-ad * iS2) * (rv < 0.0 ? -1.0 : (rv > 0.0 ? 1.0 : 0.0));
            a.c[i] += bb * (-ad * iS2) * k / h;
            a.h[i] += bb * (-ad * iS2) * (-k * c / (h * h));
        }
        if (c > 0.0) a.u[i] += a.c[i] * 5.0 / (9.0 * c);
    }
}

// -------------------------------------------------------------- stage G
// density gradient pass (final h): Omega, divv, rotv -> positions, velocities, h, rho.
// First each particle's forward sums and the adjoints of them (coef) ...
__global__ void __launch_bounds__(128) adj_density_sums(AdjState s, AdjAcc a) {
    const int sub = threadIdx.x & (LANES - 1);
    ADJ_PARTICLES(ip, s.n) {
        const bool act = ip < s.n;
        const int i = act ? ip : s.n - 1;
        const dbl4 xi = s.pos[i], vi = s.vel[i];
        const double h = s.h[i], hinv = 1.0 / h, rho = s.dens[i];
        const long long idi = s.id[i];
        // the particle itself (not in its row): W0(0) = 1, W1(0) = 0
        double Sg = sub == 0 ? xi.w * 3.0 * CEFF0 : 0.0, D = 0, Rx = 0, Ry = 0, Rz = 0;
        const Candidates cand(s.h_rows, s.h_info, s.h_off, s.h_idx, i);
        for (int e = sub; e < (act ? cand.n : 0); e += LANES) {
            const int j = cand.p[e];
            const dbl4 xj = s.pos[j];
            const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (!(r2 < h * h) || s.id[j] == idi) continue;
            const double ri = sphk::rsqrt_r(r2), q = r2 * ri * hinv;
            double w0, w0p, w1, w1p;
            wendland(q, w0, w0p, w1, w1p);
            Sg += xj.w * (3.0 * CEFF0 * w0 + CEFF1 * q * w1);
            const dbl4 vj = s.vel[j];
            const double ux = vi.x - vj.x, uy = vi.y - vj.y, uz = vi.z - vj.z;
            const double ph = xj.w * w1 * ri;
            D += (ux * dx + uy * dy + uz * dz) * ph;
            Rx += (uy * dz - uz * dy) * ph;
            Ry += (uz * dx - ux * dz) * ph;
            Rz += (ux * dy - uy * dx) * ph;
        }
        Sg = lsum(Sg); D = lsum(D); Rx = lsum(Rx); Ry = lsum(Ry); Rz = lsum(Rz);
        if (!act || sub != 0) continue;
        const double h4i = hinv * hinv * hinv * hinv;
        const double grdh = -h4i * Sg;
        const double Z = 1.0 + h * grdh / (3.0 * rho);
        const double om = 1.0 / Z;
        const double Rn = sqrt(Rx * Rx + Ry * Ry + Rz * Rz);
        const double dvb = a.divv[i], rvb = a.rotv[i];
        const double Db = dvb * (-CEFF1 * h4i * om / rho);
        const double omb = a.omega[i] + dvb * (-CEFF1 * h4i * D / rho) + rvb * CEFF1 * h4i * Rn / rho;
        double rb = dvb * CEFF1 * h4i * D * om / (rho * rho) - rvb * CEFF1 * h4i * Rn * om / (rho * rho);
        double hb = dvb * 4.0 * CEFF1 * h4i * hinv * D * om / rho - rvb * 4.0 * CEFF1 * h4i * hinv * Rn * om / rho;
        const double rs = Rn > 0.0 ? rvb * CEFF1 * h4i * om / rho / Rn : 0.0;
        const double Zb = -omb * om * om;
        hb += Zb * grdh / (3.0 * rho);
        const double grb = Zb * h / (3.0 * rho);
        rb += -Zb * h * grdh / (3.0 * rho * rho);
        hb += grb * 4.0 * h4i * hinv * Sg;
        a.h[i] += hb;
        a.rho[i] += rb;
        double *c = a.coef + 5 * (size_t)i;
        c[0] = Db;
        c[1] = rs * Rx;
        c[2] = rs * Ry;
        c[3] = rs * Rz;
        c[4] = -grb * h4i;   // adjoint of Sg
    }
}

// ... then the pairs: what the sums of both ends pass to particle i.  The
// terms of j's sums have -d and -u, and i stands at their other end: both
// signs cancel, so the two ends' coefficients add.  FP64 pipe bound (100k: 2.2 ms).
__global__ void __launch_bounds__(128) adj_density_grad(AdjState s, AdjAcc a) {
    const int sub = threadIdx.x & (LANES - 1);
    ADJ_PARTICLES(ip, s.n) {
        const bool act = ip < s.n;
        const int i = act ? ip : s.n - 1;
        const dbl4 xi = s.pos[i], vi = s.vel[i];
        const double hi_len = s.h[i], hi = 1.0 / hi_len;
        const long long idi = s.id[i];
        const double *c = a.coef + 5 * (size_t)i;
        const double Dbi = c[0], Rxi = c[1], Ryi = c[2], Rzi = c[3], Sgi = c[4];
        double hb = 0, xb0 = 0, xb1 = 0, xb2 = 0, vb0 = 0, vb1 = 0, vb2 = 0;
        const Candidates cand(s.h_rows, s.h_info, s.h_off, s.h_idx, i);
        for (int e = sub; e < (act ? cand.n : 0); e += LANES) {
            const int j = cand.p[e];
            const dbl4 xj = s.pos[j];
            const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double hj_len = s.h[j];
            const double hm = fmax(hi_len, hj_len);
            if (!(r2 < hm * hm) || s.id[j] == idi) continue;
            const dbl4 vj = s.vel[j];
            const double ux = vi.x - vj.x, uy = vi.y - vj.y, uz = vi.z - vj.z;
            const double ri = sphk::rsqrt_r(r2), r = r2 * ri;
            const double ud = ux * dx + uy * dy + uz * dz;
            const double cx = uy * dz - uz * dy, cy = uz * dx - ux * dz, cz = ux * dy - uy * dx;
            double P = 0, Qx = 0, Qy = 0, Qz = 0, r2b2 = 0;   // r2b2: twice the adjoint of r^2
            // one end's sums: coefficients, 1/h, the other end's mass
            auto end = [&](double Db, double Rx, double Ry, double Rz, double Sg, double hinv, double m) -> double {
                const double q = r * hinv;
                double w0, w0p, w1, w1p;
                wendland(q, w0, w0p, w1, w1p);
                const double ph = m * w1 * ri;
                P += Db * ph;
                Qx += ph * Rx; Qy += ph * Ry; Qz += ph * Rz;
                const double phb = Db * ud + Rx * cx + Ry * cy + Rz * cz;
                const double qb = m * (Sg * (3.0 * CEFF0 * w0p + CEFF1 * (w1 + q * w1p)) + phb * w1p * ri);
                r2b2 += (qb * hinv - phb * m * w1 * ri * ri) * ri;
                return qb;
            };
            if (r2 < hi_len * hi_len) hb -= end(Dbi, Rxi, Ryi, Rzi, Sgi, hi, xj.w) * r * hi * hi;
            if (r2 < hj_len * hj_len) {
                const double *cj = a.coef + 5 * (size_t)j;
                end(cj[0], cj[1], cj[2], cj[3], cj[4], 1.0 / hj_len, xi.w);
            }
            vb0 += P * dx + dy * Qz - dz * Qy;
            vb1 += P * dy + dz * Qx - dx * Qz;
            vb2 += P * dz + dx * Qy - dy * Qx;
            xb0 += P * ux + Qy * uz - Qz * uy + r2b2 * dx;
            xb1 += P * uy + Qz * ux - Qx * uz + r2b2 * dy;
            xb2 += P * uz + Qx * uy - Qy * ux + r2b2 * dz;
        }
        hb = lsum(hb);
        xb0 = lsum(xb0); xb1 = lsum(xb1); xb2 = lsum(xb2);
        vb0 = lsum(vb0); vb1 = lsum(vb1); vb2 = lsum(vb2);
        if (act && sub == 0) {
            a.x[3 * i] += xb0; a.x[3 * i + 1] += xb1; a.x[3 * i + 2] += xb2;
            a.v[3 * i] += vb0; a.v[3 * i + 1] += vb1; a.v[3 * i + 2] += vb2;
            a.h[i] += hb;
        }
    }
}

// -------------------------------------------------------------- stage H
// the three smoothing-length passes: (rho_2, h_3) -> positions, first guess h_0.
// FP64 pipe bound (75% busy; 100k: 5.2 ms); rows of the passes are not
// symmetric, so the j side takes atomics.
__global__ void __launch_bounds__(128) adj_density_passes(AdjState s, AdjAcc a) {
    const int sub = threadIdx.x & (LANES - 1);
    ADJ_PARTICLES(ip, s.n) {
        const bool act = ip < s.n;
        const int i = act ? ip : s.n - 1;
        const dbl4 xi = s.pos[i];
        Candidates cand(s.d_rows, s.d_info, s.d_off, s.d_idx, i);
        // forward: h_k, rho_k and S'_k = sum m q W0'(q) per pass
        double hk[4], rk[3], sp[3];
        hk[0] = s.h0[i];
        const double h_row = hk[0] * s.slack * 0.99998;
        for (int p = 0; p < 3; ++p) {
            if (p > 0 && hk[p] > h_row) {   // beyond the row: the walk's list
                const int w = s.d_info[i].y;
                cand.p = s.d_idx + s.d_off[w];
                cand.n = s.d_off[w + 1] - s.d_off[w];
            }
            const double hinv = 1.0 / hk[p];
            double S0 = 0, S1 = 0;
            for (int e = sub; e < cand.n; e += LANES) {
                const dbl4 xj = s.pos[cand.p[e]];
                const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
                const double r2 = dx * dx + dy * dy + dz * dz;
                if (!(r2 < hk[p] * hk[p])) continue;
                const double q = sphk::sqrt_r(r2) * hinv;
                double w0, w0p, w1, w1p;
                wendland(q, w0, w0p, w1, w1p);
                S0 += xj.w * w0;
                S1 += xj.w * q * w0p;
            }
            S0 = lsum(S0);
            sp[p] = lsum(S1);
            rk[p] = CEFF0 * hinv * hinv * hinv * S0;
            hk[p + 1] = s.eta_ksrh * cbrt(xi.w / rk[p]);
        }
        // reverse over the scalars
        double rhob[3], hb[4], fk[3];
        hb[3] = act ? a.h[i] : 0.0;
        rhob[2] = (act ? a.rho[i] : 0.0) + hb[3] * (-hk[3] / (3.0 * rk[2]));
        for (int p = 2; p >= 0; --p) {
            const double hinv = 1.0 / hk[p], hinv4 = hinv * hinv * hinv * hinv;
            // rho = c0 h^-3 S0(h): d rho/d h = -3 rho/h - c0 h^-4 sum m q W0'(q)
            hb[p] = rhob[p] * (-3.0 * rk[p] * hinv - CEFF0 * hinv4 * sp[p]);
            if (p > 0) rhob[p - 1] = hb[p] * (-hk[p] / (3.0 * rk[p - 1]));
            // d rho_k / d r = c0 h_k^-4 m W0'(q_k), W0'(q) = -20 q (1 - q)^3
            fk[p] = -20.0 * CEFF0 * rhob[p] * hinv4 * hinv;
        }
        // pairs: r-bar / r, times d for the separation
        double xb0 = 0, xb1 = 0, xb2 = 0;
        const double hmx = fmax(fmax(hk[0], hk[1]), hk[2]);
        const double hi0 = 1.0 / hk[0], hi1 = 1.0 / hk[1], hi2 = 1.0 / hk[2];
        for (int e = sub; e < (act ? cand.n : 0); e += LANES) {
            const int j = cand.p[e];
            const dbl4 xj = s.pos[j];
            const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (j == i || !(r2 < hmx * hmx)) continue;
            const double r = sphk::sqrt_r(r2);
            const double u0 = sphk::max0(1.0 - r * hi0), u1 = sphk::max0(1.0 - r * hi1), u2 = sphk::max0(1.0 - r * hi2);
            const double f = xj.w * (fk[0] * (u0 * u0 * u0) + fk[1] * (u1 * u1 * u1) + fk[2] * (u2 * u2 * u2));
            xb0 += f * dx; xb1 += f * dy; xb2 += f * dz;
            atomicAdd(&a.x[3 * j + 0], -f * dx);
            atomicAdd(&a.x[3 * j + 1], -f * dy);
            atomicAdd(&a.x[3 * j + 2], -f * dz);
        }
        xb0 = lsum(xb0); xb1 = lsum(xb1); xb2 = lsum(xb2);
        if (act && sub == 0) {
            atomicAdd(&a.x[3 * i + 0], xb0);
            atomicAdd(&a.x[3 * i + 1], xb1);
            atomicAdd(&a.x[3 * i + 2], xb2);
            a.h0[i] = hb[0];
        }
    }
}
#undef ADJ_PARTICLES

// work items: one per 32 i-particles of a group (offsets from an exclusive
// scan of the per-group counts)
__global__ void adj_item_counts(int n_groups, const int *gcount, int *cnt) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n_groups; g += gridDim.x * blockDim.x)
        cnt[g] = (gcount[g] + 31) / 32;
}
__global__ void adj_fill_items(int n_groups, const int *gfirst, const int *gcount, const int *off,
                               sphk::WorkItem *items) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n_groups; g += gridDim.x * blockDim.x) {
        const int c = gcount[g];
        for (int k = 0; 32 * k < c; ++k)
            items[off[g] + k] = make_int4(g, gfirst[g] + 32 * k, min(32, c - 32 * k), 0);
    }
}

}  // namespace sphadj
