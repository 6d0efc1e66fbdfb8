// adjoint.cu -- reverse-mode gradient of the FP64 DEM step (pe has no gradients; this extends the
// path): d loss / d (initial x, v, w) and d loss / d (k_n, c_n, c_t, mu).
//
// The forward map of one step is the grid-search DEM step of dem.cu (pe's linear law and
// semi-implicit Euler, DEMSolver.h:328-379, spheretrait/Default.h:149-220):
//     F_i = sum_c f_c(x, v, w; theta),  T_i = sum_c r_c x f_c
//     v+ = (v + (F/m + g) dt) drag,  x+ = x + (v + (F/m + g) dt) dt,  w+ = (w + I^-1 T dt) drag
// Its vector-Jacobian product, for post-step adjoints (lx+, lv+, lw+):
//     u = lv+ drag + lx+ dt                  (adjoint of the pre-drag velocity)
//     Fbar = u dt / m,  Tbar = lw+ drag I^-1 dt
//     lx = lx+ + sum_c d s_c / dx,  lv = u + sum_c d s_c / dv,  lw = lw+ drag + sum_c d s_c / dw
// with s_c = Fbar_1.f_1 + Tbar_1.tau_1 + Fbar_2.f_2 + Tbar_2.tau_2 for contact c.  Each thread
// owns one body and gathers d s_c over its contacts, the partners coming from the grid step's
// candidate lists.  As tau_i = R_i x f_i and f_2 = -f_1, s_c = f_1 . A with A = Fbar_1 - Fbar_2 +
// Tbar_1 x R_1 - Tbar_2 x R_2, and its derivatives are those of the contact law and geometry taken
// backwards from A by hand.  Kinks of the law (max(0, .), the Coulomb min, contact onset) take the
// branch the forward step took.
//
// Memory: the forward run keeps a checkpoint every K steps; the backward pass recomputes each
// segment from its checkpoint, keeping the K pre-step states (each step writes the next one in
// place) and, while they take at most kSearchBytes, each state's sort and candidate lists, and
// runs the adjoint steps in reverse.  Adjoints are stored by upload index, so the grid re-sorting
// of the state between steps does not matter.
#include <algorithm>
#include <vector>

#include "internal.cuh"
#include "near.cuh"

namespace peb {

namespace {

// the kept sorts and candidate lists of a segment: at most this much device memory, else each
// reversed step searches again
constexpr int64_t kSearchBytes = int64_t(1) << 30;

struct AdjArgs {
    int64_t n;
    double dt, drag;
    const int32_t *sorted, *cell_start;
    const SceneInfo *scenes;
    const MatDev *mats;
    const double4 *planes;
    const int32_t *plane_mat;
    const double *boxes;
    const int32_t *box_mat;
    const double4 *pr;
    const double *vw;
    const uint32_t *tag;
    const int32_t *uid;
    const double *lx1, *lv1, *lw1;  // post-step adjoints by upload index (3n each)
    double *lx0, *lv0, *lw0;        // pre-step adjoints
    double *gpar;                   // per-block partial parameter gradients (4 per block)
    const int32_t *near_cnt, *near_idx;   // the state's candidate lists (near.cuh)
};

__device__ __forceinline__ V3<double> ld3u(const double *a, int64_t u) {
    return v3(a[3 * u], a[3 * u + 1], a[3 * u + 2]);
}

// Fbar, Tbar of a body from its post-step adjoints
__device__ __forceinline__ void body_bars(const AdjArgs &a, int64_t u, double r, double density,
                                          V3<double> &Fb, V3<double> &Tb, V3<double> &uvel) {
    double im, ii, I;
    sphere_mass(r, density, im, ii, I);
    const V3<double> lx = ld3u(a.lx1, u), lv = ld3u(a.lv1, u), lw = ld3u(a.lw1, u);
    uvel = lv * a.drag + lx * a.dt;
    Fb = uvel * (a.dt * im);
    Tb = lw * (a.drag * ii * a.dt);
}

// The contact law (pe's response/DEMSolver.h:328-379, force f on body 1) taken backwards from A, the
// derivative of s_c with respect to f: the derivatives with respect to the normal, the distance, the
// relative velocity and the coefficients k_n, c_n, c_t, mu.
struct LawAdjoint {
    V3<double> f, n, rvel;
    double dist, par[4];
};
__device__ __forceinline__ LawAdjoint law_adjoint(const V3<double> &n, double dist, const V3<double> &rvel,
                                                  const MatDev &m1, const MatDev &m2,
                                                  const V3<double> &A) {
    const double k = 1.0 / (m1.rk + m2.rk), cn = 1.0 / (m1.rcn + m2.rcn), ct = 1.0 / (m1.rct + m2.rct);
    const double nv = dot(n, rvel);
    // friction pick on the forward values (Contact.cpp:102-105)
    const double tvel = dot(n, rvel - n * nv);
    const double mu = fabs(tvel) > kFrictionThreshold ? m1.cdf + m2.cdf : m1.csf + m2.csf;
    const V3<double> vt = n * nv - rvel;
    const double tl = sqrt(dot(vt, vt));
    double fN = k * -dist - cn * nv;
    const bool pressed = !(fN < 0.0);
    if (!pressed) fN = 0.0;
    LawAdjoint r;
    double fb = dot(A, n);                       // d s / d f_N
    V3<double> vb = v3(0.0, 0.0, 0.0);           // d s / d v_t
    r.f = n * fN;
    r.n = A * fN;
    r.par[2] = r.par[3] = 0.0;
    if (tl != 0.0) {   // Vector3::getNormalized leaves a zero vector unchanged
        if (ct * tl < mu * fN) {
            r.f = r.f + vt * ct;
            vb = A * ct;
            r.par[2] = dot(A, vt);
        } else {
            const double il = 1.0 / tl;
            const V3<double> u = vt * il;
            const double au = dot(A, u), m = mu * fN;
            r.f = r.f + u * m;
            fb += mu * au;
            r.par[3] = fN * au;
            vb = (A - u * au) * (m * il);
        }
    }
    r.n = r.n + vb * nv;
    r.rvel = -vb;
    double nvb = dot(n, vb);
    r.dist = r.par[0] = r.par[1] = 0.0;
    if (pressed) {
        r.par[0] = -dist * fb;
        r.par[1] = -nv * fb;
        r.dist = -k * fb;
        nvb -= cn * fb;
    }
    r.n = r.n + rvel * nvb;
    r.rvel = r.rvel + n * nvb;
    return r;
}

// Bound: the chain of dependent FP64 operations and loads of a sphere's contacts (a few warps per
// SM at 16,384 spheres).  With forward-mode dual numbers over the 9 state components and 4
// coefficients, and a 27-cell search in FP64, it took 135 us per step of a 16,224-sphere packing
// with 3 contacts per sphere.
__global__ void __launch_bounds__(128) k_adjoint(AdjArgs a) {
    __shared__ double s_par[4][4];
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double gp[4] = {0.0, 0.0, 0.0, 0.0};
    if (t < a.n) {
        const int32_t b = a.sorted[t];
        const double4 pi = a.pr[b];
        const uint32_t tagi = a.tag[b];
        const int64_t ui = a.uid[b];
        const int cnt = a.near_cnt[t];
        const SceneInfo &s = a.scenes[tagi >> 16];
        const MatDev &mi = a.mats[tagi & 0xffffu];
        const V3<double> xi = v3(pi.x, pi.y, pi.z);
        const V3<double> vi = ld_vw(a.vw, a.n, b, 0), wi = ld_vw(a.vw, a.n, b, 1);
        V3<double> Fbi, Tbi, ui_vel;
        body_bars(a, ui, pi.w, mi.density, Fbi, Tbi, ui_vel);
        V3<double> gx = v3(0.0, 0.0, 0.0), gv = gx, gw = gx;
        // a sphere pair, by the predicate of the forward step; this body's share of d s_c
        auto pair = [&](int32_t j) {
            if (j == b) return;
            const double4 pj = a.pr[j];
            const int64_t uj = a.uid[j];
            const bool self1 = ui < uj;   // pe's orientation: body 1 has the smaller id
            const double4 p1 = self1 ? pi : pj, p2 = self1 ? pj : pi;
            const double nx = p1.x - p2.x, ny = p1.y - p2.y, nz = p1.z - p2.z;
            const double len = length_rn(nx, ny, nz);
            const double dist = __dsub_rn(__dsub_rn(len, p1.w), p2.w);
            if (!(dist < -kContactThreshold)) return;
            const MatDev &mj = a.mats[a.tag[j] & 0xffffu];
            const V3<double> vj = ld_vw(a.vw, a.n, j, 0), wj = ld_vw(a.vw, a.n, j, 1);
            V3<double> Fbj, Tbj, uj_vel;
            body_bars(a, uj, pj.w, mj.density, Fbj, Tbj, uj_vel);
            const V3<double> V1 = self1 ? vi : vj, V2 = self1 ? vj : vi;
            const V3<double> W1 = self1 ? wi : wj, W2 = self1 ? wj : wi;
            const V3<double> Fb1 = self1 ? Fbi : Fbj, Tb1 = self1 ? Tbi : Tbj;
            const V3<double> Fb2 = self1 ? Fbj : Fbi, Tb2 = self1 ? Tbj : Tbi;
            const V3<double> d = v3(nx, ny, nz);
            const double il = 1.0 / len;
            const V3<double> n = d * il;
            const double kk = p2.w + 0.5 * dist;
            const V3<double> R2 = n * kk, R1 = R2 - d;
            const V3<double> rvel = (V1 + cross(W1, R1)) - (V2 + cross(W2, R2));
            const V3<double> A = (Fb1 - Fb2) + cross(Tb1, R1) - cross(Tb2, R2);
            const LawAdjoint g = law_adjoint(n, dist, rvel, self1 ? mi : mj, self1 ? mj : mi, A);
            // the contact point: R_1 = x_2 + n kk - x_1, R_2 = n kk, kk = r_2 + dist / 2
            const V3<double> R1b = cross(g.f, Tb1) + cross(g.rvel, W1);
            const V3<double> R2b = -(cross(g.f, Tb2) + cross(g.rvel, W2));
            const V3<double> Rb = R1b + R2b;
            const V3<double> nb = g.n + Rb * kk;
            const double db = g.dist + 0.5 * dot(n, Rb);
            // n = d / |d|, dist = |d| - r_1 - r_2
            const V3<double> xb = (nb - n * dot(n, nb)) * il + n * db - R1b;
            if (self1) {
                gx = gx + xb;
                gv = gv + g.rvel;
                gw = gw + cross(R1, g.rvel);
#pragma unroll
                for (int k = 0; k < 4; ++k) gp[k] += g.par[k];   // once per contact
            } else {
                gx = gx - xb;
                gv = gv - g.rvel;
                gw = gw - cross(R2, g.rvel);
            }
        };
        // a wall contact (the sphere is body 1, the wall does not move): the derivatives with
        // respect to the normal, the distance and R_1 are left to the wall's geometry
        auto wall = [&](const V3<double> &n, double dist, const V3<double> &R1, const MatDev &mw,
                        V3<double> &nb, double &db, V3<double> &R1b) {
            const V3<double> rvel = vi + cross(wi, R1);
            const V3<double> A = Fbi + cross(Tbi, R1);
            const LawAdjoint g = law_adjoint(n, dist, rvel, mi, mw, A);
            R1b = cross(g.f, Tbi) + cross(g.rvel, wi);
            nb = g.n;
            db = g.dist;
            gv = gv + g.rvel;
            gw = gw + cross(R1, g.rvel);
#pragma unroll
            for (int k = 0; k < 4; ++k) gp[k] += g.par[k];
        };
        if (cnt > kNear) {
            // more candidates than recorded: the 27 cells around the sphere
            int cx, cy, cz;
            cell_coords(s, pi.x, pi.y, pi.z, cx, cy, cz);
            const int x0 = max(cx - 1, 0), x1 = min(cx + 1, s.dim[0] - 1);
            for (int z = max(cz - 1, 0); z <= min(cz + 1, s.dim[2] - 1); ++z)
                for (int y = max(cy - 1, 0); y <= min(cy + 1, s.dim[1] - 1); ++y) {
                    const int64_t c0 = cell_key(s, x0, y, z);
                    const int e = a.cell_start[c0 + (x1 - x0) + 1];
                    for (int slot = a.cell_start[c0]; slot < e; ++slot) pair(a.sorted[slot]);
                }
        } else if (cnt > 0) {
            int32_t sl[kNear];
            load_near(a.near_idx, a.n, t, cnt, sl);
#pragma unroll 1
            for (int k = 0; k < cnt; ++k) {
                pair(a.sorted[sl[0]]);
                // the next candidate to the front (constant indexes keep the list in registers)
#pragma unroll
                for (int q = 0; q + 1 < kNear; ++q) sl[q] = sl[q + 1];
            }
        }
        for (int p = 0; p < s.nplanes; ++p) {
            const double4 pl = a.planes[s.plane_begin + p];
            const double kd = dot_rn(pl.x, pl.y, pl.z, pi.x, pi.y, pi.z);
            const double dist = __dsub_rn(__dsub_rn(kd, pi.w), pl.w);
            if (!(dist < -kContactThreshold)) continue;
            // dist = n . x - r - d, R_1 = -n (r + dist)
            const V3<double> n = v3(pl.x, pl.y, pl.z), R1 = n * -(pi.w + dist);
            V3<double> nb, R1b;
            double db;
            wall(n, dist, R1, a.mats[a.plane_mat[s.plane_begin + p]], nb, db, R1b);
            gx = gx + n * (db - dot(n, R1b));
        }
        for (int k = 0; k < s.nboxes; ++k) {
            const double *B = a.boxes + 15 * (int64_t)(s.box_begin + k);
            const double *R = B + 6;
            const double l[3] = {0.5 * B[3], 0.5 * B[4], 0.5 * B[5]};
            const V3<double> D = xi - v3(B[0], B[1], B[2]);
            double p[3] = {D.x * R[0] + D.y * R[3] + D.z * R[6], D.x * R[1] + D.y * R[4] + D.z * R[7],
                           D.x * R[2] + D.y * R[5] + D.z * R[8]};
            bool beyond[3];
            bool outside = false;
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                beyond[ax] = p[ax] < -l[ax] || p[ax] > l[ax];
                if (p[ax] < -l[ax]) p[ax] = -l[ax];
                else if (p[ax] > l[ax]) p[ax] = l[ax];
                outside = outside || beyond[ax];
            }
            const MatDev &mw = a.mats[a.box_mat[s.box_begin + k]];
            V3<double> nb, R1b;
            double db;
            if (!outside) {
                // the centre is inside the box: the nearest face's normal, R_1 = 0
                double dmax = fabs(p[0]) - l[0], pf = p[0];
                int face = 0;
#pragma unroll
                for (int ax = 1; ax < 3; ++ax) {
                    const double tmp = fabs(p[ax]) - l[ax];
                    if (dmax < tmp) { dmax = tmp; face = ax; pf = p[ax]; }
                }
                const double sg = (pf > 0.0) ? 1.0 : -1.0;
                const V3<double> n = v3(R[face] * sg, R[3 + face] * sg, R[6 + face] * sg);
                const double dist = dmax - pi.w;
                if (!(dist < -kContactThreshold)) continue;
                wall(n, dist, v3(0.0, 0.0, 0.0), mw, nb, db, R1b);
                gx = gx + n * db;
            } else {
                // m = D - q from the box's nearest point q; dist = |m| - r, n = m / |m|, R_1 = -m;
                // m depends on x through the axes along which the centre is beyond the box
                const V3<double> q = v3(R[0] * p[0] + R[1] * p[1] + R[2] * p[2],
                                        R[3] * p[0] + R[4] * p[1] + R[5] * p[2],
                                        R[6] * p[0] + R[7] * p[1] + R[8] * p[2]);
                const V3<double> m = D - q;
                const double L = sqrt(dot(m, m)), dist = L - pi.w;
                if (!(dist < -kContactThreshold)) continue;
                const double il = 1.0 / L;
                const V3<double> n = m * il;
                wall(n, dist, -m, mw, nb, db, R1b);
                const V3<double> mb = (nb - n * dot(n, nb)) * il + n * db - R1b;
#pragma unroll
                for (int ax = 0; ax < 3; ++ax) {
                    if (!beyond[ax]) continue;
                    const V3<double> axis = v3(R[ax], R[3 + ax], R[6 + ax]);
                    gx = gx + axis * dot(axis, mb);
                }
            }
        }
        const V3<double> lx = ld3u(a.lx1, ui), lw = ld3u(a.lw1, ui);
        const V3<double> ox = lx + gx, ov = ui_vel + gv, ow = lw * a.drag + gw;
        a.lx0[3 * ui] = ox.x; a.lx0[3 * ui + 1] = ox.y; a.lx0[3 * ui + 2] = ox.z;
        a.lv0[3 * ui] = ov.x; a.lv0[3 * ui + 1] = ov.y; a.lv0[3 * ui + 2] = ov.z;
        a.lw0[3 * ui] = ow.x; a.lw0[3 * ui + 1] = ow.y; a.lw0[3 * ui + 2] = ow.z;
    }
    // per-block parameter partials, summed in a fixed order
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) gp[k] += __shfl_down_sync(0xffffffffu, gp[k], o);
        if ((threadIdx.x & 31) == 0) s_par[k][threadIdx.x >> 5] = gp[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        const double *w = s_par[threadIdx.x];
        a.gpar[4 * blockIdx.x + threadIdx.x] += (w[0] + w[1]) + (w[2] + w[3]);
    }
}

void free_ckpt(Ctx *c, BodyBuf &b) {
    dfree(c, b.pr);
    dfree(c, b.vw);
    dfree(c, b.tag);
    dfree(c, b.uid);
    b = BodyBuf();
}

int alloc_ckpt(Ctx *c, BodyBuf &b) {
    const size_t n = (size_t)std::max<int64_t>(c->n, 1);
    PEB_CUDA(c, dmalloc(c, &b.pr, n * sizeof(double4)));
    PEB_CUDA(c, dmalloc(c, &b.vw, n * (size_t)c->vw_bytes));
    PEB_CUDA(c, dmalloc(c, &b.tag, n * sizeof(uint32_t)));
    PEB_CUDA(c, dmalloc(c, &b.uid, n * sizeof(int32_t)));
    return PE_B200_OK;
}

int copy_state(Ctx *c, BodyBuf &dst, const BodyBuf &src) {
    const size_t n = (size_t)c->n;
    PEB_CUDA(c, cudaMemcpyAsync(dst.pr, src.pr, n * sizeof(double4), cudaMemcpyDeviceToDevice, c->stream));
    PEB_CUDA(c, cudaMemcpyAsync(dst.vw, src.vw, n * (size_t)c->vw_bytes, cudaMemcpyDeviceToDevice, c->stream));
    PEB_CUDA(c, cudaMemcpyAsync(dst.tag, src.tag, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->stream));
    PEB_CUDA(c, cudaMemcpyAsync(dst.uid, src.uid, n * sizeof(int32_t), cudaMemcpyDeviceToDevice, c->stream));
    return PE_B200_OK;
}

}  // namespace

void adjoint_free(Ctx *c) {
    for (auto &b : c->adj.ckpt) free_ckpt(c, b);
    for (auto &b : c->adj.seg) free_ckpt(c, b);
    c->adj.ckpt.clear();
    c->adj.seg.clear();
    dfree(c, c->adj.search);
    c->adj.search = nullptr;
    c->adj.search_bytes = 0;
    c->adj.nsteps = 0;
}

bool adjoint_spare_free(Ctx *c) {
    AdjState &A = c->adj;
    const bool search = A.search && A.busy < 2, seg = !A.seg.empty() && A.busy < 1;
    if (search) {
        dfree(c, A.search);
        A.search = nullptr;
        A.search_bytes = 0;
    }
    if (seg) {
        for (auto &b : A.seg) free_ckpt(c, b);
        A.seg.clear();
    }
    return search || seg;
}

int adjoint_forward(Ctx *c, int32_t nsteps, double dt, int32_t every) {
    if (c->p.solver != PE_B200_DEM || c->p.precision != PE_B200_FP64 || c->p.track_orientation ||
        c->p.force_model != 0)
        return set_err(c, PE_B200_ERR_UNSUPPORTED,
                       "the adjoint needs the linear DEM law in FP64 without orientation tracking");
    if (nsteps < 1 || every < 1 || !(dt > 0.0)) return PE_B200_ERR_ARG;
    AdjState &A = c->adj;
    A.nsteps = 0;   // no run to take backwards until this one is complete
    // the buffers of an earlier run serve this one (an upload frees them); the rest goes back
    const size_t nck = ((size_t)nsteps + every - 1) / every, nseg = (size_t)std::min(nsteps, every) - 1;
    while (A.ckpt.size() > nck) { free_ckpt(c, A.ckpt.back()); A.ckpt.pop_back(); }
    while (A.seg.size() > nseg) { free_ckpt(c, A.seg.back()); A.seg.pop_back(); }
    while (A.ckpt.size() < nck) {
        BodyBuf b;
        const int rc = alloc_ckpt(c, b);
        A.ckpt.push_back(b);
        if (rc) {
            adjoint_free(c);
            return rc;
        }
    }
    c->binned = false;   // whatever ran before; each step bins the state it writes
    for (int s = 0; s < nsteps; ++s) {
        if (s % every == 0) {
            int rc = copy_state(c, A.ckpt[s / every], c->cur);
            if (rc) return rc;
        }
        int rc = dem_step(c, dt);
        if (rc) return rc;
    }
    A.nsteps = nsteps;
    A.every = every;
    A.dt = dt;
    if (c->nl.enabled) return dem_list_request_rebuild(c);
    return PE_B200_OK;
}

int adjoint_backward(Ctx *c, const double *gx, const double *gv, const double *gw, double *ox,
                     double *ov, double *ow, double *gpar) {
    AdjState &A = c->adj;
    if (A.nsteps < 1 || A.ckpt.empty())
        return set_err(c, PE_B200_ERR_STATE, "run pe_b200_adjoint_forward first");
    const int64_t n = c->n;
    const size_t vb = 3 * (size_t)n * sizeof(double);
    double *l[6] = {};
    double *d_gpar = nullptr;
    const unsigned blocks = grid_for(n, 128);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 6 && e == cudaSuccess; ++k) e = dmalloc(c, &l[k], vb);
    if (e == cudaSuccess) e = dmalloc(c, &d_gpar, 4 * sizeof(double) * blocks);
    auto cleanup = [&]() {
        for (int k = 0; k < 6; ++k) dfree(c, l[k]);
        dfree(c, d_gpar);
    };
    if (e != cudaSuccess) {
        cleanup();
        return cuda_err(c, e, "adjoint buffers");
    }
    // post-final adjoints (upload order)
    int rc = PE_B200_OK;
    {
        const double *src[3] = {gx, gv, gw};
        for (int k = 0; k < 3 && e == cudaSuccess; ++k)
            e = cudaMemcpyAsync(l[k], src[k], vb, cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(d_gpar, 0, 4 * sizeof(double) * blocks, c->stream);
        if (e != cudaSuccess) rc = cuda_err(c, e, "adjoint inputs");
    }
    // the pre-step states of a segment after its checkpoint (the forward run's last segment may
    // be shorter than the interval)
    const int seglen = std::min(A.every, A.nsteps);
    A.busy = 1;
    for (size_t k = A.seg.size(); k + 1 < (size_t)seglen && !rc; ++k) {
        BodyBuf b;
        rc = alloc_ckpt(c, b);
        if (rc) free_ckpt(c, b);
        else A.seg.push_back(b);
    }
    // what each step searches with, made here rather than by the first one, so that the kept lists can
    // stand in (and before they take what memory there is)
    if (!rc) rc = near_reserve(c);
    // the segment's sorts and candidate lists: per step the cell offsets, the order, the lists
    const int64_t nn = std::max<int64_t>(n, 1);
    const int64_t per = ((c->ncell + 2 + nn + (1 + kNear) * nn) * (int64_t)sizeof(int32_t) + 255) & ~(int64_t)255;
    const bool keep = !rc && per * seglen <= kSearchBytes;
    if (keep && A.search_bytes < per * seglen) {
        dfree(c, A.search);
        A.search = nullptr;
        A.search_bytes = 0;
        if (dmalloc(c, &A.search, (size_t)(per * seglen)) == cudaSuccess) A.search_bytes = per * seglen;
        else cudaGetLastError();
    }
    const bool kept = keep && A.search_bytes >= per * seglen;
    A.busy = 2;
    // the steps below run on the checkpoints' and the segment's buffers, and search into the kept
    // ones; the context's own state stays what it is
    const BodyBuf cur0 = c->cur, nxt0 = c->nxt;
    int32_t *const sorted0 = c->sorted, *const start0 = c->cell_start, *const near0 = c->near;
    const int32_t grid0 = c->tune.dem_grid;
    c->tune.dem_grid = 0;   // the form with candidate lists (both give the same states)
    auto use = [&](int s) {   // the search buffers of the segment's s-th state
        if (!kept) return;
        int32_t *p = (int32_t *)((char *)A.search + per * s);
        c->cell_start = p;
        c->sorted = p + c->ncell + 2;
        c->near = c->sorted + nn;
    };
    int cur_l = 0;  // l[cur_l..cur_l+2] hold the post-step adjoints
    const int nck = (int)A.ckpt.size();
    for (int seg = nck - 1; seg >= 0 && !rc; --seg) {
        const int s0 = seg * A.every;
        const int len = std::min(A.nsteps, s0 + A.every) - s0;
        auto state = [&](int s) -> const BodyBuf & { return s == 0 ? A.ckpt[seg] : A.seg[s - 1]; };
        // recompute the segment, each step writing the next pre-step state
        c->binned = false;
        for (int s = 0; s < len && !rc; ++s) {
            use(s);
            c->cur = state(s);
            if (s + 1 < len) {
                c->nxt = state(s + 1);
                rc = dem_step(c, A.dt);
            } else if (kept) {
                rc = dem_search(c);
            }
        }
        for (int s = len - 1; s >= 0 && !rc; --s) {
            c->cur = state(s);
            use(s);
            if (!kept) {
                c->binned = false;
                rc = dem_search(c);
                if (rc) break;
            }
            AdjArgs a;
            a.n = n;
            a.dt = A.dt;
            a.drag = c->p.damping < 1.0 ? pow(c->p.damping, A.dt) : 1.0;
            a.sorted = c->sorted;
            a.cell_start = c->cell_start;
            a.scenes = c->d_scenes;
            a.mats = c->d_mats;
            a.planes = c->d_planes;
            a.plane_mat = c->d_plane_mat;
            a.boxes = c->d_boxes;
            a.box_mat = c->d_box_mat;
            a.pr = c->cur.pr;
            a.vw = (const double *)c->cur.vw;
            a.tag = c->cur.tag;
            a.uid = c->cur.uid;
            a.lx1 = l[cur_l];
            a.lv1 = l[cur_l + 1];
            a.lw1 = l[cur_l + 2];
            a.lx0 = l[3 - cur_l];
            a.lv0 = l[4 - cur_l];
            a.lw0 = l[5 - cur_l];
            a.gpar = d_gpar;
            a.near_cnt = c->near;
            a.near_idx = c->near + n;
            if (n > 0) {
                k_adjoint<<<blocks, 128, 0, c->stream>>>(a);
                c->launches++;
                e = cudaGetLastError();
                if (e != cudaSuccess) rc = cuda_err(c, e, "k_adjoint");
            }
            cur_l = 3 - cur_l;
        }
    }
    c->cur = cur0;
    c->nxt = nxt0;
    c->sorted = sorted0;
    c->cell_start = start0;
    c->near = near0;
    c->tune.dem_grid = grid0;
    c->binned = false;
    A.busy = 0;
    if (!rc) {
        std::vector<double> hp(4 * (size_t)blocks);
        e = cudaMemcpyAsync(ox, l[cur_l], vb, cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ov, l[cur_l + 1], vb, cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ow, l[cur_l + 2], vb, cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(hp.data(), d_gpar, hp.size() * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) rc = cuda_err(c, e, "adjoint results");
        for (int k = 0; k < 4 && !rc; ++k) {
            double s = 0.0;
            for (unsigned b = 0; b < blocks; ++b) s += hp[4 * b + k];
            if (gpar) gpar[k] = s;
        }
    }
    if (!rc && c->nl.enabled) rc = dem_list_request_rebuild(c);
    cudaStreamSynchronize(c->stream);
    cleanup();
    return rc;
}

}  // namespace peb
