// FP64 all-pairs forces with every unordered pair formed once: Newton's third
// law for the Newtonian and the pairwise 1PN force (the pair law of
// allpairs.cu; compute_gravitational / get_pn1,
// src/physics/tool_chain_impl.cpp:110-137).
//
// Bound by the FP64 pipe. A directed Newtonian pair costs 16 FP64 operations
// (separation 3, r^2 3, r^-3 6, mass 1, update 3); formed once for both bodies
// it is 20, so 10 per directed pair. Bodies are cut into tiles of `tile`
// bodies; one block takes one unordered pair of tiles (I, J). Its warps share
// the i bodies (32 U at a time, U per lane, in registers) and split J into
// sub-tiles of 32: a warp holds one j body per lane, with its running
// acceleration, and rotates the 32 of them around the warp with shuffles, so
// after 32 steps every j has met every i of the set and is back at its lane.
// The shuffles (14 32-bit words a step) and the loop run in the issue slots
// that the FP64 pipe leaves free (one FP64 instruction every other cycle).
// j sums stay in shared memory between i sets (each warp owns its sub-tiles),
// i sums are added over the warps at the end of a set. Tile pair (I, J) writes
// the pull of J on I's bodies to slot J and of I on J's bodies to slot I of a
// partial array (slots x 3 x n), which k_sym_reduce adds in slot order: no
// atomics, the same sums every run.
//
// Measured against the directed kernel (device time of an evaluation, same box):
// Newton 1000 bodies 0.026 -> 0.015 ms, 4096 0.043 -> 0.029, 12,001 0.203 ->
// 0.134, 65,536 5.46 -> 3.09, 262,144 82.2 -> 47.8 ms; 1PN 30,011 bodies 3.13
// -> 2.14 ms. The FP64 pipe is about 75% busy (52 cycles per scheduler and
// warp's pair, 40 of them the 20 FP64 operations); 8 i bodies a lane at two
// blocks per SM beat 4 at three or four (50.1, 48.8 against 46.9 ms at
// 262,144) and 6 at two (49.5): fewer shuffles per pair count for more than
// warps. Testing every r^2's range cost 8%, hence the untested rounds below.
#include <algorithm>

#include "aster_internal.cuh"
#include "fp64_pair.cuh"
#include "pn.cuh"

namespace {

constexpr int JT = 1024;           // j bodies whose sums a block keeps in shared memory
constexpr double SYM_PAD = 1.0e90;  // where lanes past the last body sit (massless)
// Softening of at least SYM_EPS2 and coordinates below SYM_FAR keep every r^2
// within [1e-200, 1e200]: rounds between such bodies test nothing.
constexpr double SYM_FAR = 1.0e99, SYM_EPS2 = 1.0e-199;

struct SymArgs {
    int64_t n, npad;
    int set, tile, slots;  // bodies of the i sets, bodies of a tile (whole sets), tiles
    const double4* pm;
    const double4* vel;
    double eps2, G, c2;
    double* part;
};

// One body's state as a lane holds it (the velocities: 1PN only).
struct SymBody {
    double x, y, z, m, ax, ay, az;
    double vx, vy, vz, v2;
};

__device__ __forceinline__ double rot1(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// Adds the pair's force to a (and, SYM, to b): fa = m_b / r^3, fb = m_a / r^3,
// inv = 1 / r (1PN only), d = x_b - x_a.
template <int PNL, bool SYM>
__device__ __forceinline__ void sym_pair(SymBody& a, SymBody& b, double fa, double fb, double inv, double dx, double dy,
                                         double dz, double G, double c2) {
    if constexpr (PNL == 0) {
        a.ax = fma(dx, fa, a.ax); a.ay = fma(dy, fa, a.ay); a.az = fma(dz, fa, a.az);
        if constexpr (SYM) {
            b.ax = fma(-dx, fb, b.ax); b.ay = fma(-dy, fb, b.ay); b.az = fma(-dz, fb, b.az);
        }
    } else {
        // with u = d.v_a, w = d.v_b: a_a += m_b r^-3 [d (1 - c^-2 A) - (v_a - v_b) c^-2 (4u - 3w)],
        // A = 4 v_a.v_b - v_a^2 - 2 v_b^2 + 3/2 (w/r)^2 + (5 m_a + 4 m_b) G / r (get_pn1's bracket with n = -d/r)
        const double vx = a.vx - b.vx, vy = a.vy - b.vy, vz = a.vz - b.vz;
        const double w = fma(dx, b.vx, fma(dy, b.vy, dz * b.vz));
        const double u = fma(dx, a.vx, fma(dy, a.vy, dz * a.vz));
        const double vab = fma(a.vx, b.vx, fma(a.vy, b.vy, a.vz * b.vz));
        const double q = fma(4.0, vab, -a.v2) - b.v2;
        const double gs = G * inv;
        {
            const double ws = w * inv;
            double A = fma(1.5 * ws, ws, q - b.v2);
            A = fma(fma(4.0, b.m, 5.0 * a.m), gs, A);
            const double fc = fa * c2;
            const double fd = fma(-fc, A, fa), fv = fc * fma(4.0, u, -3.0 * w);
            a.ax = fma(-vx, fv, fma(dx, fd, a.ax));
            a.ay = fma(-vy, fv, fma(dy, fd, a.ay));
            a.az = fma(-vz, fv, fma(dz, fd, a.az));
        }
        if constexpr (SYM) {  // the same with a and b exchanged: d, v_a - v_b change sign, u and w swap
            const double us = u * inv;
            double A = fma(1.5 * us, us, q - a.v2);
            A = fma(fma(4.0, a.m, 5.0 * b.m), gs, A);
            const double fc = fb * c2;
            const double fd = fma(-fc, A, fb), fv = fc * fma(3.0, u, -4.0 * w);
            b.ax = fma(vx, fv, fma(-dx, fd, b.ax));
            b.ay = fma(vy, fv, fma(-dy, fd, b.ay));
            b.az = fma(vz, fv, fma(-dz, fd, b.az));
        }
    }
}

// 32 rotation steps: the warp's 32 j bodies against U i bodies per lane. CHECK:
// some r^2 may lie outside the series step's range (r2_ordinary) and is tested.
template <int PNL, int U, bool SYM, bool CHECK>
__device__ __forceinline__ void sym_round(SymBody (&bi)[U], SymBody& bj, double eps2, double G, double c2, int src) {
#pragma unroll 1
    for (int k = 0; k < 32; ++k) {
        double dx[U], dy[U], dz[U], r2[U], s3[U], inv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            dx[u] = bj.x - bi[u].x; dy[u] = bj.y - bi[u].y; dz[u] = bj.z - bi[u].z;
            r2[u] = fma(dx[u], dx[u], fma(dy[u], dy[u], fma(dz[u], dz[u], eps2)));
            if constexpr (PNL == 0) {
                s3[u] = inv_r3_fast(r2[u]);
                inv[u] = 0.0;
            } else {
                inv[u] = inv_r_fast(r2[u]);
                s3[u] = inv[u] * inv[u] * inv[u];
            }
        }
        if constexpr (CHECK) {
            double fi[U], fj[U];
            bool odd = false;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                fi[u] = s3[u] * bj.m;
                fj[u] = s3[u] * bi[u].m;
                odd = odd || !r2_ordinary(r2[u]);
            }
            if (odd) {  // a body and itself without softening, or extreme separations
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (!r2_ordinary(r2[u])) {
                        const double v = inv_r_any(r2[u]), v2 = v * v;
                        fi[u] = bj.m * v * v2;  // the mass first: r^-3 alone may leave the range
                        fj[u] = bi[u].m * v * v2;
                        inv[u] = v;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                sym_pair<PNL, SYM>(bi[u], bj, fi[u], fj[u], inv[u], dx[u], dy[u], dz[u], G, c2);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
                sym_pair<PNL, SYM>(bi[u], bj, s3[u] * bj.m, s3[u] * bi[u].m, inv[u], dx[u], dy[u], dz[u], G, c2);
        }
        bj.x = rot1(bj.x, src); bj.y = rot1(bj.y, src); bj.z = rot1(bj.z, src); bj.m = rot1(bj.m, src);
        if constexpr (SYM) { bj.ax = rot1(bj.ax, src); bj.ay = rot1(bj.ay, src); bj.az = rot1(bj.az, src); }
        if constexpr (PNL > 0) {
            bj.vx = rot1(bj.vx, src); bj.vy = rot1(bj.vy, src); bj.vz = rot1(bj.vz, src);
            bj.v2 = rot1(bj.v2, src);
        }
    }
}

template <int PNL>
__device__ __forceinline__ bool sym_load(const SymArgs& g, int64_t b, SymBody& s) {
    const bool ok = b < g.n;
    const double4 p = ok ? g.pm[b] : make_double4(SYM_PAD, SYM_PAD, SYM_PAD, 0.0);
    s.x = p.x; s.y = p.y; s.z = p.z; s.m = p.w;
    s.ax = s.ay = s.az = 0.0;
    if constexpr (PNL > 0) {
        const double4 v = ok ? g.vel[b] : make_double4(0, 0, 0, 0);
        s.vx = v.x; s.vy = v.y; s.vz = v.z;
        s.v2 = v.x * v.x + v.y * v.y + v.z * v.z;
    }
    return fmax(fabs(s.x), fmax(fabs(s.y), fabs(s.z))) < SYM_FAR;
}

// Block b: tile pair (I, J). The off-diagonal pairs come first, by distance
// J - I (mod slots), the diagonal ones (half the work) last.
template <int PNL, int U, int W>
__global__ void __launch_bounds__(32 * W, U == 2 ? 8 : 2) k_allpairs_sym(SymArgs g) {
    extern __shared__ double sym_smem[];
    constexpr int SET = 32 * U;
    const int jt = g.tile < JT ? g.tile : JT;
    double* sj = sym_smem;           // [3][jt] sums of the j bodies
    double* red = sym_smem + 3 * jt;  // [W][3][SET] the warps' sums of the i bodies
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, src = (lane + 1) & 31;
    const int S = g.slots;
    const int64_t noff = (int64_t)S * (S - 1) / 2;
    int I, J;
    if ((int64_t)blockIdx.x < noff) {
        I = (int)(blockIdx.x % S);
        J = I + 1 + (int)(blockIdx.x / S);
        if (J >= S) J -= S;
    } else {
        I = J = (int)(blockIdx.x - noff);
    }
    const bool diag = I == J;
    const int64_t i0 = (int64_t)I * g.tile, i1 = min(g.npad, i0 + g.tile);
    const int64_t j0 = (int64_t)J * g.tile, j1 = min(g.npad, j0 + g.tile);
    double* pI = g.part + (int64_t)J * 3 * g.npad;  // slot J: the pull of tile J
    double* pJ = g.part + (int64_t)I * 3 * g.npad;
    for (int64_t js = j0; js < j1; js += jt) {
        const int nsub = (int)((min(j1, js + jt) - js) >> 5);
        for (int t = warp; t < nsub; t += W)
            for (int c = 0; c < 3; ++c) sj[c * jt + 32 * t + lane] = 0.0;
        for (int64_t is = i0; is < i1; is += SET) {
            SymBody bi[U];
            bool near_i = g.eps2 >= SYM_EPS2 && g.eps2 < 1e199;
#pragma unroll
            for (int u = 0; u < U; ++u) near_i = sym_load<PNL>(g, is + 32 * u + lane, bi[u]) && near_i;
            for (int t = warp; t < nsub; t += W) {
                const int64_t jb = js + 32 * t;
                if (diag && jb < is) continue;  // met as (i, j) of the other order
                SymBody bj;
                const bool plain = __all_sync(0xffffffffu, sym_load<PNL>(g, jb + lane, bj) && near_i);
                if (diag && jb < is + SET) {  // inside the set: both orders occur, each for its i alone
                    if (plain) sym_round<PNL, U, false, false>(bi, bj, g.eps2, g.G, g.c2, src);
                    else sym_round<PNL, U, false, true>(bi, bj, g.eps2, g.G, g.c2, src);
                } else {
                    double* a = sj + 32 * t + lane;
                    bj.ax = a[0]; bj.ay = a[jt]; bj.az = a[2 * jt];
                    if (plain) sym_round<PNL, U, true, false>(bi, bj, g.eps2, g.G, g.c2, src);
                    else sym_round<PNL, U, true, true>(bi, bj, g.eps2, g.G, g.c2, src);
                    a[0] = bj.ax; a[jt] = bj.ay; a[2 * jt] = bj.az;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                double* r = red + warp * 3 * SET + 32 * u + lane;
                r[0] = bi[u].ax; r[SET] = bi[u].ay; r[2 * SET] = bi[u].az;
            }
            __syncthreads();
            for (int k = threadIdx.x; k < 3 * SET; k += 32 * W) {
                double v = red[k];
                for (int w = 1; w < W; ++w) v += red[w * 3 * SET + k];
                double* o = pI + (int64_t)(k / SET) * g.npad + is + k % SET;
                *o = js > j0 ? *o + v : v;
            }
            __syncthreads();
        }
        // the j sums of this part of J (a diagonal pair adds them to its i sums)
        for (int k = threadIdx.x; k < 3 * 32 * nsub; k += 32 * W) {
            const int c = k / (32 * nsub), b = k - c * 32 * nsub;
            double* o = pJ + (int64_t)c * g.npad + js + b;
            const double v = sj[c * jt + b];
            *o = diag ? *o + v : v;
        }
        __syncthreads();
    }
}

// Sum of a body's slots in slot order, one thread per component (a warp takes
// 32 bodies of one component), scaled by G; then the closing kick and, with pm,
// the next step's opening kick and drift (the operations of the kick-drift
// kernel in its order, so that it need not run).
__global__ void __launch_bounds__(192) k_sym_reduce(int64_t n, int64_t npad, int slots, const double* __restrict__ part,
                                                    double G, double4* __restrict__ acc, double4* __restrict__ vel,
                                                    double kick_dt, double4* __restrict__ pm, double drift_dt) {
    const int c = (threadIdx.x >> 5) % 3;
    const int64_t b = ((int64_t)blockIdx.x * 2 + threadIdx.x / 96) * 32 + (threadIdx.x & 31);
    if (b >= n) return;
    const double* p = part + (int64_t)c * npad + b;
    double a = 0.0;
#pragma unroll 8
    for (int s = 0; s < slots; ++s) a += p[(int64_t)s * 3 * npad];
    a *= G;
    double* o = reinterpret_cast<double*>(acc + b);
    o[c] = a;
    if (c == 2) o[3] = 0.0;
    if (vel) {
        double* vp = reinterpret_cast<double*>(vel + b) + c;
        double v = *vp;
        v += a * kick_dt;
        if (pm) {
            double* x = reinterpret_cast<double*>(pm + b) + c;
            v += a * kick_dt;
            *x += v * drift_dt;
        }
        *vp = v;
    }
}

// W = 4, U = 8: 24 KB of j sums and 24 KB of i sums, the 48 KB a launch gets
// without opting in
template <int PNL, int U, int W>
int launch_sym(aster_ctx* c, const SymArgs& g) {
    static_assert((3 * JT + W * 3 * 32 * U) * sizeof(double) <= 48 * 1024, "no opt-in shared memory");
    static_assert(JT % (32 * U) == 0, "tiles beyond JT bodies are whole sets");
    const int64_t blocks = (int64_t)g.slots * (g.slots + 1) / 2;
    const int jt = g.tile < JT ? g.tile : JT;
    const size_t smem = ((size_t)3 * jt + (size_t)W * 3 * 32 * U) * sizeof(double);
    k_allpairs_sym<PNL, U, W><<<(unsigned)blocks, 32 * W, smem, c->stream>>>(g);
    ASTER_CUDA(cudaGetLastError());
    return ASTER_OK;
}

// Tiles: as many as SYM_SLOTS and the limit on the partial sums (1 GB) allow. The
// partial array is 24 bytes a body and slot, and every tile pair writes two of its
// rows; 128 slots give 8256 tile pairs for the 296 resident blocks. 262,144 bodies
// with 64 / 128 / 256 slots: 55.8 / 52.9 / 52.8 ms; 40,000 bodies: 1.37 / 1.30 /
// 1.31 ms (4 bodies per lane). Beyond 349,525 bodies fewer slots fit: 699,050 with
// 128 / 64 / 24 slots 342 / 353 / 386 ms, 2^20 with 128 / 42 / 24 765 / 831 / 946.
// Fewer than SYM_SLOTS_MIN are fewer tile pairs than resident blocks, and the
// directed kernel is faster: 2^20 with 20 slots 1239 ms, directed 1141; 524,289
// with 24 slots 221, with 20 308, directed 291; 1PN there 604 ms with 128 slots,
// 688 with 24, 962 with 20, directed 872.
constexpr int SYM_SLOTS = 128, SYM_SLOTS_MIN = 24;
// Smaller systems take tiles of 64 bodies (2 per lane, 2 warps), larger ones
// of 256 (8 per lane, 4 warps; 1PN 128 and 4): Newton at 4096 bodies 0.033
// against 0.029 ms, at 8192 0.087 against 0.076; 1PN at 1000 0.021 against
// 0.028 ms, at 4096 0.068 against 0.064.
constexpr int64_t SYM_SMALL = 4000;
// Below this size a single target block with source slices is as fast.
constexpr int64_t SYM_MIN = 128;

}  // namespace

static SymArgs sym_args(const aster_ctx* c, const aster_params* p) {
    const int pnl = pn_level(p);
    SymArgs g;
    const int set = g.set = c->n < SYM_SMALL ? 64 : pnl ? 128 : 256;
    g.n = c->n;
    g.npad = (c->n + set - 1) / set * set;
    const int64_t sets = g.npad / set;
    int64_t most = std::min<int64_t>(SYM_SLOTS, (int64_t)(c->sums_limit / (24 * (size_t)g.npad)));
    if (most < 1) most = 1;
    g.tile = (int)((sets + most - 1) / most) * set;
    if (g.tile > JT) g.tile = (g.tile + JT - 1) / JT * JT;
    g.slots = (int)((g.npad + g.tile - 1) / g.tile);
    g.pm = c->pm.as<double4>();
    g.vel = c->vel.as<double4>();
    g.eps2 = p->eps2;
    g.G = p->G;
    g.c2 = make_pn(p).c2;
    g.part = nullptr;
    return g;
}

static size_t sym_bytes(const SymArgs& g) { return (size_t)g.slots * 3 * g.npad * sizeof(double); }

// Whether an evaluation of all bodies on all bodies takes this path: the
// Newtonian and 1PN laws from SYM_MIN bodies on. Trailing massless bodies
// (n_src < n) stay with the directed kernel, whose source loop leaves them out, as
// do systems for which the partial sums' limit allows too few slots.
bool aster_allpairs_sym_fits(const aster_ctx* c, const aster_params* p) {
    if (pn_level(p) > 1 || c->n < SYM_MIN || c->n_src != c->n) return false;
    const SymArgs g = sym_args(c, p);
    return g.tile == g.set || g.slots >= SYM_SLOTS_MIN;
}

// Room for the partial array. ASTER_ERR_OOM: there is none, and the evaluation
// goes to the directed kernel.
int aster_allpairs_sym_prepare(aster_ctx* c, const aster_params* p) {
    return aster_sums_ensure(c, c->scratch, sym_bytes(sym_args(c, p)));
}

// One evaluation (ASTER_ERR_OOM: nothing was launched), with the closing kick
// and, fuse_next, the next step's opening kick and drift.
int aster_allpairs_sym_launch(aster_ctx* c, const aster_params* p, bool closing_kick, bool fuse_next) {
    ASTER_TRY(aster_allpairs_sym_prepare(c, p));
    SymArgs g = sym_args(c, p);
    g.part = c->scratch.as<double>();
    const int64_t n = c->n;
    const bool small = n < SYM_SMALL;
    if (pn_level(p)) ASTER_TRY(small ? launch_sym<1, 2, 2>(c, g) : launch_sym<1, 4, 4>(c, g));
    else ASTER_TRY(small ? launch_sym<0, 2, 2>(c, g) : launch_sym<0, 8, 4>(c, g));
    k_sym_reduce<<<(unsigned)((n + 63) / 64), 192, 0, c->stream>>>(
        n, g.npad, g.slots, g.part, p->G, c->acc.as<double4>(), closing_kick ? c->vel.as<double4>() : nullptr,
        0.5 * p->dt, closing_kick && fuse_next ? c->pm.as<double4>() : nullptr, p->dt);
    ASTER_CUDA(cudaGetLastError());
    if (closing_kick) c->mixed_valid = false;  // the closing kick moves the velocities
    c->stats.kernels += 2;
    c->stats.interactions += (double)n * (double)n;
    return ASTER_OK;
}
