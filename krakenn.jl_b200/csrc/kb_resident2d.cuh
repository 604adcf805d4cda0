// Many steps of a small cavity in one launch, the populations in registers.
//
// What bounds a small grid is the time between two dependent steps, not its
// traffic: captured launches take 1.87 us per step on 128^2 FP64 whatever the
// kernel does.  Here a thread keeps its node for the whole run.  A block is a
// tile of 64 x 2 nodes; populations that stay in the tile pass through shared
// memory (two slots, one block barrier per step), populations that leave it go
// to the neighbouring thread through L2 as packets that carry the step number
// beside the value.  A reader polls its packet until the number is the step's:
// no fence and no barrier between blocks, one write and one read of L2.
//
// One B200, us per step, captured launches -> this: 32^2 FP64 1.67 -> 1.42,
// 128^2 1.67 -> 1.47, 256^2 2.57 -> 1.79; FP32 1.67 -> 1.27, 1.67 -> 1.42, 2.18
// -> 1.68, 384 x 256 (about the largest that is resident) 2.46 -> 2.02.  Narrow
// grids, FP64: 1 x 512 1.41 -> 1.19, 24 x 512 1.67 -> 1.34, 65 x 300 (tiles of
// 33 nodes) 1.80 -> 1.53, 65 x 512 1.93 -> 1.73, 1024 x 16 1.68 -> 1.50; the
// least gain of 48 grids in both precisions and with both lids is 6 % (65 x 300
// FP32, moving lid).  It wins at every resident size, so that is the rule.
// At 128^2 FP64, tiles of 32 x 4 and 128 x 1 took 4 % longer.
// Packets fetched by warps of their own (20 % longer), or read again by the
// whole row until all are in (25 %), load L2 with more polls and lose; so does
// a pair of thermal lattices, whose step has twice the packets (256 x 64: 2.0 us
// where captured launches take 2.1, 1.9 in FP32 where they take 1.9).
//
// Slot reuse (two slots, step parity): a thread overwrites its packet of step
// s - 2 to node r after it has received r's packet of step s - 1, which r sent
// after it had read the packet of step s - 2 (every link has its reverse).
// Packets are 64-bit words, 32 bits of value and 32 of step number, so a word
// is either old or new.  Blocks wait for one another, so the launch is
// cooperative; a wait that exceeds its limit sets the error flag, and its
// thread and those that see the flag wait no more: every thread still takes
// all its steps, so the launch ends, with void results.
#pragma once
#include "kb_common.cuh"

namespace kb {
namespace d2 {

constexpr int RES_W = 64, RES_H = 2, RES_T = RES_W * RES_H;
constexpr size_t RES_HEADER = 256;  // the error flag, then the packets

__host__ __device__ constexpr int rcx(int q) { return (q == 1 || q == 5 || q == 8) - (q == 3 || q == 6 || q == 7); }
__host__ __device__ constexpr int rcy(int q) { return (q == 2 || q == 5 || q == 6) - (q == 4 || q == 7 || q == 8); }
__host__ __device__ constexpr int ropp(int q) { return q == 0 ? 0 : (q < 5 ? (q + 1) % 4 + 1 : (q - 3) % 4 + 5); }

template <typename T> struct Packet;
template <> struct Packet<double> {
    ulonglong2 w;
    __device__ __forceinline__ void get(const void *p) {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
    }
    __device__ __forceinline__ bool is(unsigned s) const {
        return (unsigned)(w.x >> 32) == s && (unsigned)(w.y >> 32) == s;
    }
    __device__ __forceinline__ double value() const {
        return __hiloint2double((int)(unsigned)w.y, (int)(unsigned)w.x);
    }
    static __device__ __forceinline__ void put(void *p, double v, unsigned s) {
        const unsigned long long t = (unsigned long long)s << 32;
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p),
                     "l"(t | (unsigned)__double2loint(v)), "l"(t | (unsigned)__double2hiint(v))
                     : "memory");
    }
};
template <> struct Packet<float> {
    unsigned long long w;
    __device__ __forceinline__ void get(const void *p) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    }
    __device__ __forceinline__ bool is(unsigned s) const { return (unsigned)(w >> 32) == s; }
    __device__ __forceinline__ float value() const { return __uint_as_float((unsigned)w); }
    static __device__ __forceinline__ void put(void *p, float v, unsigned s) {
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p),
                     "l"((unsigned long long)s << 32 | __float_as_uint(v))
                     : "memory");
    }
};

// State s of the run is left in f[s & 1] for the last two steps; state 0 is
// read from f[0].
template <typename T>
struct CavityRun {
    T *f0, *f1, *rho, *ux, *uy;
    const uint8_t *solid;
    int Nx, Ny, tw;
    unsigned nsteps;
    T omega, u_lid;
    unsigned char *packets;  // [2][8][Nx Ny]
    int *err;
    long long spin;
};

template <typename T, bool MOVING>
__global__ void __launch_bounds__(RES_T) cavity_run_k(const CavityRun<T> R) {
    __shared__ T sh[2][8][RES_T];
    const int lx = threadIdx.x, ly = threadIdx.y, tid = ly * RES_W + lx;
    const int Nx = R.Nx, Ny = R.Ny, x0 = blockIdx.x * R.tw, y0 = blockIdx.y * RES_H;
    const int tw = min(R.tw, Nx - x0), th = min(RES_H, Ny - y0);
    const int i = x0 + lx, j = y0 + ly;
    const bool active = lx < tw && ly < th;
    const size_t P = (size_t)Nx * Ny, c = active ? (size_t)j * Nx + i : 0;
    unsigned wall = 0, away = 0, leave = 0;  // bit q: source beyond a wall / in another tile; target in another tile
#pragma unroll
    for (int q = 1; q < 9; ++q) {
        const int sx = i - rcx(q), sy = j - rcy(q), dx = i + rcx(q), dy = j + rcy(q);
        if (sx < 0 || sx >= Nx || sy < 0 || sy >= Ny) wall |= 1u << q;
        else if (sx < x0 || sx >= x0 + tw || sy < y0 || sy >= y0 + th) away |= 1u << q;
        if (dx >= 0 && dx < Nx && dy >= 0 && dy < Ny && (dx < x0 || dx >= x0 + tw || dy < y0 || dy >= y0 + th))
            leave |= 1u << q;
    }
    T p[9];
    bool solid = false;
    if (active) {
#pragma unroll
        for (int q = 0; q < 9; ++q) p[q] = R.f0[c + q * P];
        solid = R.solid && R.solid[c];
    }
    bool dead = false;
    for (unsigned s = 1; s <= R.nsteps; ++s) {
        const unsigned slot = s & 1u;
        unsigned char *pk = R.packets + (size_t)slot * 8 * P * sizeof(Packet<T>);
        if (active) {
#pragma unroll
            for (int q = 1; q < 9; ++q) {
                if (leave >> q & 1u) Packet<T>::put(pk + ((q - 1) * P + c) * sizeof(Packet<T>), p[q], s);
                sh[slot][q - 1][tid] = p[q];
            }
        }
        __syncthreads();
        if (active) {
            T v[9];
            v[0] = p[0];
#pragma unroll
            for (int q = 1; q < 9; ++q) {
                v[q] = p[ropp(q)];
                if (!((wall | away) >> q & 1u)) v[q] = sh[slot][q - 1][tid - rcy(q) * RES_W - rcx(q)];
            }
            unsigned need = dead ? 0u : away;
            for (long long it = 0; need; ++it) {
                Packet<T> k[9];
#pragma unroll
                for (int q = 1; q < 9; ++q)
                    if (need >> q & 1u)
                        k[q].get(pk + ((q - 1) * P + (size_t)(j - rcy(q)) * Nx + i - rcx(q)) * sizeof(Packet<T>));
#pragma unroll
                for (int q = 1; q < 9; ++q)
                    if ((need >> q & 1u) && k[q].is(s)) {
                        v[q] = k[q].value();
                        need &= ~(1u << q);
                    }
                if (need && (it > R.spin || ((it & 1023) == 1023 && *(volatile int *)R.err))) {
                    atomicExch(R.err, 1);
                    dead = true;
                    break;
                }
            }
#pragma unroll
            for (int q = 0; q < 9; ++q) p[q] = v[q];
            T r, a, b;
            if (MOVING) movingwall_node(p, j == Ny - 1, solid, R.omega, R.u_lid, r, a, b);
            else cavity_node(p, j == Ny - 1, solid, R.omega, R.u_lid);
            if (s + 1 >= R.nsteps) {
                T *o = slot ? R.f1 : R.f0;
#pragma unroll
                for (int q = 0; q < 9; ++q) o[c + q * P] = p[q];
            }
            if (s == R.nsteps) {
                if (!MOVING) macro_node(p, r, a, b);
                R.rho[c] = r; R.ux[c] = a; R.uy[c] = b;
            }
        }
    }
}

// Tiles of a grid, even in x.
inline dim3 cavity_run_grid(int Nx, int Ny, int *tw) {
    const int nx = (Nx + RES_W - 1) / RES_W;
    *tw = (Nx + nx - 1) / nx;
    return dim3((unsigned)((Nx + *tw - 1) / *tw), (unsigned)((Ny + RES_H - 1) / RES_H));
}

// Workspace of a run; 0 where the tiles are not all resident at once.
template <typename T, bool MOVING>
size_t cavity_run_bytes(int Nx, int Ny) {
    int tw, dev = 0, coop = 0, occ = 0;
    const dim3 grid = cavity_run_grid(Nx, Ny, &tw);
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, cavity_run_k<T, MOVING>, RES_T, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (!coop || (long long)grid.x * grid.y > (long long)occ * sm_count()) return 0;
    return RES_HEADER + (size_t)2 * 8 * Nx * Ny * sizeof(Packet<T>);
}

// Rounds of polls in one step before a wait gives up, about a microsecond each.
constexpr long long RES_SPIN = 1ll << 21;

template <typename T, bool MOVING>
int cavity_run(const char *what, CavityRun<T> R, void *workspace, size_t bytes, cudaStream_t s,
               long long spin = RES_SPIN) {
    const size_t need = cavity_run_bytes<T, MOVING>(R.Nx, R.Ny);
    KB_REQUIRE(need > 0, "%s: a %d x %d grid is not resident on the device at once", what, R.Nx, R.Ny);
    KB_REQUIRE(bytes >= need, "%s: workspace of %zu bytes, %zu needed", what, bytes, need);
    if (cudaMemsetAsync(workspace, 0, need, s) != cudaSuccess) return check_launch(what);
    const dim3 grid = cavity_run_grid(R.Nx, R.Ny, &R.tw);
    R.err = (int *)workspace;
    R.packets = (unsigned char *)workspace + RES_HEADER;
    R.spin = spin;
    void *args[] = {&R};
    if (cudaLaunchCooperativeKernel((void *)cavity_run_k<T, MOVING>, grid, dim3(RES_W, RES_H), args, 0, s) !=
        cudaSuccess)
        return check_launch(what);
    return KB_OK;
}

}  // namespace d2
}  // namespace kb
