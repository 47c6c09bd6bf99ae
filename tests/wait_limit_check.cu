// A sweep whose upstream columns never come ends with its error flag raised.
//
// The main sweep and an extra sweep of a small grid, on a block list without
// the first block, so that its neighbours wait for values (words) that nobody
// writes, with a limit of some thousand polls instead of a million.  The
// kernel has to return, with error bit 16, without a write before or behind
// the field, and in the main sweep with every listed node written; with the
// whole list there is no error.
//
//   nvcc -gencode arch=compute_103a,code=sm_103a -std=c++17 --expt-relaxed-constexpr -fmad=false
//        -DFM_WAIT_POLLS=4096 wait_limit_check.cu -o check && ./check
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../parallel-fast-marching-method_gb300/csrc/front.cuh"

namespace {

using namespace fm3dt;

constexpr int NR = 37, NX = 13, NZ = 19, NEV = 2, SX = 4, SZ = 8;
constexpr int NBX = (NX + SX - 1) / SX, NBZ = (NZ + SZ - 1) / SZ, NB = NBX * NBZ;
constexpr size_t LAYER = (size_t)NX * NZ, N = LAYER * NR;

template <typename T>
T *managed(size_t n)
{
    T *p = nullptr;
    if (cudaMallocManaged(&p, n * sizeof(T)) != cudaSuccess) std::exit(3);
    std::memset((void *)p, 0, n * sizeof(T));
    return p;
}

template <typename R>
struct Setup {
    R *buf = managed<R>((NEV + 2) * N), *T = buf + N;      // guards of an event either side
    R *s = managed<R>(N), *hx = managed<R>(NR), *wx = managed<R>(NR), *hz = managed<R>(NR * NX), *wz = managed<R>(NR * NX);
    uint8_t *frozen = managed<uint8_t>(NEV * LAYER);
    int *blocks = managed<int>(NB), *dir = managed<int>(NEV), *err = managed<int>(1);
    unsigned *next = managed<unsigned>(1), *act = managed<unsigned>(2 * NEV * NB);
    unsigned long long *prog = managed<unsigned long long>(NEV * NB);
    FieldArgs<R> f{};

    Setup()
    {
        for (size_t i = 0; i < N; ++i) s[i] = R(0.2);
        for (int i = 0; i < NR; ++i) hx[i] = R(5), wx[i] = R(1) / R(25);
        for (int i = 0; i < NR * NX; ++i) hz[i] = R(5), wz[i] = R(1) / R(25);
        std::memset(frozen, 1, NEV * LAYER);
        int n = 0;
        for (int h = 0; h < NBX + NBZ - 1; ++h)
            for (int b = 0; b < NBX; ++b)
                if (h - b >= 0 && h - b < NBZ) blocks[n++] = (b << 12) | (h - b);
        f.T = T; f.s = s; f.hx = hx; f.wx = wx; f.hz = hz; f.wz = wz; f.hr = R(5); f.wr = R(1) / R(25);
        f.frozen = frozen; f.nnr = NR; f.nnx = NX; f.nnz = NZ; f.order2 = 1;
    }
    // the field: ones (unwritten), or a plane wave's times; a plane wave at the
    // bottom; dir: the wave's
    void reset(bool unwritten)
    {
        for (size_t i = 0; i < (NEV + 2) * N; ++i) buf[i] = R(1e6);
        if (unwritten) std::memset((void *)T, 0xff, NEV * N * sizeof(R));
        for (int e = 0; e < NEV; ++e) {
            dir[e] = e ? 0 : 3;
            for (int r = unwritten ? NR - 1 : 0; r < NR; ++r)
                for (int x = 0; x < NX; ++x)
                    for (int z = 0; z < NZ; ++z) {
                        const int d = e ? NX - 1 - x + NZ - 1 - z : x + z;
                        T[e * N + r * LAYER + (size_t)x * NZ + z] = R(0.4) * d + R(0.8) * (NR - 1 - r);
                    }
        }
        *err = 0;
        *next = 0;
        std::memset(prog, 0, NEV * NB * sizeof *prog);
        std::memset(act, 0, 2 * NEV * NB * sizeof *act);
    }
    template <typename A>
    void fill(A &a, int first)
    {
        a.f = f;
        a.blocks = blocks + first;
        a.nblocks = NB - first;
        a.dir = dir;
        a.nev = NEV;
        a.group = NEV;
        a.nbx = NBX;
        a.nbz = NBZ;
        a.count = (unsigned)(NB - first) * NEV;
        a.next = next;
        a.err = err;
    }
    bool guards() const
    {
        for (size_t i = 0; i < N; ++i)
            if (buf[i] != R(1e6) || buf[(NEV + 1) * N + i] != R(1e6)) return false;
        return true;
    }
    // nodes still unwritten: none, or the first block's (its columns, in the
    // event's direction) above the bottom layer
    bool written(bool first_left_out) const
    {
        for (int e = 0; e < NEV; ++e)
            for (size_t i = 0; i < N; ++i) {
                const int r = (int)(i / LAYER), x = (int)(i % LAYER) / NZ, z = (int)(i % NZ);
                const bool up = dir[e] & 1;
                const int bx = up ? x / SX : NBX - 1 - x / SX, bz = up ? z / SZ : NBZ - 1 - z / SZ;
                const bool left = first_left_out && bx == 0 && bz == 0 && r < NR - 1;
                const R v = T[e * N + i];
                if ((v != v) != left) return false;
            }
        return true;
    }
};

int finish(const char *what, int first, int err, bool ok)
{
    const cudaError_t e = cudaGetLastError();
    const bool good = e == cudaSuccess && ok && err == (first ? 16 : 0);
    std::printf("%s, %s: %s, error flag %d, %s\n", what, first ? "first block left out" : "whole list", cudaGetErrorString(e), err,
                good ? "ok" : "FAILED");
    return good ? 0 : 1;
}

template <typename R>
int run()
{
    Setup<R> u;
    int bad = 0;
    for (int first = 0; first < 2; ++first) {
        for (int skew = 0; skew < 2; ++skew) {
            u.reset(true);
            FrontArgs<R> a{};
            u.fill(a, first);
            a.skew = skew;
            launch_front<R, SX, SZ>(a, 0);
            if (cudaDeviceSynchronize() != cudaSuccess) return finish("main sweep", first, -1, false);
            bad += finish(skew ? "main sweep, skewed" : "main sweep", first, *u.err, u.guards() && u.written(first));
        }
        // every step, and only where something changed (nothing did)
        for (int track = 0; track < 2; ++track) {
            u.reset(false);
            StreamArgs<R> a{};
            u.fill(a, first);
            a.prog = u.prog;
            a.act_shift = 2;
            if (track) {
                a.act_cur = u.act;
                a.act_prev = u.act + NEV * NB;
            }
            StreamKernels<R, SX, SZ>::sweep((int)a.count, a, 0);
            if (cudaDeviceSynchronize() != cudaSuccess) return finish("extra sweep", first, -1, false);
            bad += finish(track ? "extra sweep, tracked" : "extra sweep", first, *u.err, u.guards());
        }
    }
    return bad;
}

}  // namespace

int main()
{
    return run<float>() + run<double>() == 0 ? 0 : 1;
}
