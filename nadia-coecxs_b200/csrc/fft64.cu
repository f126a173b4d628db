// fft64.cu -- plans, twiddles and launch shapes of the FP64 transforms.
#include "fft64.h"

#include <algorithm>

namespace nadia {
namespace plain {

// the kernels, one file per length (powers of two) or tile width (any length)
#define NADIA_P2(N)                                                                              \
    bool rows_p2_##N(int L, RowMode mode, bool fwd, const Fft64Args &A, cudaStream_t st);        \
    bool cols_p2_##N(int L, ColMode mode, bool fwd, const Fft64Args &A, cudaStream_t st);
NADIA_P2(64)
NADIA_P2(128)
NADIA_P2(256)
NADIA_P2(512)
NADIA_P2(1024)
NADIA_P2(2048)
NADIA_P2(4096)
#undef NADIA_P2
#define NADIA_ANY(L)                                                                             \
    void rows_any##L(RowMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p, int threads, \
                     size_t smem, cudaStream_t st);                                                           \
    void cols_any##L(ColMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p, int threads, \
                     size_t smem, cudaStream_t st);
NADIA_ANY(1)
NADIA_ANY(2)
NADIA_ANY(4)
NADIA_ANY(8)
#undef NADIA_ANY

bool launch_rows_p2(int N, int L, RowMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (N) {
    case 64: return rows_p2_64(L, mode, fwd, A, st);
    case 128: return rows_p2_128(L, mode, fwd, A, st);
    case 256: return rows_p2_256(L, mode, fwd, A, st);
    case 512: return rows_p2_512(L, mode, fwd, A, st);
    case 1024: return rows_p2_1024(L, mode, fwd, A, st);
    case 2048: return rows_p2_2048(L, mode, fwd, A, st);
    case 4096: return rows_p2_4096(L, mode, fwd, A, st);
    default: return false;
    }
}

bool launch_cols_p2(int N, int L, ColMode mode, bool fwd, const Fft64Args &A, cudaStream_t st)
{
    switch (N) {
    case 64: return cols_p2_64(L, mode, fwd, A, st);
    case 128: return cols_p2_128(L, mode, fwd, A, st);
    case 256: return cols_p2_256(L, mode, fwd, A, st);
    case 512: return cols_p2_512(L, mode, fwd, A, st);
    case 1024: return cols_p2_1024(L, mode, fwd, A, st);
    case 2048: return cols_p2_2048(L, mode, fwd, A, st);
    case 4096: return cols_p2_4096(L, mode, fwd, A, st);
    default: return false;
    }
}

void launch_rows_any(int L, RowMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
                     int threads, size_t smem, cudaStream_t st)
{
    (L == 1 ? rows_any1 : L == 2 ? rows_any2 : L == 4 ? rows_any4 : rows_any8)(
        mode, fwd, A, p, threads, smem, st);
}

void launch_cols_any(int L, ColMode mode, bool fwd, const Fft64Args &A, const Fft64Plan &p,
                     int threads, size_t smem, cudaStream_t st)
{
    (L == 1 ? cols_any1 : L == 2 ? cols_any2 : L == 4 ? cols_any4 : cols_any8)(
        mode, fwd, A, p, threads, smem, st);
}

namespace {
constexpr size_t kSmemMax = 227 * 1024;

// two neighbouring radices whose passes one thread can do on its registers
bool joinable(int a, int b)
{
    return (a == 2 && (b == 3 || b == 5)) || (a == 3 && b == 3);
}
} // namespace

void Fft64Axis::init(int n)
{
    const FftPlan f = make_plan(n);
    const std::vector<double2> W = twiddles(n);
    std::vector<double2> t;
    plan = Fft64Plan{};
    plan.n = n;
    max_prime = 0;
    int Ns = 1;
    auto twiddle = [&](int R, int span) { // W[k * r * n / (span * R)], r = 1 .. R-1, k < span
        const int at = (int)t.size(), step = n / (span * R);
        if (span > 1)
            for (int r = 1; r < R; ++r)
                for (int k = 0; k < span; ++k) t.push_back(W[(size_t)k * r * step]);
        return at;
    };
    std::vector<std::pair<int *, int>> primes;
    for (int i = 0; i < f.np; ) {
        NADIA_REQUIRE(plan.np < kMaxSuper, NADIA_ERR_INVALID, "transform plan too long");
        Fft64Pass &s = plan.pass[plan.np++];
        s.r1 = f.radix[i++];
        s.r2 = 1;
        s.Ns = Ns;
        if (i < f.np && joinable(s.r1, f.radix[i])) s.r2 = f.radix[i++];
        s.tw1 = twiddle(s.r1, Ns);
        s.tw2 = s.r2 > 1 ? twiddle(s.r2, Ns * s.r1) : 0;
        s.wq1 = s.wq2 = 0;
        if (s.r1 & 1) primes.push_back({&s.wq1, s.r1});
        if (s.r2 & 1 && s.r2 > 1) primes.push_back({&s.wq2, s.r2});
        if (s.r1 > 7) max_prime = std::max(max_prime, s.r1 & 1 ? s.r1 : 0);
        s.dNs = FastDiv((unsigned)Ns);
        Ns *= s.r1 * s.r2;
        s.dm = FastDiv((unsigned)(n / (s.r1 * s.r2)));
    }
    for (auto &p : primes) { // W[t * n / R]
        *p.first = (int)t.size();
        for (int k = 0; k < p.second; ++k) t.push_back(W[(size_t)k * (n / p.second)]);
    }
    const int r0 = plan.np > 0 ? plan.pass[0].r1 * plan.pass[0].r2 : 0;
    plan.swz = r0 == 8 ? 3 : r0 == 4 ? 2 : 31;
    plan.prime_sm = 1;
    p2 = n >= 64 && n <= 4096 && (n & (n - 1)) == 0;
    if (smem_any(1) > kSmemMax) plan.prime_sm = 0; // the longest lines
    NADIA_REQUIRE(smem_any(1) <= kSmemMax, NADIA_ERR_INVALID, "grid too large for the FP64 transform");
    if (t.empty()) t.push_back(make_double2(1.0, 0.0));
    tw.alloc(t.size());
    upload_now(tw.p, t.data(), tw.bytes());
}

size_t Fft64Axis::smem_any(int L) const
{
    // never less than the error sums' scratch
    return std::max<size_t>(2 * (size_t)any_values(plan.n, L, plan.swz) +
                                (plan.prime_sm ? max_prime : 0), 64) * sizeof(double2);
}

int Fft64Axis::tile_p2(int count, bool cols) const
{
    int L;
    switch (plan.n) {
    case 64: L = 4; break;
    case 128: L = 4; break;
    case 256: case 512: case 1024: L = 4; break;
    case 2048: L = 2; break;
    default: L = cols ? 2 : 1;
    }
    const int least = plan.n <= 128 ? 4 : cols ? 2 : 1;
    // wide column tiles use whole lines, so they give way only to leave no SM idle
    while (L > least && (count + L - 1) / L < (cols ? 148 : 296)) L /= 2;
    return L;
}

// Signals and threads to a block of the any-length kernels: the pair with the
// least estimated time (in cycles; weights fitted to measurements of all pairs at
// five sizes on B200, where the pair taken is within 4% of the best one) for `count` signals.  A block's time is a latency per
// pass and round (a barrier and a trip through shared memory) plus the rounds'
// work; an SM runs as many blocks as its registers and shared memory hold.
void Fft64Axis::shape_any(int count, bool cols, int *Lout, int *threads) const
{
    double best = 1e300;
    for (int L = 1; L <= 8; L *= 2) {
        const size_t smem = smem_any(L);
        if (smem > kSmemMax) break;
        if (cols && L == 1 && smem_any(2) <= kSmemMax) continue; // half-used sectors
        for (int nt = 64; nt <= kAnyMaxThreads; nt += 32) {
            const int tiles = (count + L - 1) / L;
            int held = std::min({65536 / (kAnyRegisters * nt), (int)((size_t)kAnyCarveKB * 1024 / (smem + 1024)), 32});
            held = std::max(1, std::min(held, (tiles + 147) / 148));
            const int waves = (tiles + 148 * held - 1) / (148 * held);
            double t = 2000 + 2.0 * ((L * plan.n + nt - 1) / nt) * 40; // load and store
            double work = 0; // issue slots of the block's warps
            for (int i = 0; i < plan.np; ++i) {
                const int R = plan.pass[i].r1 * plan.pass[i].r2, m = plan.n / R;
                const bool prime = plan.pass[i].r1 > 8;
                const int items = prime ? (R + 3) / 4 * L * m : L * m;
                const int rounds = (items + nt - 1) / nt;
                t += 400 + rounds * (200 + R * (prime ? 130.0 : 25.0));
                work += prime ? (items + 31) / 32 * R * 64.0 : rounds * (nt / 32) * R * 30.0;
            }
            // four schedulers share the work of the blocks an SM holds
            const double time = waves * std::max(t, held * work / 4);
            if (time < best) {
                best = time;
                *Lout = L;
                *threads = nt;
            }
        }
    }
}

void Fft2d::init(int nx_, int ny_)
{
    nx = nx_;
    ny = ny_;
    X.init(nx);
    Y.init(ny);
}

int Fft2d::rows(RowMode mode, bool forward, Fft64Args A, cudaStream_t s) const
{
    A.nx = nx;
    A.ny = ny;
    A.tw = Y.tw.p;
    int L = Y.p2 ? Y.tile_p2(A.count, false) : 0;
    if (!(L && launch_rows_p2(ny, L, mode, forward, A, s))) {
        int nt;
        Y.shape_any(A.count, false, &L, &nt);
        launch_rows_any(L, mode, forward, A, Y.plan, nt, Y.smem_any(L), s);
    }
    NADIA_CUDA(cudaGetLastError());
    return (A.count + L - 1) / L;
}

int Fft2d::cols(ColMode mode, bool forward, Fft64Args A, cudaStream_t s) const
{
    A.nx = nx;
    A.ny = ny;
    A.tw = X.tw.p;
    if (A.hi == 0) A.hi = nx;
    const bool whole = A.lo == 0 && A.hi == nx;
    int L = X.p2 && whole ? X.tile_p2(A.count, true) : 0;
    if (!(L && launch_cols_p2(nx, L, mode, forward, A, s))) {
        int nt;
        X.shape_any(A.count, true, &L, &nt);
        launch_cols_any(L, mode, forward, A, X.plan, nt, X.smem_any(L), s);
    }
    NADIA_CUDA(cudaGetLastError());
    return (A.count + L - 1) / L;
}

void Fft2d::exec(double2 *a, bool forward, cudaStream_t s) const
{
    Fft64Args A;
    A.src = a;
    A.dst = a;
    A.count = nx;
    rows(R_PLAIN, forward, A, s);
    A.count = ny;
    cols(C_PLAIN, forward, A, s);
}

} // namespace plain
} // namespace nadia
