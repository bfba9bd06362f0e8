// ptd_tune.cu -- launch-shape choice for the fused kernels.
#include <mutex>

#include "ptd_internal.h"

namespace ptd {

int sm_count()
{
    static std::mutex mu;
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 152;   // only reached when no device is usable; launches then fail anyway
    }
    std::lock_guard<std::mutex> lk(mu);
    if (!cache[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = 152;
        }
        cache[dev] = n;
    }
    return cache[dev];
}

// The z march length of a 3D launch of bxy CTAs per z chunk on `slots`
// resident CTA slots: the longest march (512..16) whose CTA count fills the
// slots in whole waves to >= 90 % (wave quantization), else the best filling
// one.
int z_chunk(long long bxy, int nz, long long slots)
{
    int best = 16;
    double best_eff = -1.0;
    for (int chunk = 512; chunk >= 16; chunk /= 2) {
        const long long nb = bxy * ((nz - 2 + chunk - 1) / chunk);
        const long long waves = (nb + slots - 1) / slots;
        const double eff = (double)nb / (double)(waves * slots);
        if (nb >= slots && eff >= 0.9) return chunk;
        if (eff > best_eff) {
            best_eff = eff;
            best = chunk;
        }
    }
    return best;
}

namespace {

// The march length (rows in 2D, planes in 3D) of a launch: `pref` while
// `units(march)` -- the warps (2D) or CTAs (3D) of the launch -- reaches
// `hi`, halved down to `mid` otherwise; below that halved while fewer than
// `lo` units run.  A march step is a chain of dependent loads and arithmetic
// of about 1 us, so a grid too small to fill the SMs is bound by the march
// length and not by its cells; a shorter march re-evaluates one face per cell
// column and march start.
template <class Units>
int march_length(int pref, int mid, long long hi, long long lo, Units units)
{
    int m = pref;
    while (m > mid && units(m) < hi) m /= 2;
    while (m > 1 && units(m) < lo) m /= 2;
    return m;
}

long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

}  // namespace

// z march of the 16-row FP32 kernels (defect correction, rebased LIN on large
// grids): us per iteration at march 16 and at the march taken: rebased LINSTEP
// 64^3 17.6, 8.1 (4); 96^3 21.3, 17.2 (4); 128^3 35.7, 33.8 (4); 192^3 95.7 (16).
int z_march16(const ptd_params& p)
{
    const long long bxy = ceil_div(p.nx - 2, 31) * ceil_div(p.ny - 2, 15);
    const long long sm = sm_count();
    return march_length(16, 4, 17 * sm / 2, sm, [&](int m) { return bxy * ceil_div(p.nz - 2, m); });
}

// Whether the 3D rebased form runs two cells per lane (rb3d_pair_body): LIN and
// NONLIN grids that are bound by the latency of a plane (the figures are at
// rb3d_pair_body: 110^3 is the largest cube where it is faster, at 128^3 the
// one-cell kernel is).
bool rb3d_pair(int model, long long nx, long long ny, long long nz)
{
    return (model == LIN || model == NONLIN) && nx * ny * nz <= 1500000;
}

// Its march: us per iteration at marches 1, 2, 4, 8, 16: NONLIN 96^3 20.8, 18.5,
// 19.0, 19.2, 25.7; 110^3 30.1, 24.8, 23.6, 21.9, 29.9; LIN 96^3 15.3, 12.8, 12.6,
// 13.0, 18.0.
int z_march_pair(const ptd_params& p)
{
    const long long bxy = ceil_div(p.nx - 2, 62) * ceil_div(p.ny - 2, 7);
    const long long sm = sm_count();
    return march_length(16, 4, 4 * sm, 7 * sm / 4, [&](int m) { return bxy * ceil_div(p.nz - 2, m); });
}

// Rows of a CTA of the 3D rebased form's one-cell kernel: 8 (half the warps per
// barrier), for LIN grids past the L2 cache 16 (less halo).  us per iteration,
// 8 / 16 rows at the best march: NONLIN 128^3 36.2, 37.9; 256x200x180 122, 126;
// 320x255x191 187, 188; LINSTEP 48^3 6.0, 6.6; 128^3 30.3, 33.8; 320x255x191 176,
// 182; 400^3 681, 702; LIN 128^3 24.5, 26.7; 192^3 80.5, 80.3; 320x255x191 155.6,
// 152.2.
int rb3d_rows(int model, long long nx, long long ny, long long nz)
{
    return model == LIN && nx * ny * nz > 2400000 ? 16 : 8;
}

// z march of the 8-row FP32 kernels and of the adjoint, at least per_sm CTAs
// per SM down to a march of one plane.  A gradient of 72^3 over three steps at
// marches 1, 2, 3, 4, 6: rebased 12.1, 11.1, 10.4, 10.4, 10.9 ms (4 is taken);
// FP64 36.7, 34.3, 35.0, 36.2, 38.9 (2; in 16-row CTAs 38.3 at best).
int z_march8(const ptd_params& p, int per_sm)
{
    const long long bxy = ceil_div(p.nx - 2, 31) * ceil_div(p.ny - 2, 7);
    const long long sm = sm_count();
    return march_length(16, 4, 8 * sm, per_sm * sm, [&](int m) { return bxy * ceil_div(p.nz - 2, m); });
}

// March of the rebased form's base kernel (rows in 2D, planes in 3D, per warp
// of 32 cells): us of two rebases, one launch and the step's overhead (about
// 100) at march 32 and at the march taken: 2D NONLIN 256^2 308, 128 (1); 600x500
// 314, 165 (4); 2048^2 925, 830 (8); 4096^2 2907, 2832 (16); 3D NONLIN 50x40x45
// 357, 137 (1); 100x90x80 433, 395 (8); 320x255x191 3865, 3841 (16).
int rb_base_march(const ptd_params& p)
{
    const long long sm = sm_count(), line = ceil_div(p.nx, 32) * (p.ndim == 3 ? p.ny : 1), n = p.ndim == 3 ? p.nz : p.ny;
    return march_length(16, 8, 120 * sm, 15 * sm, [&](int m) { return line * ceil_div(n, m); });
}

LaunchCfg tuned_config(const ptd_params& p)
{
    LaunchCfg c;
    const long long sm = sm_count();
    const bool often = p.nchk < 4;
    if (p.ndim == 2) {
        // short y marches in small CTAs: many independent warps per SM hide
        // the memory latency of the march.  Measured over warps {1,2,4,8} x
        // rows {1..64}, us per iteration of a check block at another march (FP32
        // forms and DFH: the former fixed one) and at the one taken here:
        //   FP64 NONLIN (grids that do not fit the flow kernel) 768x600 15.2
        //     (4); 1024^2 30.6 (16), 26.5 (8); 2048^2 92.9 (8), 93.6 (16);
        //     4096^2 345.8 (8), 340.1 (16), 342.7 (32); LIN and LINSTEP alike
        //   DFH NONLIN (1 x 8) 256^2 12.0, 4.8 (1); 512^2 12.5, 7.8 (2);
        //     1021x1500 29.7, 27.3 (4); 2048^2 62.7 (8)
        //   FP32_RB NONLIN (8 x 32, marches of twice the rows) 256^2 28.9, 4.4
        //     (1); 512^2 30.2, 4.8 (1); 1024^2 30.1, 8.1 (4); 2048^2 48.9,
        //     26.0 (8); 3000^2 61.1, 48.1 (16); 4096^2 78.7 (32)
        //   FP32_RB LINSTEP 1024^2 22.3, 7.2 (4); 2048^2 39.8, 24.6 (8)
        //   FP32_DC NONLIN (2 x 16) 256^2 8.8, 4.7 (1); 512^2 8.7, 5.5 (4);
        //     1024^2 9.2, 8.0 (8)
        const bool coef = p.model == PTD_MODEL_LINSTEP || p.model == PTD_MODEL_NONLIN_EXPM;
        const bool tb = p.nchk % 2 == 0 && !(p.flags & PTD_FLAG_DC_NO_TBLOCK);   // two FP32 iterations per launch
        auto warps = [&](int cols, int rows_per) {
            const long long tiles = ceil_div(p.nx - 2, cols);
            return [&p, tiles, rows_per](int m) { return tiles * ceil_div(p.ny - 2, (long long)rows_per * m); };
        };
        switch (p.precision) {
        case PTD_PREC_FP64:
            c.warps2d = 1;
            c.chunk2d = march_length(16, 8, 52 * sm, 25 * sm / 2, warps(31, 1));
            break;
        case PTD_PREC_DFH:
        case PTD_PREC_DF64:
            c.warps2d = p.precision == PTD_PREC_DFH ? 1 : 2;
            // (with a field and checks every iteration 8 rows sooner: DF64 LINSTEP
            // 1000x1001 27.7 (4), 26.7 (8) us, DFH 34.1, 30.8)
            if (often && coef) c.chunk2d = march_length(8, 8, 52 * sm, 12 * sm, warps(62, 1));
            else c.chunk2d = march_length(8, 4, 52 * sm, 29 * sm / 2, warps(62, 1));
            break;
        case PTD_PREC_FP32_RB:
            if (coef) c.chunk2d = march_length(8, 1, 30 * sm, 30 * sm, warps(tb ? 28 : 31, tb ? 2 : 1));
            else c.chunk2d = march_length(32, 8, 26 * sm, 15 * sm, warps(tb ? 60 : 31, tb ? 2 : 1));
            c.warps2d = c.chunk2d == 32 ? 8 : 2;
            break;
        default:
            c.warps2d = 2;
            c.chunk2d = march_length(16, 8, 52 * sm, 15 * sm, warps(tb ? 28 : 31, 1));
            break;
        }
    } else if (p.ndim == 3 && (p.precision == PTD_PREC_FP32_RB || p.precision == PTD_PREC_FP32_DC)) {
        c.rows3d = 16;
        const bool pair = p.precision == PTD_PREC_FP32_RB && rb3d_pair(p.model, p.nx, p.ny, p.nz);
        const bool rb8 = p.precision == PTD_PREC_FP32_RB && rb3d_rows(p.model, p.nx, p.ny, p.nz) == 8;
        c.chunk3d = pair ? z_march_pair(p) : rb8 ? z_march8(p, 2) : z_march16(p);
        // FP32_DC with checks (nearly) every iteration: a check launch costs by
        // its CTAs.  ms of a step at the march above, at the one taken: LIN
        // 96^3 4.08 (4), 3.76 (8); 130x100x127 6.83 (4), 5.91 (16); 160x150x140
        // 15.4 (4), 14.8 (16); LINSTEP 130x100x127 9.5 (4), 8.4 (16)
        if (p.precision == PTD_PREC_FP32_DC && often) {
            const long long bxy = ceil_div(p.nx - 2, 31) * ceil_div(p.ny - 2, 15);
            c.chunk3d = march_length(16, 16, 0, 3 * sm / 2, [&](int m) { return bxy * ceil_div(p.nz - 2, m); });
        }
    } else if (p.ndim == 3) {
        // The FP64-accuracy forms: 256-thread CTAs of 31 x 7 updated cells.
        // Their per-plane barrier joins half the warps of 512-thread CTAs (31
        // x 15 cells) and their tiles waste less of a ragged grid; the larger
        // halo is not what bounds them.  us per iteration, 16 rows x best
        // march / as taken: FP64 NONLIN 128^3 96.6, 88.4 (4 planes); 256^3
        // 596, 562 (16); 512^3 4317, 4079 (32); LIN 512^3 3904, 3901; LINSTEP
        // 512^3 4881, 4496 (32); DF64 LIN 128^3 42.0, 38.9; NONLIN 512^3 2128,
        // 2142 (32); DFH 512^3 2762, 2726 (32).
        c.rows3d = 8;
        const long long bxy = ceil_div(p.nx - 2, 31) * ceil_div(p.ny - 2, 7);
        auto ctas = [&](int m) { return bxy * ceil_div(p.nz - 2, m); };
        // below 4 planes the line is where a shorter march no longer paid: FP64
        // 66^3 at 4, 2 planes 22.0, 21.0 (480, 960 CTAs), 80^3 27.6, 26.3
        // (720, 1440), 96^3 44.0, 43.2 (1344, 2632); DFH 62x72x66 13.3, 11.7
        // (320, 640), 80^3 19.3, 19.4
        const long long lo = (p.precision == PTD_PREC_FP64 ? 5 : 3) * sm;
        c.chunk3d = ctas(32) >= 52 * sm ? 32 : march_length(16, 4, 16 * sm, lo, ctas);
    }
    return c;
}

}  // namespace ptd
