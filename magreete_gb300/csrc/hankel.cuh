// Hankel functions H0, H1 (first kind) of a real argument in FP64, for the 2D
// Green's functions.
//
// Why not j0 / y0 / j1 / y1: the four calls cost about 150 clocks per argument
// and SM (the FP64 pipe does 1.7 operations a clock), and beyond x = 8 their
// absolute error is up to 5e-12.  Here both functions come from one table of
// local Taylor polynomials, 38 FP64 operations, with errors below 1e-15 of the
// amplitude sqrt(2 / (pi x)).
//
// Table: interval i is [i / 8, (i + 1) / 8), 3 <= x < 512; ten coefficients of
// H0 about its centre.  H1 = -H0' is the derivative of the same polynomial.  The
// coefficients follow from H0, H1 at the centre by the recurrence of Bessel's
// equation x y'' + y' + x y = 0; the centre values by Hankel's asymptotic
// expansion (x >= 25) or by a degree-20 expansion about the nearest of 46 nodes
// (Abramowitz and Stegun, chapter 9).  Below x = 3 CUDA's functions (accurate
// there), beyond 512 three terms of the asymptotic expansion; both are calls,
// because FP64 instructions that are predicated off still take their time.
// Measured (GB300, system assembly, complex128): 2D TE N = 1000, k0 L / 2 pi = 25
// 0.384 -> 0.133 ms; 2D TM N = 3000 1.36 -> 0.43 ms; errors 4.7e-12 -> 7e-15.
//
// The table is device memory of this translation unit, written by
// hankel_fill_kernel on the caller's stream before the kernel that reads it.  A
// block whose entries are complete returns at once, so a repeated call costs
// one empty launch and no host state exists; concurrent first calls write
// the same bits.
#pragma once
#include "common.cuh"
#include "diag.cuh"

namespace mgt {
namespace hk {

constexpr int kDeg = 9;                       // degree of the local polynomials
constexpr int kFirst = 24, kIntervals = 4096; // table: intervals kFirst .. kIntervals - 1 of width 1/8
constexpr double kMinX = kFirst / 8.0, kMaxX = kIntervals / 8.0;
constexpr int kFillThreads = 64;
constexpr int kFillBlocks = kIntervals / kFillThreads;

static __device__ double2 g_table[(size_t)kIntervals * (kDeg + 1)];   // (J0, Y0) coefficients
static __device__ int g_filled[kFillBlocks];

__constant__ const double kNode[46][4] = {
    // J0, Y0, J1, Y1 at 2.5, 3.0, ..., 25.0
    {-0.048383776468198, 0.4980703596152319, 0.49709410246427405, 0.1459181379667858},
    {-0.26005195490193345, 0.3768500100127904, 0.3390589585259365, 0.3246744247918},
    {-0.3801277399872634, 0.1890219439208265, 0.1373775273623272, 0.41018841788751187},
    {-0.39714980986384735, -0.016940739325064992, -0.06604332802354913, 0.3979257105571},
    {-0.32054250898512143, -0.19470500862950454, -0.23106043192337064, 0.3009973230696546},
    {-0.1775967713143383, -0.30851762524903376, -0.32757913759146523, 0.14786314339122683},
    {-0.006843869417819197, -0.339480592881911, -0.34143821542904335, -0.023758238956389618},
    {0.15064525725099692, -0.28819468398157916, -0.27668385812756563, -0.17501034430039825},
    {0.2600946055816064, -0.17324243491898234, -0.15384130140997185, -0.27409127395927546},
    {0.3000792705195556, -0.025949743967209265, -0.004682823482345833, -0.30266723702418485},
    {0.2663396578803784, 0.11731328614820863, 0.1352484275797055, -0.25912851048611624},
    {0.1716508071375539, 0.22352148938756622, 0.23463634685391463, -0.1580604617312475},
    {0.041939251842934504, 0.27020510536578746, 0.2731219636740537, -0.02616867939853747},
    {-0.09033361118287614, 0.24993669828502468, 0.24531178657332528, 0.10431457519671589},
    {-0.19392874768742235, 0.17121062620272384, 0.16126443075752986, 0.20317989938720768},
    {-0.24593576445134835, 0.055671167283599395, 0.04347274616886144, 0.24901542420695388},
    {-0.23664819446234714, -0.0675303724978764, -0.07885001422733148, 0.2337042283572686},
    {-0.1711903004071961, -0.16884732389207954, -0.17678529895672151, 0.16370553741494284},
    {-0.06765394811166522, -0.22523211169118787, -0.22837862066532347, 0.057942547143000823},
    {0.047689310796833535, -0.22523731263436145, -0.2234471044906276, -0.05709921826089652},
    {0.1468840547004211, -0.1712143068446693, -0.16548380461475973, -0.1538382565375012},
    {0.20692610237706782, -0.07820786452787591, -0.07031805212177837, -0.2100814084206935},
    {0.21498916588040082, 0.030077009046785588, 0.03804929208600142, -0.21402293034002892},
    {0.17107347611045867, 0.1271925685821837, 0.13337515469879324, -0.16664484185617226},
    {0.08754486801037623, 0.19030189118784452, 0.19342946359604696, -0.08104209092873875},
    {-0.014224472826780772, 0.20546429603891828, 0.20510403861352275, 0.02107362803687351},
    {-0.10923065090005017, 0.17064491122943462, 0.16721318035174715, 0.11478614251334232},
    {-0.1748990739836292, 0.0958109970807124, 0.09039717566130419, 0.17797516893941687},
    {-0.19638069293686103, 0.00018123245754096657, -0.005764213735631227, 0.19647583778590966},
    {-0.16985425215118355, -0.0926371984423237, -0.09766849275778065, 0.1672050360772337},
    {-0.10311039822868592, -0.16041119250501118, -0.1634199694257549, 0.09857279873421605},
    {-0.013355805721984111, -0.1875521596114106, -0.18799488548806959, 0.008155132278221441},
    {0.0771648214225547, -0.16865634504032312, -0.16663364001001604, -0.08174785849680946},
    {0.1466294396596512, -0.10951969138534148, -0.10570143114240926, -0.1495601138626533},
    {0.17885382704017289, -0.025451742976154466, -0.02087707014809752, -0.1795645668963179},
    {0.16702466434058316, 0.06264059680938383, 0.06683312417585005, -0.1655116143625213},
    {0.11509696025367476, 0.1334095666575905, 0.13625468819339573, -0.11187909834450974},
    {0.036579071000862745, 0.17020175842215576, 0.1711202727639001, -0.03253926075586534},
    {-0.048942043721558054, 0.16494520346148386, 0.16385208254581224, 0.05278910893417191},
    {-0.12065147570486719, 0.11988759780067156, 0.1171777896438517, 0.12340585622650763},
    {-0.1615403170277827, 0.04681853166548836, 0.0432420331907122, 0.1626199829760663},
    {-0.16241278131348655, -0.03598179027370283, -0.03951932188370151, 0.16166920099263313},
    {-0.12392823156027444, -0.10828611769479093, -0.11094614338176333, 0.12165328069026943},
    {-0.056230274166859266, -0.15283402879758778, -0.15403806518312121, 0.05305977612120217},
    {0.0236974337340679, -0.15942871774975043, -0.1589784118193281, -0.026954655331885412},
    {0.09626678327595811, -0.12724943226800614, -0.1253502495802899, -0.09882996478323741},
};

// H0 and H1 by the asymptotic expansion; x >= 25
__device__ __noinline__ inline void hankel_asymptotic(double x, double2* h0, double2* h1) {
  double P[2], Q[2];
#pragma unroll
  for (int nu = 0; nu < 2; ++nu) {
    const double mu = 4.0 * nu;
    double t = 1.0, p = 1.0, q = 0.0;
#pragma unroll 1
    for (int k = 1; k < 24; ++k) {
      const double o = 2.0 * k - 1.0;
      t = t * (mu - o * o) / (8.0 * k * x);
      const double v = (k >> 1) & 1 ? -t : t;
      if (k & 1) q += v;
      else p += v;
    }
    P[nu] = p;
    Q[nu] = q;
  }
  // e^{i (x - pi/4)} = ((c + s) + i (s - c)) / sqrt 2
  double s, c;
  sincos(x, &s, &c);
  const double a = c + s, b = s - c, amp = 1.0 / sqrt(3.14159265358979323846 * x);
  *h0 = make_double2(amp * (a * P[0] - b * Q[0]), amp * (a * Q[0] + b * P[0]));
  *h1 = make_double2(amp * (a * Q[1] + b * P[1]), -amp * (a * P[1] - b * Q[1]));
}

// the same for x >= 512, where three terms of each series are enough
__device__ __noinline__ inline void hankel_far(double x, double2* h0, double2* h1) {
  const double ix = __drcp_rn(x), y = ix * ix;
  const double p0 = fma(y, fma(y, 3675.0 / 32768, -9.0 / 128), 1.0);
  const double q0 = ix * fma(y, fma(y, -59535.0 / 262144, 75.0 / 1024), -0.125);
  const double p1 = fma(y, fma(y, -4725.0 / 32768, 15.0 / 128), 1.0);
  const double q1 = ix * fma(y, fma(y, 72765.0 / 262144, -105.0 / 1024), 0.375);
  double s, c;
  sincos(x, &s, &c);
  const double amp = sqrt(ix * (1.0 / 3.14159265358979323846)), a = amp * (c + s), b = amp * (s - c);
  *h0 = make_double2(a * p0 - b * q0, a * q0 + b * p0);
  *h1 = make_double2(a * q1 + b * p1, b * q1 - a * p1);
}

__device__ __noinline__ inline double2 hankel0_small(double x) { return make_double2(j0(x), y0(x)); }
__device__ __noinline__ inline double2 hankel1_small(double x) { return make_double2(j1(x), y1(x)); }

// Taylor coefficients a[0 .. deg] of a solution of Bessel's equation of order 0 about x
template <int DEG>
__device__ __forceinline__ void taylor(double x, double y, double dy, double* a) {
  a[0] = y;
  a[1] = dy;
#pragma unroll
  for (int k = 0; k + 2 <= DEG; ++k)
    a[k + 2] = -((double)((k + 1) * (k + 1)) * a[k + 1] + x * a[k] + (k ? a[k - 1] : 0.0)) /
               (x * (double)((k + 2) * (k + 1)));
}

static __global__ void __launch_bounds__(kFillThreads) hankel_fill_kernel() {
  if (*(volatile int*)&g_filled[blockIdx.x]) return;
  const int i = blockIdx.x * kFillThreads + threadIdx.x;
  if (i >= kFirst) {
    const double xc = (i + 0.5) / 8.0;
    double2 h0, h1;
    if (xc >= 25.0) {
      hankel_asymptotic(xc, &h0, &h1);
    } else {
      const int n = (int)((xc - 2.5) * 2.0 + 0.5);
      const double xn = 2.5 + 0.5 * n, t = xc - xn;
      double v[2], d[2];
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        double a[21];
        taylor<20>(xn, kNode[n][q], -kNode[n][2 + q], a);
        double p = a[20], dp = 0.0;
#pragma unroll
        for (int k = 19; k >= 0; --k) {
          dp = fma(dp, t, p);
          p = fma(p, t, a[k]);
        }
        v[q] = p;
        d[q] = -dp;
      }
      h0 = make_double2(v[0], v[1]);
      h1 = make_double2(d[0], d[1]);
    }
    double a[kDeg + 1], b[kDeg + 1];
    taylor<kDeg>(xc, h0.x, -h1.x, a);
    taylor<kDeg>(xc, h0.y, -h1.y, b);
#pragma unroll
    for (int k = 0; k <= kDeg; ++k) g_table[(size_t)i * (kDeg + 1) + k] = make_double2(a[k], b[k]);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *(volatile int*)&g_filled[blockIdx.x] = 1;
}

// The table, complete for every kernel launched on `s` from here on.
static inline cudaError_t ensure_table(cudaStream_t s) {
  count_launch();
  hankel_fill_kernel<<<kFillBlocks, kFillThreads, 0, s>>>();
  return cudaGetLastError();
}

// H0(x) and, with NEED1, H1(x); x > 0
template <bool NEED1>
__device__ __forceinline__ void hankel01(double x, double2& h0, double2& h1) {
  if (x >= kMinX && x < kMaxX) {
    const int i = (int)(x * 8.0);
    const double t = x - (i + 0.5) * 0.125;
    const double2* c = g_table + (size_t)i * (kDeg + 1);
    const double2 top = c[kDeg];
    double pr = top.x, pi = top.y, dr = 0.0, di = 0.0;
#pragma unroll
    for (int k = kDeg - 1; k >= 0; --k) {
      const double2 ck = c[k];
      if (k == kDeg - 1) {
        dr = pr;
        di = pi;
      } else {
        dr = fma(dr, t, pr);
        di = fma(di, t, pi);
      }
      pr = fma(pr, t, ck.x);
      pi = fma(pi, t, ck.y);
    }
    h0 = make_double2(pr, pi);
    h1 = make_double2(-dr, -di);
  } else if (x >= kMaxX) {
    hankel_far(x, &h0, &h1);
  } else {
    h0 = hankel0_small(x);
    if (NEED1) h1 = hankel1_small(x);
  }
}

}  // namespace hk
}  // namespace mgt
