// gw_log.cuh -- FP64 logarithm of the Barlow-Beeston bin term.
//
// GB300 issues a warp of FP64 operations every 16 cycles per SM, so the term's
// operation count is its time.  This is the table-driven method of Tang (ACM
// TOMS 16, 1990) with a tabulated reciprocal: x = 2^e m, m in [0.703, 1.414);
// c_j ~ 1 / m of the 128 intervals of m; r = m c_j - 1, |r| < 2^-7, and
//   log x = e ln 2 - log c_j + log1p(r),
// the last by its series to r^8.  The c_j are multiples of 2^-7 (m < 1) or 2^-8,
// so that r is exact, and 1 in the two intervals at m = 1, so that there the series
// is all of it and the error stays relative down to x = 1.  ln 2 and -log c_j are
// split so that their leading sum H (multiples of 2^-42 below 2^11) is exact, and
// H + r keeps its rounding error (Dekker's sum, |H| >= |r| or H = 0).  What is left
// to round is the last addition: at most 0.517 ulp over all exponents and down to
// x = 1 (28M arguments against 113-bit logarithms; CUDA's log 0.551).  17 FP64
// operations.
#pragma once
#include <cmath>

namespace gw {
namespace {

struct LogEntry {
  double c, hi, lo;  // c_j, -log c_j = hi + lo
};

__device__ const LogEntry kLogTable[128] = {
    {0x1.6a0p+0, -0x1.62c82f2b9c000p-2, -0x1.e54bdbd7c8a98p-44},
    {0x1.680p+0, -0x1.5d1bdbf581000p-2, 0x1.8d6bdc9c7c238p-44},
    {0x1.660p+0, -0x1.5767717456000p-2, 0x1.64ead9524d7cap-44},
    {0x1.640p+0, -0x1.51aad872e0000p-2, 0x1.f4bd8db0a7cc1p-44},
    {0x1.620p+0, -0x1.4be5f95778000p-2, 0x1.d7c92cd9ad824p-44},
    {0x1.600p+0, -0x1.4618bc21c6000p-2, 0x1.3d82f484c84ccp-46},
    {0x1.5e0p+0, -0x1.404308686a000p-2, -0x1.f8ef43049f7d3p-44},
    {0x1.5c0p+0, -0x1.3a64c55694000p-2, -0x1.7a71cbcd735d0p-44},
    {0x1.5a0p+0, -0x1.347dd9a988000p-2, 0x1.5594dd4c58092p-45},
    {0x1.580p+0, -0x1.2e8e2bae12000p-2, 0x1.67b1e99b72bd8p-45},
    {0x1.560p+0, -0x1.2895a13de8000p-2, -0x1.a8d7ad24c13f0p-44},
    {0x1.540p+0, -0x1.22941fbcf8000p-2, 0x1.a6976f5eb0963p-44},
    {0x1.520p+0, -0x1.1c898c169a000p-2, 0x1.81410e5c62affp-44},
    {0x1.500p+0, -0x1.1675cababa000p-2, -0x1.8380e731f55c4p-44},
    {0x1.500p+0, -0x1.1675cababa000p-2, -0x1.8380e731f55c4p-44},
    {0x1.4e0p+0, -0x1.1058bf9ae5000p-2, 0x1.4ab9d817d52cdp-44},
    {0x1.4c0p+0, -0x1.0a324e2739000p-2, -0x1.c6bee7ef4030ep-47},
    {0x1.4a0p+0, -0x1.0402594b4d000p-2, -0x1.036b89ef42d7fp-48},
    {0x1.480p+0, -0x1.fb9186d5e4000p-3, 0x1.d572aab993c87p-47},
    {0x1.460p+0, -0x1.ef0adcbdc6000p-3, 0x1.b26b79c86af24p-45},
    {0x1.460p+0, -0x1.ef0adcbdc6000p-3, 0x1.b26b79c86af24p-45},
    {0x1.440p+0, -0x1.e27076e2b0000p-3, 0x1.a342c2af0003cp-44},
    {0x1.420p+0, -0x1.d5c216b4fc000p-3, 0x1.1ba91bbca681bp-45},
    {0x1.400p+0, -0x1.c8ff7c79aa000p-3, 0x1.7794f689f8434p-45},
    {0x1.3e0p+0, -0x1.bc286742d8000p-3, -0x1.9ac53f39d121cp-44},
    {0x1.3e0p+0, -0x1.bc286742d8000p-3, -0x1.9ac53f39d121cp-44},
    {0x1.3c0p+0, -0x1.af3c94e80c000p-3, 0x1.a4e633fcd9066p-52},
    {0x1.3a0p+0, -0x1.a23bc1fe2c000p-3, 0x1.539cd91dc9f0bp-44},
    {0x1.380p+0, -0x1.9525a9cf46000p-3, 0x1.297137d9f158fp-44},
    {0x1.380p+0, -0x1.9525a9cf46000p-3, 0x1.297137d9f158fp-44},
    {0x1.360p+0, -0x1.87fa06520c000p-3, -0x1.22120401202fcp-44},
    {0x1.340p+0, -0x1.7ab890210e000p-3, 0x1.bdb9072534a58p-45},
    {0x1.320p+0, -0x1.6d60fe719e000p-3, 0x1.bc6e557134767p-44},
    {0x1.320p+0, -0x1.6d60fe719e000p-3, 0x1.bc6e557134767p-44},
    {0x1.300p+0, -0x1.5ff3070a7a000p-3, 0x1.8586f183bebf2p-44},
    {0x1.2e0p+0, -0x1.526e5e3a1c000p-3, 0x1.790ba37fc5238p-44},
    {0x1.2e0p+0, -0x1.526e5e3a1c000p-3, 0x1.790ba37fc5238p-44},
    {0x1.2c0p+0, -0x1.44d2b6ccb8000p-3, 0x1.70cc16135783cp-46},
    {0x1.2a0p+0, -0x1.371fc201e8000p-3, -0x1.ee8779b2d8abcp-44},
    {0x1.2a0p+0, -0x1.371fc201e8000p-3, -0x1.ee8779b2d8abcp-44},
    {0x1.280p+0, -0x1.29552f8200000p-3, 0x1.5b967f4471dfcp-44},
    {0x1.260p+0, -0x1.1b72ad52f6000p-3, -0x1.e80a41811a396p-45},
    {0x1.260p+0, -0x1.1b72ad52f6000p-3, -0x1.e80a41811a396p-45},
    {0x1.240p+0, -0x1.0d77e7cd08000p-3, -0x1.cb2cd2ee2f482p-44},
    {0x1.220p+0, -0x1.fec9131dc0000p-4, 0x1.54555d1ae6607p-44},
    {0x1.220p+0, -0x1.fec9131dc0000p-4, 0x1.54555d1ae6607p-44},
    {0x1.200p+0, -0x1.e27076e2b0000p-4, 0x1.a342c2af0003cp-45},
    {0x1.1e0p+0, -0x1.c5e548f5bc000p-4, -0x1.d0c57585fbe06p-46},
    {0x1.1e0p+0, -0x1.c5e548f5bc000p-4, -0x1.d0c57585fbe06p-46},
    {0x1.1c0p+0, -0x1.a926d3a4ac000p-4, -0x1.563650bd22a9cp-44},
    {0x1.1c0p+0, -0x1.a926d3a4ac000p-4, -0x1.563650bd22a9cp-44},
    {0x1.1a0p+0, -0x1.8c345d6318000p-4, -0x1.b20f5acb42a66p-44},
    {0x1.180p+0, -0x1.6f0d28ae58000p-4, 0x1.4b4641b664613p-44},
    {0x1.180p+0, -0x1.6f0d28ae58000p-4, 0x1.4b4641b664613p-44},
    {0x1.160p+0, -0x1.51b073f060000p-4, -0x1.83f69278e686ap-44},
    {0x1.160p+0, -0x1.51b073f060000p-4, -0x1.83f69278e686ap-44},
    {0x1.140p+0, -0x1.341d7961bc000p-4, -0x1.1d09299837610p-44},
    {0x1.120p+0, -0x1.16536eea38000p-4, 0x1.47c5e768fa309p-46},
    {0x1.120p+0, -0x1.16536eea38000p-4, 0x1.47c5e768fa309p-46},
    {0x1.100p+0, -0x1.f0a30c0118000p-5, 0x1.d599e83368e91p-45},
    {0x1.100p+0, -0x1.f0a30c0118000p-5, 0x1.d599e83368e91p-45},
    {0x1.0e0p+0, -0x1.b42dd71198000p-5, 0x1.c827ae5d6704cp-46},
    {0x1.0e0p+0, -0x1.b42dd71198000p-5, 0x1.c827ae5d6704cp-46},
    {0x1.0c0p+0, -0x1.77458f6330000p-5, 0x1.181dce586af09p-44},
    {0x1.0a0p+0, -0x1.39e87b9fe8000p-5, -0x1.eafd480ad9015p-44},
    {0x1.0a0p+0, -0x1.39e87b9fe8000p-5, -0x1.eafd480ad9015p-44},
    {0x1.080p+0, -0x1.f829b0e780000p-6, -0x1.980267c7e09e4p-45},
    {0x1.080p+0, -0x1.f829b0e780000p-6, -0x1.980267c7e09e4p-45},
    {0x1.060p+0, -0x1.7b91b07d60000p-6, 0x1.3b955b602ace4p-44},
    {0x1.060p+0, -0x1.7b91b07d60000p-6, 0x1.3b955b602ace4p-44},
    {0x1.040p+0, -0x1.fc0a8b0fc0000p-7, -0x1.f1e7cf6d3a69cp-50},
    {0x1.040p+0, -0x1.fc0a8b0fc0000p-7, -0x1.f1e7cf6d3a69cp-50},
    {0x1.020p+0, -0x1.fe02a6b100000p-8, -0x1.9e23f0dda40e4p-46},
    {0x1.020p+0, -0x1.fe02a6b100000p-8, -0x1.9e23f0dda40e4p-46},
    {0x1.000p+0, 0.0, 0.0},
    {0x1.000p+0, 0.0, 0.0},
    {0x1.fa0p-1, 0x1.82448a3880000p-7, 0x1.4554412c584e0p-44},
    {0x1.f60p-1, 0x1.432a925980000p-6, 0x1.98139928637fep-47},
    {0x1.f20p-1, 0x1.c63d2ec150000p-6, -0x1.5439ce030a687p-44},
    {0x1.ee0p-1, 0x1.252f32f8d0000p-5, 0x1.83e9ae021b67bp-45},
    {0x1.ea0p-1, 0x1.67c94f2d48000p-5, 0x1.dac20827cca0cp-44},
    {0x1.e80p-1, 0x1.894aa149f8000p-5, 0x1.9a19a8be97661p-44},
    {0x1.e40p-1, 0x1.ccb73cddd8000p-5, 0x1.965c36e09f5fep-44},
    {0x1.e00p-1, 0x1.08598b59e4000p-4, -0x1.7e5dd7009902cp-46},
    {0x1.dc0p-1, 0x1.2aa04a4470000p-4, 0x1.7a48ba8b1cb41p-44},
    {0x1.da0p-1, 0x1.3bdf5a7d20000p-4, -0x1.19bd0ad125895p-44},
    {0x1.d60p-1, 0x1.5e95a4d978000p-4, 0x1.1cb7ce1d17171p-44},
    {0x1.d20p-1, 0x1.8197e2f410000p-4, -0x1.c0fe460d20041p-44},
    {0x1.d00p-1, 0x1.9335e5d594000p-4, 0x1.3115c3abd47dap-45},
    {0x1.cc0p-1, 0x1.b6ac88dad4000p-4, 0x1.b1bdff50225c7p-44},
    {0x1.c80p-1, 0x1.da72763844000p-4, 0x1.a89401fa71733p-46},
    {0x1.c60p-1, 0x1.ec739830a0000p-4, 0x1.11fcba80cdd10p-44},
    {0x1.c20p-1, 0x1.08598b59e4000p-3, -0x1.7e5dd7009902cp-45},
    {0x1.c00p-1, 0x1.1178e8227e000p-3, 0x1.1ef78ce2d07f2p-45},
    {0x1.bc0p-1, 0x1.23d712a49c000p-3, 0x1.00d238fd3df5cp-46},
    {0x1.ba0p-1, 0x1.2d1610c868000p-3, 0x1.39d6ccb81b4a1p-47},
    {0x1.b60p-1, 0x1.3fb45a5992000p-3, 0x1.19713c0cae559p-44},
    {0x1.b40p-1, 0x1.4913d8333c000p-3, -0x1.53e43558124c4p-44},
    {0x1.b00p-1, 0x1.5bf406b544000p-3, -0x1.27023eb68981cp-46},
    {0x1.ae0p-1, 0x1.6574ebe8c2000p-3, -0x1.98c1d34f0f462p-44},
    {0x1.aa0p-1, 0x1.7898d85444000p-3, 0x1.8e67be3dbaf3fp-44},
    {0x1.a80p-1, 0x1.823c16551a000p-3, 0x1.e0ddb9a631e83p-46},
    {0x1.a60p-1, 0x1.8beafeb390000p-3, -0x1.73d54aae92cd1p-47},
    {0x1.a20p-1, 0x1.9f6c40708a000p-3, -0x1.337d94bcd3f43p-44},
    {0x1.a00p-1, 0x1.a93ed3c8ae000p-3, -0x1.8724350562169p-45},
    {0x1.9e0p-1, 0x1.b31d8575bc000p-3, 0x1.c794e562a63cbp-44},
    {0x1.9a0p-1, 0x1.c6ffbc6f00000p-3, 0x1.ee138d3a69d43p-44},
    {0x1.980p-1, 0x1.d1037f2656000p-3, -0x1.84a7e75b6f6e4p-47},
    {0x1.960p-1, 0x1.db13db0d48000p-3, 0x1.2806a847527e6p-44},
    {0x1.940p-1, 0x1.e530effe72000p-3, -0x1.fdbdbb13f7c18p-44},
    {0x1.900p-1, 0x1.f991c6cb3c000p-3, -0x1.90d04cd7cc834p-44},
    {0x1.8e0p-1, 0x1.01eae5626c000p-2, 0x1.a43dcfade85aep-44},
    {0x1.8c0p-1, 0x1.07138604d6000p-2, -0x1.e76324e912b17p-44},
    {0x1.8a0p-1, 0x1.0c42d67616000p-2, 0x1.7188b163ceae9p-45},
    {0x1.880p-1, 0x1.1178e8227e000p-2, 0x1.1ef78ce2d07f2p-44},
    {0x1.840p-1, 0x1.1bf99635a7000p-2, -0x1.1ac89575c2125p-44},
    {0x1.820p-1, 0x1.214456d0ec000p-2, -0x1.caf0428b728a3p-44},
    {0x1.800p-1, 0x1.269621134e000p-2, -0x1.1b61f10522625p-44},
    {0x1.7e0p-1, 0x1.2bef07cdc9000p-2, 0x1.a9cfa4a5004f4p-45},
    {0x1.7c0p-1, 0x1.314f1e1d36000p-2, -0x1.8e27ad3213cb8p-45},
    {0x1.7a0p-1, 0x1.36b6776be1000p-2, 0x1.16ecdb0f177c8p-46},
    {0x1.780p-1, 0x1.3c25277333000p-2, 0x1.83b54b606bd5cp-46},
    {0x1.760p-1, 0x1.419b423d5f000p-2, -0x1.ce379226de3ecp-44},
    {0x1.740p-1, 0x1.4718dc271c000p-2, 0x1.06c18fb4c14c5p-44},
    {0x1.720p-1, 0x1.4c9e09e173000p-2, -0x1.e20891b0ad8a4p-45},
    {0x1.700p-1, 0x1.522ae0738a000p-2, 0x1.ebe708164c759p-45},
    {0x1.6e0p-1, 0x1.57bf753c8d000p-2, 0x1.fadedee5d40efp-46},
    {0x1.6c0p-1, 0x1.5d5bddf596000p-2, -0x1.a0b2a08a465dcp-47},
};

// log(x), x positive, finite and normal.
__device__ __forceinline__ double log_normal(double x) {
  const int h = __double2hiint(x), t = h - 0x3fe6a000;
  const double e = (double)(t >> 20);
  const double m = __hiloint2double(h - (t & (int)0xfff00000), __double2loint(x));
  const LogEntry* L = kLogTable + ((t >> 13) & 127);
  const double r = fma(m, __ldg(&L->c), -1.0);
  double q = fma(r, -1.0 / 8, 1.0 / 7);
  q = fma(q, r, -1.0 / 6);
  q = fma(q, r, 1.0 / 5);
  q = fma(q, r, -1.0 / 4);
  q = fma(q, r, 1.0 / 3);
  q = fma(q, r, -1.0 / 2);
  const double lo = fma(e, 0x1.ef35793c76730p-45, __ldg(&L->lo));
  const double H = fma(e, 0x1.62e42fefa3800p-1, __ldg(&L->hi));
  const double S = __dadd_rn(H, r);
  const double err = __dadd_rn(__dadd_rn(H, -S), r);
  return __dadd_rn(S, __dadd_rn(err, fma(__dmul_rn(r, r), q, lo)));
}

// Whether x is positive, finite, normal and above the smallest normal's binade,
// from its high word (no FP64 operation).
__device__ __forceinline__ bool positive_normal(double x) {
  return (unsigned)(__double2hiint(x) - 0x00200000) < 0x7ff00000u - 0x00200000u;
}

}  // namespace
}  // namespace gw
