// FP64 reciprocal, reciprocal square root, logarithm and arctangent for the FP64 paths of the pair integrals.
//
// This GPU does 2 FP64 operations per clock and SM, one 64th of its FP32 rate, so an FP64 kernel's time is its count of
// FP64 instructions and nothing else. The library's log, atan2, square root and division are general; the ones here
// take fewer FP64 instructions by using a seed or a table where that costs none:
// - rcp, rsqrt: the hardware's approximation (rcp.approx.ftz.f64, rsqrt.approx.ftz.f64, about 20 bits, not on the FP64
//   pipe) and one third-order step from its residual (Householder's iteration): 3 and 5 instructions, about 1 ulp;
// - log: Tang's table-driven scheme (P. T. P. Tang, ACM TOMS 16, 1990): x = 2^k m, m within 2^-8 of a table point whose
//   reciprocal and logarithm are stored, and six terms of the series of log1p, the large part of the sum
//   exact: 12 instructions;
// - atan2: the quotient's nearest of 65 points c, one angle subtraction atan(t) = atan(c) + atan((n - c d)/(d + c n)) and
//   four terms of the series: 15 instructions.
// Arguments outside the normal range (zero, subnormal, infinite, NaN) go to the library's functions, out of line.
// Errors against 64 bits: at most 2 ulp (rcp, rsqrt, sqrt), 2^-52 max(1, |log x|) and 2^-51 (atan2's angle); the tables
// are the functions' values rounded to FP64. The functions also compile for the host (their test runs there).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

namespace f64 {

#ifdef __CUDACC__
#define F64_FN __host__ __device__ __forceinline__
#else
#define F64_FN inline
#endif

// 1/c to 20 bits, and the logarithm of its reciprocal as a multiple of 2^-42 and the rest, at c = 1 + i/128
#define F64_LOG_ROWS \
    {0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0}, \
    {0x1.fc08000000000p-1, 0x1.fdfaa6b140000p-8, -0x1.98770e7341672p-44}, \
    {0x1.f81f800000000p-1, 0x1.fc0b0b0fc0000p-7, 0x1.f8f3e86147e01p-49}, \
    {0x1.f446600000000p-1, 0x1.7b90e87d60000p-6, -0x1.daeab805daeedp-45}, \
    {0x1.f07c200000000p-1, 0x1.f82990e780000p-6, 0x1.9c0267c68b48fp-45}, \
    {0x1.ecc0800000000p-1, 0x1.39e82b9ff0000p-5, -0x1.e302b8487c536p-44}, \
    {0x1.e913200000000p-1, 0x1.7745376330000p-5, -0x1.b73b9d8eab34ap-45}, \
    {0x1.e573a00000000p-1, 0x1.b42eab1198000p-5, 0x1.da2c34eee7648p-45}, \
    {0x1.e1e1e00000000p-1, 0x1.f0a32c0118000p-5, -0x1.c599e828be3e6p-45}, \
    {0x1.de5d600000000p-1, 0x1.1653e8ea38000p-4, 0x1.7f2e8f6224536p-44}, \
    {0x1.dae6000000000p-1, 0x1.341db961bc000p-4, 0x1.9d092aed8cba6p-44}, \
    {0x1.d77b600000000p-1, 0x1.51b0a1f060000p-4, 0x1.c61692f7a3dd1p-44}, \
    {0x1.d41d400000000p-1, 0x1.6f0d38ae58000p-4, -0x1.434641b10f0bdp-44}, \
    {0x1.d0cb600000000p-1, 0x1.8c341f631c000p-4, -0x1.d5d0a66b1000cp-44}, \
    {0x1.cd85600000000p-1, 0x1.a9271fa4b0000p-4, -0x1.f549ad0747f8fp-44}, \
    {0x1.ca4b400000000p-1, 0x1.c5e4bcf5c0000p-4, -0x1.274eb0936b570p-44}, \
    {0x1.c71c800000000p-1, 0x1.e26ff6e2b0000p-4, 0x1.2e5e93fdd5937p-44}, \
    {0x1.c3f9000000000p-1, 0x1.fec8831dc0000p-4, 0x1.33aa93b51a061p-44}, \
    {0x1.c0e0800000000p-1, 0x1.0d779fcd0a000p-3, 0x1.4cb30ef8beba7p-46}, \
    {0x1.bdd2c00000000p-1, 0x1.1b728b52f6000p-3, 0x1.84851f2722772p-44}, \
    {0x1.bacfa00000000p-1, 0x1.2954eb8200000p-3, 0x1.ccd2e7e07238fp-45}, \
    {0x1.b7d6c00000000p-1, 0x1.371fd401ea000p-3, -0x1.e8f886106753dp-44}, \
    {0x1.b4e8200000000p-1, 0x1.44d2a0ccb8000p-3, -0x1.fb305f3c08ab6p-48}, \
    {0x1.b203600000000p-1, 0x1.526e713a1c000p-3, -0x1.4beba33852786p-44}, \
    {0x1.af28600000000p-1, 0x1.5ff33f0a7a000p-3, 0x1.3c8ad0cb5ddecp-51}, \
    {0x1.ac57000000000p-1, 0x1.6d6106719e000p-3, -0x1.b46e556bdf211p-44}, \
    {0x1.a98f000000000p-1, 0x1.7ab860210e000p-3, 0x1.048ddfb597060p-46}, \
    {0x1.a6d0200000000p-1, 0x1.87f9eb520c000p-3, 0x1.7d3203341831cp-44}, \
    {0x1.a41a400000000p-1, 0x1.9525b1cf46000p-3, -0x1.217137d49c039p-44}, \
    {0x1.a16d400000000p-1, 0x1.a23bbffe2c000p-3, -0x1.531cd91ddf460p-44}, \
    {0x1.9ec8e00000000p-1, 0x1.af3cc2e80c000p-3, 0x1.06db1dc1ede2cp-44}, \
    {0x1.9c2d200000000p-1, 0x1.bc283042da000p-3, -0x1.d6358f1682cc0p-45}, \
    {0x1.9999a00000000p-1, 0x1.c8ff5c79aa000p-3, -0x1.de53e4d28b97bp-47}, \
    {0x1.970e400000000p-1, 0x1.d5c264b4fe000p-3, -0x1.95547a8f12b3ap-44}, \
    {0x1.948b000000000p-1, 0x1.e270c6e2b0000p-3, 0x1.7cbd522655eddp-44}, \
    {0x1.920fc00000000p-1, 0x1.ef0aa2bdc6000p-3, 0x1.96947656c00ecp-45}, \
    {0x1.8f9c200000000p-1, 0x1.fb9162d5e4000p-3, 0x1.9d46a30b36357p-46}, \
    {0x1.8d30200000000p-1, 0x1.040246cb4d000p-2, 0x1.76ad6d1ea313fp-45}, \
    {0x1.8acba00000000p-1, 0x1.0a3227273a000p-2, -0x1.9d506ca2aed96p-45}, \
    {0x1.886e600000000p-1, 0x1.1058bd1ae5000p-2, -0x1.4799d81922822p-44}, \
    {0x1.8618600000000p-1, 0x1.1675cebaba000p-2, 0x1.8b80e7374ab1ap-44}, \
    {0x1.83c9800000000p-1, 0x1.1c8976169a000p-2, -0x1.1e8223a76fedfp-45}, \
    {0x1.8181800000000p-1, 0x1.229423bcf8000p-2, -0x1.9e976f595b40dp-44}, \
    {0x1.7f40600000000p-1, 0x1.2895a0bde8000p-2, 0x1.a8f7ad24be946p-44}, \
    {0x1.7d06000000000p-1, 0x1.2e8e0bae12000p-2, 0x1.4c2700879c369p-44}, \
    {0x1.7ad2200000000p-1, 0x1.347ddb2988000p-2, -0x1.5354dd4bc8092p-45}, \
    {0x1.78a4c00000000p-1, 0x1.3a64db5695000p-2, -0x1.938e30bb373f6p-44}, \
    {0x1.767dc00000000p-1, 0x1.40432f686b000p-2, 0x1.e2deaca7c014dp-45}, \
    {0x1.745d200000000p-1, 0x1.4618a421c6000p-2, 0x1.a13e7cbd9c022p-45}, \
    {0x1.7242800000000p-1, 0x1.4be60f5778000p-2, -0x1.cb9252c4b03d4p-45}, \
    {0x1.702e000000000p-1, 0x1.51aae872e0000p-2, -0x1.74bd8c5b5272cp-44}, \
    {0x1.6e1f800000000p-1, 0x1.5767577456000p-2, -0x1.2eadf0af80b60p-48}, \
    {0x1.6c16c00000000p-1, 0x1.5d1bdff581000p-2, -0x1.856bdc9726ce2p-44}, \
    {0x1.6a13c00000000p-1, 0x1.62c8542b9d000p-2, 0x1.2397d8a9bce27p-45}, \
    {0x1.6816800000000p-1, 0x1.686c85e9b1000p-2, 0x1.33b110b4d95a9p-44}, \
    {0x1.661ec00000000p-1, 0x1.6e08fda2ba000p-2, 0x1.2d6307205b931p-44}, \
    {0x1.642c800000000p-1, 0x1.739d8f6bbd000p-2, 0x1.034e73d0d4b01p-45}, \
    {0x1.623fa00000000p-1, 0x1.792a6b7dd5000p-2, -0x1.3040f74d3b49bp-44}, \
    {0x1.6058200000000p-1, 0x1.7eaf66b82b000p-2, 0x1.955924f90f6dbp-44}, \
    {0x1.5e75c00000000p-1, 0x1.842d10a1e9000p-2, -0x1.cb5b63e3f7b6ap-45}, \
    {0x1.5c98800000000p-1, 0x1.89a3406c14000p-2, 0x1.6d5ad3e195ddfp-45}, \
    {0x1.5ac0600000000p-1, 0x1.8f11ccf367000p-2, -0x1.d40080ea9d2d6p-44}, \
    {0x1.58ed200000000p-1, 0x1.94794ac211000p-2, 0x1.e72e9374051fbp-44}, \
    {0x1.571ee00000000p-1, 0x1.99d933917f000p-2, -0x1.432d2588872c7p-44}, \
    {0x1.5555600000000p-1, 0x1.9f321ecbfa000p-2, 0x1.2fca2f8b33125p-48}, \
    {0x1.5390a00000000p-1, 0x1.a483e68e5c000p-2, 0x1.15aaf1cbb61a2p-44}, \
    {0x1.51d0800000000p-1, 0x1.a9cec5a9a1000p-2, -0x1.e59cadf158099p-44}, \
    {0x1.5015000000000p-1, 0x1.af12972478000p-2, -0x1.dd3bb31998253p-44}, \
    {0x1.4e5e000000000p-1, 0x1.b44f97bcc9000p-2, 0x1.d8a33a6615a51p-44}, \
    {0x1.4cab800000000p-1, 0x1.b985a36931000p-2, 0x1.90d669a4fea8dp-44}, \
    {0x1.4afd600000000p-1, 0x1.beb4f8da72000p-2, 0x1.7efbd673c6f14p-45}, \
    {0x1.4953a00000000p-1, 0x1.c3dd74fcdb000p-2, -0x1.3b06263b14ed4p-45}, \
    {0x1.47ae200000000p-1, 0x1.c8ff5879aa000p-2, 0x1.106afa4608234p-44}, \
    {0x1.460cc00000000p-1, 0x1.ce1ae5b85f000p-2, 0x1.375ededc08018p-44}, \
    {0x1.446f800000000p-1, 0x1.d32ffbe00f000p-2, -0x1.0a9e16cc89426p-46}, \
    {0x1.42d6600000000p-1, 0x1.d83e79d8a3000p-2, -0x1.44beb85ef44a9p-48}, \
    {0x1.4141400000000p-1, 0x1.dd46a44c1c000p-2, 0x1.302fb98efe7cap-44}, \
    {0x1.3fb0200000000p-1, 0x1.e2485b27c7000p-2, 0x1.eea71cd044961p-44}, \
    {0x1.3e22c00000000p-1, 0x1.e7444c1d69000p-2, 0x1.67f1e28b0df24p-45}, \
    {0x1.3c99600000000p-1, 0x1.ec398aa469000p-2, -0x1.26d156a06d358p-47}, \
    {0x1.3b13c00000000p-1, 0x1.f128c5faf2000p-2, -0x1.c4d34cdf12774p-44}, \
    {0x1.3991c00000000p-1, 0x1.f61248a703000p-2, -0x1.ac67ae6830d1ep-44}, \
    {0x1.3813800000000p-1, 0x1.faf58cf78f000p-2, 0x1.9f6cd7e49d1ffp-45}, \
    {0x1.3698e00000000p-1, 0x1.ffd2de057f000p-2, 0x1.293565f2c03ddp-44}, \
    {0x1.3521c00000000p-1, 0x1.0255445a5d800p-1, 0x1.c7637bfa05d31p-44}, \
    {0x1.33ae400000000p-1, 0x1.04be035a92800p-1, 0x1.db3009c15a2ddp-48}, \
    {0x1.323e400000000p-1, 0x1.0723d2c1ce800p-1, -0x1.8dd8e6118de2ep-44}, \
    {0x1.30d1a00000000p-1, 0x1.0986da3574000p-1, 0x1.3be2f0a378f2ap-47}, \
    {0x1.2f68400000000p-1, 0x1.0be7424253000p-1, 0x1.856d8484ce2e1p-46}, \
    {0x1.2e02600000000p-1, 0x1.0e44919d1d000p-1, -0x1.5ee48b5a18b2bp-44}, \
    {0x1.2c9fc00000000p-1, 0x1.109f26e2d5000p-1, 0x1.1d7ee019a35a5p-44}, \
    {0x1.2b40400000000p-1, 0x1.12f72bd93f800p-1, -0x1.75566ef15d546p-44}, \
    {0x1.29e4200000000p-1, 0x1.154c262f4e000p-1, -0x1.d256b02b04f1cp-45}, \
    {0x1.288b000000000p-1, 0x1.179eadbd89800p-1, 0x1.b0bfc6191a4b3p-45}, \
    {0x1.2735000000000p-1, 0x1.19ee7f467d000p-1, -0x1.44cde65df292ep-47}, \
    {0x1.25e2200000000p-1, 0x1.1c3b8e3714000p-1, -0x1.830361740d9efp-45}, \
    {0x1.2492400000000p-1, 0x1.1e8605e704800p-1, -0x1.97e0ff28821b6p-44}, \
    {0x1.2345600000000p-1, 0x1.20cdda592b000p-1, -0x1.d42ca3a555a36p-45}, \
    {0x1.21fb800000000p-1, 0x1.2312ff7bec000p-1, 0x1.294167f5ee619p-44}, \
    {0x1.20b4800000000p-1, 0x1.2555a1e990000p-1, 0x1.979dcedb6f6f8p-44}, \
    {0x1.1f70400000000p-1, 0x1.2795ef289b800p-1, -0x1.ea8a3cbb0ba87p-44}, \
    {0x1.1e2f000000000p-1, 0x1.29d369ec2b800p-1, 0x1.ac82561781a00p-49}, \
    {0x1.1cf0600000000p-1, 0x1.2c0eb25449800p-1, -0x1.c1a32f62a695bp-44}, \
    {0x1.1bb4a00000000p-1, 0x1.2e474aae40000p-1, 0x1.9d402b0ed0a12p-44}, \
    {0x1.1a7ba00000000p-1, 0x1.307d6134f1800p-1, -0x1.18f03467ae9edp-44}, \
    {0x1.1945400000000p-1, 0x1.32b1251122000p-1, 0x1.7463eaebc2f85p-46}, \
    {0x1.1811800000000p-1, 0x1.34e28bd9ce000p-1, 0x1.e316eb9d83308p-45}, \
    {0x1.16e0600000000p-1, 0x1.37118b1474800p-1, 0x1.cb02f8adcc5e8p-44}, \
    {0x1.15b1e00000000p-1, 0x1.393e183562800p-1, 0x1.fed4e598857f1p-44}, \
    {0x1.1486000000000p-1, 0x1.3b6828a000800p-1, 0x1.8abc7225c382fp-47}, \
    {0x1.135c800000000p-1, 0x1.3d9028a715800p-1, -0x1.eab7f79e3094fp-46}, \
    {0x1.1235800000000p-1, 0x1.3fb5d34d17800p-1, 0x1.532dda90aa355p-44}, \
    {0x1.1111200000000p-1, 0x1.41d8e28468000p-1, -0x1.119c0d988db07p-45}, \
    {0x1.0fef000000000p-1, 0x1.43fa002f9d000p-1, -0x1.88858d79b9f46p-45}, \
    {0x1.0ecf600000000p-1, 0x1.4618aaa1c6000p-1, 0x1.c5be77c8b18a9p-44}, \
    {0x1.0db2000000000p-1, 0x1.4835511ea9000p-1, -0x1.c11800d931d97p-46}, \
    {0x1.0c97200000000p-1, 0x1.4a4f70db04800p-1, -0x1.307f043e5b6eap-44}, \
    {0x1.0b7e600000000p-1, 0x1.4c67b73ccf800p-1, 0x1.58f8ef2c9e5c1p-44}, \
    {0x1.0a68200000000p-1, 0x1.4e7d639b76800p-1, 0x1.499c2ae286b76p-45}, \
    {0x1.0954000000000p-1, 0x1.509124c017000p-1, 0x1.6b4b833a5d935p-45}, \
    {0x1.0842200000000p-1, 0x1.52a2b465bd000p-1, 0x1.dd76f5945aa1ep-44}, \
    {0x1.0732600000000p-1, 0x1.54b247b999800p-1, -0x1.b10b755d6d08cp-44}, \
    {0x1.0624e00000000p-1, 0x1.56bf97db3f800p-1, -0x1.f6df723ddf0eap-44}, \
    {0x1.0519800000000p-1, 0x1.58cada5cd7800p-1, 0x1.8d3092f1083dbp-45}, \
    {0x1.0410400000000p-1, 0x1.5ad406c35a000p-1, -0x1.8609ac955eca5p-46}, \
    {0x1.0309200000000p-1, 0x1.5cdb1486c1800p-1, 0x1.7599e58901200p-46}, \
    {0x1.0204000000000p-1, 0x1.5ee03a9241800p-1, 0x1.3ab875af5ad3dp-44}, \
    {0x1.0101000000000p-1, 0x1.60e3314478800p-1, 0x1.d194f928096c0p-46}, \
    {0x1.0000000000000p-1, 0x1.62e42fefa3800p-1, 0x1.ef35793c76730p-45}
// atan(i/64)
#define F64_ATAN_ROWS \
    0x0.0p+0, 0x1.fff555bbb729bp-7, 0x1.ffd55bba97625p-6, 0x1.7fb818430da2ap-5, \
    0x1.ff55bb72cfdeap-5, 0x1.3f59f0e7c559dp-4, 0x1.7ee182602f10fp-4, 0x1.be39ebe6f07c3p-4, \
    0x1.fd5ba9aac2f6ep-4, 0x1.1e1fafb043727p-3, 0x1.3d6eee8c6626cp-3, 0x1.5c9811e3ec26ap-3, \
    0x1.7b97b4bce5b02p-3, 0x1.9a6a8e96c8626p-3, 0x1.b90d7529260a2p-3, 0x1.d77d5df205736p-3, \
    0x1.f5b75f92c80ddp-3, 0x1.09dc597d86362p-2, 0x1.18bf5a30bf178p-2, 0x1.278372057ef46p-2, \
    0x1.362773707ebccp-2, 0x1.44aa436c2af0ap-2, 0x1.530ad9951cd4ap-2, 0x1.614840309cfe2p-2, \
    0x1.6f61941e4def1p-2, 0x1.7d5604b63b3f7p-2, 0x1.8b24d394a1b25p-2, 0x1.98cd5454d6b18p-2, \
    0x1.a64eec3cc23fdp-2, 0x1.b3a911da65c6cp-2, 0x1.c0db4c94ec9f0p-2, 0x1.cde53432c1351p-2, \
    0x1.dac670561bb4fp-2, 0x1.e77eb7f175a34p-2, 0x1.f40dd0b541418p-2, 0x1.0039c73c1a40cp-1, \
    0x1.0657e94db30d0p-1, 0x1.0c6145b5b43dap-1, 0x1.1255d9bfbd2a9p-1, 0x1.1835a88be7c13p-1, \
    0x1.1e00babdefeb4p-1, 0x1.23b71e2cc9e6ap-1, 0x1.2958e59308e31p-1, 0x1.2ee628406cbcap-1, \
    0x1.345f01cce37bbp-1, 0x1.39c391cd4171ap-1, 0x1.3f13fb89e96f4p-1, 0x1.445065b795b56p-1, \
    0x1.4978fa3269ee1p-1, 0x1.4e8de5bb6ec04p-1, 0x1.538f57b89061fp-1, 0x1.587d81f732fbbp-1, \
    0x1.5d58987169b18p-1, 0x1.6220d115d7b8ep-1, 0x1.66d663923e087p-1, 0x1.6b798920b3d99p-1, \
    0x1.700a7c5784634p-1, 0x1.748978fba8e0fp-1, 0x1.78f6bbd5d315ep-1, 0x1.7d528289fa093p-1, \
    0x1.819d0b7158a4dp-1, 0x1.85d69576cc2c5p-1, 0x1.89ff5ff57f1f8p-1, 0x1.8e17aa99cc05ep-1, \
    0x1.921fb54442d18p-1

struct LogRow {
    double inv, hi, lo;
};
#ifdef __CUDACC__
static __device__ const LogRow d_log[129] = {F64_LOG_ROWS};
static __device__ const double d_atan[65] = {F64_ATAN_ROWS};
#endif
#ifndef __CUDA_ARCH__
static const LogRow h_log[129] = {F64_LOG_ROWS};
static const double h_atan[65] = {F64_ATAN_ROWS};
#endif

F64_FN LogRow log_row(int i) {
#ifdef __CUDA_ARCH__
    const double* p = &d_log[i].inv;
    return LogRow{__ldg(p), __ldg(p + 1), __ldg(p + 2)};
#else
    return h_log[i];
#endif
}
F64_FN double atan_row(int i) {
#ifdef __CUDA_ARCH__
    return __ldg(d_atan + i);
#else
    return h_atan[i];
#endif
}

F64_FN int hi_word(double x) {
#ifdef __CUDA_ARCH__
    return __double2hiint(x);
#else
    long long v;
    memcpy(&v, &x, 8);
    return int(v >> 32);
#endif
}
F64_FN int lo_word(double x) {
#ifdef __CUDA_ARCH__
    return __double2loint(x);
#else
    long long v;
    memcpy(&v, &x, 8);
    return int(v);
#endif
}
F64_FN double from_words(int hi, int lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double(hi, lo);
#else
    long long v = ((long long)hi << 32) | (unsigned)lo;
    double x;
    memcpy(&x, &v, 8);
    return x;
#endif
}

// a positive normal number (from its high word alone, with integer instructions)
F64_FN bool normal_pos(double x) { return (unsigned)(hi_word(x) - 0x00100000) < 0x7fe00000u; }

// the hardware's approximations; on the host, a rounding of the value to 20 bits
F64_FN double rcp_seed(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
#else
    return from_words(hi_word(1.0 / x), 0);
#endif
}
F64_FN double rsqrt_seed(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
#else
    return from_words(hi_word(1.0 / ::sqrt(x)), 0);
#endif
}

#ifdef __CUDACC__
static __host__ __device__ __noinline__ double rcp_general(double x) { return 1.0 / x; }
#else
static inline double rcp_general(double x) { return 1.0 / x; }
#endif

// 1/x: y (1 + e + e^2), e = 1 - x y
F64_FN double rcp(double x) {
    if ((unsigned)((hi_word(x) & 0x7fffffff) - (3 << 20)) >= (2040u << 20)) return rcp_general(x);  // |x| outside 2^+-1020
    const double y = rcp_seed(x);
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
F64_FN double div(double a, double b) { return a * rcp(b); }

// 1/sqrt(x) for a normal x > 0: y (1 + e/2 + 3 e^2/8), e = 1 - x y^2
F64_FN double rsqrt(double x) {
    const double y = rsqrt_seed(x);
    const double e = fma(-(x * y), y, 1.0);
    return fma(fma(0.375, e, 0.5), y * e, y);
}

// sqrt(x) and 1/sqrt(x), x >= 0 (0 and +inf for x = 0)
#ifdef __CUDACC__
static __host__ __device__ __noinline__ void sqrt_general(double x, double& s, double& i) {
#else
static inline void sqrt_general(double x, double& s, double& i) {
#endif
    s = ::sqrt(x);
    i = 1.0 / s;
}
F64_FN double sqrt_inv(double x, double& inv) {
    if (!normal_pos(x)) {
        double s;
        sqrt_general(x, s, inv);
        return s;
    }
    inv = rsqrt(x);
    const double s = x * inv;
    return fma(0.5 * inv, fma(-s, s, x), s);  // one correction: about half an ulp
}
F64_FN double sqrt(double x) {
    double i;
    return sqrt_inv(x, i);
}

#ifdef __CUDACC__
static __host__ __device__ __noinline__ double log_general(double x) { return ::log(x); }
static __host__ __device__ __noinline__ double atan2_general(double y, double x) { return ::atan2(y, x); }
#else
static inline double log_general(double x) { return ::log(x); }
static inline double atan2_general(double y, double x) { return ::atan2(y, x); }
#endif

// log 2 as a multiple of 2^-42 and the rest
constexpr double LN2_HI = 0x1.62e42fefa3800p-1, LN2_LO = 0x1.ef35793c76730p-45;

// log(x 2^shift)
template <int shift = 0>
F64_FN double log(double x) {
    if (!normal_pos(x)) return log_general(x) + shift * 0.69314718055994530942;
    const int hi = hi_word(x);
    const int i = ((hi & 0xfffff) + 0x1000) >> 13;  // nearest of the 128 intervals' ends
    const double m = from_words((hi & 0xfffff) | 0x3ff00000, lo_word(x));
    const int k = (hi >> 20) - 1023 + shift;
    const LogRow t = log_row(i);
    const double r = fma(m, t.inv, -1.0);
    const double kd = from_words(0x43300000, int(unsigned(k) ^ 0x80000000u)) - from_words(0x43300000, int(0x80000000u));
    double p = fma(r, -1.0 / 6, 1.0 / 5);
    p = fma(r, p, -1.0 / 4);
    p = fma(r, p, 1.0 / 3);
    p = fma(r, p, -1.0 / 2);
    // k log 2 + log c in two parts, the first exact
    const double hi2 = fma(kd, LN2_HI, t.hi);
    return hi2 + (fma(r * r, p, fma(kd, LN2_LO, t.lo)) + r);
}

// the angle of (x, y), as atan2(y, x)
F64_FN double atan2(double y, double x) {
    const int hy = hi_word(y) & 0x7fffffff, hx = hi_word(x) & 0x7fffffff;
    const bool swap = hy > hx;  // by the high words: ties may go either way
    const double ay = fabs(y), ax = fabs(x);
    const double d = swap ? ay : ax, n = swap ? ax : ay;
    // within 2^100 of 1, so that neither the seed nor the products leave the normal range
    if ((unsigned)(hi_word(d) - ((1023 - 100) << 20)) >= (200u << 20)) return atan2_general(y, x);
    const double t = n * rcp_seed(d);  // the quotient to about 20 bits, in [0, 1 + 2^-19]
    const double big = 105553116266496.0;  // 1.5 * 2^46: adding it leaves round(64 t) in the low word
    const double tb = t + big;
    int i = lo_word(tb);
    i = i < 0 ? 0 : (i > 64 ? 64 : i);
    const double c = tb - big;
    const double u = div(fma(-c, d, n), fma(c, n, d));  // |u| <= 1/128
    const double u2 = u * u;
    double p = fma(u2, -1.0 / 7, 1.0 / 5);
    p = fma(u2, p, -1.0 / 3);
    double a = atan_row(i) + fma(u * u2, p, u);
    // octants: swapped: pi/2 - a; x < 0: pi - that; the sign of y
    const bool neg = hi_word(x) < 0;
    if (swap || neg) {
        const double base = swap ? 1.5707963267948966192 : 3.1415926535897932385;
        a = base + ((swap != neg) ? -a : a);
    }
    return from_words((hi_word(a) & 0x7fffffff) | (hi_word(y) & int(0x80000000u)), lo_word(a));
}

}  // namespace f64
