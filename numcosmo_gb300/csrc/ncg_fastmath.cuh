/*
 * ncg_fastmath.cuh -- table-driven FP64 exponential and logarithm for the
 * kernel sums (exp(lnt - gamma) and log(1 + chi^2/nu) per point-kernel pair).
 *
 * What bounds them: this part issues one FP64 warp instruction per 64 cycles
 * and SM sub-partition (measured: DADD, DFMA, DSETP and the FP64 conversions
 * all 64 cycles, no shorter for fewer lanes), so an FP64 function costs its
 * count of FP64 instructions and everything integer or in a table is nearly
 * free.  The method is the table-driven one of Tang (ACM TOMS 15, 1989 and
 * 16, 1990): reduce by a table of 256 intervals, then a short polynomial.
 *   exp: t = k ln2/256 + f, |f| <= ln2/512, 2^(j/256) from the table
 *        (j = k mod 256), 1 + f + f^2/2 + f^3/6 + f^4/24 (the next term is
 *        below 4e-17): 7 FP64 instructions, 2 more to add the result to a sum;
 *        measured beside the library's 17 for the call alone.
 *   log: u = 2^E m, r = m c_j - 1 with c_j the double nearest to 1/(1 + (j + 1/2)/256),
 *        |r| <= 2^-9 (1 + 2^-8), log u = E ln2 - log c_j + r - r^2/2 + r^3/3
 *        - r^4/4 + r^5/5 (the next term is below 1e-17): 8 FP64 instructions
 *        against 21 of the library's log1p.
 * Errors: exp within 1 ulp for |t| <= 1, relative error |t| 2^-53 beyond (the
 * reduction takes ln2/256 as one double), which the term's own weight e^t in a
 * sum makes up for (t <= 4 here); log within 1.5 ulp of max(|log u|, 1).
 * The tables hold correctly rounded values.
 */
#ifndef NCG_FASTMATH_CUH
#define NCG_FASTMATH_CUH

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

/* 2^(j/256) */
static __device__ const double ncg_exp2_tab[256] = {
  0x1.0000000000000p+0, 0x1.00b1afa5abcbfp+0, 0x1.0163da9fb3335p+0, 0x1.02168143b0281p+0,
  0x1.02c9a3e778061p+0, 0x1.037d42e11bbccp+0, 0x1.04315e86e7f85p+0, 0x1.04e5f72f654b1p+0,
  0x1.059b0d3158574p+0, 0x1.0650a0e3c1f89p+0, 0x1.0706b29ddf6dep+0, 0x1.07bd42b72a836p+0,
  0x1.0874518759bc8p+0, 0x1.092bdf66607e0p+0, 0x1.09e3ecac6f383p+0, 0x1.0a9c79b1f3919p+0,
  0x1.0b5586cf9890fp+0, 0x1.0c0f145e46c85p+0, 0x1.0cc922b7247f7p+0, 0x1.0d83b23395decp+0,
  0x1.0e3ec32d3d1a2p+0, 0x1.0efa55fdfa9c5p+0, 0x1.0fb66affed31bp+0, 0x1.1073028d7233ep+0,
  0x1.11301d0125b51p+0, 0x1.11edbab5e2ab6p+0, 0x1.12abdc06c31ccp+0, 0x1.136a814f204abp+0,
  0x1.1429aaea92de0p+0, 0x1.14e95934f312ep+0, 0x1.15a98c8a58e51p+0, 0x1.166a45471c3c2p+0,
  0x1.172b83c7d517bp+0, 0x1.17ed48695bbc0p+0, 0x1.18af9388c8deap+0, 0x1.1972658375d2fp+0,
  0x1.1a35beb6fcb75p+0, 0x1.1af99f8138a1cp+0, 0x1.1bbe084045cd4p+0, 0x1.1c82f95281c6bp+0,
  0x1.1d4873168b9aap+0, 0x1.1e0e75eb44027p+0, 0x1.1ed5022fcd91dp+0, 0x1.1f9c18438ce4dp+0,
  0x1.2063b88628cd6p+0, 0x1.212be3578a819p+0, 0x1.21f49917ddc96p+0, 0x1.22bdda27912d1p+0,
  0x1.2387a6e756238p+0, 0x1.2451ffb82140ap+0, 0x1.251ce4fb2a63fp+0, 0x1.25e85711ece75p+0,
  0x1.26b4565e27cddp+0, 0x1.2780e341ddf29p+0, 0x1.284dfe1f56381p+0, 0x1.291ba7591bb70p+0,
  0x1.29e9df51fdee1p+0, 0x1.2ab8a66d10f13p+0, 0x1.2b87fd0dad990p+0, 0x1.2c57e39771b2fp+0,
  0x1.2d285a6e4030bp+0, 0x1.2df961f641589p+0, 0x1.2ecafa93e2f56p+0, 0x1.2f9d24abd886bp+0,
  0x1.306fe0a31b715p+0, 0x1.31432edeeb2fdp+0, 0x1.32170fc4cd831p+0, 0x1.32eb83ba8ea32p+0,
  0x1.33c08b26416ffp+0, 0x1.3496266e3fa2dp+0, 0x1.356c55f929ff1p+0, 0x1.36431a2de883bp+0,
  0x1.371a7373aa9cbp+0, 0x1.37f26231e754ap+0, 0x1.38cae6d05d866p+0, 0x1.39a401b7140efp+0,
  0x1.3a7db34e59ff7p+0, 0x1.3b57fbfec6cf4p+0, 0x1.3c32dc313a8e5p+0, 0x1.3d0e544ede173p+0,
  0x1.3dea64c123422p+0, 0x1.3ec70df1c5175p+0, 0x1.3fa4504ac801cp+0, 0x1.40822c367a024p+0,
  0x1.4160a21f72e2ap+0, 0x1.423fb2709468ap+0, 0x1.431f5d950a897p+0, 0x1.43ffa3f84b9d4p+0,
  0x1.44e086061892dp+0, 0x1.45c2042a7d232p+0, 0x1.46a41ed1d0057p+0, 0x1.4786d668b3237p+0,
  0x1.486a2b5c13cd0p+0, 0x1.494e1e192aed2p+0, 0x1.4a32af0d7d3dep+0, 0x1.4b17dea6db7d7p+0,
  0x1.4bfdad5362a27p+0, 0x1.4ce41b817c114p+0, 0x1.4dcb299fddd0dp+0, 0x1.4eb2d81d8abffp+0,
  0x1.4f9b2769d2ca7p+0, 0x1.508417f4531eep+0, 0x1.516daa2cf6642p+0, 0x1.5257de83f4eefp+0,
  0x1.5342b569d4f82p+0, 0x1.542e2f4f6ad27p+0, 0x1.551a4ca5d920fp+0, 0x1.56070dde910d2p+0,
  0x1.56f4736b527dap+0, 0x1.57e27dbe2c4cfp+0, 0x1.58d12d497c7fdp+0, 0x1.59c0827ff07ccp+0,
  0x1.5ab07dd485429p+0, 0x1.5ba11fba87a03p+0, 0x1.5c9268a5946b7p+0, 0x1.5d84590998b93p+0,
  0x1.5e76f15ad2148p+0, 0x1.5f6a320dceb71p+0, 0x1.605e1b976dc09p+0, 0x1.6152ae6cdf6f4p+0,
  0x1.6247eb03a5585p+0, 0x1.633dd1d1929fdp+0, 0x1.6434634ccc320p+0, 0x1.652b9febc8fb7p+0,
  0x1.6623882552225p+0, 0x1.671c1c70833f6p+0, 0x1.68155d44ca973p+0, 0x1.690f4b19e9538p+0,
  0x1.6a09e667f3bcdp+0, 0x1.6b052fa75173ep+0, 0x1.6c012750bdabfp+0, 0x1.6cfdcddd47645p+0,
  0x1.6dfb23c651a2fp+0, 0x1.6ef9298593ae5p+0, 0x1.6ff7df9519484p+0, 0x1.70f7466f42e87p+0,
  0x1.71f75e8ec5f74p+0, 0x1.72f8286ead08ap+0, 0x1.73f9a48a58174p+0, 0x1.74fbd35d7cbfdp+0,
  0x1.75feb564267c9p+0, 0x1.77024b1ab6e09p+0, 0x1.780694fde5d3fp+0, 0x1.790b938ac1cf6p+0,
  0x1.7a11473eb0187p+0, 0x1.7b17b0976cfdbp+0, 0x1.7c1ed0130c132p+0, 0x1.7d26a62ff86f0p+0,
  0x1.7e2f336cf4e62p+0, 0x1.7f3878491c491p+0, 0x1.80427543e1a12p+0, 0x1.814d2add106d9p+0,
  0x1.82589994cce13p+0, 0x1.8364c1eb941f7p+0, 0x1.8471a4623c7adp+0, 0x1.857f4179f5b21p+0,
  0x1.868d99b4492edp+0, 0x1.879cad931a436p+0, 0x1.88ac7d98a6699p+0, 0x1.89bd0a478580fp+0,
  0x1.8ace5422aa0dbp+0, 0x1.8be05bad61778p+0, 0x1.8cf3216b5448cp+0, 0x1.8e06a5e0866d9p+0,
  0x1.8f1ae99157736p+0, 0x1.902fed0282c8ap+0, 0x1.9145b0b91ffc6p+0, 0x1.925c353aa2fe2p+0,
  0x1.93737b0cdc5e5p+0, 0x1.948b82b5f98e5p+0, 0x1.95a44cbc8520fp+0, 0x1.96bdd9a7670b3p+0,
  0x1.97d829fde4e50p+0, 0x1.98f33e47a22a2p+0, 0x1.9a0f170ca07bap+0, 0x1.9b2bb4d53fe0dp+0,
  0x1.9c49182a3f090p+0, 0x1.9d674194bb8d5p+0, 0x1.9e86319e32323p+0, 0x1.9fa5e8d07f29ep+0,
  0x1.a0c667b5de565p+0, 0x1.a1e7aed8eb8bbp+0, 0x1.a309bec4a2d33p+0, 0x1.a42c980460ad8p+0,
  0x1.a5503b23e255dp+0, 0x1.a674a8af46052p+0, 0x1.a799e1330b358p+0, 0x1.a8bfe53c12e59p+0,
  0x1.a9e6b5579fdbfp+0, 0x1.ab0e521356ebap+0, 0x1.ac36bbfd3f37ap+0, 0x1.ad5ff3a3c2774p+0,
  0x1.ae89f995ad3adp+0, 0x1.afb4ce622f2ffp+0, 0x1.b0e07298db666p+0, 0x1.b20ce6c9a8952p+0,
  0x1.b33a2b84f15fbp+0, 0x1.b468415b749b1p+0, 0x1.b59728de5593ap+0, 0x1.b6c6e29f1c52ap+0,
  0x1.b7f76f2fb5e47p+0, 0x1.b928cf22749e4p+0, 0x1.ba5b030a1064ap+0, 0x1.bb8e0b79a6f1fp+0,
  0x1.bcc1e904bc1d2p+0, 0x1.bdf69c3f3a207p+0, 0x1.bf2c25bd71e09p+0, 0x1.c06286141b33dp+0,
  0x1.c199bdd85529cp+0, 0x1.c2d1cd9fa652cp+0, 0x1.c40ab5fffd07ap+0, 0x1.c544778fafb22p+0,
  0x1.c67f12e57d14bp+0, 0x1.c7ba88988c933p+0, 0x1.c8f6d9406e7b5p+0, 0x1.ca3405751c4dbp+0,
  0x1.cb720dcef9069p+0, 0x1.ccb0f2e6d1675p+0, 0x1.cdf0b555dc3fap+0, 0x1.cf3155b5bab74p+0,
  0x1.d072d4a07897cp+0, 0x1.d1b532b08c968p+0, 0x1.d2f87080d89f2p+0, 0x1.d43c8eacaa1d6p+0,
  0x1.d5818dcfba487p+0, 0x1.d6c76e862e6d3p+0, 0x1.d80e316c98398p+0, 0x1.d955d71ff6075p+0,
  0x1.da9e603db3285p+0, 0x1.dbe7cd63a8315p+0, 0x1.dd321f301b460p+0, 0x1.de7d5641c0658p+0,
  0x1.dfc97337b9b5fp+0, 0x1.e11676b197d17p+0, 0x1.e264614f5a129p+0, 0x1.e3b333b16ee12p+0,
  0x1.e502ee78b3ff6p+0, 0x1.e653924676d76p+0, 0x1.e7a51fbc74c83p+0, 0x1.e8f7977cdb740p+0,
  0x1.ea4afa2a490dap+0, 0x1.eb9f4867cca6ep+0, 0x1.ecf482d8e67f1p+0, 0x1.ee4aaa2188510p+0,
  0x1.efa1bee615a27p+0, 0x1.f0f9c1cb6412ap+0, 0x1.f252b376bba97p+0, 0x1.f3ac948dd7274p+0,
  0x1.f50765b6e4540p+0, 0x1.f6632798844f8p+0, 0x1.f7bfdad9cbe14p+0, 0x1.f91d802243c89p+0,
  0x1.fa7c1819e90d8p+0, 0x1.fbdba3692d514p+0, 0x1.fd3c22b8f71f1p+0, 0x1.fe9d96b2a23d9p+0,
};

/* c_j (x) and -log c_j (y) */
static __device__ const double2 ncg_log_tab[256] = {
  { 0x1.ff007fc01ff00p-1, 0x1.ff802a9ab11e6p-10 }, { 0x1.fd04794a10e6ap-1, 0x1.7ee11ebd82ec4p-8 },
  { 0x1.fb0c610d5e939p-1, 0x1.3e7295d25a7d5p-7 }, { 0x1.f9182b6813bafp-1, 0x1.bcf712c743853p-7 },
  { 0x1.f727cce5f530ap-1, 0x1.1d7f7eb9eebf1p-6 }, { 0x1.f53b3a3fa204ep-1, 0x1.5c45a51b8d393p-6 },
  { 0x1.f3526859b8cecp-1, 0x1.9ace7551cc515p-6 }, { 0x1.f16d4c4401f17p-1, 0x1.d91a66c543cbep-6 },
  { 0x1.ef8bdb389ebadp-1, 0x1.0b94f7c196173p-5 }, { 0x1.edae0a9b3d3a5p-1, 0x1.2a7ec2214e879p-5 },
  { 0x1.ebd3cff850b0cp-1, 0x1.494acc34d911dp-5 }, { 0x1.e9fd21044e799p-1, 0x1.67f94f094bd92p-5 },
  { 0x1.e829f39aef509p-1, 0x1.868a83083f6d0p-5 }, { 0x1.e65a3dbe74d6bp-1, 0x1.a4fe9ffa3d233p-5 },
  { 0x1.e48df596f3394p-1, 0x1.c355dd0921f2fp-5 }, { 0x1.e2c511719ee16p-1, 0x1.e19070c276010p-5 },
  { 0x1.e0ff87c01e100p-1, 0x1.ffae9119b92fbp-5 }, { 0x1.df3d4f17de4dbp-1, 0x1.0ed839b5526fep-4 },
  { 0x1.dd7e5e316d94cp-1, 0x1.1dcb263db1944p-4 }, { 0x1.dbc2abe7d71d4p-1, 0x1.2cb0283f5de22p-4 },
  { 0x1.da0a2f3803b41p-1, 0x1.3b87598b1b6f0p-4 }, { 0x1.d854df401d855p-1, 0x1.4a50d3aa1b03fp-4 },
  { 0x1.d6a2b33ef7448p-1, 0x1.590cafdf01c26p-4 }, { 0x1.d4f3a293769cap-1, 0x1.67bb0726ec0fbp-4 },
  { 0x1.d347a4bc01d34p-1, 0x1.765bf23a6be17p-4 }, { 0x1.d19eb155f08a4p-1, 0x1.84ef898e82828p-4 },
  { 0x1.cff8c01cff8c0p-1, 0x1.9375e55595edfp-4 }, { 0x1.ce55c8eac7900p-1, 0x1.a1ef1d8061cd8p-4 },
  { 0x1.ccb5c3b636e3ap-1, 0x1.b05b49bee4403p-4 }, { 0x1.cb18a8930de60p-1, 0x1.beba818146764p-4 },
  { 0x1.c97e6fb15e44dp-1, 0x1.cd0cdbf8c13e0p-4 }, { 0x1.c7e7115d0ce95p-1, 0x1.db5270187d925p-4 },
  { 0x1.c65285fd56843p-1, 0x1.e98b54967146bp-4 }, { 0x1.c4c0c61456a8ep-1, 0x1.f7b79fec37de2p-4 },
  { 0x1.c331ca3e91679p-1, 0x1.02ebb42bf3d4ap-3 }, { 0x1.c1a58b327f576p-1, 0x1.09f561ee719c4p-3 },
  { 0x1.c01c01c01c01cp-1, 0x1.10f8e422539b1p-3 }, { 0x1.be9526d0769fap-1, 0x1.17f6458fca611p-3 },
  { 0x1.bd10f365451b6p-1, 0x1.1eed90e2dc2c3p-3 }, { 0x1.bb8f609879493p-1, 0x1.25ded0abc6ad3p-3 },
  { 0x1.ba10679bd8488p-1, 0x1.2cca0f5f5f252p-3 }, { 0x1.b89401b89401cp-1, 0x1.33af575770e4dp-3 },
  { 0x1.b71a284ee6b34p-1, 0x1.3a8eb2d31a375p-3 }, { 0x1.b5a2d4d5b081fp-1, 0x1.41682bf727bbfp-3 },
  { 0x1.b42e00da17007p-1, 0x1.483bccce6e3dcp-3 }, { 0x1.b2bba5ff26a23p-1, 0x1.4f099f4a230b1p-3 },
  { 0x1.b14bbdfd760e6p-1, 0x1.55d1ad4232d70p-3 }, { 0x1.afde42a2cb482p-1, 0x1.5c940075972b9p-3 },
  { 0x1.ae732dd1c2a09p-1, 0x1.6350a28aaa759p-3 }, { 0x1.ad0a798177693p-1, 0x1.6a079d0f7aad0p-3 },
  { 0x1.aba41fbd2e5b1p-1, 0x1.70b8f97a1aa74p-3 }, { 0x1.aa401aa401aa4p-1, 0x1.7764c128f2127p-3 },
  { 0x1.a8de64688ebabp-1, 0x1.7e0afd630c276p-3 }, { 0x1.a77ef750a56dap-1, 0x1.84abb75865137p-3 },
  { 0x1.a621cdb4f8fdfp-1, 0x1.8b46f8223625bp-3 }, { 0x1.a4c6e200d2637p-1, 0x1.91dcc8c340bdfp-3 },
  { 0x1.a36e2eb1c432dp-1, 0x1.986d3228180c8p-3 }, { 0x1.a217ae575ff2fp-1, 0x1.9ef83d2769a34p-3 },
  { 0x1.a0c35b92ecdf1p-1, 0x1.a57df28244dcbp-3 }, { 0x1.9f713117200d0p-1, 0x1.abfe5ae46124ap-3 },
  { 0x1.9e2129a7d5f0ap-1, 0x1.b2797ee46320cp-3 }, { 0x1.9cd34019cd340p-1, 0x1.b8ef670420c3bp-3 },
  { 0x1.9b876f5262dd1p-1, 0x1.bf601bb0e44e0p-3 }, { 0x1.9a3db2474fb98p-1, 0x1.c5cba543ae424p-3 },
  { 0x1.98f603fe670a0p-1, 0x1.cc320c0176501p-3 }, { 0x1.97b05f8d56652p-1, 0x1.d293581b6b3e7p-3 },
  { 0x1.966cc01966cc0p-1, 0x1.d8ef91af31d5ep-3 }, { 0x1.952b20d73ee97p-1, 0x1.df46c0c722d30p-3 },
  { 0x1.93eb7d0aa6759p-1, 0x1.e598ed5a87e2ep-3 }, { 0x1.92add0064ab74p-1, 0x1.ebe61f4dd7b0bp-3 },
  { 0x1.9172152b841ddp-1, 0x1.f22e5e72f105cp-3 }, { 0x1.903847ea1cec1p-1, 0x1.f871b28955045p-3 },
  { 0x1.8f0063c018f00p-1, 0x1.feb0233e607cep-3 }, { 0x1.8dca64397e408p-1, 0x1.0274dc16c232fp-2 },
  { 0x1.8c9644f01efbcp-1, 0x1.058f3c703ebc5p-2 }, { 0x1.8b64018b64019p-1, 0x1.08a73667c57aep-2 },
  { 0x1.8a3395c018a34p-1, 0x1.0bbccdb0d24bcp-2 }, { 0x1.8904fd503744bp-1, 0x1.0ed005f657da5p-2 },
  { 0x1.87d8340ab6e97p-1, 0x1.11e0e2dad9cb6p-2 }, { 0x1.86ad35cb59a84p-1, 0x1.14ef67f88685ap-2 },
  { 0x1.8583fe7a7c018p-1, 0x1.17fb98e15095ep-2 }, { 0x1.845c8a0ce5129p-1, 0x1.1b05791f07b4ap-2 },
  { 0x1.8336d48397a24p-1, 0x1.1e0d0c33716bdp-2 }, { 0x1.8212d9eba4018p-1, 0x1.211255986160cp-2 },
  { 0x1.80f0965dfabcbp-1, 0x1.241558bfd1405p-2 }, { 0x1.7fd005ff40180p-1, 0x1.27161913f853dp-2 },
  { 0x1.7eb124ffa053bp-1, 0x1.2a1499f762bcap-2 }, { 0x1.7d93ef9aa4b46p-1, 0x1.2d10dec508582p-2 },
  { 0x1.7c7862170949fp-1, 0x1.300aead06350cp-2 }, { 0x1.7b5e78c693733p-1, 0x1.3302c1658658ap-2 },
  { 0x1.7a463005e918cp-1, 0x1.35f865c93293ep-2 }, { 0x1.792f843c689c3p-1, 0x1.38ebdb38ed320p-2 },
  { 0x1.781a71dc01782p-1, 0x1.3bdd24eb14b69p-2 }, { 0x1.7706f5610d8d0p-1, 0x1.3ecc460ef5f50p-2 },
  { 0x1.75f50b522b17cp-1, 0x1.41b941cce0beep-2 }, { 0x1.74e4b040174e5p-1, 0x1.44a41b463c47bp-2 },
  { 0x1.73d5e0c5899f7p-1, 0x1.478cd5959b3d8p-2 }, { 0x1.72c899870f91fp-1, 0x1.4a7373cecf997p-2 },
  { 0x1.71bcd732e940ap-1, 0x1.4d57f8fefe27fp-2 }, { 0x1.70b29680e66fap-1, 0x1.503a682cb1cb3p-2 },
  { 0x1.6fa9d43244380p-1, 0x1.531ac457ee77fp-2 }, { 0x1.6ea28d118b474p-1, 0x1.55f9107a43ee2p-2 },
  { 0x1.6d9cbdf26eaefp-1, 0x1.58d54f86e02f3p-2 }, { 0x1.6c9863b1ab429p-1, 0x1.5baf846aa1b1ap-2 },
  { 0x1.6b957b34e7803p-1, 0x1.5e87b20c2954ap-2 }, { 0x1.6a94016a94017p-1, 0x1.615ddb4bec13cp-2 },
  { 0x1.6993f349cc726p-1, 0x1.64320304447c1p-2 }, { 0x1.68954dd2390bap-1, 0x1.67042c0983e30p-2 },
  { 0x1.67980e0bf08c7p-1, 0x1.69d4592a0362ep-2 }, { 0x1.669c31075ab40p-1, 0x1.6ca28d2e34986p-2 },
  { 0x1.65a1b3dd13357p-1, 0x1.6f6ecad8b2292p-2 }, { 0x1.64a893adcd25fp-1, 0x1.723914e6500e2p-2 },
  { 0x1.63b0cda236e1cp-1, 0x1.75016e0e2ba63p-2 }, { 0x1.62ba5eeade65ep-1, 0x1.77c7d901bb913p-2 },
  { 0x1.61c544c0161c5p-1, 0x1.7a8c586cdf545p-2 }, { 0x1.60d17c61da198p-1, 0x1.7d4eeef5eec6ep-2 },
  { 0x1.5fdf0317b5c6fp-1, 0x1.800f9f3dc94ccp-2 }, { 0x1.5eedd630a9fb3p-1, 0x1.82ce6bdfe4d9ep-2 },
  { 0x1.5dfdf303137b6p-1, 0x1.858b57725cc43p-2 }, { 0x1.5d0f56ec91e57p-1, 0x1.8846648600623p-2 },
  { 0x1.5c21ff51ef005p-1, 0x1.8aff95a661781p-2 }, { 0x1.5b35e99f06714p-1, 0x1.8db6ed59e272dp-2 },
  { 0x1.5a4b1346add2bp-1, 0x1.906c6e21c4753p-2 }, { 0x1.596179c29d2cep-1, 0x1.93201a7a35336p-2 },
  { 0x1.58791a9357ccep-1, 0x1.95d1f4da5ca0ap-2 }, { 0x1.5791f34015792p-1, 0x1.9881ffb46a6f0p-2 },
  { 0x1.56ac0156ac015p-1, 0x1.9b303d75a3620p-2 }, { 0x1.55c7426b79286p-1, 0x1.9ddcb0866e742p-2 },
  { 0x1.54e3b4194ce66p-1, 0x1.a0875b4a61d17p-2 }, { 0x1.5401540154015p-1, 0x1.a33040204fa64p-2 },
  { 0x1.53201fcb02fb1p-1, 0x1.a5d7616252c36p-2 }, { 0x1.5240152401524p-1, 0x1.a87cc165db199p-2 },
  { 0x1.516131c015161p-1, 0x1.ab20627bba0a0p-2 }, { 0x1.508373590ec9cp-1, 0x1.adc246f02e900p-2 },
  { 0x1.4fa6d7aeb597cp-1, 0x1.b062710af141cp-2 }, { 0x1.4ecb5c86b3d24p-1, 0x1.b300e30f402a2p-2 },
  { 0x1.4df0ffac83c01p-1, 0x1.b59d9f3bea7c3p-2 }, { 0x1.4d17bef15cb4ep-1, 0x1.b838a7cb5c1efp-2 },
  { 0x1.4c3f982c20723p-1, 0x1.bad1fef3a9167p-2 }, { 0x1.4b68893948d1cp-1, 0x1.bd69a6e698c46p-2 },
  { 0x1.4a928ffad5b5cp-1, 0x1.bfffa1d1b1084p-2 }, { 0x1.49bdaa583b401p-1, 0x1.c293f1de4137dp-2 },
  { 0x1.48e9d63e504d1p-1, 0x1.c52699316cf6cp-2 }, { 0x1.4817119f3d325p-1, 0x1.c7b799ec36eafp-2 },
  { 0x1.47455a726abf2p-1, 0x1.ca46f62b8b4e6p-2 }, { 0x1.4674aeb4717e9p-1, 0x1.ccd4b0084a5efp-2 },
  { 0x1.45a50c670938fp-1, 0x1.cf60c99752ad9p-2 }, { 0x1.44d67190f8b43p-1, 0x1.d1eb44e98b4c9p-2 },
  { 0x1.4408dc3e05b22p-1, 0x1.d474240beddd7p-2 }, { 0x1.433c4a7ee52b4p-1, 0x1.d6fb6907907eap-2 },
  { 0x1.4270ba692bc4dp-1, 0x1.d98115e1af9b6p-2 }, { 0x1.41a62a173e821p-1, 0x1.dc052c9bb79abp-2 },
  { 0x1.40dc97a843ae8p-1, 0x1.de87af334e71cp-2 }, { 0x1.4014014014014p-1, 0x1.e1089fa25d168p-2 },
  { 0x1.3f4c65072bf74p-1, 0x1.e387ffdf18d77p-2 }, { 0x1.3e85c12a9d651p-1, 0x1.e605d1dc0c931p-2 },
  { 0x1.3dc013dc013dcp-1, 0x1.e882178821d52p-2 }, { 0x1.3cfb5b51698ebp-1, 0x1.eafcd2cea9d72p-2 },
  { 0x1.3c3795c553afbp-1, 0x1.ed7605976663dp-2 }, { 0x1.3b74c1769aa5cp-1, 0x1.efedb1c692a07p-2 },
  { 0x1.3ab2dca869b81p-1, 0x1.f263d93cebbb9p-2 }, { 0x1.39f1e5a22f36ep-1, 0x1.f4d87dd7b97e6p-2 },
  { 0x1.3931daaf8f721p-1, 0x1.f74ba170d6c7ep-2 }, { 0x1.3872ba2057e04p-1, 0x1.f9bd45deb9ea5p-2 },
  { 0x1.37b4824872744p-1, 0x1.fc2d6cf47cf1cp-2 }, { 0x1.36f7317fd9212p-1, 0x1.fe9c1881e5cfep-2 },
  { 0x1.363ac622898b1p-1, 0x1.0084a529b7386p-1 }, { 0x1.357f3e9078e5bp-1, 0x1.01ba8219265a4p-1 },
  { 0x1.34c4992d87fd9p-1, 0x1.02efa3f23d29cp-1 }, { 0x1.340ad461776d3p-1, 0x1.04240b965e54cp-1 },
  { 0x1.3351ee97dbfc6p-1, 0x1.0557b9e55634ep-1 }, { 0x1.3299e6401329ap-1, 0x1.068aafbd5e9dap-1 },
  { 0x1.31e2b9cd37dc2p-1, 0x1.07bcedfb229fep-1 }, { 0x1.312c67b6173eep-1, 0x1.08ee7579c2413p-1 },
  { 0x1.3076ee7525c2cp-1, 0x1.0a1f4712d6292p-1 }, { 0x1.2fc24c8874486p-1, 0x1.0b4f639e73429p-1 },
  { 0x1.2f0e8071a5703p-1, 0x1.0c7ecbf32e532p-1 }, { 0x1.2e5b88b5e3104p-1, 0x1.0dad80e61f87ap-1 },
  { 0x1.2da963ddd3cfbp-1, 0x1.0edb834ae5f5ep-1 }, { 0x1.2cf8107590e67p-1, 0x1.1008d3f3ab146p-1 },
  { 0x1.2c478d0c9c013p-1, 0x1.113573b126281p-1 }, { 0x1.2b97d835d548ep-1, 0x1.126163529fa7ap-1 },
  { 0x1.2ae8f087718d0p-1, 0x1.138ca3a5f494fp-1 }, { 0x1.2a3ad49af0907p-1, 0x1.14b7357799cd2p-1 },
  { 0x1.298d830d13780p-1, 0x1.15e119929f4e4p-1 }, { 0x1.28e0fa7dd35a3p-1, 0x1.170a50c0b3749p-1 },
  { 0x1.2835399057efdp-1, 0x1.1832dbca262d9p-1 }, { 0x1.278a3eeaee650p-1, 0x1.195abb75ec21ap-1 },
  { 0x1.26e009370049cp-1, 0x1.1a81f089a1d56p-1 }, { 0x1.263697210aa18p-1, 0x1.1ba87bc98ec1ap-1 },
  { 0x1.258de75895121p-1, 0x1.1cce5df8a8622p-1 }, { 0x1.24e5f89029305p-1, 0x1.1df397d8953bfp-1 },
  { 0x1.243ec97d49eaep-1, 0x1.1f182a29afdb1p-1 }, { 0x1.239858d86b11fp-1, 0x1.203c15ab09c7ap-1 },
  { 0x1.22f2a55ce8fc5p-1, 0x1.215f5b1a6e729p-1 }, { 0x1.224dadc900489p-1, 0x1.2281fb34661a0p-1 },
  { 0x1.21a970ddc5ba7p-1, 0x1.23a3f6b438a52p-1 }, { 0x1.2105ed5f1e336p-1, 0x1.24c54e53f0793p-1 },
  { 0x1.20632213b6c6dp-1, 0x1.25e602cc5d448p-1 }, { 0x1.1fc10dc4fce8bp-1, 0x1.270614d516c38p-1 },
  { 0x1.1f1faf3f16b64p-1, 0x1.282585247f7d3p-1 }, { 0x1.1e7f0550db594p-1, 0x1.2944546fc777ap-1 },
  { 0x1.1ddf0ecbcb841p-1, 0x1.2a62836aeee59p-1 }, { 0x1.1d3fca840a074p-1, 0x1.2b8012c8c8cc0p-1 },
  { 0x1.1ca13750547fep-1, 0x1.2c9d033afda0fp-1 }, { 0x1.1c035409fc1dfp-1, 0x1.2db955720de23p-1 },
  { 0x1.1b661f8cde833p-1, 0x1.2ed50a1d54a5ap-1 }, { 0x1.1ac998b75eb90p-1, 0x1.2ff021eb0a221p-1 },
  { 0x1.1a2dbe6a5e3e4p-1, 0x1.310a9d8846313p-1 }, { 0x1.19928f89362b7p-1, 0x1.32247da102ca6p-1 },
  { 0x1.18f80af9b06dcp-1, 0x1.333dc2e01e776p-1 }, { 0x1.185e2fa401186p-1, 0x1.34566def5ec14p-1 },
  { 0x1.17c4fc72bfcb9p-1, 0x1.356e7f7772978p-1 }, { 0x1.172c7052e1316p-1, 0x1.3685f81ff4b06p-1 },
  { 0x1.16948a33b08fap-1, 0x1.379cd88f6de2bp-1 }, { 0x1.15fd4906c96f1p-1, 0x1.38b3216b5778dp-1 },
  { 0x1.1566abc011567p-1, 0x1.39c8d3581d7ecp-1 }, { 0x1.14d0b155b19aep-1, 0x1.3addeef921080p-1 },
  { 0x1.143b58c01143bp-1, 0x1.3bf274f0ba70dp-1 }, { 0x1.13a6a0f9cf01ep-1, 0x1.3d0665e03b98fp-1 },
  { 0x1.131288ffbb3b6p-1, 0x1.3e19c267f2182p-1 }, { 0x1.127f0fd0d2295p-1, 0x1.3f2c8b27296cdp-1 },
  { 0x1.11ec346e36092p-1, 0x1.403ec0bc2d255p-1 }, { 0x1.1159f5db29606p-1, 0x1.415063c44b02cp-1 },
  { 0x1.10c8531d0952ep-1, 0x1.426174dbd5166p-1 }, { 0x1.10374b3b480aap-1, 0x1.4371f49e23d9dp-1 },
  { 0x1.0fa6dd3f67322p-1, 0x1.4481e3a59840ep-1 }, { 0x1.0f170834f27fap-1, 0x1.4591428b9dc68p-1 },
  { 0x1.0e87cb297a51ep-1, 0x1.46a011e8ac746p-1 }, { 0x1.0df9252c8e5e6p-1, 0x1.47ae52544ae45p-1 },
  { 0x1.0d6b154fb86f9p-1, 0x1.48bc0465103d8p-1 }, { 0x1.0cdd9aa677344p-1, 0x1.49c928b0a62bep-1 },
  { 0x1.0c50b446391f3p-1, 0x1.4ad5bfcbcad23p-1 }, { 0x1.0bc4614657569p-1, 0x1.4be1ca4a52b77p-1 },
  { 0x1.0b38a0c010b39p-1, 0x1.4ced48bf2aaf3p-1 }, { 0x1.0aad71ce84d16p-1, 0x1.4df83bbc59bc9p-1 },
  { 0x1.0a22d38eaf2bfp-1, 0x1.4f02a3d302f06p-1 }, { 0x1.0998c51f624d5p-1, 0x1.500c819367434p-1 },
  { 0x1.090f45a1430aap-1, 0x1.5115d58ce769bp-1 }, { 0x1.08865436c3cf7p-1, 0x1.521ea04e05a45p-1 },
  { 0x1.07fdf0041ff7cp-1, 0x1.5326e264678adp-1 }, { 0x1.0776182f57386p-1, 0x1.542e9c5cd7d2ep-1 },
  { 0x1.06eecbe029155p-1, 0x1.5535cec348128p-1 }, { 0x1.06680a4010668p-1, 0x1.563c7a22d27ccp-1 },
  { 0x1.05e1d27a3ee9cp-1, 0x1.57429f05bb9b9p-1 }, { 0x1.055c23bb98e2ap-1, 0x1.58483df574045p-1 },
  { 0x1.04d6fd32b0c7bp-1, 0x1.594d577a9a07fp-1 }, { 0x1.04525e0fc2fcbp-1, 0x1.5a51ec1cfb5f4p-1 },
  { 0x1.03ce4584b19a0p-1, 0x1.5b55fc6396d2bp-1 }, { 0x1.034ab2c50040dp-1, 0x1.5c5988d49dddep-1 },
  { 0x1.02c7a505cffbfp-1, 0x1.5d5c91f5764f1p-1 }, { 0x1.02451b7ddb2d2p-1, 0x1.5e5f184abbe28p-1 },
  { 0x1.01c315657186bp-1, 0x1.5f611c5841d9fp-1 }, { 0x1.014191f674111p-1, 0x1.60629ea1148fep-1 },
  { 0x1.00c0906c513cfp-1, 0x1.61639fa77b069p-1 }, { 0x1.0040100401004p-1, 0x1.62641fecf8743p-1 },
};

/* E ln2 for E = 0..63 */
static __device__ const double ncg_eln2_tab[64] = {
  0x0.0p+0, 0x1.62e42fefa39efp-1, 0x1.62e42fefa39efp+0, 0x1.0a2b23f3bab73p+1,
  0x1.62e42fefa39efp+1, 0x1.bb9d3beb8c86bp+1, 0x1.0a2b23f3bab73p+2, 0x1.3687a9f1af2b1p+2,
  0x1.62e42fefa39efp+2, 0x1.8f40b5ed9812dp+2, 0x1.bb9d3beb8c86bp+2, 0x1.e7f9c1e980fa9p+2,
  0x1.0a2b23f3bab73p+3, 0x1.205966f2b4f12p+3, 0x1.3687a9f1af2b1p+3, 0x1.4cb5ecf0a9650p+3,
  0x1.62e42fefa39efp+3, 0x1.791272ee9dd8ep+3, 0x1.8f40b5ed9812dp+3, 0x1.a56ef8ec924ccp+3,
  0x1.bb9d3beb8c86bp+3, 0x1.d1cb7eea86c0ap+3, 0x1.e7f9c1e980fa9p+3, 0x1.fe2804e87b348p+3,
  0x1.0a2b23f3bab73p+4, 0x1.1542457337d43p+4, 0x1.205966f2b4f12p+4, 0x1.2b708872320e2p+4,
  0x1.3687a9f1af2b1p+4, 0x1.419ecb712c481p+4, 0x1.4cb5ecf0a9650p+4, 0x1.57cd0e7026820p+4,
  0x1.62e42fefa39efp+4, 0x1.6dfb516f20bbfp+4, 0x1.791272ee9dd8ep+4, 0x1.8429946e1af5ep+4,
  0x1.8f40b5ed9812dp+4, 0x1.9a57d76d152fdp+4, 0x1.a56ef8ec924ccp+4, 0x1.b0861a6c0f69cp+4,
  0x1.bb9d3beb8c86bp+4, 0x1.c6b45d6b09a3ap+4, 0x1.d1cb7eea86c0ap+4, 0x1.dce2a06a03dd9p+4,
  0x1.e7f9c1e980fa9p+4, 0x1.f310e368fe178p+4, 0x1.fe2804e87b348p+4, 0x1.049f9333fc28cp+5,
  0x1.0a2b23f3bab73p+5, 0x1.0fb6b4b37945bp+5, 0x1.1542457337d43p+5, 0x1.1acdd632f662bp+5,
  0x1.205966f2b4f12p+5, 0x1.25e4f7b2737fap+5, 0x1.2b708872320e2p+5, 0x1.30fc1931f09cap+5,
  0x1.3687a9f1af2b1p+5, 0x1.3c133ab16db99p+5, 0x1.419ecb712c481p+5, 0x1.472a5c30ead69p+5,
  0x1.4cb5ecf0a9650p+5, 0x1.52417db067f38p+5, 0x1.57cd0e7026820p+5, 0x1.5d589f2fe5107p+5,
};

/* exp(t) for t <= 700 or so as a scaled table value T and the polynomial p:
 * exp(t) = T + T p.  T = 0 for t < -700 (a term that small never counts beside
 * the maximum of its sum) and for NaN. */
static __device__ __forceinline__ void
ncg_exp_parts (double t, double *T, double *p)
{
  const double z  = fma (t, 0x1.71547652b82fep+8, 0x1.8p+52);     /* 256/ln2 */
  const int k     = __double2loint (z);
  const double f  = fma (z - 0x1.8p+52, -0x1.62e42fefa39efp-9, t);   /* ln2/256 */
  const double q  = f * f;
  const double h  = fma (f, fma (f, 0x1.5555555555555p-5, 0x1.5555555555555p-3), 0.5);
  const double tj = __ldg (ncg_exp2_tab + (k & 255));
  /* t < -700 or NaN, from the high word alone (no FP64 compare) */
  const uint32_t hi = (uint32_t) __double2hiint (t);
  const bool zero   = hi >= 0xc085e000u || (hi & 0x7fffffffu) >= 0x7ff00000u;

  *p = fma (q, h, f);
  *T = zero ? 0.0 : __hiloint2double (__double2hiint (tj) + ((k >> 8) << 20), __double2loint (tj));

  if (zero)
    *p = 0.0;
}

/* exp(t), t <= 700 */
static __device__ __forceinline__ double
ncg_exp (double t)
{
  double T, p;

  ncg_exp_parts (t, &T, &p);

  return fma (T, p, T);
}

/* exp(t + tl), tl far below 1, to about an ulp down to the subnormals, t <= 700: ln2/256 as two
 * doubles, the scaling in two steps */
static __device__ __forceinline__ double
ncg_exp_full (double t, double tl = -0.0)
{
  const uint32_t hi = (uint32_t) __double2hiint (t);

  if (hi >= 0xc0874a00u && hi <= 0xfff00000u)
    return 0.0;

  if ((hi & 0x7fffffffu) >= 0x7ff00000u)
    return t;   /* +inf, NaN */

  const double z  = fma (t, 0x1.71547652b82fep+8, 0x1.8p+52);
  const int k     = __double2loint (z);
  const double kd = z - 0x1.8p+52;
  const double f  = fma (kd, -0x1.abc9e3b39803fp-64, fma (kd, -0x1.62e42fefa39efp-9, t)) + tl;
  const double q  = f * f;
  const double h  = fma (f, fma (f, 0x1.5555555555555p-5, 0x1.5555555555555p-3), 0.5);
  const double tj = __ldg (ncg_exp2_tab + (k & 255));
  const double v  = fma (tj, fma (q, h, f), tj);
  const int e     = k >> 8;

  if (__builtin_expect (e >= -1021, 1))
    return __hiloint2double (__double2hiint (v) + (e << 20), __double2loint (v));

  return __hiloint2double (__double2hiint (v) + ((e + 200) << 20), __double2loint (v)) * 0x1p-200;
}

/* log(u) for u >= 1; +inf for u = +inf, NaN for NaN */
static __device__ __forceinline__ double
ncg_log_ge1 (double u)
{
  const int hi    = __double2hiint (u);
  const int E     = ((hi >> 20) & 0x7ff) - 1023;   /* a NaN of either sign: 1024 */
  const double2 c = __ldg (ncg_log_tab + ((hi >> 12) & 255));
  const double m  = __hiloint2double ((hi & 0x000fffff) | 0x3ff00000, __double2loint (u));
  const double r  = fma (m, c.x, -1.0);
  const double h  = fma (r, fma (r, fma (r, 0x1.999999999999ap-3, -0.25), 0x1.5555555555555p-2), -0.5);
  const double p  = fma (r * r, h, r);

  if (__builtin_expect ((uint32_t) E < 64u, 1))
    return (__ldg (ncg_eln2_tab + E) + c.y) + p;

  if (E == 1024)
    return u;   /* inf, NaN */

  return fma ((double) E, 0x1.62e42fefa39efp-1, c.y) + p;
}

/* -log c_j less its double in ncg_log_tab */
static __device__ const double ncg_log_lo_tab[256] = {
  0x1.e29e3a153e432p-64, 0x1.3c2d23a074505p-63, 0x1.600d65eebbc60p-61, -0x1.7b4213447a4ccp-61,
  0x1.2be019c2d240ep-61, -0x1.885b61f610d84p-63, -0x1.cbf63e207e981p-60, 0x1.4b2c67dcd0956p-60,
  -0x1.c5bc089e0b23bp-59, 0x1.042b74e00f373p-60, -0x1.9d6a40b6e333bp-59, 0x1.19f3f276b596dp-59,
  -0x1.284d2b1a4a1edp-60, -0x1.4502014926cd6p-59, -0x1.4d9501f1df1d3p-59, 0x1.a66e7585e8241p-59,
  0x1.ba13162a9c44ep-60, 0x1.1e4add513114dp-58, 0x1.7d7a7a2605718p-58, -0x1.34d66a3f7a2b6p-58,
  0x1.44d6a6b9dad0cp-58, -0x1.9308973e22a83p-61, -0x1.42a375515892ep-58, 0x1.d2da7bd644829p-59,
  0x1.cff28ef6a5931p-58, -0x1.f491a5df236ecp-58, -0x1.e463f9e4dd91fp-59, 0x1.76df97bcb1787p-60,
  -0x1.89f383dad0d65p-58, 0x1.d248382a5ecffp-62, -0x1.64af228bcf63ap-60, -0x1.9d4a8f3f05aa5p-59,
  0x1.a227143a5a99ap-58, 0x1.38176812fe880p-59, -0x1.652e70072e4b1p-57, -0x1.aae2afa34f48ap-58,
  0x1.cf798d39f1b7dp-58, -0x1.f52f6c3723f80p-57, 0x1.837097648f581p-58, 0x1.14f176448b993p-60,
  0x1.dcdca01dc0febp-57, 0x1.f28bf9ca923d6p-58, 0x1.bbbeaea81ece2p-57, -0x1.1e103f093930dp-58,
  0x1.b1391fb1b4b22p-57, 0x1.24140543648f3p-58, -0x1.4644b3703041cp-57, -0x1.1919a4664319dp-57,
  -0x1.0ea8fd38a2c66p-58, 0x1.28891a29eac08p-57, -0x1.de12ad4822814p-57, 0x1.440d1e78f44cep-57,
  -0x1.d9f13877e61b9p-57, -0x1.16fa715e8d38bp-59, 0x1.610816ebe4976p-57, -0x1.f28442017473fp-57,
  0x1.0593750fffe78p-58, -0x1.9fb3f9cdff9d3p-57, -0x1.966bc4ca8938dp-57, 0x1.2b1a83b18de21p-58,
  0x1.1adf25feae309p-57, 0x1.9990bc47005e0p-59, -0x1.beb83c874aaf3p-57, -0x1.44269756071afp-58,
  0x1.cd329bc9d42b1p-64, -0x1.204a2aa97ac8ep-58, 0x1.d01e4d9c3e3a7p-57, -0x1.4f486fc6e8c8ap-64,
  -0x1.daf3c7a62832cp-57, -0x1.9987ee52650b9p-60, -0x1.98a0bf20f9d99p-59, 0x1.8d2b5b2204b4cp-57,
  0x1.6e32d5e8c7080p-57, -0x1.6bb183e51ec40p-56, 0x1.e9432dc9528f1p-56, 0x1.2140c5a328e6dp-56,
  -0x1.2333a23204a40p-56, 0x1.0b5e955ff414ep-59, 0x1.97b8198d22e05p-56, 0x1.a6880da1b13e4p-58,
  0x1.1458b5d97ba9dp-56, -0x1.b26dc55e2d052p-56, 0x1.154d86a4ff98bp-59, -0x1.3a2eb579e2857p-59,
  -0x1.99bae06a5c863p-61, -0x1.0e09ea9b4c4a4p-56, 0x1.895c18aa47a54p-57, 0x1.f3ee1106a6ca7p-57,
  -0x1.95d2280d51407p-58, -0x1.263d5c1f755e9p-56, 0x1.8d8af2d5b0557p-59, 0x1.2d733ea6502f0p-56,
  0x1.06d1e3224d3e9p-57, -0x1.0c4f82601ebfap-60, -0x1.8027c87f91214p-57, -0x1.430c8309edcfcp-56,
  -0x1.1c0f372f6825bp-57, -0x1.51d7e6a892849p-57, 0x1.cb3fe83434321p-56, -0x1.bc78b7cdae677p-56,
  -0x1.c4826ceaff1c8p-56, -0x1.81de37d2989eep-56, -0x1.24f586adeb499p-57, 0x1.ec1e3016fc9f5p-58,
  -0x1.fa7088c705f8ap-56, -0x1.e15bd0fed391dp-56, -0x1.d617f8a08338cp-58, 0x1.b9b7b9e219186p-56,
  -0x1.fc80d000b4083p-57, -0x1.5e8e76dd346a0p-56, -0x1.fc083df227104p-59, 0x1.4caf721f626aap-57,
  0x1.a748662fc4171p-56, -0x1.29943804dfbeep-56, -0x1.9a576c0601322p-58, -0x1.58f8f27d8e90fp-57,
  -0x1.306488dd76781p-58, -0x1.dc45997fbc413p-56, 0x1.7cab36811fa33p-57, -0x1.f4419b612c65ap-57,
  0x1.9f4fca257a85dp-57, -0x1.51ec4c14526a6p-56, 0x1.dd8e962c0c0adp-56, -0x1.02711f5645823p-57,
  -0x1.f3c3fbbc738aap-57, -0x1.951ec6ae7473ep-58, 0x1.6ef49cf67f73bp-56, 0x1.0f947c24d6d15p-57,
  -0x1.66f70bc45a4eap-56, 0x1.a254f268e3b77p-57, -0x1.83875c3d29410p-56, 0x1.11178481c3254p-57,
  0x1.027ed837c8098p-56, 0x1.db9250ec7d6c0p-56, 0x1.49cdf84b4963bp-59, 0x1.2d4ebe6b64659p-57,
  0x1.46b9d39edb329p-56, 0x1.46a03ad42b053p-58, -0x1.b230b0b86cdb3p-56, -0x1.b575624ae2937p-56,
  0x1.42e6254debd1ap-56, -0x1.7f81655ffb866p-57, 0x1.6a615815805b6p-56, 0x1.b5ac6bcf865f1p-60,
  0x1.490f7d8320aa6p-56, 0x1.555ccfd34e773p-56, -0x1.392469ec4f2d1p-57, 0x1.6b1ca5b4c2326p-57,
  0x1.894972adf9532p-58, -0x1.f73153d5f3576p-58, -0x1.5033e78d17001p-56, -0x1.fc1498cd5f810p-59,
  0x1.866ba1f8898b2p-58, 0x1.0af58040358ccp-56, -0x1.f2180135bc9e9p-57, -0x1.e1ea13f7bb73cp-56,
  -0x1.2c2a607f4211fp-56, -0x1.ae71b7919fe41p-62, -0x1.f987ff7ff1891p-56, 0x1.7694d500702eep-56,
  -0x1.a045e49ba251ep-56, 0x1.259465d63197dp-57, -0x1.746e0614b6c54p-60, -0x1.a1d4ac924a114p-56,
  -0x1.4070d99441964p-56, -0x1.91c292bb5006ep-57, -0x1.ac9a15ed191cdp-56, -0x1.4059e632f810ep-59,
  0x1.01637cd0c6322p-55, 0x1.b3ca7518f79eep-55, 0x1.3956e356c4427p-55, -0x1.09c4075c537f5p-57,
  0x1.b3b5da204f2b4p-56, 0x1.cbfa8aba6b01bp-56, -0x1.637129e8e65d6p-55, 0x1.9f7b2c890500ap-57,
  0x1.12b0a6bece97ep-55, 0x1.fe2b7fa595f64p-55, -0x1.d8d54bbb0dd12p-58, -0x1.a6e6efd578cdfp-57,
  0x1.e6178fa93d276p-57, -0x1.8dc202e52373bp-55, 0x1.3fd142b10a7d5p-57, -0x1.c3f0e01a37834p-55,
  -0x1.dcf909e3864ebp-58, 0x1.97a882bf8aad4p-56, -0x1.df40f54d1f054p-55, -0x1.f81c49a23f756p-58,
  -0x1.92db65c2b36abp-55, -0x1.5ff40c85bc439p-58, 0x1.f38426184f32ap-56, 0x1.5f5b45b30e302p-55,
  -0x1.abfa36e2d19f9p-55, -0x1.5cbe32567e6afp-57, 0x1.a1afa4aeb598ap-64, -0x1.3e6cde2013e20p-55,
  0x1.4d0496643f035p-55, -0x1.5dd121bc42e34p-55, -0x1.6534a9a0dcbbdp-57, -0x1.97f4edb1f37cbp-56,
  0x1.c3fb96be5d640p-57, 0x1.9899fca1425e8p-56, -0x1.5d299abea2437p-55, 0x1.d1ff94a792f17p-55,
  -0x1.d9becbb0e4322p-56, 0x1.0f3ef07774574p-55, -0x1.e9ae735118099p-55, 0x1.dbf08ade6a75ep-55,
  -0x1.1d5ba1424b05ap-58, 0x1.d7f1bd5fda3d6p-55, 0x1.ef8b734c91c5dp-56, -0x1.2ac7fe2a95992p-56,
  -0x1.7f9c5ae27b58ap-57, -0x1.45dac4b904390p-58, 0x1.bcade2e600649p-58, 0x1.24677c50b4f2fp-57,
  -0x1.c5ab543639f33p-55, 0x1.05d28c1ee028bp-58, 0x1.5f5078dc66fcap-55, 0x1.6ff71a5d46072p-55,
  -0x1.e1b74bd7dc57dp-56, -0x1.aa1f2821f7e80p-57, 0x1.e8eac4149d261p-56, 0x1.df8a528db9e2cp-57,
  -0x1.7c4d58c23cd48p-56, 0x1.32539ce2355b0p-55, -0x1.3f8369cbbe59cp-57, -0x1.a785f94848c6cp-55,
  0x1.52017a9a0ae4fp-58, -0x1.288675d0fb1f9p-55, -0x1.dbad233fb591cp-59, -0x1.4b98fa670a3fbp-58,
  -0x1.0f6379c6918c0p-55, 0x1.f7a9713105cedp-55, 0x1.284f66c1ee3bap-59, -0x1.c9dd3f2c57232p-55,
  -0x1.6ebac541fb222p-55, -0x1.f6f07ea5faf41p-56, 0x1.dc3c55b9ff703p-56, -0x1.df05830ea2cf0p-55,
  -0x1.d864d52029c26p-55, 0x1.df1ab56bd0694p-56, 0x1.addbe1cefeccdp-63, -0x1.8997c4a22e891p-55,
  -0x1.75638d706fc01p-55, -0x1.b91f884591919p-56, -0x1.1adfd04bb2ed0p-55, -0x1.38d3c3ffe9f6ep-58,
  0x1.b46dbddbb1f4dp-56, 0x1.82ea1d0142b6cp-61, -0x1.20a591b0ba580p-55, 0x1.10c88f64cc285p-55,
  -0x1.2591e1e383d79p-55, 0x1.c6a443e72f437p-57, 0x1.5c7e902d91dc0p-56, -0x1.a40dee0981e4cp-58,
};

/* log (1 + t) as x + y for t + dt >= 0 (dt far below t; t + dt may be inf or NaN): the
 * rounding of 1 + t is taken along, below 2^-8 the series runs in t itself, and above
 * it the table's and the sums' low parts are kept.  Against quadruple precision over t =
 * 2^-60 .. 2^1010 within 2^-53 of itself just above 2^-8 and 2^-61 absolutely from there on
 * (2^-58 relative below it). */
static __device__ __forceinline__ double2
ncg_log1p_dd (double t, double dt)
{
  double h, l;

  if ((uint32_t) __double2hiint (t) < 0x3f700000u)
  {
    const double a = fma (t, fma (t, 0x1.2492492492492p-3, -0x1.5555555555555p-3), 0x1.999999999999ap-3);

    h = t;
    l = fma (t * t, fma (t, fma (t, fma (t, a, -0.25), 0x1.5555555555555p-2), -0.5), dt);
  }
  else
  {
    const double u  = 1.0 + t;
    const int hi    = __double2hiint (u);
    const int E     = ((hi >> 20) & 0x7ff) - 1023;
    const double2 c = __ldg (ncg_log_tab + ((hi >> 12) & 255));

    if (E == 1024)
      return make_double2 (u, 0.0);   /* inf, NaN */

    /* 1 + t - u, exact, in units of 2^E (nothing from 2^64) */
    const double du = ((E == 0) ? t - (u - 1.0) : 1.0 - (u - t)) + dt;
    const double d  = (E < 64) ? du * __hiloint2double ((1023 - E) << 20, 0) : 0.0;
    const double m  = __hiloint2double ((hi & 0x000fffff) | 0x3ff00000, __double2loint (u));
    const double r  = fma (m, c.x, -1.0);
    const double a  = fma (r, fma (r, -0x1.5555555555555p-3, 0x1.999999999999ap-3), -0.25);
    const double q  = fma (r, fma (r, a, 0x1.5555555555555p-2), -0.5);
    /* ln2 as 42 bits and the rest: E times the first is exact */
    const double e0 = E * 0x1.62e42fefa3800p-1, s0 = e0 + c.y, f0 = c.y - (s0 - e0);
    const double s1 = s0 + r, b1 = s1 - s0, f1 = (s0 - (s1 - b1)) + (r - b1);

    h = s1;
    l = fma (r * r, q, fma (d, c.x, fma ((double) E, 0x1.ef35793c76730p-45, __ldg (ncg_log_lo_tab + ((hi >> 12) & 255)) + (f0 + f1))));
  }

  const double x = h + l;

  return make_double2 (x, l - (x - h));
}

/* ln of a Student-t term at a large nu: kappa log (1 + t) + c.  ncg_log_ge1 sees 1 + t
 * rounded, so kappa = -(nu + d) / 2 times 1.5 2^-53 is lost there: less than the
 * rounding of the result up to nu = d, 1e-9 of it at nu = 1e9. */
static __device__ __noinline__ double
ncg_lnt_wide (double t, double kappa, double c)
{
  const double2 g = ncg_log1p_dd (t, 0.0);

  return fma (kappa, g.x, fma (kappa, g.y, c));
}

/* A Student-t kernel by itself, (1 + chi^2 / nu)^kappa, for the interpolation matrix:
 * pow's accuracy, since an error of the logarithm counts kappa log u times there.  The
 * quotient's remainder and the logarithm's and the product's low parts are kept (the
 * rounded logarithm cost up to kappa (1 + 1.5 log u) units of 2^-53, pow's base kappa). */
static __device__ __noinline__ double
ncg_st_power (double chi2, double nu, double inv_nu, double kappa)
{
  const double t  = chi2 * inv_nu;
  const double2 g = ncg_log1p_dd (t, fma (-t, nu, chi2) * inv_nu);
  const double p  = kappa * g.x;

  return ncg_exp_full (p, fma (kappa, g.x, -p) + kappa * g.y);
}

/* The nu that take ncg_lnt_wide, by a kernel of their own (KERN = NCG_KERNEL_ST_WIDE): as a branch on
 * a launch constant in the one for small nu it cost that one 2 % (d = 16, 8192 x 8192
 * 3.18 -> 3.25 ms), although it never ran.  Their own time: nu = 8 | 40 at d = 16, 8192
 * kernels, 500 points in tiles 1.47 | 1.68 ms, 8192 points in sliced products 3.13 | 6.33;
 * d = 8, 2000 kernels, 500 points 194 | 246 us.  The line: up to nu = d the lost digits are
 * below the rounding of the sum itself ((nu + d) / 2 <= 32 units of 2^-53 in a value of
 * some d), and 8 stands in for that at small d. */
#define NCG_KERNEL_ST_WIDE 2

static __host__ __device__ __forceinline__ bool
ncg_nu_wide (double nu, int d)
{
  return nu > 8.0 && nu > (double) d;
}

/* One sum over kernels kept as (g, s): the terms added so far are
 * s exp(g).  g follows the largest term closely enough (within 4) that
 * g + log s loses nothing against the maximum itself; it starts at the lowest
 * double with s = 0, where an empty sum or one of -inf terms stays. */
#define NCG_LSE_EMPTY (-0x1.fffffffffffffp+1023)

static __device__ __forceinline__ void
ncg_lse_add (double lnt, double &g, double &s)
{
  double t = lnt - g;

  /* t >= 4, not inf or NaN (an infinite or NaN term is left out): rescale; rare once g is near the maximum */
  if ((uint32_t) __double2hiint (t) - 0x40100000u < 0x7ff00000u - 0x40100000u)
  {
    s *= ncg_exp (-t);
    g = lnt;
    t = 0.0;
  }

  double T, p;

  ncg_exp_parts (t, &T, &p);
  s = fma (T, p, s + T);
}

/* the FP32 forms' (gamma, lambda) pair -- the sum is (lambda + 1) exp(gamma),
 * gamma = -inf for an empty one -- as (g, s) */
static __device__ __forceinline__ double2
ncg_lse_pair (float2 q)
{
  return (q.x > -CUDART_INF_F) ? make_double2 ((double) q.x, (double) q.y + 1.0) : make_double2 (NCG_LSE_EMPTY, 0.0);
}

/* ln of the density from its sum s exp(g): the constant taken out of the
 * mixed operand (dshift, may be NULL), the KDE's common lnnorm (shift) and d ln h */
static __device__ __forceinline__ double
ncg_lse_lnp (double g, double s, double shift, const double *dshift, double d_ln_href)
{
  const double gamma = g - shift + (dshift ? *dshift : 0.0);

  return gamma + log (s) - d_ln_href;
}

#endif /* NCG_FASTMATH_CUH */
