// exp2_table.cuh -- 2^x in FP64 with a table, for the integrands: 2^(i / 256) as
// a sum of two doubles, and the Taylor coefficients of 2^(u / 256).
#pragma once

namespace sfsim {

__device__ const double2 kExp2Table[256] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.00b1afa5abcbfp+0, -0x1.4f6b2a7609f71p-55},
    {0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54}, {0x1.02168143b0281p+0, -0x1.2bf310fc54eb6p-55},
    {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56}, {0x1.037d42e11bbccp+0, 0x1.56811eeade11ap-57},
    {0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54}, {0x1.04e5f72f654b1p+0, 0x1.4c3793aa0d08dp-55},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55}, {0x1.0650a0e3c1f89p+0, -0x1.5cb7b5799c397p-54},
    {0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55}, {0x1.07bd42b72a836p+0, 0x1.3233454458700p-55},
    {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57}, {0x1.092bdf66607e0p+0, -0x1.68063800a3fd1p-54},
    {0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54}, {0x1.0a9c79b1f3919p+0, 0x1.5d16c873d1d38p-55},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0c0f145e46c85p+0, 0x1.4f98906d21cefp-54},
    {0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54}, {0x1.0d83b23395decp+0, -0x1.bc14de43f316ap-54},
    {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59}, {0x1.0efa55fdfa9c5p+0, -0x1.49db9bc54021bp-54},
    {0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57}, {0x1.1073028d7233ep+0, 0x1.d46eb1692fdd5p-55},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.11edbab5e2ab6p+0, -0x1.ca454f703fb72p-54},
    {0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58}, {0x1.136a814f204abp+0, -0x1.7108fba48dcf0p-57},
    {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54}, {0x1.14e95934f312ep+0, -0x1.b91e839bf44abp-55},
    {0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55}, {0x1.166a45471c3c2p+0, 0x1.8f23b82ea1a32p-58},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.17ed48695bbc0p+0, 0x1.09e3fe2ac5a64p-56},
    {0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54}, {0x1.1972658375d2fp+0, 0x1.4aadd85f17e08p-54},
    {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55}, {0x1.1af99f8138a1cp+0, 0x1.7bf85a4b69280p-54},
    {0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54}, {0x1.1c82f95281c6bp+0, 0x1.009778010f8c9p-54},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.1e0e75eb44027p+0, -0x1.6fdd8088cb6dep-54},
    {0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54}, {0x1.1f9c18438ce4dp+0, -0x1.bf524a097af5cp-54},
    {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55}, {0x1.212be3578a819p+0, 0x1.3592d2cfcaac9p-54},
    {0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55}, {0x1.22bdda27912d1p+0, 0x1.d34fb5577d69fp-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.2451ffb82140ap+0, 0x1.acfcc911ca996p-55},
    {0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55}, {0x1.25e85711ece75p+0, 0x1.3e1a24ac31b2cp-54},
    {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55}, {0x1.2780e341ddf29p+0, 0x1.e067c05f9e76cp-54},
    {0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54}, {0x1.291ba7591bb70p+0, -0x1.2cc7228401cbdp-55},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55}, {0x1.2ab8a66d10f13p+0, -0x1.95743191690a7p-54},
    {0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59}, {0x1.2c57e39771b2fp+0, -0x1.50145a6eb5124p-54},
    {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54}, {0x1.2df961f641589p+0, 0x1.d16cffbbce198p-54},
    {0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56}, {0x1.2f9d24abd886bp+0, -0x1.53c55532bda93p-57},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.31432edeeb2fdp+0, 0x1.959a3f3f3fcd1p-55},
    {0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55}, {0x1.32eb83ba8ea32p+0, -0x1.c45e83cb4f318p-54},
    {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54}, {0x1.3496266e3fa2dp+0, -0x1.35a75930881a4p-55},
    {0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55}, {0x1.36431a2de883bp+0, -0x1.c3144a06cb85ep-55},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.37f26231e754ap+0, -0x1.9f5ca9eceb23cp-54},
    {0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54}, {0x1.39a401b7140efp+0, -0x1.9a9a5fc8e2934p-54},
    {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56}, {0x1.3b57fbfec6cf4p+0, 0x1.54c66e26fff18p-54},
    {0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54}, {0x1.3d0e544ede173p+0, 0x1.fe8d08c284c71p-56},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.3ec70df1c5175p+0, -0x1.af6637b8c9bcap-55},
    {0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54}, {0x1.40822c367a024p+0, 0x1.bddf8b6f4d048p-55},
    {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58}, {0x1.423fb2709468ap+0, -0x1.8462dc0b314ddp-54},
    {0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55}, {0x1.43ffa3f84b9d4p+0, 0x1.880be9704c003p-55},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.45c2042a7d232p+0, -0x1.8641982fb1f8ep-57},
    {0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54}, {0x1.4786d668b3237p+0, -0x1.c20f0ed445733p-54},
    {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56}, {0x1.494e1e192aed2p+0, -0x1.3b2895e499ea0p-55},
    {0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54}, {0x1.4b17dea6db7d7p+0, -0x1.125b87f2897f0p-55},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4ce41b817c114p+0, 0x1.05e29690abd5dp-54},
    {0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54}, {0x1.4eb2d81d8abffp+0, -0x1.5257d2e5d7a52p-54},
    {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54}, {0x1.508417f4531eep+0, 0x1.a249b49b7465fp-56},
    {0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55}, {0x1.5257de83f4eefp+0, -0x1.c998d43efef71p-56},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55}, {0x1.542e2f4f6ad27p+0, 0x1.7926d192d5f7ep-55},
    {0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55}, {0x1.56070dde910d2p+0, -0x1.0fb6e168eebf0p-54},
    {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54}, {0x1.57e27dbe2c4cfp+0, -0x1.0b98c8a57b9c4p-54},
    {0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55}, {0x1.59c0827ff07ccp+0, -0x1.7e2cee467e60fp-54},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5ba11fba87a03p+0, -0x1.b77a14c233e1ap-54},
    {0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60}, {0x1.5d84590998b93p+0, -0x1.cd6a7a8b45643p-54},
    {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54}, {0x1.5f6a320dceb71p+0, -0x1.9eadde3cdcf92p-55},
    {0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54}, {0x1.6152ae6cdf6f4p+0, 0x1.e4b3e4ab84c27p-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.633dd1d1929fdp+0, 0x1.84710beb964e5p-54},
    {0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55}, {0x1.652b9febc8fb7p+0, -0x1.ae3d5c9a73e09p-54},
    {0x1.6623882552225p+0, -0x1.bb60987591c34p-54}, {0x1.671c1c70833f6p+0, -0x1.e8732586c6134p-55},
    {0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57}, {0x1.690f4b19e9538p+0, 0x1.804bd9aeb445dp-55},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.6b052fa75173ep+0, 0x1.a38f52c9a9d0ep-56},
    {0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56}, {0x1.6cfdcddd47645p+0, 0x1.c7aa9b6f17309p-54},
    {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57}, {0x1.6ef9298593ae5p+0, -0x1.0b9749e1ac8b2p-54},
    {0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55}, {0x1.70f7466f42e87p+0, 0x1.9d644d45aa65fp-58},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.72f8286ead08ap+0, -0x1.20aa02cd62c72p-54},
    {0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54}, {0x1.74fbd35d7cbfdp+0, 0x1.047fd618a6e1cp-54},
    {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54}, {0x1.77024b1ab6e09p+0, 0x1.b7877169147f8p-54},
    {0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54}, {0x1.790b938ac1cf6p+0, 0x1.349a862aadd3ep-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7b17b0976cfdbp+0, -0x1.bebb58468dc88p-54},
    {0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54}, {0x1.7d26a62ff86f0p+0, 0x1.1bddbfb72b8b4p-54},
    {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56}, {0x1.7f3878491c491p+0, -0x1.07f11cf9311aep-55},
    {0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54}, {0x1.814d2add106d9p+0, 0x1.464370d151d4dp-54},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54}, {0x1.8364c1eb941f7p+0, 0x1.99b9a31df2bd5p-54},
    {0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55}, {0x1.857f4179f5b21p+0, -0x1.ba748f8b216d0p-58},
    {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54}, {0x1.879cad931a436p+0, 0x1.5d2d7d2db47bdp-55},
    {0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54}, {0x1.89bd0a478580fp+0, 0x1.d53954475202bp-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8be05bad61778p+0, 0x1.ecb5efc43446ep-54},
    {0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56}, {0x1.8e06a5e0866d9p+0, -0x1.7114a6fc9b2e6p-54},
    {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55}, {0x1.902fed0282c8ap+0, 0x1.592ca85fe3fd2p-54},
    {0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54}, {0x1.925c353aa2fe2p+0, -0x1.3455fa639db7fp-55},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.948b82b5f98e5p+0, -0x1.dc3d6797d2d99p-55},
    {0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56}, {0x1.96bdd9a7670b3p+0, -0x1.ba5967f19c896p-58},
    {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54}, {0x1.98f33e47a22a2p+0, 0x1.cabdaa24c78edp-56},
    {0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54}, {0x1.9b2bb4d53fe0dp+0, -0x1.dd84e4df6d518p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.9d674194bb8d5p+0, -0x1.516bea3dd8233p-54},
    {0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56}, {0x1.9fa5e8d07f29ep+0, -0x1.4a9ceaaf1facep-55},
    {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54}, {0x1.a1e7aed8eb8bbp+0, 0x1.c6618ee8be70ep-54},
    {0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54}, {0x1.a42c980460ad8p+0, -0x1.aa780589fb120p-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a674a8af46052p+0, 0x1.50f5630670366p-57},
    {0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54}, {0x1.a8bfe53c12e59p+0, -0x1.4f867b2ba15a9p-54},
    {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54}, {0x1.ab0e521356ebap+0, 0x1.89c31dae94545p-55},
    {0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55}, {0x1.ad5ff3a3c2774p+0, 0x1.7ef3bb6b1b8e5p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.afb4ce622f2ffp+0, -0x1.4b2fc0f315ecdp-54},
    {0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54}, {0x1.b20ce6c9a8952p+0, 0x1.4dd024a0756ccp-54},
    {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57}, {0x1.b468415b749b1p+0, -0x1.f763de9df7c90p-56},
    {0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54}, {0x1.b6c6e29f1c52ap+0, 0x1.2a8f352883f6ep-54},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56}, {0x1.b928cf22749e4p+0, -0x1.b721654cb65c6p-54},
    {0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54}, {0x1.bb8e0b79a6f1fp+0, -0x1.f52d1c9696205p-60},
    {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55}, {0x1.bdf69c3f3a207p+0, -0x1.c262360ea5b52p-60},
    {0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54}, {0x1.c06286141b33dp+0, -0x1.d8a5aa1fbca34p-55},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c2d1cd9fa652cp+0, -0x1.6e51617c8a5d7p-54},
    {0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54}, {0x1.c544778fafb22p+0, 0x1.12f072493b5afp-54},
    {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54}, {0x1.c7ba88988c933p+0, -0x1.e76bbbe255559p-55},
    {0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56}, {0x1.ca3405751c4dbp+0, -0x1.7f2bed10d08f5p-55},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.ccb0f2e6d1675p+0, -0x1.d220f86009093p-56},
    {0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55}, {0x1.cf3155b5bab74p+0, -0x1.a08e9b86dff57p-54},
    {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54}, {0x1.d1b532b08c968p+0, 0x1.55636219a36eep-54},
    {0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54}, {0x1.d43c8eacaa1d6p+0, 0x1.3db53bf5a1614p-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.d6c76e862e6d3p+0, 0x1.fe87a4a8165a0p-58},
    {0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54}, {0x1.d955d71ff6075p+0, 0x1.a052dbb9af6bep-54},
    {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54}, {0x1.dbe7cd63a8315p+0, -0x1.b76f1926b8be4p-54},
    {0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54}, {0x1.de7d5641c0658p+0, -0x1.ca5528e79ba8fp-54},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e11676b197d17p+0, -0x1.2b529bd5c7f44p-56},
    {0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54}, {0x1.e3b333b16ee12p+0, -0x1.9f4a431fdc68bp-54},
    {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55}, {0x1.e653924676d76p+0, -0x1.63ff87522b735p-55},
    {0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54}, {0x1.e8f7977cdb740p+0, -0x1.1089480b054b1p-54},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.eb9f4867cca6ep+0, 0x1.4832f2293e4f2p-54},
    {0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54}, {0x1.ee4aaa2188510p+0, 0x1.1c68da487568dp-54},
    {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54}, {0x1.f0f9c1cb6412ap+0, -0x1.3220065181d45p-54},
    {0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54}, {0x1.f3ac948dd7274p+0, -0x1.95a5a3ed837dep-56},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54}, {0x1.f6632798844f8p+0, 0x1.fa37b3539343ep-54},
    {0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54}, {0x1.f91d802243c89p+0, -0x1.12ea8a779f689p-57},
    {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55}, {0x1.fbdba3692d514p+0, -0x1.9677315098eb6p-56},
    {0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57}, {0x1.fe9d96b2a23d9p+0, 0x1.4a6037442fde3p-56},
};

// 2^x by the table-driven method (P. T. P. Tang, ACM TOMS 15, 1989).  For |x| <
// 1000, x = (k + u) / 256 with k whole and |u| <= 1/2, so 2^x = 2^(k >> 8)
// 2^((k & 255) / 256) 2^(u / 256), the last by its Taylor series to u^4
// (truncated below 4e-17).  In 11 FP64 operations; GB300 runs two a clock and
// SM, and the library's exp2() was half of the FP64 integrals' operations: the
// first order of 8x16x8x4 tables with 64 steps 1.44 -> 1.09 ms, a build 2.11 ->
// 1.65 (1.54 with what came later).  Largest error over [-200, 0] against long double 0.81 ulp, exp2() 0.84.
__device__ __forceinline__ double exp2_table(double x) {
  if ((__double2hiint(x) & 0x7fffffff) >= 0x408f4000) return exp2(x);  // |x| >= 1000, infinities, NaN
  const double y = x * 256.0;                         // exact
  const double m = __dadd_rn(y, 6755399441055744.0);  // 1.5 2^52: the low bits are round(y)
  const int k = __double2loint(m);
  const double u = y - __dadd_rn(m, -6755399441055744.0);
  double p = 0x1.3b2ab6fba4e77p-39;
  p = fma(p, u, 0x1.c6b08d704a0c0p-29);
  p = fma(p, u, 0x1.ebfbdff82c58fp-19);
  p = fma(p, u, 0x1.62e42fefa39efp-9);
  const double2 t = kExp2Table[k & 255];
  const double r = __dadd_rn(t.x, fma(t.x, u * p, t.y));
  return __hiloint2double(__double2hiint(r) + ((k >> 8) << 20), __double2loint(r));
}

}  // namespace sfsim
