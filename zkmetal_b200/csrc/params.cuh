// Generated by zkmetal_b200/gen_params.py -- do not edit by hand.
// All values are derived from the curve definitions in that script.
#pragma once
#include <cstdint>

namespace zkmsm {

struct Bn254Fp {
    static constexpr int N = 8;
    static constexpr int BITS = 254;
    static constexpr uint32_t N0 = 0xe4866389u;
    __host__ __device__ static constexpr uint32_t N0R() { return N0; }
    __host__ __device__ static constexpr uint32_t P(int i) { return (i == 0 ? 0xd87cfd47u : (i == 1 ? 0x3c208c16u : (i == 2 ? 0x6871ca8du : (i == 3 ? 0x97816a91u : (i == 4 ? 0x8181585du : (i == 5 ? 0xb85045b6u : (i == 6 ? 0xe131a029u : (i == 7 ? 0x30644e72u : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t ONE(int i) { return (i == 0 ? 0xc58f0d9du : (i == 1 ? 0xd35d438du : (i == 2 ? 0xf5c70b3du : (i == 3 ? 0x0a78eb28u : (i == 4 ? 0x7879462cu : (i == 5 ? 0x666ea36fu : (i == 6 ? 0x9a07df2fu : (i == 7 ? 0x0e0a77c1u : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t R2(int i) { return (i == 0 ? 0x538afa89u : (i == 1 ? 0xf32cfc5bu : (i == 2 ? 0xd44501fbu : (i == 3 ? 0xb5e71911u : (i == 4 ? 0x0a417ff6u : (i == 5 ? 0x47ab1effu : (i == 6 ? 0xcab8351fu : (i == 7 ? 0x06d89f71u : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t TWO_P(int i) { return (i == 0 ? 0xb0f9fa8eu : (i == 1 ? 0x7841182du : (i == 2 ? 0xd0e3951au : (i == 3 ? 0x2f02d522u : (i == 4 ? 0x0302b0bbu : (i == 5 ? 0x70a08b6du : (i == 6 ? 0xc2634053u : (i == 7 ? 0x60c89ce5u : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t PM2(int i) { return (i == 0 ? 0xd87cfd45u : (i == 1 ? 0x3c208c16u : (i == 2 ? 0x6871ca8du : (i == 3 ? 0x97816a91u : (i == 4 ? 0x8181585du : (i == 5 ? 0xb85045b6u : (i == 6 ? 0xe131a029u : (i == 7 ? 0x30644e72u : 0u)))))))); }
};

struct Bn254Fr {
    static constexpr int N = 8;
    static constexpr int BITS = 254;
    static constexpr uint32_t N0 = 0xefffffffu;
    __host__ __device__ static constexpr uint32_t N0R() { return N0; }
    __host__ __device__ static constexpr uint32_t P(int i) { return (i == 0 ? 0xf0000001u : (i == 1 ? 0x43e1f593u : (i == 2 ? 0x79b97091u : (i == 3 ? 0x2833e848u : (i == 4 ? 0x8181585du : (i == 5 ? 0xb85045b6u : (i == 6 ? 0xe131a029u : (i == 7 ? 0x30644e72u : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t R2(int i) { return (i == 0 ? 0xae216da7u : (i == 1 ? 0x1bb8e645u : (i == 2 ? 0xe35c59e3u : (i == 3 ? 0x53fe3ab1u : (i == 4 ? 0x53bb8085u : (i == 5 ? 0x8c49833du : (i == 6 ? 0x7f4e44a5u : (i == 7 ? 0x0216d0b1u : 0u)))))))); }
    // subtractions of r that bring any 256-bit integer below r
    static constexpr int REDUCE_PASSES = 5;
};

struct Bn254Glv {
    static constexpr bool PSI = false;  // the endomorphism is phi below
    // phi(x, y) = (BETA * x, y) = LAMBDA * (x, y) on G1
    __host__ __device__ static constexpr uint32_t BETA_MONT(int i) { return (i == 0 ? 0xd782e155u : (i == 1 ? 0x71930c11u : (i == 2 ? 0xffbe3323u : (i == 3 ? 0xa6bb947cu : (i == 4 ? 0xd4741444u : (i == 5 ? 0xaa303344u : (i == 6 ? 0x26594943u : (i == 7 ? 0x2c3b3f0du : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t LAMBDA(int i) { return (i == 0 ? 0xb99c90ddu : (i == 1 ? 0x8b17ea66u : (i == 2 ? 0x8d8daaa7u : (i == 3 ? 0x5bfc4108u : (i == 4 ? 0x41a91758u : (i == 5 ? 0xb3c4d79du : (i == 6 ? 0x00000000u : (i == 7 ? 0x00000000u : 0u)))))))); }
    // lattice basis (a1, b1), (a2, b2): a + b*lambda = 0 mod r
    static constexpr int A1_NEG = 0;
    __host__ __device__ static constexpr uint32_t A1(int i) { return (i == 0 ? 0x94d213e3u : (i == 1 ? 0x89d32568u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B1_NEG = 1;
    __host__ __device__ static constexpr uint32_t B1(int i) { return (i == 0 ? 0x7d4f1128u : (i == 1 ? 0x8211bbebu : (i == 2 ? 0xeeb859fcu : (i == 3 ? 0x6f4d8248u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int A2_NEG = 0;
    __host__ __device__ static constexpr uint32_t A2(int i) { return (i == 0 ? 0x1221250bu : (i == 1 ? 0x0be4e154u : (i == 2 ? 0xeeb859fdu : (i == 3 ? 0x6f4d8248u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B2_NEG = 0;
    __host__ __device__ static constexpr uint32_t B2(int i) { return (i == 0 ? 0x94d213e3u : (i == 1 ? 0x89d32568u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    // Babai multipliers: c1 = (k*G1 + 2^255) >> 256, c2 = (k*G2 + 2^255) >> 256
    __host__ __device__ static constexpr uint32_t G1(int i) { return (i == 0 ? 0xc7e0b3d7u : (i == 1 ? 0xd91d232eu : (i == 2 ? 0x00000002u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    __host__ __device__ static constexpr uint32_t G2(int i) { return (i == 0 ? 0x391eb18eu : (i == 1 ? 0x7a7bd9d4u : (i == 2 ? 0xa773d2cfu : (i == 3 ? 0x4ccef014u : (i == 4 ? 0x00000002u : 0u))))); }
    static constexpr int HALF_BITS = 127;  // |k1|, |k2| < 2^HALF_BITS
};

struct Bn254Gen {
    __host__ __device__ static constexpr uint32_t X_MONT(int i) { return (i == 0 ? 0xc58f0d9du : (i == 1 ? 0xd35d438du : (i == 2 ? 0xf5c70b3du : (i == 3 ? 0x0a78eb28u : (i == 4 ? 0x7879462cu : (i == 5 ? 0x666ea36fu : (i == 6 ? 0x9a07df2fu : (i == 7 ? 0x0e0a77c1u : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t Y_MONT(int i) { return (i == 0 ? 0x8b1e1b3au : (i == 1 ? 0xa6ba871bu : (i == 2 ? 0xeb8e167bu : (i == 3 ? 0x14f1d651u : (i == 4 ? 0xf0f28c58u : (i == 5 ? 0xccdd46deu : (i == 6 ? 0x340fbe5eu : (i == 7 ? 0x1c14ef83u : 0u)))))))); }
    static constexpr uint32_t B = 3u;
    // DBL_C^2 = 3b (DBL_NEG 0) or -3b (DBL_NEG 1): projective doubling chains
    static constexpr int DBL_NEG = 0;
    __host__ __device__ static constexpr uint32_t DBL_C_MONT(int i) { return (i == 0 ? 0x50ad28d7u : (i == 1 ? 0x7a17caa9u : (i == 2 ? 0xe15521b9u : (i == 3 ? 0x1f6ac17au : (i == 4 ? 0x696bd284u : (i == 5 ? 0x334bea4eu : (i == 6 ? 0xce179d8eu : (i == 7 ? 0x2a1f6744u : 0u)))))))); }
};

struct Bls381Fp {
    static constexpr int N = 12;
    static constexpr int BITS = 381;
    static constexpr uint32_t N0 = 0xfffcfffdu;
    __host__ __device__ static constexpr uint32_t N0R() { return N0; }
    __host__ __device__ static constexpr uint32_t P(int i) { return (i == 0 ? 0xffffaaabu : (i == 1 ? 0xb9feffffu : (i == 2 ? 0xb153ffffu : (i == 3 ? 0x1eabfffeu : (i == 4 ? 0xf6b0f624u : (i == 5 ? 0x6730d2a0u : (i == 6 ? 0xf38512bfu : (i == 7 ? 0x64774b84u : (i == 8 ? 0x434bacd7u : (i == 9 ? 0x4b1ba7b6u : (i == 10 ? 0x397fe69au : (i == 11 ? 0x1a0111eau : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t ONE(int i) { return (i == 0 ? 0x0002fffdu : (i == 1 ? 0x76090000u : (i == 2 ? 0xc40c0002u : (i == 3 ? 0xebf4000bu : (i == 4 ? 0x53c758bau : (i == 5 ? 0x5f489857u : (i == 6 ? 0x70525745u : (i == 7 ? 0x77ce5853u : (i == 8 ? 0xa256ec6du : (i == 9 ? 0x5c071a97u : (i == 10 ? 0xfa80e493u : (i == 11 ? 0x15f65ec3u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t R2(int i) { return (i == 0 ? 0x1c341746u : (i == 1 ? 0xf4df1f34u : (i == 2 ? 0x09d104f1u : (i == 3 ? 0x0a76e6a6u : (i == 4 ? 0x4c95b6d5u : (i == 5 ? 0x8de5476cu : (i == 6 ? 0x939d83c0u : (i == 7 ? 0x67eb88a9u : (i == 8 ? 0xb519952du : (i == 9 ? 0x9a793e85u : (i == 10 ? 0x92cae3aau : (i == 11 ? 0x11988fe5u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t TWO_P(int i) { return (i == 0 ? 0xffff5556u : (i == 1 ? 0x73fdffffu : (i == 2 ? 0x62a7ffffu : (i == 3 ? 0x3d57fffdu : (i == 4 ? 0xed61ec48u : (i == 5 ? 0xce61a541u : (i == 6 ? 0xe70a257eu : (i == 7 ? 0xc8ee9709u : (i == 8 ? 0x869759aeu : (i == 9 ? 0x96374f6cu : (i == 10 ? 0x72ffcd34u : (i == 11 ? 0x340223d4u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t PM2(int i) { return (i == 0 ? 0xffffaaa9u : (i == 1 ? 0xb9feffffu : (i == 2 ? 0xb153ffffu : (i == 3 ? 0x1eabfffeu : (i == 4 ? 0xf6b0f624u : (i == 5 ? 0x6730d2a0u : (i == 6 ? 0xf38512bfu : (i == 7 ? 0x64774b84u : (i == 8 ? 0x434bacd7u : (i == 9 ? 0x4b1ba7b6u : (i == 10 ? 0x397fe69au : (i == 11 ? 0x1a0111eau : 0u)))))))))))); }
};

struct Bls381Fr {
    static constexpr int N = 8;
    static constexpr int BITS = 255;
    static constexpr uint32_t N0 = 0xffffffffu;
    __host__ __device__ static constexpr uint32_t N0R() { return N0; }
    __host__ __device__ static constexpr uint32_t P(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0xffffffffu : (i == 2 ? 0xfffe5bfeu : (i == 3 ? 0x53bda402u : (i == 4 ? 0x09a1d805u : (i == 5 ? 0x3339d808u : (i == 6 ? 0x299d7d48u : (i == 7 ? 0x73eda753u : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t R2(int i) { return (i == 0 ? 0xf3f29c6du : (i == 1 ? 0xc999e990u : (i == 2 ? 0x87925c23u : (i == 3 ? 0x2b6cedcbu : (i == 4 ? 0x7254398fu : (i == 5 ? 0x05d31496u : (i == 6 ? 0x9f59ff11u : (i == 7 ? 0x0748d9d9u : 0u)))))))); }
    // subtractions of r that bring any 256-bit integer below r
    static constexpr int REDUCE_PASSES = 2;
};

struct Bls381Glv {
    static constexpr bool PSI = false;  // the endomorphism is phi below
    // phi(x, y) = (BETA * x, y) = LAMBDA * (x, y) on G1
    __host__ __device__ static constexpr uint32_t BETA_MONT(int i) { return (i == 0 ? 0x8671f071u : (i == 1 ? 0xcd03c9e4u : (i == 2 ? 0x1fcda5d2u : (i == 3 ? 0x5dab2246u : (i == 4 ? 0xd3851b95u : (i == 5 ? 0x587042afu : (i == 6 ? 0x01bacb9eu : (i == 7 ? 0x8eb60ebeu : (i == 8 ? 0x83d050d2u : (i == 9 ? 0x03f97d6eu : (i == 10 ? 0x54638741u : (i == 11 ? 0x18f02065u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t LAMBDA(int i) { return (i == 0 ? 0xffffffffu : (i == 1 ? 0x00000000u : (i == 2 ? 0x0001a402u : (i == 3 ? 0xac45a401u : (i == 4 ? 0x00000000u : (i == 5 ? 0x00000000u : (i == 6 ? 0x00000000u : (i == 7 ? 0x00000000u : 0u)))))))); }
    // lattice basis (a1, b1), (a2, b2): a + b*lambda = 0 mod r
    static constexpr int A1_NEG = 0;
    __host__ __device__ static constexpr uint32_t A1(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B1_NEG = 0;
    __host__ __device__ static constexpr uint32_t B1(int i) { return (i == 0 ? 0x00000000u : (i == 1 ? 0x00000001u : (i == 2 ? 0x0001a402u : (i == 3 ? 0xac45a401u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int A2_NEG = 0;
    __host__ __device__ static constexpr uint32_t A2(int i) { return (i == 0 ? 0xffffffffu : (i == 1 ? 0x00000000u : (i == 2 ? 0x0001a402u : (i == 3 ? 0xac45a401u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B2_NEG = 1;
    __host__ __device__ static constexpr uint32_t B2(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    // Babai multipliers: c1 = (k*G1 + 2^255) >> 256, c2 = (k*G2 + 2^255) >> 256
    __host__ __device__ static constexpr uint32_t G1(int i) { return (i == 0 ? 0x00000002u : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    __host__ __device__ static constexpr uint32_t G2(int i) { return (i == 0 ? 0xf6cfee30u : (i == 1 ? 0x63f6e522u : (i == 2 ? 0xe01faaddu : (i == 3 ? 0x7c6becf1u : (i == 4 ? 0x00000001u : 0u))))); }
    static constexpr int HALF_BITS = 128;  // |k1|, |k2| < 2^HALF_BITS
};

struct Bls381Gen {
    __host__ __device__ static constexpr uint32_t X_MONT(int i) { return (i == 0 ? 0xfd530c16u : (i == 1 ? 0x5cb38790u : (i == 2 ? 0x9976fff5u : (i == 3 ? 0x7817fc67u : (i == 4 ? 0x143ba1c1u : (i == 5 ? 0x154f95c7u : (i == 6 ? 0xf3d0e747u : (i == 7 ? 0xf0ae6acdu : (i == 8 ? 0x21dbf440u : (i == 9 ? 0xedce6eccu : (i == 10 ? 0x9e0bfb75u : (i == 11 ? 0x12017741u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t Y_MONT(int i) { return (i == 0 ? 0x0ce72271u : (i == 1 ? 0xbaac93d5u : (i == 2 ? 0x7918fd8eu : (i == 3 ? 0x8c22631au : (i == 4 ? 0x570725ceu : (i == 5 ? 0xdd595f13u : (i == 6 ? 0x50405194u : (i == 7 ? 0x51ac5829u : (i == 8 ? 0xad0059c0u : (i == 9 ? 0x0e1c8c3fu : (i == 10 ? 0x5008a26au : (i == 11 ? 0x0bbc3efcu : 0u)))))))))))); }
    static constexpr uint32_t B = 4u;
    // DBL_C^2 = 3b (DBL_NEG 0) or -3b (DBL_NEG 1): projective doubling chains
    static constexpr int DBL_NEG = 1;
    __host__ __device__ static constexpr uint32_t DBL_C_MONT(int i) { return (i == 0 ? 0xe6303e44u : (i == 1 ? 0x3bd8d86du : (i == 2 ? 0x20a968aeu : (i == 3 ? 0x697376c8u : (i == 4 ? 0xd282a50du : (i == 5 ? 0x4ad2b457u : (i == 6 ? 0xcd8e9378u : (i == 7 ? 0x3056d97eu : (i == 8 ? 0x3fd6f0e7u : (i == 9 ? 0xfab1c35cu : (i == 10 ? 0x126f8172u : (i == 11 ? 0x0c592c60u : 0u)))))))))))); }
};

#ifdef __CUDACC__
static __constant__ uint32_t Bls377Fp_N0_MEM = 0xffffffffu;
#endif
struct Bls377Fp {
    static constexpr int N = 12;
    static constexpr int BITS = 377;
    static constexpr uint32_t N0 = 0xffffffffu;
#ifdef __CUDACC__
    __device__ static uint32_t N0R() { return Bls377Fp_N0_MEM; }
#endif
    __host__ __device__ static constexpr uint32_t P(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x8508c000u : (i == 2 ? 0x30000000u : (i == 3 ? 0x170b5d44u : (i == 4 ? 0xba094800u : (i == 5 ? 0x1ef3622fu : (i == 6 ? 0x00f5138fu : (i == 7 ? 0x1a22d9f3u : (i == 8 ? 0x6ca1493bu : (i == 9 ? 0xc63b05c0u : (i == 10 ? 0x17c510eau : (i == 11 ? 0x01ae3a46u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t ONE(int i) { return (i == 0 ? 0xffffff68u : (i == 1 ? 0x02cdffffu : (i == 2 ? 0x7fffffb1u : (i == 3 ? 0x51409f83u : (i == 4 ? 0x8a7d3ff2u : (i == 5 ? 0x9f7db3a9u : (i == 6 ? 0x6e7c6305u : (i == 7 ? 0x7b4e97b7u : (i == 8 ? 0x803c84e8u : (i == 9 ? 0x4cf495bfu : (i == 10 ? 0xe2fdf49au : (i == 11 ? 0x008d6661u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t R2(int i) { return (i == 0 ? 0x9400cd22u : (i == 1 ? 0xb786686cu : (i == 2 ? 0xb00431b1u : (i == 3 ? 0x0329fcaau : (i == 4 ? 0x62d6b46du : (i == 5 ? 0x22a5f111u : (i == 6 ? 0x827dc3acu : (i == 7 ? 0xbfdf7d03u : (i == 8 ? 0x41790bf9u : (i == 9 ? 0x837e92f0u : (i == 10 ? 0x1e914b88u : (i == 11 ? 0x006dfccbu : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t TWO_P(int i) { return (i == 0 ? 0x00000002u : (i == 1 ? 0x0a118000u : (i == 2 ? 0x60000001u : (i == 3 ? 0x2e16ba88u : (i == 4 ? 0x74129000u : (i == 5 ? 0x3de6c45fu : (i == 6 ? 0x01ea271eu : (i == 7 ? 0x3445b3e6u : (i == 8 ? 0xd9429276u : (i == 9 ? 0x8c760b80u : (i == 10 ? 0x2f8a21d5u : (i == 11 ? 0x035c748cu : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t PM2(int i) { return (i == 0 ? 0xffffffffu : (i == 1 ? 0x8508bfffu : (i == 2 ? 0x30000000u : (i == 3 ? 0x170b5d44u : (i == 4 ? 0xba094800u : (i == 5 ? 0x1ef3622fu : (i == 6 ? 0x00f5138fu : (i == 7 ? 0x1a22d9f3u : (i == 8 ? 0x6ca1493bu : (i == 9 ? 0xc63b05c0u : (i == 10 ? 0x17c510eau : (i == 11 ? 0x01ae3a46u : 0u)))))))))))); }
};

struct Bls377Fr {
    static constexpr int N = 8;
    static constexpr int BITS = 253;
    static constexpr uint32_t N0 = 0xffffffffu;
    __host__ __device__ static constexpr uint32_t N0R() { return N0; }
    __host__ __device__ static constexpr uint32_t P(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x0a118000u : (i == 2 ? 0xd0000001u : (i == 3 ? 0x59aa76feu : (i == 4 ? 0x5c37b001u : (i == 5 ? 0x60b44d1eu : (i == 6 ? 0x9a2ca556u : (i == 7 ? 0x12ab655eu : 0u)))))))); }
    __host__ __device__ static constexpr uint32_t R2(int i) { return (i == 0 ? 0xb861857bu : (i == 1 ? 0x25d577bau : (i == 2 ? 0x8860591fu : (i == 3 ? 0xcc2c27b5u : (i == 4 ? 0xe5dc8593u : (i == 5 ? 0xa7cc008fu : (i == 6 ? 0xeff1c939u : (i == 7 ? 0x011fdae7u : 0u)))))))); }
    // subtractions of r that bring any 256-bit integer below r
    static constexpr int REDUCE_PASSES = 13;
};

struct Bls377Glv {
    static constexpr bool PSI = false;  // the endomorphism is phi below
    // phi(x, y) = (BETA * x, y) = LAMBDA * (x, y) on G1
    __host__ __device__ static constexpr uint32_t BETA_MONT(int i) { return (i == 0 ? 0x5a7b8727u : (i == 1 ? 0x2c766f92u : (i == 2 ? 0x253d58b5u : (i == 3 ? 0x03d7f6b0u : (i == 4 ? 0xec122131u : (i == 5 ? 0x838ec0deu : (i == 6 ? 0xf658bb10u : (i == 7 ? 0xbd5eb3e9u : (i == 8 ? 0x6ed3e52eu : (i == 9 ? 0x6942bd12u : (i == 10 ? 0xdd04ed6au : (i == 11 ? 0x01673786u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t LAMBDA(int i) { return (i == 0 ? 0x00000000u : (i == 1 ? 0x00000000u : (i == 2 ? 0x40000000u : (i == 3 ? 0x14885f32u : (i == 4 ? 0x5c37b001u : (i == 5 ? 0x60b44d1eu : (i == 6 ? 0x9a2ca556u : (i == 7 ? 0x12ab655eu : 0u)))))))); }
    // lattice basis (a1, b1), (a2, b2): a + b*lambda = 0 mod r
    static constexpr int A1_NEG = 0;
    __host__ __device__ static constexpr uint32_t A1(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B1_NEG = 1;
    __host__ __device__ static constexpr uint32_t B1(int i) { return (i == 0 ? 0x00000000u : (i == 1 ? 0x0a118000u : (i == 2 ? 0x90000001u : (i == 3 ? 0x452217ccu : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int A2_NEG = 0;
    __host__ __device__ static constexpr uint32_t A2(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x0a118000u : (i == 2 ? 0x90000001u : (i == 3 ? 0x452217ccu : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B2_NEG = 0;
    __host__ __device__ static constexpr uint32_t B2(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    // Babai multipliers: c1 = (k*G1 + 2^255) >> 256, c2 = (k*G2 + 2^255) >> 256
    __host__ __device__ static constexpr uint32_t G1(int i) { return (i == 0 ? 0x0000000eu : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    __host__ __device__ static constexpr uint32_t G2(int i) { return (i == 0 ? 0xaf90181eu : (i == 1 ? 0x7f72ed32u : (i == 2 ? 0x9fd37160u : (i == 3 ? 0xb3f7aa96u : (i == 4 ? 0x00000003u : 0u))))); }
    static constexpr int HALF_BITS = 126;  // |k1|, |k2| < 2^HALF_BITS
};

struct Bls377Gen {
    __host__ __device__ static constexpr uint32_t X_MONT(int i) { return (i == 0 ? 0x772451f4u : (i == 1 ? 0x260f33b9u : (i == 2 ? 0x169d5658u : (i == 3 ? 0xc54dd773u : (i == 4 ? 0x69a510ddu : (i == 5 ? 0x5c1551c4u : (i == 6 ? 0x425e1698u : (i == 7 ? 0x761662e4u : (i == 8 ? 0x6f065272u : (i == 9 ? 0xc97d78ccu : (i == 10 ? 0xb361fd4du : (i == 11 ? 0x00a41206u : 0u)))))))))))); }
    __host__ __device__ static constexpr uint32_t Y_MONT(int i) { return (i == 0 ? 0xb8cb81f3u : (i == 1 ? 0x8193961fu : (i == 2 ? 0x5f44adb8u : (i == 3 ? 0x00638d4cu : (i == 4 ? 0xd4daf54au : (i == 5 ? 0xfafaf3dau : (i == 6 ? 0xd655cd18u : (i == 7 ? 0xc27849e2u : (i == 8 ? 0x01d52814u : (i == 9 ? 0x2ec3ddb4u : (i == 10 ? 0x26303c71u : (i == 11 ? 0x007da933u : 0u)))))))))))); }
    static constexpr uint32_t B = 1u;
    // DBL_C^2 = 3b (DBL_NEG 0) or -3b (DBL_NEG 1): projective doubling chains
    static constexpr int DBL_NEG = 0;
    __host__ __device__ static constexpr uint32_t DBL_C_MONT(int i) { return (i == 0 ? 0x8894e1e4u : (i == 1 ? 0x3fabdfd0u : (i == 2 ? 0xcc1f55aau : (i == 3 ? 0xcbf921ddu : (i == 4 ? 0x460edc0cu : (i == 5 ? 0xd17deff1u : (i == 6 ? 0x7897028du : (i == 7 ? 0xd394e81eu : (i == 8 ? 0x0912681au : (i == 9 ? 0xc29c995du : (i == 10 ? 0xaff9d568u : (i == 11 ? 0x01515e6cu : 0u)))))))))))); }
};

// BN254 G2: GLV with psi(x, y) = (conj(x) * GAMMA1, conj(y) * GAMMA2) = LAMBDA * (x, y)
struct Bn254G2Glv {
    static constexpr bool PSI = true;
    __host__ __device__ static constexpr uint32_t GAMMA1_MONT(int i) { return (i == 0 ? 0x4563ab30u : (i == 1 ? 0xb5773b10u : (i == 2 ? 0xa9aa6454u : (i == 3 ? 0x347f91c8u : (i == 4 ? 0x242e0991u : (i == 5 ? 0x7a007127u : (i == 6 ? 0x118214ecu : (i == 7 ? 0x1956bcd8u : (i == 8 ? 0xa0aa4757u : (i == 9 ? 0x6e849f1eu : (i == 10 ? 0x89f89141u : (i == 11 ? 0xaa1c7b6du : (i == 12 ? 0xfae0ca3au : (i == 13 ? 0xb6e713cdu : (i == 14 ? 0x4e82ebc3u : (i == 15 ? 0x26694fbbu : 0u)))))))))))))))); }
    __host__ __device__ static constexpr uint32_t GAMMA2_MONT(int i) { return (i == 0 ? 0x2936b629u : (i == 1 ? 0xe4bbdd0cu : (i == 2 ? 0xe133bacbu : (i == 3 ? 0xbb30f162u : (i == 4 ? 0xf9645366u : (i == 5 ? 0x31a9d1b6u : (i == 6 ? 0xa500f8ddu : (i == 7 ? 0x253570beu : (i == 8 ? 0x5ffe77c7u : (i == 9 ? 0xa1d77ce4u : (i == 10 ? 0x7826d1dbu : (i == 11 ? 0x07affd11u : (i == 12 ? 0xbb7edc6bu : (i == 13 ? 0x6d16bd27u : (i == 14 ? 0x85defeccu : (i == 15 ? 0x2c872002u : 0u)))))))))))))))); }
    __host__ __device__ static constexpr uint32_t BETA_MONT(int) { return 0u; }  // unused (PSI)
    __host__ __device__ static constexpr uint32_t LAMBDA(int i) { return (i == 0 ? 0xe87cfd46u : (i == 1 ? 0xf83e9682u : (i == 2 ? 0xeeb859fbu : (i == 3 ? 0x6f4d8248u : (i == 4 ? 0x00000000u : (i == 5 ? 0x00000000u : (i == 6 ? 0x00000000u : (i == 7 ? 0x00000000u : 0u)))))))); }
    static constexpr int A1_NEG = 0;
    __host__ __device__ static constexpr uint32_t A1(int i) { return (i == 0 ? 0xe87cfd46u : (i == 1 ? 0xf83e9682u : (i == 2 ? 0xeeb859fbu : (i == 3 ? 0x6f4d8248u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B1_NEG = 1;
    __host__ __device__ static constexpr uint32_t B1(int i) { return (i == 0 ? 0x00000001u : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int A2_NEG = 0;
    __host__ __device__ static constexpr uint32_t A2(int i) { return (i == 0 ? 0xbe763ba7u : (i == 1 ? 0x9d797039u : (i == 2 ? 0x00000001u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int B2_NEG = 0;
    __host__ __device__ static constexpr uint32_t B2(int i) { return (i == 0 ? 0xa6f338efu : (i == 1 ? 0x95b806bcu : (i == 2 ? 0xeeb859fdu : (i == 3 ? 0x6f4d8248u : (i == 4 ? 0x00000000u : 0u))))); }
    __host__ __device__ static constexpr uint32_t G1(int i) { return (i == 0 ? 0xc8e01942u : (i == 1 ? 0x2cb62031u : (i == 2 ? 0xa773d2d5u : (i == 3 ? 0x4ccef014u : (i == 4 ? 0x00000002u : 0u))))); }
    __host__ __device__ static constexpr uint32_t G2(int i) { return (i == 0 ? 0x00000005u : (i == 1 ? 0x00000000u : (i == 2 ? 0x00000000u : (i == 3 ? 0x00000000u : (i == 4 ? 0x00000000u : 0u))))); }
    static constexpr int HALF_BITS = 127;  // |k1|, |k2| < 2^HALF_BITS
};

// BN254 G2 generator on the twist y^2 = x^3 + 3/(9 + u): c0 limbs, then c1 limbs
struct Bn254G2Gen {
    __host__ __device__ static constexpr uint32_t X_MONT(int i) { return (i == 0 ? 0x02bc2026u : (i == 1 ? 0x8e83b5d1u : (i == 2 ? 0x497b0172u : (i == 3 ? 0xdceb1935u : (i == 4 ? 0x97811adfu : (i == 5 ? 0xfbb82647u : (i == 6 ? 0xaf96503bu : (i == 7 ? 0x19573841u : (i == 8 ? 0xa84c6140u : (i == 9 ? 0xafb4737du : (i == 10 ? 0x5802d8c4u : (i == 11 ? 0x6043dd5au : (i == 12 ? 0x52a02f86u : (i == 13 ? 0x09e950fcu : (i == 14 ? 0x3aea7b6bu : (i == 15 ? 0x14fef083u : 0u)))))))))))))))); }
    __host__ __device__ static constexpr uint32_t Y_MONT(int i) { return (i == 0 ? 0x886be9f6u : (i == 1 ? 0x619dfa9du : (i == 2 ? 0xf59e9b78u : (i == 3 ? 0xfe7fd297u : (i == 4 ? 0x231b7dfeu : (i == 5 ? 0xff9e1a62u : (i == 6 ? 0xae9e4206u : (i == 7 ? 0x28fd7eebu : (i == 8 ? 0xc71856eeu : (i == 9 ? 0x64095b56u : (i == 10 ? 0x327d3cbbu : (i == 11 ? 0xdc57f922u : (i == 12 ? 0x33351076u : (i == 13 ? 0x55f935beu : (i == 14 ? 0x93fd6482u : (i == 15 ? 0x0da4a0e6u : 0u)))))))))))))))); }
};

}  // namespace zkmsm
