// Generated by gen_fixed_tables.py; do not edit.
#pragma once
namespace mpgb {
namespace fx {
constexpr uint64_t kLog2e63 = 0xb8aa3b295c17f0bcull;  // log2(e), 63 fraction bits
constexpr uint64_t kE1 = 0x0b17217f7d1cf79bull;  // 64 fraction bits
constexpr uint64_t kE2 = 0x003d7f7bff058b1dull;  // 64 fraction bits
constexpr uint64_t kE3 = 0x0000e35846b82506ull;  // 64 fraction bits
constexpr uint32_t kE4 = 0x4ecaadbfu;  // 53 fraction bits
constexpr uint32_t kE5 = 0x00aec3ffu;  // 53 fraction bits
constexpr uint32_t kE6 = 0x00014309u;  // 53 fraction bits
constexpr uint32_t kE7 = 0x00000200u;  // 53 fraction bits
constexpr uint64_t kL1 = 0x1000000000000000ull;  // 64 fraction bits
constexpr uint64_t kL2 = 0x0080000000000000ull;  // 64 fraction bits
constexpr uint64_t kL3 = 0x0005555555555555ull;  // 64 fraction bits
constexpr uint64_t kL4 = 0x0000400000000000ull;  // 64 fraction bits
constexpr uint32_t kL5 = 0x66666666u;  // 53 fraction bits
constexpr uint32_t kL6 = 0x05555555u;  // 53 fraction bits
constexpr uint32_t kL7 = 0x00492492u;  // 53 fraction bits
constexpr uint32_t kL8 = 0x00040000u;  // 53 fraction bits
constexpr uint32_t kL9 = 0x000038e4u;  // 53 fraction bits
constexpr uint32_t kL10 = 0x00000333u;  // 53 fraction bits
// 2^(-j/32), 63 fraction bits (1 as the largest value below it).
MPGB_FX_TABLE uint64_t kExpTab[32] = {
    0x7fffffffffffffffull, 0x7d41d96db915019dull, 0x7a92be8a92436616ull, 0x77f25ccdee6d7ae6ull,
    0x75606373ee921c97ull, 0x72dc8373be41a454ull, 0x70666f76154a7089ull, 0x6dfddbcbed791babull,
    0x6ba27e656b4eb57aull, 0x69540ec8f895722dull, 0x6712460a8fc24072ull, 0x64dcdec3371793d1ull,
    0x62b39508aa836d6full, 0x6096266533384a2bull, 0x5e8451cfac061b5full, 0x5c7dd7a3b17dcf75ull,
    0x5a827999fcef3242ull, 0x5891fac0e95612c8ull, 0x56ac1f752150a563ull, 0x54d0ad5a753e077cull,
    0x52ff6b54d8a89c75ull, 0x513821818624b40cull, 0x4f7a993048d088d7ull, 0x4dc69cdceaa72a9cull,
    0x4c1bf828c6dc54b8ull, 0x4a7a77d47f7b84b1ull, 0x48e1e9b9d588e19bull, 0x47521cc5a2e6a9e0ull,
    0x45cae0f1f545eb73ull, 0x444c0740496d4294ull, 0x42d561b3e6243d8aull, 0x4166c34c5615d0ecull,
};
// inv: the smallest multiple of 2^-31 not below 1 / (1 + j/32), 31 fraction bits;
// lg: -log(inv), 63 fraction bits.
struct alignas(16) LogEntry { uint64_t lg; uint32_t inv, pad; };
MPGB_FX_TABLE LogEntry kLogTab[32] = {
    {0x0000000000000000ull, 0x80000000u, 0u},
    {0x03f05361bf06600aull, 0x7c1f07c2u, 0u},
    {0x07c28c2f7458a999ull, 0x78787879u, 0u},
    {0x0b78694462b5a5cfull, 0x75075076u, 0u},
    {0x0f1383b6d57972f5ull, 0x71c71c72u, 0u},
    {0x129552f6fff5234dull, 0x6eb3e454u, 0u},
    {0x15ff30701793d3c9ull, 0x6bca1af3u, 0u},
    {0x19525a9bc456b478ull, 0x6906906au, 0u},
    {0x1c8ff7c6da9a21adull, 0x66666667u, 0u},
    {0x1fb9186ca63e2a8eull, 0x63e7063fu, 0u},
    {0x22ceb956b74c1c08ull, 0x61861862u, 0u},
    {0x25d1c575b23a6138ull, 0x5f417d06u, 0u},
    {0x28c3178378bd84fbull, 0x5d1745d2u, 0u},
    {0x2ba37b7d501394a3ull, 0x5b05b05cu, 0u},
    {0x2e73afec47a00d3bull, 0x590b2165u, 0u},
    {0x3134670c7a84b56cull, 0x572620afu, 0u},
    {0x33e647d87f3097e6ull, 0x55555556u, 0u},
    {0x3689eef7311ec51aull, 0x5397829du, 0u},
    {0x391fef8ec5344358ull, 0x51eb851fu, 0u},
    {0x3ba8d4086b89417full, 0x50505051u, 0u},
    {0x3e251ebefe0dd967ull, 0x4ec4ec4fu, 0u},
    {0x40954a960f43fb1bull, 0x4d4873edu, 0u},
    {0x42f9cb8fc4aa0adbull, 0x4bda12f7u, 0u},
    {0x45530f4b1357a6a7ull, 0x4a7904a8u, 0u},
    {0x47a17d78410340faull, 0x4924924au, 0u},
    {0x49e5784866c46bb1ull, 0x47dc11f8u, 0u},
    {0x4c1f5ccc2c42f880ull, 0x469ee585u, 0u},
    {0x4e4f834d08a866a7ull, 0x456c797eu, 0u},
    {0x50763f9fb9cab993ull, 0x44444445u, 0u},
    {0x5293e176a8faec09ull, 0x4325c53fu, 0u},
    {0x54a8b4978f16abbdull, 0x42108422u, 0u},
    {0x56b5012ee67cb3f0ull, 0x41041042u, 0u},
};
}  // namespace fx
}  // namespace mpgb
