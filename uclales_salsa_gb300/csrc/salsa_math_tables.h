// salsa_math_tables.h -- tables of salsa_math.cuh, from their definitions:
//   c_exp2_tab[j]  = round(2^(j/128) * 2^63),  j = 0..127
//   c_log_c[i]     = round(512 / m_i), m_i = 1 + (i + 1/2)/128 the middle of interval i of [1, 2);
//                    512 (c = 1) for the first interval and 256 (c = 1/2) for the last, so
//                    that arguments on either side of 1 keep log1p's relative accuracy
//   c_log_l[i]     = round(-ln(c_log_c[i] / 512) * 2^64); 0 for the first and last intervals
//                    (the last one's ln 2 is counted with the exponent)
#pragma once

namespace salsa {
namespace {
__device__ const unsigned long long c_exp2_tab[128] = {
    0x8000000000000000ull, 0x80b1ed4fd999ab6cull, 0x8164d1f3bc030773ull, 0x8218af4373fc25ecull,
    0x82cd8698ac2ba1d7ull, 0x8383594eefb6ee37ull, 0x843a28c3acde4046ull, 0x84f1f656379c1a29ull,
    0x85aac367cc487b15ull, 0x8664915b923fba04ull, 0x871f61969e8d1010ull, 0x87db357ff698d792ull,
    0x88980e8092da8527ull, 0x8955ee03618e5fddull, 0x8a14d575496efd9aull, 0x8ad4c6452c728924ull,
    0x8b95c1e3ea8bd6e7ull, 0x8c57c9c4646f4ddeull, 0x8d1adf5b7e5ba9e6ull, 0x8ddf042022e69cd6ull,
    0x8ea4398b45cd53c0ull, 0x8f6a8117e6c8e5c4ull, 0x9031dc431466b1dcull, 0x90fa4c8beee4b12bull,
    0x91c3d373ab11c336ull, 0x928e727d9531f9acull, 0x935a2b2f13e6e92cull, 0x9426ff0fab1c04b6ull,
    0x94f4efa8fef70961ull, 0x95c3fe86d6cc7fefull, 0x96942d3720185a00ull, 0x97657d49f17ab08eull,
    0x9837f0518db8a96full, 0x990b87e266c189aaull, 0x99e0459320b7fa65ull, 0x9ab62afc94ff864aull,
    0x9b8d39b9d54e5539ull, 0x9c6573682ec32c2dull, 0x9d3ed9a72cffb751ull, 0x9e196e189d472420ull,
    0x9ef5326091a111aeull, 0x9fd228256400dd06ull, 0xa0b0510fb9714fc2ull, 0xa18faeca8544b6e4ull,
    0xa27043030c496819ull, 0xa3520f68e802bb93ull, 0xa43515ae09e6809eull, 0xa5195786be9ef339ull,
    0xa5fed6a9b15138eaull, 0xa6e594cfeee86b1eull, 0xa7cd93b4e965356aull, 0xa8b6d5167b320e09ull,
    0xa9a15ab4ea7c0ef8ull, 0xaa8d2652ec907629ull, 0xab7a39b5a93ed337ull, 0xac6896a4be3fe929ull,
    0xad583eea42a14ac6ull, 0xae493452ca35b80eull, 0xaf3b78ad690a4375ull, 0xb02f0dcbb6e04584ull,
    0xb123f581d2ac2590ull, 0xb21a31a66618fe3bull, 0xb311c412a9112489ull, 0xb40aaea2654b9841ull,
    0xb504f333f9de6484ull, 0xb60093a85ed5f76cull, 0xb6fd91e328d17791ull, 0xb7fbefca8ca41e7cull,
    0xb8fbaf4762fb9ee9ull, 0xb9fcd2452c0b9debull, 0xbaff5ab2133e45fbull, 0xbc034a7ef2e9fb0dull,
    0xbd08a39f580c36bfull, 0xbe0f6809860993e2ull, 0xbf1799b67a731083ull, 0xc0213aa1f0d08db0ull,
    0xc12c4cca66709456ull, 0xc238d2311e3d6673ull, 0xc346ccda24976407ull, 0xc4563ecc5334cb33ull,
    0xc5672a115506daddull, 0xc67990b5aa245f79ull, 0xc78d74c8abb9b15dull, 0xc8a2d85c8ffe2c45ull,
    0xc9b9bd866e2f27a3ull, 0xcad2265e4290774eull, 0xcbec14fef2727c5dull, 0xcd078b86503dcdd2ull,
    0xce248c151f8480e4ull, 0xcf4318cf191918c1ull, 0xd06333daef2b2595ull, 0xd184df6251699ac6ull,
    0xd2a81d91f12ae45aull, 0xd3ccf099859ac379ull, 0xd4f35aabcfedfa1full, 0xd61b5dfe9f9bce07ull,
    0xd744fccad69d6af4ull, 0xd870394c6db32c84ull, 0xd99d15c278afd7b6ull, 0xdacb946f2ac9cc72ull,
    0xdbfbb797daf23755ull, 0xdd2d818508324c20ull, 0xde60f4825e0e9124ull, 0xdf9612deb8f04420ull,
    0xe0ccdeec2a94e111ull, 0xe2055afffe83d369ull, 0xe33f8972be8a5a51ull, 0xe47b6ca0373da88dull,
    0xe5b906e77c8348a8ull, 0xe6f85aaaee1fce22ull, 0xe8396a503c4bdc68ull, 0xe97c38406c4f8c57ull,
    0xeac0c6e7dd24392full, 0xec0718b64c1cbddcull, 0xed4f301ed9942b84ull, 0xee990f980da3025bull,
    0xefe4b99bdcdaf5cbull, 0xf13230a7ad094509ull, 0xf281773c59ffb13aull, 0xf3d28fde3a641a5bull,
    0xf5257d152486cc2cull, 0xf67a416c733f846eull, 0xf7d0df730ad13bb9ull, 0xf92959bb5dd4ba74ull,
    0xfa83b2db722a033aull, 0xfbdfed6ce5f09c49ull, 0xfd3e0c0cf486c175ull, 0xfe9e115c7b8f884cull};
__device__ const unsigned short c_log_c[128] = {
    512, 506, 502, 498, 495, 491, 487, 484, 480, 477, 473, 470, 466, 463, 460, 457,
    454, 450, 447, 444, 441, 438, 435, 433, 430, 427, 424, 421, 419, 416, 413, 411,
    408, 406, 403, 401, 398, 396, 394, 391, 389, 387, 384, 382, 380, 378, 376, 373,
    371, 369, 367, 365, 363, 361, 359, 357, 355, 353, 351, 350, 348, 346, 344, 342,
    340, 339, 337, 335, 334, 332, 330, 329, 327, 325, 324, 322, 320, 319, 317, 316,
    314, 313, 311, 310, 308, 307, 306, 304, 303, 301, 300, 299, 297, 296, 295, 293,
    292, 291, 289, 288, 287, 286, 284, 283, 282, 281, 279, 278, 277, 276, 275, 274,
    272, 271, 270, 269, 268, 267, 266, 265, 264, 263, 262, 261, 260, 259, 258, 256};
__device__ const unsigned long long c_log_l[128] = {
    0x0000000000000000ull, 0x0304891471145544ull, 0x050caa4966033027ull, 0x0718f4bb052abc63ull,
    0x08a4f1f2002d4675ull, 0x0ab8ae2601e77772ull, 0x0cd0c3dab9ef3dd2ull, 0x0e65b9e6eed965c3ull,
    0x108598b59e3a0689ull, 0x12207b5c78549d8dull, 0x14485e03dbdfad47ull, 0x15e95a4d9791cb7dull,
    0x18197e2f40e3f01cull, 0x19c0c32d4d25483full, 0x1b6ac88dad5b1be0ull, 0x1d17978821936434ull,
    0x1ec739830a111fccull, 0x210b316b3c740d11ull, 0x22c19004964f6169ull, 0x247ae25493840349ull,
    0x2637329a749f098full, 0x27f68b4b32519714ull, 0x29b8f712f7838f37ull, 0x2ae6f9920319baa8ull,
    0x2cae9d7d182673e3ull, 0x2e79720e9fa29957ull, 0x304782caa3478377ull, 0x3218db73f979b283ull,
    0x3350ef1bd75470faull, 0x3527da7915b3c6deull, 0x37022e617047a41aull, 0x384051562ff368f9ull,
    0x3a206fe4cabcf6b0ull, 0x3b627b61a912806bull, 0x3d48893e0955e916ull, 0x3e8e96269be451b6ull,
    0x407ab9589b1a43ddull, 0x41c4e181356189ceull, 0x4310b59d858b8c46ull, 0x45059fbcd9de0c08ull,
    0x4655b4ee6f0be97cull, 0x47a7859e2267d151ull, 0x49a58844d36e49e1ull, 0x4afbc1f3724d4e7dull,
    0x4c53c7874d738ec3ull, 0x4dad9ddaf8445bb3ull, 0x4f0949dcccc60ed5ull, 0x511647814e7d22d5ull,
    0x52769fcef3107b33ull, 0x53d8dfaeea603ea7ull, 0x553d0c6def86a255ull, 0x56a32b6efb7e8386ull,
    0x580b422bc247afa4ull, 0x5975563533802a8aull, 0x5ae16d33fe8ff33bull, 0x5c4f8ce91a85ee6dull,
    0x5dbfbb2e51c5d2eeull, 0x5f31fdf6d1a8367cull, 0x60a65b4fbe2f2ad5ull, 0x616155ddb72feab8ull,
    0x62d8e6a22cb7d28full, 0x6452a18d6fda2653ull, 0x65ce8d0c4d5ab73bull, 0x674cafa857b4ec31ull,
    0x68cd100893e9e323ull, 0x698e197eaf43af76ull, 0x6b11e3408141bc0full, 0x6c97fbed832cb830ull,
    0x6d5be81118a42549ull, 0x6ee5846e038bec2eull, 0x707181a4fe8e7640ull, 0x713866e11c8f0692ull,
    0x72c8034b3ad90b9eull, 0x745a13527d1ab9daull, 0x7524091b7be9add8ull, 0x76b9d521325856f5ull,
    0x785228689c9b3653ull, 0x791f474cb99df866ull, 0x7abb74bab26430cfull, 0x7b8a855ad04f93faull,
    0x7d2a9fb80c64b379ull, 0x7dfbab9ad5d87300ull, 0x7f9fc63ac0f4f857ull, 0x8072d72d903d588cull,
    0x821b05f3b01d6774ull, 0x82f0260d51603018ull, 0x83c5f8299e2b4091ull, 0x8573b71682a7d21bull,
    0x864ba644a18e6e05ull, 0x87fdaa109d23aef7ull, 0x88d7c11e3ad53cdcull, 0x89b29295f8432617ull,
    0x8b6a69c608cfd3afull, 0x8c47720791e53314ull, 0x8d2539c5bd19e2b1ull, 0x8ee30cef034a20dbull,
    0x8fc31afe30b2c6dfull, 0x90a3edd23d1c9d58ull, 0x9267e737c06cd34aull, 0x934b1089a6dc93c2ull,
    0x942f0421651c1c4eull, 0x9513c36876083696ull, 0x96dfaabd86fa1647ull, 0x97c6d5b1b19bccd0ull,
    0x98aed221a03458b6ull, 0x9997a18a56bcad28ull, 0x9b6bbf4e9a7eb5faull, 0x9c5710b8cbb73a43ull,
    0x9d433b392b888970ull, 0x9e304061b5fda919ull, 0x9f1e21c8c7bb62b3ull, 0xa00ce1092e5498c3ull,
    0xa1ecff97c91e267bull, 0xa2de62326449d0a3ull, 0xa3d0a93f45169a4bull, 0xa4c3d6706d5d83edull,
    0xa5b7eb7cb860fb89ull, 0xa6acea1fed5d0f66ull, 0xa7a2d41ad270c9d7ull, 0xa899ab333fe2b9caull,
    0xa991713433c2b999ull, 0xaa8a27ede5eb13adull, 0xab83d135dc633301ull, 0xac7e6ee700261c70ull,
    0xad7a02e1b24efd32ull, 0xae768f0be1ae2ad0ull, 0xaf74155120c9011cull, 0x0000000000000000ull};
}  // namespace
}  // namespace salsa
