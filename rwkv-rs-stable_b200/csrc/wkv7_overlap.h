// When the scans of the two-kernel prefill run beside the operator kernel of the next segment.  Host arithmetic alone, no CUDA.
//
// The scan is one latency-bound CTA per chain (0.85 us per chunk), the operator kernel throughput work that fills every SM (2.8 us per
// chunk and SM).  On SM partitions the scans have `chains` SMs rounded up to eight and the operator kernel the rest.  Without, the
// operator kernel leaves as many SMs' worth of CTAs out as there are chains, and the scans, on a stream of higher priority, take the
// SMs that have no operator CTA (a scan CTA's 217 KB and an operator CTA's 57 KB do not fit one SM).  Measured (B200, 148 SMs; in
// sequence / on partitions; us):
//     chains x chunks    128          192          256          320          384          512          1024
//     4                               148 / 164    198 / 213    239 / 256
//     12                 125 / 132    177 / 185    228 / 238    280 / 286    334 / 330    439 / 423    864 / 799
//     16                 132 / 137    189 / 192    247 / 246    303 / 296    359 / 343    476 / 443    935 / 823
//     20                              201 / 202    264 / 253    327 / 305
//     24                              217 / 208    282 / 263    350 / 317    415 / 365    550 / 469    1098 / 867
//     32                              241 / 225    319 / 282    392 / 338    467 / 394    618 / 502    1237 / 923
//     40                              269 / 261    354 / 329    436 / 394
//     44                              282 / 291    374 / 370    458 / 447
//     48                              294 / 310    388 / 395    482 / 475
//     56                              324 / 368    425 / 471    527 / 576
// and with few chains, whose scans leave most of their partition idle:
//     chains x chunks    384          512          768          1024         1536         2048         4096
//     2                  268 / 289    359 / 375    522 / 546    686 / 722    1020 / 1058  1358 / 1392  2702 / 2738
//     3                  275 / 291    361 / 384    532 / 561    703 / 741    1049 / 1075  1392 / 1423  2774 / 2782
//     4                  285 / 298    369 / 389    544 / 566    721 / 746    1074 / 1086  1430 / 1430  2844 / 2816
//     5                  287 / 302    378 / 393    558 / 573    739 / 753    1102 / 1097  1465 / 1449  2918 / 2844
//     6                  294 / 307    388 / 399    573 / 579    756 / 759    1129 / 1112  1501 / 1466  3002 / 2858
//     7                  300 / 311    395 / 403    585 / 585    775 / 768    1156 / 1120  1538 / 1474  3074 / 2873
//     8                  307 / 314    404 / 405    598 / 590    795 / 776    1182 / 1124  1572 / 1480  3142 / 2889
//     10                 320 / 322    421 / 415    627 / 600    829 / 788    1239 / 1141  1646 / 1495  3289 / 2905
//     11                 327 / 324    430 / 418    639 / 603    849 / 792    1264 / 1142  1682 / 1506  3360 / 2914
// Without partitions (from a captured graph, where that is what runs; with kernels of other speeds): 24 x 256 274 us against 316 in
// sequence, 24 x 512 490 (623), 32 x 256 289 (361); with fewer than 24 chains it loses (12 x 512: 537 against 502).
#pragma once

#include <cstddef>

namespace rwkv7 {

inline bool partition_overlap_pays(size_t chains, size_t nchunks, int num_sms) {
    if (num_sms <= 0) return false;
    const size_t share = chains * 1000 / (size_t)num_sms;   // chains in thousandths of the SMs
    // from which share on, and then from how many chunks on
    constexpr struct { unsigned share, chunks; } kFrom[] = {{160, 192}, {130, 256}, {105, 320}, {74, 384}, {60, 512}, {50, 768}, {45, 1024}, {33, 1536}, {27, 4096}};
    for (const auto &from : kFrom)
        if (share >= from.share) return share <= 280 && nchunks >= from.chunks;
    return false;
}
// (the schedule without partitions, where they are not to be had: 16 to 27 % as many chains as SMs, from 256 chunks on)
inline bool shared_sm_overlap_pays(size_t chains, size_t nchunks, int num_sms) {
    return chains * 100 >= (size_t)num_sms * 16 && chains * 100 <= (size_t)num_sms * 27 && nchunks >= 256;
}

}  // namespace rwkv7
