// What the genotypes and the graph near a meiosis say about toggling it, for
// 32 loci at a time (the M-sweep's kernel, and the host's check of it).
#pragma once

#include <stdint.h>

#include "sl_internal.h"

#ifdef __CUDACC__
#define SL_HD __host__ __device__ __forceinline__
#else
#define SL_HD inline
#endif

namespace sl {

// Adds to the masks of meiosis_flips (sl_host.cc) for meiosis m = (i, p), o
// being i's other parent; a mask has a bit per locus.  The founder alleles that
// p's and o's two alleles have at a locus are those of the children that
// inherited them there and of p's and o's parents.  Members outside i's
// descendants that are homozygous fix their allele's colour (such alleles are
// fixed before anything is propagated); full sibs of i that are heterozygous
// below a homozygous o tell the colour of p's allele; the other allele of a
// heterozygous p or o has the opposite one.  The moving allele's colour shows
// in i, or in a homozygous child of i that has it.
//   same:  both of p's alleles are fixed to one colour by homozygous members
//          that do not move; never: the allele moved to has the other colour
//          than the moving one (see meiosis_flips for why either decides).
// entry(r), code0(r), code1(r): relative r's entry and the two bits of its
// genotype codes; meiosis(b): meiosis b's indicators; t: m's own.  Words for 32
// loci, so a relative costs a dozen logical operations; the loci left to
// evaluate fall from 7.4% to 4.6% (120 members, 5% of the genotypes missing) and
// from 6.2% to 3.2% (400 members).
template <class Entry, class Code0, class Code1, class Meiosis>
SL_HD void relatives_rule(int m, int F, uint32_t t, Entry entry, Code0 code0, Code1 code1, Meiosis meiosis,
                          uint32_t* same, uint32_t* never) {
    struct Codes {
        uint32_t a, b, h;   // homozygous A, homozygous B, heterozygous
    };
    auto codes = [&](int r) {
        const uint32_t c0 = code0(r), c1 = code1(r);
        return Codes{c1 & ~c0, c1 & c0, c0 & ~c1};
    };
    const Codes i = codes(0), p = codes(1), o = codes(2), p0 = codes(3), p1 = codes(4), o0 = codes(5), o1 = codes(6);
    // colours of p's alleles 0 and 1: fixed by homozygous members (d), told otherwise (k); of o's alleles
    uint32_t dA0 = p0.a, dB0 = p0.b, dA1 = p1.a, dB1 = p1.b, kA0 = 0, kB0 = 0, kA1 = 0, kB1 = 0;
    uint32_t oA0 = o.a | o0.a, oB0 = o.b | o0.b, oA1 = o.a | o1.a, oB1 = o.b | o1.b;
    uint32_t tA = i.a, tB = i.b;   // the moving allele's
#ifdef __CUDACC__
#pragma unroll 1
#endif
    for (int r = 7; r < kRelatives; ++r) {
        const uint32_t en = entry(r);
        if (en == kNoRelative) break;
        const Codes k = codes(r);
        const int b0 = 2 * ((int)(en & 0xffffu) - F);
        if (en & kRelOfP) {
            const uint32_t s = meiosis(b0 + (int)((en >> 20) & 1u));
            dA1 |= s & k.a;
            dB1 |= s & k.b;
            dA0 |= ~s & k.a;
            dB0 |= ~s & k.b;
            if (en & kRelOfO) {
                kB1 |= s & k.h & o.a;
                kA1 |= s & k.h & o.b;
                kB0 |= ~s & k.h & o.a;
                kA0 |= ~s & k.h & o.b;
            }
        }
        if (en & kRelOfO) {
            const uint32_t s = meiosis(b0 + (int)((en >> 21) & 1u));
            oA1 |= s & k.a;
            oB1 |= s & k.b;
            oA0 |= ~s & k.a;
            oB0 |= ~s & k.b;
        }
        if (en & kRelOfI) {
            uint32_t s = meiosis(b0 + (int)((en >> 22) & 1u));   // which of i's alleles the child has
            if (!(m & 1)) s = ~s;
            tA |= s & k.a;
            tB |= s & k.b;
        }
    }
    const uint32_t v = meiosis(m ^ 1);   // which of o's alleles i has
    const uint32_t wA = (v & (oA1 | (o.h & oB0))) | (~v & (oA0 | (o.h & oB1)));
    const uint32_t wB = (v & (oB1 | (o.h & oA0))) | (~v & (oB0 | (o.h & oA1)));
    tA |= i.h & wB;
    tB |= i.h & wA;
    kA0 |= dA0;
    kB0 |= dB0;
    kA1 |= dA1;
    kB1 |= dB1;
    // the allele moved to: p's allele 0 where the meiosis's indicator is 1
    const uint32_t bA = (t & (kA0 | (p.h & kB1))) | (~t & (kA1 | (p.h & kB0)));
    const uint32_t bB = (t & (kB0 | (p.h & kA1))) | (~t & (kB1 | (p.h & kA0)));
    *never |= ((bA & tB) | (bB & tA)) & ~*same;
    *same |= ((dA0 & dA1) | (dB0 & dB1)) & ~*never;
}

}  // namespace sl
