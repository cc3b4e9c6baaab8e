// quant_check.cu — the encoders' float quantisers (tcb_resid.cuh: QuantPos)
// against the integer rules they stand for, on the CPU: every quantiser step of
// every QP and band with every lambda that goes with it, every coefficient
// that an 8-bit residual can have, and the level's reconstruction.  Also the
// closed form of the bit model's last-position part.  Exit code 0 when all
// match.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "../oracle/tcoracle.h"
#include "../tcodec_b200/csrc/tcb_resid.cuh"

using namespace tcb;

static long long bad = 0, checked = 0;

// The kernels' level: code_area's expressions, with the round-down add that
// takes the integer part written as floor.
static int level_of(const QuantPos &q, int a) {
    return (float)a >= q.thr ? (int)floorf(fmaf((float)a, q.r, q.off)) : 0;
}

static void check(int eff, long long lambda, bool rdoq) {
    QuantPos q(eff, rdoq ? lambda : 0);
    if (!rdoq) q.bias = (float)(eff >> 1);
    for (int c = 0; c <= 2047; ++c) {
        int want = (c + eff / 3) / eff;
        if (c == 0) want = 0;
        if (rdoq) {
            if (want != (c ? or_quant(c, eff) : 0) || or_quant(-c, eff) != -want) ++bad;
            if (want == 1) {
                const int d = or_dequant(1, eff);
                if ((long long)c * c + lambda < (long long)(c - d) * (c - d) + 2 * lambda) want = 0;
            }
        }
        const int got = level_of(q, c);
        const int dq = rdoq ? or_dequant(want, eff) : want ? want * eff + (eff >> 1) : 0;
        const float gdq = got ? fmaf((float)got, q.eff, q.bias) : 0.0f;
        bad += got != want || gdq != (float)dq || dq > 4800;
        ++checked;
    }
}

int main() {
    for (int qp = 0; qp < 64; ++qp)
        for (int band = 0; band < 4; ++band) {
            const int eff = or_eff_scale(qp, band);
            const long long lam = or_lambda(qp);
            check(eff, lam, true);               // inter frames, chroma
            check(eff, lam * 3 / 4, true);       // key frames' luma
            check(eff, 0, false);                // the 8x8 block path
        }
    for (int last = -1; last < 64; ++last) {
        // an area whose only level is 1 at `last`: 1 + 2, a term per position, the position's cost
        int want = last < 0 ? 1 : 1 + 2 + last + 4;
        want += last < 0 ? 1 : last < 4 ? 3 + last : 6;
        if (last >= 4) want += 2 * (int)floor(log2((double)(last - 4 + 1))) + 1;
        const int got = last_bits(last) + (last >= 0 ? 5 : 0);
        bad += got != want;
        ++checked;
    }
    printf("checked %lld, mismatches %lld\n", checked, bad);
    return bad ? 1 : 0;
}
