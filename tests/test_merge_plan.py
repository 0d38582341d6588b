"""Host arithmetic of the hit merge's plan (phx_merge.cuh), compiled for the CPU with the undefined-behaviour
checks of the host compiler: which key bytes the sort passes over."""
import os
import re
import subprocess

from tests.conftest import ROOT

SRC = os.path.join(ROOT, "opticks_b200", "csrc", "phx_merge.cuh")


def _extract(src, start):
    """the definition that opens with `start`, to its closing brace at column 0"""
    a = src.index(start)
    b = re.search(r"\n}(;?)\n", src[a:])
    return src[a:a + b.end()]


def test_key_bytes_in_use(tmp_path):
    src = open(SRC).read()
    main = r"""
#include <stdint.h>
#include <stdio.h>
#define __host__
#define __device__
%s
%s
int main(void)
{
    unsigned id, bk;
    while (scanf("%%u %%u", &id, &bk) == 2) {
        PhxMergeRange r = {};
        r.id_max = id; r.bk_max = bk;
        for (int b = 0; b < 8; b++) printf("%%d", phx_merge_byte_used(r, b) ? 1 : 0);
        printf("\n");
    }
}
""" % (_extract(src, "struct PhxMergeRange"), _extract(src, "__host__ __device__ inline bool phx_merge_byte_used"))
    cc = tmp_path / "plan.cc"
    cc.write_text(main)
    exe = str(tmp_path / "plan")
    subprocess.run(["g++", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover=all", str(cc), "-o", exe], check=True)
    vals = [0, 1, 0xFF, 0x100, 0xFFFF, 0x10000, 0xFFFFFFFF]
    cases = [(i, b) for i in vals if i <= 0xFFFF for b in vals]
    out = subprocess.run([exe], input="\n".join(f"{i} {b}" for i, b in cases), capture_output=True, text=True, check=True).stdout.split()
    for (i, b), got in zip(cases, out):
        k = (i << 48) | b
        # a byte is passed over only when it is zero in every key up to the largest bucket and identity
        want = "".join(str(int((b >> 8 * q) != 0 if q < 4 else q >= 6 and (i >> 8 * (q - 6)) != 0)) for q in range(8))
        assert got == want, (hex(k), got, want)
    engine = open(os.path.join(ROOT, "opticks_b200", "csrc", "phx_engine.cu")).read()
    assert "phx_merge_byte_used(range, b)" in engine
