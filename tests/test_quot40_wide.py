"""cpx_quot40_core and cpx_quot40_small for dividends up to 2^63, whose double is
rounded: the harness of test_quot40 with its bound of 2^53 raised, and operands
drawn between 2^53 and 2^63, exact multiples and their neighbours among them.
CPU only."""
import os
import subprocess

from test_quot40 import HARNESS, ROOT


def test_quot40_wide_dividends(tmp_path):
    src = HARNESS.replace("n >> 53", "n >> 63").replace(
        "        check(rnd() >> 24, d);\n",
        "        check(rnd() >> 24, d);\n"
        "        {\n"
        "            const int bn = 54 + (int)(rnd() % 10);  // dividend bit length 54 .. 63\n"
        "            const uint64_t n = (rnd() >> (64 - bn)) | (1ull << (bn - 1)), m = n / d * d;\n"
        "            for (int64_t o = -2; o <= 2; o++) {\n"
        "                check(n + o, d);\n"
        "                check(m + o, d);\n"
        "            }\n"
        "        }\n").replace("(1ull << 53) - 1, (1ull << 53) - 2", "(1ull << 53) - 1, (1ull << 63) - 3, (1ull << 62) + 1")
    assert src.count("bn = 54") == 1 and "n >> 63" in src
    f = tmp_path / "q.cpp"
    f.write_text(src)
    exe = tmp_path / "q"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "cudapix_b200", "csrc"), str(f), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), str(4 * 10**6)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout
