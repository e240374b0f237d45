"""Rules by which the host picks a kernel's form, run here as they stand in the sources."""
import re
import subprocess
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "kinetics_b200" / "csrc"


def _program(folder, source):
    (folder / "rule.cpp").write_text(source)
    subprocess.run(["g++", "-std=c++17", "-o", str(folder / "rule"), str(folder / "rule.cpp")], check=True)

    def ask(cases):
        text = "\n".join(" ".join(map(str, c)) for c in cases)
        out = subprocess.run([str(folder / "rule")], input=text, capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in out.stdout.splitlines()]
    return ask


@pytest.fixture(scope="module")
def wide(tmp_path_factory):
    """lf_wide of the recurrent step as a program: block, blocks and rows to 0 or 1, and the shared memory of either form."""
    text = (CSRC / "layers" / "ktl_lru.cu").read_text()
    parts = [re.search(p, text, re.S | re.M).group(0) for p in (
        r"^constexpr int kLfRows = [^\n]*\n", r"^[^\n]* int lf_ld\([^\n]*\n", r"^[^\n]* int lf_smem\([^\n]*\n", r"^static bool lf_wide\(.*?^}\n")]
    source = ("#include <cstdint>\n#include <cstdio>\n#define __host__\n#define __device__\nstruct ktk_lru { int blocks, block_stride; };\n"
              "static int sm_count() { return 148; }\n" + "".join(parts) +
              'int main() { int b, n, r; while (scanf("%d %d %d", &b, &n, &r) == 3) {\n'
              '    const ktk_lru a{n, b};\n    printf("%d %d %d\\n", (int)lf_wide(a, (r + kLfRows - 1) / kLfRows), lf_smem(b, 32), lf_smem(b, 64)); } }\n')
    return _program(tmp_path_factory.mktemp("wide"), source)


def test_wide_recurrent_steps_only_where_they_take_less(wide):
    cases = [(block, blocks, rows) for block in range(8, 513, 8) for blocks in (1, 3, 16, 40, 128) for rows in (1, 33, 128, 256, 1000)]
    for (block, blocks, rows), (chosen, narrow_smem, wide_smem) in zip(cases, wide(cases)):
        assert 2 * (narrow_smem + 1024) <= 228 * 1024                        # the narrow form always has two CTAs on an SM
        if chosen:
            groups = (rows + 31) // 32
            ctas = [groups * blocks * -(-block // chan) for chan in (32, 64)]
            assert 2 * (wide_smem + 1024) <= 228 * 1024 and ctas[1] < ctas[0] and ctas[0] > 2 * 148, (block, blocks, rows)
    # measured: block, blocks, rows
    assert [c for c, _, _ in wide([(256, 16, 128), (128, 32, 256), (64, 40, 256), (96, 64, 128), (200, 20, 256)])] == [1] * 5
    assert [c for c, _, _ in wide([(512, 8, 256), (304, 12, 256), (32, 64, 256), (24, 128, 256), (200, 20, 128), (256, 16, 64)])] == [0] * 6


def test_decode_steps_over_shared_rows_are_balanced_only_where_that_is_faster(tmp_path):
    text = (CSRC / "layers" / "ktl_attn_shared.cu").read_text()
    parts = [re.search(p, text, re.S | re.M).group(0) for p in (
        r"^constexpr int kAsTok = [^\n]*\n", r"^constexpr int kAsMinTiles = [^\n]*\n", r"^constexpr int kAsMaxSplits = [^\n]*\n",
        r"^struct Packing [^\n]*\n", r"^__host__ __device__ inline Packing packing_of\(.*?^}\n", r"^static int64_t splits_cost\(.*?^}\n",
        r"^static int balanced_ctas\(.*?^}\n", r"^bool attn_shared_balanced\(.*?^}\n")]
    ask = _program(tmp_path, "#include <cstdint>\n#include <cstdio>\n#define __host__\n#define __device__\nstruct ktk_attn { int heads; };\n"
                   "static int sm_count() { return 148; }\n" + "".join(parts) +
                   'int main() { int h, b, k; while (scanf("%d %d %d", &h, &b, &k) == 3) printf("%d\\n", '
                   "(int)attn_shared_balanced(ktk_attn{h}, b, k)); }\n")
    # heads, sequences, longest: measured at 576 columns, even and ragged lists
    by_sequence = [(8, 1, 16384), (16, 1, 600), (16, 1, 16384), (16, 4, 5000), (16, 16, 600), (16, 16, 5000), (16, 48, 2000), (32, 1, 16384),
                   (32, 4, 4000), (32, 16, 4000), (32, 128, 600), (32, 1, 32768), (128, 8, 8192), (128, 150, 1000), (128, 128, 2000),
                   (128, 64, 2000), (32, 0, 100), (32, 70000, 4000)]
    balanced = [(16, 32, 16384), (16, 128, 4096), (32, 100, 4000), (32, 128, 4096), (32, 150, 2000), (32, 64, 16384), (128, 64, 16384),
                (128, 150, 4000)]
    assert [c for c, (x,) in zip(by_sequence, ask(by_sequence)) if x] == []
    assert [c for c, (x,) in zip(balanced, ask(balanced)) if not x] == []


# rows, columns, inner size, gated: measured with weights that are not in L2
FASTER_HERE = {
    torch.float32: [(1, 512, 512, False), (4, 768, 512, False), (4, 1024, 512, True), (4, 512, 1024, False), (16, 512, 512, False),
                    (4, 4096, 4096, False), (16, 4096, 4096, False), (16, 12288, 4096, False), (8, 12288, 4096, True), (1, 4096, 4096, True)],
    torch.bfloat16: [(4, 768, 4096, False), (4, 1536, 4096, False), (8, 768, 4096, False), (1, 1536, 1024, False), (4, 1536, 4096, True),
                     (4, 3200, 5120, True), (8, 1536, 4096, True), (16, 1024, 1024, True), (16, 512, 512, True)]}
FASTER_THERE = {
    torch.float32: [(1, 8, 16384, False), (1, 64, 16384, False), (1, 512, 4096, False), (1, 1024, 2560, False), (1, 32, 16384, True),
                    (1, 128, 8192, True), (2, 32, 16384, False), (16, 32, 12288, False), (16, 4096, 256, False), (16, 8192, 1024, True),
                    (12, 12288, 1024, False), (8, 12288, 256, False), (8, 4096, 128, False)],
    torch.bfloat16: [(4, 8, 256, False), (4, 128, 16384, False), (8, 64, 256, False), (8, 1536, 4096, False), (8, 1024, 16384, False),
                     (8, 4096, 1024, True), (4, 6144, 1024, True), (4, 8192, 640, True), (16, 1024, 256, True), (16, 1536, 512, True)]}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_products_by_rows_only_where_they_are_faster(dtype):
    from kinetics_b200 import ops
    assert [c for c in FASTER_HERE[dtype] if not ops.linear_rows_wins(c[0], c[1], c[2], dtype, c[3])] == []
    assert [c for c in FASTER_THERE[dtype] if ops.linear_rows_wins(c[0], c[1], c[2], dtype, c[3])] == []
    assert not any(ops.linear_rows_wins(r, 512, k, dtype, g) for r, k in ((0, 512), (17, 512), (4, 500)) for g in (False, True))
