"""What choose_shape() (csrc/matmul_shape.cuh) takes, as compiled for the host: the shapes of work that the GPU tests mean to run, and
the splits of K on which the accuracy of f32 results rests."""
import shutil
import subprocess
from pathlib import Path

import pytest

from deepforge_b200.dfgpu import E4M3, E5M2

ROOT = Path(__file__).resolve().parent.parent
SIXTEEN, CODES, SCALED = 0, 1, 2
TYPES = {"FLOAT": (0, 4), "HALF": (1, 2), "BFLOAT16": (2, 2), "E4M3": (E4M3, 1), "E5M2": (E5M2, 1)}
# M, K, N whose K is split where C is stored element by element: in 16 bits with rows off the 16-byte boundaries, and as E5M2.
DIRECT = {SIXTEEN: [(128, 512, 1280), (179, 336, 128), (256, 384, 128), (70, 200, 264)], CODES: [(128, 1024, 2688), (596, 528, 336), (78, 832, 2384)]}
# M, K, N with B [K, N] that two SMs take as tiles of 192 columns, 96 of them a CTA's. The last tile has all of them, 16 (none left for the
# second CTA), 80, 96 (the first CTA's all), 112 and 144; a second round of tiles; rows past 256 and K with a remainder throughout.
N_MAJOR_192 = {kind: [(1030, 1040, 2112), (1030, 528, 2128), (1030, 528, 2192), (1030, 528, 2208), (1030, 528, 2224), (1030, 1040, 2064), several]
               for kind, several in ((SIXTEEN, (3333, 528, 1808)), (CODES, (2050, 528, 4432)))}


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    folder = tmp_path_factory.mktemp("shape")
    source = folder / "shape.cpp"
    source.write_text("""#include <cstdio>
#include "matmul_shape.cuh"
int main() {
    dfgpu::Problem p{};
    int n_major, operands, direct;
    while (scanf("%d %ld %ld %ld %d %d %d %d %d", &p.kind, &p.M, &p.K, &p.N, &n_major, &p.out_dtype, &p.out_bytes, &operands, &direct) == 9) {
        p.direct_stores = direct != 0;
        p.b_mn_major = n_major != 0;
        p.in_bytes = dfgpu::sixteen_bits(p) ? 2 : 1;
        const dfgpu::Shape s = dfgpu::choose_shape(p, operands);
        printf("%d %d %d %d\\n", s.cg, s.bn, s.splits, s.k_per_split);
    }
}
""")
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "include"), "-I", str(ROOT / "deepforge_b200" / "csrc"), str(source), "-o", str(folder / "shape")], check=True)

    def ask(kind, m, k, n, n_major, c_type, operands=0, direct=False):
        dtype, size = TYPES[c_type]
        line = f"{kind} {m} {k} {n} {int(n_major)} {dtype} {size} {operands} {int(direct)}\n"
        return tuple(int(v) for v in subprocess.run([str(folder / "shape")], input=line, check=True, capture_output=True, text=True).stdout.split())
    return ask


@pytest.mark.parametrize("kind", sorted(N_MAJOR_192))
@pytest.mark.parametrize("c_type", ["BFLOAT16", "HALF"])
def test_n_major_columns_of_one_and_a_half_boxes(shapes, kind, c_type):
    for m, k, n in N_MAJOR_192[kind]:
        assert shapes(kind, m, k, n, True, c_type)[:3] == (2, 192, 1), (m, k, n)


@pytest.mark.parametrize("m,k,n,blocks", [(128, 384, 1152, 1), (128, 640, 3840, 3), (128, 896, 3712, 4), (128, 2048, 2688, 6), (128, 3328, 1536, 7)])
def test_f32_results_split_k(shapes, m, k, n, blocks):
    assert shapes(SIXTEEN, m, k, n, True, "FLOAT")[3] == blocks


@pytest.mark.parametrize("kind,m,k,n", [(SIXTEEN, 1, 136, 3648), (SIXTEEN, 2, 240, 3680), (SIXTEEN, 4, 184, 224), (SIXTEEN, 22, 288, 192), (SCALED, 7, 736, 2624), (SCALED, 15, 704, 2448)])
def test_few_blocks_are_not_worth_an_exchange(shapes, kind, m, k, n):
    assert shapes(kind, m, k, n, True, "BFLOAT16")[2] == 1


def test_a_full_operand_is_shared_out(shapes):
    assert [shapes(SIXTEEN, 128, 384, 384, True, "HALF", operands)[2] for operands in (0, 1)] == [1, 6]
    assert shapes(SIXTEEN, 1059, 368, 104, True, "BFLOAT16", 1)[2] > 1


def test_stores_element_by_element_are_shared_out(shapes):
    for kind, c_type in ((SIXTEEN, "HALF"), (CODES, "E5M2")):
        for m, k, n in DIRECT[kind]:
            assert shapes(kind, m, k, n, False, c_type, direct=True)[2] > 1, (m, k, n)
    assert shapes(CODES, 78, 912, 336, True, "E4M3")[2] > 1


@pytest.mark.parametrize("m,k,n,blocks", [(194, 5392, 2368, 15), (128, 2432, 6016, 10), (128, 1792, 3456, 4), (924, 1776, 288, 3)])
def test_amax_comes_from_no_longer_sums(shapes, m, k, n, blocks):
    """Blocks of 128 codes in an accumulator, as many as the accuracy of Amax_C was measured with."""
    assert shapes(CODES, m, k, n, False, "BFLOAT16")[3] <= blocks
