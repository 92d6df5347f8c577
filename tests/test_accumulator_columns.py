"""The matrix instructions of the float32 product, read from its source: instructions of different shapes run in no particular order,
so those that add into the same columns of tensor memory have one shape and one accumulator."""

import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "acorninfer_b200" / "csrc" / "gemm_f32_tc.cu"


def test_instructions_of_different_shapes_have_columns_of_their_own():
    text = SOURCE.read_text()
    number = lambda name: int(re.search(rf"#define {name} (\d+)", text).group(1))
    NT = number("F3_NT")
    columns = {name: int(eval(size.replace("NT", str(NT)))) for name, size in
               re.findall(r"\b(I\d) = IDESC \| \(\(uint32_t\)\(([\d\* ]*NT) >> 3\) << 17\)", text)}
    calls = re.findall(r"umma_bf16_elect\((d[^,]*), [^;]*?, (I\d), ([^;]*)\);", text)
    assert len(columns) >= 2 and len(calls) >= 3
    ranges = set()
    for place, shape, _ in calls:
        for k in range(4):
            first = eval(place, {"d": 0, "k": k, "NT": NT})
            ranges.add((first, first + columns[shape]))
    ranges = sorted(ranges)
    for (a0, a1), (b0, b1) in zip(ranges, ranges[1:]):
        assert a1 <= b0, f"columns {b0} .. {a1 - 1} belong to accumulators of two shapes"
    sums = eval(re.search(r"#define F3_SUMS \(([^)]*)\)", text).group(1).replace("F3_NT", str(NT)))
    assert ranges[-1][1] <= sums and 2 * sums <= number("F3_TMEM_COLS") <= 512
