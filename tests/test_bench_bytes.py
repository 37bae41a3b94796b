"""The bytes that bench.py counts once for the fused stage: what its four stages
read and write of a grid."""
import bench


def test_fused_stage_bytes():
    nv = 10 * 4 ** 5 + 2
    ne, nt = 3 * nv - 6, 2 * nv - 4
    records = nt * (16 + 16 + 4) + nv * (6 * 16 + 3 * 4) + ne * 8
    words = 0
    for stage in range(4):
        words += 1                   # the stage's input
        words += stage > 0           # y_n, which is the input of stage 0
        words += stage > 0           # the accumulator, read
        words += stage < 3           # and written
        words += 1                   # the stage's output
    once = records + (nv + ne) * 4 * words / 4
    kb = bench.kernel_bytes(nv, ne, nt, "fp32", 1, fused=True)
    assert kb["cell"] == once and sum(kb.values()) == once
    assert abs(once / nv - 272) < 0.1
    # what moves is more: the tiles' rims are read twice
    assert 1.0 < bench.TRAFFIC_PER_CELL["k_stage32"] * nv / once < 1.25
