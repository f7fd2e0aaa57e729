"""CPU test of the byte model behind the benchmark's roofline record (bench.algorithmic_bytes)."""
import pytest

import bench

INFO = dict(nxt=256, nyt=192, nzt=97, nz=97, nxt2=384, nyt2=288, lhx=129)


@pytest.mark.parametrize("s", [4, 8])
@pytest.mark.parametrize("gform", [False, True])
def test_batched_launches_carry_all_fields(s, gform):
    """The batched forward pass moves what the field-by-field one moves, in fewer launches."""
    b = lambda name, n=None: bench.algorithmic_bytes(name, INFO, s, n, gform)   # noqa: E731
    assert b("rows_fwd3", 1) == pytest.approx(4 * b("rows_fwd3", 4))
    assert b("rows_fwd3") == b("rows_fwd3", 4)
    assert b("cols_fwd", 1) == pytest.approx(4 * (b("pad_cols", 4) + b("ddy_cols", 4)) +
                                             (1 if gform else 3) * b("press_fwd_cols", 3))


@pytest.mark.parametrize("name", ["rows_fwd3", "cols_fwd", "pad_cols", "ddy_cols", "press_fwd_cols", "press_gform_cols",
                                  "tdma", "tdma_mixed", "tdma_reg", "tdma_staged", "tdma_seg_solve", "tdma_seg_finish",
                                  "pinv_cols", "pinv_rows_project"])
def test_every_field_sized_launch_of_a_step_is_counted(name):
    n = INFO["nxt"] * INFO["nyt"] * (INFO["nz"] - 1) * 4
    assert n < bench.algorithmic_bytes(name, INFO, 4, 1) < 40 * n
