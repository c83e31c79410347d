"""Numbers that the Python side and the CUDA sources of the selective scan both state."""
import re
from pathlib import Path

from mstar_b200 import ops
from mstar_b200.ops import build


def test_both_sides_cut_and_route_portions_alike():
    text = (Path(build.CSRC) / "selective_scan.cu").read_text()
    stated = {name: int(v) for name, v in re.findall(r"^#define (SCAN_\w+) (\d+)", text, flags=re.M)}
    assert stated["SCAN_CUT_FROM"] == ops.SCAN_CUT_FROM and stated["SCAN_FEW"] == ops.SCAN_FEW
    # the rank up to which ``selective_scan`` lets that kernel make the step sizes' product
    assert stated["SCAN_FEW_RANK"] == 256
    # scratch holds a piece for every started 64 tokens, as the shortest piece has
    assert ops.SCAN_CUT_FROM >= 64 and ops.scan_most_pieces(ops.SCAN_CUT_FROM) >= -(-ops.SCAN_CUT_FROM // 64)
