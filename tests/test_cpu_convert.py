"""The one-launch conversion's early exits, checked on its source: a block that
leaves a cooperative kernel while others go on to a barrier hangs them, so every
block has to find the same value in the word that an exit tests."""
import re

from conftest import ROOT

SOURCE = ROOT / "relaxmap_b200" / "csrc" / "rmx_convert.cu"


def test_word_of_an_exit_is_not_written_before_the_next_barrier():
    body = SOURCE.read_text().split("k_convert(", 1)[1]
    body = body[:body.index("\n}\n")]
    exits = list(re.finditer(r"if \(__ldcg\(a\.ctl \+ (\d+)\)\) return;", body))
    assert len(exits) == 2
    for e in exits:
        before = body[:e.start()].rstrip()
        assert before.endswith("grid.sync();")  # the word is complete when it is tested
        stretch = body[e.end():].split("grid.sync();", 1)[0]
        assert f"a.ctl[{e.group(1)}] =" not in stretch and f"a.ctl + {e.group(1)}," not in stretch
