"""The benchmark's tables of what a kernel has to move name launchers that exist."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def launchers():
    text = (ROOT / "delta_b200" / "kernels" / "ops.py").read_text()
    return set(re.findall(r'_stream\(\)\),\s*"(\w+)"', text))


def test_launchers_that_do_anothers_work_exist():
    import bench
    known = launchers()
    assert "attention_rows_mma" in known and len(known) > 50
    for name, other in bench.SAME_WORK.items():
        assert name in known and other in known, (name, other)


def test_every_table_names_launchers():
    """A key that no launcher is counted under gives no fraction."""
    text = (ROOT / "bench.py").read_text()
    body = text[text.index("def design_workload("):text.index("def main()")]
    keys = set(re.findall(r'^\s+"([\w ]+)": \(.*\),', body, re.M)) - {"library batched product"}
    assert len(keys) > 20 and keys <= launchers(), keys - launchers()
    mevulix = body[body.index("def mevulix_work"):]
    mevulix = mevulix[:mevulix.index("if design ==")]
    assert "n_att" not in re.search(r'"attention_rows_mma": (.*)', mevulix).group(1) and "n_att" in re.search(r'"attention_rows_tc": (.*)', mevulix).group(1)
