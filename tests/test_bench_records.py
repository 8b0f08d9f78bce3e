"""bench.py's DRAM figure is reported only for the launch layout it was measured at."""
import importlib.util
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def _bench():
    spec = importlib.util.spec_from_file_location("bench_module", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_traffic_figure_follows_the_block_size(tmp_path):
    b = _bench()
    (tmp_path / "k_update_32x4_traffic.txt").write_text(
        f"kernel: k_update_quad\nblock: 224\nsource_digest: {b.update_kernel_digest()}\ndram_bytes_per_launch: 12345\n")
    where = ((32, 32, 32, 32), "k_update_quad", tmp_path)
    assert b.ncu_traffic_per_launch(*where, block=224)[0] == 12345
    assert b.ncu_traffic_per_launch(*where)[0] == 12345
    value, note = b.ncu_traffic_per_launch(*where, block=128)
    assert value is None and "224" in note and "128" in note


def test_committed_figure_names_its_block_size():
    text = (ROOT / "profiles" / "k_update_32x4_traffic.txt").read_text()
    assert any(line.startswith("block: ") for line in text.splitlines())
