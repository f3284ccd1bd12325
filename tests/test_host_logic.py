"""Host-side logic of the Python layer that needs no GPU: the packed Z2 sample layout and the
quartic route chosen from the optimizer's arguments (sweep_driver.py:48-50)."""
from __future__ import annotations

import subprocess
from types import SimpleNamespace

import numpy as np
import pytest

from conftest import ROOT, load_records
from oracle import fg_phi4_oracle as O


def test_pack_z2_samples_inverts_the_dense_layout():
    from rcmps_b200 import objective
    rec = load_records("packed.npz")[4]
    Q = O.left_canonical_q(rec["R"], rec["K"])
    system = O.PackedZ2System(Q, rec["R"], rec["rho"])
    packed = rec["samples"]
    dense = np.stack([system.unpack(x) for x in packed])
    assert dense.shape[1] == 7 * 4 * 4 + 1
    np.testing.assert_array_equal(objective.pack_z2_samples(dense, 4), packed)


def test_route_from_optimizer_arguments():
    from rcmps_b200 import objective
    assert objective.settings_from_args(SimpleNamespace(packed_z2=True, reduced=False)).symmetry == objective.SYMMETRY_Z2
    assert objective.settings_from_args(SimpleNamespace(packed_z2=False, reduced=True)).symmetry == objective.SYMMETRY_NONE
    assert objective.settings_from_args(SimpleNamespace(window=20.0)).symmetry == objective.SYMMETRY_NONE
    with pytest.raises(ValueError):
        objective.settings_from_args(SimpleNamespace(packed_z2=True, reduced=True))
    s = objective.settings_from_args(None, symmetry=objective.SYMMETRY_AUTO)
    assert s.symmetry == 2


def test_validation_rows_and_refined_controls():
    from rcmps_b200 import validate
    assert [name for name, _ in validate.ROWS] == ["standard_cold", "standard_warm_1", "standard_warm_2",
                                                    "refined_512", "refined_1024"]
    assert validate.REFINED == dict(window=40.0, quadrature=1024, atol=1e-14, rtol=1e-13)
    with pytest.raises(ValueError):
        validate.source_integral(0.0)


def _run_host_program(tmp_path, header, body):
    """Compile and run `body` as main() against a host-only header of csrc."""
    src = tmp_path / "main.cpp"
    src.write_text(f'#include "{ROOT / "rcmpscore.jl_b200" / "csrc" / header}"\n#include <cstdio>\n{body}')
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=60).stdout.split()


def test_a_failed_capacity_query_is_asked_again(tmp_path):
    out = _run_host_program(tmp_path, "capacity.h", """
int main() {
  std::atomic<int> known{0};
  const int answers[] = {-1, 5, 7};
  int asked = 0;
  auto ask = [&] { return answers[asked++]; };
  for (int i = 0; i < 3; ++i) std::printf("%d ", rcmps::capacity_once(known, ask));
  std::atomic<int> none{0};
  int zeros = 0;
  for (int i = 0; i < 2; ++i) std::printf("%d ", rcmps::capacity_once(none, [&] { ++zeros; return 0; }));
  std::printf("%d %d", asked, zeros);
}""")
    assert out == ["0", "5", "5", "0", "0", "2", "1"]


def test_admission_of_launches(tmp_path):
    """One kind at a time up to its capacity, in the order of arrival."""
    out = _run_host_program(tmp_path, "capacity.h", """
#include <chrono>
#include <thread>
#include <vector>
int main() {
  rcmps::Admission gate;
  std::atomic<int> inside[3] = {}, broken{0};
  const int capacity[3] = {1, 5, 21};
  std::vector<std::thread> threads;
  for (int i = 0; i < 90; ++i)
    threads.emplace_back([&, i] {
      const int kind = i / 7 % 3, count = 1 + i % capacity[kind];
      gate.enter(kind, count, capacity[kind]);
      const int now = inside[kind] += count;
      if (now > capacity[kind] || inside[(kind + 1) % 3] || inside[(kind + 2) % 3]) ++broken;
      std::this_thread::sleep_for(std::chrono::milliseconds(2));
      inside[kind] -= count;
      gate.leave(count);
    });
  for (auto& t : threads) t.join();
  // a later launch of the kind inside does not overtake one of another kind
  gate.enter(2, 1, 21);
  std::atomic<int> order{0};
  int other = 0, same = 0;
  auto wait = [] { std::this_thread::sleep_for(std::chrono::milliseconds(200)); };
  std::thread a([&] { gate.enter(0, 1, 1); other = ++order; gate.leave(1); });
  wait();
  std::thread b([&] { gate.enter(2, 1, 21); same = ++order; gate.leave(1); });
  wait();
  const int early = order;
  gate.leave(1);
  a.join();
  b.join();
  std::printf("%d %d %d %d", (int)broken, early, other, same);
}""")
    assert out == ["0", "0", "1", "2"]


def test_the_benchmark_finds_the_traffic_of_its_default_launch():
    import bench
    per = bench.launch_traffic("d64_mixed", [1])
    assert 1e4 < per < 1e7
    assert bench.launch_traffic("d64_mixed", [3, 4]) == 7 * per
    assert bench.launch_traffic("no such workload", [1]) is None
