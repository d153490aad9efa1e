"""The few-token kernels' shares of a step: their sums at the limits that a registry accepts, and what the blocks walk."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("units") / "units_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", "-o", exe,
                    os.path.join(ROOT, "tests", "units_check.cpp")], check=True)

    def run(items, cnt, blocks, walk, *parts):
        r = subprocess.run([exe] + [str(v) for v in (items, cnt, blocks, walk) + sum(parts, ())], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        return int(r.stdout)
    return run


@pytest.mark.parametrize("parts", [((16, 40),), ((512, 12288), (512, 12288)), ((64, 1000), (0, 0), (8, 24), (128, 4096))], ids=str)
@pytest.mark.parametrize("items,cnt", [(1, 1), (3, 16), (70, 9)])
def test_every_column_of_every_item_once(units, items, cnt, parts):
    units(items, cnt, 1, 0, *parts)
    units(items, cnt, 7, 0, *parts)
    units(items, cnt, 296, 0, *parts)


@pytest.mark.parametrize("items,parts", [(800, ((256, 12288), (256, 12288))),      # 12,800 tokens in a registry of rank 256
                                         (560, ((256, 34816),)),
                                         (12864, ((512, 34816),)),                 # as many items as a registry's metadata holds
                                         (12864, ((512, 20000),) * 4),             # ... over more columns than the scale allows
                                         (12864, ((512, 65536),) * 4),
                                         (600, ((16, 40000000), (512, 1000)))], ids=str)
@pytest.mark.parametrize("blocks", [64, 296])
def test_sums_past_32_bits(units, items, parts, blocks):
    total = units(items, 16, blocks, 3, *parts)
    assert total > 2 ** 31
    assert total < 1.08e11


def test_usual_layers_keep_their_costs(units):
    # (2 x 21 + 4) a column at rank 64 and 16 tokens, up to 182,361 columns
    assert units(1, 16, 1, 0, (64, 12288), (64, 12288)) == 46 * 24576
    assert units(1, 16, 1, 0, (64, 182361)) == 46 * 182361
    assert units(1, 16, 1, 0, (64, 182362)) == 45 * 182362
