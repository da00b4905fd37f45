"""The rules that pick a direct sum's form by how its targets and sources fill the SMs
(gravhopper_gb300/csrc/shape_rules.h), built for the host, against forces timed on a GB300
(152 SMs) with every form: the choice is never slower than the plainer rule that each
replaces, by more than two runs of one form differ (1 %)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 152

# FP64 force of N particles, ordered kernel with 2, 4, 5, 7 and 8 targets per CTA, in us
FORMS = (2, 4, 5, 7, 8)
ORDERED = {
    304: (22.2, 22.1, 21.9, 24.4, 26.9), 400: (28.5, 26.6, 26.3, 28.8, 33.2), 500: (33.0, 31.1, 30.5, 34.2, 38.0),
    608: (38.1, 35.1, 34.9, 39.2, 44.0), 700: (47.8, 47.6, 39.3, 44.5, 50.0), 800: (52.5, 52.5, 53.5, 49.9, 56.1),
    912: (58.9, 58.7, 61.0, 55.6, 62.7), 1000: (72.4, 63.8, 65.7, 60.1, 66.8), 1064: (75.5, 66.9, 69.0, 62.7, 70.6),
    1200: (84.8, 74.4, 76.8, 95.6, 79.0), 1216: (84.9, 75.0, 77.3, 96.8, 80.2),
    1300: (109.6, 98.2, 82.7, 103.2, 117.2), 1400: (118.2, 105.8, 88.3, 111.0, 124.8),
    1520: (126.9, 113.8, 94.7, 119.6, 136.2), 1600: (188.4, 118.2, 128.0, 124.8, 142.9),
    1700: (200.2, 125.8, 138.1, 133.4, 151.1), 1800: (212.9, 132.1, 145.1, 140.4, 159.7),
    1824: (224.4, 133.7, 146.3, 140.4, 160.7), 1900: (235.2, 168.6, 152.8, 147.1, 167.2),
    2000: (246.8, 178.0, 160.3, 154.7, 175.2), 2128: (276.4, 187.7, 169.7, 164.3, 185.0),
    2200: (285.8, 195.0, 175.0, 224.7, 192.6), 2300: (297.2, 202.5, 225.7, 236.0, 201.7),
    2432: (314.6, 214.0, 240.1, 249.0, 212.4), 2500: (349.5, 272.4, 246.9, 257.6, 292.2),
    2700: (378.5, 293.9, 266.5, 276.3, 316.4), 2900: (451.5, 314.7, 285.2, 294.6, 338.6),
    3000: (466.5, 325.7, 294.4, 305.2, 349.8), 3192: (593.2, 454.2, 389.0, 323.6, 370.1),
    3300: (629.2, 470.0, 402.3, 413.4, 382.0), 3500: (671.7, 497.8, 427.3, 438.1, 407.4),
    3648: (699.9, 551.5, 442.9, 454.2, 423.6), 3800: (762.4, 583.9, 462.7, 474.4, 538.7),
    4000: (844.0, 615.8, 614.0, 498.3, 568.0), 4256: (898.9, 700.2, 655.1, 528.4, 602.2),
    4500: (1033, 757.2, 693.0, 680.3, 638.9), 4864: (1244, 819.7, 824.1, 734.7, 688.9),
    5200: (1410, 973.1, 880.8, 785.8, 887.7), 5500: (1557, 1150, 1038, 1025, 941.0),
    6000: (1826, 1258, 1134, 1121, 1024), 6500: (2168, 1541, 1368, 1367, 1524),
    7000: (2489, 1752, 1652, 1612, 1637), 8000: (3235, 2289, 2097, 1884, 1871),
    10000: (4873, 3470, 3235, 2916, 2933), 12000: (7164, 4924, 4672, 4152, 3895),
    16000: (12465, 8670, 8017, 7313, 7129),
}


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("rules") / "shape_rules_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "shape_rules_check.cpp")],
                   check=True)

    def ask(lines):
        r = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, timeout=60, check=True)
        return [int(v) for v in r.stdout.split()]

    return ask


def test_ordered_targets(choose):
    gains = 0
    for n, t in zip(ORDERED, choose([f"ordered {n} {SMS}" for n in ORDERED])):
        us = dict(zip(FORMS, ORDERED[n]))
        plain = us[next((q for q in (8, 4) if -(-n // q) >= 2 * SMS), 2)]
        assert us[t] <= 1.01 * plain, (n, t)
        gains += us[t] < 0.9 * plain
    assert gains > 10  # and a tenth faster at many sizes


def test_ordered_targets_any_size(choose):
    sizes = list(range(1, 7000, 7)) + [10 ** 6, 10 ** 9, 2 ** 40]
    got = choose([f"ordered {n} {sms}" for sms in (1, 132, SMS) for n in sizes])
    assert len(got) == 3 * len(sizes) and set(got) <= set(FORMS)
