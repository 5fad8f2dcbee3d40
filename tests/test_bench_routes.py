"""The benchmark's prefill entries ask for the routes that their labels name."""
import os
import re

import bench

HEADER = os.path.join(os.path.dirname(os.path.abspath(bench.__file__)), "include", "mldfc.h")


def _enum(name):
    return int(re.search(rf"\b{name}\s*=\s*(\d+)", open(HEADER).read()).group(1))


def test_labels_name_the_routes_they_time():
    inline, convert, auto = (_enum("MLD_PREFILL_ROUTE_" + n) for n in ("INLINE", "CONVERT", "AUTO"))
    assert bench.PREFILL_ROUTES == {"dequantised_inside_gemm": (inline, False, "inside"),
                                    "with_weight_conversion": (convert, False, "converted"),
                                    "weights_prepared_once": (auto, True, "cached"), "auto": (auto, False, None)}
    assert bench.PREFILL_ROUTE_NAMES == {_enum("MLD_ROUTE_PREFILL_INLINE"): "inside", _enum("MLD_ROUTE_PREFILL_CONVERTED"): "converted",
                                         _enum("MLD_ROUTE_PREFILL_CACHED"): "cached"}
