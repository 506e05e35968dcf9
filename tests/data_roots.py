"""Data roots with other grids than the synthetic library's: its first ages or pixels alone, in the package's own layout."""
import json

import numpy as np


def cut_root(root, data, nt=None, ns=None):
    """The synthetic library's first nt ages and ns pixels under root (its filters' responses cut with the pixels):
    the root and the library as synthdata.load reads it."""
    from libopensps_gb300 import synthdata
    nt, ns = nt or data["log_age"].size, ns or data["lambda"].size
    out = root / "synthetic"
    out.mkdir(parents=True)
    arrays = {"lambda": data["lambda"][:ns], "log_age": data["log_age"][:nt], "zlegend": data["zlegend"],
              "ssp_spec": data["ssp_spec"][:, :nt, :ns], "ssp_mass": data["ssp_mass"][:, :nt],
              "ssp_lbol": data["ssp_lbol"][:, :nt], "line_lambda": data["line_lambda"],
              "line_lum": data["line_lum"][:, :nt]}
    for nb in data["manifest"]["filter_sets"]:
        arrays[f"filters_{nb}"] = data[f"filters_{nb}"][:, :ns]
        arrays[f"filters_{nb}_center"] = data[f"filters_{nb}_center"]
    for name, a in arrays.items():
        np.ascontiguousarray(a, dtype="<f8").tofile(out / f"{name}.f64")
    (out / "manifest.json").write_text(json.dumps(dict(data["manifest"], ntfull=nt, nspec=ns), indent=1))
    return root, synthdata.load(root)
