"""Child process of tuner tests (the tuner's memory is per process): one
calculation per kernel named on the command line, in order, of a seeded case
whose sizes come as JSON first; prints the list of {kernel_used, counts'
checksums} as JSON."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

from analisi_gb300 import engine, workloads  # noqa: E402

if __name__ == "__main__":
    c = json.loads(sys.argv[1])
    w = workloads.small_case(c["seed"], sum(c["counts"]), c["frames"], c["edge"], 0.15,
                             c["counts"], **c["params"])
    p = w["params"]
    out = []
    with engine.Engine(0) as e:
        e.set_frames(w["positions"], w["boxes"], w["type_ids"], w["ntypes"])
        for kernel in sys.argv[2:]:
            n = e.run(p["rmin"], p["rmax"], p["nbin"], p["tmax"], p["skip"], p["every"],
                      p["ntimesteps"], p["primo"], kernel=kernel)
            weight = 1 + np.arange(n.size, dtype=np.uint64)
            out.append({"kernel_used": e.stats()["kernel_used"], "sum": int(n.sum()),
                        "weighted": int((n.ravel() * weight).sum())})  # modulo 2^64
    print(json.dumps(out))
