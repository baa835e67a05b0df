"""Records tests/golden/step_paths.npz: the cases of tests/test_step_paths_gpu.py
run by the parity build of the package under --package-root.  The committed
file was recorded with a built checkout of commit a5ab038 (see the test).

    python tests/golden/make_step_paths.py --package-root DIR [--out FILE]
"""
import argparse
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(os.path.dirname(HERE))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--package-root", required=True)
    ap.add_argument("--out", default=os.path.join(HERE, "step_paths.npz"))
    args = ap.parse_args()
    root = os.path.abspath(args.package_root)
    sys.path.insert(0, os.path.join(REPO, "tests"))
    sys.path.insert(0, root)
    import dustyfargoadsg_b200 as fb
    from test_step_paths_gpu import CASES, run_case
    assert os.path.dirname(os.path.dirname(os.path.abspath(fb.__file__))) == root
    arrays = {}
    for name in sorted(CASES):
        res = run_case(fb, name, "parity")
        print(name, "substeps", res["substeps"], "stream", res.get("stream"),
              "finite", all(np.all(np.isfinite(v)) for v in res.values()), flush=True)
        arrays.update({"%s/%s" % (name, k): np.asarray(v) for k, v in res.items()})
    np.savez_compressed(args.out, **arrays)
    print("wrote %s, %d bytes" % (args.out, os.path.getsize(args.out)))


if __name__ == "__main__":
    main()
