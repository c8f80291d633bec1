"""The result line of the benchmark stays short enough for a reader that keeps the end of the output only."""
import json

import bench


def test_lists_leave_the_result_line():
    per = [{"layer": [512, 4608], "sparsity": 0.9, "V": 16, "us": 20.746666938066483, "useful_tflops": 17.831666604779354}] * 32
    keep = {"metric": "m", "value": 1.0, "config": {"workload": "w" * 700}, "roofline": {"frac": 0.5}, "e2e": {"value": 1.0},
            "encoder_layer": {"ms_sparse_weights": 0.5}, "sweep": {"matrices": 2000}}
    ref = {"ms_per_step": 11.6, "useful_tflops": 60.0, "per_product": per}
    line = {**keep, "comparators": {"cublas_dense_fp16": {"ms_per_step": 0.93}, "reference_gpu_kernel": ref}, "per_product": per,
            "per_product_note": "n", "svc": {"matrices": per}, "ffn": {"cases": per}}
    short, detail = bench.split_line(line)
    assert {k: short[k] for k in keep} == keep and set(short) == set(keep) | {"comparators"}
    assert short["comparators"] == {"cublas_dense_fp16": {"ms_per_step": 0.93}, "reference_gpu_kernel": {"ms_per_step": 11.6, "useful_tflops": 60.0}}
    assert detail["per_product"] == detail["reference_gpu_kernel_per_product"] == detail["svc"]["matrices"] == detail["ffn"]["cases"] == per
    assert len(json.dumps(short)) < 4096 and line["comparators"]["reference_gpu_kernel"] is ref
    assert bench.split_line({"metric": "m", "comparators": {"reference_gpu_kernel": {"unavailable": "x"}}})[0]["comparators"]
