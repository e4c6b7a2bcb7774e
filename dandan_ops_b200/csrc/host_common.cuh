// Error text and launch counting shared by the translation units of the C ABI (defined in b2_w4a16.cu).
#pragma once
#include <cstdint>
#include <string>

namespace b2host {

int fail(int code, const std::string& msg);      // stores the calling thread's error text, returns `code`
int after_launch(const char* what);              // counts a launch and reports its error
int check_dims(int64_t n, int64_t k);

}  // namespace b2host
